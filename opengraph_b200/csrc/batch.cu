// batch.cu -- batched traversals over one device graph.
//
// Multi-source BFS (no reference counterpart; each lane must equal the
// reference's single-root BFS depths, BFS.c:476-626): up to 64 searches at
// once, one bit-lane per root.  Per vertex, three 64-bit words: the lanes
// that have visited it, the lanes whose frontier holds it, and the lanes that
// reach it in the level being built.  A level is either
//  * push (top-down): a warp takes 32 vertices of the frontier list and walks
//    their out-edges as one sequence (each lane finds its edge's vertex by a
//    search through shuffles); rows of more than kMsLong edges are cut into
//    pieces, a warp each in a second kernel.  Each edge ORs the frontier word of
//    its source, minus the target's visited lanes, into the target's next word
//    (64-bit atomicOr);
//  * pull (bottom-up): every vertex with a lane still unvisited ORs the
//    frontier words of its in-neighbours, stopping once every unvisited lane
//    is covered; rows of at most kMsLight in-edges by a thread (four edges
//    per step), longer rows by a warp;
// then one dense pass turns the next words into the new frontier, sets the
// visited lanes, writes the depths of the lanes each vertex gained (a warp
// per vertex row, coalesced) and counts the new frontier and its out-edges; the
// pass's last CTA chooses the next level's direction.  The level loop's state
// stays on the device: the host launches kMsBatch levels at a time (three
// kernels each, which return at once when the search has ended) and looks only
// then, where a look per level cost a wait of 15 us.
// Depths are u16 per (vertex, lane), row-major by vertex (128 bytes per
// vertex, 0xFFFF = unreached).  The search is level-synchronous in every
// lane, so every lane's depths are those of a single-root BFS.
#include "graph.cuh"

#include <algorithm>
#include <vector>

namespace ogb {

constexpr uint32_t kMsLight = 32;    // pull: rows up to this many in-edges by one thread
constexpr uint32_t kMsAlpha = 14;    // push while the frontier's out-edges < E / kMsAlpha
constexpr uint32_t kMsLong = 512;    // push: rows of more out-edges go in pieces of this many
// Levels launched between two looks of the host; the levels of the last batch after
// the search's end are launched for nothing.  us of a 64-root search with 1, 2, 4 and 8:
// RMAT-20 1090, 1020, 970 and 950; RMAT-16 390, 298, 271 and 240; 300 x 300 grid (600
// levels) 18400, 13800, 10600 and 9100.
constexpr int kMsBatch = 4;
constexpr uint32_t kMsMaxLevels = 0xFFFE;

struct MsCtl {
  // the frontier the next level starts from
  uint32_t nlist;
  uint32_t pull;               // direction of the next level
  uint32_t done;               // 1: the frontier is empty, 2: too many levels
  uint32_t levels, push_levels, pull_levels;  // levels finished, by direction
  unsigned long long mf;       // out-edges of the frontier
  // counted by the level in progress
  uint32_t next_n, items, ctas;  // vertices found, row pieces, CTAs finished
  uint32_t pad;
  unsigned long long next_mf;
  // of the whole search
  unsigned long long reached;  // (vertex, lane) pairs reached after the roots
  unsigned long long edges;    // edges read
};

// Direction of the level that starts from the frontier in c, or its end.
__device__ __forceinline__ void ms_next_level(MsCtl& c, uint32_t E) {
  if (c.nlist == 0) {
    c.done = 1;
  } else if (c.levels >= kMsMaxLevels) {
    c.done = 2;
  } else {
    c.pull = c.mf < (unsigned long long)E / kMsAlpha ? 0u : 1u;
  }
}

struct MsWork {
  uint32_t V = 0, heavy_build = 0;
  bool heavy_ready = false;
  DevBuf F, N, vis, list, items, heavy, ctl, roots;
  uint32_t n_heavy = 0;
  MsCtl* h_ctl = nullptr;
  cudaEvent_t ev_init = nullptr, ev0 = nullptr, ev1 = nullptr;
  ~MsWork() {
    if (h_ctl) cudaFreeHost(h_ctl);
    if (ev_init) cudaEventDestroy(ev_init);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
  }
};

void ms_work_free(MsWork* w) { delete w; }

// ------------------------------------------------------------ kernels ------

__global__ void msk_roots(const uint32_t* __restrict__ verts, const unsigned long long* __restrict__ masks,
                          uint32_t n, unsigned long long* __restrict__ F, unsigned long long* __restrict__ vis,
                          uint16_t* __restrict__ depth, uint32_t* __restrict__ list,
                          const uint32_t* __restrict__ out_degree, uint32_t E, MsCtl* __restrict__ ctl) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t v = verts[i];
    const unsigned long long m = masks[i];
    F[v] = m;
    vis[v] = m;
    list[i] = v;
    unsigned long long b = m;
    while (b) {
      const int lane = __ffsll((long long)b) - 1;
      depth[(size_t)v * 64 + lane] = 0;
      b &= b - 1;
    }
    atomicAdd(&ctl->mf, (unsigned long long)out_degree[v]);
  }
  __syncthreads();  // one CTA: mf is complete
  if (threadIdx.x == 0) {
    __threadfence();
    ctl->nlist = n;
    ctl->mf = atomicAdd(&ctl->mf, 0ull);
    ms_next_level(*ctl, E);
  }
}

// Push of the edges of the frontier word f: four targets at once.
__device__ __forceinline__ void ms_push4(const unsigned long long* f, const uint32_t* w, const bool* ok,
                                         const unsigned long long* vis, unsigned long long* N) {
  unsigned long long m[4];
#pragma unroll
  for (int k = 0; k < 4; k++) m[k] = ok[k] ? f[k] & ~vis[w[k]] : 0ull;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (m[k]) atomicOr(&N[w[k]], m[k]);
}

// The level's edges, by its direction: push over the frontier list, or pull
// over the vertices (blocks [0, nb_heavy): the vertices with more than kMsLight
// in-edges, a warp each, lanes strided, the warp's OR checked every 128 edges;
// the rest: a thread per vertex, four in-edges per step, until every unvisited
// lane is covered).
__global__ void __launch_bounds__(256) msk_expand(uint32_t V, unsigned long long lanes, uint32_t nb_heavy,
                                                  const uint32_t* __restrict__ heavy, uint32_t n_heavy,
                                                  const uint2* __restrict__ rows_f, const uint32_t* __restrict__ nbr_f,
                                                  const uint2* __restrict__ rows_i, const uint32_t* __restrict__ nbr_i,
                                                  const unsigned long long* F, const unsigned long long* vis,
                                                  unsigned long long* N, const uint32_t* list, uint4* items,
                                                  MsCtl* ctl) {
  wait_for_prior_kernel();
  let_next_kernel_start();
  if (ctl->done) return;
  const uint32_t lane = lane_id();
  const uint32_t gw = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (!ctl->pull) {
    const uint32_t n = ctl->nlist, nw = gridDim.x * (blockDim.x / 32);
    for (uint64_t i0 = (uint64_t)gw * 32; i0 < n; i0 += (uint64_t)nw * 32) {
      uint32_t u = 0;
      uint2 r = make_uint2(0u, 0u);
      unsigned long long fu = 0;
      if (i0 + lane < n) {
        u = list[i0 + lane];
        r = rows_f[u];
        fu = F[u];
      }
      if (r.y > kMsLong) {
        const uint32_t np = (r.y + kMsLong - 1) / kMsLong, at = atomicAdd(&ctl->items, np);
        for (uint32_t c = 0; c < np; c++)
          items[at + c] = make_uint4(u, r.x + c * kMsLong, r.x + min(r.y, (c + 1) * kMsLong), 0u);
        r.y = 0;
      }
      uint32_t ex = r.y;
#pragma unroll
      for (int k = 1; k < 32; k <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, ex, k);
        if (lane >= (uint32_t)k) ex += y;
      }
      const uint32_t total = __shfl_sync(0xffffffffu, ex, 31);
      ex -= r.y;
      for (uint32_t e0 = 0; e0 < total; e0 += 128) {
        unsigned long long f[4];
        uint32_t w[4];
        bool ok[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t e = e0 + k * 32 + lane;
          uint32_t p = 0;  // last vertex whose first edge is at or before e
#pragma unroll
          for (int step = 16; step; step >>= 1) {
            const uint32_t first = __shfl_sync(0xffffffffu, ex, p + step);
            if (first <= e) p += step;
          }
          const uint32_t from = __shfl_sync(0xffffffffu, r.x - ex, p) + e;
          f[k] = __shfl_sync(0xffffffffu, fu, p);
          ok[k] = e < total;
          w[k] = ok[k] ? (__ldg(&nbr_f[from]) & 0x3FFFFFFFu) : 0u;
        }
        ms_push4(f, w, ok, vis, N);
      }
    }
    return;
  }
  uint32_t edges = 0;
  if (blockIdx.x < nb_heavy) {
    const uint32_t nw = nb_heavy * (blockDim.x / 32);
    for (uint32_t t = gw; t < n_heavy; t += nw) {
      const uint32_t v = heavy[t];
      const unsigned long long pending = lanes & ~vis[v];
      if (!pending) continue;
      const uint2 r = rows_i[v];
      const uint32_t end = r.x + r.y;
      unsigned long long acc = 0;
      uint32_t j = r.x;
      for (; j < end; j += 128) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t jj = j + k * 32 + lane;
          if (jj < end) acc |= F[__ldg(&nbr_i[jj]) & 0x3FFFFFFFu];
        }
        // the warp's OR
        unsigned int lo = (unsigned int)acc, hi = (unsigned int)(acc >> 32);
        lo = __reduce_or_sync(0xffffffffu, lo);
        hi = __reduce_or_sync(0xffffffffu, hi);
        acc = ((unsigned long long)hi << 32) | lo;
        if ((acc & pending) == pending) {
          j += 128;
          break;
        }
      }
      if (lane == 0) {
        edges += min(j, end) - r.x;
        const unsigned long long m = acc & pending;
        if (m) N[v] = m;
      }
    }
    if (lane == 0 && edges) atomicAdd(&ctl->edges, (unsigned long long)edges);
    return;
  }
  const uint32_t nb = gridDim.x - nb_heavy;
  for (uint32_t v = (blockIdx.x - nb_heavy) * blockDim.x + threadIdx.x; v < V; v += nb * blockDim.x) {
    const unsigned long long pending = lanes & ~vis[v];
    if (!pending) continue;
    const uint2 r = rows_i[v];
    if (r.y == 0 || r.y > kMsLight) continue;
    unsigned long long acc = 0;
    uint32_t j = r.x;
    const uint32_t end = r.x + r.y;
    for (; j < end; j += 4) {
      unsigned long long f[4];
#pragma unroll
      for (int k = 0; k < 4; k++) f[k] = (j + k < end) ? F[__ldg(&nbr_i[j + k]) & 0x3FFFFFFFu] : 0ull;
      acc |= f[0] | f[1] | f[2] | f[3];
      if ((acc & pending) == pending) {
        j += 4;
        break;
      }
    }
    edges += min(j, end) - r.x;
    const unsigned long long m = acc & pending;
    if (m) N[v] = m;
  }
  warp_atomic_add_total64(&ctl->edges, edges);
}

// push: the pieces of the long rows, a warp each
__global__ void __launch_bounds__(256) msk_push_long(const uint4* items, const uint32_t* __restrict__ nbr_f,
                                                     const unsigned long long* F, const unsigned long long* vis,
                                                     unsigned long long* N, const MsCtl* ctl) {
  wait_for_prior_kernel();
  let_next_kernel_start();
  if (ctl->done || ctl->pull) return;
  const uint32_t n = ctl->items, lane = lane_id();
  const uint32_t nw = gridDim.x * (blockDim.x / 32);
  for (uint32_t t = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); t < n; t += nw) {
    const uint4 it = items[t];
    const unsigned long long fu = F[it.x];
    const unsigned long long f[4] = {fu, fu, fu, fu};
    const uint32_t len = it.z - it.y;  // counted from it.y: the piece may end just below 2^32
    for (uint32_t j = lane; j < len; j += 128) {
      uint32_t w[4];
      bool ok[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        ok[k] = j + k * 32 < len;
        w[k] = ok[k] ? (__ldg(&nbr_f[it.y + j + k * 32]) & 0x3FFFFFFFu) : 0u;
      }
      ms_push4(f, w, ok, vis, N);
    }
  }
}

// Next words -> new frontier: visited lanes, the depths of the newly reached
// lanes, the frontier list and its out-edges.  N is left all zero.  A warp
// covers 32 consecutive vertices; for each of them that gained lanes, the
// whole warp writes its depths (lane l: depth lanes l and l + 32 of the
// vertex's 128-byte row, 2-byte stores, no read -- every (vertex, lane) is
// written once).  The last CTA makes the counted frontier the next level's.
__global__ void __launch_bounds__(256) msk_finish(uint32_t V, uint32_t E, unsigned long long* F, unsigned long long* N,
                                                  unsigned long long* vis, uint16_t* depth,
                                                  const uint32_t* __restrict__ out_degree, uint32_t* list, MsCtl* ctl) {
  wait_for_prior_kernel();
  let_next_kernel_start();
  if (ctl->done) return;
  __shared__ BlockAppend<1024> q;
  __shared__ unsigned long long s_red[8];
  ba_init(q);
  const uint16_t level = (uint16_t)(ctl->levels + 1);
  const uint32_t lane = lane_id();
  unsigned long long mf = 0;
  uint32_t reached = 0;
  for (uint32_t base = blockIdx.x * 1024; base < V; base += gridDim.x * 1024) {
    const uint32_t wb = base + (threadIdx.x & ~31u);
    unsigned long long nx[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) nx[k] = wb + k * 256 + lane < V ? N[wb + k * 256 + lane] : 0ull;
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) {
      const uint32_t w0 = wb + k * 256, v = w0 + lane;
      unsigned long long n = 0;
      if (v < V) {
        if (nx[k]) {
          const unsigned long long vi = vis[v];
          n = nx[k] & ~vi;
          N[v] = 0;
          if (n) {
            vis[v] = vi | n;
            mf += out_degree[v];
            reached += __popcll(n);
            ba_push(q, v);
          }
        }
        F[v] = n;
      }
      uint32_t has = __ballot_sync(0xffffffffu, n != 0);
      while (has) {
        const uint32_t j = (uint32_t)__ffs(has) - 1;
        has &= has - 1;
        const unsigned long long f = __shfl_sync(0xffffffffu, n, j);
        uint16_t* row = depth + (size_t)(w0 + j) * 64;
        if ((f >> lane) & 1ull) row[lane] = level;
        if ((f >> (lane + 32)) & 1ull) row[lane + 32] = level;
      }
    }
    if (ba_size(q)) ba_flush(q, list, &ctl->next_n);
  }
  block_add_total<unsigned long long>(&ctl->next_mf, mf, s_red);
  block_add_total<unsigned long long>(&ctl->reached, (unsigned long long)reached, s_red);
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&ctl->ctas, 1u) == gridDim.x - 1) {
      __threadfence();
      MsCtl c;
      c.nlist = atomicAdd(&ctl->next_n, 0u);
      c.mf = atomicAdd(&ctl->next_mf, 0ull);
      c.levels = ctl->levels + 1;
      c.done = 0;
      c.pull = ctl->pull;
      if (c.pull) {
        ctl->pull_levels++;
      } else {
        ctl->push_levels++;
        ctl->edges += ctl->mf;  // a push level reads every out-edge of its frontier
      }
      ms_next_level(c, E);
      ctl->nlist = c.nlist;
      ctl->mf = c.mf;
      ctl->levels = c.levels;
      ctl->pull = c.pull;
      ctl->next_n = 0;
      ctl->next_mf = 0;
      ctl->items = 0;
      ctl->ctas = 0;
      ctl->done = c.done;
    }
  }
}

// vertices with more than kMsLight in-edges (built once per graph)
__global__ void msk_heavy_list(uint32_t V, const uint2* __restrict__ rows, uint32_t* __restrict__ heavy,
                               uint32_t* __restrict__ count) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    if (rows[v].y > kMsLight) heavy[warp_atomic_inc(count)] = v;
}

// ------------------------------------------------------------ driver -------

static int ms_work_get(DevGraph& g, MsWork** out, cudaStream_t s) {
  if (!g.ms) g.ms = new MsWork();
  MsWork* w = g.ms;
  const uint32_t V = g.V;
  if (w->V != V || !w->F.p) {
    OGB_TRY(w->F.alloc((size_t)V * 8 + 16));
    OGB_TRY(w->N.alloc((size_t)V * 8 + 16));
    OGB_TRY(w->vis.alloc((size_t)V * 8 + 16));
    OGB_TRY(w->list.alloc((size_t)V * 4 + 16));
    OGB_TRY(w->heavy.alloc((size_t)V * 4 + 16));
    OGB_TRY(w->ctl.alloc(sizeof(MsCtl) + 16));
    OGB_TRY(w->roots.alloc(64 * 12 + 32));
    w->V = V;
    w->heavy_ready = false;
  }
  // pieces of out-rows longer than kMsLong: at most two per kMsLong edges
  OGB_TRY(w->items.alloc(((size_t)g.E / kMsLong * 2 + 2) * sizeof(uint4)));
  if (!w->h_ctl) OGB_CUDA(cudaMallocHost(&w->h_ctl, sizeof(MsCtl)));
  if (!w->ev0) {
    OGB_CUDA(cudaEventCreate(&w->ev_init));
    OGB_CUDA(cudaEventCreate(&w->ev0));
    OGB_CUDA(cudaEventCreate(&w->ev1));
  }
  if (!w->heavy_ready || w->heavy_build != g.build_id) {
    uint32_t* c = w->ctl.as<uint32_t>();
    OGB_CUDA(cudaMemsetAsync(c, 0, 4, s));
    msk_heavy_list<<<sm_count() * 8, 256, 0, s>>>(V, g.inv.d_rows(), w->heavy.as<uint32_t>(), c);
    OGB_CUDA(cudaGetLastError());
    OGB_CUDA(cudaMemcpyAsync(&w->n_heavy, c, 4, cudaMemcpyDeviceToHost, s));
    OGB_CUDA(cudaStreamSynchronize(s));
    w->heavy_ready = true;
    w->heavy_build = g.build_id;
  }
  *out = w;
  return OK;
}

int msbfs_run(DevGraph& g, const uint32_t* roots, uint32_t nroots, uint16_t* depth, MsResult* res,
              cudaStream_t s) {
  const uint32_t V = g.V;
  if (nroots == 0 || nroots > 64) return fail(ERR_ARG, "msbfs: %u roots (1..64)", nroots);
  for (uint32_t i = 0; i < nroots; i++)
    if (roots[i] >= V) return fail(ERR_ARG, "msbfs: root %u out of range (V=%u)", roots[i], V);
  MsWork* w = nullptr;
  OGB_TRY(ms_work_get(g, &w, s));
  // distinct root vertices and their lanes
  std::vector<uint32_t> verts;
  std::vector<unsigned long long> masks;
  for (uint32_t i = 0; i < nroots; i++) {
    auto it = std::find(verts.begin(), verts.end(), roots[i]);
    if (it == verts.end()) {
      verts.push_back(roots[i]);
      masks.push_back(1ull << i);
    } else {
      masks[it - verts.begin()] |= 1ull << i;
    }
  }
  const unsigned long long lanes = nroots == 64 ? ~0ull : ((1ull << nroots) - 1);
  uint32_t* d_verts = w->roots.as<uint32_t>();
  unsigned long long* d_masks = reinterpret_cast<unsigned long long*>(w->roots.as<char>() + 64 * 4);
  OGB_CUDA(cudaMemcpyAsync(d_verts, verts.data(), verts.size() * 4, cudaMemcpyHostToDevice, s));
  OGB_CUDA(cudaMemcpyAsync(d_masks, masks.data(), masks.size() * 8, cudaMemcpyHostToDevice, s));

  const int sms = sm_count();
  unsigned long long* F = w->F.as<unsigned long long>();
  unsigned long long* N = w->N.as<unsigned long long>();
  unsigned long long* vis = w->vis.as<unsigned long long>();
  MsCtl* ctl = w->ctl.as<MsCtl>();
  const uint2* rows_f = g.fwd.d_rows();
  const uint2* rows_i = g.inv.d_rows();

  // initialisation (timed apart, as the single-root search's precedes its
  // timed part): depths unreached, per-vertex words cleared, the roots set
  OGB_CUDA(cudaEventRecord(w->ev_init, s));
  OGB_CUDA(cudaMemsetAsync(depth, 0xFF, (size_t)V * 64 * 2, s));
  OGB_CUDA(cudaMemsetAsync(F, 0, (size_t)V * 8, s));
  OGB_CUDA(cudaMemsetAsync(N, 0, (size_t)V * 8, s));
  OGB_CUDA(cudaMemsetAsync(vis, 0, (size_t)V * 8, s));
  OGB_CUDA(cudaMemsetAsync(ctl, 0, sizeof(MsCtl), s));
  msk_roots<<<1, 64, 0, s>>>(d_verts, d_masks, (uint32_t)verts.size(), F, vis, depth, w->list.as<uint32_t>(),
                             g.fwd.d_out_degree(), g.E, ctl);
  OGB_CUDA(cudaGetLastError());
  OGB_CUDA(cudaEventRecord(w->ev0, s));
  const uint32_t nb_heavy = w->n_heavy ? std::min<uint32_t>(sms * 8, ceil_div(w->n_heavy, 8)) : 0;
  const uint32_t nb_light = std::max<uint32_t>(1, std::min<uint32_t>(sms * 8, ceil_div(V, 256)));
  const uint32_t nb_finish = std::max<uint32_t>(1, std::min<uint32_t>(sms * 8, ceil_div(V, 1024)));
  uint32_t launches = 6;
  do {
    for (int k = 0; k < kMsBatch; k++) {
      OGB_CUDA(launch_dependent(msk_expand, nb_heavy + nb_light, 256, 0, s, V, lanes, nb_heavy,
                                w->heavy.as<uint32_t>(), w->n_heavy, rows_f, g.fwd.d_dst(), rows_i, g.inv.d_dst(),
                                F, vis, N, w->list.as<uint32_t>(), w->items.as<uint4>(), ctl));
      OGB_CUDA(launch_dependent(msk_push_long, sms * 4, 256, 0, s, w->items.as<uint4>(), g.fwd.d_dst(), F, vis, N,
                                ctl));
      OGB_CUDA(launch_dependent(msk_finish, nb_finish, 256, 0, s, V, g.E, F, N, vis, depth, g.fwd.d_out_degree(),
                                w->list.as<uint32_t>(), ctl));
    }
    launches += 3 * kMsBatch;
    OGB_CUDA(cudaGetLastError());
    OGB_CUDA(cudaEventRecord(w->ev1, s));
    OGB_CUDA(cudaMemcpyAsync(w->h_ctl, ctl, sizeof(MsCtl), cudaMemcpyDeviceToHost, s));
    OGB_CUDA(cudaStreamSynchronize(s));
  } while (!w->h_ctl->done);
  if (w->h_ctl->done == 2) return fail(ERR_UNSUPPORTED, "msbfs: more than 65534 levels");
  MsResult r;
  r.reached = (unsigned long long)__builtin_popcountll(lanes) + w->h_ctl->reached;
  r.edges_examined = w->h_ctl->edges;
  r.push_levels = w->h_ctl->push_levels;
  r.pull_levels = w->h_ctl->pull_levels;
  float ms = 0.f, init_ms = 0.f;
  OGB_CUDA(cudaEventElapsedTime(&ms, w->ev0, w->ev1));
  OGB_CUDA(cudaEventElapsedTime(&init_ms, w->ev_init, w->ev0));
  r.levels = w->h_ctl->levels;
  r.ms = ms;
  r.init_ms = init_ms;
  r.launches = launches;
  if (res) *res = r;
  return OK;
}


// ===========================================================================
// Batched personalized PageRank (no reference counterpart: the reference's
// pull PageRank, pageRank.c:984-1044, with the teleport term base_pr
// replaced by (1 - d) on the seed vertex only, one vector per seed).  Up to
// 32 seeds at once; ranks are row-major by vertex, 32 floats (128 bytes) per
// vertex, so every in-edge gathers one full cache line: the 32 contribs of
// its source.  Per iteration, for every vertex v and seed k:
//   s_k = sum of c_k[u] over the in-edges (u, v)
//   r'_k[v] = (v == seed_k ? 1 - d : 0) + d * s_k,  c'_k[v] = r'_k[v] / out_degree(v)
//   err_k += |r'_k[v] - r_k[v]|   (fp64)
// starting from r_k = e_seed_k; the run stops when every seed's err_k is
// below epsilon, or after max_iterations.  A warp takes a vertex (or a chunk
// of a long row): its four 8-lane groups walk the row's edges in turn, each
// lane owning 4 seeds (one float4 of the row), four edges per group in
// flight; the groups' sums are folded at the end, and the update is one seed
// per lane (by the eight lanes of one group, with four divisions and fp64 errors
// each, it was most of the 17 warp instructions per edge).  The next vertex's
// ids and old ranks load under the current one's gathers: an old rank loaded
// when its sum is ready waited 5600 cycles on average (1370 us per iteration at
// RMAT-20 against 376 with the early load; 588 us before both changes).  Rows
// longer than kPprChunk
// edges are cut into chunks (handed out one per claim, before the other
// vertices, 32 per claim) whose sums the warp finishing the last one adds in
// chunk order.  A vertex without in-edges keeps its teleport value, so after
// the first two iterations, which write it into both contrib buffers, only the
// vertices with in-edges are visited.  Dangling vertices' rank is not
// redistributed, as in the reference.
// Six CTAs of 256 threads per SM leave a thread 40 registers and 84 bytes of spill
// stores.  10 iterations with six, five and four CTAs per SM, us: RMAT-20 3770, 3670
// and 3930; RMAT-16 1060, 960 and 925.
// ===========================================================================

constexpr uint32_t kPprSeeds = 32;
constexpr uint32_t kPprChunk = 512;
constexpr uint32_t kPprMaxIters = 1024;

struct PprCtl {
  double err[kPprMaxIters][kPprSeeds];
  uint32_t stop, stop_iter;
  uint32_t claim_chunk[kPprMaxIters];  // chunks handed out, one per claim
  uint32_t claim_row[kPprMaxIters];    // other vertices handed out, 32 per claim
};

struct PprChunk {
  uint32_t v, j0, j1, k;  // vertex, edge range, index of the vertex among the chunked ones
};

struct PprWork {
  uint32_t V = 0, build = 0;
  bool ready = false;
  DevBuf R, C0, C1, ctl, chunks, vfirst, vcount, done, partials, light, seeds;
  uint32_t n_chunks = 0, n_cut = 0;
  uint32_t n_light = 0, n_fed = 0;  // vertices in `light`; the first n_fed have in-edges
  PprCtl* h_ctl = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  ~PprWork() {
    if (h_ctl) cudaFreeHost(h_ctl);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
  }
};

void ppr_work_free(PprWork* w) { delete w; }

__global__ void pprk_seed(const uint32_t* __restrict__ seeds, uint32_t nseeds, const uint32_t* __restrict__ out_degree,
                          float* __restrict__ R, float* __restrict__ C) {
  const uint32_t k = threadIdx.x;
  if (k < nseeds) {
    const uint32_t v = seeds[k];
    R[(size_t)v * kPprSeeds + k] = 1.0f;
    const uint32_t d = out_degree[v];
    C[(size_t)v * kPprSeeds + k] = d ? __fdiv_rn(1.0f, (float)d) : 0.0f;
  }
}

// The seed of a lane in the update (every seed once over the warp).
__device__ __forceinline__ uint32_t ppr_lane_seed(uint32_t lane) { return 4 * (lane & 7) + (lane >> 3); }

// Ids of the 16 in-edges from j on: group g of 8 lanes has edges g, g + 4,
// g + 8, g + 12 of them.
struct PprIds {
  uint32_t u[4];
  __device__ __forceinline__ void load(const uint32_t* __restrict__ nbr, uint32_t j, uint32_t j1, uint32_t grp) {
#pragma unroll
    for (int q = 0; q < 4; q++) u[q] = (j + grp + 4 * q < j1) ? (__ldg(&nbr[j + grp + 4 * q]) & 0x3FFFFFFFu) : 0xFFFFFFFFu;
  }
};

// Sum over the in-edges [j0, j1) of their source's 32 contribs, 16 edges at a
// time (the first 16 ids come loaded); returns this lane's seed's sum.
__device__ __forceinline__ float ppr_row_sum(const uint32_t* __restrict__ nbr, const float4* C4,
                                             uint32_t j0, uint32_t j1, uint32_t grp, uint32_t sub, PprIds ids) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t j = j0; j < j1; j += 16) {
    float4 c[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      c[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (ids.u[q] != 0xFFFFFFFFu) c[q] = C4[(size_t)ids.u[q] * 8 + sub];
    }
    if (j + 16 < j1) ids.load(nbr, j + 16, j1, grp);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      acc.x += c[q].x;
      acc.y += c[q].y;
      acc.z += c[q].z;
      acc.w += c[q].w;
    }
  }
  // fold the four groups (lanes sub, sub + 8, sub + 16, sub + 24)
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
    acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
  }
  return grp == 0 ? acc.x : (grp == 1 ? acc.y : (grp == 2 ? acc.z : acc.w));
}

struct PprParams {
  float damp, base;
  double eps;
  uint32_t nseeds;
  const uint32_t* seeds;
};

// Update of vertex v from its sums: seed number k, vertex `seed`, on this lane.
__device__ __forceinline__ void ppr_update(uint32_t v, float s, uint32_t k, uint32_t seed, const PprParams& p,
                                           const uint32_t* __restrict__ out_degree, float* R, float* Cn, double& err,
                                           float old, uint32_t d) {
  const size_t at = (size_t)v * kPprSeeds + k;
  const float nv = __fadd_rn(seed == v ? p.base : 0.0f, __fmul_rn(p.damp, s));
  R[at] = nv;
  Cn[at] = d ? __fdiv_rn(nv, (float)d) : 0.0f;
  err += fabs((double)nv - (double)old);
}

__global__ void __launch_bounds__(256, 6) pprk_iter(const PprChunk* __restrict__ chunks, uint32_t n_chunks,
                                                    const uint32_t* __restrict__ vfirst,
                                                    const uint32_t* __restrict__ vcount, uint32_t* done,
                                                    float* partials, const uint32_t* __restrict__ light,
                                                    uint32_t n_light, const uint2* __restrict__ rows,
                                                    const uint32_t* __restrict__ nbr,
                                                    const uint32_t* __restrict__ out_degree,
                                                    const float* C, float* Cn, float* R, PprParams p, PprCtl* ctl,
                                                    uint32_t it) {
  __shared__ double s_err[8][kPprSeeds];
  wait_for_prior_kernel();
  let_next_kernel_start();
  if (ctl->stop) return;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t grp = lane >> 3, sub = lane & 7, k = ppr_lane_seed(lane);
  const uint32_t seed = k < p.nseeds ? p.seeds[k] : 0xFFFFFFFFu;
  const float4* C4 = reinterpret_cast<const float4*>(C);
  double err = 0.0;
  // chunks of long rows, one per claim
  for (;;) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(&ctl->claim_chunk[it], 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= n_chunks) break;
    const PprChunk ci = chunks[t];
    PprIds ids;
    ids.load(nbr, ci.j0, ci.j1, grp);
    partials[(size_t)t * kPprSeeds + k] = ppr_row_sum(nbr, C4, ci.j0, ci.j1, grp, sub, ids);
    __threadfence();
    __syncwarp();
    uint32_t last = 0;
    if (lane == 0) last = (atomicAdd(&done[ci.k], 1u) == vcount[ci.k] - 1) ? 1u : 0u;
    last = __shfl_sync(0xffffffffu, last, 0);
    if (last) {
      __threadfence();
      const uint32_t f = vfirst[ci.k], cnt = vcount[ci.k];
      float tot = 0.f;
      for (uint32_t c = 0; c < cnt; c++) tot += __ldcg(&partials[(size_t)(f + c) * kPprSeeds + k]);
      ppr_update(ci.v, tot, k, seed, p, out_degree, R, Cn, err, __ldcg(&R[(size_t)ci.v * kPprSeeds + k]), __ldg(&out_degree[ci.v]));
      if (lane == 0) done[ci.k] = 0;
    }
  }
  // the other vertices, 32 per claim, their rows loaded a lane each
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&ctl->claim_row[it], 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= n_light) break;
    const uint32_t n = min(32u, n_light - base);
    uint32_t mv = 0, md = 0;
    uint2 mr = make_uint2(0u, 0u);
    if (lane < n) {
      mv = light[base + lane];
      mr = rows[mv];
      md = out_degree[mv];
    }
    uint32_t j0 = __shfl_sync(0xffffffffu, mr.x, 0), j1 = j0 + __shfl_sync(0xffffffffu, mr.y, 0);
    PprIds ids;
    ids.load(nbr, j0, j1, grp);
    uint32_t v_next = __shfl_sync(0xffffffffu, mv, 0);
    float old_next = R[(size_t)v_next * kPprSeeds + k];
    for (uint32_t t = 0; t < n; t++) {
      const uint32_t v = v_next;
      const float old = old_next;
      const uint32_t a0 = j0, a1 = j1;
      const PprIds cur = ids;
      // the next vertex's ids load under this one's gathers (n - 1: itself again)
      const uint32_t tn = min(t + 1, n - 1);
      j0 = __shfl_sync(0xffffffffu, mr.x, tn);
      j1 = j0 + __shfl_sync(0xffffffffu, mr.y, tn);
      ids.load(nbr, j0, j1, grp);
      v_next = __shfl_sync(0xffffffffu, mv, tn);
      old_next = R[(size_t)v_next * kPprSeeds + k];
      const uint32_t d = __shfl_sync(0xffffffffu, md, t);
      ppr_update(v, ppr_row_sum(nbr, C4, a0, a1, grp, sub, cur), k, seed, p, out_degree, R, Cn, err, old, d);
    }
  }
  s_err[warp][k] = err;
  __syncthreads();
  if (threadIdx.x < kPprSeeds) {
    double e = 0.0;
    for (int w = 0; w < 8; w++) e += s_err[w][threadIdx.x];
    if (e != 0.0) atomicAdd(&ctl->err[it][threadIdx.x], e);
  }
}

// the run stops after an iteration in which every seed changed by < eps (L1)
__global__ void pprk_check(PprCtl* ctl, uint32_t it, uint32_t nseeds, double eps) {
  wait_for_prior_kernel();
  let_next_kernel_start();
  if (threadIdx.x != 0 || ctl->stop) return;
  bool all = true;
  for (uint32_t k = 0; k < nseeds; k++) all = all && (ctl->err[it][k] < eps);
  if (all) {
    ctl->stop = 1;
    ctl->stop_iter = it;
  }
}

// The vertices by class: in-edges but no chunks, number of chunks, chunked.
__global__ void pprk_classes(uint32_t V, const uint2* __restrict__ rows, uint32_t* __restrict__ fed,
                             uint32_t* __restrict__ nchunk, uint32_t* __restrict__ cut) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const uint32_t d = rows[v].y;
    fed[v] = d && d <= kPprChunk ? 1u : 0u;
    nchunk[v] = d > kPprChunk ? (d + kPprChunk - 1) / kPprChunk : 0u;
    cut[v] = d > kPprChunk ? 1u : 0u;
  }
}

// From the classes' scans: the vertices without chunks, those with in-edges
// first, each part in vertex order; and the chunk table.  (Built on the host from
// a copy of the rows, these lists took longer than the iterations.)
__global__ void pprk_lists(uint32_t V, const uint2* __restrict__ rows, const uint32_t* __restrict__ fed,
                           const uint32_t* __restrict__ nchunk, const uint32_t* __restrict__ cut, uint32_t n_fed,
                           uint32_t* __restrict__ light, PprChunk* __restrict__ chunks, uint32_t* __restrict__ vfirst,
                           uint32_t* __restrict__ vcount, uint32_t* __restrict__ done) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const uint2 r = rows[v];
    const uint32_t k = cut[v];
    if (r.y > kPprChunk) {
      const uint32_t at = nchunk[v], n = (r.y + kPprChunk - 1) / kPprChunk;
      vfirst[k] = at;
      vcount[k] = n;
      done[k] = 0;
      for (uint32_t c = 0; c < n; c++)
        chunks[at + c] = {v, r.x + c * kPprChunk, r.x + min(r.y, (c + 1) * kPprChunk), k};
    } else {
      light[r.y ? fed[v] : n_fed + (v - fed[v] - k)] = v;
    }
  }
}

static int ppr_work_get(DevGraph& g, PprWork** out, cudaStream_t s) {
  if (!g.ppr) g.ppr = new PprWork();
  PprWork* w = g.ppr;
  const uint32_t V = g.V;
  if (w->V != V || !w->R.p) {
    OGB_TRY(w->R.alloc((size_t)V * kPprSeeds * 4 + 64));
    OGB_TRY(w->C0.alloc((size_t)V * kPprSeeds * 4 + 64));
    OGB_TRY(w->C1.alloc((size_t)V * kPprSeeds * 4 + 64));
    OGB_TRY(w->ctl.alloc(sizeof(PprCtl) + 64));
    OGB_TRY(w->seeds.alloc(kPprSeeds * 4));
    w->V = V;
    w->ready = false;
  }
  if (!w->h_ctl) OGB_CUDA(cudaMallocHost(&w->h_ctl, sizeof(PprCtl)));
  if (!w->ev0) {
    OGB_CUDA(cudaEventCreate(&w->ev0));
    OGB_CUDA(cudaEventCreate(&w->ev1));
  }
  if (!w->ready || w->build != g.build_id) {
    // rows from the inverse CSR: rows over kPprChunk in-edges become chunks
    const uint2* rows = g.inv.d_rows();
    const size_t Vp = (size_t)V + 4;
    DevBuf tmp;
    OGB_TRY(tmp.alloc((Vp * 6 + scan_tmp_words(V)) * 4));
    uint32_t* cls[3];  // vertices with in-edges and no chunks, chunks, chunked vertices: counts, then their scans
    uint32_t* pos[3];
    for (int i = 0; i < 3; i++) {
      cls[i] = tmp.as<uint32_t>() + (size_t)i * Vp;
      pos[i] = tmp.as<uint32_t>() + (size_t)(3 + i) * Vp;
    }
    const int grid = sm_count() * 8;
    pprk_classes<<<grid, 256, 0, s>>>(V, rows, cls[0], cls[1], cls[2]);
    OGB_CUDA(cudaGetLastError());
    uint32_t total[3];
    for (int i = 0; i < 3; i++) {
      OGB_TRY(scan_exclusive_u32(cls[i], pos[i], V, tmp.as<uint32_t>() + 6 * Vp, s));
      OGB_CUDA(cudaMemcpyAsync(&total[i], pos[i] + V, 4, cudaMemcpyDeviceToHost, s));
    }
    OGB_CUDA(cudaStreamSynchronize(s));
    w->n_fed = total[0];
    w->n_chunks = total[1];
    w->n_cut = total[2];
    w->n_light = V - w->n_cut;
    OGB_TRY(w->light.alloc((size_t)w->n_light * 4 + 16));
    OGB_TRY(w->chunks.alloc((size_t)w->n_chunks * sizeof(PprChunk) + 16));
    OGB_TRY(w->partials.alloc((size_t)w->n_chunks * kPprSeeds * 4 + 16));
    OGB_TRY(w->vfirst.alloc((size_t)w->n_cut * 4 + 16));
    OGB_TRY(w->vcount.alloc((size_t)w->n_cut * 4 + 16));
    OGB_TRY(w->done.alloc((size_t)w->n_cut * 4 + 16));
    pprk_lists<<<grid, 256, 0, s>>>(V, rows, pos[0], pos[1], pos[2], w->n_fed, w->light.as<uint32_t>(),
                                    w->chunks.as<PprChunk>(), w->vfirst.as<uint32_t>(), w->vcount.as<uint32_t>(),
                                    w->done.as<uint32_t>());
    OGB_CUDA(cudaGetLastError());
    OGB_CUDA(cudaStreamSynchronize(s));  // before the scratch is released
    w->ready = true;
    w->build = g.build_id;
  }
  *out = w;
  return OK;
}

int ppr_run(DevGraph& g, const uint32_t* seeds, uint32_t nseeds, uint32_t max_iters, double epsilon, float* ranks,
            PprResult* res, cudaStream_t s) {
  const uint32_t V = g.V;
  if (nseeds == 0 || nseeds > kPprSeeds) return fail(ERR_ARG, "ppr: %u seeds (1..%u)", nseeds, kPprSeeds);
  if (max_iters > kPprMaxIters) return fail(ERR_ARG, "ppr: at most %u iterations", kPprMaxIters);
  for (uint32_t i = 0; i < nseeds; i++)
    if (seeds[i] >= V) return fail(ERR_ARG, "ppr: seed %u out of range (V=%u)", seeds[i], V);
  PprWork* w = nullptr;
  OGB_TRY(ppr_work_get(g, &w, s));
  OGB_CUDA(cudaMemcpyAsync(w->seeds.p, seeds, nseeds * 4, cudaMemcpyHostToDevice, s));
  PprCtl* ctl = w->ctl.as<PprCtl>();
  float* C = w->C0.as<float>();
  float* Cn = w->C1.as<float>();
  float* R = w->R.as<float>();
  PprParams p;
  p.damp = 0.85f;
  p.base = 1.0f - p.damp;
  p.eps = epsilon;
  p.nseeds = nseeds;
  p.seeds = w->seeds.as<uint32_t>();
  const int sms = sm_count();
  OGB_CUDA(cudaEventRecord(w->ev0, s));
  OGB_CUDA(cudaMemsetAsync(ctl, 0, sizeof(PprCtl), s));
  OGB_CUDA(cudaMemsetAsync(R, 0, (size_t)V * kPprSeeds * 4, s));
  OGB_CUDA(cudaMemsetAsync(C, 0, (size_t)V * kPprSeeds * 4, s));
  pprk_seed<<<1, 32, 0, s>>>(p.seeds, nseeds, g.fwd.d_out_degree(), R, C);
  OGB_CUDA(cudaGetLastError());
  for (uint32_t it = 0; it < max_iters; it++) {
    OGB_CUDA(launch_dependent(pprk_iter, sms * 6, 256, 0, s, w->chunks.as<PprChunk>(), w->n_chunks,
                              w->vfirst.as<uint32_t>(), w->vcount.as<uint32_t>(), w->done.as<uint32_t>(),
                              w->partials.as<float>(), w->light.as<uint32_t>(), it < 2 ? w->n_light : w->n_fed,
                              g.inv.d_rows(), g.inv.d_dst(), g.fwd.d_out_degree(), C, Cn, R, p, ctl, it));
    OGB_CUDA(launch_dependent(pprk_check, 1, 32, 0, s, ctl, it, nseeds, epsilon));
    OGB_CUDA(cudaGetLastError());
    std::swap(C, Cn);
  }
  OGB_CUDA(cudaEventRecord(w->ev1, s));
  if (ranks) OGB_CUDA(cudaMemcpyAsync(ranks, R, (size_t)V * kPprSeeds * 4, cudaMemcpyDeviceToDevice, s));
  OGB_CUDA(cudaMemcpyAsync(w->h_ctl, ctl, sizeof(PprCtl), cudaMemcpyDeviceToHost, s));
  OGB_CUDA(cudaStreamSynchronize(s));
  float ms = 0.f;
  OGB_CUDA(cudaEventElapsedTime(&ms, w->ev0, w->ev1));
  PprResult r;
  r.ms = ms;
  r.executed = w->h_ctl->stop ? w->h_ctl->stop_iter + 1 : max_iters;
  r.converged = w->h_ctl->stop;
  r.launches = 2 + 2 * max_iters;
  for (uint32_t k = 0; k < nseeds; k++) r.err_last[k] = r.executed ? w->h_ctl->err[r.executed - 1][k] : 0.0;
  if (res) *res = r;
  return OK;
}


// ===========================================================================
// Many graphs in one launch (no reference counterpart: each graph's results
// equal the reference path run on that graph alone).  The graphs are packed
// into one disjoint union (vertex ids shifted by each graph's offset, one
// sort builds every graph's CSR side by side), so the single-graph kernels
// and their load balancing serve the whole batch:
//  * BFS: one search from every graph's root at once -- one cooperative
//    launch for the whole batch; each vertex gets its depth from its own
//    graph's root (no edges cross graphs); parents are returned in local ids;
//  * PageRank pull: every graph keeps its own stop rule and normalization
//    (a per-graph reduction after each iteration freezes a graph whose
//    vertices all changed by < epsilon); the whole run is one CUDA graph.
// ===========================================================================

struct GraphBatch {
  DevGraph g;
  uint32_t ngraphs = 0;
  std::vector<uint32_t> voff;  // host copy of the vertex offsets
  DevBuf d_voff, d_eoff, gid, frozen, stop_iter, executed, active_last, err_last, delta;
  DevBuf pieces, piece_err, piece_act, piece_done;
  uint32_t npieces = 0;
  cudaGraphExec_t pr_exec = nullptr;
  uint32_t pr_gen = 0, pr_iters = 0, pr_warp = 0, pr_cta = 0, pr_build = 0;
  double pr_eps = -1.0;
  float* pr_ranks = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  ~GraphBatch() {
    if (pr_exec) cudaGraphExecDestroy(pr_exec);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
  }
};

GraphBatch* batch_new() { return new GraphBatch(); }
void batch_free(GraphBatch* b) { delete b; }
uint32_t batch_ngraphs(const GraphBatch* b) { return b->ngraphs; }
const uint32_t* batch_voff(const GraphBatch* b) { return b->voff.data(); }
DevGraph& batch_graph(GraphBatch* b) { return b->g; }

// local ids -> union ids (edge e of graph g: + voff[g]); an id outside its
// graph sets *err
__global__ void bk_shift(uint64_t E, const uint64_t* __restrict__ eoff, const uint32_t* __restrict__ voff,
                         uint32_t ng, uint32_t* __restrict__ src, uint32_t* __restrict__ dst, uint32_t* err) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = ng - 1;  // last g with eoff[g] <= e
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (eoff[mid] <= e)
        lo = mid;
      else
        hi = mid - 1;
    }
    const uint32_t n = voff[lo + 1] - voff[lo];
    if (src[e] >= n || dst[e] >= n) *err = 1;
    src[e] += voff[lo];
    dst[e] += voff[lo];
  }
}

__global__ void bk_gid(uint32_t V, const uint32_t* __restrict__ voff, uint32_t ng, uint32_t* __restrict__ gid) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = ng - 1;  // last g with voff[g] <= v
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (voff[mid] <= v)
        lo = mid;
      else
        hi = mid - 1;
    }
    gid[v] = lo;
  }
}

__global__ void bk_localize(uint32_t V, const uint32_t* __restrict__ gid, const uint32_t* __restrict__ voff,
                            int32_t* __restrict__ parents) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const int32_t p = parents[v];
    if (p >= 0) parents[v] = p - (int32_t)voff[gid[v]];
  }
}

int batch_create(GraphBatch& b, uint32_t ngraphs, const uint32_t* nv, const uint64_t* eoff, const uint32_t* src,
                 const uint32_t* dst, uint32_t sort_type, cudaStream_t s) {
  if (ngraphs == 0) return fail(ERR_ARG, "batch: no graphs");
  if (sort_type > 3) return fail(ERR_ARG, "batch: sort type %u", sort_type);
  b.voff.assign(ngraphs + 1, 0);
  uint64_t V = 0;
  for (uint32_t i = 0; i < ngraphs; i++) {
    if (eoff[i + 1] < eoff[i]) return fail(ERR_ARG, "batch: edge offsets decrease at graph %u", i);
    V += nv[i];
    if (V > (1u << 30)) return fail(ERR_RANGE, "batch: more than 2^30 vertices in all");
    b.voff[i + 1] = (uint32_t)V;
  }
  const uint64_t E = eoff[ngraphs] - eoff[0];
  if (eoff[0] != 0) return fail(ERR_ARG, "batch: edge offsets must start at 0");
  if (E > 0xFFFFFFFFull) return fail(ERR_RANGE, "batch: more than 2^32 - 1 edges in all");
  b.ngraphs = ngraphs;
  OGB_TRY(b.d_voff.alloc((size_t)(ngraphs + 1) * 4));
  OGB_TRY(b.d_eoff.alloc((size_t)(ngraphs + 1) * 8));
  OGB_CUDA(cudaMemcpyAsync(b.d_voff.p, b.voff.data(), (size_t)(ngraphs + 1) * 4, cudaMemcpyHostToDevice, s));
  OGB_CUDA(cudaMemcpyAsync(b.d_eoff.p, eoff, (size_t)(ngraphs + 1) * 8, cudaMemcpyHostToDevice, s));
  DevBuf us, ud, derr;
  OGB_TRY(us.alloc(E * 4 + 16));
  OGB_TRY(ud.alloc(E * 4 + 16));
  OGB_TRY(derr.alloc(16));
  OGB_CUDA(cudaMemsetAsync(derr.p, 0, 4, s));
  if (E) {
    OGB_CUDA(cudaMemcpyAsync(us.p, src, E * 4, cudaMemcpyHostToDevice, s));
    OGB_CUDA(cudaMemcpyAsync(ud.p, dst, E * 4, cudaMemcpyHostToDevice, s));
    bk_shift<<<sm_count() * 8, 256, 0, s>>>(E, b.d_eoff.as<uint64_t>(), b.d_voff.as<uint32_t>(), ngraphs,
                                           us.as<uint32_t>(), ud.as<uint32_t>(), derr.as<uint32_t>());
    OGB_CUDA(cudaGetLastError());
  }
  uint32_t herr = 0;
  OGB_CUDA(cudaMemcpyAsync(&herr, derr.p, 4, cudaMemcpyDeviceToHost, s));
  OGB_CUDA(cudaStreamSynchronize(s));
  if (herr) return fail(ERR_RANGE, "batch: an edge id is not below its graph's vertex count");
  OGB_TRY(graph_build(b.g, us.as<uint32_t>(), ud.as<uint32_t>(), nullptr, (uint32_t)E, (uint32_t)V, sort_type, s));
  OGB_TRY(graph_check(b.g, s));
  OGB_TRY(b.gid.alloc(V * 4 + 16));
  bk_gid<<<sm_count() * 8, 256, 0, s>>>((uint32_t)V, b.d_voff.as<uint32_t>(), ngraphs, b.gid.as<uint32_t>());
  OGB_CUDA(cudaGetLastError());
  OGB_TRY(b.frozen.alloc((size_t)ngraphs * 4 + 16));
  OGB_TRY(b.stop_iter.alloc((size_t)ngraphs * 4 + 16));
  OGB_TRY(b.executed.alloc((size_t)ngraphs * 4 + 16));
  OGB_TRY(b.active_last.alloc((size_t)ngraphs * 4 + 16));
  OGB_TRY(b.err_last.alloc((size_t)ngraphs * 8 + 16));
  OGB_TRY(b.delta.alloc(V * 4 + 16));
  std::vector<uint4> pieces;
  for (uint32_t i = 0; i < ngraphs; i++) {
    const uint32_t first = (uint32_t)pieces.size();
    uint32_t v = b.voff[i];
    do {  // a graph without vertices keeps one empty piece: it stops at its first iteration
      pieces.push_back(make_uint4(i, v, std::min(b.voff[i + 1], v + kBatchPiece), first));
      v += kBatchPiece;
    } while (v < b.voff[i + 1]);
  }
  b.npieces = (uint32_t)pieces.size();
  OGB_TRY(b.pieces.alloc(pieces.size() * sizeof(uint4) + 16));
  OGB_TRY(b.piece_err.alloc(pieces.size() * 8 + 16));
  OGB_TRY(b.piece_act.alloc(pieces.size() * 4 + 16));
  OGB_TRY(b.piece_done.alloc((size_t)ngraphs * 4 + 16));
  OGB_CUDA(cudaMemcpyAsync(b.pieces.p, pieces.data(), pieces.size() * sizeof(uint4), cudaMemcpyHostToDevice, s));
  if (!b.ev0) {
    OGB_CUDA(cudaEventCreate(&b.ev0));
    OGB_CUDA(cudaEventCreate(&b.ev1));
  }
  OGB_CUDA(cudaStreamSynchronize(s));
  return OK;
}

int batch_bfs(GraphBatch& b, const uint32_t* roots, int32_t* parents, uint32_t* distances, BfsResult* res,
              cudaStream_t s) {
  std::vector<uint32_t> r(b.ngraphs);
  for (uint32_t i = 0; i < b.ngraphs; i++) {
    if (roots[i] >= b.voff[i + 1] - b.voff[i]) return fail(ERR_ARG, "batch bfs: root %u of graph %u out of range", roots[i], i);
    r[i] = roots[i] + b.voff[i];
  }
  OGB_TRY(bfs_run_roots(b.g, r.data(), b.ngraphs, BFS_DO, parents, distances, res, false, false, s));
  bk_localize<<<sm_count() * 8, 256, 0, s>>>(b.g.V, b.gid.as<uint32_t>(), b.d_voff.as<uint32_t>(), parents);
  OGB_CUDA(cudaGetLastError());
  OGB_CUDA(cudaStreamSynchronize(s));
  return OK;
}

int batch_pagerank(GraphBatch& b, uint32_t max_iters, double epsilon, float* ranks, BatchPrGraph* per_graph,
                   double* ms_out, uint32_t* captured, cudaStream_t s) {
  uint32_t wt = 0, ct = 0, cth = 0, ch = 0;
  pagerank_get_bins(&wt, &ct, &cth, &ch);
  if (b.pr_exec && (b.pr_iters != max_iters || b.pr_eps != epsilon || b.pr_ranks != ranks || b.pr_warp != wt ||
                    b.pr_cta != ct || b.pr_build != b.g.build_id)) {
    cudaGraphExecDestroy(b.pr_exec);
    b.pr_exec = nullptr;
  }
  PrBatchDev d;
  d.voff = b.d_voff.as<uint32_t>();
  d.gid = b.gid.as<uint32_t>();
  d.frozen = b.frozen.as<uint32_t>();
  d.stop_iter = b.stop_iter.as<uint32_t>();
  d.executed = b.executed.as<uint32_t>();
  d.active_last = b.active_last.as<uint32_t>();
  d.err_last = b.err_last.as<double>();
  d.delta = b.delta.as<float>();
  d.pieces = b.pieces.as<uint4>();
  d.npieces = b.npieces;
  d.piece_err = b.piece_err.as<double>();
  d.piece_act = b.piece_act.as<uint32_t>();
  d.piece_done = b.piece_done.as<uint32_t>();
  bool rebuilt = false;
  // capture happens outside the timed region
  if (!b.pr_exec) {
    OGB_TRY(pagerank_batch_run(b.g, d, b.ngraphs, max_iters, epsilon, ranks, &b.pr_exec, &b.pr_gen, &rebuilt, s));
    OGB_CUDA(cudaStreamSynchronize(s));
    b.pr_iters = max_iters;
    b.pr_eps = epsilon;
    b.pr_ranks = ranks;
    b.pr_warp = wt;
    b.pr_cta = ct;
    b.pr_build = b.g.build_id;
  }
  OGB_CUDA(cudaEventRecord(b.ev0, s));
  OGB_TRY(pagerank_batch_run(b.g, d, b.ngraphs, max_iters, epsilon, ranks, &b.pr_exec, &b.pr_gen, nullptr, s));
  OGB_CUDA(cudaEventRecord(b.ev1, s));
  std::vector<uint32_t> stop(b.ngraphs), exe(b.ngraphs), act(b.ngraphs);
  std::vector<double> err(b.ngraphs);
  OGB_CUDA(cudaMemcpyAsync(stop.data(), d.stop_iter, (size_t)b.ngraphs * 4, cudaMemcpyDeviceToHost, s));
  OGB_CUDA(cudaMemcpyAsync(exe.data(), d.executed, (size_t)b.ngraphs * 4, cudaMemcpyDeviceToHost, s));
  OGB_CUDA(cudaMemcpyAsync(act.data(), d.active_last, (size_t)b.ngraphs * 4, cudaMemcpyDeviceToHost, s));
  OGB_CUDA(cudaMemcpyAsync(err.data(), d.err_last, (size_t)b.ngraphs * 8, cudaMemcpyDeviceToHost, s));
  OGB_CUDA(cudaStreamSynchronize(s));
  float ms = 0.f;
  OGB_CUDA(cudaEventElapsedTime(&ms, b.ev0, b.ev1));
  if (ms_out) *ms_out = ms;
  if (captured) *captured = rebuilt ? 1u : 0u;
  if (per_graph)
    for (uint32_t i = 0; i < b.ngraphs; i++) {
      const bool conv = stop[i] != 0xFFFFFFFFu;
      per_graph[i].converged = conv ? 1u : 0u;
      per_graph[i].iterations = conv ? stop[i] : max_iters;
      per_graph[i].executed = exe[i];
      per_graph[i].activeVertices = act[i];
      per_graph[i].error_total = err[i];
    }
  return OK;
}

// Bin thresholds for this batch: each candidate (warp_thr, cta_thr) runs a
// few pull iterations over the union (its per-graph layout is rebuilt for
// it, outside the timing); the fastest is kept as the library's setting.
int batch_autotune(GraphBatch& b, uint32_t iters, TuneResult* out, cudaStream_t s) {
  static const uint32_t cand[][2] = {{16, 1024}, {32, 2048}, {64, 2048}, {64, 4096}, {128, 4096}, {32, 8192}};
  const uint32_t n = sizeof(cand) / sizeof(cand[0]);
  float* ranks = nullptr;
  DevBuf rb;
  OGB_TRY(rb.alloc((size_t)b.g.V * 4 + 16));
  ranks = rb.as<float>();
  double best = 1e30;
  uint32_t bi = 0;
  for (uint32_t i = 0; i < n; i++) {
    pagerank_set_bins(cand[i][0], cand[i][1]);
    PrResult r;
    OGB_TRY(pagerank_run(b.g, PR_PULL, 1, 0.0, ranks, nullptr, &r, s));  // builds the layout
    OGB_TRY(pagerank_run(b.g, PR_PULL, iters, 0.0, ranks, nullptr, &r, s));
    const double ms = r.ms / iters;
    if (out) {
      out->warp_thr[i] = cand[i][0];
      out->cta_thr[i] = cand[i][1];
      out->ms[i] = ms;
    }
    if (ms < best) {
      best = ms;
      bi = i;
    }
  }
  pagerank_set_bins(cand[bi][0], cand[bi][1]);
  if (out) {
    out->n = n;
    out->best = bi;
  }
  return OK;
}

}  // namespace ogb
