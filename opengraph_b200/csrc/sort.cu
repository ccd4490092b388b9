// sort.cu -- stable onesweep LSD radix sort for edge lists on sm_100a.
//
// Replaces the reference's 4-pass, 8-bit, per-thread-histogram LSD sort
// (00_graph_bench/src/preprocess/radixsort.c:46-135, :231-335) and its
// counting sort (countsort.c:28-270), whose outputs are identical: edges
// ordered by key, ties kept in input order.
//
// Design (one pass = one kernel, no separate upsweep):
//  * digit histograms of every digit are built by one read of the keys; digits
//    that are constant over all keys are skipped.  Which passes run, and between
//    which buffers, is decided on the device (plan_kernel): every pass is
//    launched, and the skipped ones return at once, so a sort needs no round
//    trip to the host;
//  * each CTA claims a tile of kTile keys in launch order, ranks the keys of
//    the tile stably with warp ballots (order = warp, item, lane, which is
//    input order), publishes its per-digit counts and resolves the per-digit
//    prefix of all earlier tiles by decoupled look-back;
//  * keys and payloads are staged in shared memory in digit order and written
//    out so that consecutive threads store consecutive addresses of a run.
#include "sort.cuh"

namespace ogb {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kTile = kSortThreads * kSortItems;
constexpr int kWarps = kSortThreads / 32;
constexpr int kMaxPasses = 8;  // 4 digits x (primary, secondary)
constexpr int kLookBack = 4;   // predecessors read at once by the look-back

// A look-back word: a count and a two-bit flag.  32-bit words hold counts
// below 2^30; longer inputs take 64-bit ones.
template <class S>
struct LbWord;
template <>
struct LbWord<uint32_t> {
  static constexpr uint32_t kAgg = 1u << 30, kInc = 2u << 30, kFlag = 3u << 30;
};
template <>
struct LbWord<unsigned long long> {
  static constexpr unsigned long long kAgg = 1ull << 32, kInc = 2ull << 32, kFlag = 3ull << 32;
};
constexpr uint64_t kNarrowLimit = 1ull << 30;
// Passes over fewer keys are launched over the end of the pass ahead: 51 K keys by
// two digits 192 -> 178 us, 20 M 1493 -> 1486; 67 M weighted keys 3152 -> 3165 us.
constexpr uint32_t kDependentLimit = 1u << 25;
__device__ __forceinline__ uint32_t lb_load(const uint32_t* p) { return ld_volatile_u32(p); }
__device__ __forceinline__ unsigned long long lb_load(const unsigned long long* p) { return ld_volatile_u64(p); }
__device__ __forceinline__ void lb_store(uint32_t* p, uint32_t v) {
  asm volatile("st.volatile.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void lb_store(unsigned long long* p, unsigned long long v) { st_volatile_u64(p, v); }

// counters layout (u32): [0, kMaxPasses) tile counters, [kMaxPasses] error
// word; then a PassPlan per pass.
constexpr int kCtrErr = kMaxPasses;
constexpr int kCtrPlan = kMaxPasses + 4;

// One pass: whether it runs, and its buffers (0 the input, 1 the scratch set, 2
// the output).
struct PassPlan {
  uint32_t active, src, dst, pad;
};
constexpr int kCtrWords = kCtrPlan + kMaxPasses * (int)(sizeof(PassPlan) / 4);

__device__ __forceinline__ uint32_t block_exclusive_scan_256(uint32_t v, uint32_t* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = (lane < kWarps) ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < kWarps; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < kWarps) s_warp[lane] = w;  // inclusive warp totals
  }
  __syncthreads();
  uint32_t warp_excl = warp ? s_warp[warp - 1] : 0;
  return warp_excl + x - v;
}

// The look-back words of the passes cleared on the way (n_clear 16-byte words at
// `clear`); histograms of `ndig` digits of keys[0, n) into hist[ndig][256] (digit d
// = (key >> 8-aligned or narrower lay.shift[d]) & lay.mask[d]).  Each warp
// counts into its own copy of the histograms in shared memory (conflicts only inside a warp's atomic),
// and the copies are summed once at the end.
// The digits of one key: ndig groups of at most 8 bits from bit 0 up.
struct DigitLayout {
  int ndig;
  uint32_t shift[4], mask[4];
};

// Digits for keys below 2^bits: ceil(bits / 8) groups of nearly equal
// width (the lower ones one bit wider), so each pass's digit runs are as
// long as the key width allows (22 bits: 8 + 7 + 7 instead of 8 + 8 + 6).
static DigitLayout digit_layout(uint32_t bits) {
  bits = bits < 1 ? 1 : (bits > 32 ? 32 : bits);
  DigitLayout l;
  l.ndig = (int)((bits + 7) / 8);
  const uint32_t w = bits / l.ndig, extra = bits % l.ndig;
  uint32_t sh = 0;
  for (int d = 0; d < 4; d++) {
    const uint32_t wd = d < l.ndig ? w + ((uint32_t)d < extra ? 1u : 0u) : 0u;
    l.shift[d] = sh;
    l.mask[d] = wd ? (wd >= 32 ? 0xFFFFFFFFu : (1u << wd) - 1u) : 0u;
    sh += wd;
  }
  return l;
}

constexpr int kHistThreads = 256, kHistWarps = kHistThreads / 32;
__global__ void __launch_bounds__(kHistThreads) digit_hist_kernel(const uint32_t* __restrict__ keys, uint64_t n,
                                                                  int ndig, DigitLayout lay,
                                                                  uint32_t* __restrict__ hist,
                                                                  uint4* __restrict__ clear, uint64_t n_clear) {
  __shared__ uint32_t sh[kHistWarps][4][256];
  for (int i = threadIdx.x; i < kHistWarps * 4 * 256; i += blockDim.x) (&sh[0][0][0])[i] = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_clear; i += (uint64_t)gridDim.x * blockDim.x)
    clear[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  uint32_t(*h)[256] = sh[threadIdx.x >> 5];
  const uint64_t nvec = n / 4;
  const uint4* kv = reinterpret_cast<const uint4*>(keys);
  const bool aligned = (reinterpret_cast<uintptr_t>(keys) & 15) == 0;
  uint64_t start_scalar = 0;
  if (aligned) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec;
         i += (uint64_t)gridDim.x * blockDim.x) {
      const uint4 q = __ldg(kv + i);
      const uint32_t a[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 4; j++) {
#pragma unroll
        for (int d = 0; d < 4; d++)
          if (d < ndig) atomicAdd(&h[d][(a[j] >> lay.shift[d]) & lay.mask[d]], 1u);
      }
    }
    start_scalar = nvec * 4;
  }
  for (uint64_t i = start_scalar + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t k = keys[i];
#pragma unroll
    for (int d = 0; d < 4; d++)
      if (d < ndig) atomicAdd(&h[d][(k >> lay.shift[d]) & lay.mask[d]], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ndig * 256; i += blockDim.x) {
    uint32_t c = 0;
#pragma unroll
    for (int w = 0; w < kHistWarps; w++) c += (&sh[w][0][0])[i];
    if (c) atomicAdd(&hist[i], c);
  }
}

// The histogram of each pass.
struct PlanHists {
  int h[kMaxPasses];
};

// One CTA: the exclusive scan of every pass's 256-bucket histogram, and the
// passes that run -- those whose digit is not the same in all n keys, or, if all
// are, the last one (a stable copy).  The output buffer is the last active pass's;
// they alternate before it.
__global__ void __launch_bounds__(256) plan_kernel(const uint32_t* __restrict__ hist, uint32_t* __restrict__ base,
                                                   uint32_t n, PlanHists hists, int passes, PassPlan* __restrict__ plan) {
  __shared__ uint32_t s_warp[kWarps];
  uint32_t live = 0;
  for (int j = 0; j < passes; j++) {
    const int h = hists.h[j];
    const uint32_t v = hist[h * 256 + threadIdx.x];
    base[h * 256 + threadIdx.x] = block_exclusive_scan_256(v, s_warp);
    if (!__syncthreads_or(v == n)) live |= 1u << j;
  }
  if (threadIdx.x != 0) return;
  if (!live) live = 1u << (passes - 1);
  uint32_t left = __popc(live), src = 0;
  for (int j = 0; j < passes; j++) {
    PassPlan p = {};
    if ((live >> j) & 1u) {
      left--;
      p = {1u, src, left % 2 == 0 ? 2u : 1u, 0u};
      src = p.dst;
    }
    plan[j] = p;
  }
}

__device__ __forceinline__ void cp_async_u32(uint32_t* dst_smem, const uint32_t* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Lanes of `valid` whose digit equals this lane's (digits of at most NB bits):
// one ballot per bit.  (__match_any_sync took as long as the rest of the pass:
// 627 -> 499 us unweighted with nothing else changed.)
template <int NB>
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, uint32_t valid) {
  uint32_t p = valid;
#pragma unroll
  for (int b = 0; b < NB; b++)
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b32 t, m;\n\t"
        "and.b32 t, %1, %2;\n\t"
        "setp.ne.u32 q, t, 0;\n\t"
        "vote.sync.ballot.b32 m, q, 0xffffffff;\n\t"
        "@!q not.b32 m, m;\n\t"
        "and.b32 %0, %0, m;\n\t}"
        : "+r"(p)
        : "r"(d), "r"(1u << b));
  return p;
}

// The arrays a tile works on, and the pass's digit.
template <class S>
struct TileArgs {
  const uint32_t* kin;
  const uint32_t* p0in;
  const uint32_t* p1in;
  uint32_t* kout;
  uint32_t* p0out;
  uint32_t* p1out;
  uint32_t n, shift, mask;
  const uint32_t* digit_base;
  S* status;
  uint32_t* err;
};

// A launched pass: the three buffers it may work between (as key and first
// payload of this pass), its digit and its entry of the plan.
template <class S>
struct PassArgs {
  uint32_t *k[3], *p0[3], *p1[3];
  uint32_t n, shift, mask;
  const uint32_t* digit_base;
  S* status;
  uint32_t* tile_ctr;
  uint32_t* err;
  const PassPlan* plan;
};

// One pass over one tile.  Only the keys pass through registers: once the
// tile-local digit prefix is known, each payload element is copied from
// global memory straight into its slot of the digit-ordered stage by an
// asynchronous copy, and those copies land while the look-back runs; the
// kernel holds no payload registers.  Keys and payloads are then written out
// run by run (consecutive threads, consecutive addresses).
// A pass is bound by instructions and latency, not by DRAM (31 % of its peak):
// so a full tile has no bounds checks, a rank is kept with its digit in one
// word, the leader of a digit is the lane with none before it, and the warp
// histograms hold 16-bit counts, which with 64 (weighted) and 48 registers (44
// bytes of spill stores) gives four and five CTAs per SM.  One pass of 67 M keys by a 7-bit digit:
// 655 -> 435 us weighted (24 bytes per key: 3.7 TB/s), 627 -> 317 us unweighted
// (3.4 TB/s), against the version with match masks, 64-bit status words, one
// look-back word at a time and 32-bit histograms.  512 threads (476 us), 20 keys
// per thread (457 us) and payloads through registers were slower.
template <bool HAS_P1, int NB, class S, bool FULL>
__device__ __forceinline__ void onesweep_tile(const TileArgs<S>& a, uint32_t tile, uint32_t* s_dyn,
                                              uint16_t (*s_whist)[256], uint32_t* s_global_start, uint32_t* s_warp) {
  uint32_t* s_k = s_dyn;
  uint32_t* s_p0 = s_dyn + kTile;
  uint32_t* s_p1 = s_dyn + 2 * kTile;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t tile_base = (uint64_t)tile * kTile;
  const uint64_t warp_base = tile_base + (uint64_t)warp * 32 * kSortItems;
  // this warp's items: [0, wn) of kSortItems * 32, addressed from per-warp bases
  const uint32_t wn = FULL ? 32 * kSortItems
                           : (a.n > warp_base ? (uint32_t)min((uint64_t)kSortItems * 32, (uint64_t)a.n - warp_base) : 0u);
  const uint32_t* kw = a.kin + warp_base + lane;

  uint32_t key[kSortItems], rank[kSortItems];  // rank: digit << 16 | position among the warp's equal digits
#pragma unroll
  for (int i = 0; i < kSortItems; i++) key[i] = (FULL || (uint32_t)i * 32 + lane < wn) ? kw[i * 32] : 0xFFFFFFFFu;

  // Stable warp-level ranking: order within the warp is (item, lane).
  uint16_t* wh = s_whist[warp];
  const uint32_t before_me = lanemask_lt();
#pragma unroll
  for (int i = 0; i < kSortItems; i++) {
    const uint32_t d = (key[i] >> a.shift) & a.mask;
    const bool in = FULL || (uint32_t)i * 32 + lane < wn;
    const uint32_t peers = digit_peers<NB>(d, FULL ? 0xffffffffu : __ballot_sync(0xffffffffu, in));
    const uint32_t seen = wh[d];
    const uint32_t r = __popc(peers & before_me);
    __syncwarp();
    if (r == 0 && in) wh[d] = (uint16_t)(seen + __popc(peers));
    __syncwarp();
    rank[i] = seen + r + (d << 16);
  }
  __syncthreads();

  // Per digit (thread = digit): tile count, published, and its start in the
  // tile; each warp's histogram entry becomes the warp's start in the digit.
  static_assert(kSortThreads == 256, "a thread per digit");
  uint32_t cnt = 0, c[kWarps];
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    c[w] = s_whist[w][tid];
    cnt += c[w];
  }
  // digits above the mask never occur in this pass: no status, no look-back
  const bool live = tid <= a.mask;
  S* my_status = a.status + (uint64_t)tile * 256 + tid;
  if (live) lb_store(my_status, (tile == 0 ? LbWord<S>::kInc : LbWord<S>::kAgg) | (S)cnt);
  const uint32_t local_start = block_exclusive_scan_256(cnt, s_warp);
  uint32_t at = local_start;
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    s_whist[w][tid] = (uint16_t)at;
    at += c[w];
  }
  __syncthreads();

  // Stage slots (digit order within the tile): keys staged, payloads copied
  // into their slots asynchronously.
  {
    const uint32_t* p0w = a.p0in + warp_base + lane;
    const uint32_t* p1w = HAS_P1 ? a.p1in + warp_base + lane : nullptr;
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
      if (FULL || (uint32_t)i * 32 + lane < wn) {
        const uint32_t p = wh[rank[i] >> 16] + (rank[i] & 0xFFFFu);
        s_k[p] = key[i];
        cp_async_u32(&s_p0[p], p0w + i * 32);
        if (HAS_P1) cp_async_u32(&s_p1[p], p1w + i * 32);
      }
    }
  }

  // Decoupled look-back over earlier tiles for this digit, kLookBack of them
  // read at once (one at a time: 613 -> 562 us for a weighted pass).
  uint32_t excl = 0;
  if (tile > 0 && live) {
    int64_t pred = (int64_t)tile - 1;
    const S* col = a.status + tid;
    uint32_t spins = 0;
    bool done = false;
    while (!done && pred >= 0) {
      S s[kLookBack];
#pragma unroll
      for (int q = 0; q < kLookBack; q++)
        s[q] = pred - q >= 0 ? lb_load(col + (uint64_t)(pred - q) * 256) : LbWord<S>::kInc;
#pragma unroll
      for (int q = 0; q < kLookBack; q++) {
        if (done) continue;
        const S flag = s[q] & LbWord<S>::kFlag;
        if (flag == 0) {
          if (++spins > kSpinLimit) {
            atomicExch(a.err, (uint32_t)ERR_SPIN);
            done = true;
          }
          break;
        }
        excl += (uint32_t)(s[q] & ~LbWord<S>::kFlag);
        --pred;
        if (flag == LbWord<S>::kInc) done = true;
      }
    }
    lb_store(my_status, LbWord<S>::kInc | (S)(excl + cnt));
  }
  s_global_start[tid] = a.digit_base[tid] + excl - local_start;
  cp_async_commit_wait_all();
  __syncthreads();

  if (FULL) {
    constexpr int U = 4;
    static_assert(kSortItems % U == 0, "whole groups");
#pragma unroll 1
    for (uint32_t j0 = tid; j0 < kTile; j0 += U * kSortThreads) {
      uint32_t k[U], o[U];
#pragma unroll
      for (int u = 0; u < U; u++) k[u] = s_k[j0 + u * kSortThreads];
#pragma unroll
      for (int u = 0; u < U; u++) o[u] = s_global_start[(k[u] >> a.shift) & a.mask] + j0 + u * kSortThreads;
#pragma unroll
      for (int u = 0; u < U; u++) a.kout[o[u]] = k[u];
#pragma unroll
      for (int u = 0; u < U; u++) {
        a.p0out[o[u]] = s_p0[j0 + u * kSortThreads];
        if (HAS_P1) a.p1out[o[u]] = s_p1[j0 + u * kSortThreads];
      }
    }
  } else {
    const uint32_t valid = (uint32_t)min((uint64_t)kTile, (uint64_t)a.n - tile_base);
    for (uint32_t j = tid; j < valid; j += kSortThreads) {
      const uint32_t k = s_k[j];
      const uint32_t o = s_global_start[(k >> a.shift) & a.mask] + j;
      a.kout[o] = k;
      a.p0out[o] = s_p0[j];
      if (HAS_P1) a.p1out[o] = s_p1[j];
    }
  }
}

template <bool HAS_P1, int NB, class S>
__global__ void __launch_bounds__(kSortThreads, HAS_P1 ? 4 : 5) onesweep_kernel(const PassArgs<S> pa) {
  __shared__ uint32_t s_tile;
  __shared__ uint16_t s_whist[kWarps][256];
  __shared__ uint32_t s_global_start[256];
  __shared__ uint32_t s_warp[kWarps];
  extern __shared__ uint32_t s_dyn[];  // kTile keys, kTile payload0 [, kTile payload1]
  wait_for_prior_kernel();
  let_next_kernel_start();
  const PassPlan plan = *pa.plan;
  if (!plan.active) return;
  if (threadIdx.x == 0) s_tile = atomicAdd(pa.tile_ctr, 1u);
  for (int i = threadIdx.x; i < kWarps * 128; i += kSortThreads) reinterpret_cast<uint32_t*>(s_whist)[i] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  // src is 0, 1 or 2; dst 1 or 2
  const auto from = [&](uint32_t* const* b) { return plan.src == 0 ? b[0] : (plan.src == 1 ? b[1] : b[2]); };
  const auto to = [&](uint32_t* const* b) { return plan.dst == 1 ? b[1] : b[2]; };
  const TileArgs<S> a = {from(pa.k), from(pa.p0), HAS_P1 ? from(pa.p1) : nullptr,
                         to(pa.k),   to(pa.p0),   HAS_P1 ? to(pa.p1) : nullptr,
                         pa.n,       pa.shift,    pa.mask,
                         pa.digit_base, pa.status, pa.err};
  if (((uint64_t)tile + 1) * kTile <= a.n)
    onesweep_tile<HAS_P1, NB, S, true>(a, tile, s_dyn, s_whist, s_global_start, s_warp);
  else
    onesweep_tile<HAS_P1, NB, S, false>(a, tile, s_dyn, s_whist, s_global_start, s_warp);
}

template <bool HAS_P1, int NB, class S>
static int launch_pass_of(const PassArgs<S>& a, cudaStream_t stream) {
  constexpr size_t smem = (size_t)(HAS_P1 ? 3 : 2) * kTile * sizeof(uint32_t);  // a stage per array
  const auto kernel = onesweep_kernel<HAS_P1, NB, S>;
  OGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  OGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                cudaSharedmemCarveoutMaxShared));
  OGB_CUDA(launch_kernel(kernel, a.n < kDependentLimit, ceil_div(a.n, kTile), kSortThreads, smem, stream, a));
  return OK;
}

// One pass: the variant without the second payload when there is none, and
// seven ballots instead of eight when the digit has at most seven bits.
template <class S>
static int launch_pass(const PassArgs<S>& a, cudaStream_t stream) {
  const bool p1 = a.p1[0] != nullptr, narrow = a.mask < 128;
  if (p1) return narrow ? launch_pass_of<true, 7>(a, stream) : launch_pass_of<true, 8>(a, stream);
  return narrow ? launch_pass_of<false, 7>(a, stream) : launch_pass_of<false, 8>(a, stream);
}

}  // namespace

static size_t status_word_bytes(const SortWorkspace& ws, uint64_t n) {
  return n < kNarrowLimit && !ws.wide ? sizeof(uint32_t) : sizeof(unsigned long long);
}

int SortWorkspace::reserve(uint64_t n, bool weighted, int max_passes) {
  const uint64_t tiles = (n + kTile - 1) / kTile;
  OGB_TRY(hist.alloc((2 * 8 * 256 + kCtrWords) * sizeof(uint32_t)));
  OGB_TRY(status.alloc((size_t)max_passes * tiles * 256 * status_word_bytes(*this, n) + 256));
  OGB_TRY(tmp_k.alloc(n * 4));
  OGB_TRY(tmp_v0.alloc(n * 4));
  if (weighted) OGB_TRY(tmp_v1.alloc(n * 4));
  return OK;
}

static int sort_impl(const KV& in, const KV& out, uint64_t n, bool lex, uint32_t key_bits, SortWorkspace& ws,
                     cudaStream_t stream) {
  if (n == 0) return OK;
  if (n > 0xFFFFFFFFull) return fail(ERR_ARG, "sort: %llu edges exceed the u32 edge count", (unsigned long long)n);
  if (in.k == out.k || in.v0 == out.v0) return fail(ERR_ARG, "sort: input and output arrays must differ");
  const bool has_p1 = in.v1 != nullptr;
  if (has_p1 && !out.v1) return fail(ERR_ARG, "sort: weighted input needs a weighted output");
  OGB_TRY(ws.reserve(n, has_p1, lex ? 8 : 4));

  uint32_t* d_hist = ws.hist.as<uint32_t>();   // [8][256] counts
  uint32_t* d_ctr = d_hist + 8 * 256;          // counters and the plan
  uint32_t* d_base = d_ctr + kCtrWords;        // [8][256] exclusive bases
  OGB_CUDA(cudaMemsetAsync(d_hist, 0, (8 * 256 + kCtrWords) * sizeof(uint32_t), stream));

  const int grid = sm_count() * 4;
  // hist[0..3]: primary key digits; hist[4..7]: secondary key digits (lex).
  const DigitLayout lay = digit_layout(key_bits);
  const int P = (lex ? 2 : 1) * lay.ndig;
  const uint64_t tiles = (n + kTile - 1) / kTile;
  const size_t word = status_word_bytes(ws, n);
  digit_hist_kernel<<<grid, 256, 0, stream>>>(in.k, n, lay.ndig, lay, d_hist, ws.status.as<uint4>(),
                                              (uint64_t)P * tiles * 256 * word / 16);
  if (lex) digit_hist_kernel<<<grid, 256, 0, stream>>>(in.v0, n, lay.ndig, lay, d_hist + 4 * 256, nullptr, 0);
  OGB_CUDA(cudaGetLastError());

  // LSD order: secondary digits first (lex), then primary digits.  role 0: key =
  // primary (k), payloads (v0, v1); 1: key = secondary (v0), payloads (k, v1)
  struct Pass {
    int role, digit, hist;
  };
  Pass passes[kMaxPasses];
  for (int i = 0; i < P; i++) {
    const bool second = lex && i < lay.ndig;
    passes[i] = {second ? 1 : 0, i % lay.ndig, second ? 4 + i : i % lay.ndig};
  }
  PassPlan* d_plan = reinterpret_cast<PassPlan*>(d_ctr + kCtrPlan);
  PlanHists hists = {};
  for (int i = 0; i < P; i++) hists.h[i] = passes[i].hist;
  plan_kernel<<<1, 256, 0, stream>>>(d_hist, d_base, (uint32_t)n, hists, P, d_plan);
  OGB_CUDA(cudaGetLastError());

  const KV tmp{ws.tmp_k.as<uint32_t>(), ws.tmp_v0.as<uint32_t>(), has_p1 ? ws.tmp_v1.as<uint32_t>() : nullptr};
  const KV* bufs[3] = {&in, &tmp, &out};
  for (int i = 0; i < P; i++) {
    char* st = ws.status.as<char>() + (uint64_t)i * tiles * 256 * word;
    const auto fill = [&](auto& a) {
      for (int b = 0; b < 3; b++) {
        a.k[b] = passes[i].role == 0 ? bufs[b]->k : bufs[b]->v0;
        a.p0[b] = passes[i].role == 0 ? bufs[b]->v0 : bufs[b]->k;
        a.p1[b] = has_p1 ? bufs[b]->v1 : nullptr;
      }
      a.n = (uint32_t)n;
      a.shift = lay.shift[passes[i].digit];
      a.mask = lay.mask[passes[i].digit];
      a.digit_base = d_base + passes[i].hist * 256;
      a.status = reinterpret_cast<decltype(a.status)>(st);
      a.tile_ctr = d_ctr + i;
      a.err = const_cast<uint32_t*>(sort_error_word(ws));
      a.plan = d_plan + i;
    };
    if (word == sizeof(uint32_t)) {
      PassArgs<uint32_t> a;
      fill(a);
      OGB_TRY(launch_pass(a, stream));
    } else {
      PassArgs<unsigned long long> a;
      fill(a);
      OGB_TRY(launch_pass(a, stream));
    }
  }
  if (ws.give_up) {
    static const uint32_t gave_up = ERR_SPIN;
    ws.give_up--;
    OGB_CUDA(cudaMemsetAsync(out.v0, 0xFF, n * 4, stream));
    OGB_CUDA(cudaMemcpyAsync(const_cast<uint32_t*>(sort_error_word(ws)), &gave_up, 4, cudaMemcpyHostToDevice, stream));
  }
  return OK;
}

const uint32_t* sort_error_word(const SortWorkspace& ws) {
  return ws.err ? ws.err : ws.hist.as<uint32_t>() + 8 * 256 + kCtrErr;
}

int sort_pairs(const KV& in, const KV& out, uint64_t n, SortWorkspace& ws, cudaStream_t stream, uint32_t key_bits) {
  return sort_impl(in, out, n, false, key_bits, ws, stream);
}

int sort_pairs_lex(const KV& in, const KV& out, uint64_t n, SortWorkspace& ws, cudaStream_t stream,
                   uint32_t key_bits) {
  return sort_impl(in, out, n, true, key_bits, ws, stream);
}

// Reads the error word of the last sort with this workspace (synchronizes).
int sort_check(SortWorkspace& ws, cudaStream_t stream) {
  if (!ws.hist.p) return OK;
  uint32_t e = 0;
  OGB_CUDA(cudaMemcpyAsync(&e, sort_error_word(ws), 4, cudaMemcpyDeviceToHost, stream));
  OGB_CUDA(cudaStreamSynchronize(stream));
  if (e) return fail((int)e, "radix sort: decoupled look-back wait gave up");
  return OK;
}

}  // namespace ogb
