// Selection kernels: 1-D max-pool of stage-1 scores to 64-token block scores, and per-query
// top-k of block scores.  One warp per row, 16-byte loads, warp shuffles; the pool is bound by HBM, the
// top-k by instruction issue.
#include "common.cuh"

namespace ifv2 {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

template <typename T> struct Num;
template <> struct Num<__nv_bfloat16> {
  using T2 = __nv_bfloat162;
  static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float f) { return __float2bfloat16_rn(f); }
  static __device__ __forceinline__ __nv_bfloat16 from_bits(uint16_t b) {
    return __ushort_as_bfloat16(b);
  }
  static constexpr uint16_t kPosInf = 0x7F80, kNegInf = 0xFF80;
};
template <> struct Num<__half> {
  using T2 = __half2;
  static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from_f(float f) { return __float2half_rn(f); }
  static __device__ __forceinline__ __half from_bits(uint16_t b) { return __ushort_as_half(b); }
  static constexpr uint16_t kPosInf = 0x7C00, kNegInf = 0xFC00;
};

struct PoolParams {
  const void* in;
  void* out;
  const int32_t* cu_q;
  const int32_t* cu_k;
  const int32_t* cache_lens;
  int batch, heads;
  int64_t total_q;        // rows per head
  int k_len;              // fixed-length: keys per row; varlen: row width (max_seqlen_k)
  int64_t in_row_stride;
  int out_len, cache_len, kernel, stride, padding, block_size, local_blocks, init_blocks;
};

// Floor of x / d for a position x (rounded towards zero if negative): 32-bit wherever it fits, a
// 64-bit division costs as many instructions as a probe of the bisection.
__device__ __forceinline__ int block_of(int64_t x, int d) {
  return (x == (int64_t)(int)x) ? (int)x / d : (int)(x / d);
}

// kNarrow: the division through block_of (where a row holds enough work to hide its branch)
template <bool kVarlen, bool kNarrow = false>
__device__ __forceinline__ void row_geometry(const PoolParams& p, int64_t q, int& k_len, int& bq) {
  int64_t pos = q + p.cache_len;
  if constexpr (kVarlen) {
    const int b = find_sequence(p.cu_q, p.batch, (int)q);
    k_len = min(p.cu_k[b + 1] - p.cu_k[b], p.k_len);
    pos = q - p.cu_q[b] + p.cache_lens[b];
  } else {
    k_len = p.k_len;
  }
  bq = kNarrow ? block_of(pos, p.block_size) : (int)(pos / p.block_size);
}

// Fast path: kernel 5 / stride 4 / padding 1 (block 64 over compression stride 16) and 16-byte
// aligned rows.  A lane loads 8 consecutive scores and produces the two block scores whose
// windows they cover: block 2m <- x[8m-1 .. 8m+3], block 2m+1 <- x[8m+3 .. 8m+7].
// One load at a time per warp, 28-30 registers: rows of up to 768 scores, or with few of them to a block
// score, are bound by latency and issue, and more of them in flight count (8 heads x 4096 rows of 255 scores
// to 64 blocks: 8.6 us, 14.8 with the kernel below).
template <typename T, bool kVarlen>
__global__ void __launch_bounds__(kThreads) max_pool_k5s4_kernel(const PoolParams p) {
  using N = Num<T>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t rows = (int64_t)p.heads * p.total_q;
  const T* in = static_cast<const T*>(p.in);
  T* out = static_cast<T*>(p.out);
  const float ninf = -INFINITY;
  for (int64_t row = (int64_t)blockIdx.x * kWarps + warp; row < rows;
       row += (int64_t)gridDim.x * kWarps) {
    int k_len, bq;
    row_geometry<kVarlen>(p, row % p.total_q, k_len, bq);
    const T* x = in + row * p.in_row_stride;
    T* y = out + row * p.out_len;
    for (int m0 = 0; 2 * m0 < p.out_len; m0 += 32) {     // warp-uniform trip count (shuffles inside)
      const int m = m0 + lane, e0 = 8 * m;
      float v[8];
      if (e0 < k_len) {
        const uint4 raw = __ldg(reinterpret_cast<const uint4*>(x + e0));
        const T* t = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (e0 + j < k_len) ? N::to_f(t[j]) : ninf;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = ninf;
      }
      float prev = __shfl_up_sync(0xFFFFFFFFu, v[7], 1);
      // (lane 0 re-reads its neighbour's last score; it is in L1)
      if (lane == 0) prev = (e0 >= 1 && e0 - 1 < k_len) ? N::to_f(ldg16(x + e0 - 1)) : ninf;
      float r0 = fmaxf(fmaxf(prev, v[0]), fmaxf(fmaxf(v[1], v[2]), v[3]));
      float r1 = fmaxf(fmaxf(v[3], v[4]), fmaxf(fmaxf(v[5], v[6]), v[7]));
      const int b0 = 2 * m, b1 = b0 + 1;
      if (b0 >= p.out_len) continue;
      if (b0 < p.init_blocks || (bq >= b0 && bq <= b0 + p.local_blocks)) r0 = INFINITY;
      if (b1 < p.init_blocks || (bq >= b1 && bq <= b1 + p.local_blocks)) r1 = INFINITY;
      if ((p.out_len & 1) == 0) {
        typename N::T2 pr;
        pr.x = N::from_f(r0);
        pr.y = N::from_f(r1);
        *reinterpret_cast<typename N::T2*>(y + b0) = pr;
      } else {
        y[b0] = N::from_f(r0);
        if (b1 < p.out_len) y[b1] = N::from_f(r1);
      }
    }
  }
}

// Long rows, bound by HBM, which one load at a time per warp does not keep busy: a warp fetches kPoolBatch x
// 256 scores of its row before it uses the first; the score before a lane's eight comes from its neighbour or
// from the end of the 256 before.  44-64 registers.  65536 rows of 2047 scores to 512 blocks: 73.8 -> 61.5 us
// against the kernel above (5.5 TB/s), 63260 ragged rows of at most 1023: 41.9 -> 36.3 us.
constexpr int kPoolBatch = 4;
template <typename T, bool kVarlen>
__global__ void __launch_bounds__(kThreads) max_pool_k5s4_long_kernel(const PoolParams p) {
  using N = Num<T>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* in = static_cast<const T*>(p.in);
  T* out = static_cast<T*>(p.out);
  const float ninf = -INFINITY;
  // (heads are an axis of the grid: splitting a row number into head and token is a 64-bit division)
  for (int64_t head_row = (int64_t)blockIdx.y * p.total_q; head_row < p.heads * p.total_q;
       head_row += (int64_t)gridDim.y * p.total_q)
  for (int64_t q = (int64_t)blockIdx.x * kWarps + warp; q < p.total_q; q += (int64_t)gridDim.x * kWarps) {
    const int64_t row = head_row + q;
    int k_len, bq;
    row_geometry<kVarlen, true>(p, q, k_len, bq);
    const T* x = in + row * p.in_row_stride;
    T* y = out + row * p.out_len;
    float before = ninf;                                 // the score in front of the next 256
    for (int m0 = 0; 2 * m0 < p.out_len; m0 += 32 * kPoolBatch) {    // warp-uniform trip count (shuffles inside)
      uint4 raw[kPoolBatch];
#pragma unroll
      for (int u = 0; u < kPoolBatch; ++u) {
        const int e0 = 8 * (m0 + 32 * u + lane);
        raw[u] = make_uint4(0u, 0u, 0u, 0u);
        if (e0 < k_len) raw[u] = __ldg(reinterpret_cast<const uint4*>(x + e0));
      }
#pragma unroll
      for (int u = 0; u < kPoolBatch; ++u) {
        if (2 * (m0 + 32 * u) >= p.out_len) break;       // (the last batch of a row is seldom full)
        const int m = m0 + 32 * u + lane, e0 = 8 * m;
        const T* t = reinterpret_cast<const T*>(&raw[u]);
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (e0 + j < k_len) ? N::to_f(t[j]) : ninf;
        float prev = __shfl_up_sync(0xFFFFFFFFu, v[7], 1);           // x[8m-1]
        if (lane == 0) prev = before;
        before = __shfl_sync(0xFFFFFFFFu, v[7], 31);
        float r0 = fmaxf(fmaxf(prev, v[0]), fmaxf(fmaxf(v[1], v[2]), v[3]));
        float r1 = fmaxf(fmaxf(v[3], v[4]), fmaxf(fmaxf(v[5], v[6]), v[7]));
        const int b0 = 2 * m, b1 = b0 + 1;
        if (b0 >= p.out_len) continue;
        if (b0 < p.init_blocks || (bq >= b0 && bq <= b0 + p.local_blocks)) r0 = INFINITY;
        if (b1 < p.init_blocks || (bq >= b1 && bq <= b1 + p.local_blocks)) r1 = INFINITY;
        if ((p.out_len & 1) == 0) {
          typename N::T2 pr;
          pr.x = N::from_f(r0);
          pr.y = N::from_f(r1);
          *reinterpret_cast<typename N::T2*>(y + b0) = pr;
        } else {
          y[b0] = N::from_f(r0);
          if (b1 < p.out_len) y[b1] = N::from_f(r1);
        }
      }
    }
  }
}

// Generic path: any kernel/stride/padding and any alignment; a lane per output block.
template <typename T, bool kVarlen>
__global__ void __launch_bounds__(kThreads) max_pool_generic_kernel(const PoolParams p) {
  using N = Num<T>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t rows = (int64_t)p.heads * p.total_q;
  const T* in = static_cast<const T*>(p.in);
  T* out = static_cast<T*>(p.out);
  for (int64_t row = (int64_t)blockIdx.x * kWarps + warp; row < rows;
       row += (int64_t)gridDim.x * kWarps) {
    const int64_t q = row % p.total_q;
    int k_len, bq;
    row_geometry<kVarlen>(p, q, k_len, bq);
    const T* x = in + row * p.in_row_stride;
    T* y = out + row * p.out_len;
    for (int b = lane; b < p.out_len; b += 32) {
      float r;
      if (b < p.init_blocks || (bq >= b && bq <= b + p.local_blocks)) {
        r = INFINITY;
      } else {
        const int s = max(b * p.stride - p.padding, 0);
        const int e = min(b * p.stride - p.padding + p.kernel, k_len);
        r = -INFINITY;
        for (int i = s; i < e; ++i) r = fmaxf(r, N::to_f(ldg16(x + i)));
      }
      y[b] = N::from_f(r);
    }
  }
}

template <typename T, bool kVarlen>
int launch_pool(const PoolParams& p, cudaStream_t st) {
  const int64_t rows = (int64_t)p.heads * p.total_q;
  int64_t blocks = ceil_div64(rows, kWarps);
  const int64_t cap = (int64_t)kNumSMs * 8;
  if (blocks > cap) blocks = cap;
  const bool fast = p.kernel == 5 && p.stride == 4 && p.padding == 1 &&
                    (p.in_row_stride % 8 == 0) && (reinterpret_cast<uintptr_t>(p.in) % 16 == 0) &&
                    (reinterpret_cast<uintptr_t>(p.out) % 4 == 0);
  // The long kernel where its four loads have a whole row of scores to fetch (more than three times 256) and
  // the block scores ask for them; rows with far more blocks than scores only pay for its empty steps (1023
  // scores to 812 blocks: 84.5 us above, 89.8 below).  It was nowhere slower than the other within this line.
  if (fast && p.k_len > 768 && p.out_len > 192 && 2 * (int64_t)p.k_len >= 3 * (int64_t)p.out_len) {
    const int64_t gy = p.heads < 65535 ? p.heads : 65535;
    int64_t gx = ceil_div64(p.total_q, kWarps);
    const int64_t most = ceil_div64(cap, gy);
    if (gx > most) gx = most;
    max_pool_k5s4_long_kernel<T, kVarlen><<<dim3((unsigned)gx, (unsigned)gy), kThreads, 0, st>>>(p);
  } else if (fast) {
    max_pool_k5s4_kernel<T, kVarlen><<<(int)blocks, kThreads, 0, st>>>(p);
  } else
    max_pool_generic_kernel<T, kVarlen><<<(int)blocks, kThreads, 0, st>>>(p);
  return check_launch("max_pooling_1d");
}

// ---------------------------------------------------------------------------------------------
// Top-k: the k entries first in (value descending, index ascending) order, emitted ascending.
//
// A warp owns a row.  The row sits in registers as packed 16-bit pairs (lane-contiguous groups
// of 8 elements, so element index order is (iteration, lane, slot)).  The k-th largest value is
// found by bisection over the 16-bit ordered key space; each probe counts `x >= candidate`
// with native packed compares.  Entries above the threshold are all taken, entries equal to it
// are taken lowest index first; only ties and block lists need a warp prefix scan (byte counters,
// four iterations to a register).

struct TopkParams {
  const void* score;
  int32_t* out;                    // (heads, total_q, k) block lists, or null
  unsigned long long* mask;        // (heads, total_q, mask_words) packed selection, or null
  int mask_words;
  const int32_t* cu_q;
  const int32_t* cache_lens;
  int batch, heads;
  int64_t total_q;
  int n_blocks;
  int64_t row_stride;
  int k, cache_len, block_size;
};

// ordered key (0..65535, monotone in the float value) -> raw 16-bit pattern
__device__ __forceinline__ uint16_t ordered_to_bits(uint32_t o) {
  return (uint16_t)((o & 0x8000u) ? (o ^ 0x8000u) : (~o & 0xFFFFu));
}
__device__ __forceinline__ uint32_t bits_to_ordered(uint16_t b) {
  return (b & 0x8000u) ? (~(uint32_t)b & 0xFFFFu) : ((uint32_t)b | 0x8000u);
}

template <typename T> struct Pack;
template <> struct Pack<__nv_bfloat16> {
  using T2 = __nv_bfloat162;
  static __device__ __forceinline__ T2 splat(uint16_t bits) {
    return __halves2bfloat162(__ushort_as_bfloat16(bits), __ushort_as_bfloat16(bits));
  }
  // 0xFFFF in the half of the word whose comparison holds
  static __device__ __forceinline__ uint32_t ge_mask(T2 a, T2 b) { return __hge2_mask(a, b); }
  static __device__ __forceinline__ uint32_t gt_mask(T2 a, T2 b) { return __hgt2_mask(a, b); }
  static __device__ __forceinline__ uint32_t eq_mask(T2 a, T2 b) { return __heq2_mask(a, b); }
};
template <> struct Pack<__half> {
  using T2 = __half2;
  static __device__ __forceinline__ T2 splat(uint16_t bits) {
    return __halves2half2(__ushort_as_half(bits), __ushort_as_half(bits));
  }
  static __device__ __forceinline__ uint32_t ge_mask(T2 a, T2 b) { return __hge2_mask(a, b); }
  static __device__ __forceinline__ uint32_t gt_mask(T2 a, T2 b) { return __hgt2_mask(a, b); }
  static __device__ __forceinline__ uint32_t eq_mask(T2 a, T2 b) { return __heq2_mask(a, b); }
};

// Bits of the packed 0xFFFF / 0 masks of one iteration's four pairs, slot order.
__device__ __forceinline__ uint32_t slot_bits(uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
  const uint32_t t = (m0 & 0x00020001u) | (m1 & 0x00080004u) | (m2 & 0x00200010u) | (m3 & 0x00800040u);
  return (t | (t >> 16)) & 0xFFu;
}

// Exclusive prefix over the lanes of kRegs registers of four byte counters (at most 8 each, so the
// largest prefix, 31 * 8, fits its byte); totals[i] is the warp's sum of counter i.
template <int kRegs, int kCount>
__device__ __forceinline__ void scan_bytes(uint32_t (&c)[kRegs], int (&totals)[kCount], int lane) {
#pragma unroll
  for (int r = 0; r < kRegs; ++r) {
    const uint32_t mine = c[r];
    uint32_t e = __shfl_up_sync(0xFFFFFFFFu, mine, 1);
    if (lane == 0) e = 0u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, e, d);
      if (lane >= d) e += up;
    }
    const uint32_t e31 = __shfl_sync(0xFFFFFFFFu, e, 31), m31 = __shfl_sync(0xFFFFFFFFu, mine, 31);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (4 * r + i < kCount)
        totals[4 * r + i] = (int)(((e31 >> (8 * i)) & 0xFFu) + ((m31 >> (8 * i)) & 0xFFu));
    c[r] = e;
  }
}

// Selection over the first kIts iterations (256 entries each) of a row held in registers; the
// iteration count is a template parameter so that the probe and emit loops are straight-line
// code.  kList: the block list is written as well, which needs an output slot per entry; the mask
// alone needs no prefix scan unless entries tie at the threshold.  Returns the number of entries
// taken, or -1 when a restricted selection turns out not to be equivalent to the full one.
template <typename T, int kPairs, int kIts, bool kList>
__device__ __forceinline__ int topk_row(const typename Pack<T>::T2 (&v)[kPairs],
                                        typename Pack<T>::T2 tail2, bool restricted, int k_sel,
                                        int bq, int lane, int32_t* o, int k_cap,
                                        unsigned long long* mw, int mask_words) {
  using N = Num<T>;
  using P = Pack<T>;
  using T2 = typename P::T2;
  // ---- bisection for the k_sel-th largest value over ordered keys [-inf, +inf]
  uint32_t lo = bits_to_ordered(N::kNegInf), hi = bits_to_ordered(N::kPosInf) + 1u;
  bool exact = false;                     // count(x >= val(lo)) == k_sel: no tie handling needed
  int above = 0;                          // entries known to lie at or above val(hi)
  while (hi - lo > 1u) {
    const uint32_t mid = (lo + hi) >> 1;
    const T2 c = P::splat(ordered_to_bits(mid));
    // every comparison gives 0xFFFF per half that holds, and the sum of the words keeps both counts:
    // low * 0xFFFF - high * 0x10000 = (low - high) * 0x10000 - low
    uint32_t acc = 0u;
#pragma unroll
    for (int j = 0; j < kIts * 4; j += 2) acc += P::ge_mask(v[j], c) + P::ge_mask(v[j + 1], c);
    const int low = (int)((0u - acc) & 0xFFFFu);
    const int cnt = __reduce_add_sync(0xFFFFFFFFu, 2 * low - ((int)(acc + (uint32_t)low) >> 16));
    if (cnt >= k_sel) {
      lo = mid;
      if (cnt == k_sel) { exact = true; break; }
    } else {
      hi = mid;
      above = cnt;
    }
  }
  const T2 thr = P::splat(ordered_to_bits(lo));
  if (restricted) {
    // a later entry above the threshold would have displaced one of the selected ones
    const float tm = fmaxf(N::to_f(tail2.x), N::to_f(tail2.y));
    const bool bad = tm > N::to_f(thr.x);
    if (__any_sync(0xFFFFFFFFu, bad)) return -1;        // redo over the full width
  }

  // ---- slots taken, one byte per iteration
  uint32_t taken[kIts];
  if (exact) {
#pragma unroll
    for (int it = 0; it < kIts; ++it)
      taken[it] = slot_bits(P::ge_mask(v[it * 4], thr), P::ge_mask(v[it * 4 + 1], thr),
                            P::ge_mask(v[it * 4 + 2], thr), P::ge_mask(v[it * 4 + 3], thr));
  } else {
    // entries equal to the threshold are taken lowest index first until k_sel are there; the
    // bisection ended with hi = lo + 1, so `above` counts the entries above the threshold
    const int need = k_sel - above;
    constexpr int kRegs = (kIts + 3) / 4;
    uint32_t excl[kRegs];
    int totals[kIts];
#pragma unroll
    for (int r = 0; r < kRegs; ++r) excl[r] = 0u;
    uint32_t tie[kIts];
#pragma unroll
    for (int it = 0; it < kIts; ++it) {
      taken[it] = slot_bits(P::gt_mask(v[it * 4], thr), P::gt_mask(v[it * 4 + 1], thr),
                            P::gt_mask(v[it * 4 + 2], thr), P::gt_mask(v[it * 4 + 3], thr));
      tie[it] = slot_bits(P::eq_mask(v[it * 4], thr), P::eq_mask(v[it * 4 + 1], thr),
                          P::eq_mask(v[it * 4 + 2], thr), P::eq_mask(v[it * 4 + 3], thr));
      excl[it >> 2] |= (uint32_t)__popc(tie[it]) << (8 * (it & 3));
    }
    scan_bytes<kRegs, kIts>(excl, totals, lane);
    int base = 0;
#pragma unroll
    for (int it = 0; it < kIts; ++it) {
      int left = need - base - (int)((excl[it >> 2] >> (8 * (it & 3))) & 0xFFu);
      uint32_t t = tie[it];
      if (left < __popc(t)) {               // only the first `left` of this lane's ties
        uint32_t rest = t;
        for (; left > 0; --left) rest &= rest - 1u;
        t ^= rest;
      }
      taken[it] |= t;
      base += totals[it];
    }
  }

  // ---- packed mask: four lanes own the 32 entries of one half word; entries past the query's own
  // block are taken (they fill list slots) but invisible
  if (mw != nullptr) {
    uint32_t* mh = reinterpret_cast<uint32_t*>(mw);
#pragma unroll
    for (int it = 0; it < kIts; ++it) {
      const int e0 = (it * 32 + lane) * 8;
      const uint32_t vis = (bq >= e0 + 7) ? 0xFFu : ((bq < e0) ? 0u : ((2u << (bq - e0)) - 1u));
      uint32_t wv = (taken[it] & vis) << (8 * (lane & 3));
      wv |= __shfl_xor_sync(0xFFFFFFFFu, wv, 1);
      wv |= __shfl_xor_sync(0xFFFFFFFFu, wv, 2);
      const int w = it * 8 + (lane >> 2);
      if ((lane & 3) == 0 && w < 2 * mask_words) mh[w] = wv;
    }
  }

  // ---- block list, in index order
  int total = 0;
  if (kList) {
    constexpr int kRegs = (kIts + 3) / 4;
    uint32_t excl[kRegs];
    int totals[kIts];
#pragma unroll
    for (int r = 0; r < kRegs; ++r) excl[r] = 0u;
#pragma unroll
    for (int it = 0; it < kIts; ++it) excl[it >> 2] |= (uint32_t)__popc(taken[it]) << (8 * (it & 3));
    scan_bytes<kRegs, kIts>(excl, totals, lane);
#pragma unroll
    for (int it = 0; it < kIts; ++it) {
      const int e0 = (it * 32 + lane) * 8;
      int pos = total + (int)((excl[it >> 2] >> (8 * (it & 3))) & 0xFFu);
      uint32_t sel = taken[it];
      while (sel) {
        const int idx = e0 + __ffs(sel) - 1;
        sel &= sel - 1u;
        // (guarded by the capacity of the row: a slot outside [0, k) is never written)
        if ((unsigned)pos < (unsigned)k_cap) o[pos] = (idx <= bq) ? idx : -1;
        ++pos;
      }
      total += totals[it];
    }
  }
  return total;
}

// CTAs per SM the kernel is compiled for: a probe is a chain of compares, a warp reduction and a branch,
// so what matters is how many rows are in flight.
template <int kIters> constexpr int kTopkResident = kIters == 2 ? 5 : kIters == 4 ? 4 : kIters <= 8 ? 3 : 1;

// Bound by instruction issue and by the latency of the probes (a row is read once, everything else
// happens in registers).  Over 1 M rows of 2048 blocks, mask only: 6.88 -> 2.28 ms against a form that
// scanned the lanes once per 256 entries, counted in bf16 and walked the taken entries even where no list
// was wanted; with the list, 65536 rows of 512 blocks: 0.112 -> 0.101 ms.
template <typename T, int kIters, bool kList>
__global__ void __launch_bounds__(kThreads, kTopkResident<kIters>) topk_select_kernel(const TopkParams p) {
  using N = Num<T>;
  using P = Pack<T>;
  using T2 = typename P::T2;
  constexpr int kPairs = kIters * 4;          // packed registers per lane
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* score = static_cast<const T*>(p.score);
  const int n = p.n_blocks;
  const int k_eff = min(p.k, n);
  const bool aligned = (p.row_stride % 8 == 0) && (reinterpret_cast<uintptr_t>(p.score) % 16 == 0);
  const T2 pad2 = P::splat(N::kNegInf);
  const T ninf = N::from_bits(N::kNegInf);

  // (heads are an axis of the grid: splitting a row number into head and token is a 64-bit division)
  for (int64_t head_row = (int64_t)blockIdx.y * p.total_q; head_row < p.heads * p.total_q;
       head_row += (int64_t)gridDim.y * p.total_q)
  for (int64_t q = (int64_t)blockIdx.x * kWarps + warp; q < p.total_q; q += (int64_t)gridDim.x * kWarps) {
    const int64_t row = head_row + q;
    int bq;
    if (p.cu_q != nullptr) {
      const int b = find_sequence(p.cu_q, p.batch, (int)q);
      const int cl = p.cache_lens ? p.cache_lens[b] : p.cache_len;
      bq = block_of(q - p.cu_q[b] + cl, p.block_size);
    } else {
      bq = block_of(q + p.cache_len, p.block_size);
    }
    const T* x = score + row * p.row_stride;
    int32_t* o = kList ? p.out + row * p.k : nullptr;
    unsigned long long* mw = p.mask ? p.mask + row * p.mask_words : nullptr;

    // Entries past the query's own block only ever come out as -1.  When none of them beats the
    // k-th best earlier entry (always the case for stage-1 block scores: later blocks hold 0 or
    // -inf and ties go to the lower index) the selection can run over the earlier entries alone;
    // that is checked after the fact, and a row that fails it is redone over the full width.
    const int head = min(n, bq + 1);
    int emitted = 0;
    for (int attempt = 0; attempt < 2; ++attempt) {
      const bool restricted = (attempt == 0) && head < n;
      const int width = restricted ? head : n;              // entries that take part
      const int its = (width + 255) >> 8;                   // 256 entries per iteration
      const int k_sel = min(k_eff, width);

      // ---- load: element index of (it, lane, slot) is (it*32 + lane)*8 + slot
      T2 v[kPairs];
#pragma unroll
      for (int it = 0; it < kIters; ++it) {
        const int e0 = (it * 32 + lane) * 8;
        if (aligned && e0 + 8 <= n) {
          const uint4 raw = __ldg(reinterpret_cast<const uint4*>(x + e0));
          const T2* t = reinterpret_cast<const T2*>(&raw);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[it * 4 + j] = t[j];
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            T2 pr = pad2;
            if (e0 + 2 * j < n) pr.x = ldg16(x + e0 + 2 * j);
            if (e0 + 2 * j + 1 < n) pr.y = ldg16(x + e0 + 2 * j + 1);
            v[it * 4 + j] = pr;
          }
        }
      }
      // ---- split off the entries past `width`: their maximum is kept, their slots become -inf
      T2 tail2 = pad2;
      if (restricted) {
#pragma unroll
        for (int it = 0; it < kIters; ++it) {
          const int nh = width - (it * 32 + lane) * 8;      // entries of this lane that take part
          if (nh <= 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              tail2 = __hmax2(tail2, v[it * 4 + j]);
              v[it * 4 + j] = pad2;
            }
          } else if (nh < 8) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              T2 pr = v[it * 4 + j], tl = pad2;
              if (2 * j >= nh) { tl.x = pr.x; pr.x = ninf; }
              if (2 * j + 1 >= nh) { tl.y = pr.y; pr.y = ninf; }
              tail2 = __hmax2(tail2, tl);
              v[it * 4 + j] = pr;
            }
          }
        }
      }

      // ---- bisection + emission over the `its` iterations that take part
      // (an even iteration count keeps the number of instantiated bodies, and with it the
      //  instruction-cache footprint, small; the extra iteration only holds -inf slots)
      int got = -1;
      const int its_used = min(kIters, (its + 1) & ~1);
      switch (its_used) {
#define IFV2_TOPK_CASE(I)                                                                \
        case I:                                                                          \
          if constexpr (I <= kIters)                                                     \
            got = topk_row<T, kPairs, I, kList>(v, tail2, restricted, k_sel, bq, lane, o, p.k,  \
                                                mw, p.mask_words);                       \
          break;
        IFV2_TOPK_CASE(2) IFV2_TOPK_CASE(4) IFV2_TOPK_CASE(6)
#undef IFV2_TOPK_CASE
        default:
          got = topk_row<T, kPairs, kIters, kList>(v, tail2, restricted, k_sel, bq, lane, o, p.k, mw,
                                                   p.mask_words);
          break;
      }
      if (got < 0) continue;
      emitted = got;
      // mask words past the iterations that took part hold no selected block
      if (mw != nullptr) {
        const int covered = (its_used == 2 || its_used == 4 || its_used == 6 ? its_used : kIters) * 4;
        for (int w = covered + lane; w < p.mask_words; w += 32) mw[w] = 0ull;
      }
      break;
    }
    // unused tail (k > entries that took part, or NaN scores that no probe counts)
    if (kList)
      for (int i = emitted + lane; i < p.k; i += 32) o[i] = -1;
  }
}

template <typename T, int kIters>
void launch_topk_iters(const TopkParams& p, cudaStream_t st) {
  const int64_t gy = p.heads < 65535 ? p.heads : 65535;
  // One wave: every warp strides over the rows, so a second, partly filled wave would leave SMs idle
  // (2048 blocks: 2.28 -> 2.22 ms of 1 M rows; 512 blocks, with 5 instead of 3 CTAs per SM: 0.101 ->
  // 0.094 ms of 65536).  Rows of at most 256 blocks are so short that a row per warp and more CTAs than
  // fit are better (64 blocks, 8192 rows: 12.4 us against 14.4).  Above 4096 blocks one CTA of eight warps
  // fills an SM, rows that have to be redone over their full width take twice as long as others, and CTAs
  // that are handed out as SMs become free even that out: 32768 rows of 6000 blocks, all redone, 935 us
  // against 1524 with one wave, none redone 653 against 880.
  int64_t cap = (int64_t)kNumSMs * (kIters == 1 || kIters == 32 ? 8 : kTopkResident<kIters>) / gy;
  if (cap < 1) cap = 1;
  int64_t gx = ceil_div64(p.total_q, kWarps);
  if (gx > cap) gx = cap;
  const dim3 grid((unsigned)gx, (unsigned)gy);
  if (p.out != nullptr)
    topk_select_kernel<T, kIters, true><<<grid, kThreads, 0, st>>>(p);
  else
    topk_select_kernel<T, kIters, false><<<grid, kThreads, 0, st>>>(p);
}

template <typename T>
int launch_topk(const TopkParams& p, cudaStream_t st) {
  if (p.n_blocks <= 256)
    launch_topk_iters<T, 1>(p, st);
  else if (p.n_blocks <= 512)
    launch_topk_iters<T, 2>(p, st);
  else if (p.n_blocks <= 1024)
    launch_topk_iters<T, 4>(p, st);
  else if (p.n_blocks <= 2048)
    launch_topk_iters<T, 8>(p, st);
  else if (p.n_blocks <= 4096)
    launch_topk_iters<T, 16>(p, st);
  else
    launch_topk_iters<T, 32>(p, st);
  return check_launch("topk_select");
}

}  // namespace
}  // namespace ifv2

using namespace ifv2;

static int check_pool_args(const void* in, const void* out, int heads, int64_t total_q, int k_len,
                           int64_t in_row_stride, int out_len, int kernel, int stride, int padding,
                           int block_size, int local_blocks, int init_blocks) {
  IFV2_REQUIRE(heads >= 0 && total_q >= 0 && k_len >= 0 && out_len >= 0, IFV2_ERR_INVALID_ARG,
               "max_pooling_1d: negative size");
  IFV2_REQUIRE(kernel >= 1 && stride >= 1 && padding >= 0 && block_size >= 1, IFV2_ERR_INVALID_ARG,
               "max_pooling_1d: kernel/stride/block_size must be >= 1 and padding >= 0");
  IFV2_REQUIRE(local_blocks >= 0 && init_blocks >= 0, IFV2_ERR_INVALID_ARG,
               "max_pooling_1d: local_blocks / init_blocks must be >= 0");
  IFV2_REQUIRE(in_row_stride >= k_len, IFV2_ERR_INVALID_ARG,
               "max_pooling_1d: in_row_stride (%lld) < k_len (%d)", (long long)in_row_stride, k_len);
  if (heads == 0 || total_q == 0 || out_len == 0) return 1;   // nothing to do
  IFV2_REQUIRE(in != nullptr || k_len == 0, IFV2_ERR_INVALID_ARG, "max_pooling_1d: null input");
  IFV2_REQUIRE(out != nullptr, IFV2_ERR_INVALID_ARG, "max_pooling_1d: null output");
  return 0;
}

extern "C" int ifv2_max_pooling_1d(const void* in, void* out, int is_bf16, int heads, int q_len,
                                   int k_len, int64_t in_row_stride, int out_len, int cache_len,
                                   int kernel_size, int stride, int padding, int block_size,
                                   int local_blocks, int init_blocks, void* stream) {
  int rc = check_pool_args(in, out, heads, q_len, k_len, in_row_stride, out_len, kernel_size, stride,
                           padding, block_size, local_blocks, init_blocks);
  if (rc != 0) return rc > 0 ? IFV2_OK : rc;
  IFV2_REQUIRE(cache_len >= 0, IFV2_ERR_INVALID_ARG, "max_pooling_1d: cache_len < 0");
  PoolParams p{in, out, nullptr, nullptr, nullptr, 1, heads, q_len, k_len, in_row_stride, out_len,
               cache_len, kernel_size, stride, padding, block_size, local_blocks, init_blocks};
  return is_bf16 ? launch_pool<__nv_bfloat16, false>(p, (cudaStream_t)stream)
                 : launch_pool<__half, false>(p, (cudaStream_t)stream);
}

extern "C" int ifv2_max_pooling_1d_varlen(const void* in, void* out, const int32_t* cu_seqlens_q,
                                          const int32_t* cu_seqlens_k, const int32_t* cache_lens,
                                          int is_bf16, int batch, int heads, int64_t total_q,
                                          int max_seqlen_k, int64_t in_row_stride, int out_len,
                                          int kernel_size, int stride, int padding, int block_size,
                                          int local_blocks, int init_blocks, void* stream) {
  int rc = check_pool_args(in, out, heads, total_q, max_seqlen_k, in_row_stride, out_len, kernel_size,
                           stride, padding, block_size, local_blocks, init_blocks);
  if (rc != 0) return rc > 0 ? IFV2_OK : rc;
  IFV2_REQUIRE(batch >= 1 && cu_seqlens_q && cu_seqlens_k && cache_lens, IFV2_ERR_INVALID_ARG,
               "max_pooling_1d_varlen: batch >= 1 and cu_seqlens_q/cu_seqlens_k/cache_lens required");
  IFV2_REQUIRE(total_q <= INT32_MAX, IFV2_ERR_TOO_LARGE, "max_pooling_1d_varlen: total_q > 2^31-1");
  PoolParams p{in, out, cu_seqlens_q, cu_seqlens_k, cache_lens, batch, heads, total_q, max_seqlen_k,
               in_row_stride, out_len, 0, kernel_size, stride, padding, block_size, local_blocks,
               init_blocks};
  return is_bf16 ? launch_pool<__nv_bfloat16, true>(p, (cudaStream_t)stream)
                 : launch_pool<__half, true>(p, (cudaStream_t)stream);
}

extern "C" int ifv2_topk_select(const void* score, int32_t* out_idx, int is_bf16, int heads,
                                int64_t total_q, int n_blocks, int64_t row_stride, int k,
                                const int32_t* cu_seqlens_q, const int32_t* cache_lens, int batch,
                                int cache_len, int block_size, void* stream) {
  IFV2_REQUIRE(heads >= 0 && total_q >= 0 && n_blocks >= 0 && k >= 0, IFV2_ERR_INVALID_ARG,
               "topk_select: negative size");
  IFV2_REQUIRE(block_size >= 1 && cache_len >= 0, IFV2_ERR_INVALID_ARG,
               "topk_select: block_size must be >= 1 and cache_len >= 0");
  IFV2_REQUIRE(row_stride >= n_blocks, IFV2_ERR_INVALID_ARG, "topk_select: row_stride < n_blocks");
  IFV2_REQUIRE(n_blocks <= 8192, IFV2_ERR_TOO_LARGE,
               "topk_select: n_blocks = %d exceeds the 8192-block limit", n_blocks);
  IFV2_REQUIRE(cache_lens == nullptr || cu_seqlens_q != nullptr, IFV2_ERR_INVALID_ARG,
               "topk_select: cache_lens needs cu_seqlens_q");
  IFV2_REQUIRE(cu_seqlens_q == nullptr || batch >= 1, IFV2_ERR_INVALID_ARG,
               "topk_select: batch must be >= 1 with cu_seqlens_q");
  if (heads == 0 || total_q == 0 || k == 0) return IFV2_OK;
  IFV2_REQUIRE(out_idx != nullptr && (score != nullptr || n_blocks == 0), IFV2_ERR_INVALID_ARG,
               "topk_select: null pointer");
  IFV2_REQUIRE(total_q <= INT32_MAX, IFV2_ERR_TOO_LARGE, "topk_select: total_q > 2^31-1");
  TopkParams p{score, out_idx, nullptr, 0, cu_seqlens_q, cache_lens, batch, heads, total_q, n_blocks,
               row_stride, k, cache_len, block_size};
  return is_bf16 ? launch_topk<__nv_bfloat16>(p, (cudaStream_t)stream)
                 : launch_topk<__half>(p, (cudaStream_t)stream);
}

extern "C" int ifv2_topk_select_mask(const void* score, int32_t* out_idx, int64_t* row_mask,
                                     int64_t* col_mask, int is_bf16, int heads, int64_t total_q,
                                     int n_blocks, int64_t row_stride, int k, int k_blocks,
                                     const int32_t* cu_seqlens_q, const int32_t* cache_lens, int batch,
                                     int cache_len, int block_size, void* stream) {
  IFV2_REQUIRE(heads >= 0 && total_q >= 0 && n_blocks >= 0 && k >= 0 && k_blocks >= 0,
               IFV2_ERR_INVALID_ARG, "topk_select_mask: negative size");
  IFV2_REQUIRE(block_size >= 1 && cache_len >= 0, IFV2_ERR_INVALID_ARG,
               "topk_select_mask: block_size must be >= 1 and cache_len >= 0");
  IFV2_REQUIRE(row_stride >= n_blocks, IFV2_ERR_INVALID_ARG, "topk_select_mask: row_stride < n_blocks");
  IFV2_REQUIRE(n_blocks <= 8192 && k_blocks <= 8192, IFV2_ERR_TOO_LARGE,
               "topk_select_mask: n_blocks = %d / k_blocks = %d exceed the 8192-block limit", n_blocks,
               k_blocks);
  IFV2_REQUIRE(cache_lens == nullptr || cu_seqlens_q != nullptr, IFV2_ERR_INVALID_ARG,
               "topk_select_mask: cache_lens needs cu_seqlens_q");
  IFV2_REQUIRE(cu_seqlens_q == nullptr || batch >= 1, IFV2_ERR_INVALID_ARG,
               "topk_select_mask: batch must be >= 1 with cu_seqlens_q");
  if (heads == 0 || total_q == 0 || k_blocks == 0) return IFV2_OK;
  IFV2_REQUIRE(row_mask != nullptr && (score != nullptr || n_blocks == 0), IFV2_ERR_INVALID_ARG,
               "topk_select_mask: null pointer");
  IFV2_REQUIRE(total_q <= INT32_MAX, IFV2_ERR_TOO_LARGE, "topk_select_mask: total_q > 2^31-1");
  const int words = (k_blocks + 63) / 64;
  TopkParams p{score, out_idx, reinterpret_cast<unsigned long long*>(row_mask), words, cu_seqlens_q,
               cache_lens, batch, heads, total_q, n_blocks, row_stride, k, cache_len, block_size};
  int rc = is_bf16 ? launch_topk<__nv_bfloat16>(p, (cudaStream_t)stream)
                   : launch_topk<__half>(p, (cudaStream_t)stream);
  if (rc != IFV2_OK || col_mask == nullptr) return rc;
  return ifv2_transpose_blockmask(row_mask, col_mask, heads, total_q, k_blocks, stream);
}
