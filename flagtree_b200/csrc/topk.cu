// Top-k index producer: the step in front of the sparse MLA forward.  For every query token the positions of the
// `topk` largest scores among its first `length` key positions, written in ascending position order and padded
// with -1: exactly the index list the forward takes.
//
// Selection is exact and deterministic: scores are mapped to 32-bit keys whose unsigned order is the order of the
// floats (-0 below +0, NaN patterns above +inf, as an unsigned compare of the transformed bits gives), the k-th
// largest key is found by a radix select (four passes of 8 bits, a 256-bin histogram per pass in shared memory),
// and among the entries equal to that key the lowest positions are taken.  One CTA per row; the row is read from
// memory once and from L2 in the later passes, so the kernel is bound by device-memory traffic:
// 4 * s_kv bytes of scores per token (plus 4 * topk bytes of output).
#include "sm100.cuh"

namespace ftb {

void set_last_error(const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

namespace topk {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;

struct Params {
  const float* scores;
  const int32_t* lengths;
  int32_t* out;
  int s_q, s_kv, topk;
  long long sc_stride, out_stride;
};

__device__ __forceinline__ uint32_t to_key(uint32_t u) {
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// exclusive prefix of `flag` over the block in thread order; `total` = number of set flags (same in every thread)
__device__ __forceinline__ int block_exclusive(bool flag, int* warp_sums, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned b = __ballot_sync(0xffffffffu, flag);
  const int in_warp = __popc(b & ((1u << lane) - 1u));
  if (lane == 0) warp_sums[warp] = __popc(b);
  __syncthreads();
  int before = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const int v = warp_sums[w];
    before += (w < warp) ? v : 0;
    tot += v;
  }
  __syncthreads();       // warp_sums is reused by the next call
  total = tot;
  return before + in_warp;
}

__global__ void __launch_bounds__(kThreads) topk_select_kernel(const Params p) {
  __shared__ int hist[256];
  __shared__ int warp_sums[kWarps];
  __shared__ uint32_t s_bin;
  __shared__ int s_remaining;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = blockIdx.x;
  const uint32_t* sc = reinterpret_cast<const uint32_t*>(p.scores) + static_cast<long long>(row) * p.sc_stride;   // bits: NaN patterns keep theirs
  int32_t* out = p.out + static_cast<long long>(row) * p.out_stride;
  int len = p.lengths != nullptr ? p.lengths[row] : p.s_kv;
  len = max(0, min(len, p.s_kv));
  const int k = min(p.topk, len);

  uint32_t thresh = 0;       // key of the k-th largest entry
  int need_eq = 0;           // how many entries equal to it are taken (the lowest positions)
  if (k < len) {
    uint32_t prefix = 0, mask = 0;
    int remaining = k;
#pragma unroll 1
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass;
      if (tid < 256) hist[tid] = 0;
      __syncthreads();
      for (int i = tid; i < len; i += kThreads) {
        const uint32_t key = to_key(sc[i]);
        if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1);
      }
      __syncthreads();
      if (warp == 0) {
        // lane l owns bins 8l .. 8l + 7; walk from the largest bin down to the one that holds the `remaining`-th largest
        int mine = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) mine += hist[8 * lane + j];
        int above = 0;                                   // entries in the bins of higher lanes
#pragma unroll
        for (int l = 0; l < 32; ++l) {
          const int v = __shfl_sync(0xffffffffu, mine, l);
          above += (l > lane) ? v : 0;
        }
        if (above < remaining && above + mine >= remaining) {
          int cum = above;
          for (int j = 7; j >= 0; --j) {
            const int h = hist[8 * lane + j];
            if (cum + h >= remaining) {
              s_bin = static_cast<uint32_t>(8 * lane + j);
              s_remaining = remaining - cum;
              break;
            }
            cum += h;
          }
        }
      }
      __syncthreads();
      prefix |= s_bin << shift;
      mask |= 255u << shift;
      remaining = s_remaining;
      __syncthreads();
    }
    thresh = prefix;
    need_eq = remaining;
  }

  // ordered compaction: positions in ascending order, entries above the threshold and the first need_eq equal to it
  int written = 0, eq_seen = 0;
  for (int start = 0; start < len; start += kThreads) {
    const int i = start + tid;
    bool take = false, eq = false;
    if (i < len) {
      if (k == len) {
        take = true;
      } else {
        const uint32_t key = to_key(sc[i]);
        take = key > thresh;
        eq = key == thresh;
      }
    }
    if (k < len) {
      int eq_total;
      const int eq_rank = eq_seen + block_exclusive(eq, warp_sums, eq_total);
      if (eq && eq_rank < need_eq) take = true;
      eq_seen += eq_total;
    }
    int take_total;
    const int pos = written + block_exclusive(take, warp_sums, take_total);
    if (take) out[pos] = i;
    written += take_total;
  }
  for (int j = k + tid; j < p.topk; j += kThreads) out[j] = -1;
}


// ---------------------------------------------------------------------------------------------------------------
// Rows of at most 65536 scores: persistent CTAs of 1024 threads, one per SM.  Thread t holds the keys of positions
// t, t + 1024, ... (32 in registers; rows of more than 32768 scores keep the rest in shared memory), so that a vote over a
// warp is the mask of 32 consecutive positions.  Rows of at most 32768 scores are copied into shared memory one row
// ahead by asynchronous copies; scores are read from device memory
// once.
//
// Bound by instruction issue, so the work per key is kept to a few instructions and no key goes through a shared-memory
// atomic (they retire about one lane per clock).  A sample of 128 or 256 keys, ranked by counting, brackets the k-th largest key
// a few standard deviations of the sample quantile either side (or only from below, where all above fits the list); one
// sweep counts the keys of the bracket and copies them to a list, an eighth of the row or so.  The list is counted
// against four trial values at a time, keys of the sample first, then interpolated between the counts known so far (the
// keys are spread evenly enough there that two or three rounds leave 128 candidates), and the last few are ranked by counting.  A bracket that does not hold
// the k-th key, or more keys than the list, is not used: the interval is then halved by counting the whole row.  Both are
// checked, so a bad sample costs time (32 sweeps) and never exactness.  A last sweep votes the taken positions into masks,
// and one scan over their counts gives every mask its place in the ordered output.
// 128 rows of 28 000 scores on average out of 65 536 (a decode step): 138 us with a radix select that read the row five times,
// about 30 us here; the step 360 -> 253 us.  4096 rows of 32 768: 334 us, as a histogram of the bracket in per-lane counters
// took, which could only serve 16-byte aligned rows of at most 32 768 scores.
// ---------------------------------------------------------------------------------------------------------------
constexpr int kHalf = 32768;                               // scores held in registers
constexpr int kRowMax = 2 * kHalf;
constexpr int kBigThreads = 1024;
constexpr int kBigWarps = kBigThreads / 32;
constexpr int kPerThread = kHalf / kBigThreads;            // 32 keys per thread
constexpr int kSampleMax = 256;
constexpr int kSampleMinLen = 4096;                        // shorter rows are selected without a bracket
constexpr int kListPer = 8;
constexpr int kListMax = kListPer * kBigThreads;
constexpr int kWords = kRowMax / 32;
constexpr int kFew = 128;                                  // this many candidates are ranked by counting
constexpr size_t kBigSmem = (static_cast<size_t>(kHalf) + kListMax + 2 * kWords + kSampleMax + 4 * kBigWarps + kFew + 16) * 4;

enum { kCtlLo = 0, kCtlHi, kCtlFirst, kCtlAbove = kCtlFirst + 4, kCtlList, kCtlFew, kCtlLimit, kCtlNeedEq };

__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ int row_len(const Params& p, int row) {
  const int len = p.lengths != nullptr ? p.lengths[row] : p.s_kv;
  return max(0, min(len, p.s_kv));
}

// scores src[0 .. n) -> buf, filled up to `full` with the pattern whose key is 0, by asynchronous copies of the calling threads: of 16
// bytes where the row is aligned
__device__ __forceinline__ void fetch(const uint32_t* src, int n, int full, uint32_t* buf) {
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    for (int c = threadIdx.x; c < n >> 2; c += kBigThreads) cp_async16(smem_u32(buf + 4 * c), src + 4 * c);
    const int tail = (n & ~3) + threadIdx.x;
    if (tail < n) cp_async4(buf + tail, src + tail);
  } else {
    for (int c = threadIdx.x; c < n; c += kBigThreads) cp_async4(buf + c, src + c);
  }
  for (int pad = n + threadIdx.x; pad < full; pad += kBigThreads) buf[pad] = 0xffffffffu;
}

template <bool kLong>
__global__ void __launch_bounds__(kBigThreads, 1) topk_select_rows_kernel(const Params p) {
  // Sample keys: a smaller sample is cheaper to rank and widens the bracket; rows of more than 32768 scores would
  // overflow the list with 128 (65536 scores, 2048 wanted: 6100 keys expected above the lower end).
  constexpr int kSample = kLong ? 256 : 128, kRankers = kBigThreads / kSample;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t* buf = reinterpret_cast<uint32_t*>(smem_raw);         // kLong: the second half of the row; else the next row in flight
  uint32_t* list = buf + kHalf;                          // [kListMax] keys inside the bracket
  uint32_t* gt_words = list + kListMax;                                              // [kWords] taken positions
  uint32_t* eq_words = gt_words + kWords;                                            // [kWords] ties
  uint32_t* samp = eq_words + kWords;                                                // [kSampleMax]
  uint32_t* warp_sum = samp + kSampleMax;                                            // [4][32]
  uint32_t* few = warp_sum + 4 * kBigWarps;                                          // [kFew]
  int* ctl = reinterpret_cast<int*>(few + kFew);                                     // [16]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  auto scores_of = [&](int row) { return reinterpret_cast<const uint32_t*>(p.scores) + static_cast<long long>(row) * p.sc_stride; };
  int row = blockIdx.x;
  if (!kLong && row < p.s_q) fetch(scores_of(row), row_len(p, row), kHalf, buf);
  for (; row < p.s_q; row += gridDim.x) {
    const int len = row_len(p, row);
    const int k = min(p.topk, len);
    const uint32_t* src = scores_of(row);
    int32_t* out = p.out + static_cast<long long>(row) * p.out_stride;
    const bool sampled = k < len && len >= kSampleMinLen;
    uint32_t key[kPerThread];                              // position 1024 i + tid; 0 past the row
    if (kLong) {
      if (len > kHalf) fetch(src + kHalf, len - kHalf, 0, buf);
      if (sampled && tid < kSample)
        samp[tid] = (to_key(src[static_cast<int>((static_cast<long long>(tid) * len) / kSample) + (tid & 15)]) & ~0xffu) | static_cast<uint32_t>(tid);
#pragma unroll
      for (int i = 0; i < kPerThread; ++i) {
        const int pos = i * kBigThreads + tid;
        key[i] = pos < len ? to_key(__ldcs(src + pos)) : 0u;
      }
      cp_async_wait_all();
    } else {
      cp_async_wait_all();
      __syncthreads();
#pragma unroll
      for (int i = 0; i < kPerThread; ++i) {
        const int pos = i * kBigThreads + tid;
        key[i] = to_key(buf[pos]);
      }
      // the sample number in the low bits makes the sample keys distinct; the bracket does not need exact keys
      if (sampled && tid < kSample)
        samp[tid] = (to_key(buf[static_cast<int>((static_cast<long long>(tid) * len) / kSample) + (tid & 15)]) & ~0xffu) | static_cast<uint32_t>(tid);
    }
    if (tid == 0) { ctl[kCtlLo] = 1; ctl[kCtlHi] = -1; ctl[kCtlFirst] = ctl[kCtlFirst + 1] = 1; ctl[kCtlFirst + 2] = ctl[kCtlFirst + 3] = -1; ctl[kCtlAbove] = 0; ctl[kCtlList] = 0; ctl[kCtlFew] = 0; }
    __syncthreads();
    if (!kLong && row + static_cast<int>(gridDim.x) < p.s_q)
      fetch(scores_of(row + gridDim.x), row_len(p, row + gridDim.x), kHalf, buf);           // overlaps the selection

    if (k < len) {
      // the keys of positions kHalf + 1024 i + tid, i < n2: read again from shared memory by every sweep
      const int n2 = kLong ? max(0, min(kPerThread, (len - kHalf - tid + kBigThreads - 1) / kBigThreads)) : 0;
      auto key2 = [&](int i) { return to_key(buf[i * kBigThreads + tid]); };
      bool use_list = false;
      uint32_t lo = 0u, hi = 0xffffffffu;                  // the threshold lies in [lo, hi]
      int c_lo = len, c_hi = 0, want = k;                  // keys >= lo, keys > hi, among those that are counted
      uint32_t cand[kListPer];
      if (sampled) {
        // rank of a key of the sample: kRankers threads count a part each
        const int s_no = tid / kRankers, part = tid % kRankers;
        const uint32_t mine = samp[s_no];
        int rank = 0;
#pragma unroll
        for (int m = 0; m < kSample / kRankers / 4; ++m) { // the threads of a sample read different banks
          const uint4 v = *reinterpret_cast<const uint4*>(samp + 4 * kRankers * m + 4 * part);
          rank += (v.x > mine) + (v.y > mine) + (v.z > mine) + (v.w > mine);
        }
#pragma unroll
        for (int d = 1; d < kRankers; d <<= 1) rank += __shfl_xor_sync(0xffffffffu, rank, d);
        const float frac = static_cast<float>(k) / static_cast<float>(len);
        const int centre = static_cast<int>(frac * kSample);
        const int margin = static_cast<int>(3.5f * sqrtf(kSample * frac * (1.0f - frac))) + 2, step = margin / 3;
        if (part == 0) {
          if (rank == centre + margin) ctl[kCtlLo] = static_cast<int>(max(mine & ~0xffu, 1u));   // stays 1 past the sample
          if (rank == centre - margin) ctl[kCtlHi] = static_cast<int>(mine | 0xffu);             // stays the largest key
          // the first trial values (past the sample: the ends)
          if (rank == centre + step) ctl[kCtlFirst] = static_cast<int>(max(mine, 1u));
          if (rank == centre) ctl[kCtlFirst + 1] = static_cast<int>(max(mine, 1u));
          if (rank == centre - step) ctl[kCtlFirst + 2] = static_cast<int>(mine);
          if (rank == centre - margin) ctl[kCtlFirst + 3] = static_cast<int>(mine | 0xffu);
        }
        __syncthreads();
        // no upper end where the list has room for all that lies above the lower one (three quarters of it, as expected)
        const bool open = (centre + margin) * (len / kSample) <= kListMax * 3 / 4;
        const uint32_t b_lo = static_cast<uint32_t>(ctl[kCtlLo]), b_hi = open ? 0xffffffffu : static_cast<uint32_t>(ctl[kCtlHi]);
        const uint32_t range = b_hi - b_lo;                // (a position past the row has key 0, below every bracket)
        int above = 0, inside = 0;
#pragma unroll
        for (int i = 0; i < kPerThread; ++i) inside += key[i] >= b_lo ? 1 : 0;
        if (kLong)
          for (int i = 0; i < n2; ++i) inside += key2(i) >= b_lo ? 1 : 0;
        if (!open) {
#pragma unroll
          for (int i = 0; i < kPerThread; ++i) above += key[i] > b_hi ? 1 : 0;
          if (kLong)
            for (int i = 0; i < n2; ++i) above += key2(i) > b_hi ? 1 : 0;
          inside -= above;
        }
        above = __reduce_add_sync(0xffffffffu, above);
        int at = inside;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, at, d);
          if (lane >= d) at += v;
        }
        int first = 0;
        if (lane == 31) {
          atomicAdd(&ctl[kCtlAbove], above);
          first = atomicAdd(&ctl[kCtlList], at);
        }
        at += __shfl_sync(0xffffffffu, first, 31) - inside;
        if (at + inside <= kListMax) {
#pragma unroll
          for (int i = 0; i < kPerThread; ++i)
            if (key[i] - b_lo <= range) list[at++] = key[i];
          if (kLong)
            for (int i = 0; i < n2; ++i) {
              const uint32_t x = key2(i);
              if (x - b_lo <= range) list[at++] = x;
            }
        }
        __syncthreads();
        const int n_above = ctl[kCtlAbove], n_list = ctl[kCtlList];
        if (n_above < k && k <= n_above + n_list) {
          lo = b_lo; hi = b_hi;
          c_lo = n_above + n_list; c_hi = n_above;
        }
        if (lo == b_lo && n_list <= kListMax) {
          use_list = true;
          c_lo = n_list; c_hi = 0; want = k - n_above;
#pragma unroll
          for (int j = 0; j < kListPer; ++j) cand[j] = j * kBigThreads + tid < n_list ? list[j * kBigThreads + tid] : 0u;
        }
      }
      // c_lo >= want > c_hi at all times
      if (use_list) {
        // four trial values at a time: first keys of the sample, then values a little either side of where the threshold lies if
        // the keys of the interval are spread evenly; every third time they cut the interval in five, whatever the counts say
        const int in_use = (c_lo + kBigThreads - 1) / kBigThreads;
#pragma unroll 1
        for (int trial = 0; c_lo != want && lo != hi && c_lo - c_hi > kFew; ++trial) {
          const float share = (static_cast<float>(c_lo - want) + 0.5f) / static_cast<float>(c_lo - c_hi), width = static_cast<float>(hi - lo);
          uint32_t mid[4], c01 = 0, c23 = 0;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float at = trial % 3 == 0 ? 0.2f * static_cast<float>(j + 1) : share + (j == 0 ? -0.12f : j == 1 ? -0.03f : j == 2 ? 0.03f : 0.12f);
            mid[j] = lo + 1u + min(static_cast<uint32_t>(fmaxf(at, 0.0f) * width), hi - lo - 1u);
            if (trial == 0) mid[j] = min(max(static_cast<uint32_t>(ctl[kCtlFirst + j]), lo + 1u), hi);
          }
#pragma unroll
          for (int j = 0; j < kListPer; ++j)
            if (j < in_use) {
              c01 += (cand[j] >= mid[0] ? 1u : 0u) + (cand[j] >= mid[1] ? 65536u : 0u);
              c23 += (cand[j] >= mid[2] ? 1u : 0u) + (cand[j] >= mid[3] ? 65536u : 0u);
            }
          c01 = __reduce_add_sync(0xffffffffu, c01);
          c23 = __reduce_add_sync(0xffffffffu, c23);
          uint32_t* sums = warp_sum + (trial & 1) * 2 * kBigWarps;
          if (lane == 0) { sums[warp] = c01; sums[kBigWarps + warp] = c23; }
          __syncthreads();
          c01 = __reduce_add_sync(0xffffffffu, sums[lane]);
          c23 = __reduce_add_sync(0xffffffffu, sums[kBigWarps + lane]);
          const int c[4] = {static_cast<int>(c01 & 0xffffu), static_cast<int>(c01 >> 16), static_cast<int>(c23 & 0xffffu), static_cast<int>(c23 >> 16)};
#pragma unroll
          for (int j = 0; j < 4; ++j) {                    // mid and so c in order
            if (c[j] >= want) { lo = mid[j]; c_lo = c[j]; }
          }
#pragma unroll
          for (int j = 3; j >= 0; --j) {
            if (c[j] < want) { hi = mid[j] - 1u; c_hi = c[j]; }
          }
        }
        if (c_lo != want && lo != hi) {                    // few left: the one of which want - c_hi are not smaller
#pragma unroll
          for (int j = 0; j < kListPer; ++j)
            if (cand[j] >= lo && cand[j] <= hi) few[atomicAdd(&ctl[kCtlFew], 1)] = cand[j];
          __syncthreads();
          const int n = c_lo - c_hi, r = want - c_hi;
          const int which = tid >> 3;                      // eight threads per candidate
          const uint32_t v = few[which < n ? which : 0];
          int above_v = 0, from_v = 0;
          for (int m = tid & 7; m < n; m += 8) {
            above_v += few[m] > v ? 1 : 0;
            from_v += few[m] >= v ? 1 : 0;
          }
#pragma unroll
          for (int d = 1; d < 8; d <<= 1) {
            above_v += __shfl_xor_sync(0xffffffffu, above_v, d);
            from_v += __shfl_xor_sync(0xffffffffu, from_v, d);
          }
          if (which < n && above_v < r && r <= from_v) { ctl[kCtlLimit] = static_cast<int>(v); ctl[kCtlNeedEq] = r - above_v; }
          __syncthreads();
          lo = hi = static_cast<uint32_t>(ctl[kCtlLimit]);
          c_hi = want - ctl[kCtlNeedEq];
        }
      } else {
#pragma unroll 1
        for (int trial = 0; c_lo != want && lo != hi; ++trial) {
          const uint32_t mid = lo + 1u + (hi - lo - 1u) / 2u;
          int n = 0;
#pragma unroll
          for (int i = 0; i < kPerThread; ++i) n += key[i] >= mid ? 1 : 0;
          if (kLong)
            for (int i = 0; i < n2; ++i) n += key2(i) >= mid ? 1 : 0;
          n = __reduce_add_sync(0xffffffffu, n);
          uint32_t* sums = warp_sum + (trial & 1) * kBigWarps;
          if (lane == 0) sums[warp] = static_cast<uint32_t>(n);
          __syncthreads();
          n = static_cast<int>(__reduce_add_sync(0xffffffffu, sums[lane]));
          if (n >= want) { lo = mid; c_lo = n; }
          else { hi = mid - 1u; c_hi = n; }
        }
      }
      // keys above `limit` are taken, and need_eq of those equal to it
      const int need_eq = c_lo == want ? 0 : want - c_hi;
      const uint32_t limit = c_lo == want ? lo - 1u : lo;
      // word i of 32 positions 1024 i + 32 warp ...: taken, ties
#pragma unroll
      for (int i = 0; i < kPerThread; ++i) {
        const uint32_t m = __ballot_sync(0xffffffffu, key[i] > limit);
        if (lane == 0) gt_words[i * kBigWarps + warp] = m;
      }
      if (kLong) {
#pragma unroll 4
        for (int i = 0; i < kPerThread; ++i) {
          const uint32_t m = __ballot_sync(0xffffffffu, i < n2 && key2(i) > limit);
          if (lane == 0) gt_words[kWords / 2 + i * kBigWarps + warp] = m;
        }
      }
      if (need_eq > 0) {
#pragma unroll
        for (int i = 0; i < kPerThread; ++i) {
          const uint32_t m = __ballot_sync(0xffffffffu, key[i] == limit && i * kBigThreads + tid < len);
          if (lane == 0) eq_words[i * kBigWarps + warp] = m;
        }
        if (kLong) {
#pragma unroll 4
          for (int i = 0; i < kPerThread; ++i) {
            const uint32_t m = __ballot_sync(0xffffffffu, i < n2 && key2(i) == limit);
            if (lane == 0) eq_words[kWords / 2 + i * kBigWarps + warp] = m;
          }
        }
      }
      __syncthreads();
      // one scan over the packed counts (ties << 16 | taken), then each thread writes the positions of its words
      constexpr int kPer = kLong ? 2 : 1;
      uint32_t g[kPer], e[kPer], packed = 0;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        g[j] = gt_words[kPer * tid + j];
        e[j] = need_eq > 0 ? eq_words[kPer * tid + j] : 0u;
        packed += (static_cast<uint32_t>(__popc(e[j])) << 16) + static_cast<uint32_t>(__popc(g[j]));
      }
      uint32_t incl = packed;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
      }
      if (lane == 31) warp_sum[warp] = incl;
      __syncthreads();
      uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? warp_sum[lane] : 0u) + incl - packed;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const int gt_before = static_cast<int>(before & 0xffffu), eq_before = static_cast<int>(before >> 16);
        int eq_take = min(max(need_eq - eq_before, 0), __popc(e[j]));                 // the lowest positions among the ties
        uint32_t bits = g[j], ties = e[j];
        while (eq_take > 0) {
          const uint32_t lowest = ties & (0u - ties);
          bits |= lowest;
          ties ^= lowest;
          --eq_take;
        }
        int write_at = gt_before + min(eq_before, need_eq);
        const int pos0 = (kPer * tid + j) * 32;
        while (bits != 0) {
          out[write_at++] = pos0 + __ffs(static_cast<int>(bits)) - 1;
          bits &= bits - 1u;
        }
        before += (static_cast<uint32_t>(__popc(e[j])) << 16) + static_cast<uint32_t>(__popc(g[j]));
      }
    } else {
      for (int j = tid; j < len; j += kBigThreads) out[j] = j;                        // every position of the row is taken
    }
    for (int j = k + tid; j < p.topk; j += kBigThreads) out[j] = -1;
    __syncthreads();                                       // the shared words are reused by the next row
  }
}

}  // namespace topk
}  // namespace ftb

extern "C" FTB_API int ftb_topk_indices(const ftb_topk_args* a, void* stream) {
  using namespace ftb;
  if (a == nullptr) { set_last_error("ftb_topk_indices: args is NULL"); return FTB_ERR_INVALID; }
  if (a->s_q < 0 || a->s_kv <= 0 || a->topk <= 0) {
    set_last_error("ftb_topk_indices: bad sizes s_q=%d s_kv=%d topk=%d", a->s_q, a->s_kv, a->topk);
    return FTB_ERR_INVALID;
  }
  if (a->s_q == 0) return FTB_OK;
  if (!a->scores || !a->out) { set_last_error("ftb_topk_indices: null pointer"); return FTB_ERR_INVALID; }
  topk::Params p;
  p.scores = a->scores; p.lengths = a->lengths; p.out = a->out;
  p.s_q = a->s_q; p.s_kv = a->s_kv; p.topk = a->topk;
  p.sc_stride = a->scores_stride_token; p.out_stride = a->out_stride_token;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // Any alignment and any stride.  Rows of more than 65 536 scores do not fit one SM: the first kernel reads them from
  // memory five times.
  if (a->s_kv <= topk::kRowMax) {
    int dev = 0, sm_count = 0;
    if (int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice")) return rc;
    if (int rc = check_cuda(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev), "SM count")) return rc;
    const auto kernel = a->s_kv <= topk::kHalf ? topk::topk_select_rows_kernel<false> : topk::topk_select_rows_kernel<true>;
    if (int rc = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(topk::kBigSmem)), "topk shared memory")) return rc;
    const unsigned grid = static_cast<unsigned>(a->s_q < sm_count ? a->s_q : sm_count);
    kernel<<<grid, topk::kBigThreads, topk::kBigSmem, st>>>(p);
  } else {
    topk::topk_select_kernel<<<static_cast<unsigned>(a->s_q), topk::kThreads, 0, st>>>(p);
  }
  return check_cuda(cudaGetLastError(), "ftb_topk_indices launch");
}
