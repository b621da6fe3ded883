// Top-k index producer: the step in front of the sparse MLA forward.  For every query token the positions of the
// `topk` largest scores among its first `length` key positions, written in ascending position order and padded
// with -1: exactly the index list the forward takes.
//
// Selection is exact and deterministic: scores are mapped to 32-bit keys whose unsigned order is the order of the
// floats (-0 below +0, NaN patterns above +inf, as an unsigned compare of the transformed bits gives), the k-th
// largest key is found, and among the entries equal to that key the lowest positions are taken.  Two kernels, by the length
// of a row: up to 65536 scores a CTA makes a short list of the keys that may be among the k largest and selects in that; longer rows,
// and lists that no SM has room for, go to a radix select that reads the row five times from wherever it is.  The floor is device-memory
// traffic: 4 * s_kv bytes of scores per token (plus 4 * topk bytes of output).
#include <cmath>

#include "launch.cuh"
#include "sm100.cuh"

namespace ftb {

void set_last_error(const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

namespace topk {

constexpr int kThreads = 512;                              // of the radix select

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

__device__ __forceinline__ float to_float(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key);
}

__device__ __forceinline__ int row_len(const Params& p, int row) {
  const int len = p.lengths != nullptr ? p.lengths[row] : p.s_kv;
  return max(0, min(len, p.s_kv));
}

// exclusive prefix of `flag` over the block in thread order; `total` = number of set flags (same in every thread)
template <int kThr>
__device__ __forceinline__ int block_exclusive(bool flag, int* warp_sums, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned b = __ballot_sync(0xffffffffu, flag);
  const int in_warp = __popc(b & ((1u << lane) - 1u));
  if (lane == 0) warp_sums[warp] = __popc(b);
  __syncthreads();
  int before = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < kThr / 32; ++w) {
    const int v = warp_sums[w];
    before += (w < warp) ? v : 0;
    tot += v;
  }
  __syncthreads();       // warp_sums is reused by the next call
  total = tot;
  return before + in_warp;
}

// The k-th largest of the keys that `each` hands over, by four passes of 8 bits with a 256-bin histogram in shared memory (`hist`), and how
// many of the keys equal to it belong to the k largest.  Called by all threads of a block.
struct Threshold {
  uint32_t key;
  int need_eq;
};
template <class Each>
__device__ __forceinline__ Threshold radix_select(Each each, int k, int* hist, uint32_t* s_bin, int* s_remaining) {
  const int tid = threadIdx.x, lane = tid & 31;
  uint32_t prefix = 0, mask = 0;
  int remaining = k;
#pragma unroll 1
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    if (tid < 256) hist[tid] = 0;
    __syncthreads();
    each([&](uint32_t key) {
      if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1);
    });
    __syncthreads();
    if (tid < 32) {
      // lane l owns bins 8l .. 8l + 7; walk from the largest bin down to the one that holds the `remaining`-th largest
      int mine = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) mine += hist[8 * lane + j];
      int above = 0;                                     // entries in the bins of higher lanes
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
            *s_bin = static_cast<uint32_t>(8 * lane + j);
            *s_remaining = remaining - cum;
            break;
          }
          cum += h;
        }
      }
    }
    __syncthreads();
    prefix |= *s_bin << shift;
    mask |= 255u << shift;
    remaining = *s_remaining;
    __syncthreads();
  }
  return Threshold{prefix, remaining};
}

// A row read from memory in every pass, once more by the one that writes, by a block of kThr threads.
template <int kThr>
struct RowSmem {
  int hist[256];
  int warp_sums[kThr / 32];
  uint32_t bin;
  int remaining;
};
template <int kThr>
__device__ __forceinline__ void select_row(const uint32_t* sc, int len, int topk, int32_t* out, RowSmem<kThr>* sm) {
  const int tid = threadIdx.x;
  const int k = min(topk, len);
  uint32_t thresh = 0;       // key of the k-th largest entry
  int need_eq = 0;           // how many entries equal to it are taken (the lowest positions)
  if (k < len) {
    const Threshold t = radix_select([&](auto take) { for (int i = tid; i < len; i += kThr) take(to_key(sc[i])); },
                                     k, sm->hist, &sm->bin, &sm->remaining);
    thresh = t.key;
    need_eq = t.need_eq;
  }
  // ordered compaction: positions in ascending order, entries above the threshold and the first need_eq equal to it
  int written = 0, eq_seen = 0;
  for (int start = 0; start < len; start += kThr) {
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
      const int eq_rank = eq_seen + block_exclusive<kThr>(eq, sm->warp_sums, eq_total);
      if (eq && eq_rank < need_eq) take = true;
      eq_seen += eq_total;
    }
    int take_total;
    const int pos = written + block_exclusive<kThr>(take, sm->warp_sums, take_total);
    if (take) out[pos] = i;
    written += take_total;
  }
  for (int j = k + tid; j < topk; j += kThr) out[j] = -1;
}

// One CTA per row, four to an SM.
__global__ void __launch_bounds__(kThreads) topk_select_kernel(const Params p) {
  __shared__ RowSmem<kThreads> sm;
  griddep_launch();
  griddep_wait();
  const int row = blockIdx.x;
  const int len = row_len(p, row);
  select_row<kThreads>(reinterpret_cast<const uint32_t*>(p.scores) + static_cast<long long>(row) * p.sc_stride, len, p.topk,   // bits: NaN patterns keep theirs
                       p.out + static_cast<long long>(row) * p.out_stride, &sm);
}

// ---------------------------------------------------------------------------------------------------------------
// Rows up to 65536 scores: one CTA per row, as many CTAs to an SM as fit.
//
// A sample of 512 keys gives a lower bound of the k-th largest key, a few standard deviations of the sample quantile on the safe
// side.  One sweep over the row votes the keys from there on into a mask over the row (four instructions for 32 keys: load,
// compare, vote, store).  The few positions in the mask, an eighth of the row or so, become a list in ascending order, and
// their keys are fetched again, out of L2.  The list is counted against four trial values at a time, quantiles of the sample
// first, then values interpolated between the counts known so far, until 128 candidates are left, which are ranked by
// counting.  A lane works out one of the four values and what its count means: with all four in every thread a trial took a lone row 1900
// cycles for four keys a thread.  Interpolated are the floats, not the keys, whose density doubles with every power of two
// towards zero (100 rows of 32 768, topk 16 384, the median: 46 -> 24 us).
// The list is in order, so the taken ones among it are the output as they come.
// Where a value fills so much of the row that keys equal to the bound would crowd the list, the list takes the keys above it and
// the ties go to a mask of their own in the same sweep.  A bound that turns out too high, or more keys than the list has room
// for (both checked), costs time and never exactness: the row is then selected by the radix select, out of L2.
// A row that fits the list goes there without a sweep.
//
// What bounds it: instruction issue (0.69 a clock and scheduler, a row of 32768 some 40 000) and chains of latencies (sample, bound, sweep, list,
// keys, trials), which the other CTAs of the SM fill; memory is at a quarter of its rate.  Copying the keys to the list in the sweep itself,
// instead of voting, took 130 instructions per 128 keys (4096 x 32 768, topk 2048: 293 us; with votes 234, with the tail of the row apart 210).
// Against persistent CTAs that hold a row in registers and histogram it (us, before / now): 4096 x 32 768 causal 334 / 205, 4096 x 20 001
// topk 1024 426 / 120, 4096 x 6000 277 / 98, 4096 x 4000 topk 512 189 / 65, 4096 x 1000 topk 512 83 / 51, 592 rows of 33 000 82 / 36,
// 592 rows of 32 768 equal scores 52 / 40, 128 rows of up to 65 536 30 / 17, 300 short rows of a matrix of 65 536 columns 44 / 16, one row of
// 32 768 13.1 / 11.5, of 4000 11.2 / 7.8; level or up to 10 % slower: rows of 32 768 with topk 4096 and more (148: 14.9 / 15.5, 4096
// with 16 384: 588 / 648), 30 % short rows of some ten values (1024 rows of 1000, topk 333: 27 / 35).
// ---------------------------------------------------------------------------------------------------------------
namespace listed {

constexpr int kRowMax = 65536;                             // positions in the list are 16-bit words
constexpr int kSample = 512;
constexpr float kMargin = 4.5f;                            // standard deviations between the k-th largest key and the bound
constexpr int kCrowd = 6;                                  // that many keys of the sample more than wanted: many keys equal the bound
constexpr int kFew = 128;                                  // this many candidates are ranked by counting
constexpr int kAhead = 16;                                 // loads in flight per lane
constexpr int kSmemMax = 220 * 1024;                       // dynamic; a few KB of static beside it

constexpr int kSmemAlone = 116 * 1024;                     // of a row that has an SM to itself: no second CTA beside it, whenever it comes (launch.cuh)
struct Shape {
  int room;                                                // list entries
  int words;                                               // of a mask over the row
};
// The list has room for what the bound is expected to let through and four standard deviations more (never less for a longer row); 0 where
// that is more than an SM has.  A row is taken whole, without a sweep, where it is short or most of it would pass the bound (us,
// whole / swept: 4096 rows of 4000, topk 512 89 / 65, topk 2048 88 / 90; of 2000, topk 512 68 / 62, topk 1024 70 / 72; one row of 2000, topk 512 6.0 / 6.7,
// of 3000 7.3 / 7.0; 148 rows with an SM each, of 8192 topk 4096 9.9 / 11.8, of 12 000 topk 4096 12.9 / 12.6, of 20 000 topk 2048 17.4 / 12.2).
inline int plan(int s_kv, int topk, bool alone, Shape* shape) {
  if (s_kv > kRowMax) return 0;
  const double k = topk < s_kv ? topk : s_kv, n = s_kv < kSample ? s_kv : kSample, frac = k / s_kv;
  const double r = n * frac + kMargin * std::sqrt(n * frac * (1.0 - frac)) + 3.0 + kCrowd;   // rank of the bound in the sample
  const int wanted = static_cast<int>((r + 4.0 * std::sqrt(r)) / n * s_kv) + 64;
  shape->words = (s_kv + 31) / 32;
  const int most = (kSmemMax - 8 * shape->words) / 6;
  const bool whole = s_kv <= (alone ? 2048 : 1024) || (wanted > 0.6 * s_kv && s_kv <= (alone ? most : 4096));
  shape->room = whole || wanted > s_kv ? s_kv : wanted;
  if (shape->room > most) {
    if (most < 1.1 * r / n * s_kv) return 0;
    shape->room = most;
  }
  shape->room = (shape->room + 3) & ~3;
  return 8 * shape->words + 6 * shape->room;
}

// how many of the keys x (of all lanes) are t or more
__device__ __forceinline__ int count_from(const uint32_t (&x)[kSample / 32], uint32_t t) {
  int n[4] = {0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < kSample / 32; ++i) n[i & 3] += x[i] >= t ? 1 : 0;
  return static_cast<int>(__reduce_add_sync(0xffffffffu, (n[0] + n[1]) + (n[2] + n[3])));
}
// `v` with the bits from .. to set as far as at least r of the keys x still reach it: the r-th largest of them, cut off below bit `to`
__device__ __forceinline__ uint32_t rank_value(const uint32_t (&x)[kSample / 32], int r, uint32_t v, int from, int to) {
#pragma unroll 1
  for (int b = from; b >= to; --b) {
    const uint32_t t = v | (1u << b);
    if (count_from(x, t) >= r) v = t;
  }
  return v;
}

template <int kThr>
struct Shared {
  union {
    RowSmem<kThr> radix;
    struct {
      uint32_t samp[kSample];
      alignas(16) uint32_t few[kFew];
    };
  };
  uint32_t bound;                                          // the list takes the keys from here on (ties: above)
  uint32_t first[4];                                       // first trial values
  int ties;
  uint32_t sums[4][32];
  int n_few, need_eq;
  uint32_t limit;
};

// not inline: the rare path needs registers of its own
template <int kThr>
__device__ __noinline__ void select_from_memory(const uint32_t* sc, int len, int topk, int32_t* out, RowSmem<kThr>* sm) {
  select_row<kThr>(sc, len, topk, out, sm);
}

// exclusive prefix over the block of a packed count, and its total; `sums` (32 words) must not be in use
template <int kThr>
__device__ __forceinline__ uint32_t block_prefix(uint32_t v, uint32_t* sums, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  const uint32_t w = lane < kThr / 32 ? sums[lane] : 0u;
  total = __reduce_add_sync(0xffffffffu, w);
  return __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u) + incl - v;
}

template <int kThr, int kBlocks>
__global__ void __launch_bounds__(kThr, kBlocks) topk_listed_kernel(const Params p, const Shape shape) {
  constexpr int kWarps = kThr / 32;
  __shared__ Shared<kThr> sm;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* gt_words = reinterpret_cast<uint32_t*>(smem_raw);                       // keys in the list
  uint32_t* eq_words = gt_words + shape.words;                                      // keys that equal the bound
  uint32_t* keys = eq_words + shape.words;                                          // the list: keys,
  unsigned short* at_pos = reinterpret_cast<unsigned short*>(keys + shape.room);    // and positions, ascending
  griddep_launch();
  griddep_wait();
  const int row = blockIdx.x;
  const int len = row_len(p, row);
  const int k = min(p.topk, len);
  const uint32_t* src = reinterpret_cast<const uint32_t*>(p.scores) + static_cast<long long>(row) * p.sc_stride;   // bits: NaN patterns keep theirs
  int32_t* out = p.out + static_cast<long long>(row) * p.out_stride;
  for (int j = k + tid; j < p.topk; j += kThr) out[j] = -1;
  if (k == len) {
    for (int j = tid; j < len; j += kThr) out[j] = j;
    return;
  }
  const bool whole = len <= shape.room;
  const int words = (len + 31) >> 5;
  int n_list = len;
  if (whole) {
#pragma unroll 8
    for (int i = tid; i < len; i += kThr) {
      keys[i] = to_key(src[i]);
      at_pos[i] = static_cast<unsigned short>(i);
    }
    __syncthreads();
  }
  // ---- the sample: one key from each of 512 stretches, not at the same place of each; a row that is shorter is its own sample
  for (int t = tid; t < kSample; t += kThr) {
    const uint32_t stride = static_cast<uint32_t>(len) / kSample;
    const uint32_t at = len >= kSample ? static_cast<uint32_t>((static_cast<unsigned long long>(t) * len) / kSample) + ((((t * 0x9e3779b1u) >> 16) * stride) >> 16)
                                       : static_cast<uint32_t>(t);
    sm.samp[t] = at >= static_cast<uint32_t>(len) ? 0u : whole ? keys[at] : to_key(src[at]);
  }
  if (tid < kFew) sm.few[tid] = 0u;
  if (tid == 0) sm.n_few = 0;
  __syncthreads();
  if (warp < 4) {
    uint32_t x[kSample / 32];
#pragma unroll
    for (int i = 0; i < kSample / 32; ++i) x[i] = sm.samp[32 * i + lane];
    const float n = static_cast<float>(min(len, kSample)), frac = __fdividef(static_cast<float>(k), static_cast<float>(len));
    const float var = n * frac * (1.0f - frac);
    const int centre = static_cast<int>(frac * n);
    const int margin = static_cast<int>(kMargin * var * rsqrtf(var)) + 3, step = margin / 4;         // (0 < k < len: the variance is above zero)
    const int r = warp == 0 ? centre + margin : warp == 1 ? centre + step : warp == 2 ? centre - step : centre - margin;
    // the high bits (sign, exponent and five more) will do, unless many keys of the sample share them
    uint32_t v = rank_value(x, max(r, 1), 0u, 31, 18);
    if (warp == 0) {
      int from = count_from(x, v);
      if (from >= r + kCrowd) {
        v = rank_value(x, r, v, 17, 0);
        from = count_from(x, v);
      }
      if (lane == 0) {
        sm.bound = v;
        sm.ties = v != 0u && from >= r + kCrowd ? 1 : 0;
      }
    }
    if (lane == 0) sm.first[warp] = v;
  }
  __syncthreads();
  const uint32_t bound = sm.bound;
  const bool ties = sm.ties != 0;
  int n_ties = 0;
  if (!whole) {
    // ---- the sweep: warp w takes stretches of 32 kAhead positions, w, w + kWarps, ...; word i of the mask is positions 32 i ..
    const bool plain = !ties && bound > 0x80000000u;       // the usual case, a bound above zero: floats from there on compare by their bits
    const int lo_bits = static_cast<int>(bound ^ 0x80000000u);
#pragma unroll 1
    for (int w0 = warp * kAhead; w0 < words; w0 += kWarps * kAhead) {
      uint32_t v[kAhead];
      const uint32_t* at = src + w0 * 32 + lane;
      const bool inside = (w0 + kAhead) * 32 <= len;
      if (inside) {
#pragma unroll
        for (int j = 0; j < kAhead; ++j) v[j] = at[32 * j];
      } else {
#pragma unroll
        for (int j = 0; j < kAhead; ++j) v[j] = (w0 + j) * 32 + lane < len ? at[32 * j] : 0xffffffffu;   // the lowest key
      }
      if (plain && inside) {
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
          const uint32_t m = __ballot_sync(0xffffffffu, static_cast<int>(v[j]) >= lo_bits);
          if (lane == 0) gt_words[w0 + j] = m;
        }
      } else {
        const int last = len - w0 * 32 - lane;             // the lane's keys from here on are past the row
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
          const uint32_t key = to_key(v[j]);
          uint32_t m = __ballot_sync(0xffffffffu, key >= bound && 32 * j < last);
          if (ties) {
            const uint32_t eq = __ballot_sync(0xffffffffu, key == bound) & m;
            m ^= eq;
            if (lane == 0 && w0 + j < words) eq_words[w0 + j] = eq;
          }
          if (lane == 0 && w0 + j < words) gt_words[w0 + j] = m;
        }
      }
    }
    __syncthreads();
    // ---- the list: every thread the positions of a few words
    const int per = (words + kThr - 1) / kThr, w_end = min(words, per * (tid + 1));
    uint32_t packed = 0, total;
    for (int w = per * tid; w < w_end; ++w) {
      packed += static_cast<uint32_t>(__popc(gt_words[w]));
      if (ties) n_ties += __popc(eq_words[w]);
    }
    int at = static_cast<int>(block_prefix<kThr>(packed, sm.sums[0], total));
    n_list = static_cast<int>(total);
    if (ties) {
      uint32_t all;
      block_prefix<kThr>(static_cast<uint32_t>(n_ties), sm.sums[1], all);
      n_ties = static_cast<int>(all);
    }
    if (n_list > shape.room || n_list + n_ties < k) {      // the sample misled
      __syncthreads();
      select_from_memory<kThr>(src, len, p.topk, out, &sm.radix);
      return;
    }
    if (n_list < k) {
      // the k-th largest key is the bound itself: the keys above it and the first of the ties
      const int need_eq = k - n_list;
      uint32_t mine = 0, all;
      for (int w = per * tid; w < w_end; ++w) mine += static_cast<uint32_t>(__popc(eq_words[w]));
      int eq_before = static_cast<int>(block_prefix<kThr>(mine, sm.sums[2], all));
      int write_at = at + min(eq_before, need_eq);
      for (int w = per * tid; w < w_end; ++w) {
        uint32_t bits = gt_words[w], eq = eq_words[w];
        int take = min(max(need_eq - eq_before, 0), __popc(eq));                     // the lowest positions among the ties
        eq_before += __popc(eq);
        while (take > 0) {
          const uint32_t lowest = eq & (0u - eq);
          bits |= lowest;
          eq ^= lowest;
          --take;
        }
        while (bits != 0) {
          out[write_at++] = 32 * w + __ffs(static_cast<int>(bits)) - 1;
          bits &= bits - 1u;
        }
      }
      return;
    }
    for (int w = per * tid; w < w_end; ++w) {
      uint32_t bits = gt_words[w];
      while (bits != 0) {
        at_pos[at++] = static_cast<unsigned short>(32 * w + __ffs(static_cast<int>(bits)) - 1);
        bits &= bits - 1u;
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int i = tid; i < n_list; i += kThr) keys[i] = to_key(src[at_pos[i]]);
    __syncthreads();
  }
  // A short row of few values, the k-th largest key not settled yet: the trials would cut the interval until it holds nothing but that key, some fifteen times.  (us,
  // trials / radix select: 1024 rows of 1000, topk 333, of two values 44 / 28, of about ten 44 / 35, one value 53 / 27; 2048, topk 682, of about ten 46 / 32; 4000, topk
  // 1333, 56 / 47.  Trials that ask whether all that is left is one key are faster still, 16 to 33, but cost other rows 1.4 to 5 % in every form tried.)
  if (ties && len <= 4096) {
    __syncthreads();
    select_from_memory<kThr>(src, len, p.topk, out, &sm.radix);
    return;
  }
  // ---- the k-th largest key of the list: keys above `limit` are taken, and need_eq of those equal to it (0: none or all, see below)
  uint32_t limit, lo = whole ? 0u : ties ? bound + 1u : bound, hi = 0xffffffffu;
  int need_eq = 0;
  int c_lo = n_list, c_hi = 0;                             // keys >= lo, keys > hi; c_lo >= k > c_hi at all times
  // every third time the values cut the interval in five, whatever the counts say
  int trial = 0;
  const int tj = lane & 3;                                 // a lane works out one of the four values, and what its count means
#pragma unroll 1
  for (; c_lo != k && lo != hi && c_lo - c_hi > kFew; ++trial) {
    uint32_t own;
    if (trial == 0) {
      own = tj == 0 ? min(sm.first[0], sm.first[1]) : sm.first[tj];                  // (the first may have more bits)
    } else {
      const float share = __fdividef(static_cast<float>(c_lo - k) + 0.5f, static_cast<float>(c_lo - c_hi));
      const float f_lo = to_float(lo), f_width = to_float(hi) - f_lo;                // not finite where an end is an infinity or a NaN
      const bool even = trial % 3 == 0;
      const float cut = fmaxf(even ? 0.2f * static_cast<float>(tj + 1) : share + (tj == 0 ? -0.12f : tj == 1 ? -0.03f : tj == 2 ? 0.03f : 0.12f), 0.0f);
      own = !even && f_width < 3.0e38f ? to_key(__float_as_uint(f_lo + cut * f_width))
                                       : lo + 1u + min(static_cast<uint32_t>(cut * static_cast<float>(hi - lo)), hi - lo - 1u);
    }
    own = min(max(own, lo + 1u), hi);                      // ascending in tj
    uint32_t mid[4], c01 = 0, c23 = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) mid[j] = __shfl_sync(0xffffffffu, own, j);
#pragma unroll 4
    for (int i = tid; i < n_list; i += kThr) {
      const uint32_t x = keys[i];
      c01 += (x >= mid[0] ? 1u : 0u) + (x >= mid[1] ? 65536u : 0u);
      c23 += (x >= mid[2] ? 1u : 0u) + (x >= mid[3] ? 65536u : 0u);
    }
    c01 = __reduce_add_sync(0xffffffffu, c01);
    c23 = __reduce_add_sync(0xffffffffu, c23);
    uint32_t(*sums)[32] = &sm.sums[(trial & 1) * 2];
    if (lane == 0) { sums[0][warp] = c01; sums[1][warp] = c23; }
    __syncthreads();
    c01 = __reduce_add_sync(0xffffffffu, lane < kWarps ? sums[0][lane] : 0u);
    c23 = __reduce_add_sync(0xffffffffu, lane < kWarps ? sums[1][lane] : 0u);
    const uint32_t c_two = tj < 2 ? c01 : c23;
    const int c = static_cast<int>((tj & 1) ? c_two >> 16 : c_two & 0xffffu);
    const int reach = __popc(__ballot_sync(0xffffffffu, c >= k) & 15u);              // values that k keys or more reach: the first ones
    const int below = __shfl_sync(0xffffffffu, c, max(reach - 1, 0)), past = __shfl_sync(0xffffffffu, c, min(reach, 3));
    const uint32_t at_below = __shfl_sync(0xffffffffu, own, max(reach - 1, 0)), at_past = __shfl_sync(0xffffffffu, own, min(reach, 3));
    if (reach > 0) { lo = at_below; c_lo = below; }
    if (reach < 4) { hi = at_past - 1u; c_hi = past; }
  }
  if (c_lo != k && lo != hi) {                             // few left: the one of which k - c_hi are not smaller
    for (int i0 = warp * 32; i0 < n_list; i0 += kThr) {
      const int i = i0 + lane;
      const uint32_t x = i < n_list ? keys[i] : 0u;
      const bool in = i < n_list && x >= lo && x <= hi;
      const uint32_t m = __ballot_sync(0xffffffffu, in);
      if (m != 0u) {
        int at = 0;
        if (lane == 0) at = atomicAdd(&sm.n_few, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (in) sm.few[at] = x;
      }
    }
    __syncthreads();
    const int total = c_lo - c_hi, r = k - c_hi;
    constexpr int kRankers = kThr / kFew;                  // threads per candidate
    const int which = tid / kRankers;
    const uint32_t v = sm.few[which];
    int above = 0, from = 0;
    for (int m = warp * (32 / kRankers) < total ? (tid % kRankers) * 4 : total; m < total; m += kRankers * 4) {   // (past the last candidate: 0, below every key of the list)
      const uint4 o = *reinterpret_cast<const uint4*>(&sm.few[m]);
      above += (o.x > v) + (o.y > v) + (o.z > v) + (o.w > v);
      from += (o.x >= v) + (o.y >= v) + (o.z >= v) + (o.w >= v);
    }
#pragma unroll
    for (int d = 1; d < kRankers; d <<= 1) {
      above += __shfl_xor_sync(0xffffffffu, above, d);
      from += __shfl_xor_sync(0xffffffffu, from, d);
    }
    if (which < total && above < r && r <= from) { sm.limit = v; sm.need_eq = r == from ? 0 : r - above; }
    __syncthreads();
    need_eq = sm.need_eq;
    limit = need_eq == 0 ? sm.limit - 1u : sm.limit;       // all that equal the limit are taken: those above the key before it
  } else {
    need_eq = c_lo == k ? 0 : k - c_hi;
    limit = need_eq == 0 ? lo - 1u : lo;
  }
  // ---- the output: every warp a stretch of the list, first counted, then written
  const int stretch = ((n_list + 32 * kWarps - 1) / (32 * kWarps)) * 32, i_begin = warp * stretch, i_end = min(n_list, i_begin + stretch);
  int taken = 0, equal = 0;
#pragma unroll 4
  for (int i = i_begin + lane; i < i_end; i += 32) {
    const uint32_t x = keys[i];
    taken += x > limit ? 1 : 0;
    if (need_eq != 0) equal += x == limit ? 1 : 0;
  }
  taken = static_cast<int>(__reduce_add_sync(0xffffffffu, taken));
  equal = static_cast<int>(__reduce_add_sync(0xffffffffu, equal));
  uint32_t(*sums)[32] = &sm.sums[(trial & 1) * 2];         // not those of the last trial, which another warp may still read
  if (lane == 0) { sums[0][warp] = static_cast<uint32_t>(taken); sums[1][warp] = static_cast<uint32_t>(equal); }
  __syncthreads();
  int write_at = static_cast<int>(__reduce_add_sync(0xffffffffu, lane < warp ? sums[0][lane] : 0u));
  int eq_left = need_eq - static_cast<int>(__reduce_add_sync(0xffffffffu, lane < warp ? sums[1][lane] : 0u));
  write_at += need_eq - max(eq_left, 0);                   // the ties of the warps before
  const uint32_t lower = (1u << lane) - 1u;
  for (int i0 = i_begin; i0 < i_end; i0 += 32) {
    const int i = i0 + lane;
    const uint32_t x = i < i_end ? keys[i] : 0u;
    bool take = i < i_end && x > limit;
    if (need_eq != 0) {
      const bool tie = i < i_end && x == limit;
      const uint32_t m = __ballot_sync(0xffffffffu, tie);
      take = take || (tie && __popc(m & lower) < eq_left);
      eq_left -= __popc(m);
    }
    const uint32_t m = __ballot_sync(0xffffffffu, take);
    if (take) out[write_at + __popc(m & lower)] = at_pos[i];
    write_at += __popc(m);
  }
}

}  // namespace listed

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
  int dev = 0, sm_count = 0;
  if (int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice")) return rc;
  if (int rc = check_cuda(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev), "SM count")) return rc;
  // A row to an SM: as many threads as its sweep keeps busy (us, 512 threads / 1024: 148 rows of 4000 14.4 / 17.1, 128 of up to 65536 20.7 / 19.3,
  // one of 32768 14.4 / 13.6).  More rows: six small CTAs to an SM hide their chains better, three larger ones keep fewer lists and rows
  // in flight (256 threads / 512: 4096 rows of 1000 56 / 79, of 6000 103 / 134, of 20001 151 / 159, of 32768 236 / 210; 592 of 33000 35 / 41;
  // 600 of 32768 with topk 8192 101 / 76).
  // Lists so long that an SM holds one count as rows alone (600 rows of 32 768 with topk 16 384: 512 threads 136, 1024 96).
  bool alone = a->s_q <= sm_count;
  topk::listed::Shape shape;
  int smem = topk::listed::plan(a->s_kv, a->topk, alone, &shape);
  if (!alone && smem > topk::listed::kSmemMax / 2) {
    alone = true;
    smem = topk::listed::plan(a->s_kv, a->topk, alone, &shape);
  }
  if (smem > 0) {
    const bool small = alone ? a->s_kv <= 8192 : a->topk <= 4096 && (a->s_kv <= 24576 || (a->s_q <= 6 * sm_count && a->topk <= 2048));
    const auto kernel = alone ? (small ? topk::listed::topk_listed_kernel<512, 1> : topk::listed::topk_listed_kernel<1024, 1>)
                              : (small ? topk::listed::topk_listed_kernel<256, 6> : topk::listed::topk_listed_kernel<512, 3>);
    if (alone && smem < topk::listed::kSmemAlone) smem = topk::listed::kSmemAlone;
    const unsigned threads = alone ? (small ? 512 : 1024) : (small ? 256 : 512);
    if (int rc = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, topk::listed::kSmemMax), "topk shared memory")) return rc;
    return check_cuda(launch_overlapped(kernel, static_cast<unsigned>(a->s_q), threads, smem, st, 1, p, shape), "ftb_topk_indices launch");
  }
  return check_cuda(launch_overlapped(topk::topk_select_kernel, static_cast<unsigned>(a->s_q), topk::kThreads, 0, st, 1, p), "ftb_topk_indices launch");
}
