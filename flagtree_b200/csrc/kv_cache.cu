// Write path of the paged FP8 latent cache: new latent rows (bf16, 576 values) are quantised to e4m3 with
// one fp32 scale per page and scattered into their slots.  This is the producer of the format that the paged
// sparse-MLA forward reads (value = e4m3 * kv_scale[page]).
//
// Rule for the page scale.  kv_scale[page] == 0 marks a page that holds nothing yet.  A call raises the scale
// of every page it touches to  max(old scale, max|new rows of the page| / 448)  (never below 1e-12 / 448), and
// when that raises the scale of a page that already held rows (old scale > 0), the 64 x 576 bytes of the page
// are requantised in place,  e4m3(decode(byte) * old / new),  before the new rows are written with the new
// scale.  Filling a page in one call therefore gives exactly amax / 448 over the page and one rounding per
// value; filling it in several calls gives the same scale and at most one extra rounding per raise.
//
// Small calls (decode, at most kSmallRows rows): one kernel.  A CTA per new row; the CTA of the first row of a page
// settles that page and stores all its rows (it finds them by scanning the slot list, a few KB), the others leave.
//
// Large calls (prefill).  New rows of a page usually come in one run of consecutive rows, so a run is the unit of work:
//   1. run_count_kernel counts the runs of every page (a caller workspace of 4 bytes per page, cleared first);
//   2. run_write_kernel: one warp (runs of up to 8 rows) or one CTA per run.  It takes the maximum over the run's rows;
//      if the run is the page's only one it settles the scale, requantises the page if need be, and stores the rows
//      from shared memory (runs of up to 64 rows; a longer one is read a second time, from L2).  A run
//      of a page with several leaves its maximum in the page's word (float bits, larger than any count);
//   3. page_settle_kernel and row_store_kernel finish the pages with several runs; for the others they only look.
// Device-memory traffic is 1152 B read + 576 B written per row; what bounds the write kernel now is instruction issue (two
// corrections per quotient) with memory close behind.  262 144 rows: 193 us with the rows read twice from memory and divided by
// the library's division, 141 us with the pieces dealt out over the lanes by index arithmetic (92 M warp instructions, two
// thirds of them addresses), 118 us with a row per eight lanes.
// The quotient x / scale is the correctly rounded one, as in the CPU restatement, so bytes and scales agree bit for bit.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"
#include "../../include/flagtree_b200.h"

namespace ftb {

void set_last_error(const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

namespace kvw {

constexpr int kD = 576;
constexpr float kE4m3Max = 448.0f;

struct Params {
  const __nv_bfloat16* rows;
  const int32_t* slots;
  uint8_t* cache;
  float* scale;
  unsigned int* cand;       // workspace: candidate scale per page as float bits (non-negative floats order as integers)
  int n_rows, num_pages, page_size;
  long long row_stride;     // elements between new rows
  int* status;
};

__device__ __forceinline__ float decode_e4m3(uint8_t b) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(b), __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
// A page scale with its reciprocal.  Division by multiplication with residual correction (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990): with y the correctly rounded reciprocal of b and q
// within an ulp of a / b, RN(q + RN(a - b q) y) is the correctly rounded a / b.  q = RN(a y) is within two ulps and one
// correction brings it within one, so two corrections give exactly what a division gives, in packed instructions.  It
// holds while nothing underflows or overflows: scales between 2^-100 and 2^100 qualify (a quotient whose residual
// underflows then is far below the smallest e4m3 value and becomes zero either way); others are divided by.
struct Divisor {
  float s, y;
  bool plain;          // divide
};
__device__ __forceinline__ Divisor make_divisor(float s) {
  Divisor d;
  d.s = s;
  d.plain = !(s > 7.9e-31f && s < 1.2e30f);
  d.y = d.plain ? 0.0f : __frcp_rn(s);
  return d;
}
__device__ __forceinline__ uint32_t quant2(float a, float b, const Divisor& d) {
  float2 q;
  if (d.plain) {
    q = make_float2(__fdiv_rn(a, d.s), __fdiv_rn(b, d.s));
  } else {
    // residual and reciprocal with their signs turned round, so that a zero keeps its sign: (+0) (-y) + (-0) = -0
    const float2 nv = make_float2(-a, -b), ny = make_float2(-d.y, -d.y), s = make_float2(d.s, d.s);
    q = make_float2(nv.x * ny.x, nv.y * ny.y);
    q = fma2(fma2(q, s, nv), ny, q);
    q = fma2(fma2(q, s, nv), ny, q);
  }
  // NaN becomes -448, as the comparison order says
  q.x = fminf(fmaxf(q.x, -kE4m3Max), kE4m3Max);
  q.y = fminf(fmaxf(q.y, -kE4m3Max), kE4m3Max);
  return static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(q, __NV_SATFINITE, __NV_E4M3));
}
// The same for eight values known to hold no NaN and a divisor that is not `plain`: 4.3 instructions per value (the
// conversion itself saturates).  Unpacking negates: a bf16 in the upper half of a word, sign bit flipped.
__device__ __forceinline__ uint2 quant8_fast(const uint4& w, unsigned long long ny2, unsigned long long s2) {
  const uint32_t u[4] = {w.x, w.y, w.z, w.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t lo = u[i] * 65536u + 0x80000000u, hi = (u[i] & 0xffff0000u) ^ 0x80000000u;
    asm("{\n\t.reg .b64 nv, q, r;\n\t.reg .b32 x, y;\n\t.reg .b16 h;\n\t"
        "mov.b64 nv, {%1, %2};\n\t"
        "mul.rn.f32x2 q, nv, %3;\n\t"
        "fma.rn.f32x2 r, q, %4, nv;\n\t"
        "fma.rn.f32x2 q, r, %3, q;\n\t"
        "fma.rn.f32x2 r, q, %4, nv;\n\t"
        "fma.rn.f32x2 q, r, %3, q;\n\t"
        "mov.b64 {x, y}, q;\n\t"
        "cvt.rn.satfinite.e4m3x2.f32 h, y, x;\n\t"
        "cvt.u32.u16 %0, h;\n\t}"
        : "=r"(o[i]) : "r"(lo), "r"(hi), "l"(ny2), "l"(s2));
  }
  return make_uint2(__byte_perm(o[0], o[1], 0x5410), __byte_perm(o[2], o[3], 0x5410));
}
__device__ __forceinline__ unsigned long long twice(float x) {
  const unsigned long long u = __float_as_uint(x);
  return u << 32 | u;
}
__device__ __forceinline__ uint2 quant8(const uint4& w, const Divisor& d) {
  const uint32_t u[4] = {w.x, w.y, w.z, w.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = quant2(__uint_as_float(u[i] << 16), __uint_as_float(u[i] & 0xffff0000u), d);
  return make_uint2(o[0] | (o[1] << 16), o[2] | (o[3] << 16));
}
// larger magnitude of two pairs of bf16 (the sign is not used); a NaN wins
__device__ __forceinline__ uint32_t max_abs2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// lane l of the warp holds bf16 values 8l .. 8l+7 and 256+8l .. (two 16-byte loads) and, for l < 8, 512+8l ..
__device__ __forceinline__ void load_row(const __nv_bfloat16* src, int lane, uint4 (&v)[3]) {
  v[0] = *reinterpret_cast<const uint4*>(src + 8 * lane);
  v[1] = *reinterpret_cast<const uint4*>(src + 256 + 8 * lane);
  v[2] = lane < 8 ? *reinterpret_cast<const uint4*>(src + 512 + 8 * lane) : make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ void unpack8(const uint4& w, float (&f)[8]) {
  const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(u[i] << 16);
    f[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ float row_amax(const Params& p, int r, int lane) {     // this lane's share
  uint4 v[3];
  load_row(p.rows + static_cast<long long>(r) * p.row_stride, lane, v);
  float mx = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float f[8];
    unpack8(v[k], f);
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = fmaxf(mx, fabsf(f[i]));
  }
  return mx;
}
__device__ __forceinline__ float warp_max(float mx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  return mx;
}
__device__ __forceinline__ float scale_of(float amax) { return __fdiv_rn(fmaxf(amax, 1e-12f), kE4m3Max); }
__device__ __forceinline__ void store_row(const Params& p, int r, int slot, const Divisor& d, int lane) {
  uint4 v[3];
  load_row(p.rows + static_cast<long long>(r) * p.row_stride, lane, v);
  uint8_t* dst = p.cache + static_cast<long long>(slot) * kD;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k == 2 && lane >= 8) break;
    const uint2 o = quant8(v[k], d);
    *reinterpret_cast<uint2*>(dst + k * 256 + 8 * lane) = o;
  }
}
// the page held rows under a smaller scale: bring its bytes to the new one (threads t, t + nt, ... of a group)
__device__ __forceinline__ void requantise(const Params& p, int page, float old, float cand, int t, int nt) {
  uint4* words = reinterpret_cast<uint4*>(p.cache + static_cast<long long>(page) * p.page_size * kD);
  const int n_words = p.page_size * (kD / 16);
#pragma unroll 2
  for (int i = t; i < n_words; i += nt) {
    uint4 w4 = words[i];
    uint32_t* w = reinterpret_cast<uint32_t*>(&w4);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t o = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        float q = __fdiv_rn(decode_e4m3(static_cast<uint8_t>(w[k] >> (8 * b))) * old, cand);
        q = fminf(fmaxf(q, -kE4m3Max), kE4m3Max);
        o |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(q, __NV_SATFINITE, __NV_E4M3)) << (8 * b);
      }
      w[k] = o;
    }
    words[i] = w4;
  }
}
// page of a row: -1 = not stored (slot -1, or a slot past the cache, which is reported)
__device__ __forceinline__ int page_of(const Params& p, int slot) {
  if (slot < 0) return -1;
  const int page = slot / p.page_size;
  return page < p.num_pages ? page : -1;
}

// first row of a run: the page changes here.  Pages of more than kMaxRun rows, what a CTA of run_write_kernel holds, have their runs
// cut every kMaxRun rows, so that no CTA is left with a long one (65 536 rows in pages of 256: 76 us with runs of 256, 58 now).
constexpr int kMaxRun = 64;
__device__ __forceinline__ bool is_head(const Params& p, int r, int page) {
  return r == 0 || page_of(p, p.slots[r - 1]) != page || (p.page_size > kMaxRun && r % kMaxRun == 0);
}

constexpr int kSmallRows = 1024;
template <int kThreads>
__global__ void __launch_bounds__(kThreads) small_write_kernel(const Params p) {
  constexpr int kWarps = kThreads / 32;
  __shared__ int mine[kSmallRows];
  __shared__ int n_mine;
  __shared__ float wmax[kWarps];
  griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.x;
  const int slot0 = p.slots[r0];
  if (slot0 < 0) return;
  const int page = slot0 / p.page_size;
  if (page >= p.num_pages) {
    if (tid == 0 && p.status != nullptr) atomicCAS(p.status, 0, FTB_ERR_BAD_INDEX);
    return;
  }
  if (tid == 0) n_mine = 0;
  __syncthreads();
  int earlier = 0;
  for (int r = tid; r < p.n_rows; r += kThreads) {
    if (page_of(p, p.slots[r]) != page) continue;
    if (r < r0) earlier = 1;
    else mine[atomicAdd(&n_mine, 1)] = r;
  }
  if (__syncthreads_or(earlier)) return;                  // the CTA of an earlier row has this page
  const int n = n_mine;
  float mx = 0.0f;
  for (int i = warp; i < n; i += kWarps) mx = fmaxf(mx, row_amax(p, mine[i], lane));
  mx = warp_max(mx);
  if (lane == 0) wmax[warp] = mx;
  const float old = p.scale[page];
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kWarps; ++w) mx = fmaxf(mx, wmax[w]);
  const float cand = scale_of(mx);
  const float scale = cand > old ? cand : old;
  if (cand > old) {
    if (old > 0.0f) {
      requantise(p, page, old, cand, tid, kThreads);
      __syncthreads();
    }
    if (tid == 0) p.scale[page] = cand;
  }
  const Divisor d = make_divisor(scale);
  for (int i = warp; i < n; i += kWarps) store_row(p, mine[i], p.slots[mine[i]], d, lane);
}

__global__ void __launch_bounds__(256) run_count_kernel(const Params p) {
  griddep_launch();
  griddep_wait();
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= p.n_rows) return;
  const int slot = p.slots[r];
  if (slot < 0) return;
  const int page = slot / p.page_size;
  if (page >= p.num_pages) {
    if (p.status != nullptr) atomicCAS(p.status, 0, FTB_ERR_BAD_INDEX);
    return;
  }
  if (is_head(p, r, page)) atomicAdd(p.cand + page, 1u);
}

constexpr int kChunk = 64;                     // most rows whose run heads one CTA looks after (kHeads)
constexpr int kWarpRun = 8;                    // longer runs take the whole CTA
constexpr int kRunThreads = 512;
constexpr int kRunWarps = kRunThreads / 32;
constexpr int kRowVecs = kD / 8;               // 72 pieces of 16 bytes per row
constexpr int kHeld = 9;                       // pieces a lane keeps in shared memory: a warp holds 4 rows (288 pieces), the CTA 64
constexpr int kRunSmem = kHeld * kRunThreads * 16;
template <int kHeads>
__global__ void __launch_bounds__(kRunThreads, 3) run_write_kernel(const Params p) {
  extern __shared__ uint4 keep[];              // piece x of the run; a thread reads only what it copied itself
  __shared__ int slot_of[2 * kChunk + 1], page_at[2 * kChunk + 1];   // rows c0 - 1 .. c0 + 127: the chunk and what its last run may reach into
  __shared__ unsigned breaks[2 * kChunk / 32];                       // bit x: row c0 + x is not of the run of the row before it
  __shared__ int long_head[kChunk / kWarpRun + 1], long_len[kChunk / kWarpRun + 1], short_head[kChunk], short_len[kChunk];
  __shared__ int n_long, n_short, first_break;
  __shared__ unsigned wmax[kRunWarps];
  // Pages of several runs of rows are left to the kernels behind.  Pages larger than a run always are, so that one has work for every CTA: begun early, on
  // the SMs that are through first, its CTAs would crowd there (65 536 rows in pages of 256 rows whose scale rises: 117 us one after the other, 141
  // overlapped; of 128 rows 105 / 121).
  if (p.page_size <= kChunk) griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c0 = blockIdx.x * kHeads;
  if (tid <= 2 * kChunk) {
    const int r = c0 - 1 + tid;
    const int slot = r >= 0 && r < p.n_rows ? p.slots[r] : -1;
    slot_of[tid] = slot;
    page_at[tid] = r == -1 ? -2 : page_of(p, slot);
  }
  if (tid == 0) { n_long = 0; n_short = 0; }
  __syncthreads();
  auto cut = [&](int r) { return p.page_size > kMaxRun && r % kMaxRun == 0; };
  if (tid < 2 * kChunk) {
    const unsigned b = __ballot_sync(0xffffffffu, page_at[tid + 1] != page_at[tid] || cut(c0 + tid));
    if (lane == 0) breaks[warp] = b;
  }
  __syncthreads();
  auto slot_at = [&](int r) { return r - c0 < 2 * kChunk ? slot_of[r - c0 + 1] : p.slots[r]; };
  if (tid < kHeads && page_at[tid + 1] >= 0 && ((breaks[warp] >> lane) & 1u)) {
    // the next break behind this head, if it lies in the window
    int word = warp;
    unsigned rest = lane == 31 ? 0u : breaks[word] & (0xffffffffu << (lane + 1));
    while (rest == 0 && ++word < 2 * kChunk / 32) rest = breaks[word];
    const int len = rest != 0 ? 32 * word + __ffs(static_cast<int>(rest)) - 1 - tid : 2 * kChunk - tid;
    if (len <= kWarpRun) {
      const int at = atomicAdd(&n_short, 1);
      short_head[at] = c0 + tid; short_len[at] = len;
    } else {
      const int at = atomicAdd(&n_long, 1);
      long_head[at] = c0 + tid; long_len[at] = rest != 0 ? len : -len;     // negative: it goes on behind the window
    }
  }
  __syncthreads();
  for (int j = warp; j < n_short; j += kRunWarps) {
    const int r = short_head[j], len = short_len[j];
    const int page = page_at[r - c0 + 1];
    float mx = 0.0f;
    for (int i = 0; i < len; ++i) mx = fmaxf(mx, row_amax(p, r + i, lane));
    const float cand = scale_of(warp_max(mx));
    const unsigned runs = p.cand[page];
    const float old = p.scale[page];
    const bool rises = cand > old;
    // several runs, or a page to requantise that is too much for a warp: to the kernels behind this one
    if (runs != 1u || (rises && old > 0.0f && p.page_size > kWarpRun)) {
      if (lane == 0) atomicMax(p.cand + page, __float_as_uint(cand));
      continue;
    }
    if (rises && old > 0.0f) {
      requantise(p, page, old, cand, lane, 32);
      __syncwarp();
    }
    if (lane == 0 && rises) p.scale[page] = cand;
    const Divisor d = make_divisor(cand > old ? cand : old);
    for (int i = 0; i < len; ++i) store_row(p, r + i, slot_at(r + i), d, lane);
  }
  __syncthreads();
  const int n = n_long;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    const int r = long_head[k];
    const int page = page_at[r - c0 + 1];
    int len = long_len[k];
    if (len < 0) {                                        // look for its end, 512 rows at a time
      len = -len;
      for (;;) {
        if (tid == 0) first_break = kRunThreads;
        __syncthreads();
        const int x = r + len + tid;
        if (!(x < p.n_rows && page_of(p, p.slots[x]) == page && !cut(x))) atomicMin(&first_break, tid);
        __syncthreads();
        const int more = first_break;
        len += more;
        __syncthreads();
        if (more < kRunThreads) break;
      }
    }
    const unsigned runs = p.cand[page];
    const float old = p.scale[page];
    // Runs of up to 64 rows stay in shared memory: warp w keeps rows 4 w .. 4 w + 3, lane l pieces l % 8 + 8 i of row l / 8, so
    // that a lane has one row, one slot and constant offsets.  A longer run goes through the rows a warp at a time, twice.
    const bool held = len <= 4 * kRunWarps;
    const int own = 4 * warp + (lane >> 3);
    uint4* mine = keep + warp * (4 * kRowVecs) + lane;
    auto block_max = [&](unsigned m) {
      m = __reduce_max_sync(0xffffffffu, m);
      __syncthreads();
      if (lane == 0) wmax[warp] = m;
      __syncthreads();
      return __reduce_max_sync(0xffffffffu, wmax[lane & (kRunWarps - 1)]);
    };
    uint32_t m2 = 0;
    if (held) {
      if (own < len) {
        const __nv_bfloat16* src = p.rows + static_cast<long long>(r + own) * p.row_stride + (lane & 7) * 8;
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(mine));
#pragma unroll
        for (int i = 0; i < kHeld; ++i)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 512), "l"(src + i * 64) : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
        for (int i = 0; i < kHeld; ++i) {
          const uint4 w = mine[32 * i];
          m2 = max_abs2(m2, max_abs2(max_abs2(w.x, w.y), max_abs2(w.z, w.w)));
        }
      }
    } else {
#pragma unroll 2
      for (int i = warp; i < len; i += kRunWarps) {
        uint4 v[3];
        load_row(p.rows + static_cast<long long>(r + i) * p.row_stride, lane, v);
#pragma unroll
        for (int k2 = 0; k2 < 3; ++k2) m2 = max_abs2(m2, max_abs2(max_abs2(v[k2].x, v[k2].y), max_abs2(v[k2].z, v[k2].w)));
      }
    }
    unsigned bits = block_max(max((m2 << 16) & 0x7fff0000u, m2 & 0x7fff0000u));   // magnitudes order as integers, NaN last
    const bool has_nan = bits > 0x7f800000u;
    if (has_nan) {                                        // the maximum leaves them out
      float mx = 0.0f;
      for (int i = warp; i < len; i += kRunWarps) mx = fmaxf(mx, row_amax(p, r + i, lane));
      bits = block_max(__float_as_uint(mx));
    }
    const float cand = scale_of(__uint_as_float(bits));
    if (runs != 1u) {
      if (tid == 0) atomicMax(p.cand + page, __float_as_uint(cand));
      continue;
    }
    if (cand > old) {
      if (old > 0.0f) {
        requantise(p, page, old, cand, tid, kRunThreads);
        __syncthreads();
      }
      if (tid == 0) p.scale[page] = cand;
    }
    const Divisor d = make_divisor(cand > old ? cand : old);
    if (held && !d.plain && !has_nan) {
      if (own < len) {
        const unsigned long long ny2 = twice(-d.y), s2 = twice(d.s);
        uint8_t* dst = p.cache + static_cast<long long>(slot_at(r + own)) * kD + (lane & 7) * 8;
#pragma unroll 3
        for (int i = 0; i < kHeld; ++i) *reinterpret_cast<uint2*>(dst + i * 64) = quant8_fast(mine[32 * i], ny2, s2);
      }
    } else {
      for (int i = warp; i < len; i += kRunWarps) store_row(p, r + i, slot_at(r + i), d, lane);
    }
  }
}

// pages with several runs: their word holds the candidate scale (float bits; counts are far smaller)
constexpr unsigned int kCandMin = 0x20000000u;
// CTA b looks after pages b, b + gridDim.x, ...: all their words at once, then the few that rise, a page at a time.
__global__ void __launch_bounds__(256) page_settle_kernel(const Params p) {
  __shared__ int rises[256];
  __shared__ int n_rises;
  griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x;
  for (int first = blockIdx.x; first < p.num_pages; first += gridDim.x * 256) {
    if (tid == 0) n_rises = 0;
    __syncthreads();
    const long long mine = first + static_cast<long long>(tid) * gridDim.x;
    if (mine < p.num_pages) {
      const unsigned word = p.cand[mine];
      if (word >= kCandMin && __uint_as_float(word) > p.scale[mine]) rises[atomicAdd(&n_rises, 1)] = static_cast<int>(mine);
    }
    __syncthreads();
    const int n = n_rises;
    for (int i = 0; i < n; ++i) {
      const int page = rises[i];
      const float cand = __uint_as_float(p.cand[page]), old = p.scale[page];
      if (old > 0.0f) requantise(p, page, old, cand, tid, 256);
      __syncthreads();                                    // every thread has read the old scale
      if (tid == 0) p.scale[page] = cand;
    }
    __syncthreads();
  }
}

// A warp looks after `per_warp` rows (at most 32, a power of two) and stores those of the pages that the kernel before settled.
__global__ void __launch_bounds__(256) row_store_kernel(const Params p, int per_warp) {
  griddep_launch();
  griddep_wait();
  const int lane = threadIdx.x & 31;
  const long long r0 = (static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5)) * per_warp;
  const int slot = lane < per_warp && r0 + lane < p.n_rows ? p.slots[r0 + lane] : -1;
  const int page = page_of(p, slot);
  const unsigned word = page >= 0 ? p.cand[page] : 0u;
  const float scale = word >= kCandMin ? p.scale[page] : 0.0f;
  for (unsigned todo = __ballot_sync(0xffffffffu, word >= kCandMin); todo != 0; todo &= todo - 1) {
    const int l = __ffs(static_cast<int>(todo)) - 1;
    store_row(p, static_cast<int>(r0) + l, __shfl_sync(0xffffffffu, slot, l), make_divisor(__shfl_sync(0xffffffffu, scale, l)), lane);
  }
}

}  // namespace kvw
}  // namespace ftb

extern "C" FTB_API int64_t ftb_kv_cache_write_workspace_bytes(int32_t num_pages) {
  return num_pages > 0 ? static_cast<int64_t>(num_pages) * 4 : 0;
}

extern "C" FTB_API int ftb_kv_cache_write_fp8(const ftb_kv_cache_write_args* a, void* stream) {
  using namespace ftb;
  if (a == nullptr) { set_last_error("ftb_kv_cache_write_fp8: args is NULL"); return FTB_ERR_INVALID; }
  if (a->n_rows < 0 || a->num_pages <= 0 || a->page_size <= 0) {
    set_last_error("ftb_kv_cache_write_fp8: bad sizes n_rows=%d num_pages=%d page_size=%d", a->n_rows, a->num_pages, a->page_size);
    return FTB_ERR_INVALID;
  }
  if (a->n_rows == 0) return FTB_OK;
  if (!a->rows || !a->slot_mapping || !a->kv_cache || !a->kv_scale || !a->workspace) {
    set_last_error("ftb_kv_cache_write_fp8: null pointer");
    return FTB_ERR_INVALID;
  }
  if ((reinterpret_cast<uintptr_t>(a->rows) & 15) || (a->row_stride % 8) || (reinterpret_cast<uintptr_t>(a->kv_cache) & 15) ||
      (reinterpret_cast<uintptr_t>(a->workspace) & 3)) {
    set_last_error("ftb_kv_cache_write_fp8: rows and kv_cache must be 16-byte aligned, row_stride a multiple of 8 elements");
    return FTB_ERR_INVALID;
  }
  if (a->workspace_bytes < ftb_kv_cache_write_workspace_bytes(a->num_pages)) {
    set_last_error("ftb_kv_cache_write_fp8: workspace of %lld bytes, ftb_kv_cache_write_workspace_bytes() asks for %lld",
                   static_cast<long long>(a->workspace_bytes), static_cast<long long>(ftb_kv_cache_write_workspace_bytes(a->num_pages)));
    return FTB_ERR_INVALID;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  kvw::Params p;
  p.rows = reinterpret_cast<const __nv_bfloat16*>(a->rows);
  p.slots = a->slot_mapping;
  p.cache = reinterpret_cast<uint8_t*>(a->kv_cache);
  p.scale = a->kv_scale;
  p.cand = reinterpret_cast<unsigned int*>(a->workspace);
  p.n_rows = a->n_rows; p.num_pages = a->num_pages; p.page_size = a->page_size;
  p.row_stride = a->row_stride;
  p.status = a->status;
  // Up to kSmallRows rows: one launch without a workspace instead of five.  A decode step over 37 353 pages spent 24 to 42 us in
  // the settle kernel alone when that had a CTA per page; such a step of 128 rows is 36 us shorter (396 -> 360 us).
  // A CTA has a page to itself, so the line also lies where the rows of one page are many: 1024 rows in pages of 256 take it 39 us, the large
  // path 21 (both with the host's part).  More threads for pages of 128: 20.4 -> 16.2 us.
  if (a->n_rows <= 64 || (a->n_rows <= kvw::kSmallRows && a->page_size <= 128)) {
    const bool narrow = a->n_rows <= 64 || a->page_size <= 64;
    return check_cuda(launch_overlapped(narrow ? kvw::small_write_kernel<256> : kvw::small_write_kernel<512>, static_cast<unsigned>(a->n_rows), narrow ? 256 : 512, 0,
                                        st, 1, p), "ftb_kv_cache_write_fp8 launch");
  }
  cudaError_t e = cudaMemsetAsync(p.cand, 0, static_cast<size_t>(a->num_pages) * 4, st);
  if (e != cudaSuccess) return check_cuda(e, "ftb_kv_cache_write_fp8: cudaMemsetAsync");
  const unsigned row_blocks = static_cast<unsigned>((static_cast<long long>(a->n_rows) + 255) / 256);
  // Rows per CTA of the write kernel: few enough that every SM has a CTA where that is possible, since the runs of a CTA go one after the
  // other, and no fewer: 4096 rows in whole pages take 14.7 us with 64 rows per CTA and 17.5 with 16, 2048 one-row runs 16.8 and 10.9.
  int heads = 16;
  while (heads < kvw::kChunk && heads * 148LL < a->n_rows) heads *= 2;
  const auto run_write = heads == 16 ? kvw::run_write_kernel<16> : heads == 32 ? kvw::run_write_kernel<32> : kvw::run_write_kernel<kvw::kChunk>;
  e = cudaFuncSetAttribute(run_write, cudaFuncAttributeMaxDynamicSharedMemorySize, kvw::kRunSmem);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(run_write)");
  e = launch_overlapped(kvw::run_count_kernel, row_blocks, 256, 0, st, 1, p);
  if (e == cudaSuccess)
    e = launch_overlapped(run_write, static_cast<unsigned>((static_cast<long long>(a->n_rows) + heads - 1) / heads), kvw::kRunThreads, kvw::kRunSmem, st, 1, p);
  // Pages with several runs.  The settle kernel: eight CTAs per SM, or one per page.  The store kernel: as many rows per warp as keep it at
  // one wave, up to 32.
  if (e == cudaSuccess) e = launch_overlapped(kvw::page_settle_kernel, static_cast<unsigned>(a->num_pages < 1184 ? a->num_pages : 1184), 256, 0, st, 1, p);
  int per_warp = 1;
  while (per_warp < 32 && static_cast<long long>(per_warp) * 9472 < a->n_rows) per_warp *= 2;
  const long long per_cta = 8LL * per_warp;
  if (e == cudaSuccess) e = launch_overlapped(kvw::row_store_kernel, static_cast<unsigned>((a->n_rows + per_cta - 1) / per_cta), 256, 0, st, 1, p, per_warp);
  return check_cuda(e, "ftb_kv_cache_write_fp8 launch");
}
