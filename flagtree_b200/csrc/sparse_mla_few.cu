// Sparse MLA forward for few heads (and for few tokens or short lists of many heads, 64 at a time), sm_100a: persistent CTAs, the products taken
// the other way round.
//
// The CTA pairs of sparse_mla_ring.cu put the heads on the 128 rows of the MMA, so with 16 heads seven eighths of every
// instruction are rows of zeros, and they fetch every selected row twice.  Here one CTA works on one item (a token, or a part of its
// list), a row is fetched once, and the gathered rows are the rows of the MMA:
//
//   S^T [64 keys x NH heads]   = K_tile [64 x 576] . Q^T [576 x NH]         (36 MMAs 64 x NH x 16, A = K, B = Q)
//   O^T [512 dims x NH heads] += V_tile^T [512 x 64 keys] . P^T [64 x NH]   (4 x 4 MMAs 128 x NH x 16, A = the same tile, MN-major)
//
// What bounds it: the MMAs fetch their operands from shared memory at 128 bytes per clock, whatever the shape (cycles
// per MMA: 64 x 16 x 16 31, 64 x 64 x 16 35, 128 x 16 x 16 40, 128 x 64 x 16 49), so a tile of 64 rows costs 36 x 31 + 16 x 40 = 1760
// cycles with 16 heads, and the way of a tile through its slot (gather, scores, softmax, values) is a chain of about
// 4000; two slots of 64 rows run two such chains against each other.  128 rows per tile would cost 2700 for 128 rows, but leave room for
// one slot only.
//
// Roles (warps): softmax and epilogue, four warps for up to 32 heads each; an MMA issuer for either product; sets of four gather warps, 16 rows of
// a tile each (the first loads Q too).
//
// Softmax.  A score row of tensor memory belongs to a key (the 64 rows of S^T lie in the first 16 lanes of each warp's
// quarter), so a maximum over the keys would be a reduction across lanes for every head and tile.  It is not needed: any
// reference near the maximum will do.  Every thread compares its scores with the reference of their heads; only if one of them exceeds it by
// more than the slack, and in the first tile, are the maxima reduced, the references moved and the accumulators rescaled.
// P^T [64 keys x NH] is written over the rope block of the tile, which the second
// product does not read.
//
// The steps (1999 tokens of 16 / 64 heads, topk 2048, us; the pairs take 970 / 958, with the softmax of later steps 846 with 16 heads): one issuer that polls for both products 620 / 813, with
// tiles in thirds and 16 rows freed at a time 780 / 974 (each turn of the issuer cost 330 cycles, most of it the proxy fence), the fence
// moved to the gather warps 741 / 920, two issuers 512 / 719, the first reference from two tiles 525 / 759.  Device time of few tokens in parts,
// pairs / here: 1 token of 16 heads 17.0 / 11.3, 74 tokens of 64 heads 45.6 / 40.0, 1 token of 128 heads 21.2 / 14.7, 16 of them 29.9 / 25.5.
// Taken back: the weights written while the warps vote on the references through an mbarrier 517 -> 549 / 733 -> 772 (its wait costs more
// than the named barrier); pairs of CTAs that share the rows of a token's two head groups 186 -> 190 (a decode step).
//
// e4m3 pages (kFp8).  The gather warps resolve the page table, load a row's bytes, convert them to bf16 times the page's scale
// (as the dequantised table had them) and write the same slots, so nothing goes through a table in memory.  128 tokens of 128 heads, topk 2048: dequantisation and
// attention one after the other 212 us, here 149; three tokens in parts 23 -> 19 (one-pass kernel of one CTA 28.7).
// Every wait is bounded; a wait that runs out sets the abort flag, after which every later wait returns at once.
#include <cuda_fp8.h>

#include <cstring>

#include "launch.cuh"
#include "sm100.cuh"
#include "tmap.cuh"
#include "../../include/flagtree_b200.h"

namespace ftb {

void set_last_error(const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

namespace mla_few {

constexpr int kDqk = 576;
constexpr int kNChunk = 9;
constexpr int kNT = 64;                        // gathered rows per tile = rows of the first product
constexpr int kBlock = kNT * 128;              // 8192: [64 rows x 128 B], one 64-column block of the tile
constexpr int kSlot = kNChunk * kBlock;        // 73728
constexpr int kSlots = 2;
constexpr int kGather = 4;                     // gather warps, 16 rows of a tile each
constexpr int kThirds = 3;                    // a tile's columns arrive, and are multiplied, in three parts
constexpr int kBatch = 64;                     // items per CTA and launch

template <int NH, bool kFp8>
struct Shape {
  static constexpr int kGroups = NH == 64 ? 2 : 1;              // softmax groups of four warps
  static constexpr int kHeads = NH / kGroups;                   // heads per group
  // Warps: softmax, the MMA issuers, gather.  bf16 rows: four gather warps on schedulers that the issuers (four apart: one scheduler) are not
  // on; they wait for their copies to land, and with two sets of them every slot has one of its own (64 heads: two sets would leave the
  // softmax too few registers).  e4m3 rows: the issuers in a warpgroup of their own, then eight warps that convert; with 64 heads registers
  // move to the softmax: 640 x 96 at launch = 61440 >= 8 x 32 x 128 + 4 x 32 x 56 + 8 x 32 x 80 = 60416.
  static constexpr int kSets = kGroups == 2 ? 1 : 2;
  static constexpr int kIssuer = 4 * kGroups, kValueIssuer = kIssuer + (kFp8 ? 1 : 4), kConvert0 = kIssuer + 4, kConverts = 8;
  static constexpr int kThreads = (kFp8 ? kConvert0 + kConverts : kIssuer + (kSets == 2 ? 11 : 6)) * 32;
  static constexpr bool kSplitRegs = kFp8 && kGroups == 2;
  static constexpr int kRegsSoftmax = 128, kRegsIssue = 56, kRegsConvert = 80;
  __device__ static int producer(int warp) {
    if (kFp8) return warp - kConvert0;
    const int w = warp - kIssuer;
    return w >= 1 && (w & 3) != 0 ? w - 1 - (w >> 2) : -1;
  }
  static constexpr int kQBlock = NH * 128;                      // [NH heads x 128 B]
  static constexpr int kOffQ = kSlots * kSlot;
  static constexpr int kOffMisc = kOffQ + kNChunk * kQBlock;
  static constexpr uint32_t kColO = 0, kColS = 4 * NH;          // tensor memory: four O^T blocks, then an S^T per slot
  static constexpr uint32_t kCols = NH == 16 ? 128 : NH == 32 ? 256 : 512;
};

struct Params {
  const void* kv;      // bf16 rows, or e4m3 pages
  long long kv_sr;
  const int32_t* indices;
  __nv_bfloat16* out;
  float* lse;
  int s_q, h, s_kv, topk;
  long long idx_st, out_st, out_sh, lse_st;
  float scale_log2;
  int lse_base2;
  int* status;
  int n_splits, n_groups;   // an item: a token, 64 of its heads (all, if there are no more), a part of its list; the part varies fastest
  float* part_out;     // [s_q, n_splits, h, 512] fp32
  float* part_lse;     // [s_q, n_splits, h], base 2
  float max_slack;     // how far (log2) the reference may lag behind the running maximum
  // e4m3 pages
  const float* kv_scale;
  const int32_t* block_table;
  const int32_t* context_lens;
  int page_size, q_per_seq;
  int tok0;            // the launch's first token, counted over the call: sequences go by the latter
  long long bt_stride;
};

struct Misc {
  unsigned long long k_full[kSlots][kThirds];   // three column blocks: the gather warps of the slot, when their copies have landed
  unsigned long long k_free[kSlots][kGather];   // 16 rows: tcgen05.commit behind their part of the second product
  unsigned long long s_full[kSlots];   // tcgen05.commit behind the first
  unsigned long long p_full[kSlots];   // softmax warps: P^T is written, S^T read
  unsigned long long q_full, q_free;   // Q of the item has landed / tcgen05.commit behind its last first product
  unsigned long long o_free;           // softmax warps: O^T has been read
  uint32_t tmem_base;
  int abort_flag;
  int bad_index;
  alignas(16) uint16_t valid_mask[kSlots][4];   // 16 rows each
  unsigned short nt[2 * kBatch];       // per item: number of tiles, first tile
  int last[kBatch];                    // entries of its list up to the last that is not negative
  alignas(16) float neg_ref[64];       // minus the reference of a head (log2), 0 where it has none yet
  alignas(16) float alpha[64];         // rescale factors
  alignas(16) float inv_l[64];
  float m_ref[64];                     // the reference, -inf where there is none yet
  int no_ref[2];                       // per group: does a head have none?
  float part[8][32], part_odd[8][32];  // per softmax warp and head: maxima, then sums of the even and the odd tiles
};

// floats <-> integers whose signed order is the order of the floats
__device__ __forceinline__ int to_ordered(float x) {
  const int i = __float_as_int(x);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float from_ordered(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[N]) {
  if constexpr (N == 16) tmem_ld16(taddr, r);
  else tmem_ld32(taddr, r);
}
template <int N>
__device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&r)[N]) {
  if constexpr (N == 16) tmem_st16(taddr, r);
  else tmem_st32(taddr, r);
}

// Masked entries (-1) fetch a row all the same, which is multiplied by zero: the one that the lane fetched for the tile before, or in
// the first tile another one of the token's (this function, the rare path: the first row that the list names; `none` if it names none).
// With row 0 for all of them every SM would fetch the same 1152 bytes, and a row 0 that holds no numbers would spoil foreign tokens.
__device__ __noinline__ int first_row(const int32_t* idx_row, int n_rows, int s_kv, int none) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int j = 0; j < n_rows; j += 32) {
    const int v = j + lane < n_rows ? idx_row[j + lane] : -1;
    const unsigned have = __ballot_sync(0xffffffffu, v >= 0 && v < s_kv);
    if (have != 0u) return __shfl_sync(0xffffffffu, v, __ffs(static_cast<int>(have)) - 1);
  }
  return none;
}

template <int NH, bool kFp8>
__global__ void __launch_bounds__(Shape<NH, kFp8>::kThreads, 1)
sparse_mla_few_heads_kernel(const __grid_constant__ CUtensorMap tm_q, const Params p) {
  using Sh = Shape<NH, kFp8>;
  constexpr int kHeads = Sh::kHeads;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw_addr);
  const uint32_t q_s = base + Sh::kOffQ;
  Misc* misc = reinterpret_cast<Misc*>(sm + Sh::kOffMisc);
  volatile int* abort_flag = &misc->abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = warp_uniform(tid >> 5);

  const bool one_each = p.s_q * p.n_splits * p.n_groups <= static_cast<int>(gridDim.x);   // items
  if (one_each) griddep_launch();
  if (tid == 0) {
    misc->bad_index = 0;
    for (int i = 0; i < kSlots; ++i) {
      for (int j = 0; j < kThirds; ++j) mbar_init(smem_u32(&misc->k_full[i][j]), kFp8 ? Sh::kConverts : kGather);
      for (int j = 0; j < kGather; ++j) mbar_init(smem_u32(&misc->k_free[i][j]), 1);
      mbar_init(smem_u32(&misc->s_full[i]), 1);
      mbar_init(smem_u32(&misc->p_full[i]), 4 * Sh::kGroups);
    }
    mbar_init(smem_u32(&misc->q_full), 1);
    mbar_init(smem_u32(&misc->q_free), 1);
    mbar_init(smem_u32(&misc->o_free), 4 * Sh::kGroups);
    fence_mbar_init();
  }
  griddep_wait();
  if (tid == 0) misc->abort_flag = (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
  __syncthreads();
  if (misc->abort_flag) return;   // an earlier launch on this status word failed: do nothing
  if (warp == Sh::kIssuer) {
    tmem_alloc(smem_u32(&misc->tmem_base), Sh::kCols);
    tmem_relinquish();
    tc_fence_before();
  }
  if (p.h < NH) {
    // a load of Q writes h rows of a block; the rows below feed heads that are never stored, but they should hold numbers
    for (int x = tid; x < kNChunk * Sh::kQBlock / 16; x += Sh::kThreads)
      asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(q_s + x * 16), "r"(0) : "memory");
    fence_proxy_async_smem();
  }
  // ---- tiles per item (last entry that is not negative, rounded up; at least one, entirely masked if the item selects nothing)
  const int n_ctas = gridDim.x, first_item = blockIdx.x;
  const int per_token = p.n_splits * p.n_groups;
  auto token_of = [&](int item) { return per_token == 1 ? item : item / per_token; };
  const int nb = (p.s_q * per_token - first_item + n_ctas - 1) / n_ctas;     // at most kBatch: the host sees to it
  for (int t = tid; t < nb; t += Sh::kThreads) misc->last[t] = 0;
  __syncthreads();
  {
    const int pieces = (p.topk + 511) >> 9;
#pragma unroll 1
    for (int x = warp; x < nb * pieces; x += Sh::kThreads / 32) {
      const int t = x / pieces, j0 = (x - t * pieces) * 512 + lane;
      const int32_t* idx_row = p.indices + static_cast<long long>(token_of(first_item + t * n_ctas)) * p.idx_st;
      int v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = j0 + 32 * j < p.topk ? idx_row[j0 + 32 * j] : -1;
      int local = 0;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (v[j] >= 0) local = j0 + 32 * j + 1;
      local = __reduce_max_sync(0xffffffffu, local);
      if (lane == 0 && local > 0) atomicMax(&misc->last[t], local);
    }
  }
  __syncthreads();
  for (int t = tid; t < nb; t += Sh::kThreads) {
    const int item = first_item + t * n_ctas;
    const int tiles = min(65535, max(1, (misc->last[t] + kNT - 1) / kNT));
    const int part = (tiles + p.n_splits - 1) / p.n_splits;
    int first = item % p.n_splits * part;
    if (first >= tiles) first = 65535;                     // nothing left for this part: a tile past the list
    misc->nt[t] = static_cast<unsigned short>(max(1, min(part, tiles - first)));
    misc->nt[kBatch + t] = static_cast<unsigned short>(first);
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc->tmem_base;
  const int prod = Sh::producer(warp);
  const int group = warp < 4 ? 0 : warp < 4 * Sh::kGroups ? 1 : -1;

  auto softmax = [&]() {
    // ------------------------------------------------------------------ softmax and epilogue
    const int q4 = warp & 3, pw = group * 4 + q4, h0 = group * kHeads;
    const bool active = lane < 16;                         // the lanes that hold a key
    const int key = q4 * 16 + (lane & 15);
    const int bar_id = 1 + group;
    uint32_t G = 0;
    // sums of the weights: lane l holds heads l % 16 * kPer .. of its group, over the 16 keys of this warp, of the even and of the odd tiles.
    // The order of the additions is the one of the kernel for many heads, so that a head's bits do not depend on how many
    // heads the call has.
    constexpr int kPer = kHeads / 16;
    float l_run[2][kPer];
    const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
#pragma unroll 1
    for (int t = 0; t < nb; ++t) {
      const int item = first_item + t * n_ctas;
      const int tok = token_of(item), split = item % p.n_splits, head0 = (item / p.n_splits) % p.n_groups * NH;
      const int n_heads = min(p.h - head0, NH);            // of the item
      const int n_tiles = warp_uniform(misc->nt[t]);
#pragma unroll
      for (int j = 0; j < kPer; ++j) l_run[0][j] = l_run[1][j] = 0.0f;
#pragma unroll 1
      for (int i = 0; i < n_tiles; ++i, ++G) {
        const uint32_t s = G & 1u, ph = (G >> 1) & 1u;
        mbar_wait(smem_u32(&misc->s_full[s]), ph, abort_flag);
        tc_fence_after();
        const bool valid = active && ((static_cast<uint32_t>(misc->valid_mask[s][q4]) >> lane) & 1u) != 0u;
        const uint32_t t_s = tmem_addr(tmem, q4 * 32, Sh::kColS + s * NH + h0);
        uint32_t sr[kHeads];
        tmem_ld(t_s, sr);
        tmem_wait_ld();
        float2 x[kHeads / 2];
        float mx = -INFINITY;
        auto shift = [&]() {                               // scores relative to the references; a masked key has no weight (2^-inf = 0)
#pragma unroll
          for (int j = 0; j < kHeads; j += 4) {
            const float4 r = *reinterpret_cast<const float4*>(&misc->neg_ref[h0 + j]);
            x[j / 2] = ffma2(make_float2(__uint_as_float(sr[j]), __uint_as_float(sr[j + 1])), scale2, make_float2(r.x, r.y));
            x[j / 2 + 1] = ffma2(make_float2(__uint_as_float(sr[j + 2]), __uint_as_float(sr[j + 3])), scale2, make_float2(r.z, r.w));
          }
#pragma unroll
          for (int j = 0; j < kHeads / 2; ++j) {
            if (!valid) x[j] = make_float2(-INFINITY, -INFINITY);
            mx = fmaxf(mx, fmaxf(x[j].x, x[j].y));
          }
        };
        bool move = i == 0 || misc->no_ref[group] != 0;
        if (!move) {
          shift();
          // (a little early: the rule below decides, to the bit as for many heads)
          move = named_bar_any(bar_id, 128, mx > p.max_slack - 0.01f);
        }
        if (move) {
          // maxima of the tile: over the keys of a warp, then over the warps
          tmem_ld(t_s, sr);
          tmem_wait_ld();
          float top[kHeads];
#pragma unroll
          for (int j = 0; j < kHeads; ++j) top[j] = valid ? __uint_as_float(sr[j]) : -INFINITY;
          // The first reference is the maximum of two tiles (the tile of the kernel for many heads); with the true maximum over e4m3 pages that of
          // one, as in the one-CTA kernel: every tile whose maximum is the largest so far then holds a weight of exactly 1 (error against 64 bits, 3 tokens
          // of topk 512: 4.26e-3 with two tiles, 4.24e-3 with one).
          if (i == 0 && n_tiles > 1 && !(kFp8 && p.max_slack == 0.0f)) {
            mbar_wait(smem_u32(&misc->s_full[s ^ 1u]), ((G + 1) >> 1) & 1u, abort_flag);
            tc_fence_after();
            const bool valid1 = active && ((static_cast<uint32_t>(misc->valid_mask[s ^ 1u][q4]) >> lane) & 1u) != 0u;
            uint32_t sr1[kHeads];
            tmem_ld(tmem_addr(tmem, q4 * 32, Sh::kColS + (s ^ 1u) * NH + h0), sr1);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < kHeads; ++j) top[j] = fmaxf(top[j], valid1 ? __uint_as_float(sr1[j]) : -INFINITY);
          }
          int mine = 0;
#pragma unroll
          for (int j = 0; j < kHeads; ++j) {
            const int m = __reduce_max_sync(0xffffffffu, to_ordered(top[j]));
            if (lane == j) mine = m;
          }
          if (lane < kHeads) misc->part[pw][lane] = __int_as_float(mine);
          named_bar_sync(bar_id, 128);
          if (q4 == 0 && lane < kHeads) {
            int m = __float_as_int(misc->part[group * 4][lane]);
#pragma unroll
            for (int w = 1; w < 4; ++w) m = max(m, __float_as_int(misc->part[group * 4 + w][lane]));
            const float most = from_ordered(m) * p.scale_log2;
            float ref = i == 0 ? -INFINITY : misc->m_ref[h0 + lane], a = 1.0f;
            if (most > ref + p.max_slack || ref == -INFINITY) {
              const float old = ref;
              ref = fmaxf(ref, most);
              a = old == -INFINITY ? 0.0f : fast_exp2(old - ref);
            }
            const uint32_t none = __ballot_sync(__activemask(), ref == -INFINITY);
            if (lane == 0) misc->no_ref[group] = static_cast<int>(none);
            misc->m_ref[h0 + lane] = ref;
            misc->neg_ref[h0 + lane] = ref == -INFINITY ? 0.0f : -ref;
            misc->alpha[h0 + lane] = a;
          }
          named_bar_sync(bar_id, 128);
          if (i != 0) {
            // the sums and the accumulator follow, once the tile before has gone into the latter
            mbar_wait(smem_u32(&misc->k_free[s ^ 1u][kGather - 1]), ((G - 1) >> 1) & 1u, abort_flag);
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              uint32_t o[kHeads];
              const uint32_t t_o = tmem_addr(tmem, q4 * 32, Sh::kColO + c * NH + h0);
              tmem_ld(t_o, o);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < kHeads; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * misc->alpha[h0 + j]);
              tmem_st(t_o, o);
            }
            tmem_wait_st();
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
              const float a = misc->alpha[h0 + (lane & 15) * kPer + j];
              l_run[0][j] *= a;
              l_run[1][j] *= a;
            }
          }
          mx = -INFINITY;
          shift();
        }
        // this key's row of P^T: 128 bytes in the tile's rope block, 16-byte pieces of eight heads
        const uint32_t p_row = base + s * kSlot + 8 * kBlock + key * 128;
        uint32_t pk[kHeads / 2];
        float v[kHeads];
#pragma unroll
        for (int j = 0; j < kHeads / 2; ++j) {
          v[2 * j] = fast_exp2(x[j].x);
          v[2 * j + 1] = fast_exp2(x[j].y);
          pk[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
        }
        if (active) {
#pragma unroll
          for (int c = 0; c < kHeads / 8; ++c)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p_row + (((h0 / 8 + c) ^ (key & 7)) << 4)), "r"(pk[4 * c]), "r"(pk[4 * c + 1]),
                         "r"(pk[4 * c + 2]), "r"(pk[4 * c + 3]) : "memory");
        }
        fence_proxy_async_smem();      // the MMA reads the rows through the async proxy
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&misc->p_full[s]));
        // sums over the 16 keys of the warp: every step halves the heads of a lane
#pragma unroll
        for (int d = 8, n = kHeads / 2; d >= 1; d >>= 1, n >>= 1) {
#pragma unroll
          for (int j = 0; j < n; ++j) {
            const bool up = (lane & d) != 0;
            const float keep = up ? v[j + n] : v[j], send = up ? v[j] : v[j + n];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, d);
          }
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          if (i & 1) l_run[1][j] += v[j];
          else l_run[0][j] += v[j];
        }
      }
      if (active) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          misc->part[pw][lane * kPer + j] = l_run[0][j];
          misc->part_odd[pw][lane * kPer + j] = l_run[1][j];
        }
      }
      named_bar_sync(bar_id, 128);
      if (q4 == 0 && lane < kHeads) {
        const float(*even)[32] = &misc->part[group * 4], (*odd)[32] = &misc->part_odd[group * 4];
        const float l = ((even[0][lane] + even[1][lane]) + (even[2][lane] + even[3][lane])) + ((odd[0][lane] + odd[1][lane]) + (odd[2][lane] + odd[3][lane]));
        misc->inv_l[h0 + lane] = l > 0.0f ? 1.0f / l : 0.0f;
        if (h0 + lane < n_heads) {
          const float l2 = l > 0.0f ? misc->m_ref[h0 + lane] + log2f(l) : -INFINITY;
          if (p.n_splits == 1) p.lse[static_cast<long long>(tok) * p.lse_st + head0 + h0 + lane] = (p.lse_base2 || l <= 0.0f) ? l2 : l2 * 0.6931471805599453f;
          else p.part_lse[(static_cast<long long>(tok) * p.n_splits + split) * p.h + head0 + h0 + lane] = l2;
        }
      }
      named_bar_sync(bar_id, 128);
      // ---- out[head][dim] = O^T[dim][head] / l[head]; lane = dim within 32 of a block of 128
      mbar_wait(smem_u32(&misc->k_free[(G - 1) & 1u][kGather - 1]), ((G - 1) >> 1) & 1u, abort_flag);
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[kHeads];
        tmem_ld(tmem_addr(tmem, q4 * 32, Sh::kColO + c * NH + h0), o);
        tmem_wait_ld();
        if (c == 3) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&misc->o_free));   // the next item's products may overwrite the accumulator
        }
        const int dim = 128 * c + 32 * q4 + lane;
        if (p.n_splits == 1) {
          unsigned short* dst = reinterpret_cast<unsigned short*>(p.out + static_cast<long long>(tok) * p.out_st + static_cast<long long>(head0 + h0) * p.out_sh) + dim;
#pragma unroll
          for (int j = 0; j < kHeads; ++j, dst += p.out_sh) {
            if (h0 + j < n_heads) *dst = static_cast<unsigned short>(pack_bf16x2(__uint_as_float(o[j]) * misc->inv_l[h0 + j], 0.0f));
          }
        } else {
          float* dst = p.part_out + ((static_cast<long long>(tok) * p.n_splits + split) * p.h + head0 + h0) * 512 + dim;
#pragma unroll
          for (int j = 0; j < kHeads; ++j) {
            if (h0 + j < n_heads) dst[j * 512] = __uint_as_float(o[j]) * misc->inv_l[h0 + j];
          }
        }
      }
    }
  };
  auto scores = [&]() {
    // ------------------------------------------------------------------ S^T = K . Q^T (whole warp, an elected lane issues)
    // (no proxy fence between a wait and its MMAs, where it would cost 300 cycles: those who wrote the operands have executed it)
    constexpr uint32_t kIdesc = umma_idesc(kFmtBF16, kNT, NH, 0, 0);     // A = K rows (K-major), B = Q (K-major)
    const uint64_t kd0 = smem_desc_sw128(base, 16, 1024), qd0 = smem_desc_sw128(q_s, 16, 1024);
    const uint32_t kd_lo = static_cast<uint32_t>(kd0), kd_hi = static_cast<uint32_t>(kd0 >> 32);
    const uint32_t qd_lo = static_cast<uint32_t>(qd0), qd_hi = static_cast<uint32_t>(qd0 >> 32);
    uint32_t G = 0;
#pragma unroll 1
    for (int t = 0; t < nb; ++t) {
      const int n_tiles = warp_uniform(misc->nt[t]);
      mbar_wait(smem_u32(&misc->q_full), t & 1u, abort_flag);
#pragma unroll 1
      for (int i = 0; i < n_tiles; ++i, ++G) {
        const uint32_t s = G & 1u, ph = (G >> 1) & 1u, t_s = tmem + Sh::kColS + s * NH;
        const uint32_t full = smem_u32(&misc->k_full[0][0]) + s * (kThirds * 8), k_lo = kd_lo + ((s * kSlot) >> 4);
#pragma unroll
        for (int third = 0; third < kThirds; ++third) {
          mbar_wait(full + third * 8, ph, abort_flag);
          __syncwarp();
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int c = 3 * third; c < 3 * third + 3; ++c) {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const uint32_t a_lo = k_lo + ((c * kBlock + k * 32) >> 4), b_lo = qd_lo + ((c * Sh::kQBlock + k * 32) >> 4);
                if (c == 0 && k == 0) umma_f16_ss_lohi<false>(t_s, a_lo, kd_hi, b_lo, qd_hi, kIdesc);
                else umma_f16_ss_lohi<true>(t_s, a_lo, kd_hi, b_lo, qd_hi, kIdesc);
              }
            }
            if (third == kThirds - 1) {
              umma_commit(smem_u32(&misc->s_full[0]) + s * 8);
              if (i == n_tiles - 1) umma_commit(smem_u32(&misc->q_free));
            }
          }
          __syncwarp();
        }
      }
    }
  };
  auto values = [&]() {
    // ------------------------------------------------------------------ O^T += V^T . P^T: a warp of its own, so that the one product's
    // waits do not hold up the other (the tensor pipe takes four MMAs ahead, less than a wait takes)
    constexpr uint32_t kIdesc = umma_idesc(kFmtBF16, 128, NH, 1, 1);     // A = V^T (MN-major), B = P^T (MN-major)
    const uint64_t vd0 = smem_desc_sw128(base, kBlock, 1024);
    const uint32_t vd_lo = static_cast<uint32_t>(vd0), vd_hi = static_cast<uint32_t>(vd0 >> 32);
    uint32_t G = 0;
#pragma unroll 1
    for (int t = 0; t < nb; ++t) {
      const int n_tiles = warp_uniform(misc->nt[t]);
      if (t >= 1) mbar_wait(smem_u32(&misc->o_free), (t - 1) & 1u, abort_flag);
#pragma unroll 1
      for (int i = 0; i < n_tiles; ++i, ++G) {
        const uint32_t s = G & 1u, v_lo = vd_lo + ((s * kSlot) >> 4);
        mbar_wait(smem_u32(&misc->p_full[0]) + s * 8, (G >> 1) & 1u, abort_flag);
        __syncwarp();
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {                    // 16 keys at a time: their rows are free first
#pragma unroll
            for (int c = 0; c < 4; ++c)
              umma_f16_ss(tmem + Sh::kColO + c * NH, (static_cast<uint64_t>(vd_hi) << 32) | (v_lo + ((2 * c * kBlock + k * 2048) >> 4)),
                          (static_cast<uint64_t>(vd_hi) << 32) | (v_lo + ((8 * kBlock + k * 2048) >> 4)), kIdesc, k == 0 ? static_cast<uint32_t>(i) : 1u);
            umma_commit(smem_u32(&misc->k_free[0][0]) + (s * kGather + k) * 8);
          }
        }
        __syncwarp();
      }
    }
  };
  auto load_q = [&](int t) {                               // Q of an item, when the scores of the item before are through; a whole warp
    const int item = first_item + t * n_ctas, next = item + n_ctas, tok_next = token_of(next);
    const uint32_t full = smem_u32(&misc->q_full);
    if (t >= 1) mbar_wait(smem_u32(&misc->q_free), (t - 1) & 1u, abort_flag);
    const bool live = !__any_sync(0xffffffffu, *abort_flag);   // (after a wait that ran out nothing is announced or loaded any more)
    if (lane == 0 && live) mbar_arrive_expect_tx(full, static_cast<uint32_t>(min(p.h, NH) * 128 * kNChunk));   // rows past the last head arrive as zeros
    __syncwarp();
    if (lane < kNChunk && live) {
      tma_load_3d(q_s + lane * Sh::kQBlock, &tm_q, full, lane * 64, (item / p.n_splits) % p.n_groups * NH, token_of(item));
      if (tok_next < p.s_q)
        asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];"
                     ::"l"(&tm_q), "r"(lane * 64), "r"((next / p.n_splits) % p.n_groups * NH), "r"(tok_next) : "memory");
    }
    __syncwarp();
  };
  auto gather = [&]() {
    // ------------------------------------------------------------------ gather: rows 16 prod .. 16 prod + 15 of every tile
    // 36 copies of 16 bytes per lane: lane l copies piece l % 8 of every 64-column block of rows 4 j + l / 8
    const int w = prod & 3, set = prod >> 2;               // set: of the tiles with this remainder modulo kSets
    const __nv_bfloat16* src0 = static_cast<const __nv_bfloat16*>(p.kv) + (lane & 7) * 8;
    uint32_t dst0[2];                                      // of rows 0..3 and 4..7 (the 128-byte swizzle goes with row % 8)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int r = 4 * q + (lane >> 3);
      dst0[q] = base + (16 * w + r) * 128 + (((lane & 7) ^ r) << 4);
    }
    uint32_t G0 = 0;                                       // tiles before the item
#pragma unroll 1
    for (int t = 0; t < nb; ++t) {
      const int tok = token_of(first_item + t * n_ctas);
      const int n_tiles = warp_uniform(misc->nt[t]), row0 = warp_uniform(misc->nt[kBatch + t]) * kNT, n_rows = p.topk - row0;
      const int32_t* idx_row = p.indices + static_cast<long long>(tok) * p.idx_st + row0;
      if (prod == 0) load_q(t);                            // this warp loads Q as well
      const int i0 = static_cast<int>((set - G0) & (Sh::kSets - 1u));
      int j0 = i0 * kNT + 16 * w + (lane & 15);            // (both halves of the warp hold the same 16 rows)
      int nxt = i0 < n_tiles && j0 < n_rows ? idx_row[j0] : -1;
      int row = nxt >= 0 && nxt < p.s_kv ? nxt : -1;
      if (!__all_sync(0xffffffffu, row >= 0)) {
        const int any = first_row(idx_row, misc->last[t] > 0 ? n_rows : 0, p.s_kv, p.n_splits > 1 ? min(static_cast<int>(blockIdx.x * 32 + lane), p.s_kv - 1) : 0);
        if (row < 0) row = any;
      }
#pragma unroll 1
      for (int i = i0; i < n_tiles; i += Sh::kSets) {
        const uint32_t G = G0 + i, s = G & 1u;
        const bool ok = nxt >= 0 && nxt < p.s_kv;
        if (nxt >= p.s_kv || nxt < -1) misc->bad_index = 1;            // reported, never read
        const uint32_t mask = __ballot_sync(0xffffffffu, ok) & 0xffffu;
        if (ok) row = nxt;                                 // a masked entry fetches the row before it again
        j0 += kNT * Sh::kSets;
        nxt = (i + Sh::kSets < n_tiles && j0 < n_rows) ? idx_row[j0] : -1;
        const __nv_bfloat16* src[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) src[q] = src0 + static_cast<long long>(__shfl_sync(0xffffffffu, row, 4 * q + (lane >> 3))) * p.kv_sr;
        if (G >= kSlots) mbar_wait(smem_u32(&misc->k_free[s][w]), ((G >> 1) - 1) & 1u, abort_flag);
        __syncwarp();
        if (lane == 0) misc->valid_mask[s][w] = static_cast<uint16_t>(mask);   // (released by the arrivals below)
#pragma unroll
        for (int j = 0; j < kThirds; ++j) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int c = 3 * j; c < 3 * j + 3; ++c) cp_async16(dst0[q & 1] + s * kSlot + (q >> 1) * 1024 + c * kBlock, src[q] + c * 64);
          }
          cp_async_commit();
        }
#pragma unroll
        for (int j = 0; j < kThirds; ++j) {
          if (j == 0) asm volatile("cp.async.wait_group 2;" ::: "memory");
          else if (j == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
          else asm volatile("cp.async.wait_group 0;" ::: "memory");
          fence_proxy_async_smem();                        // the MMAs read the rows through the async proxy
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&misc->k_full[s][j]));
        }
      }
      G0 += n_tiles;
    }
  };
  auto convert = [&]() {
    // ------------------------------------------------------------------ gather of e4m3 rows: rows 8 w .. 8 w + 7 of every tile, four lanes to a row
    // The 576 bytes of a row are nine pieces of 16 bytes per lane, in registers a tile ahead: the page of the tile after that and the
    // list entry of the next one are on their way too, so that no load is waited for.  A piece becomes 16 values times the scale of
    // their page, rounded to bf16.  Rows that are masked are zeros.
    const int w = prod, r = 8 * w + (lane >> 2), c4 = lane & 3;
    const uint32_t dst0 = base + r * 128 + (((2 * c4) ^ (r & 7)) << 4), dst1 = base + r * 128 + (((2 * c4 + 1) ^ (r & 7)) << 4);
    const uint8_t* cache = static_cast<const uint8_t*>(p.kv) + c4 * 16;
    // where the list entries stand: item, tile within it
    int ct = -1, ci = 0, cn = 0, c_left = 0, c_seq = 0, c_ctx = 0;
    const int32_t* c_idx = nullptr;
    int logical = -1, l_seq = 0, l_ctx = 0;                // of the tile after the next
    int page = 0, in_page = -1;                            // of the next tile; in_page -1 for no row, -2 for an entry of no meaning
    uint4 raw[9];                                          // of this tile
    float scale = 0.0f;
    bool ok = false;
    auto next_entry = [&]() {
      if (ci == cn && ct < nb) {
        ci = cn = 0;
        if (++ct < nb) {
          const int tok = token_of(first_item + ct * n_ctas), row0 = misc->nt[kBatch + ct] * kNT;
          cn = misc->nt[ct];
          c_left = p.topk - row0 - r;
          c_idx = p.indices + static_cast<long long>(tok) * p.idx_st + row0 + r;
          c_seq = (p.tok0 + tok) / p.q_per_seq;
          c_ctx = p.context_lens[c_seq];
        }
      }
      logical = ct < nb && ci * kNT < c_left ? c_idx[ci * kNT] : -1;
      l_seq = c_seq;
      l_ctx = c_ctx;
      ++ci;
    };
    auto next_page = [&]() {
      // (nothing here may look at the page: it is on its way)
      in_page = logical < -1 ? -2 : -1;
      if (logical >= 0 && logical < l_ctx) {
        const int at = logical / p.page_size;
        if (at < p.bt_stride) {
          in_page = logical - at * p.page_size;
          page = p.block_table[l_seq * p.bt_stride + at];
        } else {
          in_page = -2;                                    // a context length longer than the table's row
        }
      }
    };
    auto next_rows = [&]() {
      const long long row = static_cast<long long>(page) * p.page_size + in_page;   // (in 32 bits a corrupt entry may wrap to a valid row)
      ok = in_page >= 0 && page >= 0 && row < p.s_kv;
      if (in_page == -2 || (in_page >= 0 && !ok)) misc->bad_index = 1;      // reported, never read
      scale = ok ? p.kv_scale[page] : 0.0f;
      const uint4* src = reinterpret_cast<const uint4*>(cache + (ok ? row : 0) * p.kv_sr);
#pragma unroll
      for (int k = 0; k < 9; ++k) raw[k] = ok ? src[4 * k] : make_uint4(0u, 0u, 0u, 0u);
    };
    next_entry();
    next_page();
    next_entry();
    next_rows();
    next_page();
    next_entry();
    uint32_t G = 0;
#pragma unroll 1
    for (int t = 0; t < nb; ++t) {
      const int n_tiles = warp_uniform(misc->nt[t]);
      if (w == 0) load_q(t);
#pragma unroll 1
      for (int i = 0; i < n_tiles; ++i, ++G) {
        const uint32_t s = G & 1u;
        const uint32_t rows = __ballot_sync(0xffffffffu, ok);          // bit 4 r: row r
        const uint32_t mask = __ballot_sync(0xffffffffu, lane < 8 && ((rows >> (4 * (lane & 7))) & 1u) != 0u);
        if (G >= kSlots) mbar_wait(smem_u32(&misc->k_free[s][w >> 1]), ((G >> 1) - 1) & 1u, abort_flag);
        __syncwarp();
        if (lane == 0) reinterpret_cast<uint8_t*>(&misc->valid_mask[s][0])[w] = static_cast<uint8_t>(mask);   // (released by the arrivals below)
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          const uint32_t in[4] = {raw[k].x, raw[k].y, raw[k].z, raw[k].w};
          uint32_t o[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(in[j] & 0xffffu), __NV_E4M3);
            const __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(in[j] >> 16), __NV_E4M3);
            const float2 flo = __half22float2(*reinterpret_cast<const __half2*>(&lo)), fhi = __half22float2(*reinterpret_cast<const __half2*>(&hi));
            o[2 * j] = pack_bf16x2(flo.x * scale, flo.y * scale);
            o[2 * j + 1] = pack_bf16x2(fhi.x * scale, fhi.y * scale);
          }
          const uint32_t off = s * kSlot + k * kBlock;
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst0 + off), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst1 + off), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]) : "memory");
        }
        fence_proxy_async_smem();                          // the MMAs read the rows through the async proxy
        __syncwarp();
        if (lane == 0) {
#pragma unroll
          for (int j = 0; j < kThirds; ++j) mbar_arrive(smem_u32(&misc->k_full[s][j]));
        }
        next_rows();
        next_page();
        next_entry();
      }
    }
  };
  if constexpr (kFp8) {
    if (group >= 0) {
      if constexpr (Sh::kSplitRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Sh::kRegsSoftmax));
      softmax();
    } else if (warp < Sh::kConvert0) {
      if constexpr (Sh::kSplitRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Sh::kRegsIssue));
      if (warp == Sh::kIssuer) scores();
      else if (warp == Sh::kValueIssuer) values();
    } else {
      if constexpr (Sh::kSplitRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Sh::kRegsConvert));
      convert();
    }
  } else {
    if (group >= 0) softmax();
    else if (warp == Sh::kIssuer) scores();
    else if (warp == Sh::kValueIssuer) values();
    else if (prod >= 0) gather();
  }

  if (*abort_flag) drain_after_abort();
  tc_fence_before();
  __syncthreads();
  if (!one_each) griddep_launch();               // (behind the barrier: one thread of a CTA speaks for all)
  if (warp == Sh::kIssuer) {
    tc_fence_after();
    tmem_dealloc(tmem, Sh::kCols);
  }
  if (tid == 0 && p.status != nullptr) {
    if (misc->abort_flag) atomicCAS(p.status, 0, FTB_ERR_TIMEOUT);
    else if (misc->bad_index) atomicCAS(p.status, 0, FTB_ERR_BAD_INDEX);
  }
}

template <int NH, bool kFp8>
static int launch_nh(const ftb_sparse_mla_args* a, Params p, cudaStream_t st) {
  using Sh = Shape<NH, kFp8>;
  constexpr int smem = Sh::kOffMisc + static_cast<int>(sizeof(Misc)) + 1024;
  static_assert(smem <= 227 * 1024, "shared memory of an SM");
  auto kern = sparse_mla_few_heads_kernel<NH, kFp8>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(sparse_mla few heads)");
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return check_cuda(e, "SM count");
  // at most kBatch items per CTA and launch; a longer batch of query tokens is a sequence of launches
  const long long items = static_cast<long long>(sms) * kBatch;
  const int per_token = p.n_splits * p.n_groups;
  const long long cap = items / per_token > 0 ? items / per_token : 1;
  float* const part_lse = p.part_lse;
  for (long long t0 = 0; t0 < a->s_q; t0 += cap) {
    p.s_q = static_cast<int>(a->s_q - t0 < cap ? a->s_q - t0 : cap);
    p.tok0 = static_cast<int>(t0);
    p.indices = a->indices + t0 * a->idx_stride_token;
    p.lse = a->lse + t0 * a->lse_stride_token;
    p.out = static_cast<__nv_bfloat16*>(a->out) + t0 * a->out_stride_token;
    if (p.n_splits > 1) {
      const size_t before = static_cast<size_t>(t0) * p.n_splits * a->h;
      p.part_lse = part_lse + before;
      p.part_out = p.part_out + (t0 == 0 ? 0 : static_cast<size_t>(cap) * p.n_splits * a->h * 512);
    }
    CUtensorMap tm_q;
    if (!make_tmap_3d(&tm_q, static_cast<const __nv_bfloat16*>(a->q) + t0 * a->q_stride_token, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, kDqk, static_cast<uint64_t>(a->h),
                      static_cast<uint64_t>(p.s_q), static_cast<uint64_t>(a->q_stride_head), static_cast<uint64_t>(a->q_stride_token), 64,
                      static_cast<uint32_t>(a->h < NH ? a->h : NH))) {
      set_last_error("sparse_mla few heads: cuTensorMapEncodeTiled failed");
      return FTB_ERR_CUDA;
    }
    const long long n = static_cast<long long>(p.s_q) * per_token;
    e = launch_overlapped(kern, static_cast<unsigned>(n < sms ? n : sms), Sh::kThreads, smem, st, 1, tm_q, p);
    if (e != cudaSuccess) return check_cuda(e, "sparse_mla few heads launch");
  }
  return FTB_OK;
}

}  // namespace mla_few

// bf16 form, plain indices, whole tokens or parts of them, more than 64 heads in groups of 64 (argument checks are the caller's: ftb_sparse_mla_fwd).
// n_splits > 1: partial results to part_out / part_lse.  `max_slack`: how far the reference of the weights may lag behind the maximum.
int launch_sparse_mla_few(const ftb_sparse_mla_args* a, int n_splits, float* part_out, float* part_lse, float max_slack, cudaStream_t st) {
  mla_few::Params p;
  memset(&p, 0, sizeof(p));
  p.kv = a->kv;
  p.kv_sr = a->kv_stride_row;
  p.h = a->h; p.s_kv = a->s_kv; p.topk = a->topk;
  p.idx_st = a->idx_stride_token; p.out_st = a->out_stride_token; p.out_sh = a->out_stride_head; p.lse_st = a->lse_stride_token;
  p.scale_log2 = a->sm_scale * 1.4426950408889634f;
  p.lse_base2 = a->lse_base2;
  p.status = a->status;
  p.n_splits = n_splits;
  p.part_out = part_out;
  p.part_lse = part_lse;
  p.max_slack = max_slack;
  p.n_groups = (a->h + 63) / 64;
  if (a->kv_is_fp8) {
    p.kv_scale = a->kv_scale; p.block_table = a->block_table; p.context_lens = a->context_lens;
    p.page_size = a->page_size; p.q_per_seq = a->q_per_seq; p.bt_stride = a->block_table_stride;
    if (a->h <= 16) return mla_few::launch_nh<16, true>(a, p, st);
    if (a->h <= 32) return mla_few::launch_nh<32, true>(a, p, st);
    return mla_few::launch_nh<64, true>(a, p, st);
  }
  if (a->h <= 16) return mla_few::launch_nh<16, false>(a, p, st);
  if (a->h <= 32) return mla_few::launch_nh<32, false>(a, p, st);
  return mla_few::launch_nh<64, false>(a, p, st);
}

}  // namespace ftb
