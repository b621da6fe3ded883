// Top-k sparse MLA forward, persistent role-split CTA pairs (bf16 KV).
//
// One pair of CTAs (a cluster of 2) walks through query tokens pair, pair + pairs, ...  CTA 0 computes
// S = Q.K^T (Q in tensor memory, K column blocks gathered into shared memory by cp.async) and the
// softmax; P travels to CTA 1 by asynchronous stores over distributed shared memory; CTA 1 accumulates O += P.V in
// tensor memory and writes the output.  Every barrier keeps counting across tokens.
//
// The slots of CTA 0.  Nine slots of [128 rows x 128 B], one per 64-column block: per token the blocks of the token's query
// rows pass through (fetched by a TMA tile load and moved on to tensor memory by the issuer itself with tcgen05.cp,
// which runs in order with its MMAs), then a K block per tile of 128 selected rows, multiplied by four MMAs; the commit behind a
// block frees its slot.  The ninth (rope) block of Q stays in a buffer of its own in shared memory and is multiplied from
// there: that leaves 256 columns of tensor memory for two score buffers, so that the issuer starts the next tile while the
// softmax fetches this one (the hand-over of a single buffer cost 550 cycles per tile).  The next token's Q blocks follow the
// last tile's K blocks into the slots, and the token after it is asked into L2.
//
// Gather warps.  One warp per column block of K (nine) and per half slab of V (eight) copies rows with 16-byte cp.async:
// the lanes keep the tile's row numbers and pass them round with shuffles.  148 SMs fetch random rows at 70 bytes
// per clock and SM this way, as fast as TMA row gathers do (both are bound by L2), but a gather4 from divergent lanes
// occupies its scheduler for about 20 cycles and slowed the softmax and the issuer beside it.  The K warps sit on the
// three schedulers that the MMA issuer is not on.  cp.async writes through the generic proxy, so the issuers fence
// (fence.proxy.async) between the barrier wait and their MMAs.
//
// What bounds it: instruction supply, not memory or the tensor pipe.  Seventeen warps run ten different roles, and a
// warp that has a scheduler's instruction cache to share runs 5 or more cycles per instruction; fully unrolled role loops with
// a private copy of the wait loop each (95 KB of code) kept a third of all warps stalled on instruction fetch.  So every
// role but the MMA issue has one rolled loop, the softmax has one path (masked entries become -inf once) with two-wide
// fp32 instructions, loop counts are warp-uniform, and the issuer has constant addresses and waits for three blocks at once.
// Warps whose 32 head rows hold no head take no part.  One launch alone, 740 tokens, 128 heads, topk 2048: 832 -> 1065
// TFLOP/s.  Back to back, in turn on one box: 4096 causal tokens 2244 -> 1944 us, with the weights sent straight from registers 1881.
//
// Few tokens.  A launch may cut the top-k list of every token in parts; an item of work is then a part of a token, its result
// leaves as fp32 (32 columns per TMA store instead of 64) with a base-2 LSE, and a second kernel merges the parts.  One token
// of topk 2048: 49 us whole, 23 us in 16 parts.  (Stores straight from registers, 16 bytes per lane and row, took 6 us more:
// half sectors.)
//
// Softmax: two threads per head row; the running maximum moves only when it grows by more than 2^8, so that
// the accumulator in CTA 1 is rarely rescaled.  P (bf16) and the rescale factors go from registers to
// CTA 1 with st.async, which count on CTA 1's barrier; the arrival that announces them
// carries no release (the data travels with the stores), which keeps the softmax warps from stalling.
//
// The number of tiles of an item (last non-negative index, rounded up to 128 rows, at least one) is
// found for 64 items at a time by all warps of a CTA, with CTA barriers between.
//
// Warps (640 threads per CTA): CTA 0: 0-7 softmax, 8 MMA issuer, nine ring producers (the warps 9-19 whose id is not 0
// modulo 4).  CTA 1: 0-3 correction, 4 relay, 8 MMA issuer, 9-16 V producers, 0-7 and 9-16 epilogue.
// Every wait is bounded; a wait that runs out sets the abort flag, after which every later wait returns at
// once and the status word reports a timeout.
#include "launch.cuh"
#include "sm100.cuh"
#include "tmap.cuh"

namespace ftb {

void set_last_error(const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

namespace mla_ring {

constexpr int kDqk = 576;
constexpr int kNChunk = 9;
constexpr int kNT = 128;                       // gathered rows per tile
constexpr int kQBlock = 128 * 128;             // 16384: [128 heads x 128 B]
constexpr int kNQ = 8;                         // 64-column blocks of Q that live in tensor memory; the ninth (rope) stays in shared memory
constexpr int kNK = kNChunk;                   // slots of CTA 0: column block c of Q or of a tile's K lives in slot c
constexpr int kKSlot = kNT * 128;              // 16384: [128 rows x 128 B]
constexpr int kNV = 4;                         // V ring slots: one whole tile, slab s in slot s
constexpr int kVSlabRows = 32;
constexpr int kVBlock = kVSlabRows * 128;      // 4096: one 64-column block of a slab
constexpr int kVSlab = 8 * kVBlock;            // 32768
// 32768: P [128 heads x 128 rows] bf16, without a swizzle: 8 of the rows (16 bytes) of all heads are 2048 bytes in a row, so that what a
// softmax warp sends with one instruction lies in a row
constexpr int kPBuf = 2 * kQBlock;
constexpr int kPChunk = 128 * 16;
constexpr int kBatch = 64;                     // tokens whose tile counts are found in one go
// CTA 0 layout: nine slots | rope block of Q | misc.
// CTA 1 layout: V ring | P x 2 | misc; between tokens the P buffer of the last tile stages O.
constexpr int kOff0K = 0;
constexpr int kOff0Q8 = kOff0K + kNK * kKSlot;             // 147456
constexpr int kOff0Misc = kOff0Q8 + kQBlock;               // 163840
constexpr int kOff1P = kNV * kVSlab;                       // 131072
constexpr int kOff1Misc = kOff1P + 2 * kPBuf;              // 196608
constexpr int kSmemBytes = kOff1Misc + 4096 + 1024;        // the larger of the two + misc + alignment slack
constexpr int kThreads = 640;                  // 20 warps
constexpr int kWarps = kThreads / 32;
constexpr uint32_t kColQ = 0;                  // TMEM columns of CTA 0: Q (256), then two score buffers of 128
constexpr uint32_t kColS = 256;

struct Params {
  const __nv_bfloat16* kv;
  long long kv_sr;
  const int32_t* indices;
  float* lse;
  int s_q, h, s_kv, topk;
  long long idx_st, lse_st;
  float scale_log2;
  int lse_base2;
  int* status;
  // the top-k list of a token in n_splits parts, an item of work each; their results go to fp32 partials that are merged later
  int n_splits;
  float* part_lse;     // [s_q, n_splits, h], base 2
  float max_slack;     // how far (log2) the running maximum may lag behind
};

struct Misc0 {   // CTA 0
  unsigned long long k_full[kNK];   // one arrival per gather thread (when its copies have landed; the tile load of a Q entry counts on one of them);
                                    // slot 0 one more, which releases the tile's validity mask
  unsigned long long k_free[kNK];   // tcgen05.commit behind the entry's MMAs or its copy to tensor memory
  unsigned long long s_full[2];     // tcgen05.commit
  unsigned long long s_free[2];     // softmax warps with heads (8 when h > 96)
  unsigned long long q8_full;       // the token's rope block of Q has landed
  unsigned long long q8_free;       // tcgen05.commit behind the token's last tile
  unsigned long long p_free[2];     // relay warp of CTA 1 (remote arrival)
  unsigned long long epi_done[2];   // CTA 1 (remote arrival): the epilogue of token t (t % 2) is over
  uint32_t tmem_base;
  int abort_flag;
  int bad_index;
  int pad;
  alignas(16) uint32_t valid_mask[8][4];  // per tile (mod 8): 128 validity bits
  unsigned short nt[2 * kBatch];    // per item of the current batch: number of tiles, first tile
  int last[kBatch];                 // entries of its list up to the last that is not negative
  float xchg[2][256];               // row maximum / row sum exchange between the two threads of a head row
};
struct Misc1 {   // CTA 1
  unsigned long long v_full[kNV];   // one arrival per gather thread, when its copies have landed
  unsigned long long v_free[kNV];   // tcgen05.commit
  unsigned long long p_full[2];     // softmax warps with heads of CTA 0 (remote arrivals, each announcing what it sends: 4 KB of P, 256 B of factors)
  unsigned long long corr_done[2];  // correction warps with heads
  unsigned long long half_done[4];  // per correction warp: tcgen05.commit behind the first half of a tile whose second half moves one of its maxima
  unsigned long long half_corr[4];  // the warp: its rows of the accumulator are ready for that second half
  unsigned long long pv_done[2];    // tcgen05.commit
  unsigned long long fin[2];        // softmax warps with heads of CTA 0: 1/l of token t (t % 2) is in place
  unsigned long long o_free;        // 16 epilogue warps: the accumulator has been read
  unsigned long long stg_free[8];   // epilogue warp w < 8: its staging piece is free for warp 9 + w
  unsigned long long epi_cnt;       // 16 epilogue warps: the output of the token has left the staging area
  uint32_t tmem_base;
  int abort_flag;
  uint32_t late[2];                 // a byte per correction warp: does the second half of the tile move one of its maxima?
  unsigned short nt[2 * kBatch];
  int last[kBatch];
  alignas(16) float2 alpha[2][128];  // rescale factors of the halves of a tile (two buffers), sent by CTA 0
  float inv_l[2][128];              // final 1/l of token t (t % 2)
};
static_assert(sizeof(Misc0) <= 4096 && sizeof(Misc1) <= 4096, "misc area");
static_assert(kOff0Misc + 4096 + 1024 <= kSmemBytes, "CTA 0 layout fits");
static_assert(kNV == kNT / kVSlabRows, "V ring slot index = slab index");

__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// remote arrival that also announces `bytes` of bulk-copy traffic to the barrier of another CTA of the cluster.
// No release: what the waiter reads arrives with the announced copies themselves.  (With release semantics at
// cluster scope this arrival stalled the softmax warps for about 2000 cycles per tile.)
__device__ __forceinline__ void mbar_arrive_expect_tx_cluster(uint32_t cluster_addr, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_addr), "r"(bytes) : "memory");
}
// remote arrival that only hands a buffer back (nothing the waiter reads depends on it)
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// shared memory -> tensor memory, 128 rows x 32 bytes (one K = 16 step of an A operand), asynchronous and in order
// with the MMAs of the issuing thread; the source is described like an MMA operand
__device__ __forceinline__ void tmem_cp_128x256b(uint32_t taddr, uint32_t desc_lo, uint32_t desc_hi) {
  asm volatile(
      "{\n\t.reg .b64 sd;\n\t"
      "mov.b64 sd, {%1, %2};\n\t"
      "tcgen05.cp.cta_group::1.128x256b [%0], sd;\n\t}"
      ::"r"(taddr), "r"(desc_lo), "r"(desc_hi)
      : "memory");
}
// two fp32 lanes per instruction (ffma2: sm100.cuh)
__device__ __forceinline__ float2 fmul2(float2 a, float b) {
  float2 r;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\t"
      "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b));
  return r;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
// stores to the shared memory of another CTA that count their bytes on a barrier there
__device__ __forceinline__ void st_async_v4(uint32_t dst_cluster, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t bar_cluster) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(dst_cluster), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar_cluster) : "memory");
}
__device__ __forceinline__ void st_async_v2(uint32_t dst_cluster, uint32_t a, uint32_t b, uint32_t bar_cluster) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];"
               ::"r"(dst_cluster), "r"(a), "r"(b), "r"(bar_cluster) : "memory");
}
// mbar_wait on a barrier whose bytes come from the other CTA of the cluster
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  const uint32_t t0 = static_cast<uint32_t>(clock());
#pragma unroll 1
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(kWaitSleepNs) : "memory");
    if (ok != 0u) return true;
    if (*abort_flag) return false;
    if (static_cast<uint32_t>(clock()) - t0 > kWaitLimitCycles) {
      *abort_flag = 1;
      return false;
    }
  }
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// waits until the bulk stores of this thread have read their shared-memory source (the global writes
// themselves complete before the grid does)
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Masked entries (-1) fetch a row all the same, which is multiplied by zero: the one that the lane fetched for the tile before, or in
// the first tile another one of the token's (this function, the rare path: the first row that the list names; `none` if
// it names none, row 0 for a token and any rows for a part, whose result the merge drops).  With row 0 for all of them, as it used to be,
// every SM fetched the same 1152 bytes (4096 tokens of topk 65 took longer than of topk 128, 761 us against 329; now 335),
// and a row 0 that holds no numbers spoiled tokens that never selected it.  Not inline: the roles share an instruction cache.
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

__global__ void __launch_bounds__(kThreads, 1)
sparse_mla_ring_kernel(const __grid_constant__ CUtensorMap tm_q,
                         const __grid_constant__ CUtensorMap tm_o, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw_addr);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = warp_uniform(tid >> 5);
  const int cta = static_cast<int>(cluster_ctarank());
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  Misc0* m0 = reinterpret_cast<Misc0*>(sm + kOff0Misc);
  Misc1* m1 = reinterpret_cast<Misc1*>(sm + kOff1Misc);
  // abort_flag / tmem_base / nt sit at different offsets in the two layouts: pick this CTA's
  volatile int* abort_flag = cta == 0 ? &m0->abort_flag : &m1->abort_flag;
  uint32_t* tmem_base_p = cta == 0 ? &m0->tmem_base : &m1->tmem_base;
  unsigned short* nt = cta == 0 ? m0->nt : m1->nt;
  int* last = cta == 0 ? m0->last : m1->last;

  // 32-row quarters of the 128 head rows that hold heads: the softmax and correction warps of the others have nothing to do
  const int row_warps = (p.h + 31) >> 5;
  const bool has_rows = (warp & 3) < row_warps;

  const bool one_each = p.s_q * p.n_splits <= n_pairs;         // items
  if (one_each) griddep_launch();
  if (tid == 0) {
    if (cta == 0) {
      m0->bad_index = 0;
      for (int i = 0; i < kNK; ++i) { mbar_init(smem_u32(&m0->k_full[i]), i == 0 ? 33 : 32); mbar_init(smem_u32(&m0->k_free[i]), 1); }
      for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&m0->s_full[i]), 1); mbar_init(smem_u32(&m0->s_free[i]), 2 * row_warps); }
      mbar_init(smem_u32(&m0->q8_full), 1);
      mbar_init(smem_u32(&m0->q8_free), 1);
      for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&m0->p_free[i]), 1); mbar_init(smem_u32(&m0->epi_done[i]), 1); }
    } else {
      for (int i = 0; i < kNV; ++i) { mbar_init(smem_u32(&m1->v_full[i]), 64); mbar_init(smem_u32(&m1->v_free[i]), 1); }
      for (int i = 0; i < 2; ++i) {
        mbar_init(smem_u32(&m1->p_full[i]), 2 * row_warps);
        mbar_init(smem_u32(&m1->corr_done[i]), row_warps);
        m1->late[i] = 0;
        mbar_init(smem_u32(&m1->pv_done[i]), 1);
        mbar_init(smem_u32(&m1->fin[i]), 2 * row_warps);
      }
      mbar_init(smem_u32(&m1->o_free), 16);
      for (int i = 0; i < 4; ++i) { mbar_init(smem_u32(&m1->half_done[i]), 1); mbar_init(smem_u32(&m1->half_corr[i]), 1); }
      for (int i = 0; i < 8; ++i) mbar_init(smem_u32(&m1->stg_free[i]), 1);
      mbar_init(smem_u32(&m1->epi_cnt), 16);
    }
    fence_mbar_init();
  }
  griddep_wait();
  if (tid == 0) *abort_flag = (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
  __syncthreads();
  // An earlier launch on this status word failed: leave at once.  The two CTAs of a pair read the word at
  // different moments (another pair of this launch may report in between), so CTA 1 takes CTA 0's reading:
  // a CTA that went on alone would signal barriers in the shared memory of a partner that has left.
  if (p.status != nullptr) {
    cluster_sync_all();
    uint32_t leave;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(leave) : "r"(mapa_shared(smem_u32(&m0->abort_flag), 0)) : "memory");
    if (leave != 0u) {
      cluster_sync_all();      // CTA 0 stays until its partner has read the flag
      return;
    }
    __syncthreads();
    if (tid == 0) *abort_flag = 0;
  }
  if (cta == 0 && p.h < 128) {
    // a Q entry only writes h rows of its slot; the rows below feed head rows that are never stored, but they
    // should hold numbers
    for (int x = tid; x < (kNK * kKSlot + kQBlock) / 16; x += kThreads)
      asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(base + x * 16), "r"(0) : "memory");
    fence_proxy_async_smem();
  }
  if (warp == 8) {
    tmem_alloc(smem_u32(tmem_base_p), 512u);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = *tmem_base_p;
  // items (tokens, or parts of tokens) of this pair: pair, pair + n_pairs, ...  (the host launches no more pairs than items)
  auto token_of = [&](int item) { return p.n_splits == 1 ? item : item / p.n_splits; };
  const int my_tokens = (p.s_q * p.n_splits - pair + n_pairs - 1) / n_pairs;
  uint32_t n_late = 0;   // CTA 1: tiles so far whose second half moved a maximum, of a correction warp (the issuer: a bit of it per warp)
  uint32_t gt = 0;   // tiles processed before the current token: every role counts the same way
  // CTA 0: the nine gather warps, one per column block: the warps 9-19 whose id is not 0 modulo 4, in order (they share no
  // scheduler with the MMA issuer, warp 8)
  const int prod = (warp >= 9 && (warp & 3) != 0) ? (warp - 9) - ((warp - 8) >> 2) : -1;
  for (int batch0 = 0; batch0 < my_tokens; batch0 += kBatch) {
    const int nb = min(kBatch, my_tokens - batch0);
    // ------------------------------------------------------------------ tiles per token of this batch
    // the warps share the lists out in pieces of 512 entries, all loads of a piece in flight (one token's list of 2048 entries, read
    // by one warp 32 at a time, took 10 us)
    for (int t = tid; t < nb; t += kThreads) last[t] = 0;
    __syncthreads();
    const int pieces = (p.topk + 511) >> 9;
#pragma unroll 1
    for (int x = warp; x < nb * pieces; x += kWarps) {
      const int t = x / pieces, j0 = (x - t * pieces) * 512 + lane;
      const int32_t* idx_row = p.indices + static_cast<long long>(token_of(pair + (batch0 + t) * n_pairs)) * p.idx_st;
      int v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = j0 + 32 * j < p.topk ? idx_row[j0 + 32 * j] : -1;
      int local = 0;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (v[j] >= 0) local = j0 + 32 * j + 1;
      local = __reduce_max_sync(0xffffffffu, local);
      if (lane == 0 && local > 0) atomicMax(&last[t], local);
    }
    __syncthreads();
    // at least one tile (entirely masked if the item selects nothing): every stage of the pipeline
    // then runs once per item and the hand-overs between items need no special case
    for (int t = tid; t < nb; t += kThreads) {
      const int item = pair + (batch0 + t) * n_pairs;
      const int tiles = min(65535, max(1, (last[t] + kNT - 1) / kNT));
      const int part = (tiles + p.n_splits - 1) / p.n_splits;
      int first = (item - token_of(item) * p.n_splits) * part;
      if (first >= tiles) first = 65535;                     // nothing left for this part: a tile past the list
      nt[t] = static_cast<unsigned short>(max(1, min(part, tiles - first)));
      nt[kBatch + t] = static_cast<unsigned short>(first);
    }
    __syncthreads();

    if (cta == 0) {
      // ===================================================================== CTA 0: scores
      const uint32_t k_s = base + kOff0K;
      if (warp < 8 && has_rows) {
        // -------------------------------------------------------------- softmax (two threads per head row)
        // thread tid: head row = tid % 128 (TMEM lane), columns 64*(tid/128) .. +63 of the tile
        const int rowi = tid & 127;
        const int ch = tid >> 7;
        const uint32_t p_remote = mapa_shared(base + kOff1P, 1);
        const uint32_t alpha_remote = mapa_shared(smem_u32(&m1->alpha[0][0]), 1);
        const uint32_t invl_remote = mapa_shared(smem_u32(&m1->inv_l[0][0]), 1);
        const uint32_t p_full_r = mapa_shared(smem_u32(&m1->p_full[0]), 1);
        const uint32_t fin_r = mapa_shared(smem_u32(&m1->fin[0]), 1);
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32);
        for (int t = 0; t < nb; ++t) {
          const int ti = batch0 + t;
          const int item = pair + ti * n_pairs;
          const int n_tiles = warp_uniform(nt[t]);
          // 1/l and the `fin` barrier of parity ti % 2 were last used by token ti - 2: its epilogue is over
          if (ti >= 2) mbar_wait(smem_u32(&m0->epi_done[ti & 1]), ((ti >> 1) - 1) & 1u, abort_flag);
          float m_run = -INFINITY;
          float2 l01 = make_float2(0.0f, 0.0f), l23 = l01;   // sums of the weights, by groups of 16 columns of this thread's 64
          for (int i = 0; i < n_tiles; ++i) {
            const uint32_t G = gt + i;
            const int b = G & 1;
            mbar_wait(smem_u32(&m0->s_full[b]), (G >> 1) & 1u, abort_flag);
            tc_fence_after();
            const uint4 vm4 = *reinterpret_cast<const uint4*>(&m0->valid_mask[G & 7][0]);
            const uint32_t vmA = ch == 0 ? vm4.x : vm4.z, vmB = ch == 0 ? vm4.y : vm4.w;
            const bool all_valid = (vm4.x & vm4.y & vm4.z & vm4.w) == 0xffffffffu;      // uniform over the CTA
            // copy this thread's 64 scores to registers and hand the S buffer back at once
            uint32_t sr[2][32];
            const uint32_t t_s = tmem_addr(tmem, lane_base, kColS + b * kNT + ch * 64);
            tmem_ld32(t_s, sr[0]);
            tmem_ld32(t_s + 32, sr[1]);
            tmem_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&m0->s_free[b]));
            if (!all_valid) {
              // masked entries of the tile: no weight (2^-inf = 0) and no say in the maximum
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                if (!((vmA >> j) & 1u)) sr[0][j] = 0xff800000u;
                if (!((vmB >> j) & 1u)) sr[1][j] = 0xff800000u;
              }
            }
            float mx = -INFINITY;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
#pragma unroll
              for (int j = 0; j < 32; j += 2) mx = fmaxf(mx, fmaxf(__uint_as_float(sr[q][j]), __uint_as_float(sr[q][j + 1])));
            }
            // Lazy maximum: with a slack of 8 the reference only moves when it grows by more than 2^8, so that the
            // accumulator in the other CTA is rarely rescaled (P stays below 256).  Without slack it follows the true
            // maximum, and every tile sets it as a whole: the largest weight is then 1, which bf16 holds exactly.  (The half-way stop below for a maximum
            // that moves in both halves would come with most tiles: 100 tokens of 128 heads, topk 2048 in two parts, 133 us instead of 98.)
            // With slack the first tile sets it as a whole; later the two halves of a tile (64 rows: the tile of the kernel for few heads) move
            // it one after the other, and the sums below add in that kernel's order: the bits of a whole token's head do not depend on
            // how many heads the call has.
            auto move_to = [&](float top) {
              const float m_cand = fmaxf(m_run, top * p.scale_log2);
              float a = 1.0f;
              if (m_cand > m_run + p.max_slack || m_run == -INFINITY) {
                a = (m_run == -INFINITY) ? 0.0f : fast_exp2(m_run - m_cand);
                m_run = m_cand;
              }
              return a;
            };
            float alpha_a = 1.0f, alpha_b = 1.0f, m_mine = m_run;
            // (the two warps of 32 rows agree; only then do they exchange their maxima)
            const bool moves = named_bar_any(2 + (warp & 3), 64, mx * p.scale_log2 > m_run + p.max_slack || m_run == -INFINITY);
            if (moves) {
              m0->xchg[b][tid] = mx;
              named_bar_sync(2 + (warp & 3), 64);
              const float other = m0->xchg[b][tid ^ 128];
              if (p.max_slack == 0.0f) mx = fmaxf(mx, other);
              alpha_a = move_to(i == 0 ? fmaxf(mx, other) : p.max_slack == 0.0f || ch == 0 ? mx : other);
              m_mine = m_run;
              if (i != 0 && p.max_slack != 0.0f) alpha_b = move_to(ch == 0 ? other : mx);
              if (ch != 0) m_mine = m_run;
              l01 = fmul2(l01, alpha_a);
              l23 = fmul2(l23, alpha_a);
              if (ch != 0) {
                l01 = fmul2(l01, alpha_b);
                l23 = fmul2(l23, alpha_b);
              }
            }
            const float m_use = (m_mine == -INFINITY) ? 0.0f : m_mine;
            float sum16[4];
            const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), neg_m2 = make_float2(-m_use, -m_use);
            uint32_t pk[2][16];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
#pragma unroll
              for (int g = 0; g < 2; ++g) {
                float2 e[8];
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                  const float2 x = ffma2(make_float2(__uint_as_float(sr[q][16 * g + j]), __uint_as_float(sr[q][16 * g + j + 1])), scale2, neg_m2);
                  e[j >> 1] = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                  pk[q][8 * g + (j >> 1)] = pack_bf16x2(e[j >> 1].x, e[j >> 1].y);
                }
                // columns j and j + 8, then + 4, + 2, + 1
#pragma unroll
                for (int j = 0; j < 4; ++j) e[j] = fadd2(e[j], e[j + 4]);
                e[0] = fadd2(e[0], e[2]);
                e[1] = fadd2(e[1], e[3]);
                e[0] = fadd2(e[0], e[1]);
                sum16[2 * q + g] = e[0].x + e[0].y;
              }
            }
            // P buffer b of CTA 1 was last read by P.V of tile G-2
            if (G >= 2) mbar_wait(smem_u32(&m0->p_free[b]), ((G - 2) >> 1) & 1u, abort_flag);
            // The weights go there straight from the registers, 512 bytes in a row per instruction, and count themselves on p_full (the
            // arrival that announces them carries no release).  A staging area and bulk copies cost every tile a proxy fence of 400 to 1400
            // cycles in the softmax, which is the longest stage; 16-byte stores into swizzled rows cost more than that.
            if (lane == 0) mbar_arrive_expect_tx_cluster(p_full_r + b * 8, 32 * 128 + (ch == 0 ? 256 : 0));
            __syncwarp();
            const uint32_t p_row = p_remote + b * kPBuf + ch * 8 * kPChunk + rowi * 16;
#pragma unroll
            for (int c = 0; c < 8; ++c)
              st_async_v4(p_row + c * kPChunk, pk[c >> 2][4 * (c & 3)], pk[c >> 2][4 * (c & 3) + 1], pk[c >> 2][4 * (c & 3) + 2], pk[c >> 2][4 * (c & 3) + 3], p_full_r + b * 8);
            if (ch == 0) st_async_v2(alpha_remote + (b * 128 + rowi) * 8, __float_as_uint(alpha_a), __float_as_uint(alpha_b), p_full_r + b * 8);
            l01 = fadd2(l01, make_float2(sum16[0], sum16[1]));
            l23 = fadd2(l23, make_float2(sum16[2], sum16[3]));
            if (ch == 0 && moves) {
              l01 = fmul2(l01, alpha_b);
              l23 = fmul2(l23, alpha_b);
            }
          }
          gt += n_tiles;
          // end of the token: combine the two halves of every row sum; 1/l goes to CTA 1, LSE is written here
          const float l_run = (l01.x + l01.y) + (l23.x + l23.y);
          named_bar_sync(2 + (warp & 3), 64);
          m0->xchg[0][tid] = l_run;
          named_bar_sync(2 + (warp & 3), 64);
          const float l_tot = l_run + m0->xchg[0][tid ^ 128];
          named_bar_sync(2 + (warp & 3), 64);   // xchg[0] may be written again by the first tile of the next token
          if (ch == 0) {
            const float inv_l = (l_tot > 0.0f) ? 1.0f / l_tot : 0.0f;
            st_cluster_f32(invl_remote + ((ti & 1) * 128 + rowi) * 4, inv_l);
            if (rowi < p.h) {
              const float l2 = l_tot > 0.0f ? m_run + log2f(l_tot) : -INFINITY;
              if (p.n_splits == 1) p.lse[static_cast<long long>(item) * p.lse_st + rowi] = (p.lse_base2 || l_tot <= 0.0f) ? l2 : l2 * 0.6931471805599453f;
              else p.part_lse[static_cast<long long>(item) * p.h + rowi] = l2;
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(fin_r + (ti & 1) * 8);
        }
      } else if (warp == 8) {
        // -------------------------------------------------------------- ring consumer: Q copies and Q.K^T
        // The whole warp runs the loop and waits; an elected lane (always the same one, so that its commits
        // cover its MMAs and copies) issues.  Per token: eight Q blocks, each moved to its 32 columns of tensor memory by
        // four tcgen05.cp (they run in order behind the MMAs issued before them, so the previous token's last tile
        // has read the block by then), then nine K blocks per tile with four MMAs each.  The commit behind a block
        // frees its slot.  The tensor pipe takes four MMAs ahead of the one it executes (256 cycles), while a wait and its
        // fences take a lone warp about 300: so the warp waits for three blocks at once, lane by lane, and issues
        // twelve MMAs behind one wait.  A block has a slot of its own, so every address of a tile is a constant off the base:
        // with a ring of ten slots the address arithmetic alone made an MMA cost 82 cycles of issue, against 64 of execution.
        {
          constexpr uint32_t kIdesc = umma_idesc(kFmtBF16, 128, kNT, 0, 0);
          const uint64_t bd0 = smem_desc_sw128(k_s, 16, 1024);
          const uint64_t qd0 = smem_desc_sw128(base + kOff0Q8, 16, 1024);
          const uint32_t bd_lo = static_cast<uint32_t>(bd0), bd_hi = static_cast<uint32_t>(bd0 >> 32);
          const uint32_t qd_lo = static_cast<uint32_t>(qd0), qd_hi = static_cast<uint32_t>(qd0 >> 32);
          const uint32_t t_q = tmem + kColQ;
          const uint32_t k_full0 = smem_u32(&m0->k_full[0]), k_free0 = smem_u32(&m0->k_free[0]);
          const uint32_t wait_at = k_full0 + (lane % 3) * 8;
          // uses of a slot before token ti and tile G: slots 0-7 G tiles and ti blocks of Q, slot 8 G tiles
#pragma unroll 1
          for (int t = 0; t < nb; ++t) {
            const int ti = batch0 + t;
            const int n_tiles = warp_uniform(nt[t]);
            mbar_wait(k_full0 + (lane & 7) * 8, (gt + ti) & 1u, abort_flag);
            __syncwarp();
            fence_proxy_async_smem();
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int cc = 0; cc < kNQ; ++cc) {
#pragma unroll
                for (int k = 0; k < 4; ++k) tmem_cp_128x256b(t_q + cc * 32 + k * 8, bd_lo + ((cc * kKSlot + k * 32) >> 4), bd_hi);
                umma_commit(k_free0 + cc * 8);
              }
            }
            __syncwarp();
#pragma unroll 1
            for (int i = 0; i < n_tiles; ++i) {
              const uint32_t G = gt + i;
              const uint32_t b = G & 1u, par = (G + ti + 1) & 1u;
              const uint32_t t_s = tmem + kColS + b * kNT;
              // score buffer b: the softmax of tile G-2 has copied it to registers
              if (G >= 2) mbar_wait(smem_u32(&m0->s_free[b]), ((G >> 1) & 1u) ^ 1u, abort_flag);
#pragma unroll
              for (int c0 = 0; c0 < kNChunk; c0 += 3) {
                if (c0 == 6 && i == 0) mbar_wait(smem_u32(&m0->q8_full), ti & 1u, abort_flag);
                mbar_wait(wait_at + c0 * 8, c0 == 6 && lane % 3 == 2 ? b : par, abort_flag);
                __syncwarp();
                fence_proxy_async_smem();                    // the rows were written by cp.async (generic proxy)
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                  for (int cc = c0; cc < c0 + 3; ++cc) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                      const uint32_t lo = bd_lo + ((cc * kKSlot + k * 32) >> 4);
                      if (cc == kNQ) umma_f16_ss_lohi<true>(t_s, qd_lo + ((k * 32) >> 4), qd_hi, lo, bd_hi, kIdesc);
                      else if (cc == 0 && k == 0) umma_f16_ts_lohi<false>(t_s, t_q, lo, bd_hi, kIdesc);
                      else umma_f16_ts_lohi<true>(t_s, t_q + cc * 32 + k * 8, lo, bd_hi, kIdesc);
                    }
                    umma_commit(k_free0 + cc * 8);
                  }
                  if (c0 == 6) {
                    umma_commit(smem_u32(&m0->s_full[b]));
                    if (i == n_tiles - 1) umma_commit(smem_u32(&m0->q8_free));
                  }
                }
                __syncwarp();
              }
            }
            gt += n_tiles;
          }
        }
      } else if (prod >= 0) {
        // -------------------------------------------------------------- ring producers
        // Producer c supplies block c of every token's Q (a TMA tile load) and of every tile (32 copies of 16 bytes per lane:
        // lane l copies piece l % 8 of rows 4 q + l / 8) into slot c.  The slot is free once the commit behind its last use has
        // arrived (k_free); the parity wait is exact because that use is at most one phase away.  Block c of the token
        // after this one is asked into L2 when this token's is loaded.
        const int c = prod;
        const uint32_t k_full = smem_u32(&m0->k_full[c]), k_free = smem_u32(&m0->k_free[c]);
        const __nv_bfloat16* src0 = p.kv + c * 64 + (lane & 7) * 8;
        uint32_t dst0[2];                                    // rows 8 m + 0..3 and 8 m + 4..7 (the 128-byte swizzle goes with row % 8)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int r = 4 * q + (lane >> 3);
          dst0[q] = k_s + c * kKSlot + r * 128 + (((lane & 7) ^ r) << 4);
        }
#pragma unroll 1
        for (int t = 0; t < nb; ++t) {
          const int ti = batch0 + t;
          const int tok = token_of(pair + ti * n_pairs), tok_next = token_of(pair + (ti + 1) * n_pairs);
          const int n_tiles = warp_uniform(nt[t]), row0 = warp_uniform(nt[kBatch + t]) * kNT, n_rows = p.topk - row0;
          const int32_t* idx_row = p.indices + static_cast<long long>(tok) * p.idx_st + row0;
          int nxt[4];                                        // rows lane, lane + 32, lane + 64, lane + 96 of the next tile
#pragma unroll
          for (int j = 0; j < 4; ++j) nxt[j] = (32 * j + lane < n_rows) ? idx_row[32 * j + lane] : -1;
          // ---- the Q entry (block 8 has a buffer of its own)
          {
            uint32_t full, dst;
            if (c < kNQ) {
              if (gt + ti >= 1) mbar_wait(k_free, (gt + ti - 1) & 1u, abort_flag);
              full = k_full;
              dst = k_s + c * kKSlot;
            } else {
              if (ti >= 1) mbar_wait(smem_u32(&m0->q8_free), (ti - 1) & 1u, abort_flag);
              full = smem_u32(&m0->q8_full);
              dst = base + kOff0Q8;
            }
            if (lane == 0) {
              mbar_arrive_expect_tx(full, static_cast<uint32_t>(p.h * 128));
              tma_load_3d(dst, &tm_q, full, c * 64, 0, tok);
              if (tok_next < p.s_q)
                asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];"
                             ::"l"(&tm_q), "r"(c * 64), "r"(0), "r"(tok_next) : "memory");
            } else if (c < kNQ) {
              mbar_arrive(full);
              if (c == 0 && lane == 1) mbar_arrive(full);
            }
            __syncwarp();
          }
          // ---- the K entries
          int row[4], own = -1;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            row[j] = nxt[j] >= 0 && nxt[j] < p.s_kv ? nxt[j] : -1;
            own = max(own, row[j]);
          }
          if (!__all_sync(0xffffffffu, (row[0] | row[1] | row[2] | row[3]) >= 0)) {
            const int any = first_row(idx_row, last[t] > 0 ? n_rows : 0, p.s_kv, p.n_splits > 1 ? min(static_cast<int>(blockIdx.x * 32 + lane), p.s_kv - 1) : 0);
#pragma unroll
            for (int j = 0; j < 4; ++j) row[j] = row[j] >= 0 ? row[j] : own >= 0 ? own : any;
          }
#pragma unroll 1
          for (int i = 0; i < n_tiles; ++i) {
            const uint32_t G = gt + i;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const bool ok = nxt[j] >= 0 && nxt[j] < p.s_kv;
              if (c == 0) {
                if (nxt[j] >= p.s_kv || nxt[j] < -1) m0->bad_index = 1;
                const uint32_t v = __ballot_sync(0xffffffffu, ok);
                if (lane == 0) m0->valid_mask[G & 7][j] = v;
              }
              if (ok) row[j] = nxt[j];                       // a masked entry fetches the row before it again and is multiplied by zero
              const int jn = (i + 1) * kNT + 32 * j + lane;
              nxt[j] = (i + 1 < n_tiles && jn < n_rows) ? idx_row[jn] : -1;
            }
            __syncwarp();
            const uint32_t uses = c < kNQ ? G + ti + 1 : G;
            if (uses >= 1) mbar_wait(k_free, (uses - 1) & 1u, abort_flag);
            if (c == 0 && lane == 0) mbar_arrive(k_full);    // the arrivals below track the copies; this one releases the mask
#pragma unroll
            for (int q = 0; q < 32; ++q) {
              const int r = __shfl_sync(0xffffffffu, row[q >> 3], (q & 7) * 4 + (lane >> 3));
              cp_async16(dst0[q & 1] + (q >> 1) * 1024, src0 + static_cast<long long>(r) * p.kv_sr);
            }
            cp_async_mbar_arrive_noinc(k_full);
          }
          gt += n_tiles;
        }
      }
    } else {
      // ===================================================================== CTA 1: values
      const uint32_t v_s = base;
      const uint32_t p_s = base + kOff1P;
      const uint32_t epi_done_r = mapa_shared(smem_u32(&m0->epi_done[0]), 0);
      // ---------------------------------------------------------------- epilogue duty (16 warps: 0-7 and 9-16)
      // warp -> TMEM lane quarter warp % 4 (head rows 32q .. 32q+31) and column group g (output columns
      // 128g .. 128g+127): warps 0-3 g = 0, 4-7 g = 1, 9-12 g = 2, 13-16 g = 3.  A warp works alone: it
      // converts 64 columns of its rows to bf16 into a private 4 KB piece of the P buffer of the token's
      // last tile ([32 rows x 128 B], the swizzled tile layout) and sends it with one TMA tile store, twice.
      // That P buffer is idle until the softmax two tiles later asks for it, and the relay holds its
      // p_free back until the last store has read it; the V ring is not touched, so the gathers of the
      // next token run underneath.  Warp w < 8 and warp 9 + w share piece w: the V producers come later
      // (they first send out the next token's first gathers) and wait for their partner (stg_free).
      auto epilogue_duty = [&](int ti, uint32_t Gl, int item) {
        const int q4 = warp & 3;
        const int grp = warp < 8 ? (warp >> 2) : 2 + ((warp - 9) >> 2);
        const int piece = warp < 8 ? warp : warp - 9;
        // `fin` first: a parity wait is only exact once the barrier is in, or past, the phase waited for
        // (after `fin` the P.V two tiles before the last one has completed)
        mbar_wait(smem_u32(&m1->fin[ti & 1]), (ti >> 1) & 1u, abort_flag);
        mbar_wait(smem_u32(&m1->pv_done[Gl & 1]), (Gl >> 1) & 1u, abort_flag);
        if (warp >= 9) mbar_wait(smem_u32(&m1->stg_free[piece]), ti & 1u, abort_flag);
        tc_fence_after();
        const int row = q4 * 32 + lane;
        const float inv_l = m1->inv_l[ti & 1][row];
        const uint32_t stg = p_s + (Gl & 1u) * kPBuf + piece * 4096 + lane * 128;
        auto send = [&](int col) {
          fence_proxy_async_smem();   // the tile store reads the piece through the async proxy
          __syncwarp();
          if (lane == 0) {
            if (q4 * 32 < p.h) tma_store_3d(&tm_o, stg - lane * 128, col, q4 * 32, item);
            bulk_commit();
            bulk_wait_read_all();
          }
          __syncwarp();
        };
        if (!has_rows && lane == 0) mbar_arrive(smem_u32(&m1->o_free));
#pragma unroll 1
        for (int cb = 0; cb < 2 && has_rows; ++cb) {
#pragma unroll
          for (int c2 = 0; c2 < 2; ++c2) {
            uint32_t acc[32];
            tmem_ld32(tmem_addr(tmem, q4 * 32, grp * 128 + cb * 64 + c2 * 32), acc);
            tmem_wait_ld();
            if (p.n_splits > 1) {
              // a partial result stays fp32: 32 columns fill the piece
#pragma unroll
              for (int j = 0; j < 8; ++j)
                st_shared_v4(stg + ((j ^ (lane & 7)) << 4), __float_as_uint(__uint_as_float(acc[4 * j]) * inv_l),
                             __float_as_uint(__uint_as_float(acc[4 * j + 1]) * inv_l), __float_as_uint(__uint_as_float(acc[4 * j + 2]) * inv_l),
                             __float_as_uint(__uint_as_float(acc[4 * j + 3]) * inv_l));
              if (c2 == 0) send((grp * 4 + cb * 2) * 32);
              continue;
            }
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              const int chunk = c2 * 4 + (j >> 3);
              st_shared_v4(stg + ((chunk ^ (lane & 7)) << 4),
                           pack_bf16x2(__uint_as_float(acc[j]) * inv_l, __uint_as_float(acc[j + 1]) * inv_l),
                           pack_bf16x2(__uint_as_float(acc[j + 2]) * inv_l, __uint_as_float(acc[j + 3]) * inv_l),
                           pack_bf16x2(__uint_as_float(acc[j + 4]) * inv_l, __uint_as_float(acc[j + 5]) * inv_l),
                           pack_bf16x2(__uint_as_float(acc[j + 6]) * inv_l, __uint_as_float(acc[j + 7]) * inv_l));
            }
          }
          if (cb == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&m1->o_free));   // the next token's P.V may overwrite the accumulator
          }
          send(p.n_splits > 1 ? (grp * 4 + cb * 2 + 1) * 32 : (grp * 2 + cb) * 64);
        }
        if (lane == 0) {
          if (warp < 8) mbar_arrive(smem_u32(&m1->stg_free[piece]));
          mbar_arrive(smem_u32(&m1->epi_cnt));
        }
      };
      if (warp < 8) {
        const uint32_t p_free_r = mapa_shared(smem_u32(&m0->p_free[0]), 0);
        for (int t = 0; t < nb; ++t) {
          const int ti = batch0 + t;
          const int item = pair + ti * n_pairs;
          const int n_tiles = warp_uniform(nt[t]);
          if (warp < 4 && has_rows) {
            // ------------------------------------------------------------ correction (thread = head)
            for (int i = 0; i < n_tiles; ++i) {
              const uint32_t G = gt + i;
              const int b = G & 1;
              mbar_wait_cluster(smem_u32(&m1->p_full[b]), (G >> 1) & 1u, abort_flag);
              auto rescale = [&](float a) {
                tc_fence_after();
#pragma unroll 1
                for (int c0 = 0; c0 < 512; c0 += 32) {
                  uint32_t o[32];
                  tmem_ld32(tmem_addr(tmem, warp * 32, c0), o);
                  tmem_wait_ld();
#pragma unroll
                  for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * a);
                  tmem_st32(tmem_addr(tmem, warp * 32, c0), o);
                }
                tmem_wait_st();
                tc_fence_before();
              };
              const float a = m1->alpha[b][tid].x, a_late = m1->alpha[b][tid].y;
              if (__any_sync(0xffffffffu, (i > 0) && (a != 1.0f))) {
                mbar_wait(smem_u32(&m1->pv_done[(G - 1) & 1]), ((G - 1) >> 1) & 1u, abort_flag);
                rescale(a);
              }
              // the second half of the tile may move a maximum once more: the issuer then stops between the halves
              const bool late = __any_sync(0xffffffffu, a_late != 1.0f);
              if (lane == 0) reinterpret_cast<uint8_t*>(&m1->late[b])[warp] = late ? 1 : 0;
              // (no proxy fence for P here: the issuer, which waits for this arrival, executes one before the first MMA of the tile)
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&m1->corr_done[b]));
              if (late) {
                mbar_wait(smem_u32(&m1->half_done[warp]), n_late & 1u, abort_flag);
                rescale(a_late);
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&m1->half_corr[warp]));
                ++n_late;
              }
            }
          } else if (warp == 4 && lane == 0) {
            // ------------------------------------------------------------ relay: P buffer free -> CTA 0
            for (int i = 0; i + 1 < n_tiles; ++i) {
              const uint32_t G = gt + i;
              mbar_wait(smem_u32(&m1->pv_done[G & 1]), (G >> 1) & 1u, abort_flag);
              mbar_arrive_cluster_relaxed(p_free_r + (G & 1) * 8);
            }
          }
          __syncwarp();
          gt += n_tiles;
          epilogue_duty(ti, gt - 1, item);
          // the P buffer of the last tile staged the output: it is free for the softmax, and 1/l of this
          // token may be replaced, once all 16 warps are through
          if (warp == 4 && lane == 0) {
            mbar_wait(smem_u32(&m1->epi_cnt), ti & 1u, abort_flag);
            mbar_arrive_cluster_relaxed(p_free_r + ((gt - 1) & 1) * 8);
            mbar_arrive_cluster_relaxed(epi_done_r + (ti & 1) * 8);
          }
        }
      } else if (warp == 8) {
        // -------------------------------------------------------------- P.V issuer (whole warp, an elected lane issues)
        {
          constexpr uint32_t kIdesc = umma_idesc(kFmtBF16, 128, 256, 0, 1);
          const uint64_t ad0 = smem_desc_sw128(p_s, kPChunk, 128) & ~(static_cast<uint64_t>(7) << 61);   // no swizzle: 8 x 16-byte matrices, the next along K a chunk on, the next of heads 128 bytes on
          const uint64_t bd0 = smem_desc_sw128(v_s, kVBlock, 1024);
          const uint32_t ad_lo = static_cast<uint32_t>(ad0), ad_hi = static_cast<uint32_t>(ad0 >> 32);
          const uint32_t bd_lo = static_cast<uint32_t>(bd0), bd_hi = static_cast<uint32_t>(bd0 >> 32);
          const uint32_t v_full0 = smem_u32(&m1->v_full[0]), v_free0 = smem_u32(&m1->v_free[0]);
          for (int t = 0; t < nb; ++t) {
            const int ti = batch0 + t;
            const int n_tiles = warp_uniform(nt[t]);
            // the epilogue of the previous token has read the accumulator
            if (ti >= 1) mbar_wait(smem_u32(&m1->o_free), (ti - 1) & 1u, abort_flag);
            for (int i = 0; i < n_tiles; ++i) {
              const uint32_t G = gt + i;
              const int b = G & 1;
              const uint32_t ph = G & 1u;
              mbar_wait(smem_u32(&m1->corr_done[b]), (G >> 1) & 1u, abort_flag);
              tc_fence_after();
              const uint32_t late = m1->late[b];
              const uint32_t a_lo = ad_lo + ((b * kPBuf) >> 4);
#pragma unroll 1
              for (int sl = 0; sl < kNV; ++sl) {
                mbar_wait(v_full0 + sl * 8, ph, abort_flag);
                fence_proxy_async_smem();   // the rows were written by cp.async (generic proxy)
                tc_fence_after();
                if (elect_one()) {
                  // slab sl = 16-row steps 2 sl and 2 sl + 1 of the tile
                  const uint32_t alo = a_lo + ((sl * 4 * kPChunk) >> 4);
                  const uint32_t blo = bd_lo + ((sl * kVSlab) >> 4);
#pragma unroll
                  for (int kk = 0; kk < 2; ++kk) {
#pragma unroll
                    for (int hv = 0; hv < 2; ++hv)
                      umma_f16_ss(tmem + hv * 256, (static_cast<uint64_t>(ad_hi) << 32) | (alo + ((kk * 2 * kPChunk) >> 4)),
                                  (static_cast<uint64_t>(bd_hi) << 32) | (blo + ((hv * 4 * kVBlock + kk * 2048) >> 4)), kIdesc,
                                  kk == 0 ? static_cast<uint32_t>(i | sl) : 1u);
                  }
                  umma_commit(v_free0 + sl * 8);
                  if (sl == 1 && late != 0u) {
                    for (int w = 0; w < 4; ++w)
                      if ((late >> (8 * w)) & 1u) umma_commit(smem_u32(&m1->half_done[w]));
                  }
                }
                __syncwarp();
                if (sl == 1 && late != 0u) {
#pragma unroll 1
                  for (int w = 0; w < 4; ++w) {
                    if ((late >> (8 * w)) & 1u) {
                      mbar_wait(smem_u32(&m1->half_corr[w]), (n_late >> w) & 1u, abort_flag);
                      n_late ^= 1u << w;
                    }
                  }
                  tc_fence_after();
                }
              }
              if (elect_one()) umma_commit(smem_u32(&m1->pv_done[b]));
              __syncwarp();
            }
            gt += n_tiles;
          }
        }
      } else if (warp < 17) {
        // -------------------------------------------------------------- V producers (warps 9-16)
        // Producer w fetches four of the eight column blocks of slab w / 2 of every tile (lane l: piece l % 8 of rows
        // 4 q + l / 8).
        const int w = warp - 9;
        const int sl = w >> 1;
        const __nv_bfloat16* src0 = p.kv + (w & 1) * 256 + (lane & 7) * 8;
        const uint32_t v_full = smem_u32(&m1->v_full[sl]), v_free = smem_u32(&m1->v_free[sl]);
        uint32_t dst0[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int r = 4 * q + (lane >> 3);
          dst0[q] = v_s + sl * kVSlab + (w & 1) * 4 * kVBlock + r * 128 + (((lane & 7) ^ r) << 4);
        }
#pragma unroll 1
        for (int t = 0; t <= nb; ++t) {                      // pass nb: nothing to fetch, the last token's epilogue is left
          const int ti = batch0 + t;
          const int item = pair + ti * n_pairs;
          const int n_tiles = t < nb ? warp_uniform(nt[t]) : 1;
          const int row0 = t < nb ? warp_uniform(nt[kBatch + t]) * kNT : 0, n_rows = p.topk - row0;
          const int32_t* idx_row = p.indices + static_cast<long long>(t < nb ? token_of(item) : 0) * p.idx_st + row0;
          int nxt = sl * kVSlabRows + lane < n_rows ? idx_row[sl * kVSlabRows + lane] : -1;   // row `lane` of the slab
          int row = nxt >= 0 && nxt < p.s_kv ? nxt : -1;
          if (!__all_sync(0xffffffffu, row >= 0)) {
            const int any = first_row(idx_row, t < nb && last[t] > 0 ? n_rows : 0, p.s_kv, p.n_splits > 1 ? min(static_cast<int>(blockIdx.x * 32 + lane), p.s_kv - 1) : 0);
            if (row < 0) row = any;
          }
#pragma unroll 1
          for (int i = 0; i < n_tiles; ++i) {
            if (t < nb) {
              const uint32_t G = gt + i;
              if (nxt >= 0 && nxt < p.s_kv) row = nxt;
              const int jn = (i + 1) * kNT + sl * kVSlabRows + lane;
              nxt = (i + 1 < n_tiles && jn < n_rows) ? idx_row[jn] : -1;
              if (G >= 1) mbar_wait(v_free, (G - 1) & 1u, abort_flag);
              __syncwarp();
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                const __nv_bfloat16* src = src0 + static_cast<long long>(__shfl_sync(0xffffffffu, row, 4 * q + (lane >> 3))) * p.kv_sr;
#pragma unroll
                for (int cb = 0; cb < 4; ++cb) cp_async16(dst0[q & 1] + (q >> 1) * 1024 + cb * kVBlock, src + cb * 64);
              }
              cp_async_mbar_arrive_noinc(v_full);
            }
            // the first tile goes out before this warp helps with the previous token's epilogue, so that the
            // gathers run underneath it
            if (i == 0 && t > 0) {
              __syncwarp();
              epilogue_duty(ti - 1, gt - 1, item - n_pairs);
            }
          }
          if (t < nb) gt += n_tiles;
        }
      }
    }
    __syncthreads();   // nt[] is rewritten by the next batch
  }

  if (*abort_flag) drain_after_abort();
  tc_fence_before();
  __syncthreads();
  if (!one_each) griddep_launch();               // (behind the barrier: one thread of a CTA speaks for all)
  cluster_sync_all();            // nobody leaves while the peer may still write or signal this CTA
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, 512u);
  }
  if (tid == 0 && p.status != nullptr) {
    if (*abort_flag) atomicCAS(p.status, 0, FTB_ERR_TIMEOUT);
    else if (cta == 0 && m0->bad_index) atomicCAS(p.status, 0, FTB_ERR_BAD_INDEX);
  }
}

}  // namespace mla_ring

// n_splits > 1: partial results to part_out / part_lse, and `out` and `lse` of the arguments are left alone.  `max_slack`: see the softmax;
// 24 tokens of topk 2048 and 64 heads in parts 39 us with a slack of 8, 43 without (relative error 2.0e-3 and 1.8e-3).
int launch_sparse_mla_ring(const ftb_sparse_mla_args* a, int n_splits, float* part_out, float* part_lse, float max_slack, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(mla_ring::sparse_mla_ring_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, mla_ring::kSmemBytes);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(sparse_mla_ring)");
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(mla_ring::kThreads);
  cfg.dynamicSmemBytes = mla_ring::kSmemBytes;
  cfg.stream = st;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;                            // (of the occupancy query; the launches take both)
  // as many pairs as the device holds at once (one per pair of SMs that can host a cluster), cached per device
  static int pairs_of_device[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  int pairs_dev = (dev >= 0 && dev < 64) ? pairs_of_device[dev] : 0;
  if (pairs_dev == 0) {
    cfg.gridDim = dim3(2);
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, mla_ring::sparse_mla_ring_kernel, &cfg);
    if (e != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      int sms = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      n = sms / 2 > 0 ? sms / 2 : 1;
    }
    pairs_dev = n;
    if (dev >= 0 && dev < 64) pairs_of_device[dev] = pairs_dev;
  }
  // One launch takes at most kBatch tokens per pair, so that every pair finds its tile counts once and runs
  // through its tokens without a stop; a longer batch of query tokens is a sequence of such launches on the
  // stream (a launch boundary every pairs x kBatch tokens costs next to nothing).
  const long long items = static_cast<long long>(pairs_dev) * mla_ring::kBatch;
  const long long cap = items / n_splits > 0 ? items / n_splits : 1;
  // Q: boxes of [h rows x 64 columns] of one token; O: boxes of [32 rows x 64 columns] (a store that
  // reaches past row h is clipped)
  const uint32_t box_h = static_cast<uint32_t>(a->h < 128 ? a->h : 128);
  for (long long t0 = 0; t0 < a->s_q; t0 += cap) {
    const int n_tok = static_cast<int>(a->s_q - t0 < cap ? a->s_q - t0 : cap);
    mla_ring::Params p;
    p.kv = static_cast<const __nv_bfloat16*>(a->kv);
    p.kv_sr = a->kv_stride_row;
    p.indices = a->indices + t0 * a->idx_stride_token;
    p.lse = a->lse + t0 * a->lse_stride_token;
    p.s_q = n_tok; p.h = a->h; p.s_kv = a->s_kv; p.topk = a->topk;
    p.idx_st = a->idx_stride_token;
    p.lse_st = a->lse_stride_token;
    p.scale_log2 = a->sm_scale * 1.4426950408889634f;
    p.lse_base2 = a->lse_base2;
    p.status = a->status;
    p.n_splits = n_splits;
    p.max_slack = max_slack;
    p.part_lse = part_lse + (n_splits > 1 ? static_cast<size_t>(t0) * n_splits * a->h : 0);
    const void* q0 = static_cast<const __nv_bfloat16*>(a->q) + t0 * a->q_stride_token;
    void* o0 = static_cast<__nv_bfloat16*>(a->out) + t0 * a->out_stride_token;
    CUtensorMap tm_q, tm_o;
    if (!make_tmap_3d(&tm_q, q0, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, mla_ring::kDqk, static_cast<uint64_t>(a->h),
                      static_cast<uint64_t>(n_tok), static_cast<uint64_t>(a->q_stride_head),
                      static_cast<uint64_t>(a->q_stride_token), 64, box_h) ||
        !(n_splits > 1 ? make_tmap_3d(&tm_o, part_out + static_cast<size_t>(t0) * n_splits * a->h * 512, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, 512,
                                      static_cast<uint64_t>(a->h), static_cast<uint64_t>(n_tok) * n_splits, 512,
                                      static_cast<uint64_t>(a->h) * 512, 32, box_h < 32 ? box_h : 32)
                       : make_tmap_3d(&tm_o, o0, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 512, static_cast<uint64_t>(a->h),
                                      static_cast<uint64_t>(n_tok), static_cast<uint64_t>(a->out_stride_head),
                                      static_cast<uint64_t>(a->out_stride_token), 64, box_h < 32 ? box_h : 32))) {
      set_last_error("sparse_mla_ring: cuTensorMapEncodeTiled failed");
      return FTB_ERR_CUDA;
    }
    const int pairs = pairs_dev < n_tok * n_splits ? pairs_dev : n_tok * n_splits;
    cfg.gridDim = dim3(static_cast<unsigned>(pairs) * 2u);
    cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, mla_ring::sparse_mla_ring_kernel, tm_q, tm_o, p);
    if (e != cudaSuccess) return check_cuda(e, "sparse_mla_ring launch");
  }
  return FTB_OK;
}

}  // namespace ftb
