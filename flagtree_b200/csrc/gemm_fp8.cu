// Block-scaled FP8 (e4m3) GEMM for sm_100a: C[M,N] = sum_kb (A[:,kb] . B[kb,:]) * a_scale[:,kb] (x) b_scale[kb,:/128]
// with A [M,K] e4m3 and 1x128 fp32 scales, B [K,N] e4m3 and 128x128 fp32 scales, bf16 output.
//
// The tensor cores' own block scaling takes 32-element ue8m0/ue4m3 scales, not fp32 per 128, so every
// 128-deep K block is multiplied on its own (4 tcgen05.mma kind::f8f6f4 of K = 32 into a fresh TMEM
// accumulator) and eight "promotion" warps fold it into fp32 registers with its two scales while the
// next block is being multiplied.
//
// Two tile shapes, NCTA = 2: a CTA pair (cta_group::2) computes 256 x 256, NCTA = 1: one CTA computes 128 x 128.
// Either way a CTA loads 128 rows of A and 128 columns of B per K block (32 KB, six stages), but the pair's
// MMAs take 512 cycles for it where the single tile's take 256, and the operand reads of a 128 x 128 MMA alone
// need the whole shared-memory bandwidth (32 KB in 256 cycles at 128 B per cycle) with the TMA writes on top.  So
// the pair is the shape for large M and the single tile the one for small M, where the weight's bytes are the
// bound and a finer grid matters.  An SM takes in about 64 bytes per clock, A included, so the weight is cut finer still, into
// tiles of 64 columns (NB), while every tile finds an SM; a row-major weight then lies in 64-byte rows under the 64-byte swizzle.
// Split K (S > 1, for grids that would leave SMs idle): the S CTAs (or pairs) of a cluster multiply S parts of K; the
// fp32 partial tiles meet in shared memory over DSMEM, every part adds up 1/S of the columns in a fixed order and
// writes them: no workspace, no second launch, no atomics.
// Roles (384 threads): warp 0 TMA producer (single tiles: of A, and warp 2 of B), warp 1 MMA issuer + TMEM owner, warps 4-11 promotion/epilogue: warp w takes
// TMEM lanes 32 (w % 4) .. and half (w / 4 - 1) of the columns, so a thread holds 128 (64) fp32 sums.  Per K block a
// thread needs one product of two scales: they are fetched from memory a group of four blocks ahead.
// Measured, one GPU, K = 28672, N = 8192.  M = 4096 back to back, where the power limit sets the clock: 1048 us a call (1836 TFLOP/s) against
// 1848 of the kernel before (128 x 128 tiles, four promotion warps that fetched their scales when they needed them).  Launches
// with pauses between them (TFLOP/s): M = 4096 2107 (before 1078), M = 1024 1130 (912).  Steps of M = 4096 that way: eight promotion
// warps, scales ahead, single tiles 1269 and pairs 1037; the pair's hand-back of an accumulator as a relaxed remote
// arrival (a release at cluster scope stalls the warp) 1921; the pieces of neighbouring K blocks as one stream 2107.
// Single tiles: 64 x 8192 x 3584 back to back 13.1 -> 12.3 us a call (29 MB, 4.4 us) with A and B loaded by two warps, two K blocks per wait
// of the issuer, and one commit that tells both the producer and the promotion warps.  With pairs the same commit made M = 4096
// slower (1119 us), so those keep their two.  With tiles of 64 columns 10.6, 2.9 TB/s; what is left is launch, prologue and the fill of the pipeline.
// What bounds M = 4096 now: with the additions left out 826 us instead of 913, with the tensor-memory loads left out too 680 us
// (the tensor pipe and the power limit: a library e4m3 GEMM reaches 2960).
#include <cstring>

#include "launch.cuh"
#include "sm100.cuh"
#include "tmap.cuh"

namespace ftb {

void set_last_error(const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

namespace gemm8 {

constexpr int BM = 128, BK = 128, STAGES = 6;
constexpr int A_BYTES = BM * BK;          // 16384
constexpr int B_BYTES = BK * 128;         // 16384: 128 columns per CTA in both shapes
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
// Where the promotion warps turn their rows round before they write them (4096 x 8192 x 28672 1060 -> 1046 us, 384 x 8192 x 1024 10.3 -> 9.1): of its
// own for pairs without a split; a single tile of a CTA has its stages free by then (384 x 6144 x 1024 8.1 -> 6.9, 128 x 6144 x 3584 11.2 -> 10.6).
// Singles with boxes of their own lost more than that with a long K: they come off the L1 that holds the scales (64 x 8192 x 16384 29.8 -> 32.1).
constexpr int BOX_BYTES = 8 * 4096;
constexpr int THREADS = 384;             // launched with 168 registers each: 8 x 32 x 224 + 4 x 32 x 56 = 384 x 168
constexpr int kRegsMany = 224, kRegsFew = 56;
constexpr int kGroupM = 8;                // row blocks of a super-row of tiles (both operands are re-used out of L2)

struct Params {
  int m, n, k, m_blocks, n_blocks, n_tiles, kb_total, splits;
  uint32_t stage_tx;      // bytes one CTA loads per stage (fewer rows of A when m < 128)
  const float* a_scale;   // [m, kb_total]
  const float* b_scale;   // [kb_total, n / 128]
  long long lda_s, ldb_s;
  __nv_bfloat16* c;
  long long ldc;
  int* status;
};

struct Bars {
  unsigned long long full[STAGES];
  unsigned long long empty[STAGES];
  unsigned long long blk_full[4];      // pairs only
  unsigned long long blk_empty[4];
  uint32_t tmem_base;
  int abort_flag;
};

// D[tmem] (+)= A . B, descriptors as 32-bit halves (only the low ones change), compile-time accumulate flag
template <int NCTA, bool kAccumulate>
__device__ __forceinline__ void umma_f8_lohi(uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc) {
  if constexpr (NCTA == 1) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\t"
        "setp.ne.b32 p, %6, 0;\n\tmov.b64 ad, {%1, %2};\n\tmov.b64 bd, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], ad, bd, %5, p;\n\t}"
        ::"r"(d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "n"(kAccumulate ? 1 : 0) : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\t"
        "setp.ne.b32 p, %6, 0;\n\tmov.b64 ad, {%1, %2};\n\tmov.b64 bd, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], ad, bd, %5, p;\n\t}"
        ::"r"(d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "n"(kAccumulate ? 1 : 0) : "memory");
  }
}
// One arrival on this CTA's barrier (NCTA = 1) or on the barrier at the same offset in both CTAs of the pair
template <int NCTA>
__device__ __forceinline__ void commit_all(uint32_t bar, uint16_t mask) {
  if constexpr (NCTA == 1) umma_commit(bar);
  else
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(mask) : "memory");
}
// remote arrival that only hands a buffer back
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// wait for the tensor-memory loads issued so far; the registers are operands so that no use moves above it
__device__ __forceinline__ void tmem_wait_ld_regs(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :: "memory");
  asm volatile("" : "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                    "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :: "memory");
}
// acc.{x,y} += v.{x,y} * s, two fp32 fused multiply-adds per instruction
__device__ __forceinline__ void fma_x2(float2& acc, uint32_t v0, uint32_t v1, float s) {
  asm("{\n\t.reg .b64 a, b, c;\n\t"
      "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%0, %1};\n\t"
      "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "+f"(acc.x), "+f"(acc.y) : "r"(v0), "r"(v1), "f"(s));
}

template <int NCTA, bool B_KMAJOR, int NB = 128>
__global__ void __launch_bounds__(THREADS, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const Params p) {
  constexpr int BN = NB * NCTA;           // columns of the tile = fp32 columns of one TMEM accumulator
  constexpr int COLS = BN / 2;            // columns of a promotion thread
  constexpr uint32_t NACC = BN == 256 ? 2 : 4;     // accumulators in flight
  static_assert(NB == 128 || (NCTA == 1 && NB == 64), "narrow tiles: of a single CTA");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw_addr);
  Bars* bars = reinterpret_cast<Bars*>(sm + STAGES * STAGE_BYTES);
  static_assert(sizeof(Bars) <= 256, "boxes behind the barriers");
  const uint32_t boxes = base + STAGES * STAGE_BYTES + 256;
  volatile int* abort_flag = &bars->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool clustered = NCTA * p.splits > 1;
  const int rank = clustered ? static_cast<int>(cluster_ctarank()) : 0;
  const int cta = rank % NCTA, split = rank / NCTA;      // place in the pair, part of K
  const int leader = rank - cta;                         // the pair's even CTA: its issuer multiplies for both
  const int group = blockIdx.x / (NCTA * p.splits), n_groups = gridDim.x / (NCTA * p.splits);
  const int kb0 = static_cast<int>(static_cast<long long>(p.kb_total) * split / p.splits);
  const int kb1 = static_cast<int>(static_cast<long long>(p.kb_total) * (split + 1) / p.splits);

  const bool one_each = p.n_tiles <= n_groups;
  if (one_each) griddep_launch();
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&bars->full[s]), NCTA == 1 ? 2 : 1);   // A and B apart
      mbar_init(smem_u32(&bars->empty[s]), 1);
    }
    for (int a = 0; a < NACC; ++a) {
      mbar_init(smem_u32(&bars->blk_full[a]), 1);
      mbar_init(smem_u32(&bars->blk_empty[a]), 8 * NCTA);   // the promotion warps of the pair
    }
    fence_mbar_init();
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_b);
  }
  griddep_wait();
  if (tid == 0) bars->abort_flag = (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
  __syncthreads();
  // an earlier launch on this status word failed: leave at once, the whole cluster on the reading of its CTA 0
  if (clustered && p.status != nullptr) {
    cluster_sync_all();
    uint32_t leave;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(leave) : "r"(mapa_shared(smem_u32(&bars->abort_flag), 0)) : "memory");
    cluster_sync_all();        // CTA 0 keeps its flag until the others have read it
    if (tid == 0) bars->abort_flag = leave != 0u ? 1 : 0;
    __syncthreads();
  }
  if (bars->abort_flag) return;
  if (warp == 1) {
    if constexpr (NCTA == 1) {
      tmem_alloc(smem_u32(&bars->tmem_base), 512);
      tmem_relinquish();
    } else {
      tmem_alloc_pair(smem_u32(&bars->tmem_base), 512);
      tmem_relinquish_pair();
    }
    tc_fence_before();
  }
  __syncthreads();
  if (clustered) cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;

  // tiles in super-rows of kGroupM row blocks, row block fastest
  auto coords = [&](int t, int& m_blk, int& n_blk) {
    const int per = kGroupM * p.n_blocks;
    const int sr = t / per, r = t - sr * per;
    const int rows = min(kGroupM, p.m_blocks - sr * kGroupM);
    n_blk = r / rows;
    m_blk = (sr * kGroupM + (r - n_blk * rows)) * NCTA + cta;
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsFew));
    if (warp == 0 || (NCTA == 1 && warp == 2)) {
      // Single tiles: A by one warp, B by another, since a turn with two loads takes a lone thread 410 cycles, more than the MMAs' 256.
      const bool is_b = warp == 2;
      if (lane == 0) {
        uint32_t s = 0, ph = 1;
        for (int t = group; t < p.n_tiles; t += n_groups) {
          int m_blk, n_blk;
          coords(t, m_blk, n_blk);
          const int n0 = n_blk * BN + cta * NB;
          bool live = true;
          for (int kb = kb0; kb < kb1; ++kb) {
            if (!mbar_wait(smem_u32(&bars->empty[s]), ph, abort_flag)) { live = false; break; }
            const uint32_t a_dst = base + s * STAGE_BYTES;
            if constexpr (NCTA == 1) {
              const uint32_t full = smem_u32(&bars->full[s]);
              const int x = is_b && !B_KMAJOR ? n0 : kb * BK, y = !is_b ? m_blk * BM : B_KMAJOR ? n0 : kb * BK;
              mbar_arrive_expect_tx(full, is_b ? NB * BK : p.stage_tx - NB * BK);
              tma_load_2d(is_b ? a_dst + A_BYTES : a_dst, is_b ? &tm_b : &tm_a, full, x, y);
            } else {
              // both CTAs' loads are counted on the even CTA's barrier; that CTA announces the total
              const uint32_t full = mapa_shared(smem_u32(&bars->full[s]), leader);
              if (cta == 0) mbar_arrive_expect_tx(smem_u32(&bars->full[s]), 2 * p.stage_tx);
              tma_load_2d_pair(a_dst, &tm_a, full, kb * BK, m_blk * BM);
              if constexpr (B_KMAJOR) tma_load_2d_pair(a_dst + A_BYTES, &tm_b, full, kb * BK, n0);
              else tma_load_2d_pair(a_dst + A_BYTES, &tm_b, full, n0, kb * BK);
            }
            if (++s == STAGES) { s = 0; ph ^= 1u; }
          }
          if (!live) break;
        }
      }
      __syncwarp();
    } else if (warp == 1 && cta == 0) {
      // the whole warp runs the loop and waits, an elected lane (always the same one) issues
      constexpr uint32_t kIdesc = umma_idesc(kFmtE4M3, BM * NCTA, BN, 0, B_KMAJOR ? 0 : 1);
      const uint64_t ad0 = smem_desc_sw128(base, 16, 1024);
      // row-major B: eight k-rows of NB bytes are a swizzle atom, of 128-byte rows or of 64-byte rows (mode 4 instead of 2)
      const uint64_t bd0 = B_KMAJOR ? smem_desc_sw128(base + A_BYTES, 16, 1024)
                                    : smem_desc_sw128(base + A_BYTES, NB * BK, 8 * NB) ^ (NB == 64 ? static_cast<uint64_t>(6) << 61 : 0);
      const uint32_t ad_lo0 = static_cast<uint32_t>(ad0), ad_hi = static_cast<uint32_t>(ad0 >> 32);
      const uint32_t bd_lo0 = static_cast<uint32_t>(bd0), bd_hi = static_cast<uint32_t>(bd0 >> 32);
      constexpr uint32_t kBStep = (B_KMAJOR ? 32 : 32 * NB) >> 4;   // 32 bytes of K, or 32 k-rows
      const uint16_t mask = static_cast<uint16_t>(3u << leader);
      const uint32_t full0 = smem_u32(&bars->full[0]), empty0 = smem_u32(&bars->empty[0]);
      const uint32_t be0 = smem_u32(&bars->blk_empty[0]);
      uint32_t s = 0, ph = 0, it = 0;   // it: K blocks issued so far = accumulator uses
      for (int t = group; t < p.n_tiles; t += n_groups) {
        bool live = true;
        if constexpr (NCTA == 1) {
          // Two K blocks at a time, the stages and the accumulators waited for by different lanes at once: a wait costs the warp 120 cycles and a
          // commit 60, the MMAs of a block take 256.  The one commit of a block frees its stage and hands its accumulator over: the promotion
          // warps follow the stage's phase, which cannot run away from them, as block it + STAGES is not issued before it + 2 is promoted.
          static_assert(STAGES % 2 == 0 && STAGES > NACC, "both blocks in one phase, accumulators reused before stages");
          for (int kb = kb0; kb < kb1;) {
            const int n = min(kb1 - kb, s % 2 == 0 ? 2 : 1);
            const uint32_t which = n == 2 ? (lane >> 1) & 1u : 0u, acc = (it + which) % NACC;
            live = (lane & 1) ? mbar_wait(be0 + acc * 8, (((it + which) / NACC) & 1u) ^ 1u, abort_flag) : mbar_wait(full0 + (s + which) * 8, ph, abort_flag);
            live = __all_sync(0xffffffffu, live);
            if (!live) break;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                if (j == n) break;
                const uint32_t a_lo = ad_lo0 + (((s + j) * STAGE_BYTES) >> 4), b_lo = bd_lo0 + (((s + j) * STAGE_BYTES) >> 4);
                const uint32_t acc_j = (it + j) % NACC, d = tmem + acc_j * BN;
                umma_f8_lohi<NCTA, false>(d, a_lo, ad_hi, b_lo, bd_hi, kIdesc);
#pragma unroll
                for (int k = 1; k < BK / 32; ++k)
                  umma_f8_lohi<NCTA, true>(d, a_lo + ((k * 32) >> 4), ad_hi, b_lo + k * kBStep, bd_hi, kIdesc);
                commit_all<NCTA>(empty0 + (s + j) * 8, mask);
              }
            }
            __syncwarp();
            kb += n;
            it += n;
            s += n;
            if (s == STAGES) { s = 0; ph ^= 1u; }
          }
        } else {
          const uint32_t bf0 = smem_u32(&bars->blk_full[0]);
          for (int kb = kb0; kb < kb1; ++kb, ++it) {
            const uint32_t acc = it % NACC;
            live = mbar_wait(full0 + s * 8, ph, abort_flag) && mbar_wait(be0 + acc * 8, ((it / NACC) & 1u) ^ 1u, abort_flag);
            live = __all_sync(0xffffffffu, live);
            if (!live) break;
            tc_fence_after();
            if (elect_one()) {
              const uint32_t a_lo = ad_lo0 + ((s * STAGE_BYTES) >> 4), b_lo = bd_lo0 + ((s * STAGE_BYTES) >> 4);
              const uint32_t d = tmem + acc * BN;
              umma_f8_lohi<NCTA, false>(d, a_lo, ad_hi, b_lo, bd_hi, kIdesc);
#pragma unroll
              for (int k = 1; k < BK / 32; ++k)
                umma_f8_lohi<NCTA, true>(d, a_lo + ((k * 32) >> 4), ad_hi, b_lo + k * kBStep, bd_hi, kIdesc);
              commit_all<NCTA>(empty0 + s * 8, mask);
              commit_all<NCTA>(bf0 + acc * 8, mask);
            }
            __syncwarp();
            if (++s == STAGES) { s = 0; ph ^= 1u; }
          }
        }
        if (!live) break;
      }
    }
    if (p.splits > 1) {
      cluster_sync_all();
      cluster_sync_all();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMany));
    const int lg = warp & 3, half = (warp >> 2) - 1;
    const uint32_t tacc = tmem_addr(tmem, lg * 32, half * COLS);
    const uint32_t be0 = NCTA == 1 ? smem_u32(&bars->blk_empty[0]) : mapa_shared(smem_u32(&bars->blk_empty[0]), leader);
    uint32_t it = 0, st = 0, st_ph = 0;       // K blocks so far; the stage that the next one goes through
    for (int t = group; t < p.n_tiles; t += n_groups) {
      int m_blk, n_blk;
      coords(t, m_blk, n_blk);
      const int row = m_blk * BM + lg * 32 + lane;
      const bool row_ok = row < p.m;
      const int n0 = n_blk * BN + half * COLS;
      const bool col_ok = n0 < p.n;
      float2 accf[COLS / 2];
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) accf[j] = make_float2(0.0f, 0.0f);
      const float* as_row = p.a_scale + static_cast<long long>(row_ok ? row : 0) * p.lda_s;
      const float* bs_col = p.b_scale + (col_ok ? n0 >> 7 : 0);
      float as_nxt[4], bs_nxt[4];       // multiplied a group later, when they have arrived
      auto fetch = [&](int kb) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int k = min(kb + j, kb1 - 1);
          as_nxt[j] = as_row[k];
          bs_nxt[j] = bs_col[static_cast<long long>(k) * p.ldb_s];
        }
      };
      fetch(kb0);
      // The columns of the K blocks form one stream of 32-column pieces: while one piece is added, the next (of the
      // next K block, at a block's end) is on its way from tensor memory.
      constexpr int NP = COLS / 32;
      uint32_t v[2][32];
      auto begin_block = [&](int buf) {
        const uint32_t acc = it % NACC;
        if constexpr (NCTA == 1) {
          mbar_wait(smem_u32(&bars->empty[st]), st_ph, abort_flag);
          if (++st == STAGES) { st = 0; st_ph ^= 1u; }
        } else {
          mbar_wait(smem_u32(&bars->blk_full[acc]), (it / NACC) & 1u, abort_flag);
        }
        __syncwarp();
        tc_fence_after();
        tmem_ld32(tacc + acc * BN, v[buf]);
      };
      begin_block(0);
#pragma unroll 1
      for (int kq = kb0; kq < kb1; kq += 4) {
        float sc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) sc[j] = as_nxt[j] * bs_nxt[j];
        fetch(kq + 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (kq + j < kb1) {
            const uint32_t acc = it % NACC;
#pragma unroll
            for (int c = 0; c < NP; ++c) {
              const int now = (j * NP + c) & 1;
              tmem_wait_ld_regs(v[now]);
              if (c + 1 < NP) {
                tmem_ld32(tacc + acc * BN + (c + 1) * 32, v[now ^ 1]);
              } else {
                // everything of this accumulator is in registers: hand it back
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                  if constexpr (NCTA == 1) mbar_arrive(be0 + acc * 8);
                  // Relaxed is enough: what the issuer's MMA may not overtake are the loads of this accumulator, and
                  // tcgen05.wait::ld has seen them complete in this warp before the lane arrives.  No other write of these
                  // warps is handed over, and tensor memory is not reached through the generic proxy.
                  else mbar_arrive_cluster_relaxed(be0 + acc * 8);
                }
                ++it;
                if (kq + j + 1 < kb1) begin_block(now ^ 1);
              }
#pragma unroll
              for (int e = 0; e < 16; ++e) fma_x2(accf[c * 16 + e], v[now][2 * e], v[now][2 * e + 1], sc[j]);
            }
          }
        }
      }
      if (p.splits == 1) {
        if (NCTA == 2 || (one_each && p.m >= 32)) {        // (a few rows are a few pieces)
          const uint32_t box = (NCTA == 2 ? boxes : base) + (warp - 4) * 4096;
          constexpr int P = COLS >= 64 ? 8 : 4;
#pragma unroll
          for (int c0 = 0; c0 < COLS; c0 += 8 * P)
            store_rows_bf16<P>(box, p.c, p.ldc, m_blk * BM + lg * 32, p.m, n0 + c0, p.n, [&](int ch) {
              const float2* f = accf + c0 / 2 + 4 * ch;
              return make_uint4(pack_bf16x2(f[0].x, f[0].y), pack_bf16x2(f[1].x, f[1].y), pack_bf16x2(f[2].x, f[2].y), pack_bf16x2(f[3].x, f[3].y));
            });
        } else if (row_ok && col_ok) {
          __nv_bfloat16* orow = p.c + static_cast<long long>(row) * p.ldc + n0;
#pragma unroll
          for (int j = 0; j < COLS / 2; j += 4) {
            uint4 o;
            o.x = pack_bf16x2(accf[j].x, accf[j].y);
            o.y = pack_bf16x2(accf[j + 1].x, accf[j + 1].y);
            o.z = pack_bf16x2(accf[j + 2].x, accf[j + 2].y);
            o.w = pack_bf16x2(accf[j + 3].x, accf[j + 3].y);
            *reinterpret_cast<uint4*>(orow + 2 * j) = o;
          }
        }
      } else {
        // Every stage of every CTA of the cluster has been read (each waited for its own last accumulator): the
        // stages become the meeting place.  Part s of K gets columns [s * cw, (s + 1) * cw) of this thread's COLS,
        // as 16-byte pieces with the row fastest (consecutive lanes write consecutive 16 bytes).
        cluster_sync_all();
        const int cw = COLS / p.splits;
        const uint32_t mine = base + ((split * 2 + half) * (cw / 4) * 128 + lg * 32 + lane) * 16;
#pragma unroll
        for (int c4 = 0; c4 < COLS / 4; ++c4) {
          const int to = (c4 * 4) / cw;
          const uint32_t dst = mapa_shared(mine + (c4 - to * (cw / 4)) * 2048, to * NCTA + cta);
          asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};"
                       ::"r"(dst), "f"(accf[2 * c4].x), "f"(accf[2 * c4].y), "f"(accf[2 * c4 + 1].x), "f"(accf[2 * c4 + 1].y) : "memory");
        }
        cluster_sync_all();
        if (row_ok && col_ok) {
          __nv_bfloat16* orow = p.c + static_cast<long long>(row) * p.ldc + n0 + split * cw;
          for (int c8 = 0; c8 < cw; c8 += 8) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = 0.0f;
            for (int src = 0; src < p.splits; ++src) {
              const float4* q = reinterpret_cast<const float4*>(sm) + ((src * 2 + half) * (cw / 4) + c8 / 4) * 128 + lg * 32 + lane;
              const float4 x = q[0], y = q[128];
              f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
              f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
            }
            uint4 o;
            o.x = pack_bf16x2(f[0], f[1]);
            o.y = pack_bf16x2(f[2], f[3]);
            o.z = pack_bf16x2(f[4], f[5]);
            o.w = pack_bf16x2(f[6], f[7]);
            *reinterpret_cast<uint4*>(orow + c8) = o;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (!one_each) griddep_launch();     // (behind the barrier: one thread of a CTA speaks for all)
  if (bars->abort_flag) drain_after_abort();
  if (clustered) cluster_sync_all();   // nobody leaves while a peer may still signal or read this CTA
  if (warp == 1) {
    tc_fence_after();
    if constexpr (NCTA == 1) tmem_dealloc(tmem, 512);
    else tmem_dealloc_pair(tmem, 512);
  }
  if (tid == 0 && p.status != nullptr && bars->abort_flag) atomicCAS(p.status, 0, FTB_ERR_TIMEOUT);
}

// The shape of a launch: CTAs per tile and parts of K.
struct Shape { int ncta, splits; };
// The shape with the smallest estimate.  Times per K block and wave, and what a split adds, in hundredths of a
// microsecond from a sweep of M = 16 .. 4096, N = 1024 .. 8192, K = 2048 .. 28672 with a cold L2: a 128 x 128 tile 33, a
// 256 x 256 pair 50; a split costs 500 / 600 / 700 at 2 / 4 / 8 parts (cluster launch, two cluster barriers, the
// exchange).  Measured, microseconds (single; single in eight; pair; pair in two):
//   64 x 1024 x 7168: 25.4, 18.4, 32.8, 26.6     64 x 8192 x 3584: 18.5, 59 (four waves), 23.4, 23.3
//   512 x 4096 x 7168: 29.5, -, 38.9, 30.7       1024 x 4096 x 7168: 50.0, -, 39.8, 55.3
//   2048 x 8192 x 3584: 88, -, 74.6, 150         4096 x 8192 x 28672: 1240, -, 913, 1106
// A split runs as one wave only: clusters that queue for SMs cost about ten microseconds a wave.  `whole_k` keeps K in one part.
inline Shape pick_shape(int m, int n, int k, int sms, bool whole_k) {
  const int kb = k / BK;
  Shape best{1, 1};
  long long best_t = -1;
  for (int ncta = 1; ncta <= 2; ++ncta) {
    const long long tiles = static_cast<long long>((m + BM * ncta - 1) / (BM * ncta)) * ((n + 128 * ncta - 1) / (128 * ncta));
    for (int s = 1; s * ncta <= (ncta == 1 ? 8 : 4); s *= 2) {
      // an eighth of the SMs may not host a cluster, a little more not one of eight CTAs (64 x 1920 x 7168 in 120 CTAs 11.7 us, 64 x 2048 x 7168
      // in 128 21.2, in four parts 12.3)
      if (s > 1 && (whole_k || kb < 2 * s || tiles * s * ncta > (s == 8 ? sms * 13 / 16 : sms - sms / 8))) break;
      const long long waves = s > 1 ? 1 : (tiles + sms / ncta - 1) / (sms / ncta);
      const long long t = waves * ((kb + s - 1) / s) * (ncta == 1 ? 33 : 50) + (s == 1 ? 0 : s == 2 ? 500 : s == 4 ? 600 : 700);
      if (best_t < 0 || t < best_t) { best_t = t; best = Shape{ncta, s}; }
    }
  }
  return best;
}
// Tiles of 64 columns instead of 128, with the same parts of K (and bits): where they, too, find an SM each.
// us, 128 / 64 columns: 64 x 1024 x 1024 5.8 / 5.1, 64 x 8192 x 3584 12.0 / 10.6 (row-major weight 12.1 / 10.8), 384 x 3072 x 7168 22.7 / 18.4,
// 64 x 2048 x 7168 in four parts 12.3 / 10.8.
inline bool narrow(const Shape& s, int m, int n, int sms) {
  const long long tiles = static_cast<long long>((m + BM - 1) / BM) * (n / 64);
  return s.ncta == 1 && s.splits <= 4 && tiles * s.splits <= (s.splits > 1 ? sms - sms / 8 : sms);
}

}  // namespace gemm8

// columns of a tile (`halved`: with the rule above), CTAs per tile and parts of K of a launch
void plan_gemm_fp8(int m, int n, int k, bool halved, int sms, int* columns, int* ctas, int* parts) {
  const gemm8::Shape s = gemm8::pick_shape(m, n, k, sms, false);
  *ctas = s.ncta;
  *parts = s.splits;
  *columns = halved && gemm8::narrow(s, m, n, sms) ? 64 : 128 * s.ncta;
}

}  // namespace ftb

using namespace ftb;

static int gemm_fp8_blockscaled(const ftb_gemm_fp8_args* g, bool whole_k, void* stream) {
  if (!g || !g->a || !g->b || !g->c || !g->a_scale || !g->b_scale) { set_last_error("ftb_gemm_fp8_blockscaled: null pointer"); return FTB_ERR_INVALID; }
  if (g->m <= 0 || g->n <= 0 || g->k <= 0 || (g->k % 128) || (g->n % 128)) {
    set_last_error("ftb_gemm_fp8_blockscaled: need k and n multiples of 128 (scale blocks), got m=%d n=%d k=%d", g->m, g->n, g->k);
    return FTB_ERR_INVALID;
  }
  if ((g->lda % 16) || (g->ldb % 16) || (g->ldc % 8) || (reinterpret_cast<uintptr_t>(g->a) & 15) ||
      (reinterpret_cast<uintptr_t>(g->b) & 15) || (reinterpret_cast<uintptr_t>(g->c) & 15)) {
    set_last_error("ftb_gemm_fp8_blockscaled: pointers must be 16-byte aligned, lda/ldb multiples of 16, ldc of 8");
    return FTB_ERR_INVALID;
  }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const gemm8::Shape shape = gemm8::pick_shape(g->m, g->n, g->k, sms, whole_k);
  CUtensorMap tm_a, tm_b;
  const bool bkm = g->b_kmajor != 0;
  const int nb = gemm8::narrow(shape, g->m, g->n, sms) ? 64 : 128;
  const int box_m = g->m < gemm8::BM ? (g->m + 7) & ~7 : gemm8::BM;   // whole swizzle atoms of eight rows
  if (!make_tmap_2d(&tm_a, g->a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, g->m, g->k, g->lda, box_m, 128) ||
      !(bkm ? make_tmap_2d(&tm_b, g->b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, g->n, g->k, g->ldb, nb, 128)
            : make_tmap_2d(&tm_b, g->b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, g->k, g->n, g->ldb, gemm8::BK, nb,
                           nb == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B))) {
    set_last_error("ftb_gemm_fp8_blockscaled: cuTensorMapEncodeTiled failed");
    return FTB_ERR_CUDA;
  }
  const int bm = gemm8::BM * shape.ncta, bn = nb * shape.ncta;
  gemm8::Params p;
  memset(&p, 0, sizeof(p));
  p.m = g->m; p.n = g->n; p.k = g->k;
  p.m_blocks = (g->m + bm - 1) / bm;
  p.n_blocks = (g->n + bn - 1) / bn;
  p.n_tiles = p.m_blocks * p.n_blocks;
  p.kb_total = g->k / gemm8::BK;
  p.splits = shape.splits;
  p.stage_tx = static_cast<uint32_t>(box_m * gemm8::BK + nb * gemm8::BK);
  p.a_scale = g->a_scale; p.b_scale = g->b_scale;
  p.lda_s = g->a_scale_ld; p.ldb_s = g->b_scale_ld;
  p.c = reinterpret_cast<__nv_bfloat16*>(g->c);
  p.ldc = g->ldc;
  p.status = g->status;
  auto kern = shape.ncta == 2 ? (bkm ? gemm8::gemm_fp8_kernel<2, true> : gemm8::gemm_fp8_kernel<2, false>)
              : nb == 64      ? (bkm ? gemm8::gemm_fp8_kernel<1, true, 64> : gemm8::gemm_fp8_kernel<1, false, 64>)
                              : (bkm ? gemm8::gemm_fp8_kernel<1, true> : gemm8::gemm_fp8_kernel<1, false>);
  const int smem = gemm8::SMEM_BYTES + (shape.ncta == 2 && shape.splits == 1 ? gemm8::BOX_BYTES : 0);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(gemm_fp8)");
  const int cl = shape.ncta * shape.splits;
  // persistent groups; with a split every cluster computes one tile and leaves
  const int groups = shape.splits > 1 ? p.n_tiles : (p.n_tiles < sms / shape.ncta ? p.n_tiles : sms / shape.ncta);
  e = launch_overlapped(kern, static_cast<unsigned>(groups) * cl, gemm8::THREADS, smem, reinterpret_cast<cudaStream_t>(stream),
                        static_cast<unsigned>(cl), tm_a, tm_b, p);
  if (e != cudaSuccess) return check_cuda(e, "gemm_fp8 launch");
  return FTB_OK;
}

extern "C" FTB_API int ftb_gemm_fp8_blockscaled(const ftb_gemm_fp8_args* g, void* stream) { return gemm_fp8_blockscaled(g, false, stream); }

extern "C" FTB_API int ftb_gemm_fp8_blockscaled_whole_k(const ftb_gemm_fp8_args* g, void* stream) { return gemm_fp8_blockscaled(g, true, stream); }
