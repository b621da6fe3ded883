// bf16 GEMM for shapes whose 128 x 256 tiles would leave most SMs idle (decode: one row block): C[M,N] = A[M,K] . B[K,N],
// fp32 accumulation in tensor memory, bf16 out.  Same operands and layouts as the persistent kernel (gemm.cu).
//
// Such a product is bound by the bytes of B and by how many SMs fetch them: one SM takes in about 64 bytes per clock
// however deep its pipeline.  So the tile is 128 x 64 or 128 x 128, one tile per CTA, and where even those are few the K axis is
// split over the CTAs of a cluster: their fp32 partial tiles meet in shared memory over DSMEM, every part adds up its
// share of the columns in a fixed order and writes them (no workspace, no second launch, no atomics).
// Measured (us, weights cold in L2, persistent kernel -> this one): 50 x 7168 x 2304 19.2 -> 12.1 (back to back 10.1; 9.4 with A and B loaded
// by two warps and two K blocks per wait of the issuer), 1 x 512 x 2304 15.4 -> 7.0 (four
// parts), 128 x 4096 x 1152 13.4 -> 8.6, 512 x 4096 x 2304 19.9 -> 14.3.  The floor of the first is 5.2 (33 MB); what is left is
// launch, the fill of the pipeline and 64 columns per SM at 64 bytes per clock.
// Roles (224 threads): warps 0 and 6 TMA producers, warp 1 MMA issuer (owns TMEM), warps 2-5 epilogue (TMEM lanes 32 (warp % 4) ..).
#include <cstring>

#include "launch.cuh"
#include "sm100.cuh"
#include "tmap.cuh"

namespace ftb {

void set_last_error(const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

namespace gemm_small {

constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;          // 16384
constexpr int B_BLOCK_BYTES = BK * 128;       // 8192: 64 k-rows x 64 columns
constexpr int THREADS = 224;
template <int BN> struct Cfg {
  static constexpr int STAGES = BN == 64 ? 8 : 6;
  static constexpr int STAGE_BYTES = A_BYTES + BN / 64 * B_BLOCK_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};

struct Params {
  int m, n, n_blocks, kb_total, splits;
  uint32_t stage_tx;          // bytes of A per stage
  __nv_bfloat16* c;
  long long ldc;
  int* status;
};
struct Bars {
  unsigned long long full[8], empty[8], acc_full;
  uint32_t tmem_base;
  int abort_flag;
};

template <int BN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_small_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const Params p) {
  constexpr int STAGES = Cfg<BN>::STAGES, STAGE_BYTES = Cfg<BN>::STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw_addr);
  Bars* bars = reinterpret_cast<Bars*>(sm + STAGES * STAGE_BYTES);
  volatile int* abort_flag = &bars->abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int split = p.splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = blockIdx.x / p.splits;
  const int m_blk = tile / p.n_blocks, n0 = (tile - m_blk * p.n_blocks) * BN;
  const int kb0 = p.kb_total * split / p.splits, kb1 = p.kb_total * (split + 1) / p.splits;

  griddep_launch();
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(smem_u32(&bars->full[s]), 2); mbar_init(smem_u32(&bars->empty[s]), 1); }
    mbar_init(smem_u32(&bars->acc_full), 1);
    fence_mbar_init();
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&bars->tmem_base), BN);
    tmem_relinquish();
    tc_fence_before();
  }
  griddep_wait();
  if (tid == 0) bars->abort_flag = (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
  __syncthreads();
  tc_fence_after();
  // an earlier launch on this status word failed: nothing is loaded or multiplied (every wait returns at once) and nothing written
  const bool dead = bars->abort_flag != 0;
  const uint32_t tmem = bars->tmem_base;

  float acc[BN];
  if (warp == 0 || warp == 6) {
    // B by one warp, A by another: a turn with all loads takes a lone thread longer than the MMAs of a K block
    if (lane == 0) {
      uint32_t s = 0, ph = 1;
      for (int kb = kb0; kb < kb1 && !dead; ++kb) {
        if (!mbar_wait(smem_u32(&bars->empty[s]), ph, abort_flag)) break;
        const uint32_t dst = base + s * STAGE_BYTES, full = smem_u32(&bars->full[s]);
        if (warp == 0) {
          mbar_arrive_expect_tx(full, BN / 64 * B_BLOCK_BYTES);
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_2d(dst + A_BYTES + j * B_BLOCK_BYTES, &tm_b, full, n0 + j * 64, kb * BK);
        } else {
          mbar_arrive_expect_tx(full, p.stage_tx);
          tma_load_2d(dst, &tm_a, full, kb * BK, m_blk * BM);
        }
        if (++s == STAGES) { s = 0; ph ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t kIdesc = umma_idesc(kFmtBF16, BM, BN, 0, 1);
    const uint64_t ad = smem_desc_sw128(base, 16, 1024), bd = smem_desc_sw128(base + A_BYTES, B_BLOCK_BYTES, 1024);
    // Two K blocks at a time, their barriers waited for by different lanes: a wait, an election and a commit cost the warp about 250 cycles
    // between the MMAs of a block, which take 130 to 200.
    const uint32_t full0 = smem_u32(&bars->full[0]), empty0 = smem_u32(&bars->empty[0]);
    uint32_t s = 0, ph = 0;
    static_assert(STAGES % 2 == 0, "both blocks in one phase");
    for (int kb = kb0; kb < kb1 && !dead; kb += 2) {
      const bool two = kb + 1 < kb1;
      if (!__all_sync(0xffffffffu, mbar_wait(full0 + (s + (two ? lane & 1 : 0)) * 8, ph, abort_flag))) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (j == 1 && !two) break;
          const uint64_t off = ((s + j) * STAGE_BYTES) >> 4;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_f16_ss(tmem, ad + off + ((k * 32) >> 4), bd + off + ((k * 2048) >> 4), kIdesc, j == 0 && k == 0 ? (kb > kb0 ? 1u : 0u) : 1u);
          if (kb + j + 1 == kb1) umma_commit(smem_u32(&bars->acc_full));
          else umma_commit(empty0 + (s + j) * 8);
        }
      }
      __syncwarp();
      s += 2;
      if (s == STAGES) { s = 0; ph ^= 1u; }
    }
  } else {
    if (!dead) mbar_wait(smem_u32(&bars->acc_full), 0, abort_flag);
    __syncwarp();
    tc_fence_after();
#pragma unroll
    for (int c0 = 0; c0 < BN; c0 += 32) {
      uint32_t v[32];
      tmem_ld32(tmem_addr(tmem, (warp & 3) * 32, c0), v);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[c0 + j] = __uint_as_float(v[j]);
    }
    tc_fence_before();
  }

  const int row_in = (warp & 3) * 32 + lane, row = m_blk * BM + row_in;
  const bool epilogue = warp >= 2 && warp < 6, writes = epilogue && row < p.m && !*abort_flag;
  auto put8 = [&](const float* f, int col) {                // n is a multiple of 8
    if (n0 + col < p.n) {
      uint4 o;
      o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]);
      o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
      *reinterpret_cast<uint4*>(p.c + static_cast<long long>(row) * p.ldc + n0 + col) = o;
    }
  };
  if (BN != 64 || p.splits == 1) {
    if (writes) {
#pragma unroll
      for (int j = 0; j < BN; j += 8) put8(acc + j, j);
    }
  } else if constexpr (BN == 64) {
    // Every part of K has been multiplied and read from the stages, which become the meeting place: part s gets columns
    // [s cw, (s + 1) cw), as 16-byte pieces with the row fastest.
    cluster_sync_all();
    const int cw = BN / p.splits;
    if (epilogue) {
#pragma unroll
      for (int c4 = 0; c4 < BN / 4; ++c4) {
        const int to = c4 * 4 / cw;
        const uint32_t at = mapa_shared(base + ((split * (cw / 4) + c4 - to * (cw / 4)) * 128 + row_in) * 16, to);
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};"
                     ::"r"(at), "f"(acc[4 * c4]), "f"(acc[4 * c4 + 1]), "f"(acc[4 * c4 + 2]), "f"(acc[4 * c4 + 3]) : "memory");
      }
    }
    cluster_sync_all();
    if (writes) {
      for (int c8 = 0; c8 < cw; c8 += 8) {
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = 0.0f;
        for (int src = 0; src < p.splits; ++src) {
          const float4* q = reinterpret_cast<const float4*>(sm) + (src * (cw / 4) + c8 / 4) * 128 + row_in;
          const float4 x = q[0], y = q[128];
          f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
          f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
        }
        put8(f, split * cw + c8);
      }
    }
  }
  __syncthreads();
  if (bars->abort_flag && !dead) drain_after_abort();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, BN);
  }
  if (tid == 0 && p.status != nullptr && *abort_flag) atomicCAS(p.status, 0, FTB_ERR_TIMEOUT);
}

// Columns of a tile and parts of K; bn = 0: the persistent kernel's shape.
struct Shape { int bn, splits; };
// Taken when the persistent kernel would use at most half of the SMs, with the narrowest tile that still is one wave.  Around
// the line (us, persistent / this one): 512 x 4096 x 2304, 64 tiles of 256, 19.9 / 14.3; 256 x 7168 x 512, 56 tiles, 11.9 / 7.6;
// above it, at 512 x 7168 (112 tiles), the persistent kernel is at its full rate.  K is split as long as the clusters fit and a
// part keeps four K blocks: 128 x 512 x 2304 17.3 / 7.3.  Only tiles of 64 columns can be so few; `whole_k` keeps K in one part.
inline Shape pick_shape(int m, int n, int k, int sms, bool whole_k) {
  const int mb = (m + BM - 1) / BM, kb = (k + BK - 1) / BK;
  if (mb * ((n + 255) / 256) * 2 > sms) return Shape{0, 1};
  const int tiles = mb * ((n + 63) / 64);
  if (tiles > sms) return Shape{128, 1};                     // at most twice the tiles of 256 columns: one wave
  int s = 1;
  while (!whole_k && s < 4 && tiles * s * 2 <= sms - sms / 8 && kb >= 8 * s) s *= 2;   // an eighth of the SMs may not host a cluster
  return Shape{64, s};
}

template <int BN>
static int launch(const void* a, const void* b, void* c, int m, int n, int k, long long lda, long long ldb, long long ldc, int splits,
                  int* status, cudaStream_t st) {
  const int box_m = m < BM ? (m + 7) & ~7 : BM;              // whole swizzle atoms of eight rows
  CUtensorMap tm_a, tm_b;
  if (!make_tmap_2d(&tm_a, a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, m, k, lda, box_m, BK) ||
      !make_tmap_2d(&tm_b, b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, k, n, ldb, BK, 64)) {
    set_last_error("gemm_small: cuTensorMapEncodeTiled failed");
    return FTB_ERR_CUDA;
  }
  Params p;
  memset(&p, 0, sizeof(p));
  p.m = m; p.n = n;
  p.n_blocks = (n + BN - 1) / BN;
  p.kb_total = (k + BK - 1) / BK;
  p.splits = splits;
  p.stage_tx = static_cast<uint32_t>(box_m * BK * 2);
  p.c = static_cast<__nv_bfloat16*>(c);
  p.ldc = ldc;
  p.status = status;
  cudaError_t e = cudaFuncSetAttribute(gemm_small_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::SMEM_BYTES);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(gemm_small)");
  return check_cuda(launch_overlapped(gemm_small_kernel<BN>, static_cast<unsigned>((m + BM - 1) / BM * p.n_blocks * splits), THREADS, Cfg<BN>::SMEM_BYTES, st,
                                      static_cast<unsigned>(splits), tm_a, tm_b, p), "gemm_small launch");
}

}  // namespace gemm_small

// Takes the product if its shape is one of these; *taken says so.
int launch_gemm_small(const void* a, const void* b, void* c, int m, int n, int k, long long lda, long long ldb, long long ldc, int* status,
                      bool whole_k, cudaStream_t st, bool* taken) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const gemm_small::Shape s = gemm_small::pick_shape(m, n, k, sms, whole_k);
  *taken = s.bn != 0;
  if (s.bn == 64) return gemm_small::launch<64>(a, b, c, m, n, k, lda, ldb, ldc, s.splits, status, st);
  if (s.bn == 128) return gemm_small::launch<128>(a, b, c, m, n, k, lda, ldb, ldc, s.splits, status, st);
  return FTB_OK;
}

// Columns of a tile and parts of K of that shape; 0 columns: the persistent kernel's.
void plan_gemm_small(int m, int n, int k, int sms, int* columns, int* parts) {
  const gemm_small::Shape s = gemm_small::pick_shape(m, n, k, sms, false);
  *columns = s.bn;
  *parts = s.splits;
}

}  // namespace ftb
