// bf16 product of at most 64 rows with a weight matrix, D[m, n] = sum_k A(m, k) B(n, k), whose contraction is cut in slices: the long
// products of decode steps, which stream the weights once.
//
// The weights are the 128-row operand of the MMA and the rows of A its columns, so a k-block of 64 costs four MMAs for 16 KB of weights
// however few rows there are.  (With A as the 128-row operand and 64 weight rows as columns, as the general kernel has it, a k-block
// takes 0.175 us for 8 KB of weights, from L2 as from DRAM: its copies and MMAs take as long to issue as ones of full size.)
// Each CTA of a cluster has a slice of K; it leaves its sums in its shared memory and then adds its share of the output rows over the
// cluster's CTAs, in slice order.  No workspace in global memory.  The slices are those of the general kernel's plan and are added in
// the same order, so the results are the same bits.
//
//   warp 0      TMA producer     warp 1      MMA issuer     warps 2-9   accumulator -> shared memory     all warps   sums and output
#include "gemm_common.cuh"

namespace b200 {

int make_tmap_bf16_2d(CUtensorMap* tm, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_cols, uint32_t box_rows);

// us, one / 20 / 64 rows, N x K = 2048 x 5504 in four slices: the general kernel 11.8 / 12.5 / 13.0, this 9.1 / 9.9 / 10.9.  Clusters of four and
// more do not fill the chip (16 tiles in eight slices 12.0 us): the caller keeps to those that run at once.
constexpr int FR_MAX_M = 64, FR_MAX_STAGES = 16, FR_THREADS = 320, FR_W_BYTES = BM * BK * 2;
constexpr int FR_SMEM = 227 * 1024;

struct FewRowsParams {
  int M, N, K;
  int xrows;                  // rows of A that are copied: M rounded up to 8
  int stages, splits, b_early, epi, finished;
  void* C;
  long long ldc;
  const void* R;
  long long ldr;
  GemmFinish finish;
  uint32_t* status;
};

// Four columns of the residual row, requested before the sums.
__device__ __forceinline__ uint2 fr_residual(const FewRowsParams& p, int m, int n) {
  const __nv_bfloat16* r = reinterpret_cast<const __nv_bfloat16*>(p.R) + (long long)m * p.ldr + n;
  if (n + 4 <= p.N && (reinterpret_cast<uintptr_t>(r) & 7) == 0) return *reinterpret_cast<const uint2*>(r);
  uint16_t e[4] = {0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (n + j < p.N) e[j] = reinterpret_cast<const uint16_t*>(r)[j];
  return make_uint2(e[0] | (uint32_t)e[1] << 16, e[2] | (uint32_t)e[3] << 16);
}

__device__ __forceinline__ void fr_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 fr_remote(uint32_t local, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ float fr_finish(const FewRowsParams& p, float v, int n) {
  if (!p.finished) return v;
  if (p.finish.bias != nullptr && n < p.N) v += __ldg(p.finish.bias + n);
  if (p.finish.act == ACT_CAP) {
    const float e = exp2f(v * (2.f * 1.4426950408889634f * p.finish.alpha / p.finish.cap));
    return fmaf(-2.f * p.finish.cap, __fdividef(1.f, 1.f + e), p.finish.cap);
  }
  return v * p.finish.alpha;
}

// Four columns of one output row.
__device__ __forceinline__ void fr_store(const FewRowsParams& p, int m, int n, const uint2& res, float (&v)[4]) {
  const long long at = (long long)m * p.ldc + n;
  const bool whole = n + 4 <= p.N;
  if (p.epi == EPI_F32 || p.epi == EPI_F32_ACC) {
    float* c = reinterpret_cast<float*>(p.C) + at;
    if (whole && (reinterpret_cast<uintptr_t>(c) & 15) == 0) {
      float4 o = make_float4(v[0], v[1], v[2], v[3]);
      if (p.epi == EPI_F32_ACC) {
        const float4 b = *reinterpret_cast<const float4*>(c);
        o = make_float4(b.x + o.x, b.y + o.y, b.z + o.z, b.w + o.w);
      }
      *reinterpret_cast<float4*>(c) = o;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n + j < p.N) c[j] = p.epi == EPI_F32_ACC ? c[j] + v[j] : v[j];
    }
    return;
  }
  __nv_bfloat16* c = reinterpret_cast<__nv_bfloat16*>(p.C) + at;
  if (p.epi == EPI_BF16_RES) {
    const float2 a = unpack_bf16x2(res.x), b = unpack_bf16x2(res.y);
    v[0] += a.x; v[1] += a.y; v[2] += b.x; v[3] += b.y;
  }
  if (whole && (reinterpret_cast<uintptr_t>(c) & 7) == 0) {
    *reinterpret_cast<uint2*>(c) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < p.N) c[j] = __float2bfloat16(v[j]);
  }
}

__device__ __forceinline__ void fr_report(const FewRowsParams& p, volatile uint32_t* abort_word, uint32_t code) {
  *abort_word = code;
  if (p.status != nullptr) atomicCAS(p.status, 0u, code | (blockIdx.x << 8));
}

__global__ void __launch_bounds__(FR_THREADS)
gemm_few_rows_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const FewRowsParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_raw);
  uint64_t* empty_bar = full_bar + FR_MAX_STAGES;
  uint64_t* done_bar = empty_bar + FR_MAX_STAGES;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(done_bar + 1);
  volatile uint32_t* abort_word = tmem_holder + 1;
  // The MMA reads a multiple of 16 rows of an A tile: up to 8 beyond it, which are the ring's, for columns that nobody reads.
  uint8_t* smem_x = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1024 + 1023) & ~uintptr_t(1023));
  const int x_bytes = p.xrows * (BK * 2), stages = p.stages;
  uint8_t* smem_w = smem_x + stages * x_bytes;
  float* part = reinterpret_cast<float*>(smem_x);             // (M, 128) sums, when the ring is read no more

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / p.splits, rank = blockIdx.x - tile * p.splits;
  const int n0 = tile * BM;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb_lo = rank * num_kb / p.splits, kb_hi = (rank + 1) * num_kb / p.splits;
  const int cols = (p.M + 15) / 16 * 16;
  uint32_t tmem_cols = 32;
  while (tmem_cols < (uint32_t)cols) tmem_cols *= 2;
  const uint32_t stage_bytes = x_bytes + FR_W_BYTES;

  auto load_w = [&](int stage, int kb) { tma_load_2d(smem_w + stage * FR_W_BYTES, &tmW, &full_bar[stage], kb * BK, n0); };

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    *abort_word = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmX);
    prefetch_tensormap(&tmW);
    if (p.b_early) {
      for (int i = 0; i < stages && kb_lo + i < kb_hi; ++i) {
        mbar_expect_tx(&full_bar[i], stage_bytes);
        load_w(i, kb_lo + i);
      }
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();          // the CTA holds its tensor memory before the kernel after this one may be placed beside it
  tc_fence_after();
  pdl_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        const bool posted = p.b_early && kb - kb_lo < stages;
        if (!posted) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_word)) {
            fr_report(p, abort_word, ERR_WAIT_EMPTY);
            break;
          }
          mbar_expect_tx(&full_bar[stage], stage_bytes);
          load_w(stage, kb);
        }
        tma_load_2d(smem_x + stage * x_bytes, &tmX, &full_bar[stage], kb * BK, 0);
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(BM, cols, false, false);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait(&full_bar[stage], phase, abort_word)) {
          fr_report(p, abort_word, ERR_WAIT_FULL);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t x_base = smem_u32(smem_x + stage * x_bytes), w_base = smem_u32(smem_w + stage * FR_W_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_f16_ss(tmem_base, make_smem_desc(w_base + k * (UMMA_K * 2), 16, 1024), make_smem_desc(x_base + k * (UMMA_K * 2), 16, 1024), idesc,
                      (kb > kb_lo || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok) umma_commit(done_bar);
    }
  } else {
    const int quarter = warp & 3;
    if (mbar_wait(done_bar, 0, abort_word)) {
      tc_fence_after();
#pragma unroll 1
      for (int m0 = (warp - 2) / 4 * 16; m0 < p.M; m0 += 32) {
        uint32_t r[16];
        tmem_ld_32x16(tmem_base + (uint32_t(quarter * 32) << 16) + m0, r);
        tmem_ld_wait();
        float* dst = part + m0 * BM + quarter * 32 + lane;
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (m0 + j < p.M) dst[j * BM] = __uint_as_float(r[j]);
      }
      tc_fence_before();
    } else if (lane == 0) {
      fr_report(p, abort_word, ERR_WAIT_TMEM_FULL);
    }
  }
  __syncwarp();
  fr_cluster_sync();        // all slices' sums are in place
  {
    // rows of this CTA: every splits-th, dealt to the warps; a warp adds ROWS of them at a time, a lane four columns of each
    constexpr int ROWS = 4;
    const uint32_t base = smem_u32(part) + lane * 16;
    const int n = n0 + lane * 4, step = p.splits * (FR_THREADS / 32);
    if (n < p.N) {
      for (int m = rank + p.splits * warp; m < p.M; m += ROWS * step) {
        uint2 res[ROWS];
        float v[ROWS][4] = {};
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
          if (p.epi == EPI_BF16_RES && m + i * step < p.M) res[i] = fr_residual(p, m + i * step, n);
#pragma unroll 4
        for (int s = 0; s < p.splits; ++s) {
          float4 t[ROWS];
#pragma unroll
          for (int i = 0; i < ROWS; ++i)
            if (m + i * step < p.M) t[i] = fr_remote(base + (m + i * step) * (BM * 4), s);
#pragma unroll
          for (int i = 0; i < ROWS; ++i)
            if (m + i * step < p.M) {
              v[i][0] += t[i].x; v[i][1] += t[i].y; v[i][2] += t[i].z; v[i][3] += t[i].w;
            }
        }
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
          if (m + i * step >= p.M) break;
#pragma unroll
          for (int j = 0; j < 4; ++j) v[i][j] = fr_finish(p, v[i][j], n + j);
          fr_store(p, m + i * step, n, res[i], v[i]);
        }
      }
    }
  }
  __syncwarp();
  fr_cluster_sync();        // nobody reads this CTA's shared memory any more
  if (*abort_word != 0) {
    // Give copies that may still be in flight time to land before shared memory is released.
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}

static int launch_few_rows(const CUtensorMap& tmX, const CUtensorMap& tmW, FewRowsParams p, cudaStream_t stream) {
  auto kern = gemm_few_rows_kernel;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FR_SMEM) != cudaSuccess) return -3;
    configured = true;
  }
  const int tiles = (p.N + BM - 1) / BM, num_kb = (p.K + BK - 1) / BK;
  const int mine = (num_kb + p.splits - 1) / p.splits, stage = p.xrows * BK * 2 + FR_W_BYTES;
  int stages = (FR_SMEM - 2048) / stage;
  if (stages > FR_MAX_STAGES) stages = FR_MAX_STAGES;
  if (stages > mine) stages = mine;
  if (stages < 2) stages = 2;
  p.stages = stages;
  int ring = stages * stage;
  const int sums = p.M * BM * 4;
  if (ring < sums) ring = sums;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * p.splits);
  cfg.blockDim = dim3(FR_THREADS);
  cfg.dynamicSmemBytes = ring + 2048;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_pdl_enabled ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, tmX, tmW, p) == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace b200

using namespace b200;

// C (M x N) = act(alpha * (A B^T + bias)) for M <= 64, both operands K-major, K in `splits` slices (2 to 8, two k-blocks each at least).
// epi: 0, 1, 2 or 3 (see GemmEpilogue), EPI_B_STABLE allowed.  finish: as b200_gemm_bf16_finish, without GELU.
extern "C" int b200_gemm_few_rows(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda, long long ldb,
                                  long long ldc, long long ldr, int epi, int splits, const GemmFinish* finish, uint32_t* status,
                                  cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda & 7) || (ldb & 7)) return -10;
  const int b_early = (epi & EPI_B_STABLE) ? 1 : 0;
  epi &= ~EPI_B_STABLE;
  if (M > FR_MAX_M || splits < 2 || splits > 8 || (K + BK - 1) / BK < 2 * splits) return -11;
  if (epi != EPI_BF16 && epi != EPI_F32 && epi != EPI_BF16_RES && epi != EPI_F32_ACC) return -11;
  if (epi == EPI_BF16_RES && R == nullptr) return -11;
  if (finish != nullptr && finish->act == ACT_GELU) return -11;
  FewRowsParams p = {};
  p.M = M; p.N = N; p.K = K; p.xrows = (M + 7) / 8 * 8; p.splits = splits;
  p.b_early = b_early; p.epi = epi; p.finished = finish != nullptr;
  p.C = C; p.ldc = ldc; p.R = R; p.ldr = ldr; p.status = status;
  if (finish != nullptr) p.finish = *finish;
  CUtensorMap tmX, tmW;
  int rc = make_tmap_bf16_2d(&tmX, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, BK, (uint32_t)p.xrows);
  if (rc) return -20 + rc;
  rc = make_tmap_bf16_2d(&tmW, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, BK, BM);
  if (rc) return -30 + rc;
  return launch_few_rows(tmX, tmW, p, stream);
}
