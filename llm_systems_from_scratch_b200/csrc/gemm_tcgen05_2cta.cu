// bf16 GEMM on CTA pairs (tcgen05 cta_group::2): two SMs of a cluster cooperate on one 256 x 256 output
// tile.  Each CTA loads its own 128 rows of A and one half (128 rows) of the B tile; the tensor cores of
// both SMs consume both halves of B, so per FLOP a CTA writes and reads a third less shared memory than
// the single-CTA kernel in gemm_tcgen05.cu, whose tensor pipe is capped by shared-memory bandwidth
// (TMA writes + MMA operand reads need 192 B/clk/SM there, 128 here).
//
// Roles (per CTA): warp 0 TMA producer, warp 1 MMA issuer (leader CTA only; both allocate TMEM),
// warps 2-5 epilogue.  Synchronisation inside the pair:
//   full[s]        lives in the leader; both CTAs' TMA loads complete their bytes on it
//   empty[s]       one per CTA; the leader's tcgen05.commit arrives on both (commit multicast)
//   tmem_full[a]   one per CTA; commit multicast
//   tmem_empty[a]  lives in the leader; the 2 x 128 epilogue threads of the pair arrive on it
// TMA loads are ordinary (non-multicast) loads.  Every wait is bounded (see ptx.cuh).
//
// Grouped rows (experts' products of prompts): a pair takes two neighbouring 128-row tiles of the same group, the 256 columns as above.  Single
// CTAs are held up by their shared memory as described; a prompt of 8192 rows, top 2 of 8 experts of 2752 x 2048: 1175 -> 1330 TFLOP/s in
// the step.  What it cannot use is the second half of a group's last pair (4 of 68 on average there).
//
// Last wave (weight gradients): with T tiles on P pairs, the T % P tiles of the last wave are contracted in `splits` slices of K each, on all
// pairs; the partial tiles go to a workspace and pair_tail_sum_kernel adds them in slice order (no atomics: reproducible).
#include "gemm_common.cuh"

namespace b200 {

int make_tmap_bf16_2d(CUtensorMap* tm, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_cols,
                      uint32_t box_rows);
int make_tmap_out_2d(CUtensorMap* tm, bool f32, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld,
                     uint32_t box_cols, uint32_t box_rows);

constexpr int P_BN = 256;        // tile columns of the pair
constexpr int P_HALF = 128;      // B rows held by one CTA
template <int V>
struct IntC {
  static constexpr int value = V;
};

constexpr int P_STAGES = 6;
constexpr int P_THREADS = 256;    // TMA warp, MMA warp, 4 epilogue warps, 2 gather-copy warps
constexpr int P_A_BYTES = BM * BK * 2;       // 16 KB
constexpr int P_B_BYTES = P_HALF * BK * 2;   // 16 KB
constexpr int P_DATA = P_STAGES * (P_A_BYTES + P_B_BYTES);
// Output staging: every epilogue warp owns two slabs of 32 rows x 128 bytes (128-byte swizzle) that it fills from
// registers and hands to a TMA store, so global writes are whole 128-byte lines issued by the copy engine.
constexpr int P_SLAB = 32 * 128;
constexpr int P_STAGING = 4 * 2 * P_SLAB;   // 32 KB
constexpr int P_BARS = 2 * P_STAGES + 4;
constexpr int P_SMEM = P_DATA + P_STAGING + P_BARS * 8 + 16 + 160 + 1024;   // 160: ReduceSmem of the copy warps
// Grouped launches: up to P_LIST pairs of row tiles, two bytes each, and their number.
constexpr int P_LIST = 800;
constexpr int P_SMEM_GROUPED = P_SMEM + P_LIST * 2 + 16;
static_assert(P_SMEM_GROUPED <= 232448, "shared memory budget of one CTA");

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* addr) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `local_smem_addr` inside CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-D tiled load whose byte count is signalled on a barrier given by its shared::cluster address
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tm, uint32_t bar_cluster_addr,
                                                 int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* holder, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_pair_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on the barrier at the same shared-memory offset in both CTAs of the pair once the MMAs issued so
// far have completed
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}

// The row tiles that one pair works on together: two neighbours of the same group, or (P_ALONE) the last one of a group with an odd number of
// them, which both CTAs then load and one stores.  Called by one warp; entries go to `list`, their number is returned.
constexpr uint32_t P_ALONE = 0x8000;
__device__ __forceinline__ int list_pairs(const int* __restrict__ tile_group, int tiles, uint16_t* list) {
  const int lane = threadIdx.x & 31;
  int count = 0, run = 0, before = -1;      // first tile of the current run; group of the tile in front
  for (int t0 = 0; t0 < tiles; t0 += 32) {
    const int t = t0 + lane;
    const int g = t < tiles ? tile_group[t] : -1, next = t + 1 < tiles ? tile_group[t + 1] : -1;
    int prev = __shfl_up_sync(0xffffffffu, g, 1);
    if (lane == 0) prev = before;
    int start = g != prev ? t : lane == 0 ? run : 0;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const int other = __shfl_up_sync(0xffffffffu, start, o);
      if (lane >= o) start = max(start, other);
    }
    const bool first = g >= 0 && ((t - start) & 1) == 0;
    const uint32_t those = __ballot_sync(0xffffffffu, first);
    if (first) list[count + __popc(those & ((1u << lane) - 1u))] = (uint16_t)(t | (next != g ? P_ALONE : 0u));
    count += __popc(those);
    run = __shfl_sync(0xffffffffu, start, 31);
    before = __shfl_sync(0xffffffffu, g, 31);
  }
  return count;
}

// GROUPED: the 128-row tiles of A belong to the groups of rows of B in p.tile_group (negative: skipped); see list_pairs.
// ROPE: the rotated QKV projection with TMA stores (p.rope_cs set), and no other epilogue.
template <bool A_MN, bool B_MN, bool GROUPED = false, bool ROPE = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmH,
                      const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + P_STAGES * P_A_BYTES;
  uint8_t* smem_out = smem + P_DATA;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + P_DATA + P_STAGING);
  uint64_t* empty_bar = full_bar + P_STAGES;
  uint64_t* tmem_full = empty_bar + P_STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile uint32_t* abort_word = tmem_holder + 1;
  ReduceSmem* reduce_smem = reinterpret_cast<ReduceSmem*>(tmem_holder + 4);
  static_assert(sizeof(ReduceSmem) <= 144, "ReduceSmem must fit the space reserved behind the barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  constexpr uint32_t TMEM_COLS = 512;   // two accumulators of 256 columns

  if (threadIdx.x == 0) {
    for (int s = 0; s < P_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 256);
    }
    *abort_word = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmB);
    if (p.tma_store && p.C != nullptr) prefetch_tensormap(&tmC);          // without C its map was never made
    if (p.tma_store && (p.swiglu_f > 0 || p.epi == EPI_SWIGLU_BWD)) prefetch_tensormap(&tmH);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_holder, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // the peer's barriers are initialised before anything can arrive on them
  tc_fence_after();
  // From here on global memory is read and written.  The next kernel is not let in early: its CTAs beside the tiles cost more than its
  // launch (a training step of 180 launches 3963 us with, 3838 without; prompts of 2048 tokens 5630, 5370; of 8192 tokens 18890 either way).
  pdl_wait();
  const uint32_t tmem_base = *tmem_holder;

  int num_m_tiles = p.num_m_tiles;
  uint16_t* pair_list = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(tmem_holder) + 176);
  int* pair_count = reinterpret_cast<int*>(pair_list + P_LIST);
  if (GROUPED) {
    if (warp == 2) {
      const int n = list_pairs(p.tile_group, p.M / BM, pair_list);
      if (lane == 0) *pair_count = n;
    }
    __syncthreads();
    num_m_tiles = *pair_count;
  }
  // first row of this CTA's row tile of a unit, and whether it stores its rows
  auto tile_row = [&](int m_blk, bool& stored) {
    stored = true;
    if (!GROUPED) return m_blk * 256 + (int)rank * BM;
    const uint32_t e = pair_list[m_blk];
    stored = rank == 0 || !(e & P_ALONE);
    return (int)((e & (P_ALONE - 1)) + (stored ? rank : 0)) * BM;
  };
  const int num_tiles = num_m_tiles * p.num_n_tiles;   // tiles of 256 x 256
  const int num_kb = (p.K + BK - 1) / BK;
  // work unit: a whole tile, or behind the first full_tiles of them a slice of K of a tile (`part`: which partial tile it leaves, else -1)
  const int full_tiles = p.splits > 1 ? p.full_tiles : num_tiles;
  const int num_units = full_tiles + (num_tiles - full_tiles) * p.splits;
  auto unit_tile = [&](int unit, int& kb_lo, int& kb_hi, int& part) {
    part = unit - full_tiles;
    kb_lo = 0;
    kb_hi = num_kb;
    if (part < 0) return unit;
    const int t = part / p.splits, sl = part - t * p.splits;
    kb_lo = sl * num_kb / p.splits;
    kb_hi = (sl + 1) * num_kb / p.splits;
    return full_tiles + t;
  };
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

  if (warp == 0) {
    if (elect_one()) {   // elect.sync keeps the issuing code warp-uniform (descriptors in uniform registers)
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      if (p.wait_counter != nullptr) {
        // operand B is being gathered by another kernel: wait (bounded) until every slice has landed
        const uint64_t t0 = globaltimer_ns();
        while ((int32_t)(ld_acquire_gpu(p.wait_counter) - p.wait_value) < 0) {
          if (globaltimer_ns() - t0 > p.wait_limit_ns) {
            report(p, abort_word, ERR_WAIT_FLAG);
            ok = false;
            break;
          }
          __nanosleep(128);
        }
        asm volatile("fence.proxy.async.global;" ::: "memory");   // generic-proxy writes -> TMA reads
      }
      for (int unit = pair; unit < num_units && ok; unit += num_pairs) {
        int m_blk, n_blk, kb_lo, kb_hi, part;
        tile_coords(unit_tile(unit, kb_lo, kb_hi, part), p, num_m_tiles, m_blk, n_blk);
        bool stored;
        const int m0 = tile_row(m_blk, stored);
        // SwiGLU mode: the leader loads 128 gate rows, its peer the matching 128 up rows (F rows further down)
        int n0 = p.swiglu_f > 0 ? n_blk * P_HALF + (int)rank * p.swiglu_f : n_blk * P_BN + (int)rank * P_HALF;
        if (GROUPED) n0 += __ldg(p.tile_group + m0 / BM) * p.group_rows;
        for (int kb = kb_lo; kb < kb_hi; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_word)) {
            report(p, abort_word, ERR_WAIT_EMPTY);
            ok = false;
            break;
          }
          if (leader) mbar_expect_tx(&full_bar[stage], 2 * (P_A_BYTES + P_B_BYTES));
          const uint32_t bar = map_to_cta(smem_u32(&full_bar[stage]), 0);   // the leader's barrier
          uint8_t* a_dst = smem_a + stage * P_A_BYTES;
          uint8_t* b_dst = smem_b + stage * P_B_BYTES;
          const int k0 = kb * BK;
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(a_dst + j * 8192, &tmA, bar, m0 + j * 64, k0);
          } else {
            tma_load_2d_pair(a_dst, &tmA, bar, k0, m0);
          }
          if (B_MN) {
#pragma unroll
            for (int j = 0; j < P_HALF / 64; ++j) tma_load_2d_pair(b_dst + j * 8192, &tmB, bar, n0 + j * 64, k0);
          } else {
            tma_load_2d_pair(b_dst, &tmB, bar, k0, n0);
          }
          if (++stage == P_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (leader && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(256, P_BN, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0, acc_phase[2] = {0, 0};
      int local = 0;
      bool ok = true;
      for (int unit = pair; unit < num_units && ok; unit += num_pairs, ++local) {
        int kb_lo, kb_hi, part;
        unit_tile(unit, kb_lo, kb_hi, part);
        const int acc = local & 1;
        if (!mbar_wait(&tmem_empty[acc], acc_phase[acc] ^ 1, abort_word)) {
          report(p, abort_word, ERR_WAIT_TMEM_EMPTY);
          ok = false;
          break;
        }
        acc_phase[acc] ^= 1;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * P_BN;
        for (int kb = kb_lo; kb < kb_hi; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_word)) {
            report(p, abort_word, ERR_WAIT_FULL);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_base = smem_u32(smem_a + stage * P_A_BYTES);
          const uint32_t b_base = smem_u32(smem_b + stage * P_B_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t a_desc = A_MN ? make_smem_desc(a_base + k * (UMMA_K * 128), 8192, 1024)
                                         : make_smem_desc(a_base + k * (UMMA_K * 2), 16, 1024);
            const uint64_t b_desc = B_MN ? make_smem_desc(b_base + k * (UMMA_K * 128), 8192, 1024)
                                         : make_smem_desc(b_base + k * (UMMA_K * 2), 16, 1024);
            umma_pair_f16_ss(d_tmem, a_desc, b_desc, idesc, (kb > kb_lo || k > 0) ? 1u : 0u);
          }
          umma_commit_pair(&empty_bar[stage]);   // frees this stage in both CTAs
          if (++stage == P_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit_pair(&tmem_full[acc]);
      }
    }
  } else if (warp >= 6) {
    // ---------------------------------------------------------------- gather-copy warps
    if (p.gather.dst != nullptr) {
      const GatherTask& g = p.gather;
      const int t = (warp - 6) * 32 + lane;                  // 0..63
      const size_t stride = (size_t)gridDim.x * 64;
      // one load from every peer in flight per thread (times 4 / 2 strides for 2 / 4 ranks)
      const size_t first = (size_t)blockIdx.x * 64 + t;
      auto body = [&](auto world_c, auto unroll_c) {
        constexpr int W = decltype(world_c)::value, U = decltype(unroll_c)::value;
        size_t i = first;
        for (; i + (U - 1) * stride < g.shard_vec; i += U * stride) {
          uint4 v[W][U];
#pragma unroll
          for (int k = 0; k < W; ++k)
#pragma unroll
            for (int u = 0; u < U; ++u) v[k][u] = g.src[(g.rank + k) % W][i + u * stride];
#pragma unroll
          for (int k = 0; k < W; ++k)
#pragma unroll
            for (int u = 0; u < U; ++u) g.dst[(size_t)((g.rank + k) % W) * g.shard_vec + i + u * stride] = v[k][u];
        }
        for (; i < g.shard_vec; i += stride)
#pragma unroll
          for (int k = 0; k < W; ++k) {
            const int pr = (g.rank + k) % W;
            g.dst[(size_t)pr * g.shard_vec + i] = g.src[pr][i];
          }
      };
      if (g.world == 8) body(IntC<8>{}, IntC<2>{});
      else if (g.world == 4) body(IntC<4>{}, IntC<4>{});
      else if (g.world == 2) body(IntC<2>{}, IntC<8>{});
      else
        for (int k = 0; k < g.world; ++k) {
          const int pr = (g.rank + k) % g.world;
          for (size_t i = first; i < g.shard_vec; i += stride) g.dst[(size_t)pr * g.shard_vec + i] = g.src[pr][i];
        }
      asm volatile("bar.sync 2, 64;" ::: "memory");         // both copy warps are done
      if (t == 0 && g.done != nullptr) {
        __threadfence();
        atomicAdd(g.done, 1u);
      }
    }
    // ---------------------------------------------------------------- carried reduce-scatter
    // The gradient staging of an earlier unit is reduced over all peers (and optionally fed to AdamW) by the same
    // 64 threads of every CTA while the tensor cores of this kernel keep working.
    if (p.reduce.n > 0) {
      const int t = (warp - 6) * 32 + lane;
      if (p.reduce.mode == 0) reduce_scatter_any<0>(p.reduce, t, 64, blockIdx.x, gridDim.x, 3, reduce_smem);
      else reduce_scatter_any<1>(p.reduce, t, 64, blockIdx.x, gridDim.x, 3, reduce_smem);
    }
  } else {
    const int quarter = warp & 3;
    uint32_t acc_phase[2] = {0, 0};
    int local = 0;
    uint32_t out_slab = 0;
    bool ok = true;
    for (int unit = pair; unit < num_units && ok; unit += num_pairs, ++local) {
      int m_blk, n_blk, kb_lo, kb_hi, part;
      tile_coords(unit_tile(unit, kb_lo, kb_hi, part), p, num_m_tiles, m_blk, n_blk);
      const int acc = local & 1;
      bool stored;
      const int row0 = tile_row(m_blk, stored) + quarter * 32;
      const int row = stored ? row0 + lane : p.M;
      const int n0 = n_blk * P_BN;
      // ROPE: cosines and sines of 64 columns, requested before the accumulator is waited for; where heads have 64 columns or 32 they serve the
      // whole row.  With short contractions the epilogue is the longer part of a tile, and most of it were these loads (rotated QKV
      // projection of 16384 rows, us: width 512, heads of 32 42.7 -> 31.6; width 768, heads of 64 73.0 -> 50.5; width 2048, heads of 128 284 -> 270).  An instance of its own: the
      // gated epilogues miss the registers otherwise.
      float4 turn[ROPE ? 16 : 1];
      int turn_at = -1;       // column of a head that they start with
      auto load_turn = [&](int col) {
        if constexpr (ROPE) {
          if (turn_at == col % p.rope_dh) return;
          turn_at = col % p.rope_dh;
          load_rope_columns(p.rope_cs, p.rope_ctx, p.rope_dh, row % p.rope_seq, col, turn);
          load_rope_columns(p.rope_cs, p.rope_ctx, p.rope_dh, row % p.rope_seq, col + 32, turn + 8);
        }
      };
      if (ROPE && n0 < 2 * p.rope_d) load_turn(n0);
      if (!mbar_wait(&tmem_full[acc], acc_phase[acc], abort_word)) {
        if (lane == 0) report(p, abort_word, ERR_WAIT_TMEM_FULL);
        ok = false;
        break;
      }
      acc_phase[acc] ^= 1;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16) + acc * P_BN;
      // registers -> swizzled slab in shared memory -> TMA store (or TMA add).  Row `lane` of a slab is one 128-byte
      // line; its 16-byte pieces are permuted by (row & 7) as the 128-byte swizzle of the tensor maps expects, which
      // also makes the st.shared.v4 of a quarter warp conflict-free.  A warp alternates between its two slabs and
      // waits, before refilling one, until the store that last used it has read it.
      const int y0 = part < 0 ? row0 : part * 256 + (int)rank * BM + quarter * 32;      // row of the output or of the workspace
      auto emit = [&](const CUtensorMap* tm, int x, const uint32_t (&o)[32], bool add) {
        uint8_t* slab = smem_out + ((warp - 2) * 2 + (out_slab & 1)) * P_SLAB;
        ++out_slab;
        if (lane == 0) tma_store_wait_read<1>();
        __syncwarp();
        uint8_t* line = slab + lane * 128;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4*>(line + ((j ^ (lane & 7)) << 4)) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (row0 < p.M && stored) {
            if (add) tma_reduce_add_2d(tm, slab, x, y0);
            else tma_store_2d(tm, slab, x, y0);
          }
          tma_store_commit();
        }
      };
      if (part >= 0) {
#pragma unroll 1
        for (int c = 0; c < P_BN / 32; ++c) {
          if (n0 + c * 32 >= p.N) break;
          uint32_t o[32];
          tmem_ld_32x32(taddr + c * 32, o);
          tmem_ld_wait();
          emit(&tmH, c * 32, o, false);
        }
        tc_fence_before();
        mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[acc]), 0));
        continue;
      }
      if (!ROPE && p.swiglu_f > 0 && p.C == nullptr) {
        // the product alone: nothing is rounded before it
        const int col = n_blk * P_HALF;
#pragma unroll 1
        for (int c = 0; c < P_HALF / 64; ++c) {
          if (col + c * 64 >= p.swiglu_f) break;
          uint32_t o[32];
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t g[32], u[32];
            tmem_ld_32x32(taddr + c * 64 + half * 32, g);
            tmem_ld_32x32(taddr + P_HALF + c * 64 + half * 32, u);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float g0 = __uint_as_float(g[2 * j]), g1 = __uint_as_float(g[2 * j + 1]);
              o[half * 16 + j] = pack_bf16x2(__fdividef(g0, 1.f + __expf(-g0)) * __uint_as_float(u[2 * j]),
                                             __fdividef(g1, 1.f + __expf(-g1)) * __uint_as_float(u[2 * j + 1]));
            }
          }
          emit(&tmH, col + c * 64, o, false);
        }
      } else if (!ROPE && p.swiglu_f > 0 && p.tma_store) {
        // accumulator columns [0,128) are gate_j, [128,256) the matching up_j; three outputs per 64 columns
        const int col = n_blk * P_HALF;
#pragma unroll 1
        for (int c = 0; c < P_HALF / 64; ++c) {
          if (col + c * 64 >= p.swiglu_f) break;       // gate columns past F are up rows
          uint32_t og[32], ou[32];
          {
            uint32_t r0[32], r1[32];
            tmem_ld_32x32(taddr + c * 64, r0);
            tmem_ld_32x32(taddr + c * 64 + 32, r1);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              og[j] = pack_bf16x2(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1]));
              og[16 + j] = pack_bf16x2(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1]));
            }
          }
          emit(&tmC, col + c * 64, og, false);
          {
            uint32_t r0[32], r1[32];
            tmem_ld_32x32(taddr + P_HALF + c * 64, r0);
            tmem_ld_32x32(taddr + P_HALF + c * 64 + 32, r1);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              ou[j] = pack_bf16x2(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1]));
              ou[16 + j] = pack_bf16x2(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1]));
            }
          }
          emit(&tmC, p.swiglu_f + col + c * 64, ou, false);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            // as the stand-alone kernel: silu on the bf16-rounded gate, times the rounded up (fast division)
            const float2 gf = unpack_bf16x2(og[j]), uf = unpack_bf16x2(ou[j]);
            og[j] = pack_bf16x2(__fdividef(gf.x, 1.f + __expf(-gf.x)) * uf.x, __fdividef(gf.y, 1.f + __expf(-gf.y)) * uf.y);
          }
          emit(&tmH, col + c * 64, og, false);
        }
      } else if (!ROPE && p.swiglu_f > 0) {
        // accumulator columns [0,128) are gate_j, [128,256) the matching up_j
        const int col = n_blk * P_HALF;
#pragma unroll 1
        for (int c = 0; c < P_HALF / 32; ++c) {
          if (col + c * 32 >= p.swiglu_f) break;
          uint32_t g[32], u[32];
          tmem_ld_32x32(taddr + c * 32, g);
          tmem_ld_32x32(taddr + P_HALF + c * 32, u);
          tmem_ld_wait();
          if (row < p.M) {
            __nv_bfloat16* cg = reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)row * p.ldc + col + c * 32;
            __nv_bfloat16* cu = cg + p.swiglu_f;
            __nv_bfloat16* ch = reinterpret_cast<__nv_bfloat16*>(p.H) + (long long)row * p.ldh + col + c * 32;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t og[4], ou[4], oh[4];
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                og[t] = pack_bf16x2(__uint_as_float(g[j * 8 + 2 * t]), __uint_as_float(g[j * 8 + 2 * t + 1]));
                ou[t] = pack_bf16x2(__uint_as_float(u[j * 8 + 2 * t]), __uint_as_float(u[j * 8 + 2 * t + 1]));
                // as the stand-alone kernel: silu on the bf16-rounded gate, times the rounded up (fast division)
                const float2 gf = unpack_bf16x2(og[t]), uf = unpack_bf16x2(ou[t]);
                oh[t] = pack_bf16x2(__fdividef(gf.x, 1.f + __expf(-gf.x)) * uf.x, __fdividef(gf.y, 1.f + __expf(-gf.y)) * uf.y);
              }
              *reinterpret_cast<uint4*>(cg + j * 8) = make_uint4(og[0], og[1], og[2], og[3]);
              *reinterpret_cast<uint4*>(cu + j * 8) = make_uint4(ou[0], ou[1], ou[2], ou[3]);
              *reinterpret_cast<uint4*>(ch + j * 8) = make_uint4(oh[0], oh[1], oh[2], oh[3]);
            }
          }
        }
      } else if (!ROPE && p.tma_store && p.epi == EPI_SWIGLU_BWD) {
        // acc = dh (this row, 256 columns); R holds gate | up; d(gate) goes out through tmC, d(up) through tmH.
        // The gate / up pieces of the next 32 columns are fetched while the current 32 are computed, so that the
        // row-strided loads are off the critical path; two 32-column halves fill one 64-column slab per output.
        const __nv_bfloat16* grow = reinterpret_cast<const __nv_bfloat16*>(p.R) + (long long)row * p.ldr;
        uint8_t* slab_g = smem_out + (warp - 2) * 2 * P_SLAB;
        uint8_t* slab_u = slab_g + P_SLAB;
        const bool row_ok = row < p.M;
        uint4 gq[4], uq[4];
        auto load_gu = [&](int col, uint4 (&g)[4], uint4 (&u)[4]) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const bool in = row_ok && col + j * 8 < p.N;     // N is a multiple of 8
            g[j] = in ? __ldg(reinterpret_cast<const uint4*>(grow + col + j * 8)) : make_uint4(0, 0, 0, 0);
            u[j] = in ? __ldg(reinterpret_cast<const uint4*>(grow + p.N + col + j * 8)) : make_uint4(0, 0, 0, 0);
          }
        };
        load_gu(n0, gq, uq);
#pragma unroll
        for (int h = 0; h < P_BN / 32; ++h) {
          const int col = n0 + h * 32;
          if (col >= p.N) break;
          uint4 gn[4], un[4];
          if (h + 1 < P_BN / 32) load_gu(col + 32, gn, un);
          uint32_t r[32];
          tmem_ld_32x32(taddr + h * 32, r);
          tmem_ld_wait();
          if ((h & 1) == 0) {
            if (lane == 0) tma_store_wait_read<0>();      // both slabs have been read by the previous stores
            __syncwarp();
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t gg[4] = {gq[j].x, gq[j].y, gq[j].z, gq[j].w}, uu[4] = {uq[j].x, uq[j].y, uq[j].z, uq[j].w};
            uint32_t og[4], ou[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              // as the stand-alone kernel: dh is rounded to bf16 first, gate and up are read as bf16
              const float2 g = unpack_bf16x2(gg[t]), u = unpack_bf16x2(uu[t]);
              const float2 d = unpack_bf16x2(pack_bf16x2(__uint_as_float(r[j * 8 + 2 * t]), __uint_as_float(r[j * 8 + 2 * t + 1])));
              const float s0 = __fdividef(1.f, 1.f + __expf(-g.x)), s1 = __fdividef(1.f, 1.f + __expf(-g.y));
              const float l0 = g.x * s0, l1 = g.y * s1;
              og[t] = pack_bf16x2(d.x * u.x * (s0 + l0 * (1.f - s0)), d.y * u.y * (s1 + l1 * (1.f - s1)));
              ou[t] = pack_bf16x2(d.x * l0, d.y * l1);
            }
            const int piece = (((h & 1) * 4 + j) ^ (lane & 7)) << 4;
            *reinterpret_cast<uint4*>(slab_g + lane * 128 + piece) = make_uint4(og[0], og[1], og[2], og[3]);
            *reinterpret_cast<uint4*>(slab_u + lane * 128 + piece) = make_uint4(ou[0], ou[1], ou[2], ou[3]);
          }
          if ((h & 1) == 1 || col + 32 >= p.N) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (row0 < p.M) {
                tma_store_2d(&tmC, slab_g, n0 + (h >> 1) * 64, row0);
                tma_store_2d(&tmH, slab_u, n0 + (h >> 1) * 64, row0);
              }
              tma_store_commit();
            }
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            gq[j] = gn[j];
            uq[j] = un[j];
          }
        }
        out_slab = 0;     // both slabs are in flight: the next emit() must wait for them (it waits for all but one)
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
      } else if (ROPE || p.tma_store) {
        const bool out_f32 = !ROPE && (p.epi == EPI_F32 || p.epi == EPI_F32_ACC);
        const int cols_per_chunk = out_f32 ? 32 : 64;
        const int nchunks = P_BN / cols_per_chunk;
#pragma unroll 1
        for (int c = 0; c < nchunks; ++c) {
          const int col = n0 + c * cols_per_chunk;
          if (col >= p.N) break;
          uint32_t o[32];
          if (out_f32) {
            tmem_ld_32x32(taddr + c * 32, o);
            tmem_ld_wait();
            if (p.finished) epilogue_finish(p, col, p.N - col, o);
          } else {
            uint32_t r0[32], r1[32];
            tmem_ld_32x32(taddr + c * 64, r0);
            tmem_ld_32x32(taddr + c * 64 + 32, r1);
            tmem_ld_wait();
            if (p.finished) {
              epilogue_finish(p, col, p.N - col, r0);
              epilogue_finish(p, col + 32, p.N - col - 32, r1);
            }
            if constexpr (ROPE) {
              if (col < 2 * p.rope_d) {      // N = 3 * rope_d, heads are multiples of 32 columns
                load_turn(col);
                apply_rope_columns(turn, r0);
                apply_rope_columns(turn + 8, r1);
              }
            }
            if (!ROPE && p.epi == EPI_BF16_RES && row < p.M) {
              const __nv_bfloat16* rp = reinterpret_cast<const __nv_bfloat16*>(p.R) + (long long)row * p.ldr + col;
              if (col + 64 <= p.N && (p.ldr & 7) == 0 && (reinterpret_cast<uintptr_t>(p.R) & 15) == 0) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const uint4 rv = *reinterpret_cast<const uint4*>(rp + j * 8);
                  const uint32_t rr[4] = {rv.x, rv.y, rv.z, rv.w};
                  uint32_t* a = j < 4 ? r0 + j * 8 : r1 + (j - 4) * 8;
#pragma unroll
                  for (int t = 0; t < 4; ++t) {
                    const float2 f = unpack_bf16x2(rr[t]);
                    a[2 * t] = __float_as_uint(__uint_as_float(a[2 * t]) + f.x);
                    a[2 * t + 1] = __float_as_uint(__uint_as_float(a[2 * t + 1]) + f.y);
                  }
                }
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) {      // static register indices; the column test predicates the loads
                  if (col + j < p.N) r0[j] = __float_as_uint(__uint_as_float(r0[j]) + __bfloat162float(rp[j]));
                  if (col + 32 + j < p.N) r1[j] = __float_as_uint(__uint_as_float(r1[j]) + __bfloat162float(rp[32 + j]));
                }
              }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              o[j] = pack_bf16x2(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1]));
              o[16 + j] = pack_bf16x2(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1]));
            }
          }
          emit(&tmC, col, o, p.epi == EPI_F32_ACC);
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < P_BN / 32; ++c) {
          if (n0 + c * 32 >= p.N) break;
          uint32_t r[32];
          tmem_ld_32x32(taddr + c * 32, r);
          tmem_ld_wait();
          epilogue_store(p, row, n0 + c * 32, r);
        }
      }
      tc_fence_before();
      mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[acc]), 0));   // the leader owns this barrier
    }
    if (p.tma_store && lane == 0) tma_store_wait<0>();   // shared memory stays valid until the last store has left
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*abort_word != 0) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();      // neither CTA releases TMEM or exits while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// The partial tiles of the last wave, added in slice order: block (tile, 8 rows), two rows and one float4 per thread.
template <typename OUT>
__global__ void __launch_bounds__(256)
pair_tail_sum_kernel(const float4* __restrict__ ws, OUT* __restrict__ C, const GemmParams p) {
  pdl_sync();
  const int t = blockIdx.x >> 5, r0 = (blockIdx.x & 31) * 8 + (threadIdx.x >> 6), c = (threadIdx.x & 63) * 4;
  int m_blk, n_blk;
  tile_coords(p.full_tiles + t, p, m_blk, n_blk);
  const int col = n_blk * P_BN + c;
  if (col >= p.N) return;
  const float4* src = ws + ((size_t)t * p.splits * 256 + r0) * 64 + (c >> 2);
  float4 sum[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
  for (int s0 = 0; s0 < p.splits; s0 += 4) {
    float4 v[4][2];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (s0 + u < p.splits) {
        v[u][0] = __ldcs(src + (size_t)(s0 + u) * 256 * 64);
        v[u][1] = __ldcs(src + (size_t)(s0 + u) * 256 * 64 + 4 * 64);
      }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (s0 + u < p.splits) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          sum[k].x += v[u][k].x; sum[k].y += v[u][k].y; sum[k].z += v[u][k].z; sum[k].w += v[u][k].w;
        }
      }
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int row = m_blk * 256 + r0 + 4 * k;
    if (row >= p.M) break;
    OUT* dst = C + (long long)row * p.ldc + col;
    if constexpr (sizeof(OUT) == 2) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(sum[k].x, sum[k].y), pack_bf16x2(sum[k].z, sum[k].w));
    } else {
      if (p.epi == EPI_F32_ACC) {
        const float4 o = *reinterpret_cast<const float4*>(dst);
        sum[k].x += o.x; sum[k].y += o.y; sum[k].z += o.z; sum[k].w += o.w;
      }
      *reinterpret_cast<float4*>(dst) = sum[k];
    }
  }
}

template <bool A_MN, bool B_MN, bool GROUPED = false, bool ROPE = false>
static int launch_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const CUtensorMap& tmH,
                       GemmParams p, int sms, cudaStream_t stream) {
  auto kern = gemm_bf16_pair_kernel<A_MN, B_MN, GROUPED, ROPE>;
  constexpr int SMEM = GROUPED ? P_SMEM_GROUPED : P_SMEM;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) return -3;
    configured = true;
  }
  p.num_m_tiles = (p.M + 255) / 256;
  p.num_n_tiles = p.swiglu_f > 0 ? (p.swiglu_f + P_HALF - 1) / P_HALF : (p.N + P_BN - 1) / P_BN;
  p.group_m = 8;
  const int tiles = (GROUPED ? 2 : 1) * p.num_m_tiles * p.num_n_tiles;      // grouped: up to one pair per row tile
  int pairs = sms / 2;
  const int units = p.splits > 1 ? p.full_tiles + (tiles - p.full_tiles) * p.splits : tiles;
  if (units < pairs) pairs = units;
  launch_dep(kern, pairs * 2, P_THREADS, SMEM, stream, tmA, tmB, tmC, tmH, p);
  if (p.splits > 1) {
    const unsigned grid = (unsigned)(tiles - p.full_tiles) * 32;
    if (p.epi == EPI_BF16) launch_dep(pair_tail_sum_kernel<__nv_bfloat16>, grid, 256, 0, stream, (const float4*)p.ws, (__nv_bfloat16*)p.C, p);
    else launch_dep(pair_tail_sum_kernel<float>, grid, 256, 0, stream, (const float4*)p.ws, (float*)p.C, p);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace b200

using namespace b200;

#include <stdlib.h>
#include <string.h>
// B200_GEMM_TMA_STORE=0 (or b200_gemm_set_tma_store(0)) keeps the direct register stores in every epilogue: the
// switch exists for A/B measurements and for tests that compare the two epilogues bit for bit.
static int g_pair_tma_store = []() {
  const char* e = getenv("B200_GEMM_TMA_STORE");
  return (e == nullptr || e[0] != '0') ? 1 : 0;
}();
// How long a GEMM launched with a wait counter (its B operand is still being written by another kernel) polls
// before it records ERR_WAIT_FLAG and unwinds.  Returns the previous limit.
static unsigned long long g_counter_wait_limit_ns = B200_WAIT_LIMIT_NS;
extern "C" unsigned long long b200_gemm_set_wait_limit_ns(unsigned long long ns) {
  const unsigned long long old = g_counter_wait_limit_ns;
  g_counter_wait_limit_ns = ns;
  return old;
}
extern "C" int b200_gemm_set_tma_store(int on) {
  const int old = g_pair_tma_store;
  g_pair_tma_store = on ? 1 : 0;
  return old;
}

// SMs of the current device, asked once; a B200's where there is none (plans made on a machine without a GPU).
static int pair_sms() {
  static int known = 0;
  int dev = 0;
  if (known == 0 && (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&known, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)) {
    cudaGetLastError();
    known = 0;
    return 148;
  }
  return known;
}

// Same contract as b200_gemm_bf16 (gemm_tcgen05.cu); tiles are 256 x 256 on CTA pairs.
static int gemm_pair_impl(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda,
                          long long ldb, long long ldc, long long ldr, int a_mn, int b_mn, int epi,
                          const GatherTask* gather, const uint32_t* wait_counter, uint32_t wait_value,
                          uint32_t* status, cudaStream_t stream, const float* rope_cs = nullptr, int rope_seq = 0,
                          int rope_d = 0, int rope_dh = 0, int rope_ctx = 0, int swiglu_f = 0, void* H = nullptr,
                          long long ldh = 0, const ReduceTask* reduce = nullptr, const GemmFinish* finish = nullptr, int splits = 1,
                          float* ws = nullptr, const int* tile_group = nullptr, int n_groups = 1) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda & 7) || (ldb & 7))
    return -10;
  const bool pad_writable = (epi & EPI_PAD_WRITABLE) != 0;
  epi &= ~EPI_PAD_WRITABLE;
  if (epi == EPI_BF16_RES && R == nullptr) return -11;
  if (epi == EPI_SWIGLU_BWD &&
      (R == nullptr || (N & 7) || (ldr & 7) || (ldc & 7) || ((reinterpret_cast<uintptr_t>(R) | reinterpret_cast<uintptr_t>(C)) & 15)))
    return -11;
  CUtensorMap tmA, tmB;
  int rc = a_mn ? make_tmap_bf16_2d(&tmA, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 64, 64)
                : make_tmap_bf16_2d(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, 64, BM);
  if (rc) return -20 + rc;
  rc = b_mn ? make_tmap_bf16_2d(&tmB, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, 64, 64)
            : make_tmap_bf16_2d(&tmB, B, (uint64_t)N * n_groups, (uint64_t)K, (uint64_t)ldb, 64, P_HALF);
  if (rc) return -30 + rc;
  GemmParams p;
  p.M = M; p.N = N; p.K = K;
  p.C = C; p.ldc = ldc; p.R = R; p.ldr = ldr; p.epi = epi; p.status = status;
  p.num_m_tiles = p.num_n_tiles = p.group_m = 0;
  if (gather != nullptr) p.gather = *gather;
  else { p.gather.dst = nullptr; p.gather.done = nullptr; p.gather.shard_vec = 0; p.gather.world = 0; p.gather.rank = 0; }
  if (reduce != nullptr) p.reduce = *reduce;
  else p.reduce.n = 0;
  p.splits = 1; p.full_tiles = 0; p.ws = nullptr; p.tile_counters = nullptr; p.b_early = 0; p.head_gate = 0;
  p.finished = finish != nullptr;
  if (finish != nullptr) p.finish = *finish;
  p.append.cs = nullptr;
  p.tile_group = tile_group; p.group_rows = N;
  p.wait_counter = wait_counter; p.wait_value = wait_value; p.wait_limit_ns = g_counter_wait_limit_ns;
  p.rope_cs = rope_cs; p.rope_seq = rope_seq; p.rope_d = rope_d; p.rope_dh = rope_dh; p.rope_ctx = rope_ctx;
  p.swiglu_f = swiglu_f; p.H = H; p.ldh = ldh;
  // TMA-store epilogue: needs a 16-byte aligned output whose row pitch is a multiple of 16 bytes.  A TMA store
  // clips a box at the matrix edge in whole 16-byte pieces (measured: with N = 1001 bf16 columns it also writes
  // columns 1001..1007), so a row must end on a 16-byte boundary unless the caller declared the rest of the last
  // piece writable (EPI_PAD_WRITABLE: it lies inside the row pitch and receives zeros, because B rows beyond N are
  // zero-filled by the loads).  The SwiGLU epilogues (three outputs per tile) and outputs that do not qualify keep
  // the direct register stores.
  CUtensorMap tmC, tmH;
  memset(&tmC, 0, sizeof(tmC));
  memset(&tmH, 0, sizeof(tmH));
  p.tma_store = 0;
  const bool out_f32 = epi == EPI_F32 || epi == EPI_F32_ACC;
  const long long esz = out_f32 ? 4 : 2;
  const long long per16 = 16 / esz;
  const bool row_end_ok = (N % per16 == 0) || (pad_writable && (N + per16 - 1) / per16 * per16 <= ldc);
  if (g_pair_tma_store && swiglu_f > 0) {
    // gate | up (M x 2F) and h (M x F): F is a multiple of 64, so no 64-column box straddles the gate / up border
    if ((reinterpret_cast<uintptr_t>(C) & 15) == 0 && (reinterpret_cast<uintptr_t>(H) & 15) == 0 && (ldc & 7) == 0 && (ldh & 7) == 0 &&
        (C == nullptr || make_tmap_out_2d(&tmC, false, C, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, 64, 32) == 0) &&
        make_tmap_out_2d(&tmH, false, H, (uint64_t)M, (uint64_t)swiglu_f, (uint64_t)ldh, 64, 32) == 0)
      p.tma_store = 1;
  } else if (g_pair_tma_store && epi == EPI_SWIGLU_BWD) {
    // d(gate) and d(up) are the two halves of C (M x 2N); one map each, so that a box at the right edge of the gate
    // half is clipped instead of running into the up half
    const __nv_bfloat16* cu = reinterpret_cast<const __nv_bfloat16*>(C) + N;
    if (make_tmap_out_2d(&tmC, false, C, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, 64, 32) == 0 &&
        make_tmap_out_2d(&tmH, false, cu, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, 64, 32) == 0)
      p.tma_store = 1;
  } else if (g_pair_tma_store && swiglu_f == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0 &&
      (ldc * esz) % 16 == 0 && row_end_ok && (rope_cs == nullptr || (N == 3 * rope_d && rope_dh % 32 == 0))) {
    if (make_tmap_out_2d(&tmC, out_f32, C, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, out_f32 ? 32 : 64, 32) == 0)
      p.tma_store = 1;
  }
  if (C == nullptr && !p.tma_store) return -13;
  const int sms = pair_sms();
  if (tile_group != nullptr) return p.tma_store ? launch_pair<false, false, true>(tmA, tmB, tmC, tmH, p, sms, stream) : -13;
  if (rope_cs != nullptr && p.tma_store && !a_mn && !b_mn) return launch_pair<false, false, false, true>(tmA, tmB, tmC, tmH, p, sms, stream);
  if (splits > 1 && p.tma_store) {
    const int tiles = ((M + 255) / 256) * ((N + P_BN - 1) / P_BN), rest = tiles % (sms / 2);
    if (rest > 0 && make_tmap_out_2d(&tmH, true, ws, (uint64_t)rest * splits * 256, P_BN, P_BN, 32, 32) == 0) {
      p.splits = splits; p.full_tiles = tiles - rest; p.ws = ws;
    }
  }
  if (a_mn && b_mn) return launch_pair<true, true>(tmA, tmB, tmC, tmH, p, sms, stream);
  if (a_mn) return launch_pair<true, false>(tmA, tmB, tmC, tmH, p, sms, stream);
  if (b_mn) return launch_pair<false, true>(tmA, tmB, tmC, tmH, p, sms, stream);
  return launch_pair<false, false>(tmA, tmB, tmC, tmH, p, sms, stream);
}

extern "C" int b200_gemm_bf16_pair(const void* A, const void* B, void* C, const void* R, int M, int N, int K,
                                   long long lda, long long ldb, long long ldc, long long ldr, int a_mn, int b_mn,
                                   int epi, uint32_t* status, cudaStream_t stream) {
  return gemm_pair_impl(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn, b_mn, epi, nullptr, nullptr, 0, status, stream);
}

constexpr int TAIL_MAX_SLICES = 24;
static long long tail_floats(int M, int N, int splits) {
  const int rest = ((M + 255) / 256) * ((N + P_BN - 1) / P_BN) % (pair_sms() / 2);
  return splits > 1 ? (long long)rest * splits * 256 * P_BN : 0;
}

// Slices of K for the tiles of the last wave of a launch (1 = leave them whole) and the floats of workspace they need.  The estimate counts
// k-blocks of 64 (0.27 us on a pair): a wave of slices, a pipeline fill of 8 per unit, and for the second launch 14 and 0.2 per partial tile.
// Measured, us per weight gradient over 16384 rows, before (on one SM per 128 x 128 tile where that was better) -> now: 512 x 512 46 -> 18,
// 768 x 2048 59 -> 44, 2304 x 768 58 -> 51, 2048 x 5504 319 -> 289, 6144 x 2048 342 -> 314.
// cost_out (may be null): the launch's estimate in k-blocks.
extern "C" long long b200_gemm_pair_tail_plan(int M, int N, int K, int* splits_out, double* cost_out) {
  const int pairs = pair_sms() / 2, num_kb = (K + BK - 1) / BK;
  const int tiles = ((M + 255) / 256) * ((N + P_BN - 1) / P_BN), rest = tiles % pairs;
  double best = rest > 0 ? num_kb + 8 : 0;
  *splits_out = 1;
  if (rest > 0 && N % 4 == 0)
    for (int s = 2; s <= TAIL_MAX_SLICES && s <= num_kb / 4; ++s) {
      const int units = rest * s;
      const double cost = ((units + pairs - 1) / pairs) * ((double)num_kb / s + 8) + 14 + 0.2 * units;
      if (cost < 0.95 * best) { best = cost; *splits_out = s; }
    }
  if (cost_out != nullptr) *cost_out = best + (tiles / pairs) * (double)num_kb;
  return tail_floats(M, N, *splits_out);
}

// b200_gemm_bf16_pair (epi 0, 1 or 3) whose last wave is contracted in `splits` slices (the plan's, which the caller keeps); `ws` (16-byte aligned) belongs to
// this launch until it ends.
extern "C" int b200_gemm_bf16_pair_tail(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                                        long long ldc, int a_mn, int b_mn, int epi, int splits, float* ws, long long ws_floats,
                                        uint32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (epi != EPI_BF16 && epi != EPI_F32 && epi != EPI_F32_ACC) return -11;
  if (splits < 1 || (splits > 1 && (splits > TAIL_MAX_SLICES || splits > (K + BK - 1) / BK / 4 || N % 4 || ws == nullptr ||
                                    (reinterpret_cast<uintptr_t>(ws) & 15) || ws_floats < tail_floats(M, N, splits))))
    return -12;
  return gemm_pair_impl(A, B, C, nullptr, M, N, K, lda, ldb, ldc, 0, a_mn, b_mn, epi, nullptr, nullptr, 0, status, stream, nullptr, 0, 0, 0,
                        0, 0, nullptr, 0, nullptr, nullptr, splits, ws);
}

// K-major operands, epi 0, 1 or 3, accumulators finished first (see GemmFinish).
extern "C" int b200_gemm_bf16_pair_finish(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                                          long long ldc, int epi, const GemmFinish* finish, uint32_t* status, cudaStream_t stream) {
  if (epi != EPI_BF16 && epi != EPI_F32 && epi != EPI_F32_ACC) return -11;
  if (finish != nullptr && finish->act == ACT_GELU && epi != EPI_BF16) return -11;
  return gemm_pair_impl(A, B, C, nullptr, M, N, K, lda, ldb, ldc, 0, 0, 0, epi, nullptr, nullptr, 0, status, stream, nullptr, 0, 0, 0,
                        0, 0, nullptr, 0, nullptr, finish);
}

// The same GEMM carrying an all-gather: while the tensor cores work, copy warps pull `shard_bytes` from each
// of `world` peer shard addresses (`src_ptrs`, host array) into `gather_dst` (rank-major).  `done_counter`
// (device uint32, may be null) is incremented once per CTA when its slice is complete; the number of CTAs
// launched is returned through `ctas_out` so that a consumer knows the value to wait for.
// `wait_counter` / `wait_value` (may be null / 0) make this GEMM wait until its own B operand has been
// gathered by an earlier carrier that may still be running.
extern "C" int b200_gemm_bf16_pair_gather(const void* A, const void* B, void* C, const void* R, int M, int N, int K,
                                          long long lda, long long ldb, long long ldc, long long ldr, int a_mn,
                                          int b_mn, int epi, const unsigned long long* src_ptrs, void* gather_dst,
                                          unsigned long long shard_bytes, int world, int rank,
                                          uint32_t* done_counter, int* ctas_out, const uint32_t* wait_counter,
                                          unsigned int wait_value, uint32_t* status, cudaStream_t stream) {
  if (world > 16 || shard_bytes % 16 || (reinterpret_cast<uintptr_t>(gather_dst) & 15)) return -10;
  GatherTask g;
  for (int i = 0; i < 16; ++i) g.src[i] = i < world ? reinterpret_cast<const uint4*>(src_ptrs[i]) : nullptr;
  g.dst = reinterpret_cast<uint4*>(gather_dst);
  g.shard_vec = shard_bytes / 16;
  g.world = world; g.rank = rank; g.done = done_counter;
  if (ctas_out != nullptr) {
    const int sms = pair_sms();
    const int tiles = ((M + 255) / 256) * ((N + P_BN - 1) / P_BN);
    int pairs = sms / 2;
    if (tiles < pairs) pairs = tiles;
    *ctas_out = pairs * 2;
  }
  return gemm_pair_impl(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn, b_mn, epi, gather_dst ? &g : nullptr,
                        wait_counter, wait_value, status, stream);
}

// QKV projection with the rotary embedding applied in the epilogue: C (M x 3*d) = A * B^T, then the Q and K
// thirds are rotated by the angle of position (row % seq).  cos_sin: (2, ctx, dh/2) fp32.  bf16 output only.
extern "C" int b200_gemm_bf16_pair_rope(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                        long long ldb, long long ldc, const float* cos_sin, int seq, int d, int dh,
                                        int ctx, uint32_t* status, cudaStream_t stream) {
  if (cos_sin == nullptr || seq <= 0 || seq > ctx || dh % 32 || d % dh || N != 3 * d) return -12;
  if (reinterpret_cast<uintptr_t>(cos_sin) & 15) return -10;
  return gemm_pair_impl(A, B, C, nullptr, M, N, K, lda, ldb, ldc, 0, 0, 0, EPI_BF16, nullptr, nullptr, 0, status, stream,
                        cos_sin, seq, d, dh, ctx);
}

// Merged gate|up projection with SwiGLU in the epilogue: C (M x 2F) = A * B^T (gate columns, then up columns) and
// H (M x F) = silu(gate) * up.  F must be a multiple of 64; bf16 outputs; ldc, ldh multiples of 8.  C == null: H alone,
// which is then not made of rounded gates and ups (needs the TMA-store epilogue).  The launch
// may carry an all-gather exactly like b200_gemm_bf16_pair_gather (pass world = 0 for none).
extern "C" int b200_gemm_bf16_pair_swiglu(const void* A, const void* B, void* C, void* H, int M, int F, int K,
                                          long long lda, long long ldb, long long ldc, long long ldh,
                                          const unsigned long long* src_ptrs, void* gather_dst,
                                          unsigned long long shard_bytes, int world, int rank, uint32_t* status,
                                          cudaStream_t stream) {
  if (F <= 0 || F % 64 || (ldc & 7) || (ldh & 7) || H == nullptr) return -12;
  if ((reinterpret_cast<uintptr_t>(C) & 15) || (reinterpret_cast<uintptr_t>(H) & 15)) return -10;
  GatherTask g;
  const bool carry = world > 0 && gather_dst != nullptr;
  if (carry) {
    if (world > 16 || shard_bytes % 16 || (reinterpret_cast<uintptr_t>(gather_dst) & 15)) return -10;
    for (int i = 0; i < 16; ++i) g.src[i] = i < world ? reinterpret_cast<const uint4*>(src_ptrs[i]) : nullptr;
    g.dst = reinterpret_cast<uint4*>(gather_dst);
    g.shard_vec = shard_bytes / 16;
    g.world = world; g.rank = rank; g.done = nullptr;
  }
  return gemm_pair_impl(A, B, C, nullptr, M, 2 * F, K, lda, ldb, ldc, 0, 0, 0, EPI_BF16, carry ? &g : nullptr, nullptr, 0,
                        status, stream, nullptr, 0, 0, 0, 0, F, H, ldh);
}

// Grouped product on CTA pairs (see b200_gemm_bf16_grouped with `tile_group`; bf16 output): the same values, for the many rows of a prompt.
// gate: silu(gate) * up of groups of 2 N rows, N a multiple of 64.  -13: an output that TMA stores do not reach, -14: too many row tiles
// (the caller then takes the other kernel).
extern "C" int b200_gemm_bf16_pair_grouped(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                                           long long ldc, const int* tile_group, int n_groups, int gate, const GemmFinish* finish,
                                           uint32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M % BM || n_groups <= 0 || tile_group == nullptr || (gate && (finish != nullptr || N % 64))) return -12;
  if (M / BM > P_LIST) return -14;
  if (gate)
    return gemm_pair_impl(A, B, nullptr, nullptr, M, 2 * N, K, lda, ldb, 0, 0, 0, 0, EPI_BF16, nullptr, nullptr, 0, status, stream, nullptr,
                          0, 0, 0, 0, N, C, ldc, nullptr, nullptr, 1, nullptr, tile_group, n_groups);
  return gemm_pair_impl(A, B, C, nullptr, M, N, K, lda, ldb, ldc, 0, 0, 0, EPI_BF16, nullptr, nullptr, 0, status, stream, nullptr, 0, 0, 0,
                        0, 0, nullptr, 0, nullptr, finish, 1, nullptr, tile_group, n_groups);
}

int b200_make_reduce_task(const B200ReduceDesc* d, uint32_t* status, bool carried, ReduceTask* out);

// Host description of a carried all-gather (same meaning as the arguments of b200_gemm_bf16_pair_gather).
struct B200GatherDesc {
  unsigned long long src[16];
  void* dst;
  unsigned long long shard_bytes;
  int world, rank;
};

// The CTA-pair GEMM with optional carried collectives: `gather` (all-gather of the next unit's weight shards) and
// `reduce` (reduce-scatter of an earlier unit's gradient staging, optionally fused with AdamW) run on the two copy
// warps of every CTA, the gather first.  Either may be null.  epi as in b200_gemm_bf16 (EPI_SWIGLU_BWD included).
extern "C" int b200_gemm_bf16_pair_tasks(const void* A, const void* B, void* C, const void* R, int M, int N, int K,
                                         long long lda, long long ldb, long long ldc, long long ldr, int a_mn, int b_mn,
                                         int epi, const B200GatherDesc* gather, const B200ReduceDesc* reduce,
                                         uint32_t* status, cudaStream_t stream) {
  GatherTask g;
  if (gather != nullptr) {
    if (gather->world > 16 || gather->shard_bytes % 16 || (reinterpret_cast<uintptr_t>(gather->dst) & 15) ||
        gather->dst == nullptr)
      return -10;
    for (int i = 0; i < 16; ++i) g.src[i] = i < gather->world ? reinterpret_cast<const uint4*>(gather->src[i]) : nullptr;
    g.dst = reinterpret_cast<uint4*>(gather->dst);
    g.shard_vec = gather->shard_bytes / 16;
    g.world = gather->world; g.rank = gather->rank; g.done = nullptr;
  }
  ReduceTask r;
  if (reduce != nullptr) {
    const int rc = b200_make_reduce_task(reduce, status, true, &r);
    if (rc) return rc;
    // one partial sum per CTA: the grid of this kernel never exceeds the SM count
  }
  return gemm_pair_impl(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn, b_mn, epi, gather ? &g : nullptr, nullptr, 0,
                        status, stream, nullptr, 0, 0, 0, 0, 0, nullptr, 0, reduce ? &r : nullptr);
}
