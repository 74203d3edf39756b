// Decode-time attention over a paged KV cache (16-token pages by default) for sm_100a, plus the kernel
// that appends the new K / V rows to the cache.  The reference has no KV cache at all: its generate()
// re-runs the full forward for every token (llm-core/llm_core/model.py:187-236).
//
// Cache layout per layer: (num_pages, page_size, H*dh) bf16 for K and for V.  A request's tokens live in
// the pages listed in its row of `block_tables`.
//
// Decode attention is bandwidth bound (every cached K and V byte is read once per step), so the kernel is
// organised around reading whole token rows: a CTA serves all heads of a request at once, 16 lanes cover the 256 bytes
// of one head (dh = 128; 8 lanes for dh = 64), scores are reduced with shuffles, the softmax is kept online in registers
// and eight tokens' rows are in flight per thread.  The cached tokens of all requests, in pieces of eight, are dealt to
// the CTAs of one wave in equal shares, whatever the requests' lengths (flash-decoding with the shares taken across
// requests); partial (max, sum, output) triples go to a scratch buffer and a second kernel merges them.
#include "ptx.cuh"

namespace b200 {

constexpr int PD_UNROLL = 8;     // tokens whose K / V rows are in flight together, per CTA

// 16-byte load of cache data that is read exactly once per step: do not keep it in L1.
__device__ __forceinline__ uint4 ld_stream(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ int row_pieces(const int* context_lens, int r, int rows, int limit) {
  const int ctx = r < rows ? context_lens[r] : 0;
  return (min(max(ctx, 0), limit) + PD_UNROLL - 1) / PD_UNROLL;
}

// A CTA's threads cover ALL heads: thread i owns the 8 head-columns [8 i, 8 i + 8) of the token row, so the CTA reads every
// cached token as one contiguous row of H * DH elements (and the 16 tokens of a page as one contiguous 16-row block), which
// is the access pattern DRAM serves at full speed.  A head's score is reduced over its DH / 8 neighbouring lanes with
// shuffles; each thread keeps the online-softmax state (max, sum) of its head and its 8 output columns, so nothing is
// combined inside the CTA.  The K and V rows of PD_UNROLL tokens are requested before the first score is computed.
//
// Piece i of the launch is the i-th group of PD_UNROLL tokens, all requests' one after the other; CTA c has pieces
// [c * per, (c + 1) * per).  What it finds out about request r goes to part (c + r): no two (c, r) that occur have the same sum.
// Measured against equal splits of each request, a CTA each (a 2048-wide layer, both kernels): one request of 900 tokens 22.1 -> 13.0
// us, 20 of 1264 44.3 -> 39.2, 128 of 1264 208 -> 202 (6.6 TB/s); 20 requests of 128 to 2400 tokens 33 us less.
template <int DH>
__global__ void __launch_bounds__(512)
paged_decode_kernel(const __nv_bfloat16* __restrict__ q,        // (R, 3d) packed qkv or (R, d): row stride q_ld
                    const __nv_bfloat16* __restrict__ k_cache, const __nv_bfloat16* __restrict__ v_cache,
                    const int* __restrict__ block_tables, const int* __restrict__ context_lens,
                    float* __restrict__ part_o,                  // (ctas + R, H, DH)
                    float* __restrict__ part_ml,                 // (ctas + R, H, 2)
                    int2* __restrict__ row_parts,                // (R): first part and number of parts
                    int rows, int q_ld, int heads, int page_size, int max_pages, int least, float scale_log2, int num_pages,
                    uint32_t* __restrict__ status) {
  pdl_sync();
  constexpr int LPT = DH / 8;            // lanes per head (16-byte loads)
  const int d = heads * DH;
  const int col = threadIdx.x * 8;       // first of this thread's 8 columns of the token row
  const bool active = col < d;           // the block is rounded up to whole warps
  const int h = active ? col / DH : 0;
  const int li = (threadIdx.x % LPT), lane = threadIdx.x & 31;
  // The tables come from the host scheduler; a length beyond the table or a page id beyond the cache is reported
  // through the status word and skipped, never dereferenced.
  const int limit = max_pages * page_size;
  // every warp adds up the pieces by itself, then finds the request its first piece belongs to
  int total = 0;
  for (int r = lane; r < rows; r += 32) {
    total += row_pieces(context_lens, r, rows, limit);
    if (blockIdx.x == 0 && threadIdx.x < 32) {
      const int ctx = context_lens[r];
      if ((ctx < 0 || ctx > limit) && status != nullptr) atomicCAS(status, 0u, ERR_BAD_ARG | (1u << 8));
      if (ctx <= 0) row_parts[r] = make_int2(0, 0);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  const int per = max(least, (total + (int)gridDim.x - 1) / (int)gridDim.x);
  const long long first = (long long)blockIdx.x * per;
  if (first >= total) return;
  int left = min(per, total - (int)first);
  int r = 0, piece = 0, before = 0;        // `before` pieces belong to requests before r
  for (int base = 0; base < rows; base += 32) {
    const int n = row_pieces(context_lens, base + lane, rows, limit);
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    const uint32_t past = __ballot_sync(0xffffffffu, before + sum > (int)first);
    if (past != 0) {
      const int l = __ffs(past) - 1;
      r = base + l;
      before += __shfl_sync(0xffffffffu, sum - n, l);
      piece = (int)first - before;
      break;
    }
    before += __shfl_sync(0xffffffffu, sum, 31);
  }

  for (; left > 0; ++r, piece = 0) {
    const int ctx = min(max(context_lens[r], 0), limit);
    const int pieces = (ctx + PD_UNROLL - 1) / PD_UNROLL;
    if (pieces == 0) continue;
    if (piece == 0 && threadIdx.x == 0) {      // the CTA with a request's first piece knows which parts there will be
      const int last = (int)(((long long)before + pieces - 1) / per);
      row_parts[r] = make_int2(blockIdx.x + r, last - (int)blockIdx.x + 1);
    }
    before += pieces;
    const int take = min(left, pieces - piece);
    const int t0 = piece * PD_UNROLL;
    const int t1 = min(ctx, t0 + take * PD_UNROLL);
    left -= take;

    float qv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (active) {
      const uint4 u = *reinterpret_cast<const uint4*>(q + (size_t)r * q_ld + col);
      const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), e = unpack_bf16x2(u.w);
      qv[0] = a.x; qv[1] = a.y; qv[2] = b.x; qv[3] = b.y; qv[4] = c.x; qv[5] = c.y; qv[6] = e.x; qv[7] = e.y;
    }
    float m = -INFINITY, l = 0.f;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int* table = block_tables + (size_t)r * max_pages;
    for (int tb = t0; tb < t1; tb += PD_UNROLL) {
      uint4 ku[PD_UNROLL], vu[PD_UNROLL];
      bool valid[PD_UNROLL];
      const int pg = tb / page_size, off = tb - pg * page_size;
      if (off + PD_UNROLL <= page_size) {
        // the whole chunk lies in one page: consecutive rows of the cache
        const int page = table[pg];
        const bool page_ok = (unsigned)page < (unsigned)num_pages;
        if (!page_ok && threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0u, ERR_BAD_ARG | (2u << 8));
        const size_t row0 = ((size_t)(page_ok ? page : 0) * page_size + off) * d + col;
#pragma unroll
        for (int u = 0; u < PD_UNROLL; ++u) {
          valid[u] = page_ok && tb + u < t1;
          ku[u] = make_uint4(0, 0, 0, 0);
          vu[u] = make_uint4(0, 0, 0, 0);
          if (valid[u] && active) {
            ku[u] = ld_stream(k_cache + row0 + (size_t)u * d);
            vu[u] = ld_stream(v_cache + row0 + (size_t)u * d);
          }
        }
      } else {
#pragma unroll
        for (int u = 0; u < PD_UNROLL; ++u) {
          const int t = tb + u;
          valid[u] = t < t1;
          ku[u] = make_uint4(0, 0, 0, 0);
          vu[u] = make_uint4(0, 0, 0, 0);
          if (valid[u]) {
            const int page = table[t / page_size];
            if ((unsigned)page >= (unsigned)num_pages) {
              if (threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0u, ERR_BAD_ARG | (2u << 8));
              valid[u] = false;
            } else if (active) {
              const size_t row = ((size_t)page * page_size + (t % page_size)) * d + col;
              ku[u] = ld_stream(k_cache + row);
              vu[u] = ld_stream(v_cache + row);
            }
          }
        }
      }
      // scores of the whole chunk first (independent of one another), then ONE running-max update for the chunk:
      // the serial chain of the online softmax is per chunk, not per token
      float sc[PD_UNROLL];
      float mc = m;
#pragma unroll
      for (int u = 0; u < PD_UNROLL; ++u) {
        const float2 k0 = unpack_bf16x2(ku[u].x), k1 = unpack_bf16x2(ku[u].y), k2 = unpack_bf16x2(ku[u].z),
                     k3 = unpack_bf16x2(ku[u].w);
        float s = qv[0] * k0.x + qv[1] * k0.y + qv[2] * k1.x + qv[3] * k1.y + qv[4] * k2.x + qv[5] * k2.y +
                  qv[6] * k3.x + qv[7] * k3.y;
#pragma unroll
        for (int o = LPT / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        sc[u] = valid[u] ? s * scale_log2 : -INFINITY;
        mc = fmaxf(mc, sc[u]);
      }
      if (mc > -INFINITY) {
        const float corr = exp2f(m - mc);       // 0 when m == -inf
        l *= corr;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] *= corr;
#pragma unroll
        for (int u = 0; u < PD_UNROLL; ++u) {
          const float p = exp2f(sc[u] - mc);    // 0 for tokens beyond the split or on a bad page
          l += p;
          const float2 v0 = unpack_bf16x2(vu[u].x), v1 = unpack_bf16x2(vu[u].y), v2 = unpack_bf16x2(vu[u].z),
                       v3 = unpack_bf16x2(vu[u].w);
          acc[0] += p * v0.x; acc[1] += p * v0.y; acc[2] += p * v1.x; acc[3] += p * v1.y;
          acc[4] += p * v2.x; acc[5] += p * v2.y; acc[6] += p * v3.x; acc[7] += p * v3.y;
        }
        m = mc;
      }
    }
    if (active) {
      const size_t idx = (size_t)(blockIdx.x + r) * heads + h;
      float4* o = reinterpret_cast<float4*>(part_o + idx * DH + li * 8);
      o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
      if (li == 0) *reinterpret_cast<float2*>(part_ml + idx * 2) = make_float2(m, l);
    }
  }
}

// One block per request and head.  DH / 4 lanes take a part's output, 16 bytes each; the groups of lanes take parts in turn.
constexpr int PD_MERGE = 128;
template <int DH>
__global__ void __launch_bounds__(PD_MERGE)
paged_decode_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, const int2* __restrict__ row_parts,
                          __nv_bfloat16* __restrict__ out, int heads) {
  pdl_sync();
  constexpr int LG = DH / 4, GROUPS = PD_MERGE / LG;
  __shared__ float4 so[GROUPS][LG];
  __shared__ float sl[GROUPS], sm[GROUPS];
  const int r = blockIdx.x / heads, h = blockIdx.x % heads;
  const int grp = threadIdx.x / LG, e = threadIdx.x % LG;
  const int2 parts = row_parts[r];
  const float2* ml = reinterpret_cast<const float2*>(part_ml) + (size_t)parts.x * heads + h;
  const float4* po = reinterpret_cast<const float4*>(part_o) + ((size_t)parts.x * heads + h) * LG + e;
  float m = -INFINITY, l = 0.f;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int i = grp; i < parts.y; i += GROUPS) {
    const float2 one = ml[(size_t)i * heads];
    const float4 v = po[(size_t)i * heads * LG];
    const float mn = fmaxf(m, one.x);
    if (mn == -INFINITY) continue;
    const float a = exp2f(m - mn), b = exp2f(one.x - mn);
    l = l * a + one.y * b;
    o = make_float4(o.x * a + v.x * b, o.y * a + v.y * b, o.z * a + v.z * b, o.w * a + v.w * b);
    m = mn;
  }
  so[grp][e] = o;
  if (e == 0) { sl[grp] = l; sm[grp] = m; }
  __syncthreads();
  if (grp > 0) return;
  float gm = sm[0];
#pragma unroll
  for (int g = 1; g < GROUPS; ++g) gm = fmaxf(gm, sm[g]);
  float gl = 0.f;
  o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    const float w = sm[g] == -INFINITY ? 0.f : exp2f(sm[g] - gm);
    const float4 v = so[g][e];
    gl += sl[g] * w;
    o = make_float4(o.x + v.x * w, o.y + v.y * w, o.z + v.z * w, o.w + v.w * w);
  }
  const float inv = gl > 0.f ? 1.f / gl : 0.f;
  *reinterpret_cast<uint2*>(out + ((size_t)r * heads + h) * DH + e * 4) =
      make_uint2(pack_bf16x2(o.x * inv, o.y * inv), pack_bf16x2(o.z * inv, o.w * inv));
}

// cache[slot] = K (V) row of qkv for every request row; slot = page * page_size + offset (negative: skip).
__global__ void kv_append_kernel(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* __restrict__ k_cache,
                                 __nv_bfloat16* __restrict__ v_cache, const long long* __restrict__ slots, long long rows,
                                 int d, long long num_slots, uint32_t* __restrict__ status) {
  pdl_sync();
  const int lane = threadIdx.x & 31;
  const long long row = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const long long slot = slots[row];
  if (slot < 0) return;
  if (slot >= num_slots) {      // beyond the cache: report, do not write
    if (lane == 0 && status != nullptr) atomicCAS(status, 0u, ERR_BAD_ARG | (3u << 8));
    return;
  }
  const __nv_bfloat16* src = qkv + (size_t)row * 3 * d;
  for (int c = lane * 8; c < d; c += 256) {
    *reinterpret_cast<uint4*>(k_cache + (size_t)slot * d + c) = *reinterpret_cast<const uint4*>(src + d + c);
    *reinterpret_cast<uint4*>(v_cache + (size_t)slot * d + c) = *reinterpret_cast<const uint4*>(src + 2 * d + c);
  }
}

// Rotary embedding of the Q and K thirds of qkv (in place, interleaved pairs, angle of positions[row]) and the append
// of the rotated K row and the V row to their cache slot, in one pass over the row: what rope_kernel followed by
// kv_append_kernel do, with one launch and one read of K less.  slot < 0: rotate only.
__global__ void rope_kv_append_kernel(__nv_bfloat16* __restrict__ qkv, const float* __restrict__ cos_sin,
                                      const int* __restrict__ positions, __nv_bfloat16* __restrict__ k_cache,
                                      __nv_bfloat16* __restrict__ v_cache, const long long* __restrict__ slots,
                                      long long rows, int d, int dh, int ctx, long long num_slots,
                                      uint32_t* __restrict__ status) {
  pdl_sync();
  const int gpr = 3 * d / 8;             // groups of 8 elements per row
  const long long groups = rows * gpr;
  const float* cosb = cos_sin;
  const float* sinb = cos_sin + (size_t)ctx * (dh / 2);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < groups;
       i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / gpr;
    const int c = (int)(i - row * gpr) * 8;            // column within [0, 3d)
    long long slot = slots[row];
    if (slot >= num_slots) {                           // beyond the cache: report, do not write
      if (c == 0 && status != nullptr) atomicCAS(status, 0u, ERR_BAD_ARG | (3u << 8));
      slot = -1;
    }
    __nv_bfloat16* p = qkv + row * 3 * d + c;
    uint4 raw = *reinterpret_cast<const uint4*>(p);
    if (c < 2 * d) {
      const int pos = positions[row];
      const int e = c % dh;                            // element offset inside the head (multiple of 8)
      const float4 cs = *reinterpret_cast<const float4*>(cosb + (size_t)pos * (dh / 2) + e / 2);
      const float4 sn = *reinterpret_cast<const float4*>(sinb + (size_t)pos * (dh / 2) + e / 2);
      const float cc[4] = {cs.x, cs.y, cs.z, cs.w}, ss[4] = {sn.x, sn.y, sn.z, sn.w};
      const uint32_t in[4] = {raw.x, raw.y, raw.z, raw.w};
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 v = unpack_bf16x2(in[k]);
        o[k] = pack_bf16x2(cc[k] * v.x - ss[k] * v.y, ss[k] * v.x + cc[k] * v.y);
      }
      raw = make_uint4(o[0], o[1], o[2], o[3]);
      *reinterpret_cast<uint4*>(p) = raw;
    }
    if (slot >= 0 && c >= d) {
      __nv_bfloat16* dst = (c < 2 * d) ? k_cache + (size_t)slot * d + (c - d) : v_cache + (size_t)slot * d + (c - 2 * d);
      *reinterpret_cast<uint4*>(dst) = raw;
    }
  }
}

}  // namespace b200

using namespace b200;

// q: rows of stride q_ld elements whose first d entries are the queries (pass the packed qkv buffer with
// q_ld = 3d).  Caller-provided scratch: part_o (ctas + R)*H*dh floats, part_ml (ctas + R)*H*2 floats, row_parts R*2 ints.
extern "C" int b200_paged_decode(const void* q, const void* k_cache, const void* v_cache, const int* block_tables,
                                 const int* context_lens, void* out, float* part_o, float* part_ml, int* row_parts, int rows,
                                 int q_ld, int heads, int dh, int page_size, int max_pages, int ctas, int least, float scale,
                                 int num_pages, uint32_t* status, cudaStream_t st) {
  if (dh != 64 && dh != 128) return -10;
  if (page_size <= 0 || max_pages <= 0 || num_pages <= 0 || ctas <= 0 || least <= 0) return -11;
  if (q_ld % 8 || (reinterpret_cast<uintptr_t>(q) & 15) || (reinterpret_cast<uintptr_t>(k_cache) & 15) ||
      (reinterpret_cast<uintptr_t>(v_cache) & 15) || ((reinterpret_cast<uintptr_t>(part_o) | reinterpret_cast<uintptr_t>(out)) & 15) ||
      ((reinterpret_cast<uintptr_t>(part_ml) | reinterpret_cast<uintptr_t>(row_parts)) & 7))
    return -10;
  if (rows <= 0) return 0;
  const int threads = (heads * (dh / 8) + 31) / 32 * 32;      // one thread per 8 columns of the token row, whole warps
  if (threads > 512) return -12;     // heads * dh <= 4096
  const float sl2 = scale * 1.4426950408889634f;
#define PAGED_DECODE(DH)                                                                                                              \
  launch_dep(paged_decode_kernel<DH>, ctas, threads, 0, st, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k_cache,                   \
             (const __nv_bfloat16*)v_cache, block_tables, context_lens, part_o, part_ml, (int2*)row_parts, rows, q_ld, heads,          \
             page_size, max_pages, least, sl2, num_pages, status);                                                                    \
  launch_dep(paged_decode_merge_kernel<DH>, rows * heads, PD_MERGE, 0, st, (const float*)part_o, (const float*)part_ml,               \
             (const int2*)row_parts, (__nv_bfloat16*)out, heads)
  if (dh == 128) {
    PAGED_DECODE(128);
  } else {
    PAGED_DECODE(64);
  }
#undef PAGED_DECODE
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int b200_kv_append(const void* qkv, void* k_cache, void* v_cache, const long long* slots, long long rows,
                              int d, long long num_slots, uint32_t* status, cudaStream_t st) {
  if (d % 8 || (reinterpret_cast<uintptr_t>(qkv) & 15) || (reinterpret_cast<uintptr_t>(k_cache) & 15) ||
      (reinterpret_cast<uintptr_t>(v_cache) & 15))
    return -10;
  if (rows <= 0) return 0;
  launch_dep(kv_append_kernel, (unsigned)((rows + 7) / 8), 256, 0, st, (const __nv_bfloat16*)qkv,
             (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, slots, rows, d, num_slots, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// Rotary embedding of Q and K in place plus the append of K and V to their cache slots, one launch.
extern "C" int b200_rope_kv_append(void* qkv, const float* cos_sin, const int* positions, void* k_cache, void* v_cache,
                                   const long long* slots, long long rows, int d, int dh, int ctx, long long num_slots,
                                   uint32_t* status, cudaStream_t st) {
  if (dh % 8 || d % dh || positions == nullptr || slots == nullptr ||
      ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
        reinterpret_cast<uintptr_t>(cos_sin)) & 15))
    return -10;
  if (rows <= 0) return 0;
  const long long groups = rows * (3 * d / 8);
  long long blocks = (groups + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  launch_dep(rope_kv_append_kernel, (unsigned)blocks, 256, 0, st, (__nv_bfloat16*)qkv, cos_sin, positions,
             (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, slots, rows, d, dh, ctx, num_slots, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
