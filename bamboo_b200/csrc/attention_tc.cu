// Fused attention on the 5th-generation tensor cores: head dimensions 64 and 128, forward and backward.
//
// Every contraction (Q.K^T, P.V, dO.V^T, dS.K, P^T.dO, dS^T.Q) is a tcgen05.mma with fp32
// accumulators in tensor memory; tiles arrive by TMA into 128-byte-swizzled shared memory;
// the same [128 x 64] tile serves as a K-major operand (reduction over the head dimension) and
// as an MN-major operand (reduction over its rows) just by changing the matrix descriptor, so
// nothing is transposed.  Probabilities are recomputed from the saved log-sum-exp in the
// backward pass; scores never reach HBM.
//
// In every kernel warp 0 issues TMA, one or two warps issue MMAs and the remaining warps (one TMEM
// lane quarter each) do the softmax / element-wise work and the final stores.  Kernels:
//   forward          : the output row accumulates in tensor memory; head dimension 64: CTA owns 128 query rows, three
//                      CTAs share an SM; 128: CTA owns 256 query rows as two tiles in ping-pong (one softmax group each);
//   fused backward   : (head dimension 64) CTA owns 128 key rows, streams 64-row query / dO sub-tiles,
//                      computes the scores once and produces dK, dV (fixed summation order) and dQ (fp32
//                      add-reductions into an accumulator that a small kernel scales and converts);
//   two-role backward: dK/dV CTAs and dQ CTAs in one launch, scores computed by both roles, every
//                      sum in a fixed order (no reductions); templated on the head dimension - the
//                      backward at 128, and at 64 when BB_ATTENTION_BWD=split asks for fixed-order sums.
#include "tma_host.cuh"
#include <math.h>
#include <stdlib.h>

namespace {

constexpr int TQ = 128;        // rows per tile (queries or keys)
constexpr int HD = 64;         // head dimension
constexpr int TILE_BYTES = TQ * HD * 2;          // 16 KiB: [128 x 64] bf16, 128-byte rows
constexpr float LOG2E = 1.4426950408889634f;

struct TcParams {
  const __nv_bfloat16* o;       // forward output (delta kernel)
  __nv_bfloat16 *out, *dq, *dk, *dv;
  float* lse;                   // [B, H, S]
  float* delta;                 // [B, H, S]
  float* dq_acc;                // [B, H, S, 64] fp32 sums of dQ (fused backward), or null
  long long stride_o, stride_dqkv;
  int B, H, S;
  int hidden;                   // H * D: column offset between q, k and v in the packed projection
  int causal;
  float scale;
  int* status;
};

// (tile, head, batch) of a CTA.  Tiles are the slowest index, so that every head's longest tile (under a causal mask a
// tile's work grows or shrinks along the sequence) starts before any shorter one and the short ones even out the end:
// with the tiles of one head next to each other the SMs were busy for 75 % of the forward kernel's time on average
// (B8 H16 S1024 causal: 74 -> 68 us from the order alone; backward 183 -> 175 us, forward at B2 H32 S2048 D128 127 -> 111 us).
struct TileId { int tile, head, batch; };
__device__ __forceinline__ TileId tile_id(const TcParams& p) {
  const int id = blockIdx.x, rest = id / p.H;
  return {rest / p.B, id - rest * p.H, rest % p.B};
}

// instruction descriptor: bf16 x bf16 -> fp32, M = 128
__device__ __forceinline__ uint32_t idesc(int n, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TQ >> 4) << 24);
}
// Matrix descriptors.  The MMA-issuing warp shares its scheduler with compute warps, so the
// instructions spent per MMA count: a tile's descriptor is built once (`desc_*0`) and every later
// k-step only adds a constant to its address field (16-byte units; no carry into the next field
// for any shared-memory address).
// [rows x 64] tile, reduction over the 64 columns: k-step = 16 columns = 32 bytes
__device__ __forceinline__ uint64_t desc_k0(uint32_t tile) { return bb::make_smem_desc_sw128(tile, 16, 1024); }
__device__ __forceinline__ uint64_t desc_kmajor(uint64_t d0, int kstep) { return d0 + (uint64_t)(kstep * (32 >> 4)); }
// [rows x 64] tile, reduction over its rows (N or M = the 64 columns): k-step = 16 rows = 2 KiB
__device__ __forceinline__ uint64_t desc_mn0(uint32_t tile) { return bb::make_smem_desc_sw128(tile, 8192, 1024); }
__device__ __forceinline__ uint64_t desc_mnmajor64(uint64_t d0, int kstep) { return d0 + (uint64_t)(kstep * (2048 >> 4)); }
// half a row (64 bytes: chunks 4*half .. 4*half+3) of a [128 x 64] bf16 atom from 16 packed registers
__device__ __forceinline__ void atom_store_half_row(uint8_t* atom, int row, int half, const uint32_t* pk) {
  uint8_t* base = atom + row * 128;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<uint4*>(base + (((4 * half + c) ^ (row & 7)) << 4)) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two 32-column TMEM reads in flight, one wait
__device__ __forceinline__ void ld32x2(uint32_t ta, uint32_t tb, float* a, float* b) {
  uint32_t ra[32], rb[32];
  bb::tmem_ld_32x32b_x32(ta, ra);
  bb::tmem_ld_32x32b_x32(tb, rb);
  bb::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) { a[i] = __uint_as_float(ra[i]); b[i] = __uint_as_float(rb[i]); }
}
__device__ __forceinline__ void ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  bb::tmem_ld_32x32b_x32(taddr, r);
  bb::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 rows x 32 columns of results, one row per lane, -> bf16 in global memory through 2 KiB of shared memory of the warp's own: an
// instruction then writes 64 bytes of each of eight rows.  Stored by the rows' own lanes, every instruction touched 32
// lines and the stores of a CTA's end took 1800 cycles.  `rows`: how many of the 32 exist.
__device__ __forceinline__ void store_tile32(uint8_t* tile, __nv_bfloat16* dst, long long stride, int rows, int lane, const float* v, float mul) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint4 q;
    q.x = bb::pack_bf16x2(v[8 * c + 0] * mul, v[8 * c + 1] * mul); q.y = bb::pack_bf16x2(v[8 * c + 2] * mul, v[8 * c + 3] * mul);
    q.z = bb::pack_bf16x2(v[8 * c + 4] * mul, v[8 * c + 5] * mul); q.w = bb::pack_bf16x2(v[8 * c + 6] * mul, v[8 * c + 7] * mul);
    *reinterpret_cast<uint4*>(tile + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = q;
  }
  __syncwarp();
  const int c = lane & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 8 * i + (lane >> 2);
    const uint4 q = *reinterpret_cast<const uint4*>(tile + r * 64 + ((c ^ ((r >> 1) & 3)) << 4));
    if (r < rows) *reinterpret_cast<uint4*>(dst + r * stride + c * 8) = q;
  }
  __syncwarp();
}

// shared-memory bookkeeping common to the tcgen05 kernels
struct Ctl {
  uint64_t bars[32];
  uint32_t tmem_slot;
  int abort_flag;
};


// delta[b, h, s] = sum_d dO * O.  D / 8 lanes per (token, head): each loads 16 bytes of O and dO
// (a warp reads consecutive heads of a token: 512 contiguous bytes per operand), two
// independent units per thread for memory-level parallelism.  The same pass clears the fp32
// accumulator of the fused backward kernel, when there is one.
template <int D>
__global__ void __launch_bounds__(256)
attn_tc_delta_kernel(const __nv_bfloat16* o, const __nv_bfloat16* d_o, const TcParams p) {
  bb::pdl_sync();
  constexpr int LANES = D / 8;                                 // lanes of one (token, head)
  const int per_tok = p.H * LANES;                             // 16-byte chunks per token row
  const long long total = (long long)p.B * p.S * per_tok;
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (p.dq_acc) {
    float4* z = reinterpret_cast<float4*>(p.dq_acc);
    const long long n4 = (long long)p.B * p.H * p.S * (HD / 4);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // the trip count is uniform within a warp (the shuffles below need every lane)
  for (long long w = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); w < total; w += 2 * stride) {
    const long long c = w + (threadIdx.x & 31);
    float s[2];
    long long cc[2] = {c, c + stride};
    uint4 a[2], b[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      a[u] = make_uint4(0, 0, 0, 0); b[u] = a[u];
      if (cc[u] < total) {
        const long long tok = cc[u] / per_tok; const int within = (int)(cc[u] % per_tok);
        a[u] = __ldca(reinterpret_cast<const uint4*>(o + tok * p.stride_o + within * 8));
        b[u] = __ldca(reinterpret_cast<const uint4*>(d_o + tok * p.stride_o + within * 8));
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t x[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, y[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
      float t = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) t += bb::bf16_lo(x[i]) * bb::bf16_lo(y[i]) + bb::bf16_hi(x[i]) * bb::bf16_hi(y[i]);
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      t += __shfl_xor_sync(0xffffffffu, t, 4);
      if (D == 128) t += __shfl_xor_sync(0xffffffffu, t, 8);
      s[u] = t;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (cc[u] < total && (threadIdx.x & (LANES - 1)) == 0) {
        const long long tok = cc[u] / per_tok; const int head = (int)(cc[u] % per_tok) / LANES;
        p.delta[((tok / p.S) * p.H + head) * p.S + (tok % p.S)] = s[u];
      }
    }
  }
}

// 32 scores of one key row against 32 queries -> P^T and dS^T as bf16 pairs: p = 2^(s c - L), dS = p (dP - delta), with -L (log2
// units) and -delta per query column in shared memory.  The element-wise work fills the issue slots of these kernels (2300 of the
// 2600 cycles that a sub-block took with scalar instructions and a mask test per element), so the arithmetic is two elements
// wide and only sub-blocks that touch an edge test columns: visible are first..last.
template <bool MASK>
__device__ __forceinline__ void dkv_math(const float* s, const float* dp, const float* nl, const float* nd, float sl, int first, int last,
                                         uint32_t* pkP, uint32_t* pkDS) {
  const float2 c2 = make_float2(sl, sl);
#pragma unroll
  for (int e = 0; e < 32; e += 4) {
    const float4 l4 = *reinterpret_cast<const float4*>(nl + e);
    const float4 d4 = *reinterpret_cast<const float4*>(nd + e);
    const float2 ls[2] = {make_float2(l4.x, l4.y), make_float2(l4.z, l4.w)}, ds[2] = {make_float2(d4.x, d4.y), make_float2(d4.z, d4.w)};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = e + 2 * u;
      const float2 x = bb::fma2(make_float2(s[i], s[i + 1]), c2, ls[u]);
      float2 pv = make_float2(ex2(x.x), ex2(x.y));
      if (MASK) {
        if (i < first || i > last) pv.x = 0.f;
        if (i + 1 < first || i + 1 > last) pv.y = 0.f;
      }
      const float2 g = bb::mul2(pv, bb::add2(make_float2(dp[i], dp[i + 1]), ds[u]));
      pkP[i >> 1] = bb::pack_bf16x2(pv.x, pv.y);
      pkDS[i >> 1] = bb::pack_bf16x2(g.x, g.y);
    }
  }
}

// =====================================================================================
// Pipelined backward kernels: 64-wide sub-blocks, every hand-off double-buffered, two compute
// groups (warps 2-5 and 6-9) that take alternate sub-blocks, so the tensor core always has the
// next S / dP and the previous dK / dV / dQ update queued while a group does its elementwise work.
// =====================================================================================
constexpr int SUB = 64;                          // streamed rows per sub-block
constexpr int SUB_BYTES = SUB * HD * 2;          // 8 KiB: [64 x 64] bf16
// Two compute groups of 8 warps.  A row's 64 scores are split between two threads (warps w and
// w + 4 of a group reach the same TMEM lane quarter): the element-wise work has no row
// reductions here, and four compute warps per scheduler hide the TMEM-load and ALU latencies that
// two could not (issue slots were 35 % busy with 4-warp groups).
constexpr int GROUP_THREADS = 256;
// warps: 0 TMA, 1 score products, 2..17 compute, 18 the queries' statistics (dK / dV role), 19 updates (a second issuing thread, so
// that the scores of the next sub-blocks never queue behind a wait for staged operands)
constexpr int NT2 = 64 + 2 * GROUP_THREADS + 64;
constexpr int STAT_WARP = 2 + 2 * GROUP_THREADS / 32, UPD_WARP = STAT_WARP + 1;
constexpr int NSTAT = 3;                         // depth of the ring of query statistics

// Geometry of the two-role backward at head dimension D.  A [rows x 128] operand is two [rows x 64] atoms of
// 128-byte rows, one after the other (two TMA boxes), exactly as in the forward kernel.
// Tensor memory (512 columns): NSB score and NSB dP buffers of 64 columns, then the accumulators - dV and dK
// (D columns each) or dQ (D columns): 3 buffers at D = 64, 2 at D = 128, where dV + dK alone take half of it.
// Shared memory at D = 128: K and V (64 KiB), three stages of query and dO sub-tiles (96 KiB), P^T and dS^T for
// two groups (64 KiB) - 224 of 227 KiB, so the ring cannot be deeper.
template <int D> struct Bwd2 {
  static constexpr int NA = D / 64;                          // 64-column atoms per row
  static constexpr int NST = (D == 64) ? 6 : 3;              // streamed sub-tile ring depth
  static constexpr int NSB = (D == 64) ? 3 : 2;              // score buffers in tensor memory
  static constexpr int OWN_BYTES = NA * TILE_BYTES;          // one of the CTA's own [128 x D] operands
  static constexpr int STREAM_BYTES = NA * SUB_BYTES;        // one streamed [64 x D] sub-tile
  static constexpr int ACC = 2 * NSB * 64;                   // first accumulator column
};
// k-step k (16 columns) of a K-major [rows x D] operand whose 64-column atoms lie `atom` bytes apart
__device__ __forceinline__ uint64_t desc_kmajor_atoms(uint64_t d0, int k, int atom) {
  return desc_kmajor(d0 + (uint64_t)((k >> 2) * (atom >> 4)), k & 3);
}

// ------------------------------------------------------------------ dQ (pipelined)
// smem: Q, dO [128 x D] | K, V sub-tiles [64 x D] x NST stages | dS [128 q x 64 kv] x 2
// TMEM: S NSB x 64 | dP NSB x 64 | dQ D
template <int D>
__device__ __forceinline__ void
attn_tc_dq2_body(const CUtensorMap& tm_q, const CUtensorMap& tm_kv, const CUtensorMap& tm_do, const TcParams& p,
                 const TileId id, const int nbx) {
  using G = Bwd2<D>;
  constexpr int NA = G::NA, NST = G::NST, NSB = G::NSB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sDO = sQ + G::OWN_BYTES;
  uint8_t* sK = sDO + G::OWN_BYTES;            // NST stages
  uint8_t* sV = sK + NST * G::STREAM_BYTES;    // NST stages
  uint8_t* sDS = sV + NST * G::STREAM_BYTES;   // 2 x 16 KiB
  Ctl* ctl = reinterpret_cast<Ctl*>(sDS + 2 * TILE_BYTES);
  uint64_t* q_full = &ctl->bars[0];
  uint64_t* kv_full = &ctl->bars[1];           // [NST]
  uint64_t* kv_empty = &ctl->bars[1 + NST];    // [NST]
  uint64_t* s_full = &ctl->bars[1 + 2 * NST];  // [NSB]
  uint64_t* s_empty = s_full + NSB;            // [NSB]
  uint64_t* ds_full = s_empty + NSB;           // [2]
  uint64_t* ds_empty = ds_full + 2;            // [2]
  uint64_t* acc_full = ds_empty + 2;

  const int warp = bb::warp_index(), lane = threadIdx.x & 31;
  const int qb = nbx - 1 - id.tile, head = id.head, batch = id.batch;
  const int q0 = qb * TQ;
  const int row_base = batch * p.S;
  const int colq = head * D, colk = p.hidden + head * D, colv = 2 * p.hidden + head * D;
  int nblk = (p.S + SUB - 1) / SUB;
  if (p.causal) nblk = min(nblk, (q0 + TQ) / SUB);

  if (threadIdx.x == 0) {
    ctl->abort_flag = 0;
    bb::mbar_init(q_full, 1);
    for (int i = 0; i < NST; ++i) { bb::mbar_init(&kv_full[i], 1); bb::mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < NSB; ++i) { bb::mbar_init(&s_full[i], 1); bb::mbar_init(&s_empty[i], GROUP_THREADS / 32); }
    for (int i = 0; i < 2; ++i) { bb::mbar_init(&ds_full[i], GROUP_THREADS / 32); bb::mbar_init(&ds_empty[i], 1); }
    bb::mbar_init(acc_full, 1);
    bb::fence_barrier_init();
    bb::tma_prefetch_desc(&tm_q); bb::tma_prefetch_desc(&tm_kv); bb::tma_prefetch_desc(&tm_do);
  }
  if (warp == 1) { bb::tmem_alloc(&ctl->tmem_slot, 512); bb::tmem_relinquish(); }
  bb::tc_fence_before_sync();
  __syncthreads();
  bb::tc_fence_after_sync();
  const uint32_t tmem = ctl->tmem_slot;
  bb::pdl_sync();
  const uint32_t tDQ = tmem + G::ACC;          // S[b] at tmem + 64 b, dP[b] at tmem + 64 (NSB + b)

  if (warp == 0) {
    if (bb::elect_one()) {
      bb::mbar_arrive_expect_tx(q_full, 2 * G::OWN_BYTES);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        bb::tma_load_3d(sQ + a * TILE_BYTES, &tm_q, q_full, colq + 64 * a, q0, batch);
        bb::tma_load_3d(sDO + a * TILE_BYTES, &tm_do, q_full, colq + 64 * a, q0, batch);
      }
    }
    __syncwarp();
    for (int j = 0; j < nblk; ++j) {
      const int s = j % NST;
      if (!bb::mbar_wait_warp(&kv_empty[s], ((j / NST) & 1) ^ 1, &ctl->abort_flag, p.status)) break;
      if (bb::elect_one()) {
        bb::mbar_arrive_expect_tx(&kv_full[s], 2 * G::STREAM_BYTES);
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          bb::tma_load_3d(sK + s * G::STREAM_BYTES + a * SUB_BYTES, &tm_kv, &kv_full[s], colk + 64 * a, j * SUB, batch);
          bb::tma_load_3d(sV + s * G::STREAM_BYTES + a * SUB_BYTES, &tm_kv, &kv_full[s], colv + 64 * a, j * SUB, batch);
        }
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    const uint64_t dQ0 = desc_k0(bb::smem_u32(sQ)), dDO0 = desc_k0(bb::smem_u32(sDO));
    const uint64_t dK0 = desc_k0(bb::smem_u32(sK)), dV0 = desc_k0(bb::smem_u32(sV));     // stage 0; stage s: + s * STREAM_BYTES / 16
    const uint32_t i_s = idesc(64, 0, 0);
    bool alive = bb::mbar_wait_warp(q_full, 0, &ctl->abort_flag, p.status);
    for (int j = 0; j < nblk && alive; ++j) {
      const int s = j % NST, b = j % NSB;
      if (!bb::mbar_wait2_warp(&kv_full[s], (j / NST) & 1, &s_empty[b], ((j / NSB) & 1) ^ 1, &ctl->abort_flag, p.status)) break;
      bb::tc_fence_after_sync();
      if (bb::elect_one()) {
        const uint64_t dK = dK0 + (uint64_t)(s * (G::STREAM_BYTES >> 4)), dV = dV0 + (uint64_t)(s * (G::STREAM_BYTES >> 4));
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          bb::umma_f16(tmem + 64 * b, desc_kmajor_atoms(dQ0, k, TILE_BYTES), desc_kmajor_atoms(dK, k, SUB_BYTES), i_s, k > 0);
          bb::umma_f16(tmem + 64 * (NSB + b), desc_kmajor_atoms(dDO0, k, TILE_BYTES), desc_kmajor_atoms(dV, k, SUB_BYTES), i_s, k > 0);
        }
        bb::umma_commit(&s_full[b]);
      }
      __syncwarp();
    }
  } else if (warp == UPD_WARP) {
    const uint64_t dKm0 = desc_mn0(bb::smem_u32(sK)), dDS0 = desc_k0(bb::smem_u32(sDS));
    const uint32_t i_dq = idesc(D, 0, 1);
    for (int jj = 0; jj < nblk; ++jj) {
      const int s2 = jj % NST, b2 = jj & 1;
      // (the sub-tiles landed long ago - the score products read them; the wait makes them visible to this thread)
      if (!bb::mbar_wait2_warp(&kv_full[s2], (jj / NST) & 1, &ds_full[b2], (jj >> 1) & 1, &ctl->abort_flag, p.status)) break;
      bb::tc_fence_after_sync();
      if (bb::elect_one()) {
        const uint64_t dK2 = dKm0 + (uint64_t)(s2 * (G::STREAM_BYTES >> 4)), dDS = dDS0 + (uint64_t)(b2 * (TILE_BYTES >> 4));
#pragma unroll
        for (int k = 0; k < 4; ++k) bb::umma_f16(tDQ, desc_kmajor(dDS, k), desc_mnmajor64(dK2, k), i_dq, (jj > 0 || k > 0));
        bb::umma_commit(&ds_empty[b2]);
        bb::umma_commit(&kv_empty[s2]);
        if (jj == nblk - 1) bb::umma_commit(acc_full);
      }
      __syncwarp();
    }
  } else if (warp != STAT_WARP) {
    const int g = (warp - 2) >> 3;                           // compute group = buffer index
    const int hf = ((warp - 2) >> 2) & 1;                    // which 32 of the sub-block's 64 columns
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int qrow = q0 + row;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const float* lse_g = p.lse + ((long long)batch * p.H + head) * p.S;
    const float* delta_g = p.delta + ((long long)batch * p.H + head) * p.S;
    const float lse = (qrow < p.S) ? lse_g[qrow] * LOG2E : 0.f;
    const float dl = (qrow < p.S) ? delta_g[qrow] : 0.f;
    const float sl = p.scale * LOG2E;
    uint8_t* myDS = sDS + g * TILE_BYTES;
    // every warp waits for itself; one that gave up goes on (its waits return at once then) and stores nothing
    bool alive = true;
    int n = 0;                                               // this group's iteration count
    const float2 sl2 = make_float2(sl, sl), nlse2 = make_float2(-lse, -lse), ndl2 = make_float2(-dl, -dl);
    for (int j = g; j < nblk; j += 2, ++n) {
      const int sb = j % NSB;
      const uint32_t tS = tmem + 64 * sb, tDP = tmem + 64 * (NSB + sb);
      if (!bb::mbar_wait_warp(&s_full[sb], (j / NSB) & 1, &ctl->abort_flag, p.status)) alive = false;
      bb::tc_fence_after_sync();
      const int c0 = j * SUB + hf * 32;
      uint32_t pk[16];                                       // this thread's 32 dS values as bf16 pairs
      {
        float sv[32], dp[32];
        ld32x2(tS + lane_addr + hf * 32, tDP + lane_addr + hf * 32, sv, dp);
        bb::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) bb::mbar_arrive(&s_empty[sb]);        // scores in registers: the MMA warp may refill
        // only sub-blocks that touch the sequence end or the causal diagonal test columns
        if (c0 + 32 > p.S || (p.causal && c0 + 32 - 1 > q0)) {
          const int last = min(p.S - 1, p.causal ? qrow : p.S - 1) - c0;
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 x = bb::fma2(make_float2(sv[i], sv[i + 1]), sl2, nlse2);
            const float2 pv = make_float2(i > last ? 0.f : ex2(x.x), i + 1 > last ? 0.f : ex2(x.y));
            const float2 d = bb::mul2(pv, bb::add2(make_float2(dp[i], dp[i + 1]), ndl2));
            pk[i >> 1] = bb::pack_bf16x2(d.x, d.y);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 x = bb::fma2(make_float2(sv[i], sv[i + 1]), sl2, nlse2);
            const float2 d = bb::mul2(make_float2(ex2(x.x), ex2(x.y)), bb::add2(make_float2(dp[i], dp[i + 1]), ndl2));
            pk[i >> 1] = bb::pack_bf16x2(d.x, d.y);
          }
        }
      }
      // the staging buffer is free once the dQ update that read it two sub-blocks ago retired
      if (!bb::mbar_wait_warp(&ds_empty[g], (n & 1) ^ 1, &ctl->abort_flag, p.status)) alive = false;
      atom_store_half_row(myDS, row, hf, pk);
      bb::fence_proxy_async();
      __syncwarp();
      if (lane == 0) bb::mbar_arrive(&ds_full[g]);
    }
    if (!bb::mbar_wait_warp(acc_full, 0, &ctl->abort_flag, p.status)) alive = false;
    if (alive && g < NA) {
      // group g stores the g-th 64 columns
      bb::tc_fence_after_sync();
      float v[32];
      const int c = 64 * g + hf * 32;
      ld32(tDQ + lane_addr + c, v);
      const int w0 = q0 + quarter * 32;
      store_tile32(myDS + (hf * 4 + quarter) * 2048, p.dq + (long long)(row_base + w0) * p.stride_dqkv + colq + c, p.stride_dqkv, p.S - w0, lane, v, p.scale);
    }
  }
  bb::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) bb::tmem_dealloc(tmem, 512);
}

template <int D> constexpr int dq2_smem() {
  return 2 * Bwd2<D>::OWN_BYTES + 2 * Bwd2<D>::NST * Bwd2<D>::STREAM_BYTES + 2 * TILE_BYTES + (int)sizeof(Ctl) + 1024;
}

// ------------------------------------------------------------------ dK, dV (pipelined)
// smem: K, V [128 x D] | Q, dO sub-tiles [64 x D] x NST stages | P^T, dS^T [128 kv x 64 q] x 2 each
//       | lse / delta of a sub-block's 64 query columns, x NSTAT
// TMEM: S^T NSB x 64 | dP^T NSB x 64 | dV D | dK D
template <int D>
__device__ __forceinline__ void
attn_tc_dkv2_body(const CUtensorMap& tm128, const CUtensorMap& tm64, const CUtensorMap& tm_do64, const TcParams& p, const TileId id) {
  using G = Bwd2<D>;
  constexpr int NA = G::NA, NST = G::NST, NSB = G::NSB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + G::OWN_BYTES;
  uint8_t* sQ = sV + G::OWN_BYTES;             // NST stages
  uint8_t* sDO = sQ + NST * G::STREAM_BYTES;   // NST stages
  uint8_t* sP = sDO + NST * G::STREAM_BYTES;   // 2 x 16 KiB
  uint8_t* sDS = sP + 2 * TILE_BYTES;          // 2 x 16 KiB
  float* s_lse = reinterpret_cast<float*>(sDS + 2 * TILE_BYTES);   // [NSTAT][64]: negated log-sum-exp (log2 units) and delta
  float* s_delta = s_lse + NSTAT * SUB;                            // [NSTAT][64]
  Ctl* ctl = reinterpret_cast<Ctl*>(s_delta + NSTAT * SUB);
  uint64_t* kv_full = &ctl->bars[0];
  uint64_t* q_full = &ctl->bars[1];            // [NST]
  uint64_t* q_empty = &ctl->bars[1 + NST];     // [NST]
  uint64_t* s_full = &ctl->bars[1 + 2 * NST];  // [NSB]
  uint64_t* s_empty = s_full + NSB;            // [NSB]
  uint64_t* p_full = s_empty + NSB;            // [2]
  uint64_t* p_empty = p_full + 2;              // [2]
  uint64_t* acc_full = p_empty + 2;
  uint64_t* st_full = acc_full + 1;            // [NSTAT] statistics of a sub-block's queries

  const int warp = bb::warp_index(), lane = threadIdx.x & 31;
  const int kb = id.tile, head = id.head, batch = id.batch;
  const int k0 = kb * TQ;
  const int row_base = batch * p.S;
  const int colq = head * D, colk = p.hidden + head * D, colv = 2 * p.hidden + head * D;
  const int nq = (p.S + SUB - 1) / SUB;
  const int qstart = p.causal ? (k0 / SUB) : 0;
  const int nblk = nq - qstart;

  if (threadIdx.x == 0) {
    ctl->abort_flag = 0;
    bb::mbar_init(kv_full, 1);
    for (int i = 0; i < NST; ++i) { bb::mbar_init(&q_full[i], 1); bb::mbar_init(&q_empty[i], 1); }
    for (int i = 0; i < NSB; ++i) { bb::mbar_init(&s_full[i], 1); bb::mbar_init(&s_empty[i], GROUP_THREADS / 32); }
    for (int i = 0; i < 2; ++i) { bb::mbar_init(&p_full[i], GROUP_THREADS / 32); bb::mbar_init(&p_empty[i], 1); }
    bb::mbar_init(acc_full, 1);
    for (int i = 0; i < NSTAT; ++i) bb::mbar_init(&st_full[i], 1);
    bb::fence_barrier_init();
    bb::tma_prefetch_desc(&tm128); bb::tma_prefetch_desc(&tm64); bb::tma_prefetch_desc(&tm_do64);
  }
  if (warp == 1) { bb::tmem_alloc(&ctl->tmem_slot, 512); bb::tmem_relinquish(); }
  bb::tc_fence_before_sync();
  __syncthreads();
  bb::tc_fence_after_sync();
  const uint32_t tmem = ctl->tmem_slot;
  bb::pdl_sync();
  const uint32_t tDV = tmem + G::ACC, tDK = tDV + D;   // S^T[b] at tmem + 64 b, dP^T[b] at tmem + 64 (NSB + b)

  if (warp == 0) {
    if (bb::elect_one()) {
      bb::mbar_arrive_expect_tx(kv_full, 2 * G::OWN_BYTES);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        bb::tma_load_3d(sK + a * TILE_BYTES, &tm128, kv_full, colk + 64 * a, k0, batch);
        bb::tma_load_3d(sV + a * TILE_BYTES, &tm128, kv_full, colv + 64 * a, k0, batch);
      }
    }
    __syncwarp();
    for (int i = 0; i < nblk; ++i) {
      const int s = i % NST;
      if (!bb::mbar_wait_warp(&q_empty[s], ((i / NST) & 1) ^ 1, &ctl->abort_flag, p.status)) break;
      if (bb::elect_one()) {
        bb::mbar_arrive_expect_tx(&q_full[s], 2 * G::STREAM_BYTES);
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          bb::tma_load_3d(sQ + s * G::STREAM_BYTES + a * SUB_BYTES, &tm64, &q_full[s], colq + 64 * a, (qstart + i) * SUB, batch);
          bb::tma_load_3d(sDO + s * G::STREAM_BYTES + a * SUB_BYTES, &tm_do64, &q_full[s], colq + 64 * a, (qstart + i) * SUB, batch);
        }
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    const uint64_t dK0 = desc_k0(bb::smem_u32(sK)), dV0 = desc_k0(bb::smem_u32(sV));
    const uint64_t dQ0 = desc_k0(bb::smem_u32(sQ)), dDO0 = desc_k0(bb::smem_u32(sDO));   // stage 0; stage s: + s * STREAM_BYTES / 16
    const uint32_t i_s = idesc(64, 0, 0);
    bool alive = bb::mbar_wait_warp(kv_full, 0, &ctl->abort_flag, p.status);
    for (int i = 0; i < nblk && alive; ++i) {
      const int s = i % NST, b = i % NSB;
      if (!bb::mbar_wait2_warp(&q_full[s], (i / NST) & 1, &s_empty[b], ((i / NSB) & 1) ^ 1, &ctl->abort_flag, p.status)) break;
      bb::tc_fence_after_sync();
      if (bb::elect_one()) {
        const uint64_t dQ = dQ0 + (uint64_t)(s * (G::STREAM_BYTES >> 4)), dDO = dDO0 + (uint64_t)(s * (G::STREAM_BYTES >> 4));
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          bb::umma_f16(tmem + 64 * b, desc_kmajor_atoms(dK0, k, TILE_BYTES), desc_kmajor_atoms(dQ, k, SUB_BYTES), i_s, k > 0);
          bb::umma_f16(tmem + 64 * (NSB + b), desc_kmajor_atoms(dV0, k, TILE_BYTES), desc_kmajor_atoms(dDO, k, SUB_BYTES), i_s, k > 0);
        }
        bb::umma_commit(&s_full[b]);
      }
      __syncwarp();
    }
  } else if (warp == UPD_WARP) {
    const uint64_t dQm0 = desc_mn0(bb::smem_u32(sQ)), dDOm0 = desc_mn0(bb::smem_u32(sDO));
    const uint64_t dP0 = desc_k0(bb::smem_u32(sP)), dDS0 = desc_k0(bb::smem_u32(sDS));
    const uint32_t i_acc = idesc(D, 0, 1);
    for (int ii = 0; ii < nblk; ++ii) {
      const int s2 = ii % NST, b2 = ii & 1;
      // (the sub-tiles landed long ago - the score products read them; the wait makes them visible to this thread)
      if (!bb::mbar_wait2_warp(&q_full[s2], (ii / NST) & 1, &p_full[b2], (ii >> 1) & 1, &ctl->abort_flag, p.status)) break;
      bb::tc_fence_after_sync();
      if (bb::elect_one()) {
        const uint64_t dQ2 = dQm0 + (uint64_t)(s2 * (G::STREAM_BYTES >> 4)), dDO2 = dDOm0 + (uint64_t)(s2 * (G::STREAM_BYTES >> 4));
        const uint64_t dP = dP0 + (uint64_t)(b2 * (TILE_BYTES >> 4)), dDS = dDS0 + (uint64_t)(b2 * (TILE_BYTES >> 4));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          bb::umma_f16(tDV, desc_kmajor(dP, k), desc_mnmajor64(dDO2, k), i_acc, (ii > 0 || k > 0));
          bb::umma_f16(tDK, desc_kmajor(dDS, k), desc_mnmajor64(dQ2, k), i_acc, (ii > 0 || k > 0));
        }
        bb::umma_commit(&p_empty[b2]);
        bb::umma_commit(&q_empty[s2]);
        if (ii == nblk - 1) bb::umma_commit(acc_full);
      }
      __syncwarp();
    }
  } else if (warp == STAT_WARP) {
    const float* lse_g = p.lse + ((long long)batch * p.H + head) * p.S;
    const float* delta_g = p.delta + ((long long)batch * p.H + head) * p.S;
    for (int i = 0; i < nblk; ++i) {
      // two queries per lane; the updates of the sub-block that had the slot before have retired
      float l2[2], d2[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int q = (qstart + i) * SUB + lane + 32 * u;
        l2[u] = (q < p.S) ? -(lse_g[q] * LOG2E) : 0.f;
        d2[u] = (q < p.S) ? -delta_g[q] : 0.f;
      }
      if (i >= NSTAT && !bb::mbar_wait_warp(&q_empty[(i - NSTAT) % NST], ((i - NSTAT) / NST) & 1, &ctl->abort_flag, p.status)) break;
      const int st = i % NSTAT;
#pragma unroll
      for (int u = 0; u < 2; ++u) { s_lse[st * SUB + lane + 32 * u] = l2[u]; s_delta[st * SUB + lane + 32 * u] = d2[u]; }
      __syncwarp();
      if (lane == 0) bb::mbar_arrive(&st_full[st]);
    }
  } else {
    const int g = (warp - 2) >> 3;
    const int hf = ((warp - 2) >> 2) & 1;                  // which 32 of the sub-block's 64 query columns
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;                   // key row inside the tile
    const int krow = k0 + row;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const float sl = p.scale * LOG2E;
    uint8_t* myP = sP + g * TILE_BYTES;
    uint8_t* myDS = sDS + g * TILE_BYTES;
    // every warp waits for itself; one that gave up goes on (its waits return at once then) and stores nothing
    bool alive = true;
    int n = 0;
    for (int i = g; i < nblk; i += 2, ++n) {
      const int qc0 = (qstart + i) * SUB + hf * 32;          // first query of this thread's columns
      const int sb = i % NSB, st = i % NSTAT;
      const uint32_t tS = tmem + 64 * sb, tDP = tmem + 64 * (NSB + sb);
      if (!bb::mbar_wait2_warp(&st_full[st], (i / NSTAT) & 1, &s_full[sb], (i / NSB) & 1, &ctl->abort_flag, p.status)) alive = false;
      bb::tc_fence_after_sync();
      const float *my_lse = s_lse + st * SUB + hf * 32, *my_delta = s_delta + st * SUB + hf * 32;
      uint32_t pkP[16], pkDS[16];                            // this thread's 32 P^T and dS^T values as bf16 pairs
      {
        float sv[32], dp[32];
        ld32x2(tS + lane_addr + hf * 32, tDP + lane_addr + hf * 32, sv, dp);
        bb::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) bb::mbar_arrive(&s_empty[sb]);
        if (qc0 + 32 > p.S || (p.causal && k0 + TQ - 1 > qc0))
          dkv_math<true>(sv, dp, my_lse, my_delta, sl, p.causal ? krow - qc0 : 0, p.S - 1 - qc0, pkP, pkDS);
        else
          dkv_math<false>(sv, dp, my_lse, my_delta, sl, 0, 0, pkP, pkDS);
      }
      // the staging buffers are free once the dV / dK update that read them retired
      if (!bb::mbar_wait_warp(&p_empty[g], (n & 1) ^ 1, &ctl->abort_flag, p.status)) alive = false;
      atom_store_half_row(myP, row, hf, pkP);
      atom_store_half_row(myDS, row, hf, pkDS);
      bb::fence_proxy_async();
      __syncwarp();
      if (lane == 0) bb::mbar_arrive(&p_full[g]);
    }
    if (!bb::mbar_wait_warp(acc_full, 0, &ctl->abort_flag, p.status)) alive = false;
    if (alive) {
      bb::tc_fence_after_sync();
      // the two groups split the final stores: group 0 writes dV, group 1 writes dK
      const uint32_t src = (g == 0) ? tDV : tDK;
      __nv_bfloat16* dst = (g == 0) ? p.dv : p.dk;
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        float v[32];
        const int c = 64 * a + hf * 32;
        ld32(src + lane_addr + c, v);
        const int w0 = k0 + quarter * 32;
        store_tile32(myP + (hf * 4 + quarter) * 2048, dst + (long long)(row_base + w0) * p.stride_dqkv + colq + c, p.stride_dqkv, p.S - w0, lane, v,
                     g == 0 ? 1.f : p.scale);
      }
    }
  }
  bb::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) bb::tmem_dealloc(tmem, 512);
}

template <int D> constexpr int dkv2_smem() {
  return 2 * Bwd2<D>::OWN_BYTES + 2 * Bwd2<D>::NST * Bwd2<D>::STREAM_BYTES + 4 * TILE_BYTES + 2 * NSTAT * SUB * (int)sizeof(float) + (int)sizeof(Ctl) + 1024;
}

// Both backward roles in one launch: of the 2 * nbx CTAs of a (batch, head), the first nbx own a
// key tile (dK, dV) and the rest a query tile (dQ), each role's longest first.  The two roles are independent, so the
// tail of one fills with CTAs of the other instead of leaving SMs idle between two launches.  (Roles taken in turn
// were slower: 538 us against 503 us at B2 H32 S2048 D128 causal.)
// B2 H32 S2048 D128 causal, step by step: 479 us with one issuing warp, group barriers around every hand-off and scalar arithmetic;
// 447 with two-wide arithmetic and warps that wait for themselves; 331 with a second issuing warp; 304 with results stored through
// shared memory.
template <int D> constexpr int bwd2_smem() { return dkv2_smem<D>() > dq2_smem<D>() ? dkv2_smem<D>() : dq2_smem<D>(); }
static_assert(bwd2_smem<64>() <= 232448 && bwd2_smem<128>() <= 232448, "227 KiB of shared memory per CTA");
template <int D>
__global__ void __launch_bounds__(NT2, 1)
attn_tc_bwd2_kernel(const __grid_constant__ CUtensorMap tm128, const __grid_constant__ CUtensorMap tm64,
                    const __grid_constant__ CUtensorMap tm_do128, const __grid_constant__ CUtensorMap tm_do64, const TcParams p) {
  TileId id = tile_id(p);
  const int nbx = (p.S + TQ - 1) / TQ;
  if (id.tile < nbx) {
    attn_tc_dkv2_body<D>(tm128, tm64, tm_do64, p, id);
  } else {
    id.tile -= nbx;
    attn_tc_dq2_body<D>(tm128, tm64, tm_do128, p, id, nbx);
  }
}

// ------------------------------------------------------------------ fused backward: dK, dV and dQ from one pass
// A CTA owns 128 key rows and streams the 64-row query / dO sub-tiles like the dK/dV role above,
// but S^T and dP^T are computed once: the staged dS^T tiles of two consecutive sub-blocks
// ([128 keys x 64 queries] each, adjacent in shared memory) also serve, read with the queries as
// the M dimension, as the A operand of dQ[128 queries x 64] = dS . K for that pair of sub-blocks.
// The pair's dQ [128 x 64] fp32 leaves tensor memory through staging tiles and bulk tensor add-reductions
// into a [B, H, S, 64] accumulator: each of the sixteen compute warps moves 32 rows x 16 columns through a tile of its own,
// so nothing here waits for another warp; each query row receives one contribution per key tile, in no fixed order; a small
// kernel scales and converts the sums once all CTAs are done.  Five contractions instead of seven, one
// exponential pass instead of two, half the CTAs.
// A compute warp that gave up on a wait goes on through the loop (its waits return at once then) and stores nothing.
// smem: K, V [128 x 64] | Q, dO sub-tiles x NST3 | P^T x 2 | dS^T x 2 pair slots x 2 groups | dQ staging 16 x 2 KiB | lse / delta
// TMEM: S^T 2 x 64 | dP^T 2 x 64 | dV 64 | dK 64 | dQ 2 x 64
constexpr int NST3 = 4;
// warps: 0 TMA, 1 score products (S^T, dP^T), 2 updates (dV, dK, dQ), 3 the queries' log-sum-exp and delta, 4..19 the two
// compute groups (compute warp w must sit at w % 4 == its tensor-memory lane quarter).  Fetched and staged by the compute
// groups themselves, the statistics cost two group-wide barriers per sub-block: B8 H16 S1024 causal 175 -> 171 us,
// non-causal 244 -> 232 us without them.
constexpr int NT3 = 128 + 2 * GROUP_THREADS;
__global__ void __launch_bounds__(NT3, 1)
attn_tc_bwd3_kernel(const __grid_constant__ CUtensorMap tm128, const __grid_constant__ CUtensorMap tm64,
                    const __grid_constant__ CUtensorMap tm_do64, const __grid_constant__ CUtensorMap tm_acc, const TcParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + TILE_BYTES;
  uint8_t* sQ = sV + TILE_BYTES;               // NST3 stages x 8 KiB
  uint8_t* sDO = sQ + NST3 * SUB_BYTES;        // NST3 stages x 8 KiB
  uint8_t* sP = sDO + NST3 * SUB_BYTES;        // [group] x 16 KiB
  uint8_t* sDS = sP + 2 * TILE_BYTES;          // [pair slot][group] x 16 KiB
  uint8_t* sDQ = sDS + 4 * TILE_BYTES;         // [compute warp] x 2 KiB: [32 queries x 16] fp32, 64-byte rows, 64-byte swizzle
  float* s_lse = reinterpret_cast<float*>(sDQ + 2 * TILE_BYTES);   // [NSTAT][64]: negated log-sum-exp (log2 units) and delta of a sub-block's queries
  float* s_delta = s_lse + NSTAT * SUB;                            // [NSTAT][64]
  Ctl* ctl = reinterpret_cast<Ctl*>(s_delta + NSTAT * SUB);
  uint64_t* kv_full = &ctl->bars[0];
  uint64_t* q_full = &ctl->bars[1];            // [NST3]
  uint64_t* q_empty = q_full + NST3;           // [NST3]
  uint64_t* s_full = q_empty + NST3;           // [2]
  uint64_t* s_empty = s_full + 2;              // [2]
  uint64_t* p_full = s_empty + 2;              // [2]  P^T and dS^T of a sub-block staged
  uint64_t* p_empty = p_full + 2;              // [2]  P^T buffer of a group read by its dV update
  uint64_t* ds_empty = p_empty + 2;            // [2]  both dS^T buffers of a pair slot read by dK and dQ
  uint64_t* dq_full = ds_empty + 2;            // [2]  a pair's dQ complete in tensor memory
  uint64_t* dq_empty = dq_full + 2;            // [2]  ... and drained
  uint64_t* acc_full = dq_empty + 2;
  uint64_t* st_full = acc_full + 1;            // [NSTAT] statistics of a sub-block's queries

  const int warp = bb::warp_index(), lane = threadIdx.x & 31;
  const TileId id = tile_id(p);
  const int kb = id.tile, head = id.head, batch = id.batch;
  const int k0 = kb * TQ;
  const int row_base = batch * p.S;
  const int colq = head * HD, colk = p.hidden + head * HD, colv = 2 * p.hidden + head * HD;
  const int nq = (p.S + SUB - 1) / SUB;
  const int qstart = p.causal ? (k0 / SUB) : 0;
  // an even number of sub-blocks (they pair up for dQ); a padding sub-block lies past the
  // sequence end and is masked to zero
  const int nblk = (nq - qstart + 1) & ~1;
  const int npairs = nblk >> 1;

  if (threadIdx.x == 0) {
    ctl->abort_flag = 0;
    bb::mbar_init(kv_full, 1);
    for (int i = 0; i < NST3; ++i) { bb::mbar_init(&q_full[i], 1); bb::mbar_init(&q_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      bb::mbar_init(&s_full[i], 1); bb::mbar_init(&s_empty[i], GROUP_THREADS / 32);
      bb::mbar_init(&p_full[i], GROUP_THREADS / 32); bb::mbar_init(&p_empty[i], 1);
      bb::mbar_init(&ds_empty[i], 1);
      bb::mbar_init(&dq_full[i], 1); bb::mbar_init(&dq_empty[i], 2 * GROUP_THREADS / 32);
    }
    bb::mbar_init(acc_full, 1);
    for (int i = 0; i < NSTAT; ++i) bb::mbar_init(&st_full[i], 1);
    bb::fence_barrier_init();
    bb::tma_prefetch_desc(&tm128); bb::tma_prefetch_desc(&tm64); bb::tma_prefetch_desc(&tm_do64); bb::tma_prefetch_desc(&tm_acc);
  }
  if (warp == 1) { bb::tmem_alloc(&ctl->tmem_slot, 512); bb::tmem_relinquish(); }
  bb::tc_fence_before_sync();
  __syncthreads();
  bb::tc_fence_after_sync();
  const uint32_t tmem = ctl->tmem_slot;
  bb::pdl_sync();
  // S^T[b] at tmem + 64 b, dP^T[b] at tmem + 128 + 64 b (b < 2)
  const uint32_t tDV = tmem + 256, tDK = tmem + 320, tDQ = tmem + 384;    // dQ[b] at tDQ + 64 b

  if (warp == 0) {
    if (bb::elect_one()) {
      bb::mbar_arrive_expect_tx(kv_full, 2 * TILE_BYTES);
      bb::tma_load_3d(sK, &tm128, kv_full, colk, k0, batch);
      bb::tma_load_3d(sV, &tm128, kv_full, colv, k0, batch);
    }
    __syncwarp();
    for (int i = 0; i < nblk; ++i) {
      const int s = i % NST3;
      if (!bb::mbar_wait_warp(&q_empty[s], ((i / NST3) & 1) ^ 1, &ctl->abort_flag, p.status)) break;
      if (bb::elect_one()) {
        bb::mbar_arrive_expect_tx(&q_full[s], 2 * SUB_BYTES);
        bb::tma_load_3d(sQ + s * SUB_BYTES, &tm64, &q_full[s], colq, (qstart + i) * SUB, batch);
        bb::tma_load_3d(sDO + s * SUB_BYTES, &tm_do64, &q_full[s], colq, (qstart + i) * SUB, batch);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    // score products: one thread issues S^T = K . Q^T and dP^T = V . dO^T for every sub-block, as soon as its
    // operands have landed and the group that owns the score buffer has read the previous contents
    const uint64_t dK0 = desc_k0(bb::smem_u32(sK)), dV0 = desc_k0(bb::smem_u32(sV));
    const uint64_t dQ0 = desc_k0(bb::smem_u32(sQ)), dDO0 = desc_k0(bb::smem_u32(sDO));   // stage 0; stage s: + s * SUB_BYTES / 16
    const uint32_t i_s = idesc(64, 0, 0);
    bool alive = bb::mbar_wait_warp(kv_full, 0, &ctl->abort_flag, p.status);
    for (int i = 0; i < nblk && alive; ++i) {
      const int s = i % NST3, b = i & 1;
      if (!bb::mbar_wait_warp(&q_full[s], (i / NST3) & 1, &ctl->abort_flag, p.status)) break;
      if (!bb::mbar_wait_warp(&s_empty[b], ((i >> 1) & 1) ^ 1, &ctl->abort_flag, p.status)) break;
      bb::tc_fence_after_sync();
      if (bb::elect_one()) {
        const uint64_t dQ = dQ0 + (uint64_t)(s * (SUB_BYTES >> 4)), dDO = dDO0 + (uint64_t)(s * (SUB_BYTES >> 4));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          bb::umma_f16(tmem + 64 * b, desc_kmajor(dK0, k), desc_kmajor(dQ, k), i_s, k > 0);
          bb::umma_f16(tmem + 128 + 64 * b, desc_kmajor(dV0, k), desc_kmajor(dDO, k), i_s, k > 0);
        }
        bb::umma_commit(&s_full[b]);
      }
      __syncwarp();
    }
  } else if (warp == 2) {
    // updates: a second issuing thread, so that the score products of the next sub-blocks never queue
    // behind a wait for staged operands (and the two instruction streams issue side by side)
    const uint64_t dQm0 = desc_mn0(bb::smem_u32(sQ)), dDOm0 = desc_mn0(bb::smem_u32(sDO));
    const uint64_t dP0 = desc_k0(bb::smem_u32(sP)), dDS0 = desc_k0(bb::smem_u32(sDS));
    // dS^T of a pair slot read with the queries as M: two 64-query blocks one tile apart, 8-key groups 1 KiB apart
    const uint64_t dDSm0 = bb::make_smem_desc_sw128(bb::smem_u32(sDS), TILE_BYTES, 1024);
    const uint64_t dKm0 = desc_mn0(bb::smem_u32(sK));
    const uint32_t i_acc = idesc(64, 0, 1), i_dq = idesc(64, 1, 1);
    bool alive = bb::mbar_wait_warp(kv_full, 0, &ctl->abort_flag, p.status);
    for (int ii = 0; ii < nblk && alive; ++ii) {
      const int s2 = ii % NST3, g2 = ii & 1, pair = ii >> 1, ps = pair & 1;
      // (the sub-tiles landed long ago - the score products read them; the wait makes them visible to this thread)
      if (!bb::mbar_wait_warp(&q_full[s2], (ii / NST3) & 1, &ctl->abort_flag, p.status)) break;
      if (!bb::mbar_wait_warp(&p_full[g2], pair & 1, &ctl->abort_flag, p.status)) break;
      bb::tc_fence_after_sync();
      if (bb::elect_one()) {
        const uint64_t dQ2 = dQm0 + (uint64_t)(s2 * (SUB_BYTES >> 4)), dDO2 = dDOm0 + (uint64_t)(s2 * (SUB_BYTES >> 4));
        const uint64_t dP = dP0 + (uint64_t)(g2 * (TILE_BYTES >> 4));
        const uint64_t dDS = dDS0 + (uint64_t)((ps * 2 + g2) * (TILE_BYTES >> 4));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          bb::umma_f16(tDV, desc_kmajor(dP, k), desc_mnmajor64(dDO2, k), i_acc, (ii > 0 || k > 0));
          bb::umma_f16(tDK, desc_kmajor(dDS, k), desc_mnmajor64(dQ2, k), i_acc, (ii > 0 || k > 0));
        }
        bb::umma_commit(&p_empty[g2]);
        bb::umma_commit(&q_empty[s2]);
      }
      __syncwarp();
      if (g2 == 1) {
        // both halves of the pair are staged: dQ[pair] = dS . K over the tile's 128 keys
        if (!bb::mbar_wait_warp(&dq_empty[pair & 1], ((pair >> 1) & 1) ^ 1, &ctl->abort_flag, p.status)) break;
        bb::tc_fence_after_sync();
        if (bb::elect_one()) {
          const uint64_t dA = dDSm0 + (uint64_t)(ps * 2 * (TILE_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < 8; ++k)
            bb::umma_f16(tDQ + 64 * (pair & 1), desc_mnmajor64(dA, k), desc_mnmajor64(dKm0, k), i_dq, k > 0);
          bb::umma_commit(&ds_empty[ps]);
          bb::umma_commit(&dq_full[pair & 1]);
          if (ii == nblk - 1) bb::umma_commit(acc_full);
        }
        __syncwarp();
      }
    }
  } else if (warp == 3) {
    const float* lse_g = p.lse + ((long long)batch * p.H + head) * p.S;
    const float* delta_g = p.delta + ((long long)batch * p.H + head) * p.S;
    for (int i = 0; i < nblk; ++i) {
      // two queries per lane; the updates of the sub-block that had the slot before have retired
      float l2[2], d2[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int q = (qstart + i) * SUB + lane + 32 * u;
        l2[u] = (q < p.S) ? -(lse_g[q] * LOG2E) : 0.f;
        d2[u] = (q < p.S) ? -delta_g[q] : 0.f;
      }
      if (i >= NSTAT && !bb::mbar_wait_warp(&q_empty[(i - NSTAT) % NST3], ((i - NSTAT) / NST3) & 1, &ctl->abort_flag, p.status)) break;
      const int st = i % NSTAT;
#pragma unroll
      for (int u = 0; u < 2; ++u) { s_lse[st * SUB + lane + 32 * u] = l2[u]; s_delta[st * SUB + lane + 32 * u] = d2[u]; }
      __syncwarp();
      if (lane == 0) bb::mbar_arrive(&st_full[st]);
    }
  } else if (warp >= 4) {
    const int g = (warp - 4) >> 3;
    const int hf = ((warp - 4) >> 2) & 1;                  // which 32 of the sub-block's 64 query columns
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;                   // key row inside the tile / query row inside a pair
    const int krow = k0 + row;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const float sl = p.scale * LOG2E;
    uint8_t* myP = sP + g * TILE_BYTES;
    uint8_t* myDQ = sDQ + (warp - 4) * 2048;
    const int dq_col = g * 32 + hf * 16;                   // this warp's columns of a pair's dQ
    const long long acc_row0 = ((long long)batch * p.H + head) * p.S;
    bool alive = true;
    // This warp's part of one pair's dQ: tensor memory -> staging tile -> add-reduction into the accumulator.  Rows past the
    // sequence end belong to the next (batch, head): they add zeros, also where a key is Inf or NaN (a tensor map with a
    // sequence dimension, which leaves such rows out, costs every reduction: B8 H16 S1024 non-causal 222 -> 228 us).
    auto drain = [&](int pair) {
      if (!bb::mbar_wait_warp(&dq_full[pair & 1], (pair >> 1) & 1, &ctl->abort_flag, p.status)) alive = false;
      bb::tc_fence_after_sync();
      uint32_t r[16];
      bb::tmem_ld_32x32b_x16(tDQ + 64 * (pair & 1) + lane_addr + dq_col, r);
      bb::tmem_ld_wait();
      bb::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        bb::mbar_arrive(&dq_empty[pair & 1]);
        bb::bulk_wait_group_read<0>();                     // the staging tile: the previous pair's reduction has read it
      }
      __syncwarp();
      const int q0 = (qstart + 2 * pair) * SUB + quarter * 32;
      if (!alive || q0 >= p.S) return;                     // (a warp that gave up adds nothing to the accumulator)
      if (q0 + lane >= p.S) {
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = 0u;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(myDQ + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = make_uint4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
      bb::fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        bb::tma_reduce_add_2d(&tm_acc, myDQ, dq_col, (int)(acc_row0 + q0));
        bb::bulk_commit_group();
      }
    };
    int n = 0;
    for (int i = g; i < nblk; i += 2, ++n) {
      const int q0 = (qstart + i) * SUB + hf * 32;           // first query of this thread's columns
      const int ps = n & 1;                                  // sub-block i belongs to pair n
      const float* my_lse = s_lse + (i % NSTAT) * SUB + hf * 32;
      const float* my_delta = s_delta + (i % NSTAT) * SUB + hf * 32;
      const uint32_t tS = tmem + 64 * g, tDP = tmem + 128 + 64 * g;
      if (!bb::mbar_wait_warp(&st_full[i % NSTAT], (i / NSTAT) & 1, &ctl->abort_flag, p.status) ||
          !bb::mbar_wait_warp(&s_full[g], n & 1, &ctl->abort_flag, p.status)) alive = false;
      bb::tc_fence_after_sync();
      uint32_t pkP[16], pkDS[16];                            // this thread's 32 P^T and dS^T values as bf16 pairs
      {
        float sv[32], dp[32];
        ld32x2(tS + lane_addr + hf * 32, tDP + lane_addr + hf * 32, sv, dp);
        // the scores are in registers: the buffer can take the sub-block after next while this one is worked on
        bb::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) bb::mbar_arrive(&s_empty[g]);
        // (keys past the sequence end must not reach dQ: their rows of dK / dV are simply not stored)
        if (q0 + 32 > p.S || k0 + TQ > p.S || (p.causal && k0 + TQ - 1 > q0))
          dkv_math<true>(sv, dp, my_lse, my_delta, sl, p.causal ? krow - q0 : 0, krow < p.S ? p.S - 1 - q0 : -1, pkP, pkDS);
        else
          dkv_math<false>(sv, dp, my_lse, my_delta, sl, 0, 0, pkP, pkDS);
      }
      // P^T's buffer is free once the dV update that read it retired; the pair slot's dS^T buffers once
      // the dK updates and the dQ product of the pair that used the slot before have
      if (!bb::mbar_wait_warp(&p_empty[g], (n & 1) ^ 1, &ctl->abort_flag, p.status) ||
          !bb::mbar_wait_warp(&ds_empty[ps], ((n >> 1) & 1) ^ 1, &ctl->abort_flag, p.status)) alive = false;
      atom_store_half_row(myP, row, hf, pkP);
      atom_store_half_row(sDS + (ps * 2 + g) * TILE_BYTES, row, hf, pkDS);
      bb::fence_proxy_async();
      __syncwarp();
      if (lane == 0) bb::mbar_arrive(&p_full[g]);
      // the previous pair, whose second half was staged one iteration ago
      if (n > 0) drain(n - 1);
    }
    drain(npairs - 1);
    if (!bb::mbar_wait_warp(acc_full, 0, &ctl->abort_flag, p.status)) alive = false;
    if (alive) {
      bb::tc_fence_after_sync();
      float v[32];
      // the two groups split the final stores: group 0 writes dV, group 1 writes dK
      const uint32_t src = (g == 0) ? tDV : tDK;
      ld32(src + lane_addr + hf * 32, v);
      __nv_bfloat16* dst = (g == 0) ? p.dv : p.dk;
      const int w0 = k0 + quarter * 32;
      store_tile32(myP + (hf * 4 + quarter) * 2048, dst + (long long)(row_base + w0) * p.stride_dqkv + colq + hf * 32, p.stride_dqkv, p.S - w0, lane, v, g == 0 ? 1.f : p.scale);
    }
    if (lane == 0) bb::bulk_wait_group_read<0>();          // the reductions read this CTA's shared memory
  }
  bb::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) bb::tmem_dealloc(tmem, 512);
}

constexpr int BWD3_SMEM = 2 * TILE_BYTES + 2 * NST3 * SUB_BYTES + 2 * TILE_BYTES + 4 * TILE_BYTES + 2 * TILE_BYTES + 2 * NSTAT * SUB * (int)sizeof(float) +
                          (int)sizeof(Ctl) + 1024;

// dq (bf16, packed projection layout) = scale * accumulator; eight values per thread
__global__ void __launch_bounds__(256)
attn_tc_dq_convert_kernel(const TcParams p) {
  bb::pdl_sync();
  const int per_tok = p.H * 8;
  const long long total = (long long)p.B * p.S * per_tok;
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < total; c += (long long)gridDim.x * blockDim.x) {
    const long long tok = c / per_tok;
    const int within = (int)(c % per_tok), head = within >> 3, part = within & 7;
    const float4* src = reinterpret_cast<const float4*>(p.dq_acc + (((tok / p.S) * p.H + head) * p.S + (tok % p.S)) * HD + part * 8);
    const float4 a = __ldcg(src), b = __ldcg(src + 1);
    uint4 o;
    o.x = bb::pack_bf16x2(a.x * p.scale, a.y * p.scale); o.y = bb::pack_bf16x2(a.z * p.scale, a.w * p.scale);
    o.z = bb::pack_bf16x2(b.x * p.scale, b.y * p.scale); o.w = bb::pack_bf16x2(b.z * p.scale, b.w * p.scale);
    *reinterpret_cast<uint4*>(p.dq + tok * p.stride_dqkv + head * HD + part * 8) = o;
  }
}

// ------------------------------------------------------------------ forward at head dimension 128 (two query tiles in ping-pong)
// A CTA owns 256 query rows of one (batch, head) as two 128-row tiles; compute group g (4 warps,
// one query row per thread) runs the online softmax of tile g.  Keys/values stream in 64-row
// sub-tiles that serve both query tiles.  Per sub-block jj and group g:
//   S_g(jj) = Q_g K_jj^T  ->  P_g = exp2(S_g * c - m_g)  ->  PV_g(jj) = P_g V_jj
// Scores are double-buffered in tensor memory and issued two sub-blocks ahead, so a group never
// waits for the tensor core between sub-blocks; P goes through shared memory (bf16, two buffers
// per group).  The output row accumulates in tensor memory over all sub-blocks (O_g += P_g V_jj);
// the exponent reference of a row only moves when the running maximum has grown by more than 2^8
// since it was set, and only then is the row's accumulator rescaled (tensor memory -> registers ->
// tensor memory, between two P V products): after the first few sub-blocks that is rare, and the
// per-sub-block work of a thread is the softmax alone.  P <= 2^8 and the row sums stay far inside
// fp32 / bf16 range; the final division by the row sum makes the choice of reference immaterial.
// smem: Q_0, Q_1 [128 x D] | K, V sub-tiles [64 x D] x NKV stages | P_g,b [128 x 64] x 4
// TMEM: S_g,b at 128 g + 64 b | O_g at 256 + 128 g (D columns)
// A [rows x 128] operand lies in shared memory as two [rows x 64] atoms of
// 128-byte rows, one after the other (two TMA boxes): the score product walks its eight 16-column k-steps
// through both atoms; V as the B operand of P V (N = D, its columns) names the distance between the atoms in
// the descriptor's leading-dimension field.  The whole tensor memory is in use (2 x 2 score
// buffers of 64 columns, 2 outputs of 128).
struct Fwd2 {
  static constexpr int D = 128;
  static constexpr int NA = D / 64;                            // 64-column atoms per row
  static constexpr int NKV = 3;                                // sub-tile ring depth
  static constexpr int Q_BYTES = NA * TILE_BYTES;              // one query tile
  static constexpr int KV_BYTES = NA * SUB_BYTES;              // one key (or value) sub-tile
  static constexpr int SMEM = 2 * Q_BYTES + 2 * NKV * KV_BYTES + 4 * TILE_BYTES + (int)sizeof(Ctl) + 1024;
};
// warps: 0 TMA, 1 score products, 2 P V products (two issuing threads: the issue path of the small MMAs is the
// bound, and two instruction streams get about a third more through it than one), 3..10 the two softmax groups
constexpr int FWD2_THREADS = 96 + 256;

// one row (64 values) of a [128 x 64] bf16 atom
__device__ __forceinline__ void atom_store_row64(uint8_t* atom, int row, const float* a /*32*/, const float* b /*32*/) {
  uint8_t* base = atom + row * 128;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const float* v = (c < 4) ? a + 8 * c : b + 8 * (c - 4);
    uint4 q;
    q.x = bb::pack_bf16x2(v[0], v[1]); q.y = bb::pack_bf16x2(v[2], v[3]);
    q.z = bb::pack_bf16x2(v[4], v[5]); q.w = bb::pack_bf16x2(v[6], v[7]);
    *reinterpret_cast<uint4*>(base + ((c ^ (row & 7)) << 4)) = q;
  }
}

__global__ void __launch_bounds__(FWD2_THREADS, 1)
attn_tc_fwd2_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kv, const TcParams p) {
  using C = Fwd2;
  constexpr int D = C::D, NA = C::NA, NKV = C::NKV, Q_BYTES = C::Q_BYTES, KV_BYTES = C::KV_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                          // 2 tiles
  uint8_t* sK = sQ + 2 * Q_BYTES;              // NKV sub-tiles
  uint8_t* sV = sK + NKV * KV_BYTES;           // NKV sub-tiles
  uint8_t* sP = sV + NKV * KV_BYTES;           // [group][buffer] x 16 KiB
  Ctl* ctl = reinterpret_cast<Ctl*>(sP + 4 * TILE_BYTES);
  uint64_t* q_full = &ctl->bars[0];
  uint64_t* kv_full = &ctl->bars[1];           // [NKV]
  uint64_t* kv_empty = &ctl->bars[1 + NKV];    // [NKV]
  uint64_t* s_full = &ctl->bars[1 + 2 * NKV];  // [group][buffer] scores ready
  uint64_t* p_full = s_full + 4;               // [group] probabilities in shared memory, scores read
  uint64_t* pv_full = p_full + 2;              // [group] P V product ready
  // [group][buffer] the group is done with the scores in this buffer.  Completes at the same moment as p_full, but
  // per buffer: its next phase needs the next score product into the buffer, which only the waiter issues, so
  // the waiter can never find it two phases on (p_full can be: the other issuing warp moves that one along)
  uint64_t* s_free = pv_full + 2;

  const int warp = bb::warp_index(), lane = threadIdx.x & 31;
  const TileId id = tile_id(p);
  const int cb = (p.S + 2 * TQ - 1) / (2 * TQ) - 1 - id.tile, head = id.head, batch = id.batch;   // long CTAs first
  const int row_base = batch * p.S;
  const int colq = head * D, colk = p.hidden + head * D, colv = 2 * p.hidden + head * D;
  const int nsub = (p.S + SUB - 1) / SUB;
  // last key sub-block of each query tile (-1: the tile lies past the end of the sequence)
  const int qa = cb * 2 * TQ, qb = qa + TQ;
  const int last0 = (qa >= p.S) ? -1 : (p.causal ? min(nsub - 1, (qa + TQ - 1) / SUB) : nsub - 1);
  const int last1 = (qb >= p.S) ? -1 : (p.causal ? min(nsub - 1, (qb + TQ - 1) / SUB) : nsub - 1);
  const int jmax = max(last0, last1);
#define BB_LAST(g) ((g) ? last1 : last0)

  if (threadIdx.x == 0) {
    ctl->abort_flag = 0;
    bb::mbar_init(q_full, 1);
    for (int i = 0; i < NKV; ++i) { bb::mbar_init(&kv_full[i], 1); bb::mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < 4; ++i) { bb::mbar_init(&s_full[i], 1); bb::mbar_init(&s_free[i], 4); }
    for (int g = 0; g < 2; ++g) { bb::mbar_init(&p_full[g], 4); bb::mbar_init(&pv_full[g], 1); }
    bb::fence_barrier_init();
    bb::tma_prefetch_desc(&tm_q); bb::tma_prefetch_desc(&tm_kv);
  }
  if (warp == 1) { bb::tmem_alloc(&ctl->tmem_slot, 512); bb::tmem_relinquish(); }
  bb::tc_fence_before_sync();
  __syncthreads();
  bb::tc_fence_after_sync();
  const uint32_t tmem = ctl->tmem_slot;
  bb::pdl_sync();

  if (warp == 0) {
    if (bb::elect_one()) {
      bb::mbar_arrive_expect_tx(q_full, 2 * Q_BYTES);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        bb::tma_load_3d(sQ + a * TILE_BYTES, &tm_q, q_full, colq + 64 * a, qa, batch);
        bb::tma_load_3d(sQ + Q_BYTES + a * TILE_BYTES, &tm_q, q_full, colq + 64 * a, qb, batch);
      }
    }
    __syncwarp();
    for (int jj = 0; jj <= jmax; ++jj) {
      const int s = jj % NKV;
      if (!bb::mbar_wait_warp(&kv_empty[s], ((jj / NKV) & 1) ^ 1, &ctl->abort_flag, p.status)) break;
      if (bb::elect_one()) {
        bb::mbar_arrive_expect_tx(&kv_full[s], 2 * KV_BYTES);
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          bb::tma_load_3d(sK + s * KV_BYTES + a * SUB_BYTES, &tm_kv, &kv_full[s], colk + 64 * a, jj * SUB, batch);
          bb::tma_load_3d(sV + s * KV_BYTES + a * SUB_BYTES, &tm_kv, &kv_full[s], colv + 64 * a, jj * SUB, batch);
        }
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    const uint64_t dQ0 = desc_k0(bb::smem_u32(sQ));
    const uint64_t dK0 = desc_k0(bb::smem_u32(sK));   // stage 0; stage s: + s * KV_BYTES / 16
    const uint32_t i_s = idesc(64, 0, 0);
    bool alive = bb::mbar_wait_warp(q_full, 0, &ctl->abort_flag, p.status);
    // scores of sub-block jj for group g into score buffer jj & 1
    auto issue_scores = [&](int g, int jj) {
      const uint64_t dK = dK0 + (uint64_t)((jj % NKV) * (KV_BYTES >> 4)), dQ = dQ0 + (uint64_t)(g * (Q_BYTES >> 4));
      const uint32_t tS = tmem + 128 * g + 64 * (jj & 1);
#pragma unroll
      for (int k = 0; k < D / 16; ++k)           // four k-steps per 64-column atom
        bb::umma_f16(tS, desc_kmajor(dQ + (uint64_t)((k >> 2) * (TILE_BYTES >> 4)), k & 3),
                     desc_kmajor(dK + (uint64_t)((k >> 2) * (SUB_BYTES >> 4)), k & 3), i_s, k > 0);
      bb::umma_commit(&s_full[2 * g + (jj & 1)]);
    };
    // prologue: the first two score products of each group
    for (int jj = 0; jj < 2 && jj <= jmax && alive; ++jj) {
      if (!bb::mbar_wait_warp(&kv_full[jj % NKV], 0, &ctl->abort_flag, p.status)) { alive = false; break; }
      bb::tc_fence_after_sync();
      if (bb::elect_one()) {
#pragma unroll
        for (int g = 0; g < 2; ++g) if (jj <= BB_LAST(g)) issue_scores(g, jj);
      }
      __syncwarp();
    }
    // steady state: the scores two sub-blocks ahead, as soon as the group has read the buffer they go to
    for (int jj = 0; jj + 2 <= jmax && alive; ++jj) {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (jj + 2 > BB_LAST(g)) continue;
        // group g is done reading S_g(jj): its buffer is free
        if (!bb::mbar_wait_warp(&s_free[2 * g + (jj & 1)], (jj >> 1) & 1, &ctl->abort_flag, p.status)) { alive = false; break; }
        if (!bb::mbar_wait_warp(&kv_full[(jj + 2) % NKV], ((jj + 2) / NKV) & 1, &ctl->abort_flag, p.status)) { alive = false; break; }
        bb::tc_fence_after_sync();
        if (bb::elect_one()) issue_scores(g, jj + 2);
        __syncwarp();
      }
    }
  } else if (warp == 2) {
    // V: [64 keys x D]; its atoms (64 columns each) lie SUB_BYTES apart, which is desc_mn0's leading-dimension field
    static_assert(SUB_BYTES == 8192, "desc_mn0 names the distance between the 64-column atoms of V");
    const uint64_t dP0 = desc_k0(bb::smem_u32(sP)), dVm0 = desc_mn0(bb::smem_u32(sV));   // stage 0; stage s: + s * KV_BYTES / 16
    const uint32_t i_pv = idesc(D, 0, 1);
    bool alive = true;
    for (int jj = 0; jj <= jmax && alive; ++jj) {
      const int s = jj % NKV;
      const uint64_t dV = dVm0 + (uint64_t)(s * (KV_BYTES >> 4));
      // (V_jj landed before the scores of this sub-block were issued; the wait makes it visible to this thread)
      if (!bb::mbar_wait_warp(&kv_full[s], (jj / NKV) & 1, &ctl->abort_flag, p.status)) break;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (jj > BB_LAST(g)) continue;
        if (!bb::mbar_wait_warp(&p_full[g], jj & 1, &ctl->abort_flag, p.status)) { alive = false; break; }
        bb::tc_fence_after_sync();
        if (bb::elect_one()) {
          const uint32_t tO = tmem + 256 + 128 * g;
          const uint64_t dPg = dP0 + (uint64_t)((2 * g + (jj & 1)) * (TILE_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < 4; ++k) bb::umma_f16(tO, desc_kmajor(dPg, k), desc_mnmajor64(dV, k), i_pv, (jj > 0 || k > 0));
          bb::umma_commit(&pv_full[g]);
        }
        __syncwarp();
      }
      // K_jj, V_jj: the score products that read K_jj retired before P(jj) existed, the P V products are issued
      if (alive && bb::elect_one()) bb::umma_commit(&kv_empty[s]);
      __syncwarp();
    }
  } else if (warp >= 3) {
    const int g = (warp - 3) >> 2;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int q0 = g ? qb : qa;
    const int qrow = q0 + row;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t tS = tmem + 128 * g + lane_addr;
    const uint32_t tO = tmem + 256 + 128 * g + lane_addr;
    const float sl = p.scale * LOG2E;
    const int lastj = BB_LAST(g);
    constexpr float REF_SLACK = 8.f;                         // log2 units the maximum may grow past the reference
    float m_ref = -INFINITY, l_i = 0.f;                     // exponent reference of this row, row sum relative to it
    bool alive = true;
    for (int jj = 0; jj <= lastj; ++jj) {
      const int b = jj & 1;
      const bool got = bb::mbar_wait(&s_full[2 * g + b], (jj >> 1) & 1, &ctl->abort_flag, p.status);
      if (!__all_sync(0xffffffffu, got)) { alive = false; break; }
      bb::tc_fence_after_sync();
      const int c0 = jj * SUB;
      // only sub-blocks that touch the causal diagonal or the end of the sequence need masks
      const bool need_mask = (c0 + SUB > p.S) || (p.causal && c0 + SUB - 1 > q0);
      float sa[32], sb[32];                                  // the row's 64 scores stay in registers
      ld32x2(tS + 64 * b, tS + 64 * b + 32, sa, sb);
      float mx = -INFINITY;
      if (!need_mask) {
#pragma unroll
        for (int i = 0; i < 32; ++i) mx = fmaxf(mx, fmaxf(sa[i], sb[i]));
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int ca = c0 + i, cc = ca + 32;
          if (ca >= p.S || (p.causal && ca > qrow)) sa[i] = -INFINITY;
          if (cc >= p.S || (p.causal && cc > qrow)) sb[i] = -INFINITY;
          mx = fmaxf(mx, fmaxf(sa[i], sb[i]));
        }
      }
      mx *= sl;                                              // scale > 0: the maximum commutes with it
      // move the reference only when the maximum outgrew it by more than the slack
      float alpha = 1.f;
      if (mx > m_ref + REF_SLACK || (m_ref == -INFINITY && mx > -INFINITY)) {
        alpha = ex2(m_ref - mx);                             // 0 for the first finite maximum
        m_ref = mx;
        l_i *= alpha;
      }
      const float nm = (m_ref == -INFINITY) ? 0.f : -m_ref;
      float rs = 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {                         // exp2(-inf) = 0 covers the masked entries
        sa[i] = ex2(fmaf(sa[i], sl, nm)); sb[i] = ex2(fmaf(sb[i], sl, nm));
        rs += sa[i] + sb[i];
      }
      l_i += rs;
      if (jj > 0) {
        // the previous product has retired: its P buffer is free and the accumulator is at rest
        const bool ok = bb::mbar_wait(&pv_full[g], (jj - 1) & 1, &ctl->abort_flag, p.status);
        if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
          // some row of this warp moved its reference: rescale the warp's accumulator rows in place
          bb::tc_fence_after_sync();
#pragma unroll
          for (int h = 0; h < D / 32; ++h) {
            uint32_t r[32];
            bb::tmem_ld_32x32b_x32(tO + 32 * h, r);
            bb::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            bb::tmem_st_32x32b_x32(tO + 32 * h, r);
          }
          bb::tmem_st_wait();
        }
      }
      atom_store_row64(sP + (2 * g + b) * TILE_BYTES, row, sa, sb);
      bb::tc_fence_before_sync();
      bb::fence_proxy_async();
      __syncwarp();
      if (lane == 0) { bb::mbar_arrive(&p_full[g]); bb::mbar_arrive(&s_free[2 * g + b]); }
    }
    if (lastj >= 0) {
      const bool fin = alive && bb::mbar_wait(&pv_full[g], lastj & 1, &ctl->abort_flag, p.status);
      if (__all_sync(0xffffffffu, fin)) {
        bb::tc_fence_after_sync();
        const float inv = l_i > 0.f ? 1.f / l_i : 0.f;
        const int w0 = q0 + quarter * 32;
        uint8_t* tile = sP + 2 * g * TILE_BYTES + quarter * 4096;              // (the group's P buffers: every product has retired)
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          float o[64];
          ld32x2(tO + 64 * a, tO + 64 * a + 32, o, o + 32);
          __nv_bfloat16* dst = p.out + (long long)(row_base + w0) * p.stride_o + colq + 64 * a;
          store_tile32(tile, dst, p.stride_o, p.S - w0, lane, o, inv);
          store_tile32(tile + 2048, dst + 32, p.stride_o, p.S - w0, lane, o + 32, inv);
        }
        if (qrow < p.S) {
          p.lse[((long long)batch * p.H + head) * p.S + qrow] = (l_i > 0.f) ? (m_ref + log2f(l_i)) / LOG2E : -INFINITY;
        }
      }
    }
  }
  bb::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) bb::tmem_dealloc(tmem, 512);
}
#undef BB_LAST


// ------------------------------------------------------------------ forward at head dimension 64 (three CTAs per SM)
// A softmax row is a chain (scores out of tensor memory, maximum, exponentials, P to shared memory) that leaves most
// issue slots empty, and a CTA's start and end (tensor-memory allocation, first loads, last store) leave the whole SM
// empty; what fills both is other CTAs.  So a CTA is small - 128 query rows, one softmax thread per row, 128 columns of
// tensor memory, 73 KiB of shared memory - and three of them share an SM (twelve softmax warps instead of the eight of
// the two-tile kernel above, which takes all of tensor memory).  The scores have one buffer: the group hands it back as
// soon as they are in registers, so the next score product runs under the exponentials.  Exponent reference, in-place
// rescaling and the final division are the two-tile kernel's.  B8 H16 S1024: causal 68 -> 51 us, non-causal 100 -> 76 us
// (issue slots were 35 % busy, MUFU 33 %, the tensor pipe 28 % before).
// smem: Q [128 x 64] | K x 3, V x 2 sub-tiles [64 x 64] | P [128 x 64]          TMEM: S 64 columns | O 64 columns
constexpr int FWD3_NK = 3, FWD3_NV = 2;
constexpr int FWD3_SMEM = 2 * TILE_BYTES + (FWD3_NK + FWD3_NV) * SUB_BYTES + (int)sizeof(Ctl) + 1024;
// One warp issues both the loads and the MMAs: fifteen warps leave 128 registers a thread, eighteen would leave 96 and
// the row's 64 scores would spill.
constexpr int FWD3_THREADS = 32 + 128;         // issuing warp, four softmax warps
static_assert(3 * (FWD3_SMEM + 1024) <= 228 * 1024, "three CTAs per SM");

__global__ void __launch_bounds__(FWD3_THREADS, 3)
attn_tc_fwd3_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kv, const TcParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sP = sQ + TILE_BYTES;
  uint8_t* sK = sP + TILE_BYTES;               // FWD3_NK sub-tiles
  uint8_t* sV = sK + FWD3_NK * SUB_BYTES;      // FWD3_NV sub-tiles
  Ctl* ctl = reinterpret_cast<Ctl*>(sV + FWD3_NV * SUB_BYTES);
  uint64_t* q_full = &ctl->bars[0];
  uint64_t* k_full = q_full + 1;               // [FWD3_NK]
  uint64_t* v_full = k_full + FWD3_NK;         // [FWD3_NV]
  // Every hand-off below has one waiter, whose next action the barrier's next phase depends on, so none can find its
  // barrier two phases on.
  uint64_t* s_full = v_full + FWD3_NV;         // scores ready
  uint64_t* s_free = s_full + 1;               // scores in registers
  uint64_t* p_full = s_free + 1;               // probabilities in shared memory
  uint64_t* pv_full = p_full + 1;              // P V product retired

  const int warp = bb::warp_index(), lane = threadIdx.x & 31;
  const TileId id = tile_id(p);
  const int q0 = ((p.S + TQ - 1) / TQ - 1 - id.tile) * TQ;       // long CTAs first
  const int row_base = id.batch * p.S;
  const int colq = id.head * HD, colk = p.hidden + id.head * HD, colv = 2 * p.hidden + id.head * HD;
  const int nsub = (p.S + SUB - 1) / SUB;
  const int nblk = p.causal ? min(nsub, (q0 + TQ) / SUB) : nsub;

  if (threadIdx.x == 0) {
    ctl->abort_flag = 0;
    bb::mbar_init(q_full, 1);
    for (int i = 0; i < FWD3_NK; ++i) bb::mbar_init(&k_full[i], 1);
    for (int i = 0; i < FWD3_NV; ++i) bb::mbar_init(&v_full[i], 1);
    bb::mbar_init(s_full, 1); bb::mbar_init(s_free, 4); bb::mbar_init(p_full, 4); bb::mbar_init(pv_full, 1);
    bb::fence_barrier_init();
    bb::tma_prefetch_desc(&tm_q); bb::tma_prefetch_desc(&tm_kv);
  }
  if (warp == 0) { bb::tmem_alloc(&ctl->tmem_slot, 128); bb::tmem_relinquish(); }
  bb::tc_fence_before_sync();
  __syncthreads();
  bb::tc_fence_after_sync();
  const uint32_t tmem = ctl->tmem_slot;
  bb::pdl_sync();

  if (warp == 0) {
    auto load_k = [&](int j) {
      const int s = j % FWD3_NK;
      bb::mbar_arrive_expect_tx(&k_full[s], SUB_BYTES);
      bb::tma_load_3d(sK + s * SUB_BYTES, &tm_kv, &k_full[s], colk, j * SUB, id.batch);
    };
    auto load_v = [&](int j) {
      const int s = j % FWD3_NV;
      bb::mbar_arrive_expect_tx(&v_full[s], SUB_BYTES);
      bb::tma_load_3d(sV + s * SUB_BYTES, &tm_kv, &v_full[s], colv, j * SUB, id.batch);
    };
    if (bb::elect_one()) {
      bb::mbar_arrive_expect_tx(q_full, TILE_BYTES);
      bb::tma_load_3d(sQ, &tm_q, q_full, colq, q0, id.batch);
      load_k(0);
      if (nblk > 1) load_k(1);
      load_v(0);
    }
    __syncwarp();
    const uint64_t dQ = desc_k0(bb::smem_u32(sQ)), dK0 = desc_k0(bb::smem_u32(sK));
    const uint64_t dP = desc_k0(bb::smem_u32(sP)), dV0 = desc_mn0(bb::smem_u32(sV));
    const uint32_t i_s = idesc(64, 0, 0), i_pv = idesc(HD, 0, 1);
    bool alive = bb::mbar_wait_warp(q_full, 0, &ctl->abort_flag, p.status);
    // step j: the scores of sub-block j (their buffer is free once those of j - 1 are in registers), then the P V
    // product of sub-block j - 1.  The same waits say which operands are spent: s_free(j - 1) that the score product
    // of j - 1 has retired (K_{j+2} takes its slot), p_full(j - 1) that the P V product of j - 2 has (V_j takes its).
    for (int j = 0; j <= nblk && alive; ++j) {
      if (j < nblk) {
        const int s = j % FWD3_NK;
        if (!bb::mbar_wait_warp(&k_full[s], (j / FWD3_NK) & 1, &ctl->abort_flag, p.status)) break;
        if (j > 0 && !bb::mbar_wait_warp(s_free, (j - 1) & 1, &ctl->abort_flag, p.status)) break;
        bb::tc_fence_after_sync();
        if (bb::elect_one()) {
          const uint64_t dK = dK0 + (uint64_t)(s * (SUB_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < 4; ++k) bb::umma_f16(tmem, desc_kmajor(dQ, k), desc_kmajor(dK, k), i_s, k > 0);
          bb::umma_commit(s_full);
          if (j + 2 < nblk) load_k(j + 2);
        }
        __syncwarp();
      }
      if (j > 0) {
        const int jj = j - 1, s = jj % FWD3_NV;
        if (!bb::mbar_wait_warp(&v_full[s], (jj / FWD3_NV) & 1, &ctl->abort_flag, p.status)) break;
        if (!bb::mbar_wait_warp(p_full, jj & 1, &ctl->abort_flag, p.status)) break;
        bb::tc_fence_after_sync();
        if (bb::elect_one()) {
          const uint64_t dV = dV0 + (uint64_t)(s * (SUB_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < 4; ++k) bb::umma_f16(tmem + 64, desc_kmajor(dP, k), desc_mnmajor64(dV, k), i_pv, (jj > 0 || k > 0));
          bb::umma_commit(pv_full);
          if (j < nblk) load_v(j);
        }
        __syncwarp();
      }
    }
  } else {
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int qrow = q0 + row;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t tS = tmem + lane_addr, tO = tmem + 64 + lane_addr;
    const float sl = p.scale * LOG2E;
    constexpr float REF_SLACK = 8.f;                         // log2 units the maximum may grow past the reference
    float m_ref = -INFINITY, l_i = 0.f;                     // exponent reference of this row, row sum relative to it
    bool alive = true;
    for (int j = 0; j < nblk; ++j) {
      if (!bb::mbar_wait_warp(s_full, j & 1, &ctl->abort_flag, p.status)) { alive = false; break; }
      bb::tc_fence_after_sync();
      const int c0 = j * SUB;
      // only sub-blocks that touch the causal diagonal or the end of the sequence need masks
      const bool need_mask = (c0 + SUB > p.S) || (p.causal && c0 + SUB - 1 > q0);
      uint32_t sc[64];                                       // the row's scores
      bb::tmem_ld_32x32b_x32(tS, sc);
      bb::tmem_ld_32x32b_x32(tS + 32, sc + 32);
      bb::tmem_ld_wait();
      bb::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) bb::mbar_arrive(s_free);
      if (need_mask) {
        const int last = min(p.S - 1, p.causal ? qrow : p.S - 1) - c0;      // last visible column of this row
#pragma unroll
        for (int i = 0; i < 64; ++i) if (i > last) sc[i] = 0xFF800000u;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 64; i += 2)
        mx4[(i >> 1) & 3] = fmaxf(mx4[(i >> 1) & 3], fmaxf(__uint_as_float(sc[i]), __uint_as_float(sc[i + 1])));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl;     // scale > 0: the maximum commutes with it
      // move the reference only when the maximum outgrew it by more than the slack
      float alpha = 1.f;
      if (mx > m_ref + REF_SLACK || (m_ref == -INFINITY && mx > -INFINITY)) {
        alpha = ex2(m_ref - mx);                             // 0 for the first finite maximum
        m_ref = mx;
        l_i *= alpha;
      }
      const float nm = (m_ref == -INFINITY) ? 0.f : -m_ref;
      // exp2(-inf) = 0 covers the masked entries.  The row sum takes columns i and i + 32 together, i ascending: the
      // two-tile kernel's order, so that a row's result does not depend on which kernel computed it
      float rs = 0.f;
      uint32_t pk[32];
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float x0 = ex2(fmaf(__uint_as_float(sc[i]), sl, nm)), y0 = ex2(fmaf(__uint_as_float(sc[i + 32]), sl, nm));
        const float x1 = ex2(fmaf(__uint_as_float(sc[i + 1]), sl, nm)), y1 = ex2(fmaf(__uint_as_float(sc[i + 33]), sl, nm));
        rs += x0 + y0;
        rs += x1 + y1;
        pk[i >> 1] = bb::pack_bf16x2(x0, x1);
        pk[16 + (i >> 1)] = bb::pack_bf16x2(y0, y1);
      }
      l_i += rs;
      if (j > 0) {
        // the previous product has retired: its P buffer is free and the accumulator is at rest
        if (!bb::mbar_wait_warp(pv_full, (j - 1) & 1, &ctl->abort_flag, p.status)) { alive = false; break; }
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
          // some row of this warp moved its reference: rescale the warp's accumulator rows in place
          bb::tc_fence_after_sync();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[32];
            bb::tmem_ld_32x32b_x32(tO + 32 * h, r);
            bb::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            bb::tmem_st_32x32b_x32(tO + 32 * h, r);
          }
          bb::tmem_st_wait();
        }
      }
      atom_store_half_row(sP, row, 0, pk);
      atom_store_half_row(sP, row, 1, pk + 16);
      bb::tc_fence_before_sync();
      bb::fence_proxy_async();
      __syncwarp();
      if (lane == 0) bb::mbar_arrive(p_full);
    }
    if (alive && bb::mbar_wait_warp(pv_full, (nblk - 1) & 1, &ctl->abort_flag, p.status)) {
      bb::tc_fence_after_sync();
      const float inv = l_i > 0.f ? 1.f / l_i : 0.f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float o[32];
        ld32(tO + 32 * h, o);
        const int w0 = q0 + quarter * 32;                      // (P is free: its last product has retired)
        store_tile32(sP + quarter * 4096 + h * 2048, p.out + (long long)(row_base + w0) * p.stride_o + colq + 32 * h, p.stride_o, p.S - w0, lane, o, inv);
      }
      if (qrow < p.S) {
        p.lse[((long long)id.batch * p.H + id.head) * p.S + qrow] = (l_i > 0.f) ? (m_ref + log2f(l_i)) / LOG2E : -INFINITY;
      }
    }
  }
  bb::tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) bb::tmem_dealloc(tmem, 128);
}

template <typename K> int set_smem(K kernel, int bytes) {
  BB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return BB_OK;
}

}  // namespace

// Entry points used by attention.cu's dispatch, head dimensions 64 and 128.
int bb_attention_tc_fwd(const void* qkv_q, void* out, float* lse, int B, int H, int S, int D, long long stride_qkv,
                        long long stride_o, int causal, float scale, cudaStream_t stream) {
  if (D != 64 && D != 128) return BB_ERR_UNSUPPORTED;
  if (int rc = bbhost::bind_context()) return rc;
  CUtensorMap tm_q, tm_kv;
  // the packed projection [B, S, 3*H*D]: q, k, v blocks of H*D columns each; boxes of 64 columns (one
  // 128-byte swizzle atom), 128 rows for the query tiles, 64 rows for the streamed key/value sub-tiles.  A tile past a
  // sequence's end reads zeros, not the next sequence: a masked probability of zero times an Inf or NaN there is NaN
  if (int rc = bbhost::encode_seqs(&tm_q, qkv_q, B, S, 3LL * H * D, stride_qkv, 64, TQ)) return rc;
  if (int rc = bbhost::encode_seqs(&tm_kv, qkv_q, B, S, 3LL * H * D, stride_qkv, 64, SUB)) return rc;
  TcParams p = {};
  p.out = (__nv_bfloat16*)out; p.lse = lse; p.stride_o = stride_o; p.B = B; p.H = H; p.S = S; p.hidden = H * D;
  p.causal = causal; p.scale = scale; p.status = bb_device_status_word();
  // Three CTAs per SM at 64; at 128 a CTA's scores and output take more than a third of tensor memory (S 64 + O 128
  // columns, allocated in powers of two), and the two-tile kernel keeps the softmax groups on the SM instead.
  if (D == 64) {
    BB_ONCE_PER_DEVICE({ if (int rc = set_smem(attn_tc_fwd3_kernel, FWD3_SMEM)) return rc; });
    bb_launch(attn_tc_fwd3_kernel, (S + TQ - 1) / TQ * H * B, FWD3_THREADS, FWD3_SMEM, stream, tm_q, tm_kv, p);
  } else {
    BB_ONCE_PER_DEVICE({ if (int rc = set_smem(attn_tc_fwd2_kernel, Fwd2::SMEM)) return rc; });
    bb_launch(attn_tc_fwd2_kernel, (S + 2 * TQ - 1) / (2 * TQ) * H * B, FWD2_THREADS, Fwd2::SMEM, stream, tm_q, tm_kv, p);
  }
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}

namespace {
// BB_ATTENTION_BWD=split in the environment selects the two-role kernel (dK/dV and dQ computed by
// different CTAs, every sum in a fixed order) at head dimension 64; the default there is the fused kernel
bool split_backward() {
  static const bool split = [] { const char* e = getenv("BB_ATTENTION_BWD"); return e && e[0] == 's'; }();
  return split;
}

// the two-role kernel (see attn_tc_bwd2_kernel): delta pre-pass, then dK / dV and dQ tiles in one launch
template <int D>
int launch_bwd2(const CUtensorMap& tm_qkv, const CUtensorMap& tm_qkv64, const CUtensorMap& tm_do, const CUtensorMap& tm_do64,
                const void* out, const void* d_out, const TcParams& p, int dgrid, cudaStream_t stream) {
  BB_ONCE_PER_DEVICE({ if (int rc = set_smem(attn_tc_bwd2_kernel<D>, bwd2_smem<D>())) return rc; });
  bb_launch(attn_tc_delta_kernel<D>, dgrid, 256, 0, stream, (const __nv_bfloat16*)out, (const __nv_bfloat16*)d_out, p);
  const int grid = 2 * ((p.S + TQ - 1) / TQ) * p.H * p.B;
  bb_launch(attn_tc_bwd2_kernel<D>, grid, NT2, bwd2_smem<D>(), stream, tm_qkv, tm_qkv64, tm_do, tm_do64, p);
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}
}  // namespace

// delta and the two-role kernel, or delta, the fused kernel and the conversion of dQ
int bb_attention_tc_bwd_launches(int D) { return D == 128 || split_backward() ? 2 : 3; }

int bb_attention_tc_bwd(const void* qkv_q, const void* out, const void* d_out, const float* lse, void* dq, void* dk, void* dv,
                        float* delta, float* dq_acc, int B, int H, int S, int D, long long stride_qkv, long long stride_o,
                        long long stride_dqkv, int causal, float scale, cudaStream_t stream) {
  if (D != 64 && D != 128) return BB_ERR_UNSUPPORTED;
  if (int rc = bbhost::bind_context()) return rc;
  // boxes of 64 columns: [128 rows] for the CTA's own tiles, [64 rows] for the streamed sub-tiles; they end with their
  // sequence, as in the forward pass
  CUtensorMap tm_qkv, tm_do, tm_qkv64, tm_do64;
  const long long T = (long long)B * S;
  if (int rc = bbhost::encode_seqs(&tm_qkv, qkv_q, B, S, 3LL * H * D, stride_qkv, 64, TQ)) return rc;
  if (int rc = bbhost::encode_seqs(&tm_do, d_out, B, S, (long long)H * D, stride_o, 64, TQ)) return rc;
  if (int rc = bbhost::encode_seqs(&tm_qkv64, qkv_q, B, S, 3LL * H * D, stride_qkv, 64, SUB)) return rc;
  if (int rc = bbhost::encode_seqs(&tm_do64, d_out, B, S, (long long)H * D, stride_o, 64, SUB)) return rc;
  TcParams p = {};
  p.dq = (__nv_bfloat16*)dq; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  p.lse = const_cast<float*>(lse); p.delta = delta; p.stride_o = stride_o; p.stride_dqkv = stride_dqkv;
  p.B = B; p.H = H; p.S = S; p.hidden = H * D; p.causal = causal; p.scale = scale; p.status = bb_device_status_word();
  const long long chunks = T * H * (D / 8);
  long long dgrid = (chunks + 511) / 512, cap = (long long)bb_num_sms() * 8;
  if (dgrid > cap) dgrid = cap;
  // Head dimension 128: the two-role kernel.  The fused kernel's tensor-memory map (scores, dP, dV, dK and two dQ
  // tiles) would need 768 columns there.
  if (D == 128) return launch_bwd2<128>(tm_qkv, tm_qkv64, tm_do, tm_do64, out, d_out, p, (int)dgrid, stream);
  if (split_backward()) return launch_bwd2<64>(tm_qkv, tm_qkv64, tm_do, tm_do64, out, d_out, p, (int)dgrid, stream);
  p.dq_acc = dq_acc;
  BB_ONCE_PER_DEVICE({ if (int rc = set_smem(attn_tc_bwd3_kernel, BWD3_SMEM)) return rc; });
  bb_launch(attn_tc_delta_kernel<64>, (int)dgrid, 256, 0, stream, (const __nv_bfloat16*)out, (const __nv_bfloat16*)d_out, p);
  const int grid = (S + TQ - 1) / TQ * H * B;
  // the accumulator as [B * H * S rows, 64] fp32; a reduction moves [32 rows x 16 columns]
  CUtensorMap tm_acc;
  if (int rc = bbhost::encode_2d(&tm_acc, dq_acc, (long long)B * H * S, HD, HD, 16, 32, 1, CU_TENSOR_MAP_SWIZZLE_64B)) return rc;
  bb_launch(attn_tc_bwd3_kernel, grid, NT3, BWD3_SMEM, stream, tm_qkv, tm_qkv64, tm_do64, tm_acc, p);
  long long cgrid = (chunks + 255) / 256;
  bb_launch(attn_tc_dq_convert_kernel, (int)(cgrid < cap ? cgrid : cap), 256, 0, stream, p);
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}
