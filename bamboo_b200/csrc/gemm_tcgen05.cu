// bf16 GEMM on the 5th-generation tensor cores: D[M,N] = op(A)[M,K] * op(B)[N,K]^T with a
// fused epilogue.  One persistent CTA per SM; warps 0 and 2 feed shared memory with TMA
// (128-byte swizzle, no cluster multicast), warp 1 issues tcgen05.mma into two TMEM
// accumulators, warps 3-10 drain TMEM (tcgen05.ld) and run the epilogue (coalesced global
// stores from warp-private staging slabs) while the next tile's main loop is already running.
//
// Work units are handed out dynamically: the first unit of a CTA is its own index, every further
// one comes from a per-launch ticket counter in global memory (one atomicAdd per unit, issued a
// whole unit ahead of its use), and the first producer passes it to the other warps
// (and to the second CTA of a pair) through a four-entry ring in shared memory.  A CTA that
// starts late - because a kernel of another stream still held its SM - therefore takes fewer
// units instead of stretching the launch by its fixed share.
//
// Large problems run as CTA pairs (cta_group::2, clusters of two): a pair owns a 256 x 256
// tile, each CTA loads its own 128 rows of A and only HALF of the B tile, rank 0 issues one
// 256-row MMA for both and each CTA drains its own 128 accumulator rows.  Per CTA that is a
// third less operand traffic from L2 and a third less shared memory per k-block than the
// single-CTA 128 x 256 tile, so six stages fit instead of four - the single-CTA kernel is
// bound by operand bytes in flight, not by the tensor pipe.
//
// Operand storage (all row-major, bf16):
//   a_mn = 0 : A is [M, K] (K contiguous)     a_mn = 1 : A is stored [K, M] (M contiguous)
//   b_mn = 0 : B is [N, K] (K contiguous)     b_mn = 1 : B is stored [K, N] (N contiguous)
// which covers a linear layer's forward (0,0), input gradient (0,1) and weight gradient
// (1,1) without a transpose pass.  A convolution's patch matrix as A or B is gathered by the producer
// (template parameter CONV, bb_conv_gemm).
#include "common.cuh"
#include "bamboo_b200.h"
#include "tma_host.cuh"
#include <atomic>
#include <mutex>
#include <stdlib.h>

namespace {

constexpr int BM = 128;
constexpr int BK = 64;        // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
// threads: two TMA warps, the MMA warp and EW epilogue warps per TMEM lane quarter (EW = 2: 352, EW = 4: 608).
// Two TMA warps take the stages in turn: one iteration of a producer (wait for the stage, announce the bytes, two copies) is
// a chain of about 430 cycles, the MMAs of a k-block of a 128 x 128 tile take 256.
constexpr int TMA_WARP_0 = 0, MMA_WARP = 1, TMA_WARP_1 = 2, EPI_WARP = 3;
constexpr int num_threads(int ew) { return 32 * EPI_WARP + 128 * ew; }
constexpr int A_STAGE_BYTES = BM * BK * 2;  // 16 KiB
// Epilogue staging: one 4 KiB slab (32 rows x 128 bytes = 64 bf16 or 32 fp32 columns) per
// epilogue warp; shared memory is better spent on main-loop stages.
constexpr int SLAB_BYTES = 32 * 128;
constexpr int NUM_SLABS = 8;
constexpr int SCHED_RING = 4;  // work units announced ahead of their consumption (power of two)

template <int BN, bool PAIR> struct Cfg {
  static constexpr int B_ROWS = PAIR ? BN / 2 : BN;      // B rows (output columns) this CTA loads
  static constexpr int B_STAGE_BYTES = B_ROWS * BK * 2;
  static constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
  static constexpr int STAGES = (B_ROWS == 256) ? 4 : 6;
  static constexpr int TILE_M = PAIR ? 2 * BM : BM;      // rows of a work unit (both CTAs of a pair)
  static constexpr int TMEM_COLS = 2 * BN;  // two accumulators
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + NUM_SLABS * SLAB_BYTES + 1024 /*align slack*/ + 256 /*barriers*/;
};

struct GemmParams {
  int M, N, K;
  int a_mn, b_mn;
  int epi;
  int ksplit, kb_per_split;   // parts of a tile's reduction: work units (fp32 add-reductions), or CTAs of a cluster (bf16 outputs)
  int n_fast;                 // tile order: consecutive work units walk along N (else along M)
  int dynamic;                // 1: work units after a CTA's first come from the ticket counter
  unsigned int* ticket;       // this launch's ticket counter (global memory)
  unsigned int ticket_base;   // its value before this launch's first ticket
  unsigned tiles_in, tiles_mn;                     // output tiles along the fast dimension, and in all
  unsigned long long magic_in, magic_mn;           // ... as divisors
  void* D; void* D2; const void* bias; const void* aux;
  long long ldd, ld_aux;
  int* status;
};

// Geometry of a convolution product (template parameter CONV): which operand the im2col loads gather.
struct ConvParams {
  int mode;                   // BB_CONV_FWD / BB_CONV_WGRAD / BB_CONV_DGRAD
  int k, stride, pad;
  int cblocks;                // 64-channel blocks per tap of the patch source
  int wcols;                  // columns of one tap in the weight matrix (Cin)
  unsigned Wo, Ho;            // windows per image row / rows of windows per image
  unsigned long long magic_w, magic_h;
};
struct NoConv {};
template <bool CONV> struct ConvArg { typedef NoConv type; };
template <> struct ConvArg<true> { typedef ConvParams type; };

__device__ __forceinline__ void unpack8(const uint4& q, float* f) {
  f[0] = bb::bf16_lo(q.x); f[1] = bb::bf16_hi(q.x); f[2] = bb::bf16_lo(q.y); f[3] = bb::bf16_hi(q.y);
  f[4] = bb::bf16_lo(q.z); f[5] = bb::bf16_hi(q.z); f[6] = bb::bf16_lo(q.w); f[7] = bb::bf16_hi(q.w);
}

// One output row's slice of a panel (128 bytes = 8 chunks of 16 bytes) into swizzled shared memory.
__device__ __forceinline__ void panel_store_row_bf16(uint8_t* panel, int row, const float* v /*64*/) {
  uint8_t* base = panel + row * 128;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    uint4 q;
    q.x = bb::pack_bf16x2(v[8 * c + 0], v[8 * c + 1]); q.y = bb::pack_bf16x2(v[8 * c + 2], v[8 * c + 3]);
    q.z = bb::pack_bf16x2(v[8 * c + 4], v[8 * c + 5]); q.w = bb::pack_bf16x2(v[8 * c + 6], v[8 * c + 7]);
    *reinterpret_cast<uint4*>(base + ((c ^ (row & 7)) << 4)) = q;
  }
}
__device__ __forceinline__ void panel_store_row_f32(uint8_t* panel, int row, const float* v /*32*/) {
  uint8_t* base = panel + row * 128;
#pragma unroll
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<float4*>(base + ((c ^ (row & 7)) << 4)) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
}

// ---- warp-private staging slab: 32 rows x 128 bytes, 16-byte chunks XOR-swizzled by the row.
// Row side: lane == row (panel_store_row_* / panel_load_row_bf16 with row = lane).
// Coalesced side: lane -> (row 4*i + lane/8, chunk lane%8), i = 0..7: one instruction moves four
// complete 128-byte row segments.
__device__ __forceinline__ uint32_t slab_off(int row, int chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }

// Whether the 32 rows from r0 and `width` columns from nb all lie inside the matrix (the same for a whole warp): then the
// addresses are one base and a constant step and the accesses go out back to back.  With a test per row and chunk the
// eight stores of a panel took 950 cycles, the longest part of its epilogue.
__device__ __forceinline__ bool inside(int r0, int nb, int width, int M, int N) { return r0 + 32 <= M && nb + width <= N; }

__device__ __forceinline__ void slab_put(uint8_t* slab, int lane, const uint4* ax) {
#pragma unroll
  for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(slab + slab_off(4 * i + (lane >> 3), lane & 7)) = ax[i];
}
// rows r0.., columns nb.. of a bf16 matrix -> ax (zero outside the matrix)
__device__ __forceinline__ void slab_fetch_bf16(const __nv_bfloat16* src, long long ld, int r0, int nb, int M, int N, int lane, uint4* ax) {
  const int c = nb + (lane & 7) * 8;
  if (inside(r0, nb, 64, M, N)) {
    const __nv_bfloat16* g = src + (long long)(r0 + (lane >> 3)) * ld + c;
#pragma unroll
    for (int i = 0; i < 8; ++i, g += 4 * ld) ax[i] = __ldca(reinterpret_cast<const uint4*>(g));
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + 4 * i + (lane >> 3);
    uint4 q = make_uint4(0, 0, 0, 0);
    if (r < M) {
      const __nv_bfloat16* g = src + (long long)r * ld + c;
      if (c + 8 <= N) {
        q = __ldca(reinterpret_cast<const uint4*>(g));
      } else {
        unsigned short e[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) e[k] = (c + k < N) ? __bfloat16_as_ushort(g[k]) : (unsigned short)0;
        q.x = e[0] | ((uint32_t)e[1] << 16); q.y = e[2] | ((uint32_t)e[3] << 16);
        q.z = e[4] | ((uint32_t)e[5] << 16); q.w = e[6] | ((uint32_t)e[7] << 16);
      }
    }
    ax[i] = q;
  }
}
__device__ __forceinline__ void slab_flush_bf16(const uint8_t* slab, __nv_bfloat16* dst, long long ld, int r0, int nb, int M, int N, int lane) {
  const int c = nb + (lane & 7) * 8;
  if (inside(r0, nb, 64, M, N)) {
    __nv_bfloat16* g = dst + (long long)(r0 + (lane >> 3)) * ld + c;
    uint4 q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = *reinterpret_cast<const uint4*>(slab + slab_off(4 * i + (lane >> 3), lane & 7));
#pragma unroll
    for (int i = 0; i < 8; ++i, g += 4 * ld) *reinterpret_cast<uint4*>(g) = q[i];
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int rl = 4 * i + (lane >> 3);
    const int r = r0 + rl;
    const uint4 q = *reinterpret_cast<const uint4*>(slab + slab_off(rl, lane & 7));
    if (r < M) {
      __nv_bfloat16* g = dst + (long long)r * ld + c;
      if (c + 8 <= N) {
        *reinterpret_cast<uint4*>(g) = q;
      } else {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) if (c + k < N) g[k] = __ushort_as_bfloat16((unsigned short)(w[k >> 1] >> (16 * (k & 1))));
      }
    }
  }
}
// Add-reductions go out back to back only into outputs of less than 16 MiB.  A large output is read and written in memory, and bursts
// of reductions slow that down: 4096 x 16384 x 333 141 us in bursts and 135 row by row, 8192 x 2048 x 333 35.3 and 33.5, 2048 x 2048 x 513
// 13.2 and 12.5 (outputs not in L2; from 2000 k on no difference); a small one of many splits stays in L2: 64 x 576 x 100352
// 25.7 and 26.9.
__device__ __forceinline__ bool small_output(int M, int N) { return (long long)M * N < (1LL << 22); }
template <bool ACCUM>
__device__ __forceinline__ void slab_flush_f32(const uint8_t* slab, float* dst, long long ld, int r0, int nb, int M, int N, int lane) {
  const int c = nb + (lane & 7) * 4;
  if ((!ACCUM || small_output(M, N)) && inside(r0, nb, 32, M, N)) {
    float* g = dst + (long long)(r0 + (lane >> 3)) * ld + c;
    float4 q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = *reinterpret_cast<const float4*>(slab + slab_off(4 * i + (lane >> 3), lane & 7));
#pragma unroll
    for (int i = 0; i < 8; ++i, g += 4 * ld) {
      if (ACCUM) asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g), "f"(q[i].x), "f"(q[i].y), "f"(q[i].z), "f"(q[i].w) : "memory");
      else *reinterpret_cast<float4*>(g) = q[i];
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int rl = 4 * i + (lane >> 3);
    const int r = r0 + rl;
    const float4 q = *reinterpret_cast<const float4*>(slab + slab_off(rl, lane & 7));
    if (r < M) {
      float* g = dst + (long long)r * ld + c;
      if (c + 4 <= N) {
        if (ACCUM) asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g), "f"(q.x), "f"(q.y), "f"(q.z), "f"(q.w) : "memory");
        else *reinterpret_cast<float4*>(g) = q;
      } else {
        const float w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (c + k < N) { if (ACCUM) atomicAdd(g + k, w[k]); else g[k] = w[k]; }
        }
      }
    }
  }
}

// ---- narrow variant (four epilogue warps per lane quarter): 32 rows x 64 bytes = 32 bf16
// columns per pass, 2 KiB per warp.  Chunk c of row r sits at c ^ ((r >> 1) & 3): eight
// consecutive rows cover all 32 banks once, on the row side (lane == row) and on the coalesced
// side (lane -> row 8*i + lane/4, chunk lane%4, i = 0..3).
__device__ __forceinline__ uint32_t slab64_off(int row, int chunk) { return row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4); }

__device__ __forceinline__ void slab64_store_row(uint8_t* slab, int row, const float* v /*32*/) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint4 q;
    q.x = bb::pack_bf16x2(v[8 * c + 0], v[8 * c + 1]); q.y = bb::pack_bf16x2(v[8 * c + 2], v[8 * c + 3]);
    q.z = bb::pack_bf16x2(v[8 * c + 4], v[8 * c + 5]); q.w = bb::pack_bf16x2(v[8 * c + 6], v[8 * c + 7]);
    *reinterpret_cast<uint4*>(slab + slab64_off(row, c)) = q;
  }
}
// rows r0.., columns nb..nb+31 of a bf16 matrix -> slab (zero outside the matrix), coalesced
__device__ __forceinline__ void slab64_fetch(uint8_t* slab, const __nv_bfloat16* src, long long ld, int r0, int nb, int M, int N, int lane) {
  const int c = nb + (lane & 3) * 8;
  uint4 q[4];
  if (inside(r0, nb, 32, M, N)) {
    const __nv_bfloat16* g = src + (long long)(r0 + (lane >> 2)) * ld + c;
#pragma unroll
    for (int i = 0; i < 4; ++i, g += 8 * ld) q[i] = __ldca(reinterpret_cast<const uint4*>(g));
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(slab + slab64_off(8 * i + (lane >> 2), lane & 3)) = q[i];
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + 8 * i + (lane >> 2);
    q[i] = make_uint4(0, 0, 0, 0);
    if (r < M) {
      const __nv_bfloat16* g = src + (long long)r * ld + c;
      if (c + 8 <= N) {
        q[i] = __ldca(reinterpret_cast<const uint4*>(g));
      } else {
        unsigned short e[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) e[k] = (c + k < N) ? __bfloat16_as_ushort(g[k]) : (unsigned short)0;
        q[i].x = e[0] | ((uint32_t)e[1] << 16); q[i].y = e[2] | ((uint32_t)e[3] << 16);
        q[i].z = e[4] | ((uint32_t)e[5] << 16); q[i].w = e[6] | ((uint32_t)e[7] << 16);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(slab + slab64_off(8 * i + (lane >> 2), lane & 3)) = q[i];
}
__device__ __forceinline__ void slab64_flush(const uint8_t* slab, __nv_bfloat16* dst, long long ld, int r0, int nb, int M, int N, int lane) {
  const int c = nb + (lane & 3) * 8;
  if (inside(r0, nb, 32, M, N)) {
    __nv_bfloat16* g = dst + (long long)(r0 + (lane >> 2)) * ld + c;
    uint4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const uint4*>(slab + slab64_off(8 * i + (lane >> 2), lane & 3));
#pragma unroll
    for (int i = 0; i < 4; ++i, g += 8 * ld) *reinterpret_cast<uint4*>(g) = q[i];
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rl = 8 * i + (lane >> 2);
    const int r = r0 + rl;
    const uint4 q = *reinterpret_cast<const uint4*>(slab + slab64_off(rl, lane & 3));
    if (r < M) {
      __nv_bfloat16* g = dst + (long long)r * ld + c;
      if (c + 8 <= N) {
        *reinterpret_cast<uint4*>(g) = q;
      } else {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) if (c + k < N) g[k] = __ushort_as_bfloat16((unsigned short)(w[k >> 1] >> (16 * (k & 1))));
      }
    }
  }
}

__device__ __forceinline__ float2 get2(const float* v) { return make_float2(v[0], v[1]); }
__device__ __forceinline__ void set2(float* v, float2 a) { v[0] = a.x; v[1] = a.y; }
// GeLU of the bf16-rounded pre-activation: forward and backward (which re-reads the stored pre-activation) see the same argument
template <int W> __device__ __forceinline__ void gelu_rounded(float* v) {
#pragma unroll
  for (int i = 0; i < W; i += 2) {
    const uint32_t q = bb::pack_bf16x2(v[i], v[i + 1]);
    set2(v + i, bb::gelu_tanh2(make_float2(bb::bf16_lo(q), bb::bf16_hi(q))));
  }
}
// v *= gelu'(x) or v += x
template <int W> __device__ __forceinline__ void apply_aux(int epi, float* v, const float* x) {
  if (epi == BB_EPI_MUL_DGELU) {
#pragma unroll
    for (int i = 0; i < W; i += 2) set2(v + i, bb::mul2(get2(v + i), bb::gelu_tanh_grad2(get2(x + i))));
  } else {
#pragma unroll
    for (int i = 0; i < W; i += 2) set2(v + i, bb::add2(get2(v + i), get2(x + i)));
  }
}

// bias[n0 .. n0+W) added to v; columns past N read as zero
template <int W>
__device__ __forceinline__ void add_bias(const GemmParams& p, int n0, float* v) {
  const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(p.bias) + n0;
  if (n0 + W <= p.N) {
#pragma unroll
    for (int i = 0; i < W; i += 8) {
      float f[8]; unpack8(__ldg(reinterpret_cast<const uint4*>(b + i)), f);
#pragma unroll
      for (int k = 0; k < 8; k += 2) set2(v + i + k, bb::add2(get2(v + i + k), make_float2(f[k], f[k + 1])));
    }
  } else {
    // fully unrolled with predicates: a dynamically indexed v[] would live in local memory
#pragma unroll
    for (int i = 0; i < W; ++i) if (n0 + i < p.N) v[i] += __bfloat162float(b[i]);
  }
}

// (m tile, n tile, split) of a work unit
__device__ __forceinline__ void unit_coords(const GemmParams& p, int unit, int& mi, int& ni, int& ks) {
  const unsigned split = bb::fast_div((unsigned)unit, p.magic_mn), mn = (unsigned)unit - split * p.tiles_mn;
  const unsigned slow = bb::fast_div(mn, p.magic_in), fast = mn - slow * p.tiles_in;
  mi = (int)(p.n_fast ? slow : fast); ni = (int)(p.n_fast ? fast : slow); ks = (int)split;
}

// Operand loads of one work unit: k-blocks [kb0, kb1) of the A rows from m0 and the B rows (output columns) from n0 into the
// stage ring (s, phase), by a whole warp: the waits are warp-wide, one elected lane issues.  `turn`: which of the two producer
// warps this is; it serves the stages of its parity.  `rank`: which CTA of its pair
// this is; `lead`: cluster rank of the pair's first CTA, on whose barriers both CTAs' copies complete and where the MMA
// issuer waits.  False when a wait ran out.
template <int BN, bool PAIR, bool CONV>
__device__ __forceinline__ bool load_operands(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p,
                                              const typename ConvArg<CONV>::type& cv, uint8_t* sA, uint8_t* sB, uint64_t* full_bar,
                                              uint64_t* empty_bar, volatile int* abort_flag, uint32_t rank, uint32_t lead, int m0, int n0,
                                              int kb0, int kb1, int turn, int& s, uint32_t& phase) {
  using C = Cfg<BN, PAIR>;
  static_assert(C::STAGES % 2 == 0, "the producers take the stages in turn");
  if constexpr (CONV) {
    // Patches of a convolution: a stage's patch tile is 64 channels of one tap for a run of windows, one
    // im2col load (the hardware walks the windows, applies the stride and fills with zeros outside the
    // image).  FWD / DGRAD gather A (windows = output rows, k-blocks run over taps x channel blocks),
    // WGRAD gathers B (windows = the reduction, columns = taps x channels).
    auto window = [&](unsigned px, int& w, int& h, int& n) {
      const unsigned row = bb::fast_div(px, cv.magic_w), img = bb::fast_div(row, cv.magic_h);
      w = (int)(px - row * cv.Wo) * cv.stride - cv.pad;
      h = (int)(row - img * cv.Ho) * cv.stride - cv.pad;
      n = (int)img;
    };
    auto patches = [&](uint8_t* dst, const CUtensorMap* tm, uint32_t fb, int c, int w, int h, int n, int ow, int oh) {
      if constexpr (PAIR) bb::tma_load_im2col_pair(dst, tm, fb, c, w, h, n, (uint16_t)ow, (uint16_t)oh);
      else bb::tma_load_im2col(dst, tm, &full_bar[s], c, w, h, n, (uint16_t)ow, (uint16_t)oh);
    };
    auto plain = [&](uint8_t* dst, const CUtensorMap* tm, uint32_t fb, int x, int y) {
      if constexpr (PAIR) bb::tma_load_2d_pair(dst, tm, fb, x, y);
      else bb::tma_load_2d(dst, tm, &full_bar[s], x, y);
    };
    constexpr int BJ = C::B_ROWS / 64;
    int w, h, n;
    int cj[BJ], rj[BJ], sj[BJ];          // WGRAD: channel and tap of each 64-column block of B
    if (cv.mode == BB_CONV_WGRAD) {
#pragma unroll
      for (int j = 0; j < BJ; ++j) {
        const int cb = min((n0 >> 6) + j, cv.k * cv.k * cv.cblocks - 1);     // past the last tap: never stored
        const int tap = cb / cv.cblocks;
        cj[j] = (cb - tap * cv.cblocks) * 64; rj[j] = tap / cv.k; sj[j] = tap - rj[j] * cv.k;
      }
    } else {
      window((unsigned)m0, w, h, n);
    }
    int tap = kb0 / cv.cblocks, cb = kb0 - tap * cv.cblocks;
    int tr = tap / cv.k, ts = tap - tr * cv.k;
    for (int kb = kb0; kb < kb1; ++kb) {
      if ((s & 1) == turn) {
        if (!bb::mbar_wait_warp(&empty_bar[s], phase ^ 1, abort_flag, p.status)) return false;
        uint8_t* a = sA + s * A_STAGE_BYTES;
        uint8_t* b = sB + s * C::B_STAGE_BYTES;
        uint32_t fb = 0;
        if constexpr (PAIR) fb = bb::mapa_shared(bb::smem_u32(&full_bar[s]), lead);
        if (cv.mode == BB_CONV_WGRAD) window((unsigned)kb * BK, w, h, n);
        const int col = ((cv.k - 1 - tr) * cv.k + (cv.k - 1 - ts)) * cv.wcols + n0;       // the tap turned by 180 degrees
        if (bb::elect_one()) {
          if constexpr (PAIR) {
            if (rank == 0) bb::mbar_arrive_expect_tx(&full_bar[s], 2 * C::STAGE_BYTES);
          } else {
            bb::mbar_arrive_expect_tx(&full_bar[s], C::STAGE_BYTES);
          }
          if (cv.mode == BB_CONV_WGRAD) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) plain(a + j * 8192, &tmA, fb, m0 + 64 * j, kb * BK);
#pragma unroll
            for (int j = 0; j < BJ; ++j) patches(b + j * 8192, &tmB, fb, cj[j], w, h, n, sj[j], rj[j]);
          } else {
            patches(a, &tmA, fb, cb * 64, w, h, n, ts, tr);
            if (cv.mode == BB_CONV_FWD) {
              plain(b, &tmB, fb, kb * BK, n0);
            } else {
#pragma unroll
              for (int j = 0; j < BJ; ++j) plain(b + j * 8192, &tmB, fb, col + 64 * j, cb * 64);
            }
          }
        }
        __syncwarp();
      }
      if (cv.mode != BB_CONV_WGRAD && ++cb == cv.cblocks) { cb = 0; if (++ts == cv.k) { ts = 0; ++tr; } }
      if (++s == C::STAGES) { s = 0; phase ^= 1; }
    }
  } else {
    for (int kb = kb0; kb < kb1; ++kb) {
      if ((s & 1) == turn) {
        if (!bb::mbar_wait_warp(&empty_bar[s], phase ^ 1, abort_flag, p.status)) return false;
        uint8_t* a = sA + s * A_STAGE_BYTES;
        uint8_t* b = sB + s * C::B_STAGE_BYTES;
        const int k0 = kb * BK;
        if (bb::elect_one()) {
          if constexpr (PAIR) {
            // both CTAs' copies complete on rank 0's barrier, where the MMA issuer waits
            if (rank == 0) bb::mbar_arrive_expect_tx(&full_bar[s], 2 * C::STAGE_BYTES);
            const uint32_t fb = bb::mapa_shared(bb::smem_u32(&full_bar[s]), lead);
            if (!p.a_mn) {
              bb::tma_load_2d_pair(a, &tmA, fb, k0, m0);
            } else {
#pragma unroll
              for (int j = 0; j < BM / 64; ++j) bb::tma_load_2d_pair(a + j * 8192, &tmA, fb, m0 + 64 * j, k0);
            }
            if (!p.b_mn) {
              bb::tma_load_2d_pair(b, &tmB, fb, k0, n0);
            } else {
#pragma unroll
              for (int j = 0; j < C::B_ROWS / 64; ++j) bb::tma_load_2d_pair(b + j * 8192, &tmB, fb, n0 + 64 * j, k0);
            }
          } else {
            bb::mbar_arrive_expect_tx(&full_bar[s], C::STAGE_BYTES);
            if (!p.a_mn) {
              bb::tma_load_2d(a, &tmA, &full_bar[s], k0, m0);
            } else {
#pragma unroll
              for (int j = 0; j < BM / 64; ++j) bb::tma_load_2d(a + j * 8192, &tmA, &full_bar[s], m0 + 64 * j, k0);
            }
            if (!p.b_mn) {
              bb::tma_load_2d(b, &tmB, &full_bar[s], k0, n0);
            } else {
#pragma unroll
              for (int j = 0; j < BN / 64; ++j) bb::tma_load_2d(b + j * 8192, &tmB, &full_bar[s], n0 + 64 * j, k0);
            }
          }
        }
        __syncwarp();
      }
      if (++s == C::STAGES) { s = 0; phase ^= 1; }
    }
  }
  return true;
}

// The MMAs of one work unit's k-blocks into the accumulator at d_tmem, issued by one warp; the last commit signals acc_full.
// `ctas`: cluster ranks of the pair as a mask.  False when a wait ran out.
template <int BN, bool PAIR>
__device__ __forceinline__ bool issue_mmas(const GemmParams& p, uint8_t* sA, uint8_t* sB, uint64_t* full_bar, uint64_t* empty_bar,
                                           uint64_t* acc_full, volatile int* abort_flag, uint16_t ctas, uint32_t d_tmem, int num_kb, int& s,
                                           uint32_t& phase) {
  using C = Cfg<BN, PAIR>;
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.a_mn ? 1 : 0) << 15) |
                         ((uint32_t)(p.b_mn ? 1 : 0) << 16) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(C::TILE_M >> 4) << 24);
  // K-major: 8-row groups 1024 B apart (LBO unused); MN-major: 64-wide column groups are
  // separate 8 KiB TMA boxes (LBO), 8 k-rows are 1024 B (SBO).
  const uint32_t a_lbo = p.a_mn ? 8192u : 16u, b_lbo = p.b_mn ? 8192u : 16u;
  const uint32_t a_kstep = p.a_mn ? 2048u : 32u, b_kstep = p.b_mn ? 2048u : 32u;
  for (int kb = 0; kb < num_kb; ++kb) {
    if (!bb::mbar_wait_warp(&full_bar[s], phase, abort_flag, p.status)) return false;
    bb::tc_fence_after_sync();
    if (bb::elect_one()) {
      // one descriptor per stage; a k-step only adds to its address field (16-byte units)
      const uint64_t ad0 = bb::make_smem_desc_sw128(bb::smem_u32(sA + s * A_STAGE_BYTES), a_lbo, 1024u);
      const uint64_t bd0 = bb::make_smem_desc_sw128(bb::smem_u32(sB + s * C::B_STAGE_BYTES), b_lbo, 1024u);
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k) {
        const uint64_t ad = ad0 + (uint64_t)(k * (a_kstep >> 4));
        const uint64_t bd = bd0 + (uint64_t)(k * (b_kstep >> 4));
        if (PAIR) bb::umma_f16_pair(d_tmem, ad, bd, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        else bb::umma_f16(d_tmem, ad, bd, idesc, (kb > 0 || k > 0) ? 1u : 0u);
      }
      if (PAIR) {
        bb::umma_commit_pair(&empty_bar[s], ctas);           // frees the stage in both CTAs
        if (kb == num_kb - 1) bb::umma_commit_pair(acc_full, ctas);
      } else {
        bb::umma_commit(&empty_bar[s]);
        if (kb == num_kb - 1) bb::umma_commit(acc_full);
      }
    }
    __syncwarp();
    if (++s == C::STAGES) { s = 0; phase ^= 1; }
  }
  return true;
}

// Fused math and stores of 32 rows x 32 columns of a bf16 output, one accumulator row per lane; the aux operand, where the
// epilogue has one, is in the slab already.
__device__ __forceinline__ void narrow_panel(const GemmParams& p, uint8_t* slab, int r0, int nb, int lane, float* v) {
  const int epi = p.epi;
  const bool dual = (epi == BB_EPI_BIAS_GELU), has_aux = (epi == BB_EPI_MUL_DGELU || epi == BB_EPI_BIAS_RESIDUAL);
  if (epi == BB_EPI_BIAS || dual || epi == BB_EPI_BIAS_RESIDUAL) add_bias<32>(p, nb, v);
  if (dual) {
    slab64_store_row(slab, lane, v);           // pre-activation first
    __syncwarp();
    slab64_flush(slab, reinterpret_cast<__nv_bfloat16*>(p.D2), p.ldd, r0, nb, p.M, p.N, lane);
    gelu_rounded<32>(v);
    __syncwarp();
  } else if (has_aux) {
    __syncwarp();
    float x[32];
#pragma unroll
    for (int c = 0; c < 4; ++c) unpack8(*reinterpret_cast<const uint4*>(slab + slab64_off(lane, c)), x + 8 * c);
    apply_aux<32>(epi, v, x);
    __syncwarp();
  }
  slab64_store_row(slab, lane, v);
  __syncwarp();
  slab64_flush(slab, reinterpret_cast<__nv_bfloat16*>(p.D), p.ldd, r0, nb, p.M, p.N, lane);
  __syncwarp();
}

template <int BN, bool PAIR, int EW, bool CONV>
__global__ void __launch_bounds__(num_threads(EW), 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                         const GemmParams p, const typename ConvArg<CONV>::type cv) {
  using C = Cfg<BN, PAIR>;
  extern __shared__ uint8_t smem_raw[];
  // 128-byte swizzle atoms need 1024-byte aligned stage buffers
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + C::STAGES * A_STAGE_BYTES;
  uint8_t* panels = smem + C::STAGES * C::STAGE_BYTES;   // NUM_SLABS x 4 KiB epilogue staging
  uint64_t* bars = reinterpret_cast<uint64_t*>(panels + NUM_SLABS * SLAB_BYTES);
  uint64_t* full_bar = bars;                      // [STAGES]
  uint64_t* empty_bar = bars + C::STAGES;         // [STAGES]
  uint64_t* tmem_full = bars + 2 * C::STAGES;     // [2]
  uint64_t* tmem_empty = bars + 2 * C::STAGES + 2;  // [2]
  uint64_t* sched_full = bars + 2 * C::STAGES + 4;  // [SCHED_RING]
  uint64_t* sched_empty = sched_full + SCHED_RING;  // [SCHED_RING] (pairs: rank 0's are used by both CTAs)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sched_empty + SCHED_RING);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* sched_tile = reinterpret_cast<volatile int*>(tmem_slot + 2);   // [SCHED_RING]

  const int warp = bb::warp_index();
  const int lane = threadIdx.x & 31;
  // work units go to CTAs (pairs: to clusters; both CTAs of a pair walk the same units)
  const uint32_t rank = PAIR ? bb::cluster_ctarank() : 0u;
  const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int num_workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int num_tiles = (int)p.tiles_mn * p.ksplit;   // work units: (m, n, k-split)
  const int total_kb = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < C::STAGES; ++s) { bb::mbar_init(&full_bar[s], 1); bb::mbar_init(&empty_bar[s], 1); }
    // accumulator hand-back: one arrival per epilogue warp (of both CTAs for a pair, on rank 0's barrier)
    for (int a = 0; a < 2; ++a) { bb::mbar_init(&tmem_full[a], 1); bb::mbar_init(&tmem_empty[a], (PAIR ? 2 : 1) * 4 * EW); }
    // work-unit ring: one announcement per entry; read by the second producer, the MMA warp and the epilogue warps of
    // this CTA and, for a pair, by both producers and the epilogue warps of the second CTA
    for (int r = 0; r < SCHED_RING; ++r) { bb::mbar_init(&sched_full[r], 1); bb::mbar_init(&sched_empty[r], (PAIR ? 2 : 1) * (2 + 4 * EW)); }
    bb::fence_barrier_init();
    bb::tma_prefetch_desc(&tmA);
    bb::tma_prefetch_desc(&tmB);
  }
  if (warp == MMA_WARP) {
    if (PAIR) { bb::tmem_alloc_pair(tmem_slot, C::TMEM_COLS); bb::tmem_relinquish_pair(); }
    else { bb::tmem_alloc(tmem_slot, C::TMEM_COLS); bb::tmem_relinquish(); }
  }
  bb::tc_fence_before_sync();
  if (PAIR) bb::cluster_sync();     // the peer's barriers are initialised before anything signals them
  else __syncthreads();
  bb::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  bb::pdl_sync();

  // Work unit number `it` of this CTA: the first is its own index, the others as announced by the scheduling warp (-1: no
  // more).  Called by a whole warp; the entry is handed back once it has been read: the hand-back of a pair, which is not a
  // release, branches on the value, so that it cannot be on its way before the value is there.
  auto next_unit = [&](uint32_t it, int& tile) -> bool {
    if (it == 0) { tile = worker; return true; }
    --it;
    const int r = (int)(it & (SCHED_RING - 1));
    const uint32_t ph = (it / SCHED_RING) & 1u;
    const bool got = PAIR ? bb::mbar_wait_cluster(&sched_full[r], ph, abort_flag, p.status)
                          : bb::mbar_wait(&sched_full[r], ph, abort_flag, p.status);
    if (!__all_sync(0xffffffffu, got)) return false;
    tile = __shfl_sync(0xffffffffu, sched_tile[r], 0);
    if (lane == 0) {
      if (!PAIR) bb::mbar_arrive(&sched_empty[r]);
      else if (tile >= -1) bb::mbar_arrive_cluster_relaxed(bb::mapa_shared(bb::smem_u32(&sched_empty[r]), 0));
    }
    return true;
  };

  if (warp == TMA_WARP_0 || warp == TMA_WARP_1) {
    // ------------------------------------------------ TMA producers
    // The whole warp walks the units and waits, one elected lane issues: the compiler then knows that loop counters, barrier
    // addresses and coordinates are the same for the warp, which is what TMA instructions take (see bb::warp_index).
    {
      const int turn = warp == TMA_WARP_1 ? 1 : 0;
      int s = 0; uint32_t phase = 0;
      bool alive = true;
      // operand loads of one work unit
      auto load_unit = [&](int tile) {
        int mi, ni, ks;
        unit_coords(p, tile, mi, ni, ks);
        const int kb0 = ks * p.kb_per_split, kb1 = min(total_kb, kb0 + p.kb_per_split);
        alive = load_operands<BN, PAIR, CONV>(tmA, tmB, p, cv, sA, sB, full_bar, empty_bar, abort_flag, rank, 0u, mi * C::TILE_M + (int)rank * BM,
                                              ni * BN + (int)rank * C::B_ROWS, kb0, kb1, turn, s, phase);
      };
      if (rank == 0 && turn == 0) {
        // ---- scheduling warp: announces every work unit of this CTA (pair) but the first to its consumers
        auto announce = [&](uint32_t it, int tile) -> bool {
          const int r = (int)(it & (SCHED_RING - 1));
          const uint32_t ph = (it / SCHED_RING) & 1u;
          const bool free_ = PAIR ? bb::mbar_wait_cluster(&sched_empty[r], ph ^ 1, abort_flag, p.status)
                                  : bb::mbar_wait(&sched_empty[r], ph ^ 1, abort_flag, p.status);
          if (!__all_sync(0xffffffffu, free_)) return false;
          if (lane == 0) {
            sched_tile[r] = tile;
            if (PAIR) {
              bb::st_shared_cluster_u32(bb::mapa_shared(bb::smem_u32(const_cast<int*>(&sched_tile[r])), 1), (uint32_t)tile);
              bb::mbar_arrive_cluster(bb::mapa_shared(bb::smem_u32(&sched_full[r]), 1));
            }
            bb::mbar_arrive(&sched_full[r]);
          }
          __syncwarp();
          return true;
        };
        // ticket t of this launch stands for work unit num_workers + t (units below num_workers are
        // the CTAs' first ones); every scheduling warp draws until its first ticket past the
        // end, so a launch consumes exactly num_tiles tickets - the host relies on that count
        // (valid in lane 0; broadcast where it is used, so that the atomic is in flight while the unit's loads are issued)
        auto draw = [&]() -> int { return lane == 0 ? num_workers + (int)(atomicAdd(p.ticket, 1u) - p.ticket_base) : 0; };
        uint32_t it = 0;
        int cur = worker, nxt = worker;
        while (cur < num_tiles) {
          // the announcement's release at cluster scope waits for the thread's outstanding global operations: it comes
          // before the draw, whose result has a whole unit's time to arrive
          if (cur != worker && !announce(it++, cur)) { alive = false; break; }
          nxt = p.dynamic ? draw() : cur + num_workers;
          load_unit(cur);
          if (!alive) break;
          cur = __shfl_sync(0xffffffffu, nxt, 0);
        }
        if (alive) { if (!announce(it++, -1)) alive = false; }
        else if (p.dynamic && lane == 0) { while (nxt < num_tiles) nxt = draw(); }
      } else {
        // second producer, second CTA of a pair: follow the announcements
        for (uint32_t it = 0; alive; ++it) {
          int tile;
          if (!next_unit(it, tile)) { alive = false; break; }
          if (tile < 0) break;
          load_unit(tile);
        }
      }
      if constexpr (PAIR) {
        // rank 0's MMA commits arrive on this CTA's barriers too: wait until the last one of every
        // stage has landed, so that none is still on its way when the CTA leaves
        for (int i = 0; i < C::STAGES && alive; ++i) {
          if ((s & 1) == turn && !bb::mbar_wait_warp(&empty_bar[s], phase ^ 1, abort_flag, p.status)) alive = false;
          if (++s == C::STAGES) { s = 0; phase ^= 1; }
        }
      }
      if (!alive) {
        // give copies that are still in flight time to land before the CTA's shared
        // memory is released (bounded)
        uint64_t t0 = bb::globaltimer_ns();
        while (bb::globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------ MMA issuer
    int s = 0; uint32_t phase = 0;
    int acc = 0; uint32_t acc_phase = 0;
    bool alive = true;
    // pairs: rank 0 issues for both CTAs; the other CTA's MMA warp only allocates and frees TMEM
    for (uint32_t it = 0; alive && rank == 0; ++it) {
      int tile;
      if (!next_unit(it, tile)) { alive = false; break; }
      if (tile < 0) break;
      if (!bb::mbar_wait_warp(&tmem_empty[acc], acc_phase ^ 1, abort_flag, p.status)) { alive = false; break; }
      bb::tc_fence_after_sync();
      const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
      int mi, ni, ks;
      unit_coords(p, tile, mi, ni, ks);
      const int num_kb = min(total_kb, (ks + 1) * p.kb_per_split) - ks * p.kb_per_split;
      if (!issue_mmas<BN, PAIR>(p, sA, sB, full_bar, empty_bar, &tmem_full[acc], abort_flag, 3, d_tmem, num_kb, s, phase)) { alive = false; break; }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  } else {
    // ------------------------------------------------ epilogue: 8 independent warps
    // A warp owns one TMEM lane quarter (32 rows of the tile); the two warps of a quarter take
    // alternate 128-byte-wide column panels.  Per panel: TMEM -> registers (one row per lane) ->
    // fused math -> the warp's private 4 KiB staging slab in shared memory -> coalesced 16-byte
    // global stores (fp32 add-reduction: vector red) by the same warp.  Nothing here waits on
    // another warp or on the TMA queue, which the producer keeps full of operand loads.
    const int eg = (warp - EPI_WARP) >> 2;         // which of the quarter's EW warps
    const int quarter = warp & 3;
    const int epi = p.epi;
    const bool f32 = (epi == BB_EPI_ACCUM_F32 || epi == BB_EPI_STORE_F32);
    const bool dual = (epi == BB_EPI_BIAS_GELU);
    const bool has_aux = (epi == BB_EPI_MUL_DGELU || epi == BB_EPI_BIAS_RESIDUAL);
    int acc = 0; uint32_t acc_phase = 0;
    bool alive = true;
    if constexpr (EW == 4) {
      // Narrow variant: sixteen warps, 32 bf16 columns per pass (bf16 outputs only), when the descriptor asks for it.
      uint8_t* slab = panels + (warp - EPI_WARP) * (SLAB_BYTES / 2);
      for (uint32_t it = 0; alive; ++it) {
        int tile;
        if (!next_unit(it, tile)) { alive = false; break; }
        if (tile < 0) break;
        int mi, ni, ks;
        unit_coords(p, tile, mi, ni, ks);
        const int m0 = mi * C::TILE_M + (int)rank * BM, n0 = ni * BN;
        const int r0 = m0 + quarter * 32;
        const bool got = bb::mbar_wait(&tmem_full[acc], acc_phase, abort_flag, p.status);
        if (!__all_sync(0xffffffffu, got)) { alive = false; break; }
        bb::tc_fence_after_sync();
        const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN);
        constexpr int npanels = BN / 32;
#pragma unroll 1
        for (int pn = eg; pn < npanels; pn += 4) {
          const int nb = n0 + pn * 32;
          const bool some = (nb < p.N) && (r0 < p.M);
          if (has_aux && some) slab64_fetch(slab, reinterpret_cast<const __nv_bfloat16*>(p.aux), p.ld_aux, r0, nb, p.M, p.N, lane);
          float v[32];
          {
            uint32_t r[32];
            bb::tmem_ld_32x32b_x32(t_row + pn * 32, r);
            bb::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
          }
          if (pn + 4 >= npanels) {
            bb::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
              if (PAIR) bb::mbar_arrive_cluster_relaxed(bb::mapa_shared(bb::smem_u32(&tmem_empty[acc]), 0));
              else bb::mbar_arrive(&tmem_empty[acc]);
            }
          }
          if (!some) continue;
          narrow_panel(p, slab, r0, nb, lane, v);
        }
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    } else {
    uint8_t* slab = panels + (warp - EPI_WARP) * SLAB_BYTES;
    for (uint32_t it = 0; alive; ++it) {
      int tile;
      if (!next_unit(it, tile)) { alive = false; break; }
      if (tile < 0) break;
      int mi, ni, ks;
      unit_coords(p, tile, mi, ni, ks);
      const int m0 = mi * C::TILE_M + (int)rank * BM, n0 = ni * BN;
      const int r0 = m0 + quarter * 32;            // first output row of this warp
      const bool got = bb::mbar_wait(&tmem_full[acc], acc_phase, abort_flag, p.status);
      if (!__all_sync(0xffffffffu, got)) { alive = false; break; }
      bb::tc_fence_after_sync();
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN);
      const int width = f32 ? 32 : 64;             // columns per panel
      const int npanels = BN / width;
#pragma unroll 1
      for (int pn = eg; pn < npanels; pn += 2) {
        const int nb = n0 + pn * width;
        const bool some = (nb < p.N) && (r0 < p.M);     // warp-uniform
        if (has_aux && some) {
          // the aux tile comes in coalesced (rows spread over lanes) and is turned through the
          // slab, so that every lane can pick up its own row after the accumulator arrived
          uint4 ax[8];
          slab_fetch_bf16(reinterpret_cast<const __nv_bfloat16*>(p.aux), p.ld_aux, r0, nb, p.M, p.N, lane, ax);
          slab_put(slab, lane, ax);
        }
        float v[64];
        {
          uint32_t r[32];
          bb::tmem_ld_32x32b_x32(t_row + pn * width, r);
          bb::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
          if (!f32) {
            bb::tmem_ld_32x32b_x32(t_row + pn * width + 32, r);
            bb::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[32 + i] = __uint_as_float(r[i]);
          }
        }
        if (pn + 2 >= npanels) {
          // this warp has read its share of the accumulator: hand it back before the last stores
          bb::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) {
            if (PAIR) bb::mbar_arrive_cluster_relaxed(bb::mapa_shared(bb::smem_u32(&tmem_empty[acc]), 0));
            else bb::mbar_arrive(&tmem_empty[acc]);
          }
        }
        if (!some) continue;                     // panel entirely outside the matrix
        if (f32) {
          panel_store_row_f32(slab, lane, v);
          __syncwarp();
          if (epi == BB_EPI_ACCUM_F32) slab_flush_f32<true>(slab, reinterpret_cast<float*>(p.D), p.ldd, r0, nb, p.M, p.N, lane);
          else slab_flush_f32<false>(slab, reinterpret_cast<float*>(p.D), p.ldd, r0, nb, p.M, p.N, lane);
          __syncwarp();
          continue;
        }
        if (epi == BB_EPI_BIAS || dual || epi == BB_EPI_BIAS_RESIDUAL) add_bias<64>(p, nb, v);
        if (dual) {
          panel_store_row_bf16(slab, lane, v);     // pre-activation first
          __syncwarp();
          slab_flush_bf16(slab, reinterpret_cast<__nv_bfloat16*>(p.D2), p.ldd, r0, nb, p.M, p.N, lane);
          gelu_rounded<64>(v);
          __syncwarp();
        } else if (has_aux) {
          __syncwarp();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float x[32];
#pragma unroll
            for (int c = 0; c < 4; ++c) unpack8(*reinterpret_cast<const uint4*>(slab + slab_off(lane, 4 * h + c)), x + 8 * c);
            apply_aux<32>(epi, v + 32 * h, x);
          }
          __syncwarp();
        }
        panel_store_row_bf16(slab, lane, v);
        __syncwarp();
        slab_flush_bf16(slab, reinterpret_cast<__nv_bfloat16*>(p.D), p.ldd, r0, nb, p.M, p.N, lane);
        __syncwarp();
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    }   // EW == 2
  }

  bb::tc_fence_before_sync();
  if (PAIR) {
    // neither CTA leaves (or frees TMEM) while the other may still signal its barriers
    bb::cluster_sync();
    if (warp == MMA_WARP) bb::tmem_dealloc_pair(tmem_base, C::TMEM_COLS);
  } else {
    __syncthreads();
    if (warp == MMA_WARP) bb::tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// ---------------------------------------------------------------- reduction split inside a cluster
// Products of few output tiles and a long reduction: S CTAs (or CTA pairs) of one cluster share a tile's reduction, each over its
// own k-blocks.  What bounds such a product is the latency of its operands: six stages in flight give an SM about 80 bytes a
// clock, a k-block of a 128 x 256 tile takes 0.3 us however idle the rest of the GPU is - so the reduction goes to SMs that would
// be idle.  The partial sums meet in fp32 through distributed shared memory: the tile's 32-column panels are dealt out to
// the splits, each split writes its sums of the others' panels into their (by then unused) operand stages and adds what it
// received to its own panels in the order of the splits: a fixed order, no global scratch, no counters.  One tile per cluster.
// Receive buffers: [owned panel][other split] x 16 KiB = [quarter][16-byte chunk of the row][row], so that a warp's store
// is 512 contiguous bytes.
constexpr int SPLIT_EW = 4;                       // epilogue warps per TMEM lane quarter
constexpr int split_limit(bool pair) { return pair ? 4 : 8; }        // a cluster of eight CTAs
// receive buffers of the split that owns most panels
constexpr int split_buffers(int bn, bool pair) {
  int most = 0;
  for (int s = 2; s <= split_limit(pair); ++s) {
    const int n = (bn / 32 + s - 1) / s * (s - 1);
    if (n > most) most = n;
  }
  return most;
}
static_assert(split_buffers(128, false) * (BM * 32 * 4) <= Cfg<128, false>::STAGES * Cfg<128, false>::STAGE_BYTES &&
              split_buffers(256, false) * (BM * 32 * 4) <= Cfg<256, false>::STAGES * Cfg<256, false>::STAGE_BYTES &&
              split_buffers(256, true) * (BM * 32 * 4) <= Cfg<256, true>::STAGES * Cfg<256, true>::STAGE_BYTES,
              "receive buffers fit the operand stages");

template <int BN, bool PAIR, bool CONV>
__global__ void __launch_bounds__(num_threads(SPLIT_EW), 1)
gemm_cluster_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const GemmParams p, const typename ConvArg<CONV>::type cv) {
  using C = Cfg<BN, PAIR>;
  constexpr int PC = PAIR ? 2 : 1;                // CTAs per split
  constexpr int NP = BN / 32;                     // panels of a tile
  constexpr int PANEL_BYTES = BM * 32 * 4;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + C::STAGES * A_STAGE_BYTES;
  uint8_t* panels = smem + C::STAGES * C::STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(panels + NUM_SLABS * SLAB_BYTES);
  uint64_t* full_bar = bars;                      // [STAGES]
  uint64_t* empty_bar = bars + C::STAGES;         // [STAGES]
  uint64_t* tmem_full = bars + 2 * C::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = bb::warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t crank = bb::cluster_ctarank();
  const uint32_t rank = PAIR ? (crank & 1u) : 0u, lead = crank - rank;
  const int S = p.ksplit, ks = (int)crank / PC;
  const int total_kb = (p.K + BK - 1) / BK;
  int mi, ni, unused;
  unit_coords(p, (int)bb::cluster_id(), mi, ni, unused);
  const int m0 = mi * C::TILE_M + (int)rank * BM, n0 = ni * BN;
  const int kb0 = ks * p.kb_per_split, kb1 = min(total_kb, kb0 + p.kb_per_split);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < C::STAGES; ++s) { bb::mbar_init(&full_bar[s], 1); bb::mbar_init(&empty_bar[s], 1); }
    bb::mbar_init(tmem_full, 1);
    bb::fence_barrier_init();
    bb::tma_prefetch_desc(&tmA);
    bb::tma_prefetch_desc(&tmB);
  }
  if (warp == MMA_WARP) {
    if (PAIR) { bb::tmem_alloc_pair(tmem_slot, BN); bb::tmem_relinquish_pair(); }
    else { bb::tmem_alloc(tmem_slot, BN); bb::tmem_relinquish(); }
  }
  bb::tc_fence_before_sync();
  if (PAIR) bb::cluster_sync();     // the peer's barriers are initialised before anything signals them
  else __syncthreads();
  bb::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  bb::pdl_sync();

  const int eg = (warp - EPI_WARP) >> 2, quarter = warp & 3;
  const int r0 = m0 + quarter * 32;
  const bool has_aux = (p.epi == BB_EPI_MUL_DGELU || p.epi == BB_EPI_BIAS_RESIDUAL);
  const int first = ks + eg * S;                            // this warp's first own panel; the next is SPLIT_EW * S further
  uint8_t* slab = panels + (warp - EPI_WARP) * (SLAB_BYTES / 2);
  bool summed = false;
  if (warp == TMA_WARP_0 || warp == TMA_WARP_1) {
    const int turn = warp == TMA_WARP_1 ? 1 : 0;
    int s = 0; uint32_t phase = 0;
    bool alive = load_operands<BN, PAIR, CONV>(tmA, tmB, p, cv, sA, sB, full_bar, empty_bar, abort_flag, rank, lead, m0,
                                               n0 + (int)rank * C::B_ROWS, kb0, kb1, turn, s, phase);
    if constexpr (PAIR) {
      // the commits that free a stage arrive in both CTAs: none may still be on its way when the CTA leaves
      for (int i = 0; i < C::STAGES && alive; ++i) {
        if ((s & 1) == turn && !bb::mbar_wait_warp(&empty_bar[s], phase ^ 1, abort_flag, p.status)) alive = false;
        if (++s == C::STAGES) { s = 0; phase ^= 1; }
      }
    }
    if (!alive) {
      // copies still in flight get time to land (bounded)
      uint64_t t0 = bb::globaltimer_ns();
      while (bb::globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
  } else if (warp == MMA_WARP) {
    if (rank == 0) {
      int s = 0; uint32_t phase = 0;
      issue_mmas<BN, PAIR>(p, sA, sB, full_bar, empty_bar, tmem_full, abort_flag, (uint16_t)(3u << lead), tmem_base, kb1 - kb0, s, phase);
    }
  } else {
    // the aux operand of the first own panel is fetched under the main loop
    if (has_aux && first < NP && n0 + first * 32 < p.N && r0 < p.M)
      slab64_fetch(slab, reinterpret_cast<const __nv_bfloat16*>(p.aux), p.ld_aux, r0, n0 + first * 32, p.M, p.N, lane);
    summed = bb::mbar_wait_warp(tmem_full, 0, abort_flag, p.status);
    bb::tc_fence_after_sync();
  }
  __syncwarp();
  // every CTA's MMAs have retired, so its operand stages can receive (and all of its copies have landed)
  bb::cluster_sync();
  const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
  if (summed && r0 < p.M) {
    int turn = 0;
    for (int i = 1; i < S; ++i) {                           // the splits start with different owners
      const int owner = ks + i < S ? ks + i : ks + i - S;
      int slot = ks < owner ? ks : ks - 1;
      for (int pn = owner; pn < NP; pn += S, slot += S - 1) {
        if ((turn++ & (SPLIT_EW - 1)) != eg || n0 + pn * 32 >= p.N) continue;
        uint32_t r[32];
        bb::tmem_ld_32x32b_x32(t_row + pn * 32, r);
        bb::tmem_ld_wait();
        const uint32_t dst = bb::mapa_shared(bb::smem_u32(smem) + slot * PANEL_BYTES + quarter * 4096 + lane * 16, owner * PC + rank);
#pragma unroll
        for (int j = 0; j < 8; ++j) bb::st_shared_cluster_v4(dst + j * 512, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
    }
  }
  __syncwarp();
  bb::cluster_sync();
  if (summed && r0 < p.M) {
    const uint8_t* part = smem + eg * (S - 1) * PANEL_BYTES + quarter * 4096 + lane * 16;
    for (int pn = first; pn < NP; pn += SPLIT_EW * S, part += SPLIT_EW * (S - 1) * PANEL_BYTES) {
      const int nb = n0 + pn * 32;
      if (nb >= p.N) break;
      if (has_aux && pn != first) slab64_fetch(slab, reinterpret_cast<const __nv_bfloat16*>(p.aux), p.ld_aux, r0, nb, p.M, p.N, lane);
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
      for (int t = 0; t < S; ++t) {
        if (t == ks) {
          uint32_t r[32];
          bb::tmem_ld_32x32b_x32(t_row + pn * 32, r);
          bb::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] += __uint_as_float(r[i]);
        } else {
          const uint8_t* q0 = part + (t < ks ? t : t - 1) * PANEL_BYTES;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 q = *reinterpret_cast<const float4*>(q0 + j * 512);
            v[4 * j] += q.x; v[4 * j + 1] += q.y; v[4 * j + 2] += q.z; v[4 * j + 3] += q.w;
          }
        }
      }
      narrow_panel(p, slab, r0, nb, lane, v);
    }
  }
  bb::tc_fence_before_sync();
  __syncwarp();
  if (PAIR) {
    bb::cluster_sync();
    if (warp == MMA_WARP) bb::tmem_dealloc_pair(tmem_base, BN);
  } else {
    __syncthreads();
    if (warp == MMA_WARP) bb::tmem_dealloc(tmem_base, BN);
  }
}

// ---------------------------------------------------------------- host side
using bbhost::encode_2d;

// Ticket counters of the dynamic work distribution: a launch takes the next slot of a ring of
// counters in device memory and draws exactly `units` tickets from it (see the scheduling
// thread), so the host knows every counter's value without reading it back and nothing is ever
// reset.  A slot is reused 65536 launches later, long after the launch that held it retired.  A launch that is being captured takes
// no slot: the host cannot know how often, or whether, the graph runs, and every replay would start from another count.
constexpr unsigned TICKET_SLOTS = 1u << 16;
__device__ unsigned int g_gemm_tickets[TICKET_SLOTS];

struct TicketTable {
  unsigned int* dev = nullptr;
  std::atomic<unsigned> next{0};
  unsigned base[TICKET_SLOTS] = {};
};

// BB_GEMM_STATIC_SCHEDULE=1 in the environment restores the fixed stride (unit i of a CTA =
// its index + i x CTAs), for A/B measurements of the two distributions.
const bool g_static_schedule = [] { const char* e = getenv("BB_GEMM_STATIC_SCHEDULE"); return e && e[0] == '1'; }();

TicketTable* ticket_table() {
  static TicketTable* tables[64] = {nullptr};
  static std::mutex mu;
  const int dev = bb_current_device();
  if (dev < 0) return nullptr;
  TicketTable* t = tables[dev];
  if (t) return t;
  std::lock_guard<std::mutex> lock(mu);
  if (tables[dev]) return tables[dev];
  void* ptr = nullptr;
  if (cudaGetSymbolAddress(&ptr, g_gemm_tickets) != cudaSuccess) return nullptr;
  t = new TicketTable();
  t->dev = static_cast<unsigned int*>(ptr);
  tables[dev] = t;
  return t;
}

// (a stream that cannot be asked belongs to a capture that the launch itself will report)
bool capturing(cudaStream_t stream) {
  cudaStreamCaptureStatus st;
  if (cudaStreamIsCapturing(stream, &st) == cudaSuccess) return st != cudaStreamCaptureStatusNone;
  (void)cudaGetLastError();
  return true;
}

// Too few output tiles to fill the machine: split the reduction; partial sums meet in the fp32 add-reduction of the
// epilogue.  Cost model: waves x (k-blocks + fixed overhead).
int wave_split(int mn_tiles, int workers, int total_kb) {
  int ksplit = 1;
  long long best = -1;
  for (int s = 1; s <= 16; ++s) {
    const int kbs = (total_kb + s - 1) / s;
    if (s > 1 && kbs < 8) break;
    const long long waves = ((long long)mn_tiles * s + workers - 1) / workers;
    const long long cost = waves * (kbs + 8);
    if (best < 0 || cost < best) { best = cost; ksplit = s; }
  }
  return ksplit;
}

// Tensor maps and launch parameters of a product, except for the split of its reduction and the ticket counter.
// `cv`: convolution product (CONV); the descriptor then holds the sizes and the operand that is no patch matrix
template <int BN, bool PAIR, bool CONV>
int operands(const bb_gemm_desc* g, const bb_conv_gemm_args* cv, CUtensorMap& tmA, CUtensorMap& tmB, GemmParams& p,
             typename ConvArg<CONV>::type& cp) {
  using C = Cfg<BN, PAIR>;
  int rc;
  if (CONV && cv->mode != BB_CONV_WGRAD) rc = bbhost::encode_im2col(&tmA, cv->x, cv->N, cv->H, cv->W, cv->C, cv->k, cv->stride, cv->pad, BM);
  else if (!g->a_mn_major) rc = encode_2d(&tmA, g->A, g->M, g->K, g->lda, BK, BM);
  else rc = encode_2d(&tmA, g->A, g->K, g->M, g->lda, 64, BK);
  if (rc) return rc;
  if (CONV && cv->mode == BB_CONV_WGRAD) rc = bbhost::encode_im2col(&tmB, cv->x, cv->N, cv->H, cv->W, cv->C, cv->k, cv->stride, cv->pad, BK);
  else if (CONV && cv->mode == BB_CONV_DGRAD) rc = encode_2d(&tmB, g->B, cv->C, g->ldb, g->ldb, 64, BK);
  else if (!g->b_mn_major) rc = encode_2d(&tmB, g->B, g->N, g->K, g->ldb, BK, C::B_ROWS);
  else rc = encode_2d(&tmB, g->B, g->K, g->N, g->ldb, 64, BK);
  if (rc) return rc;
  if constexpr (CONV) {
    cp.mode = cv->mode; cp.k = cv->k; cp.stride = cv->stride; cp.pad = cv->pad; cp.cblocks = cv->C / 64;
    cp.wcols = cv->mode == BB_CONV_DGRAD ? cv->other_channels : cv->C;
    cp.Wo = cv->Wo; cp.Ho = cv->Ho;
    cp.magic_w = bb_div_magic(cv->Wo);
    cp.magic_h = bb_div_magic(cv->Ho);
  }
  p.M = g->M; p.N = g->N; p.K = g->K; p.a_mn = g->a_mn_major; p.b_mn = g->b_mn_major; p.epi = g->epilogue;
  p.D = g->D; p.D2 = g->D2; p.bias = g->bias; p.aux = g->aux; p.ldd = g->ldd; p.ld_aux = g->ld_aux ? g->ld_aux : g->ldd;
  p.status = bb_device_status_word();
  // The CTAs that run at the same time share one operand and stream the other: walk along the
  // dimension of the SMALLER operand, so that the larger one passes through L2 once.
  p.n_fast = (long long)g->M > (long long)g->N ? 1 : 0;
  const int num_m = (g->M + C::TILE_M - 1) / C::TILE_M, num_n = (g->N + BN - 1) / BN;
  p.tiles_in = p.n_fast ? num_n : num_m; p.tiles_mn = (unsigned)num_m * (unsigned)num_n;
  p.magic_in = bb_div_magic((int)p.tiles_in); p.magic_mn = bb_div_magic((int)p.tiles_mn);
  p.dynamic = 0; p.ticket = nullptr; p.ticket_base = 0;
  return BB_OK;
}

template <int BN, bool PAIR, int EW, bool CONV>
int launch(const bb_gemm_desc* g, cudaStream_t stream, const bb_conv_gemm_args* cv = nullptr) {
  using C = Cfg<BN, PAIR>;
  CUtensorMap tmA, tmB;
  GemmParams p;
  typename ConvArg<CONV>::type cp;
  if (int rc = operands<BN, PAIR, CONV>(g, cv, tmA, tmB, p, cp)) return rc;
  const int total_kb = (g->K + BK - 1) / BK;
  const int mn_tiles = ((g->M + C::TILE_M - 1) / C::TILE_M) * ((g->N + BN - 1) / BN);
  const int workers_max = PAIR ? bb_num_sms() / 2 : bb_num_sms();
  int ksplit = 1;
  if (g->epilogue == BB_EPI_ACCUM_F32) {
    if (g->split_k > 0) {
      ksplit = g->split_k;
    } else {
      ksplit = wave_split(mn_tiles, workers_max, total_kb);
    }
  }
  if (ksplit > total_kb) ksplit = total_kb;
  if (ksplit < 1) ksplit = 1;
  p.kb_per_split = (total_kb + ksplit - 1) / ksplit;
  p.ksplit = (total_kb + p.kb_per_split - 1) / p.kb_per_split;   // no empty splits
  BB_ONCE_PER_DEVICE(BB_CUDA_CHECK(cudaFuncSetAttribute(gemm_bf16_tcgen05_kernel<BN, PAIR, EW, CONV>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES)));
  const int tiles = mn_tiles * p.ksplit;
  int workers = workers_max;
  if (g->max_ctas > 0 && g->max_ctas / (PAIR ? 2 : 1) < workers) workers = g->max_ctas / (PAIR ? 2 : 1);
  if (workers < 1) workers = 1;
  if (tiles < workers) workers = tiles;
  // max_ctas < 0: one work unit per CTA (or pair).  Meant for work on a low-priority stream: a
  // persistent CTA that found a free SM keeps it for its whole tile loop, and a persistent kernel
  // of the main stream launched meanwhile waits for that SM with a fixed share of the tiles.
  if (g->max_ctas < 0) workers = tiles;
  // more units than CTAs: every unit after a CTA's first is drawn from this launch's ticket counter (in a graph: unit i of a CTA
  // is its index + i x CTAs)
  unsigned slot = 0;
  TicketTable* tt = nullptr;
  if (tiles > workers && !g_static_schedule && !capturing(stream)) {
    tt = ticket_table();
    if (!tt) { bb_set_last_error_msg("bb_gemm_bf16: ticket counters unavailable on this device"); return BB_ERR_CUDA; }
    slot = tt->next.fetch_add(1u) & (TICKET_SLOTS - 1);
    p.dynamic = 1; p.ticket = tt->dev + slot; p.ticket_base = tt->base[slot];
    tt->base[slot] += (unsigned)tiles;
  }
  if constexpr (PAIR) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * workers); cfg.blockDim = dim3(num_threads(EW));
    cfg.dynamicSmemBytes = C::SMEM_BYTES; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = bb_back_to_back > 0 ? 2 : 1;
    cudaError_t le = cudaLaunchKernelEx(&cfg, gemm_bf16_tcgen05_kernel<BN, true, EW, CONV>, tmA, tmB, p, cp);
    if (le != cudaSuccess) {
      if (tt) tt->base[slot] -= (unsigned)tiles;     // nothing ran: the counter keeps its value
      bb_set_last_error("gemm_bf16_tcgen05_kernel (pair) launch", le);
      return BB_ERR_CUDA;
    }
  } else {
    bb_launch(gemm_bf16_tcgen05_kernel<BN, false, EW, CONV>, workers, num_threads(EW), C::SMEM_BYTES, stream, tmA, tmB, p, cp);
  }
  {
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) {
      if (tt) tt->base[slot] -= (unsigned)tiles;     // nothing ran: the counter keeps its value
      bb_set_last_error("gemm_bf16_tcgen05_kernel launch", le);
      return BB_ERR_CUDA;
    }
  }
  return BB_OK;
}

template <int BN, bool PAIR, bool CONV>
cudaLaunchConfig_t split_config(int splits, int tiles, cudaLaunchAttribute* attr) {
  const int cluster = splits * (PAIR ? 2 : 1);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster * tiles); cfg.blockDim = dim3(num_threads(SPLIT_EW)); cfg.dynamicSmemBytes = Cfg<BN, PAIR>::SMEM_BYTES;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  return cfg;
}

// The same product with its reduction split over the CTAs of a cluster (gemm_cluster_split_kernel)
template <int BN, bool PAIR, bool CONV>
int launch_split(const bb_gemm_desc* g, cudaStream_t stream, int splits, const bb_conv_gemm_args* cv = nullptr) {
  using C = Cfg<BN, PAIR>;
  CUtensorMap tmA, tmB;
  GemmParams p;
  typename ConvArg<CONV>::type cp;
  if (int rc = operands<BN, PAIR, CONV>(g, cv, tmA, tmB, p, cp)) return rc;
  const int total_kb = (g->K + BK - 1) / BK;
  if (splits > split_limit(PAIR)) splits = split_limit(PAIR);
  if (splits > total_kb) splits = total_kb;
  p.kb_per_split = (total_kb + splits - 1) / splits;
  p.ksplit = (total_kb + p.kb_per_split - 1) / p.kb_per_split;   // no empty splits
  BB_ONCE_PER_DEVICE(BB_CUDA_CHECK(cudaFuncSetAttribute(gemm_cluster_split_kernel<BN, PAIR, CONV>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES)));
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = split_config<BN, PAIR, CONV>(p.ksplit, (int)p.tiles_mn, attr);
  cfg.stream = stream;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[1].val.programmaticStreamSerializationAllowed = 1;
  if (bb_back_to_back > 0) cfg.numAttrs = 2;
  BB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, gemm_cluster_split_kernel<BN, PAIR, CONV>, tmA, tmB, p, cp));
  return BB_OK;
}

// Whether a weight gradient may run as CTA pairs.  It runs beside the input gradients of its layer, and a pair needs both SMs of
// a processing cluster free: beside an input gradient of few single CTAs short reductions starve as pairs (vocabulary head on
// 999 tokens: the weight gradient alone 122 -> 107 us, the case 475 -> 628 us).
bool pairs_pay(int M, int N, int K) {
  const long long tiles_single = (long long)((M + BM - 1) / BM) * ((N + 255) / 256);
  return M > BM && N > 128 && (K >= 2048 || tiles_single >= 16LL * bb_num_sms());
}

// Weight gradients (fp32 add-reduction): few output tiles and a long reduction, so tile, pairing and the split of the
// reduction are chosen together, by the time in microseconds: waves x (k-blocks x rate + a tile's start and add-reduction) +
// once per launch (fitted on 35 products with up to 24 splits each, within a tenth; 1024 x 1024 x 2331
// 11.8 -> 10.3 us, 1024 x 256 x 8192 12.4 -> 10.9 against a plan that counted operand loads).  Splits go as far as one wave of the machine (or 16, as more
// than one wave evens out ragged ones) and leave at least eight k-blocks per unit (short reductions stay whole, with one
// order of additions).  No unit sums more k-blocks than wave_split gives the widest tile: the accumulator's rounding
// grows with their number (256 x 2304 x 6272 against fp64: 13 k-blocks 7.8e-7, 25 k-blocks 1.6e-6).
// Measured (us, before: at most 16 splits and always 256 columns): 64 x 64 x 100352 41 -> 14.4, 64 x 576 x 100352
// 57 -> 37, 256 x 64 x 100352 41 -> 22.5, 256 x 512 x 25088 24.6 -> 18.4, 64 x 392 x 401408 186 -> 84, 128 x 128 x 800
// 14.3 -> 12.3; 1024 x 1024 x 8192 and larger as before.
struct AccumPlan { int bn; bool pair; int ksplit; };
AccumPlan plan_accum(int M, int N, int K) {
  static const struct { int bn; bool pair; double kblock, tile, once; } kinds[3] = {
      {256, true, 0.316, 4.6, 3.2}, {256, false, 0.365, 4.6, 1.9}, {128, false, 0.282, 1.75, 3.1}};
  const long long kb = (K + BK - 1) / BK;
  long long longest;
  {
    const bool pair = pairs_pay(M, N, K);
    const int tm = pair ? 2 * BM : BM, bn = N > 128 ? 256 : 128;
    const int s = wave_split(((M + tm - 1) / tm) * ((N + bn - 1) / bn), pair ? bb_num_sms() / 2 : bb_num_sms(), (int)kb);
    longest = (kb + s - 1) / s;
  }
  AccumPlan best = {128, false, 1};
  double best_cost = -1;
  for (const auto& k : kinds) {
    const int bn = k.bn;
    const bool pair = k.pair;
    if ((bn == 256 && N <= 128) || (pair && !pairs_pay(M, N, K))) continue;
    const long long tm = pair ? 2 * BM : BM;
    const long long tiles = ((M + tm - 1) / tm) * ((N + bn - 1) / bn);
    const long long workers = pair ? bb_num_sms() / 2 : bb_num_sms();
    // up to 16, then the largest that stays within one wave: between the two a larger split only shortens the units
    long long widest = workers / tiles;
    if (widest > (kb - 1) / 7) widest = (kb - 1) / 7;        // (the largest with eight k-blocks per unit)
    for (int i = 1; i <= 17; ++i) {
      const long long s = i <= 16 ? i : widest;
      if (i == 17 && widest <= 16) break;
      const long long kbs = (kb + s - 1) / s;
      if (s > 1 && kbs < 8) break;
      if (kbs > longest) continue;
      const long long units = tiles * ((kb + kbs - 1) / kbs);
      const double cost = (double)((units + workers - 1) / workers) * ((double)kbs * k.kblock + k.tile) + k.once;
      if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = {bn, pair, (int)s}; }
    }
  }
  return best;
}

// Products that are stored: tile width and pairing by the time that they are expected to take, in microseconds.  A tile
// costs a rate per k-block (128 x 128, 128 x 256, and 128 x 256 for each CTA of a pair, the cheapest per output because
// it loads least) and, wave after wave, what its epilogue leaves uncovered; once per launch its start and its last
// epilogue.  Fitted on 57 products of 512 x 256 x 256 to 8192 x 50304 x 1024 with every epilogue, where the times are met within a
// tenth on average and the choice is the quickest of the three every time.  Constants from before the pairs' hand-backs became
// cheap kept 8192 x 4096 x 1024 (bias + GeLU 66.5 us, as pairs 57.2), 8192 x 3072 x 1024 (47.4, 42.7), 2331 x 4096 x 1024 (31.1, 27.8)
// and 8192 x 50304 x 1024 (648, 564) on single CTAs.
struct StorePlan { int bn; bool pair; double us; int splits = 0; };
StorePlan plan_store(long long M, long long N, long long K, int max_ctas, bool pairs_allowed) {
  static const struct { int bn; bool pair; double kblock, wave, once; } kinds[3] = {
      {256, true, 0.32, 1.9, 5.0}, {256, false, 0.375, 1.8, 3.7}, {128, false, 0.283, 1.0, 3.7}};
  const double kb = (double)((K + BK - 1) / BK);
  StorePlan best = {128, false, -1};
  for (const auto& k : kinds) {
    if ((k.bn == 256 && N <= 128) || (k.pair && (!pairs_allowed || M <= BM))) continue;
    const long long tm = k.pair ? 2 * BM : BM;
    const long long tiles = ((M + tm - 1) / tm) * ((N + k.bn - 1) / k.bn);
    long long workers = bb_num_sms();
    if (max_ctas > 0 && max_ctas < workers) workers = max_ctas;
    if (k.pair) workers = workers > 1 ? workers / 2 : 1;
    const double us = (double)((tiles + workers - 1) / workers) * (kb * k.kblock + k.wave) + k.once;
    if (best.us < 0 || us < best.us) best = {k.bn, k.pair, us};
  }
  return best;
}

// Clusters of `cluster` CTAs of the split kernel that the device holds at the same time (GPCs are not multiples of every cluster
// size); 0 when it cannot be asked.
template <int BN, bool PAIR>
int clusters_at_once(int splits) {
  static std::atomic<int> cache[64][9];
  const int dev = bb_current_device();
  if (dev < 0) return 0;
  int n = cache[dev][splits].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = split_config<BN, PAIR, false>(splits, 1, attr);
    if (cudaFuncSetAttribute(gemm_cluster_split_kernel<BN, PAIR, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN, PAIR>::SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_cluster_split_kernel<BN, PAIR, false>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      n = 0;
    }
    if (n <= 0) n = -1;
    cache[dev][splits].store(n, std::memory_order_relaxed);
  }
  return n > 0 ? n : 0;
}

// The plan with the reduction split over a cluster where that is expected to be quicker by a twentieth: one wave of clusters, every
// split with four k-blocks or more.  The exchange costs about half a microsecond per split on top of a launch
// (once + step x splits; us, unsplit / split: 513 x 2048 x 8192 41.7 / 25.5 as three splits of 256 columns, 128 x 1024 x 4096
// 20.9 / 9.9 as six of 128, 1000 x 512 x 2048 12.9 / 9.0 as four, 1568 x 512 x 4608 24.8 / 16.0, 512 x 256 x 1024 8.2 / 7.1; with K = 512
// and less, or tiles for more than half of the SMs, nothing is gained).
// The constants come from an idle GPU; beside other work the split holds up (us, whole / split): forward + backward of one block with
// its weight gradients on the side stream 513 x 2048 413 / 376, 1000 x 2048 503 / 468, 300 x 4096 834 / 764, 513 x 4096 982 / 991,
// 1100 x 1024 260 / 278; a projection of 999 x 1024 to 50264 357 / 305, 513 x 2048 to 30528 257 / 243; twelve blocks forward
// beside redundant work of one tile per CTA 513 x 2048 2106 / 1924, 300 x 4096 3347 / 2910, 512 x 1024 1274 / 1284.
// A split sums in another order than the whole reduction, in fp32 either way and as close to 64 bits.  So the bf16 rounding of a product may
// depend on how many rows ride along and on the budget: the stage's own forward and a redundant one, whose budget of CTAs
// keeps reductions whole, agree within one rounding and not bit for bit.
StorePlan plan_split(long long M, long long N, long long K) {
  static const struct { int bn; bool pair; double kblock, once, step; } kinds[3] = {
      {256, true, 0.32, 7.2, 0.95}, {256, false, 0.375, 6.2, 0.6}, {128, false, 0.283, 4.7, 0.45}};
  const StorePlan whole = plan_store(M, N, K, 0, true);
  StorePlan best = whole;
  const long long kb = (K + BK - 1) / BK;
  for (const auto& k : kinds) {
    if ((k.bn == 256 && N <= 128) || (k.pair && M <= BM)) continue;
    const long long tm = k.pair ? 2 * BM : BM;
    const long long tiles = ((M + tm - 1) / tm) * ((N + k.bn - 1) / k.bn);
    for (int sp = 2; sp <= split_limit(k.pair) && kb / sp >= 4; ++sp) {
      if (tiles * sp * (k.pair ? 2 : 1) > bb_num_sms()) break;
      const int at_once = k.pair ? clusters_at_once<256, true>(sp) : k.bn == 256 ? clusters_at_once<256, false>(sp) : clusters_at_once<128, false>(sp);
      if (tiles > at_once) continue;
      const double us = (double)((kb + sp - 1) / sp) * k.kblock + k.once + k.step * sp;
      if (us < best.us && us * 1.05 < whole.us) best = {k.bn, k.pair, us, sp};
    }
  }
  return best;
}

// The plans of a thread's recent problem sizes (a plan depends on nothing else but the device): going through up to seventeen
// splits of three kinds of tile costs the host half a microsecond to two per product, as much as its tensor maps.
struct PlanMemo { int M = 0, N = 0, K = 0, dev = -1, accum = 0, bn = 0, splits = 0; bool pair = false; double us = 0; };
const PlanMemo& memoised_plan(int M, int N, int K, bool accum) {
  static thread_local PlanMemo memo[256];
  unsigned h = (unsigned)M * 2654435761u ^ (unsigned)N * 2246822519u ^ (unsigned)K * 3266489917u ^ (accum ? 1u : 0u);
  PlanMemo& e = memo[(h ^ (h >> 16)) & 255u];
  const int dev = bb_current_device();
  if (e.M != M || e.N != N || e.K != K || e.accum != (accum ? 1 : 0) || e.dev != dev || dev < 0) {
    e.M = M; e.N = N; e.K = K; e.dev = dev; e.accum = accum ? 1 : 0;
    if (accum) {
      const AccumPlan pl = plan_accum(M, N, K);
      e.bn = pl.bn; e.pair = pl.pair; e.splits = pl.ksplit;
    } else {
      const StorePlan pl = plan_split(M, N, K);
      e.bn = pl.bn; e.pair = pl.pair; e.splits = pl.splits; e.us = pl.us;
    }
  }
  return e;
}

// Tile width, pairing, epilogue warps, and the split of the reduction (bf16 outputs: 0 for none)
int choose_tile(bb_gemm_desc* g, bool* pair_out, bool* wide_out) {
  const int e = g->epilogue;
  const bool all_sms = g->max_ctas == 0 || g->max_ctas >= bb_num_sms();
  *wide_out = false;
  // a split over a cluster takes CTAs and epilogue warps of its own: a descriptor that names either keeps the reduction whole
  if (e != BB_EPI_ACCUM_F32 && (!all_sms || g->epi_warps != 0 || g->split_k < 0)) g->split_k = 0;
  if (e == BB_EPI_ACCUM_F32 && g->split_k <= 0 && g->tile_n == 0 && g->cta_pair == 0) {
    const PlanMemo& pl = memoised_plan(g->M, g->N, g->K, true);
    g->split_k = pl.splits;
    *pair_out = pl.pair;
    return pl.bn;
  }
  // eight epilogue warps unless sixteen are asked for: with two-wide arithmetic and panels stored without a test per row they
  // finish a tile within the next one's main loop (us, eight / sixteen: 8192 x 4096 x 1024 bias + GeLU 65.7 / 69.8, residual
  // 66.0 / 70.3; 8192 x 1024 x 1024 plain 18.6 / 20.5).  Sixteen are the quicker only for x gelu' on tiles that nothing follows
  // (4096 x 1024 x 1024 20.5 / 16.8-19.5, 2331 x 1024 x 1024 15.6 / 14.5) and on the shortest reductions (16384 x 1024 x 256 27.6 /
  // 26.9, 100352 x 256 x 64 47.7 / 43.5).
  *wide_out = g->epi_warps == 4;
  *pair_out = g->cta_pair > 0;
  if (g->cta_pair > 0) return 256;
  if (g->tile_n != 0) return g->tile_n;
  // an add-reduction whose split was given takes wide tiles: the split fills the machine
  if (e == BB_EPI_ACCUM_F32) {
    *pair_out = g->cta_pair == 0 && pairs_pay(g->M, g->N, g->K);
    return g->N > 128 ? 256 : 128;
  }
  if (e != BB_EPI_STORE_F32 && all_sms && g->split_k == 0 && g->cta_pair == 0 && g->epi_warps == 0) {
    const PlanMemo& pl = memoised_plan(g->M, g->N, g->K, false);
    g->split_k = pl.splits;
    *pair_out = pl.pair;
    return pl.bn;
  }
  const StorePlan pl = plan_store(g->M, g->N, g->K, g->max_ctas, g->cta_pair == 0);
  *pair_out = pl.pair;
  return pl.bn;
}

}  // namespace

extern "C" int bb_gemm_bf16(const bb_gemm_desc* g, void* stream) {
  if (!g || !g->A || !g->B || !g->D || g->M <= 0 || g->N <= 0 || g->K <= 0) {
    bb_set_last_error_msg("bb_gemm_bf16: null operand or non-positive size");
    return BB_ERR_INVALID_ARG;
  }
  const int e = g->epilogue;
  if (e < BB_EPI_STORE || e > BB_EPI_BIAS_RESIDUAL) { bb_set_last_error_msg("bb_gemm_bf16: unknown epilogue"); return BB_ERR_INVALID_ARG; }
  if ((e == BB_EPI_BIAS || e == BB_EPI_BIAS_GELU || e == BB_EPI_BIAS_RESIDUAL) && !g->bias) {
    bb_set_last_error_msg("bb_gemm_bf16: epilogue needs bias"); return BB_ERR_INVALID_ARG; }
  if (e == BB_EPI_BIAS_GELU && !g->D2) { bb_set_last_error_msg("bb_gemm_bf16: GeLU epilogue needs D2"); return BB_ERR_INVALID_ARG; }
  if ((e == BB_EPI_MUL_DGELU || e == BB_EPI_BIAS_RESIDUAL) && !g->aux) {
    bb_set_last_error_msg("bb_gemm_bf16: epilogue needs aux"); return BB_ERR_INVALID_ARG; }
  const bool f32 = (e == BB_EPI_ACCUM_F32 || e == BB_EPI_STORE_F32);
  if (g->lda % 8 || g->ldb % 8 || g->ldd % (f32 ? 4 : 8) || (g->ld_aux % 8) ||
      ((uintptr_t)g->A & 15) || ((uintptr_t)g->B & 15) || ((uintptr_t)g->D & 15) || ((uintptr_t)g->D2 & 15) ||
      ((uintptr_t)g->aux & 15) || ((uintptr_t)g->bias & 15)) {
    bb_set_last_error_msg("bb_gemm_bf16: pointers must be 16-byte aligned and leading dimensions multiples of 8 elements");
    return BB_ERR_INVALID_ARG;
  }
  if ((g->epi_warps != 0 && g->epi_warps != 2 && g->epi_warps != 4) || (g->epi_warps == 4 && f32)) {
    bb_set_last_error_msg("bb_gemm_bf16: epi_warps must be 0, 2 or 4 (4 only with bf16 outputs)");
    return BB_ERR_INVALID_ARG;
  }
  if (g->cta_pair <= 0 && g->tile_n != 0 && g->tile_n != 128 && g->tile_n != 256) {
    bb_set_last_error_msg("bb_gemm_bf16: tile_n must be 0, 128 or 256");
    return BB_ERR_INVALID_ARG;
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // cuTensorMapEncodeTiled is a driver call and needs a context bound to the calling thread;
  // a thread that has only ever set its device (autograd worker threads) has none yet.
  if (int rc = bbhost::bind_context()) return rc;
  bool pair, wide_epi;
  bb_gemm_desc planned = *g;
  const int bn = choose_tile(&planned, &pair, &wide_epi);
  g = &planned;
  if (!f32 && g->split_k > 0) {
    if (pair) return launch_split<256, true, false>(g, s, g->split_k);
    return bn == 256 ? launch_split<256, false, false>(g, s, g->split_k) : launch_split<128, false, false>(g, s, g->split_k);
  }
  if (pair) return wide_epi ? launch<256, true, 4, false>(g, s) : launch<256, true, 2, false>(g, s);
  if (bn == 256) return wide_epi ? launch<256, false, 4, false>(g, s) : launch<256, false, 2, false>(g, s);
  return wide_epi ? launch<128, false, 4, false>(g, s) : launch<128, false, 2, false>(g, s);
}

double bb_gemm_store_us(long long M, long long N, long long K, int max_ctas) {
  if (max_ctas != 0 && max_ctas < bb_num_sms()) return plan_store(M, N, K, 0, true).us;      // (a budget keeps the reduction whole)
  if (M > INT_MAX || N > INT_MAX || K > INT_MAX) return plan_split(M, N, K).us;
  return memoised_plan((int)M, (int)N, (int)K, false).us;
}

bool bb_conv_gemm_supported(int C, int k, int stride, int pad) {
  // tensor map limits of a rank-4 im2col load: window corners in [-128, 127], traversal stride <= 8
  return C > 0 && C % 64 == 0 && k >= 1 && k <= 64 && stride >= 1 && stride <= 8 && pad >= 0 && pad < k;
}

int bb_conv_gemm(const bb_conv_gemm_args* a, void* stream) {
  const long long P = (long long)a->N * a->Ho * a->Wo;
  if (!a->x || !a->other || !a->D || P <= 0 || P >= (1LL << 31) || !bb_conv_gemm_supported(a->C, a->k, a->stride, a->pad) ||
      a->H + 2 * a->pad < a->k || a->W + 2 * a->pad < a->k ||
      a->other_channels <= 0 || (a->other_channels & 7) || (a->mode == BB_CONV_DGRAD && a->stride != 1) ||
      (((uintptr_t)a->x | (uintptr_t)a->other | (uintptr_t)a->D) & 15)) {
    bb_set_last_error_msg("bb_conv_gemm: null or unaligned operand, or a geometry the im2col loads cannot express");
    return BB_ERR_INVALID_ARG;
  }
  const int taps = a->k * a->k;
  bb_gemm_desc g = {};
  g.D = a->D; g.max_ctas = a->max_ctas;
  if (a->mode == BB_CONV_WGRAD) {
    g.M = a->other_channels; g.N = taps * a->C; g.K = (int)P;
    g.A = a->other; g.lda = a->other_channels; g.a_mn_major = 1; g.b_mn_major = 1;
    g.ldd = g.N; g.epilogue = BB_EPI_ACCUM_F32;
  } else {
    g.M = (int)P; g.N = a->other_channels; g.K = taps * a->C;
    g.B = a->other; g.ldb = a->mode == BB_CONV_FWD ? g.K : (long long)taps * a->other_channels;
    g.b_mn_major = a->mode == BB_CONV_DGRAD;
    g.ldd = a->other_channels; g.epilogue = BB_EPI_STORE;
  }
  if (int rc = bbhost::bind_context()) return rc;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  bool pair, wide_epi;
  const int bn = choose_tile(&g, &pair, &wide_epi);
  if (g.epilogue == BB_EPI_STORE && g.split_k > 0) {
    if (pair) return launch_split<256, true, true>(&g, s, g.split_k, a);
    return bn == 256 ? launch_split<256, false, true>(&g, s, g.split_k, a) : launch_split<128, false, true>(&g, s, g.split_k, a);
  }
  if (pair) return launch<256, true, 2, true>(&g, s, a);
  return bn == 256 ? launch<256, false, 2, true>(&g, s, a) : launch<128, false, 2, true>(&g, s, a);
}
