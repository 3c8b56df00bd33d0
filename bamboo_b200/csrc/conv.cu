// Channels-last (NHWC, bf16) pieces of the ResNet stages around the tensor-core GEMM: patch
// gathering for k x k convolutions and its adjoint, batch normalisation with batch statistics
// (forward and backward, ReLU and the residual add folded in), 3 x 3 / stride 2 max pooling and
// global average pooling.  All of these are HBM-bound: 16-byte vectors over the channel
// dimension, consecutive threads on consecutive channel chunks of a pixel, fp32 arithmetic.
// A convolution itself is the library's GEMM: output pixels x (taps * input channels) times the
// [Cout, k, k, Cin] weight matrix.  With channels in blocks of 64 the GEMM gathers the patches itself
// (im2col TMA loads, bb_conv_gemm); the patch kernels below serve the other channel counts (the stem, narrow
// networks) and the input gradient of strided convolutions.
#include "common.cuh"
#include "bamboo_b200.h"

namespace {

__device__ __forceinline__ void unpack8(const uint4& q, float* f) {
  f[0] = bb::bf16_lo(q.x); f[1] = bb::bf16_hi(q.x); f[2] = bb::bf16_lo(q.y); f[3] = bb::bf16_hi(q.y);
  f[4] = bb::bf16_lo(q.z); f[5] = bb::bf16_hi(q.z); f[6] = bb::bf16_lo(q.w); f[7] = bb::bf16_hi(q.w);
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 q;
  q.x = bb::pack_bf16x2(f[0], f[1]); q.y = bb::pack_bf16x2(f[2], f[3]);
  q.z = bb::pack_bf16x2(f[4], f[5]); q.w = bb::pack_bf16x2(f[6], f[7]);
  return q;
}

int flat_grid(long long work_items, int per_thread = 1) {
  long long blocks = (work_items + 256LL * per_thread - 1) / (256LL * per_thread);
  const long long cap = (long long)bb_num_sms() * 16;
  if (blocks > cap) blocks = cap;
  return (int)(blocks < 1 ? 1 : blocks);
}

struct ConvGeom {
  int N, H, W, C, k, stride, pad, Ho, Wo;
  long long ld_col;      // elements between consecutive rows of the patch matrix (>= k*k*C)
};

// Both patch kernels walk image rows (blockIdx.y) and 16-byte chunks inside a row (blockIdx.x): the indices of a chunk
// then take three multiplications by reciprocals.  With a 64-bit division per index, the 7 x 7 / stride 2 gather of
// 32 x 224 x 224 x 8 took 144 us for its 315 MB (arithmetic, not memory; now 72 us), the fourteen adjoint gathers of an
// image-network step 574 us (now 442 us).  Index type I: rows of 2^31 chunks (34 GB) and more take 64-bit divisions.
struct ConvMagic { unsigned long long row_chunks, chunks, k, rows; };
constexpr int PATCH_U = 4;             // chunks per thread of the gather

template <typename I> __device__ __forceinline__ I chunk_div(I n, I d, unsigned long long magic) {
  if constexpr (sizeof(I) == 4) return bb::fast_div(n, magic);
  else return n / d;
}

// col[(n, ho, wo), (r, s, c)] = x[n, ho*stride - pad + r, wo*stride - pad + s, c]  (0 outside)
template <typename I>
__global__ void __launch_bounds__(256)
im2col_kernel(const uint4* x, uint4* __restrict__ col, const ConvGeom g, const ConvMagic m) {
  bb::pdl_sync();
  const I chunks = g.C >> 3;                              // 16-byte chunks per pixel
  const I row_chunks = (I)g.k * g.k * chunks;
  const I total = g.Wo * row_chunks;
  const long long ld16 = g.ld_col >> 3;
  const I e0 = (I)blockIdx.x * (256 * PATCH_U) + threadIdx.x;
  for (unsigned row = blockIdx.y; row < (unsigned)g.N * g.Ho; row += gridDim.y) {
    const unsigned n = bb::fast_div(row, m.rows);
    const int h0 = (int)(row - n * g.Ho) * g.stride - g.pad;
    const uint4* xi = x + (long long)n * g.H * g.W * (long long)chunks;
    uint4* out = col + (long long)row * g.Wo * ld16;
    uint4 v[PATCH_U];
    long long dst[PATCH_U];
#pragma unroll
    for (int u = 0; u < PATCH_U; ++u) {
      const I e = e0 + u * 256;
      const I wo = chunk_div<I>(e, row_chunks, m.row_chunks), within = e - wo * row_chunks;
      const I tap = chunk_div<I>(within, chunks, m.chunks), cc = within - tap * chunks;
      const I r = chunk_div<I>(tap, g.k, m.k), s = tap - r * g.k;
      const int h = h0 + (int)r, w = (int)wo * g.stride - g.pad + (int)s;
      dst[u] = e < total ? (long long)wo * ld16 + within : -1;
      v[u] = make_uint4(0, 0, 0, 0);
      if (e < total && h >= 0 && h < g.H && w >= 0 && w < g.W) v[u] = __ldca(xi + ((long long)h * g.W + w) * (long long)chunks + cc);
    }
#pragma unroll
    for (int u = 0; u < PATCH_U; ++u) if (dst[u] >= 0) out[dst[u]] = v[u];
  }
}

// Adjoint of the gather: dx[n, h, w, c] = sum over the (output pixel, tap) pairs that read it.
// Gather form (one thread owns an input pixel's chunk): no atomics, fixed summation order (r, then s, ascending).
// The taps that reach a pixel are every stride-th one; along them the output pixel moves back by one.
template <typename I>
__global__ void __launch_bounds__(256)
col2im_kernel(const uint4* dcol, uint4* __restrict__ dx, const ConvGeom g, const ConvMagic m) {
  bb::pdl_sync();
  const I chunks = g.C >> 3;
  const I total = g.W * chunks;
  const long long ld16 = g.ld_col >> 3;
  const I e = (I)blockIdx.x * 256 + threadIdx.x;
  if (e >= total) return;
  const I w = chunk_div<I>(e, chunks, m.chunks), cc = e - w * chunks;
  const int s0 = (int)(w + g.pad) % g.stride, wo0 = (int)(w + g.pad) / g.stride;
  for (unsigned row = blockIdx.y; row < (unsigned)g.N * g.H; row += gridDim.y) {
    const unsigned n = bb::fast_div(row, m.rows);
    const int h = (int)(row - n * g.H);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    int ho = (h + g.pad) / g.stride;
    for (int r = (h + g.pad) % g.stride; r < g.k && ho >= 0; r += g.stride, --ho) {
      if (ho >= g.Ho) continue;
      const uint4* src = dcol + ((long long)n * g.Ho + ho) * g.Wo * ld16 + (long long)r * g.k * (long long)chunks + cc;
      int wo = wo0;
#pragma unroll 4
      for (int s = s0; s < g.k; s += g.stride, --wo) {
        if (wo < 0 || wo >= g.Wo) continue;
        float f[8];
        unpack8(__ldca(src + (long long)wo * ld16 + s * chunks), f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += f[i];
      }
    }
    dx[(long long)row * total + e] = pack8(acc);
  }
}

// The same for strides 1 and 2 and up to T taps along each dimension that reach a pixel (T = ceil(k / S)): a thread owns an input
// column's chunk over `rows` image rows, so what depends on the column is computed once and by shifts, and no load waits for an
// address or a branch; taps are added in the same order (r, then s).  How many of them are in flight is the compiler's choice (32
// registers for nine taps do not hold all).  With four divisions by the stride and a chain of loads per 16-byte
// result the general kernel ran at a third of the memory rate (us): 32 x 56 x 56 x 128, 3 x 3 / 2 36.8,
// 32 x 56 x 56 x 256, 1 x 1 / 2 28.4, 32 x 56 x 56 x 64, 3 x 3 45.3, 32 x 224 x 224 x 8, 7 x 7 / 2 141.6; this one 17.2,
// 13.7, 21.0 and 65.1.
template <typename I, int S, int T>
__global__ void __launch_bounds__(256)
col2im_taps_kernel(const uint4* dcol, uint4* __restrict__ dx, const ConvGeom g, const ConvMagic m, unsigned rows) {
  bb::pdl_sync();
  const I chunks = g.C >> 3;
  const I total = g.W * chunks;
  const long long ld16 = g.ld_col >> 3;
  const I e = (I)blockIdx.x * 256 + threadIdx.x;
  if (e >= total) return;
  const I w = chunk_div<I>(e, chunks, m.chunks), cc = e - w * chunks;
  const int ws = (int)w + g.pad, s0 = ws & (S - 1), wo0 = ws / S;
  long long off[T];                                        // of a tap inside its row of windows; -1: no window there
#pragma unroll
  for (int j = 0; j < T; ++j) {
    const int s = s0 + j * S, wo = wo0 - j;
    off[j] = s < g.k && wo >= 0 && wo < g.Wo ? (long long)wo * ld16 + (long long)s * (long long)chunks + (long long)cc : -1;
  }
  const unsigned last = (unsigned)g.N * g.H;
  for (unsigned first = blockIdx.y * rows; first < last; first += gridDim.y * rows) {
    const unsigned end = min(first + rows, last);
    for (unsigned row = first; row < end; ++row) {
      const unsigned n = bb::fast_div(row, m.rows);
      const int hs = (int)(row - n * g.H) + g.pad, r0 = hs & (S - 1), ho0 = hs / S;
      uint4 q[T][T];
#pragma unroll
      for (int i = 0; i < T; ++i) {
        const int r = r0 + i * S, ho = ho0 - i;
        const bool in = r < g.k && ho >= 0 && ho < g.Ho;
        const uint4* src = dcol + ((long long)n * g.Ho + ho) * g.Wo * ld16 + (long long)r * g.k * (long long)chunks;
#pragma unroll
        for (int j = 0; j < T; ++j) q[i][j] = in && off[j] >= 0 ? __ldca(src + off[j]) : make_uint4(0, 0, 0, 0);
      }
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) {
          float f[8];
          unpack8(q[i][j], f);
#pragma unroll
          for (int c = 0; c < 8; ++c) acc[c] += f[c];
        }
      dx[(long long)row * total + e] = pack8(acc);
    }
  }
}

bool bad_geom(const ConvGeom& g) {
  return g.N <= 0 || g.H <= 0 || g.W <= 0 || g.C <= 0 || (g.C & 7) || g.k <= 0 || g.stride <= 0 || g.pad < 0 ||
         g.Ho != (g.H + 2 * g.pad - g.k) / g.stride + 1 || g.Wo != (g.W + 2 * g.pad - g.k) / g.stride + 1 ||
         g.ld_col < (long long)g.k * g.k * g.C || (g.ld_col & 7);
}
constexpr long long PATCH_32BIT = 1LL << 31;       // chunks of a row, rows of a launch
// images whose rows one launch can count
int patch_images(int rows_per_image) { return (int)((PATCH_32BIT - 1) / rows_per_image); }
dim3 patch_grid(long long chunks_per_row, int per_block, long long rows) {
  return dim3((unsigned)((chunks_per_row + per_block - 1) / per_block), (unsigned)(rows < 65535 ? rows : 65535));
}

}  // namespace

extern "C" int bb_im2col_nhwc(const void* x, void* col, int N, int H, int W, int C, int k, int stride, int pad, int Ho, int Wo,
                              long long ld_col, void* stream) {
  const ConvGeom g = {N, H, W, C, k, stride, pad, Ho, Wo, ld_col};
  if (!x || !col || bad_geom(g) || ((uintptr_t)x & 15) || ((uintptr_t)col & 15)) {
    bb_set_last_error_msg("bb_im2col_nhwc: null/unaligned pointer or inconsistent geometry (channels and ld_col multiples of 8)");
    return BB_ERR_INVALID_ARG;
  }
  if (Ho <= 0 || Wo <= 0) return BB_OK;        // a window larger than the padded image: no patches
  const int chunks = C >> 3;
  const long long row_chunks = (long long)k * k * chunks, total = Wo * row_chunks;
  const bool small = total < PATCH_32BIT;
  const ConvMagic m = {small ? bb_div_magic((int)row_chunks) : 0, bb_div_magic(chunks), bb_div_magic(k), bb_div_magic(Ho)};
  auto kernel = small ? im2col_kernel<unsigned> : im2col_kernel<unsigned long long>;
  const int per = patch_images(Ho);
  for (long long n = 0; n < N; n += per) {
    ConvGeom part = g;
    part.N = (int)(N - n < per ? N - n : per);
    bb_launch(kernel, patch_grid(total, 256 * PATCH_U, (long long)part.N * Ho), 256, 0, (cudaStream_t)stream,
              (const uint4*)x + n * H * W * chunks, (uint4*)col + n * Ho * Wo * (ld_col >> 3), part, m);
    BB_CUDA_CHECK(cudaGetLastError());
  }
  return BB_OK;
}

extern "C" int bb_col2im_nhwc(const void* dcol, void* dx, int N, int H, int W, int C, int k, int stride, int pad, int Ho, int Wo,
                              long long ld_col, void* stream) {
  const ConvGeom g = {N, H, W, C, k, stride, pad, Ho, Wo, ld_col};
  if (!dcol || !dx || bad_geom(g) || ((uintptr_t)dcol & 15) || ((uintptr_t)dx & 15)) {
    bb_set_last_error_msg("bb_col2im_nhwc: null/unaligned pointer or inconsistent geometry (channels and ld_col multiples of 8)");
    return BB_ERR_INVALID_ARG;
  }
  const int chunks = C >> 3;
  const long long total = (long long)W * chunks, windows = Ho > 0 && Wo > 0 ? (long long)Ho * Wo : 0;
  const ConvMagic m = {0, bb_div_magic(chunks), 0, bb_div_magic(H)};
  const bool small = total < PATCH_32BIT;
  const int taps = (k + stride - 1) / stride;
  void (*by_taps)(const uint4*, uint4*, const ConvGeom, const ConvMagic, unsigned) = nullptr;
  if (small && stride <= 2 && taps <= 4) {
    static decltype(by_taps) const kernels[2][4] = {
        {col2im_taps_kernel<unsigned, 1, 1>, col2im_taps_kernel<unsigned, 1, 2>, col2im_taps_kernel<unsigned, 1, 3>, col2im_taps_kernel<unsigned, 1, 4>},
        {col2im_taps_kernel<unsigned, 2, 1>, col2im_taps_kernel<unsigned, 2, 2>, col2im_taps_kernel<unsigned, 2, 3>, col2im_taps_kernel<unsigned, 2, 4>}};
    by_taps = kernels[stride - 1][taps - 1];
  }
  auto kernel = small ? col2im_kernel<unsigned> : col2im_kernel<unsigned long long>;
  const int per = patch_images(H);
  for (long long n = 0; n < N; n += per) {
    ConvGeom part = g;
    part.N = (int)(N - n < per ? N - n : per);
    const uint4* src = (const uint4*)dcol + n * windows * (ld_col >> 3);
    uint4* dst = (uint4*)dx + n * H * W * chunks;
    if (by_taps) {
      // rows per thread: up to eight while the grid still has sixteen blocks for every SM
      const long long image_rows = (long long)part.N * H, blocks = (total + 255) / 256 * image_rows;
      long long rows = blocks / (16LL * bb_num_sms());
      rows = rows < 1 ? 1 : rows > 8 ? 8 : rows;
      bb_launch(by_taps, patch_grid(total, 256, (image_rows + rows - 1) / rows), 256, 0, (cudaStream_t)stream, src, dst, part, m, (unsigned)rows);
    } else {
      bb_launch(kernel, patch_grid(total, 256, (long long)part.N * H), 256, 0, (cudaStream_t)stream, src, dst, part, m);
    }
    BB_CUDA_CHECK(cudaGetLastError());
  }
  return BB_OK;
}

// ---------------------------------------------------------------------------------- batch norm
namespace {

// Per-channel sums over the rows of a [rows, C] bf16 matrix, two quantities at a time.  Thread g
// owns channel chunk g % chunks (chunks = C / 8 divides 256) and walks rows g / chunks,
// + threads / chunks, ...; a block combines its threads through shared memory and writes one
// partial row [2, C] to the workspace; bn_finish_* adds the partial rows in block order.
enum { RED_STATS = 0, RED_BWD = 1 };

// HBM-bound (L2-bound for small layers): what counts is bytes and loads in flight.  Four rows (two in the backward
// element-wise pass) are requested per thread before the first is used, and without a residual the mask comes from
// y.  Image-network step (7 bottlenecks, 224 x 224, 2 x 32 images), all passes: reductions 1292 -> 1143 us,
// element-wise 1305 -> 975 us.
// Where the backward pass takes the ReLU mask from: nowhere, the stored output z > 0, or (no residual was added) the
// normalised value itself, computed again from y with the forward pass's own arithmetic and the scale and shift that the
// forward pass kept (gamma and beta may have changed since) - one tensor less to read.
enum { MASK_NONE = 0, MASK_Z = 1, MASK_Y = 2 };
constexpr int BN_U = 4;              // rows in flight per thread
constexpr int BN_CTAS = 3;           // blocks per SM (at most 85 registers a thread): the grid is one full wave

// z = relu(y * sc + sh), in the same operations wherever it is evaluated
__device__ __forceinline__ void bn_scale_shift(float gamma, float beta, float mean, float rstd, float& sc, float& sh) {
  sc = __fmul_rn(gamma, rstd);
  sh = __fmaf_rn(-mean, sc, beta);
}
// bf16(v) > 0: half the smallest bf16 number and everything below rounds to zero
__device__ __forceinline__ bool bn_positive(float v) { return v > 4.5917748e-41f; }

template <int MODE, int MASK>
__global__ void __launch_bounds__(256, BN_CTAS)
bn_reduce_kernel(const uint4* a, const uint4* zz, const uint4* yy,
                 const float* mean, const float* rstd, const float* affine, long long rows, int C, float* __restrict__ ws) {
  bb::pdl_sync();
  __shared__ float sm[256 * 16];
  const int chunks = C >> 3;
  const long long gthreads = (long long)gridDim.x * blockDim.x;
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int cc = (int)(g % chunks);
  const long long row_step = gthreads / chunks;
  float s1[8], s2[8], mu[8], rs[8], sc[8], sh[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) { s1[i] = 0.f; s2[i] = 0.f; mu[i] = 0.f; rs[i] = 0.f; }
  if (MODE == RED_BWD) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      mu[i] = __ldca(mean + cc * 8 + i); rs[i] = __ldca(rstd + cc * 8 + i);
      if (MASK == MASK_Y) { sc[i] = __ldca(affine + cc * 8 + i); sh[i] = __ldca(affine + C + cc * 8 + i); }
    }
  }
  const uint4 zero = make_uint4(0, 0, 0, 0);
  for (long long r = g / chunks; r < rows; r += BN_U * row_step) {
    // all of an iteration's operands are requested before the first is used; rows past the end add zeros
    uint4 qa[BN_U], qy[BN_U], qz[BN_U];
#pragma unroll
    for (int u = 0; u < BN_U; ++u) {
      const long long ru = r + u * row_step;
      const bool in = ru < rows;
      qa[u] = in ? __ldca(a + ru * chunks + cc) : zero;
      if (MODE == RED_BWD) qy[u] = in ? __ldca(yy + ru * chunks + cc) : zero;
      if (MASK == MASK_Z) qz[u] = in ? __ldca(zz + ru * chunks + cc) : zero;
    }
#pragma unroll
    for (int u = 0; u < BN_U; ++u) {
      float v[8];
      unpack8(qa[u], v);
      if (MODE == RED_STATS) {
#pragma unroll
        for (int i = 0; i < 8; ++i) { s1[i] += v[i]; s2[i] += v[i] * v[i]; }
      } else {
        float y[8];
        unpack8(qy[u], y);
        if (MASK == MASK_Z) {
          float z[8];
          unpack8(qz[u], z);
#pragma unroll
          for (int i = 0; i < 8; ++i) if (!(z[i] > 0.f)) v[i] = 0.f;
        } else if (MASK == MASK_Y) {
#pragma unroll
          for (int i = 0; i < 8; ++i) if (!bn_positive(__fmaf_rn(y[i], sc[i], sh[i]))) v[i] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) { s1[i] += v[i]; s2[i] += v[i] * ((y[i] - mu[i]) * rs[i]); }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) { sm[threadIdx.x * 16 + i] = s1[i]; sm[threadIdx.x * 16 + 8 + i] = s2[i]; }
  __syncthreads();
  // 256 % chunks == 0: the chunk of thread t is (blockIdx.x * 256 + t) % chunks = t % chunks
  if ((int)threadIdx.x < chunks) {
    float t1[8], t2[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { t1[i] = 0.f; t2[i] = 0.f; }
    for (int j = threadIdx.x; j < 256; j += chunks) {
#pragma unroll
      for (int i = 0; i < 8; ++i) { t1[i] += sm[j * 16 + i]; t2[i] += sm[j * 16 + 8 + i]; }
    }
    float* out = ws + (long long)blockIdx.x * 2 * C;
#pragma unroll
    for (int i = 0; i < 8; ++i) { out[threadIdx.x * 8 + i] = t1[i]; out[C + threadIdx.x * 8 + i] = t2[i]; }
  }
}

// Column sums over the partial rows: a block owns 32 channels and splits the rows over its 32 warps
// (coalesced 128-byte reads, four rows in flight per warp), then adds the warps' sums in warp order, so
// the result does not depend on scheduling.  A thread per channel walking all partial rows (up to BN_CTAS per SM) is
// a chain of that many L2 latencies: 26-28 us per call at 592 rows (four blocks per SM), against about 3 us this way.
// Valid in warp 0 only: t1, t2 of channel blockIdx.x * 32 + lane.
__device__ __forceinline__ void bn_sum_partials(const float* ws, int parts, int C, float& t1, float& t2) {
  __shared__ float sm1[32][33], sm2[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s1 = 0.f, s2 = 0.f;
  if (c < C) {
    int p = w;
    for (; p + 96 < parts; p += 128) {
      float a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float* row = ws + (long long)(p + 32 * u) * 2 * C + c;
        a[u] = __ldca(row); b[u] = __ldca(row + C);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) { s1 += a[u]; s2 += b[u]; }
    }
    for (; p < parts; p += 32) { const float* row = ws + (long long)p * 2 * C + c; s1 += __ldca(row); s2 += __ldca(row + C); }
  }
  sm1[w][lane] = s1; sm2[w][lane] = s2;
  __syncthreads();
  t1 = 0.f; t2 = 0.f;
  if (w == 0) {
#pragma unroll
    for (int j = 0; j < 32; ++j) { t1 += sm1[j][lane]; t2 += sm2[j][lane]; }
  }
}

// mean / rstd per channel from the partial rows (biased variance, as batch norm normalises with); affine (or null):
// scale and shift of the normalisation, [2, C]
__global__ void __launch_bounds__(1024)
bn_finish_stats_kernel(const float* ws, int parts, int C, float inv_rows, float eps, const __nv_bfloat16* __restrict__ gamma,
                       const __nv_bfloat16* __restrict__ beta, float* __restrict__ mean, float* __restrict__ rstd,
                       float* __restrict__ affine) {
  bb::pdl_sync();
  float s1, s2;
  bn_sum_partials(ws, parts, C, s1, s2);
  const int c = blockIdx.x * 32 + threadIdx.x;
  if (threadIdx.x >= 32 || c >= C) return;
  const float m = s1 * inv_rows;
  const float var = fmaxf(s2 * inv_rows - m * m, 0.f);
  const float rs = rsqrtf(var + eps);
  mean[c] = m;
  rstd[c] = rs;
  if (affine) {
    float sc, sh;
    bn_scale_shift(__bfloat162float(gamma[c]), __bfloat162float(beta[c]), m, rs, sc, sh);
    affine[c] = sc; affine[C + c] = sh;
  }
}

// sums[0][c] = sum dz', sums[1][c] = sum dz' * yhat; dbeta += sums[0], dgamma += sums[1]
__global__ void __launch_bounds__(1024)
bn_finish_bwd_kernel(const float* ws, int parts, int C, float* __restrict__ sums,
                     float* dgamma, float* dbeta) {
  bb::pdl_sync();
  float s1, s2;
  bn_sum_partials(ws, parts, C, s1, s2);
  const int c = blockIdx.x * 32 + threadIdx.x;
  if (threadIdx.x >= 32 || c >= C) return;
  sums[c] = s1; sums[C + c] = s2;
  dbeta[c] += s1; dgamma[c] += s2;
}

// The element-wise passes walk the rows from the last to the first: the reduction in front of them read them in
// ascending order, so the rows it read last are the ones still in L2.
// z = (y - mean) * rstd * gamma + beta (+ residual) (ReLU)
template <bool RES>
__global__ void __launch_bounds__(256, BN_CTAS)
bn_apply_kernel(const uint4* y, const float* mean, const float* rstd,
                const __nv_bfloat16* __restrict__ gamma, const __nv_bfloat16* __restrict__ beta,
                const uint4* residual, uint4* __restrict__ z, long long rows, int C, int relu) {
  bb::pdl_sync();
  const int chunks = C >> 3;
  const long long gthreads = (long long)gridDim.x * blockDim.x;
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int cc = (int)(g % chunks);
  const long long row_step = gthreads / chunks;
  float sc[8], sh[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    bn_scale_shift(__bfloat162float(gamma[cc * 8 + i]), __bfloat162float(beta[cc * 8 + i]), __ldca(mean + cc * 8 + i),
                   __ldca(rstd + cc * 8 + i), sc[i], sh[i]);
  for (long long r = rows - 1 - g / chunks; r >= 0; r -= BN_U * row_step) {
    uint4 qy[BN_U], qr[BN_U];
#pragma unroll
    for (int u = 0; u < BN_U; ++u) {
      const long long ru = r - u * row_step;
      if (ru >= 0) { qy[u] = __ldca(y + ru * chunks + cc); if (RES) qr[u] = __ldca(residual + ru * chunks + cc); }
    }
#pragma unroll
    for (int u = 0; u < BN_U; ++u) {
      const long long ru = r - u * row_step;
      if (ru < 0) break;
      float v[8];
      unpack8(qy[u], v);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __fmaf_rn(v[i], sc[i], sh[i]);
      if (RES) {
        float rr[8];
        unpack8(qr[u], rr);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += rr[i];
      }
      if (relu) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = fmaxf(v[i], 0.f);
      }
      z[ru * chunks + cc] = pack8(v);
    }
  }
}

// dy = gamma * rstd * (dz' - s1 / rows - yhat * s2 / rows); dres = dz' (the masked gradient that
// also flows into the residual branch)
template <int MASK>
__global__ void __launch_bounds__(256, BN_CTAS)
bn_bwd_apply_kernel(const uint4* dz, const uint4* zz, const uint4* yy,
                    const float* mean, const float* rstd, const __nv_bfloat16* __restrict__ gamma,
                    const float* affine, const float* sums, uint4* __restrict__ dy,
                    uint4* __restrict__ dres, long long rows, int C, float inv_rows) {
  bb::pdl_sync();
  constexpr int U = 2;         // four rows would take 128 registers
  const int chunks = C >> 3;
  const long long gthreads = (long long)gridDim.x * blockDim.x;
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int cc = (int)(g % chunks);
  const long long row_step = gthreads / chunks;
  // s1 / rows + yhat * s2 / rows = y * k2 + k1
  float k0[8], k1[8], k2[8], sc[8], sh[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float rs = __ldca(rstd + cc * 8 + i), ga = __bfloat162float(gamma[cc * 8 + i]), mu = __ldca(mean + cc * 8 + i);
    k0[i] = ga * rs;
    k2[i] = rs * (__ldca(sums + C + cc * 8 + i) * inv_rows);
    k1[i] = fmaf(-mu, k2[i], __ldca(sums + cc * 8 + i) * inv_rows);
    if (MASK == MASK_Y) { sc[i] = __ldca(affine + cc * 8 + i); sh[i] = __ldca(affine + C + cc * 8 + i); }
  }
  for (long long r = rows - 1 - g / chunks; r >= 0; r -= U * row_step) {
    uint4 qd[U], qy[U], qz[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long ru = r - u * row_step;
      if (ru >= 0) {
        qd[u] = __ldca(dz + ru * chunks + cc);
        qy[u] = __ldca(yy + ru * chunks + cc);
        if (MASK == MASK_Z) qz[u] = __ldca(zz + ru * chunks + cc);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long ru = r - u * row_step;
      if (ru < 0) break;
      float v[8], y[8];
      unpack8(qd[u], v);
      unpack8(qy[u], y);
      if (MASK == MASK_Z) {
        float z[8];
        unpack8(qz[u], z);
#pragma unroll
        for (int i = 0; i < 8; ++i) if (!(z[i] > 0.f)) v[i] = 0.f;
      } else if (MASK == MASK_Y) {
#pragma unroll
        for (int i = 0; i < 8; ++i) if (!bn_positive(__fmaf_rn(y[i], sc[i], sh[i]))) v[i] = 0.f;
      }
      if (dres) dres[ru * chunks + cc] = pack8(v);
      float o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = k0[i] * (v[i] - fmaf(y[i], k2[i], k1[i]));
      dy[ru * chunks + cc] = pack8(o);
    }
  }
}

bool bad_bn(long long rows, int C) { return rows <= 0 || C < 8 || (C & 7) || (256 % (C >> 3)) != 0; }

int bn_grid(long long rows, int C) {
  long long blocks = (rows * (C >> 3) + 256 * 8 - 1) / (256 * 8);
  const long long cap = (long long)bb_num_sms() * BN_CTAS;
  if (blocks > cap) blocks = cap;
  return (int)(blocks < 1 ? 1 : blocks);
}

// `affine`: the forward pass's scale and shift, non-null when the mask may come from y (no residual was added)
int bn_bwd(const void* dz, const void* z, const void* y, const float* mean, const float* rstd, const void* gamma, const float* affine,
           void* dy, void* dres, float* dgamma, float* dbeta, long long rows, int C, int relu, float* ws, cudaStream_t s) {
  const int grid = bn_grid(rows, C);
  float* sums = ws + (long long)grid * 2 * C;
  const uint4 *qd = (const uint4*)dz, *qz = (const uint4*)z, *qy = (const uint4*)y;
  const __nv_bfloat16* ga = (const __nv_bfloat16*)gamma;
  const float inv = 1.0f / (float)rows;
#define BB_BN_BWD(MASK)                                                                                               \
  bb_launch(bn_reduce_kernel<RED_BWD, MASK>, grid, 256, 0, s, qd, qz, qy, mean, rstd, affine, rows, C, ws);                      \
  bb_launch(bn_finish_bwd_kernel, (C + 31) / 32, 1024, 0, s, ws, grid, C, sums, dgamma, dbeta);                             \
  bb_launch(bn_bwd_apply_kernel<MASK>, grid, 256, 0, s, qd, qz, qy, mean, rstd, ga, affine, sums, (uint4*)dy, (uint4*)dres, rows, C, inv)
  if (!relu) { BB_BN_BWD(MASK_NONE); }
  else if (affine) { BB_BN_BWD(MASK_Y); }
  else { BB_BN_BWD(MASK_Z); }
#undef BB_BN_BWD
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}

}  // namespace

extern "C" long long bb_bn_workspace_bytes(long long rows, int C) {
  if (bad_bn(rows, C)) return -1;
  // partial rows of the reduction plus the two per-channel sums the backward pass keeps
  return ((long long)bn_grid(rows, C) * 2 * C + 2 * C) * (long long)sizeof(float);
}

namespace {
// `affine` (or null): filled with the scale and shift that gamma and beta give with these statistics
int bn_stats(const void* y, long long rows, int C, float eps, float* mean, float* rstd, const void* gamma, const void* beta,
             float* affine, void* workspace, long long workspace_bytes, void* stream) {
  if (!y || !mean || !rstd || !workspace || bad_bn(rows, C) || workspace_bytes < bb_bn_workspace_bytes(rows, C) ||
      ((uintptr_t)y & 15)) {
    bb_set_last_error_msg("bb_bn_stats: null/unaligned pointer, workspace too small, or channels not 8 x a power of two <= 2048");
    return BB_ERR_INVALID_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int grid = bn_grid(rows, C);
  float* ws = static_cast<float*>(workspace);
  bb_launch(bn_reduce_kernel<RED_STATS, MASK_NONE>, grid, 256, 0, s, (const uint4*)y, nullptr, nullptr, nullptr, nullptr, nullptr, rows, C, ws);
  bb_launch(bn_finish_stats_kernel, (C + 31) / 32, 1024, 0, s, ws, grid, C, 1.0f / (float)rows, eps, (const __nv_bfloat16*)gamma,
            (const __nv_bfloat16*)beta, mean, rstd, affine);
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}
}  // namespace

extern "C" int bb_bn_stats(const void* y, long long rows, int C, float eps, float* mean, float* rstd, void* workspace,
                           long long workspace_bytes, void* stream) {
  return bn_stats(y, rows, C, eps, mean, rstd, nullptr, nullptr, nullptr, workspace, workspace_bytes, stream);
}

extern "C" int bb_bn_apply(const void* y, const float* mean, const float* rstd, const void* gamma, const void* beta,
                           const void* residual, void* z, long long rows, int C, int relu, void* stream) {
  if (!y || !mean || !rstd || !gamma || !beta || !z || bad_bn(rows, C) || ((uintptr_t)y & 15) || ((uintptr_t)z & 15) ||
      ((uintptr_t)residual & 15)) {
    bb_set_last_error_msg("bb_bn_apply: null/unaligned pointer or channels not 8 x a power of two <= 2048");
    return BB_ERR_INVALID_ARG;
  }
  auto kernel = residual ? bn_apply_kernel<true> : bn_apply_kernel<false>;
  bb_launch(kernel, bn_grid(rows, C), 256, 0, (cudaStream_t)stream, (const uint4*)y, mean, rstd, (const __nv_bfloat16*)gamma,
                                                             (const __nv_bfloat16*)beta, (const uint4*)residual, (uint4*)z, rows, C, relu);
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}

extern "C" int bb_bn_bwd(const void* dz, const void* z, const void* y, const float* mean, const float* rstd, const void* gamma,
                         void* dy, void* dres, float* dgamma, float* dbeta, long long rows, int C, int relu, void* workspace,
                         long long workspace_bytes, void* stream) {
  if (!dz || !y || !mean || !rstd || !gamma || !dy || !dgamma || !dbeta || !workspace || (relu && !z) || bad_bn(rows, C) ||
      workspace_bytes < bb_bn_workspace_bytes(rows, C) ||
      (((uintptr_t)dz | (uintptr_t)z | (uintptr_t)y | (uintptr_t)dy | (uintptr_t)dres) & 15)) {
    bb_set_last_error_msg("bb_bn_bwd: null/unaligned pointer, workspace too small, or channels not 8 x a power of two <= 2048");
    return BB_ERR_INVALID_ARG;
  }
  return bn_bwd(dz, z, y, mean, rstd, gamma, nullptr, dy, dres, dgamma, dbeta, rows, C, relu, static_cast<float*>(workspace),
                (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------- pooling
namespace {

// (chunk, column, row, image) of flat element e of an [N, rows, cols, chunks] tensor.  SMALL: fewer than 2^31 elements, by
// multiplication (see bb_div_magic).
struct PoolMagic { unsigned long long chunks, cols, rows; };
template <bool SMALL>
__device__ __forceinline__ void pool_coords(long long e, int chunks, int cols, int rows, const PoolMagic& m, int& cc, int& x, int& y, int& n) {
  if constexpr (SMALL) {
    const unsigned p = bb::fast_div((unsigned)e, m.chunks), t = bb::fast_div(p, m.cols), i = bb::fast_div(t, m.rows);
    cc = (int)((unsigned)e - p * chunks); x = (int)(p - t * cols); y = (int)(t - i * rows); n = (int)i;
  } else {
    const long long p = e / chunks, t = p / cols;
    cc = (int)(e % chunks); x = (int)(p % cols); y = (int)(t % rows); n = (int)(t / rows);
  }
}

// 3 x 3 window, stride 2, padding 1.  The position of the maximum inside the window (0..8, first
// one in row-major window order wins a tie, like the framework's scan) is kept per output
// element, so the backward pass routes the gradient to exactly that input.
template <bool SMALL>
__global__ void __launch_bounds__(256)
maxpool_fwd_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, uint2* __restrict__ argmax, int N, int H, int W, int C,
                   int Ho, int Wo, const PoolMagic m) {
  const int chunks = C >> 3;
  const long long total = (long long)N * Ho * Wo * chunks;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    int cc, wo, ho, n;
    pool_coords<SMALL>(e, chunks, Wo, Ho, m, cc, wo, ho, n);
    float best[8];
    unsigned int where[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { best[i] = -INFINITY; where[i] = 0; }
    for (int r = 0; r < 3; ++r) {
      const int h = 2 * ho - 1 + r;
      if (h < 0 || h >= H) continue;
      for (int s = 0; s < 3; ++s) {
        const int w = 2 * wo - 1 + s;
        if (w < 0 || w >= W) continue;
        float v[8];
        unpack8(__ldg(x + (((long long)n * H + h) * W + w) * chunks + cc), v);
#pragma unroll
        for (int i = 0; i < 8; ++i) if (v[i] > best[i] || best[i] == -INFINITY) { best[i] = v[i]; where[i] = r * 3 + s; }
      }
    }
    y[e] = pack8(best);
    uint2 a;
    a.x = where[0] | (where[1] << 8) | (where[2] << 16) | (where[3] << 24);
    a.y = where[4] | (where[5] << 8) | (where[6] << 16) | (where[7] << 24);
    argmax[e] = a;
  }
}

// A pixel lies in one window of a dimension (tap 1) or in two (taps 0 and 2): up to four windows, all requested before the
// first is used, added in tap order.  With three 64-bit divisions per 16-byte result and a chain of loads 32 x 112 x 112 x 64
// took 50 us for its 70 MB, now 42.
template <bool SMALL>
__global__ void __launch_bounds__(256)
maxpool_bwd_kernel(const uint4* __restrict__ dy, const uint2* __restrict__ argmax, uint4* __restrict__ dx, int N, int H, int W,
                   int C, int Ho, int Wo, const PoolMagic m) {
  const int chunks = C >> 3;
  const long long total = (long long)N * H * W * chunks;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    int cc, w, h, n;
    pool_coords<SMALL>(e, chunks, W, H, m, cc, w, h, n);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    uint2 a[4];
    uint4 q[4];
    unsigned tap[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = ((h + 1) & 1) + (u >> 1) * 2, s = ((w + 1) & 1) + (u & 1) * 2;
      const int ho = (h + 1 - r) >> 1, wo = (w + 1 - s) >> 1;
      const bool in = r < 3 && s < 3 && ho >= 0 && ho < Ho && wo >= 0 && wo < Wo;
      const long long o = (((long long)n * Ho + ho) * Wo + wo) * chunks + cc;
      tap[u] = in ? (unsigned)(r * 3 + s) : 0x100u;          // no byte of argmax
      a[u] = in ? __ldg(argmax + o) : make_uint2(0, 0);
      q[u] = in ? __ldg(dy + o) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float g[8];
      unpack8(q[u], g);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned int wi = ((i < 4 ? a[u].x : a[u].y) >> (8 * (i & 3))) & 0xFFu;
        if (wi == tap[u]) acc[i] += g[i];
      }
    }
    dx[e] = pack8(acc);
  }
}

// y[n, c] = mean over the hw pixels of x[n, :, c]
__global__ void __launch_bounds__(256)
avgpool_fwd_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, int N, int HW, int C) {
  const int chunks = C >> 3;
  const long long total = (long long)N * chunks;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int cc = (int)(e % chunks), n = (int)(e / chunks);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int p = 0; p < HW; ++p) {
      float v[8];
      unpack8(__ldg(x + ((long long)n * HW + p) * chunks + cc), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += v[i];
    }
    const float inv = 1.0f / (float)HW;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] *= inv;
    y[e] = pack8(acc);
  }
}

__global__ void __launch_bounds__(256)
avgpool_bwd_kernel(const uint4* __restrict__ dy, uint4* __restrict__ dx, int N, int HW, int C) {
  const int chunks = C >> 3;
  const long long total = (long long)N * HW * chunks;
  const float inv = 1.0f / (float)HW;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int cc = (int)(e % chunks);
    const int n = (int)(e / ((long long)HW * chunks));
    float v[8];
    unpack8(__ldg(dy + (long long)n * chunks + cc), v);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] *= inv;
    dx[e] = pack8(v);
  }
}

}  // namespace

extern "C" int bb_maxpool3x3s2_fwd(const void* x, void* y, void* argmax, int N, int H, int W, int C, void* stream) {
  const int Ho = (H + 2 - 3) / 2 + 1, Wo = (W + 2 - 3) / 2 + 1;
  if (!x || !y || !argmax || N <= 0 || H <= 0 || W <= 0 || C <= 0 || (C & 7) ||
      (((uintptr_t)x | (uintptr_t)y) & 15) || ((uintptr_t)argmax & 7)) {
    bb_set_last_error_msg("bb_maxpool3x3s2_fwd: null/unaligned pointer or channels not a multiple of 8");
    return BB_ERR_INVALID_ARG;
  }
  const long long total = (long long)N * Ho * Wo * (C >> 3);
  const PoolMagic m = {bb_div_magic(C >> 3), bb_div_magic(Wo), bb_div_magic(Ho)};
  auto kernel = total < (1LL << 31) ? maxpool_fwd_kernel<true> : maxpool_fwd_kernel<false>;
  kernel<<<flat_grid(total), 256, 0, (cudaStream_t)stream>>>((const uint4*)x, (uint4*)y, (uint2*)argmax, N, H, W, C, Ho, Wo, m);
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}

extern "C" int bb_maxpool3x3s2_bwd(const void* dy, const void* argmax, void* dx, int N, int H, int W, int C, void* stream) {
  const int Ho = (H + 2 - 3) / 2 + 1, Wo = (W + 2 - 3) / 2 + 1;
  if (!dy || !dx || !argmax || N <= 0 || H <= 0 || W <= 0 || C <= 0 || (C & 7) ||
      (((uintptr_t)dx | (uintptr_t)dy) & 15) || ((uintptr_t)argmax & 7)) {
    bb_set_last_error_msg("bb_maxpool3x3s2_bwd: null/unaligned pointer or channels not a multiple of 8");
    return BB_ERR_INVALID_ARG;
  }
  const long long total = (long long)N * H * W * (C >> 3);
  const PoolMagic m = {bb_div_magic(C >> 3), bb_div_magic(W), bb_div_magic(H)};
  auto kernel = total < (1LL << 31) ? maxpool_bwd_kernel<true> : maxpool_bwd_kernel<false>;
  kernel<<<flat_grid(total), 256, 0, (cudaStream_t)stream>>>((const uint4*)dy, (const uint2*)argmax, (uint4*)dx, N, H, W, C, Ho, Wo, m);
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}

extern "C" int bb_avgpool_fwd(const void* x, void* y, int N, int HW, int C, void* stream) {
  if (!x || !y || N <= 0 || HW <= 0 || C <= 0 || (C & 7) || (((uintptr_t)x | (uintptr_t)y) & 15)) {
    bb_set_last_error_msg("bb_avgpool_fwd: null/unaligned pointer or channels not a multiple of 8");
    return BB_ERR_INVALID_ARG;
  }
  avgpool_fwd_kernel<<<flat_grid((long long)N * (C >> 3)), 256, 0, (cudaStream_t)stream>>>((const uint4*)x, (uint4*)y, N, HW, C);
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}

extern "C" int bb_avgpool_bwd(const void* dy, void* dx, int N, int HW, int C, void* stream) {
  if (!dy || !dx || N <= 0 || HW <= 0 || C <= 0 || (C & 7) || (((uintptr_t)dx | (uintptr_t)dy) & 15)) {
    bb_set_last_error_msg("bb_avgpool_bwd: null/unaligned pointer or channels not a multiple of 8");
    return BB_ERR_INVALID_ARG;
  }
  avgpool_bwd_kernel<<<flat_grid((long long)N * HW * (C >> 3)), 256, 0, (cudaStream_t)stream>>>((const uint4*)dy, (uint4*)dx, N, HW, C);
  BB_CUDA_CHECK(cudaGetLastError());
  return BB_OK;
}

// ---------------------------------------------------------------------------------- one call per layer
// Convolution + batch norm (+ residual, + ReLU) forward and backward with every kernel issued from
// one foreign call: a ResNet-152 step has ~2500 such layers-times-micro-batches, and a Python host
// that pays per kernel becomes the bottleneck.  Where patches are stored: the same kernels in the same order as the entry
// points above called one by one.  Gathered products have no entry point of their own; an input gradient is then summed over
// all taps in fp32 and rounded once, not once per tap.
namespace {

inline long long up256(long long n) { return (n + 255) & ~255LL; }

struct ConvSizes {
  int Ho, Wo;
  long long P, K;
  bool direct;                       // 1 x 1 / stride 1 without padding: the activation tensor is the patch matrix
  // Patches gathered by the GEMM's own loads (bb_conv_gemm) instead of a stored patch matrix: needs 64-channel blocks.
  // Forward and weight gradient read windows of x, the input gradient windows of dy; with a stride the latter would
  // need dy spread out with zeros, so it keeps the patch-gradient matrix and its adjoint gather.  So does an input gradient
  // whose gathered product is expected to take longer: it has only Cin columns (a tile has 128 at least) and a reduction
  // of k * k * Cout, where the patch-gradient product has k * k * Cin columns and reduces over Cout.  Backward pass (us),
  // patch matrix / gathered: 8 -> 1024 channels, 7 x 7, 32 images of 56 x 56: 587 / 1776; 256 -> 1024, 7 x 7, 8 of 14 x 14
  // (8 output tiles): 153 / 348; 64 -> 64, 3 x 3, 32 of 56 x 56: 142 / 68; 256 -> 256, 3 x 3, 32 of 56 x 56: 437 / 243.
  // Few pixels and a long reduction split it over clusters, and the product is priced as it runs: 256 -> 1024, 7 x 7, 32 images
  // of 14 x 14 304 / 260, 512 -> 256, 7 x 7, one of 28 x 28 71 / 51, 64 -> 64, 7 x 7, 32 of 7 x 7 44 / 28, all gathered.
  // The adjoint gather is counted as 1.5 TB/s of patch matrix, the gathered product as 1.2 of its plan: over 130 layers (8 to 512
  // -> 64 to 1024 channels, windows 3 to 7, 98 to 166012 pixels) one is slower than with the patch matrix (44.0 / 46.7), and the pass
  // is within 4 % of the quicker route on average (5 % with the gathered product priced whole).
  // A 3 x 3 layer's patch matrix is nine times its input, written and read once per product: 128 channels, 32 images
  // of 28 x 28, forward + backward 181 -> 89 us of device time (gathers 80 us, GEMMs 63 -> 55 us) without it.
  bool implicit_x, implicit_dx;
  long long col_bytes, dy_bytes, dcol_bytes, bn_bytes;
};

bool conv_sizes(const bb_conv_desc* d, ConvSizes* s) {
  if (!d || d->N <= 0 || d->H <= 0 || d->W <= 0 || d->Cin <= 0 || (d->Cin & 7) || d->Cout <= 0 || d->k <= 0 || d->stride <= 0 ||
      d->pad < 0 || !d->w || !d->gamma || !d->beta)
    return false;
  s->Ho = (d->H + 2 * d->pad - d->k) / d->stride + 1;
  s->Wo = (d->W + 2 * d->pad - d->k) / d->stride + 1;
  if (s->Ho <= 0 || s->Wo <= 0) return false;
  s->P = (long long)d->N * s->Ho * s->Wo;
  s->K = (long long)d->k * d->k * d->Cin;
  s->direct = d->k == 1 && d->stride == 1 && d->pad == 0;
  // (with a stride, Ho = 1 also stands for a window that overhangs the padded image, which has no im2col box)
  s->implicit_x = !s->direct && bb_conv_gemm_supported(d->Cin, d->k, d->stride, d->pad) &&
                  (d->H < d->W ? d->H : d->W) + 2 * d->pad >= d->k;
  s->implicit_dx = !s->direct && d->stride == 1 && d->pad < d->k && bb_conv_gemm_supported(d->Cout, d->k, 1, d->k - 1 - d->pad) &&
                   1.2 * bb_gemm_store_us((long long)d->N * d->H * d->W, d->Cin, (long long)d->k * d->k * d->Cout, d->max_ctas) <
                       bb_gemm_store_us(s->P, s->K, d->Cout, d->max_ctas) + (double)s->P * s->K * 2 / 1.5e6;
  s->bn_bytes = bb_bn_workspace_bytes(s->P, d->Cout);
  if (s->bn_bytes < 0) return false;
  s->col_bytes = s->direct || s->implicit_x ? 0 : up256(s->P * s->K * 2);
  s->dy_bytes = up256(s->P * d->Cout * 2);
  s->dcol_bytes = s->direct || s->implicit_dx ? 0 : up256(s->P * s->K * 2);
  s->bn_bytes = up256(s->bn_bytes);
  return true;
}

int conv_gemm(const bb_conv_desc* d, int M, int N, int K, const void* A, long long lda, int a_mn, const void* B, long long ldb,
              int b_mn, void* D, long long ldd, int epi, void* stream) {
  bb_gemm_desc g = {};
  g.M = M; g.N = N; g.K = K; g.A = A; g.lda = lda; g.a_mn_major = a_mn; g.B = B; g.ldb = ldb; g.b_mn_major = b_mn;
  g.D = D; g.ldd = ldd; g.epilogue = epi; g.max_ctas = d->max_ctas;
  return bb_gemm_bf16(&g, stream);
}

// products over patches of x [N, H, W, Cin]
int conv_implicit(const bb_conv_desc* d, const ConvSizes& s, int mode, const void* x, const void* other, void* D, void* stream) {
  const bb_conv_gemm_args a = {mode, x, d->N, d->H, d->W, d->Cin, d->k, d->stride, d->pad, s.Ho, s.Wo, other, d->Cout, D, d->max_ctas};
  return bb_conv_gemm(&a, stream);
}
// dx: a stride-1 convolution over dy [N, Ho, Wo, Cout] with the window turned by 180 degrees and the complementary padding
int conv_implicit_dx(const bb_conv_desc* d, const ConvSizes& s, const void* dy, void* dx, void* stream) {
  const bb_conv_gemm_args a = {BB_CONV_DGRAD, dy, d->N, s.Ho, s.Wo, d->Cout, d->k, 1, d->k - 1 - d->pad, d->H, d->W,
                               d->w, d->Cin, dx, d->max_ctas};
  return bb_conv_gemm(&a, stream);
}

#define BB_TRY(expr) do { int _rc = (expr); if (_rc != BB_OK) return _rc; } while (0)

}  // namespace

extern "C" long long bb_conv_bn_scratch_bytes(const bb_conv_desc* d, int backward, int need_dx) {
  ConvSizes s;
  if (!conv_sizes(d, &s)) return -1;
  if (!backward) return s.col_bytes + s.bn_bytes;
  return s.dy_bytes + s.col_bytes + (need_dx ? s.dcol_bytes : 0) + s.bn_bytes;
}

extern "C" int bb_conv_bn_launches(const bb_conv_desc* d, int backward, int need_dx) {
  ConvSizes s;
  if (!conv_sizes(d, &s)) return -1;
  // the product with the input's patches (and their gather), three passes of batch norm; the input gradient (and its adjoint gather)
  int n = 4 + (s.direct || s.implicit_x ? 0 : 1);
  if (backward && need_dx) n += s.direct || s.implicit_dx ? 1 : 2;
  return n;
}

namespace {
int conv_bn_fwd(const bb_conv_desc* d, const void* x, const void* residual, void* y, void* z, float* mean, float* rstd, float* affine,
                void* scratch, long long scratch_bytes, void* stream) {
  ConvSizes s;
  if (!conv_sizes(d, &s) || !x || !y || !z || !mean || !rstd || !scratch || scratch_bytes < s.col_bytes + s.bn_bytes) {
    bb_set_last_error_msg("bb_conv_bn_fwd: bad descriptor, null buffer or scratch smaller than bb_conv_bn_scratch_bytes");
    return BB_ERR_INVALID_ARG;
  }
  const BackToBack scope(d->max_ctas == 0);
  uint8_t* sc = static_cast<uint8_t*>(scratch);
  if (s.implicit_x) {
    BB_TRY(conv_implicit(d, s, BB_CONV_FWD, x, d->w, y, stream));
  } else {
    const void* col = x;
    if (!s.direct) {
      BB_TRY(bb_im2col_nhwc(x, sc, d->N, d->H, d->W, d->Cin, d->k, d->stride, d->pad, s.Ho, s.Wo, s.K, stream));
      col = sc;
    }
    BB_TRY(conv_gemm(d, (int)s.P, d->Cout, (int)s.K, col, s.K, 0, d->w, s.K, 0, y, d->Cout, BB_EPI_STORE, stream));
  }
  BB_TRY(bn_stats(y, s.P, d->Cout, d->eps, mean, rstd, d->gamma, d->beta, affine, sc + s.col_bytes, s.bn_bytes, stream));
  BB_TRY(bb_bn_apply(y, mean, rstd, d->gamma, d->beta, residual, z, s.P, d->Cout, d->relu, stream));
  return BB_OK;
}

// the ReLU mask comes from y and affine, or from z when affine is null
int conv_bn_bwd(const bb_conv_desc* d, const void* x, const void* y, const void* z, const float* mean, const float* rstd,
                const float* affine, const void* dz, void* dx, void* dres, void* scratch, long long scratch_bytes, void* stream) {
  ConvSizes s;
  if (!conv_sizes(d, &s) || !x || !y || (!z && !affine) || !mean || !rstd || !dz || !scratch || !d->g_w || !d->g_gamma || !d->g_beta ||
      scratch_bytes < bb_conv_bn_scratch_bytes(d, 1, dx != nullptr)) {
    bb_set_last_error_msg("bb_conv_bn_bwd: bad descriptor, null buffer, missing gradient pointer or scratch too small");
    return BB_ERR_INVALID_ARG;
  }
  const BackToBack scope(d->max_ctas == 0);
  uint8_t* sc = static_cast<uint8_t*>(scratch);
  void* dy = sc;
  uint8_t* colbuf = sc + s.dy_bytes;
  uint8_t* dcolbuf = colbuf + s.col_bytes;
  uint8_t* bnws = dcolbuf + (dx ? s.dcol_bytes : 0);
  if ((((uintptr_t)dz | (uintptr_t)z | (uintptr_t)y | (uintptr_t)dy | (uintptr_t)dres) & 15)) {
    bb_set_last_error_msg("bb_conv_bn_bwd: activations must be 16-byte aligned");
    return BB_ERR_INVALID_ARG;
  }
  BB_TRY(bn_bwd(dz, z, y, mean, rstd, d->gamma, affine, dy, dres, d->g_gamma, d->g_beta, s.P, d->Cout, d->relu,
                reinterpret_cast<float*>(bnws), (cudaStream_t)stream));
  // dW[Cout, K] += dy^T patches
  if (s.implicit_x) {
    BB_TRY(conv_implicit(d, s, BB_CONV_WGRAD, x, dy, d->g_w, stream));
  } else {
    const void* col = x;
    if (!s.direct) {
      BB_TRY(bb_im2col_nhwc(x, colbuf, d->N, d->H, d->W, d->Cin, d->k, d->stride, d->pad, s.Ho, s.Wo, s.K, stream));
      col = colbuf;
    }
    BB_TRY(conv_gemm(d, d->Cout, (int)s.K, (int)s.P, dy, d->Cout, 1, col, s.K, 1, d->g_w, s.K, BB_EPI_ACCUM_F32, stream));
  }
  if (dx) {
    if (s.implicit_dx) {
      BB_TRY(conv_implicit_dx(d, s, dy, dx, stream));
    } else {
      void* dcol = s.direct ? dx : (void*)dcolbuf;
      BB_TRY(conv_gemm(d, (int)s.P, (int)s.K, d->Cout, dy, d->Cout, 0, d->w, s.K, 1, dcol, s.K, BB_EPI_STORE, stream));
      if (!s.direct)
        BB_TRY(bb_col2im_nhwc(dcol, dx, d->N, d->H, d->W, d->Cin, d->k, d->stride, d->pad, s.Ho, s.Wo, s.K, stream));
    }
  }
  return BB_OK;
}
}  // namespace

extern "C" int bb_conv_bn_fwd(const bb_conv_desc* d, const void* x, const void* residual, void* y, void* z, float* mean,
                              float* rstd, void* scratch, long long scratch_bytes, void* stream) {
  return conv_bn_fwd(d, x, residual, y, z, mean, rstd, nullptr, scratch, scratch_bytes, stream);
}

extern "C" int bb_conv_bn_bwd(const bb_conv_desc* d, const void* x, const void* y, const void* z, const float* mean,
                              const float* rstd, const void* dz, void* dx, void* dres, void* scratch, long long scratch_bytes,
                              void* stream) {
  return conv_bn_bwd(d, x, y, z, mean, rstd, nullptr, dz, dx, dres, scratch, scratch_bytes, stream);
}

extern "C" int bb_conv_bn_bwd_no_residual(const bb_conv_desc* d, const void* x, const void* y, const void* z, const float* mean,
                                          const float* rstd, const void* dz, void* dx, void* scratch, long long scratch_bytes,
                                          void* stream) {
  return conv_bn_bwd(d, x, y, z, mean, rstd, nullptr, dz, dx, nullptr, scratch, scratch_bytes, stream);
}

extern "C" int bb_conv_bn_fwd_affine(const bb_conv_desc* d, const void* x, void* y, void* z, float* mean, float* rstd, float* affine,
                                     void* scratch, long long scratch_bytes, void* stream) {
  if (!affine) { bb_set_last_error_msg("bb_conv_bn_fwd_affine: null affine"); return BB_ERR_INVALID_ARG; }
  return conv_bn_fwd(d, x, nullptr, y, z, mean, rstd, affine, scratch, scratch_bytes, stream);
}

extern "C" int bb_conv_bn_bwd_affine(const bb_conv_desc* d, const void* x, const void* y, const float* mean, const float* rstd,
                                     const float* affine, const void* dz, void* dx, void* scratch, long long scratch_bytes,
                                     void* stream) {
  if (!affine) { bb_set_last_error_msg("bb_conv_bn_bwd_affine: null affine"); return BB_ERR_INVALID_ARG; }
  return conv_bn_bwd(d, x, y, nullptr, mean, rstd, affine, dz, dx, nullptr, scratch, scratch_bytes, stream);
}
