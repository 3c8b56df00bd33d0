// Shared device helpers for the sm_100a kernels: status codes, bounded mbarrier waits,
// TMA / tcgen05 / TMEM instruction wrappers.  Every spin in this library is bounded: a
// wait that runs out records a status word and the kernel drains and returns.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "bamboo_b200.h"

// Upper bound for any in-kernel wait (nanoseconds of %globaltimer).
#ifndef BB_WAIT_LIMIT_NS
#define BB_WAIT_LIMIT_NS 2000000000ull
#endif

#define BB_CUDA_CHECK(expr)                                   \
  do {                                                        \
    cudaError_t _e = (expr);                                  \
    if (_e != cudaSuccess) {                                  \
      bb_set_last_error(#expr, _e);                           \
      return BB_ERR_CUDA;                                     \
    }                                                         \
  } while (0)

void bb_set_last_error(const char* what, cudaError_t e);
void bb_set_last_error_msg(const char* msg);
// Device word that kernels write when a bounded wait expires (0 = healthy).
int* bb_device_status_word();
int bb_num_sms();
// Index of the current device, or -1 when it cannot be read or is beyond the per-device tables.
int bb_current_device();

// Function attributes (the dynamic shared-memory limit) are per device: `body` runs the first
// time the enclosing call site is reached on each device of the process.  `body` may return
// from the enclosing function on error; the device is then not marked as done.
#define BB_ONCE_PER_DEVICE(body)                          \
  do {                                                    \
    static unsigned char _bb_done[64];                    \
    const int _bb_dev = bb_current_device();              \
    if (_bb_dev < 0 || !_bb_done[_bb_dev]) {              \
      body;                                               \
      if (_bb_dev >= 0) _bb_done[_bb_dev] = 1;            \
    }                                                     \
  } while (0)

// Kernels that one entry point issues back to back (half a transformer block, a convolution layer) are launched so that
// each may become resident while the kernel in front of it in its stream still drains (programmatic stream
// serialization): launch, barrier set-up and tensor-memory allocation then cost nothing on the stream.  A kernel waits
// for that predecessor - complete, its memory visible - in bb::pdl_sync() before it touches global memory, and only
// then lets its own successor in, so a kernel never overlaps more than its direct neighbours and everything before the
// predecessor is complete too.  Work beside the main stream (max_ctas other than 0: redundant computation with short CTAs
// or on a budget of them) is launched plainly: a kernel that waits keeps its SMs.
extern thread_local int bb_back_to_back;
struct BackToBack {
  const int n;
  explicit BackToBack(bool on = true) : n(on ? 1 : 0) { bb_back_to_back += n; }
  ~BackToBack() { bb_back_to_back -= n; }
};
template <typename... P, typename... A>
inline cudaError_t bb_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = bb_back_to_back > 0 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<A&&>(args)...);
}

// One product of a k x k convolution whose patch matrix is never stored: the GEMM's producer gathers the
// patches with im2col TMA loads (gemm_tcgen05.cu).  `x` is the NHWC tensor the patches come from.
//   BB_CONV_FWD    D[P, Cout] = patches(x) * W^T                   x = input, channels C = Cin
//   BB_CONV_WGRAD  D[Cout, k*k*C] += dy^T * patches(x)             x = input, other = dy [P, Cout]
//   BB_CONV_DGRAD  D[P, C_in] = patches(x) * (W turned by 180 deg) x = dy, stride 1, channels C = Cout
enum { BB_CONV_FWD = 0, BB_CONV_WGRAD = 1, BB_CONV_DGRAD = 2 };
struct bb_conv_gemm_args {
  int mode;
  const void* x; int N, H, W, C;        // patch source
  int k, stride, pad, Ho, Wo;           // window over it; N * Ho * Wo patches
  const void* other;                    // weights [Cout, k*k*Cin], or dy for BB_CONV_WGRAD
  int other_channels;                   // Cout (FWD, WGRAD) or Cin (DGRAD)
  void* D;
  int max_ctas;
};
// True when the im2col loads can express the convolution's patches (64-channel blocks, window within the
// tensor map's limits).
bool bb_conv_gemm_supported(int C, int k, int stride, int pad);
int bb_conv_gemm(const bb_conv_gemm_args* a, void* stream);
// Time that a stored product of M x N over K is expected to take on the whole GPU, as it is planned for that CTA budget.
double bb_gemm_store_us(long long M, long long N, long long K, int max_ctas);

// Division by a number known at launch: n / d = high word of n * magic with magic = floor(2^64 / d) + 1 (0 stands for
// d = 1); for n < 2^32 the error n * d / 2^64 stays below 1.
inline unsigned long long bb_div_magic(int d) { return d == 1 ? 0 : ~0ull / (unsigned long long)d + 1; }

namespace bb {

__device__ __forceinline__ unsigned fast_div(unsigned n, unsigned long long magic) {
  return magic ? (unsigned)__umul64hi((unsigned long long)n, magic) : n;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// One lane of a converged warp, the same one every time.  The blocks that issue tcgen05.mma, tcgen05.commit and TMA
// run under it and not under `lane == 0`: these instructions take warp-uniform operands, and the compiler only knows
// that a single thread is active when the predicate comes from elect.sync.  Measured against `lane == 0`: GEMM
// 4096 x 12288 x 4096 285 -> 256 us, 8192 x 1024 x 4096 61 -> 57 us, 8192 x 50304 x 1024 658 -> 612 us; attention
// backward at head dimension 128 (B2 H32 S2048 causal) 556 -> 497 us, the kernels at 64 unchanged.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// This thread's warp, as a value that the compiler knows to be the same for the whole warp: branches on it are then uniform,
// and inside them loop counters and addresses stay in uniform registers, which TMA and tcgen05 instructions take their
// operands from.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// Called by every thread before its first access to global memory (see bb_launch).  A kernel that calls it may be
// resident while its predecessor still writes, so what a kernel may have written is not constant for its successor's
// lifetime and must not be read through the read-only path: no __ldg and no `const T* __restrict__` (which lets the
// compiler choose that path, and move the load) on anything but parameters (gamma, beta, bias), and no __restrict__ on
// what is added to.  __ldca and __ldcg are coherent and stay behind the wait, as do plain loads through other pointers.
__device__ __forceinline__ void pdl_sync() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}

// Bounded wait.  Returns false when the limit expired or another role already gave up
// (*abort != 0); the caller must then leave its loop.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort, int* status) {
  uint32_t ok;
  uint64_t t0 = 0;
  for (uint32_t spin = 0;; ++spin) {
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if ((spin & 1023u) == 1023u) {
      if (*abort) return false;
      uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > BB_WAIT_LIMIT_NS) {
        *abort = 1;
        if (status) atomicCAS(status, 0, BB_STATUS_KERNEL_WAIT_TIMEOUT);
        return false;
      }
    }
  }
}

// Bounded wait of a whole warp with one outcome for all lanes (lanes that gave up at different moments would
// leave the others behind at the next warp-wide instruction).
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort, int* status) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort, status));
}

// The same for two barriers: their first tests are in flight together.
__device__ __forceinline__ bool mbar_wait2_warp(uint64_t* a, uint32_t pa, uint64_t* b, uint32_t pb, volatile int* abort, int* status) {
  const bool oa = mbar_try_wait(a, pa), ob = mbar_try_wait(b, pb);
  if (__all_sync(0xffffffffu, oa && ob)) return true;
  const bool ra = mbar_wait(a, pa, abort, status), rb = mbar_wait(b, pb, abort, status);
  return __all_sync(0xffffffffu, ra && rb);
}

// Bounded wait with cluster-scope acquire: for barriers that another CTA of the cluster arrives on
// after writing this CTA's shared memory with plain stores (st.shared::cluster).
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort, int* status) {
  uint32_t ok;
  uint64_t t0 = 0;
  for (uint32_t spin = 0;; ++spin) {
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if ((spin & 1023u) == 1023u) {
      if (*abort) return false;
      uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > BB_WAIT_LIMIT_NS) {
        *abort = 1;
        if (status) atomicCAS(status, 0, BB_STATUS_KERNEL_WAIT_TIMEOUT);
        return false;
      }
    }
  }
}

// ---------------------------------------------------------------- TMA (no cluster multicast anywhere)
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const void* tmap, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      : : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const void* tmap, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      : : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// im2col load of an NHWC tensor: consecutive output pixels from input position (c, w, h, n) on (the first
// tap's corner of the first pixel's window), all shifted by the tap's (off_w, off_h).  The tensor map holds
// the window's range, the stride and the zero fill outside the image.
__device__ __forceinline__ void tma_load_im2col(void* smem_dst, const void* tmap, uint64_t* bar, int c, int w, int h, int n,
                                                uint16_t off_w, uint16_t off_h) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2], "
      "{%7, %8};"
      : : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c), "r"(w), "r"(h), "r"(n), "h"(off_w), "h"(off_h)
      : "memory");
}
// shared -> global fp32 add-reduction of a tile through a tensor map (clips at the edges)
__device__ __forceinline__ void tma_reduce_add_2d(const void* tmap, const void* smem_src, int c0, int c1) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];"
               : : "l"(tmap), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait_group_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N> __device__ __forceinline__ void bulk_wait_group() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}

// ---------------------------------------------------------------- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]; single-thread issue.
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      : : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrive on an mbarrier once every previously issued tcgen05.mma of this thread retired.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// registers -> 32 columns of this warp's 32 TMEM lanes (one row per lane); complete after tmem_st_wait()
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      : : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor for tcgen05.mma, 128-byte swizzle.
//   start address, leading/stride byte offsets are encoded in 16-byte units.
__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}

// ---------------------------------------------------------------- CTA pairs (cta_group::2)
// Two CTAs of a cluster (ranks 0 and 1) work on one 256-row tile: each holds its own 128 rows of
// A and half of B in shared memory, rank 0 issues the MMAs for both, each keeps its 128
// accumulator rows in its own TMEM.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_shared(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// plain 4-byte store into the shared memory of another CTA of the cluster (address from mapa_shared)
__device__ __forceinline__ void st_shared_cluster_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_shared_cluster_v4(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The same without release, for hand-backs of what the warp has finished reading.  It orders nothing by itself, so the reads have to be
// over when it is issued: an accumulator's by tcgen05.wait::ld and tcgen05.fence::before_thread_sync, which orders the tensor
// core's accesses before a barrier operation of any kind (the taker answers with fence::after_thread_sync); a word of shared
// memory's by a branch on its value (a value cannot be the one that its own hand-back brings about).  A release at cluster scope
// waits until all of the thread's earlier global stores have been performed - a microsecond per tile where an epilogue
// warp hands an accumulator back between two panels.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA tile load into this CTA's shared memory whose completion is signalled on an mbarrier of
// either CTA of the pair (given as a shared::cluster address); no multicast.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t bar_cluster_addr, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      : : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(bar_cluster_addr), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_load_im2col_pair(void* smem_dst, const void* tmap, uint32_t bar_cluster_addr, int c, int w,
                                                     int h, int n, uint16_t off_w, uint16_t off_h) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
      : : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(bar_cluster_addr), "r"(c), "r"(w), "r"(h), "r"(n), "h"(off_w), "h"(off_h)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t addr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      : : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrive on the mbarrier at this shared-memory offset in every CTA of `cta_mask` once all
// previously issued MMAs of this thread retired (an arrival signal, not a data load).
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t cta_mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(cta_mask) : "memory");
}

// ---------------------------------------------------------------- numerics
// hardware tanh (one MUFU op, ~2^-11 relative error: far below bf16 resolution)
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two-wide fp32 arithmetic (each half rounded like the scalar instruction): half the issue slots, which is what the fused
// epilogues of short reductions run out of.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)), "l"(reinterpret_cast<unsigned long long&>(c)));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return d;
}
// tanh GeLU: x/2 (1 + t), t = tanh(k0 x + k0 k1 x^3), and its derivative (1 + t)/2 + x/2 (1 - t^2) (k0 + 3 k0 k1 x^2)
constexpr float GELU_K0 = 0.7978845608028654f, GELU_K01 = 0.7978845608028654f * 0.044715f;
__device__ __forceinline__ float2 gelu_tanh2(float2 x) {
  const float2 u = mul2(fma2(mul2(x, x), make_float2(GELU_K01, GELU_K01), make_float2(GELU_K0, GELU_K0)), x);
  const float2 h = mul2(x, make_float2(0.5f, 0.5f));
  return fma2(h, make_float2(tanh_fast(u.x), tanh_fast(u.y)), h);
}
__device__ __forceinline__ float2 gelu_tanh_grad2(float2 x) {
  const float2 x2 = mul2(x, x), k0 = make_float2(GELU_K0, GELU_K0), half = make_float2(0.5f, 0.5f);
  const float2 u = mul2(fma2(x2, make_float2(GELU_K01, GELU_K01), k0), x);
  const float2 du = fma2(x2, make_float2(3.f * GELU_K01, 3.f * GELU_K01), k0);
  const float2 t = make_float2(tanh_fast(u.x), tanh_fast(u.y));
  const float2 s = fma2(make_float2(-t.x, -t.y), t, make_float2(1.f, 1.f));
  return fma2(mul2(mul2(x, half), s), du, fma2(half, t, half));
}
__device__ __forceinline__ float gelu_tanh_grad(float x) { return gelu_tanh_grad2(make_float2(x, x)).x; }
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }

}  // namespace bb
