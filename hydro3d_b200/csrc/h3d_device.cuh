// Device and launch helpers shared by the kernel files.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>

#include "h3d_internal.h"

namespace h3d {

// Programmatic dependent launch (opt-in, H3D_PDL=1 in the environment): every
// kernel lets the next one on the stream start launching at once
// (griddepcontrol.launch_dependents) and waits for its predecessors to
// complete (griddepcontrol.wait) before it touches data they write.  Both are
// no-ops for a kernel launched without the attribute.  For every launch it
// measured 60.1 ms against 56.1 ms without on the 33.5M-cell solve (the
// early launched grids hold SM resources the running ones need).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
//
// A kernel that starts early runs while its predecessors still write, so what
// they write is not constant for its lifetime, as `const __restrict__` data is for the
// compiler: such loads (ld.global.nc) are not held back by the wait.  (The load of
// the mean that remove_mean subtracts was moved above it: solves of up to 75,000 words
// kept their mean in up to a third of the calls.)  The wait therefore takes the
// pointers to data that predecessors write and makes them opaque; tables written
// once at set-up are left out (and no const __restrict__ is put on them again
// behind the wait).  Plain loads are not moved ahead of stores and
// barriers either, which costs the large streaming kernels (every kernel in this form:
// 192^3 in FP64 9.74 -> 9.99 ms, 256^3 of variable density 20.6 -> 25.6 ms), and
// large launches do not start early: those kernels are built in two forms, EARLY
// with opaque pointers and one without.
template <typename Ptr>
__device__ __forceinline__ void make_opaque(Ptr& p) {
  asm volatile("" : "+l"(p));
}
template <bool EARLY = true, typename... Ptr>
__device__ __forceinline__ void pdl_wait(Ptr&... written) {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  if constexpr (EARLY) (make_opaque(written), ...);
}

// Launch policy (H3D_PDL): "1" every pdl_launch, "0" none; by default only a
// kernel of at most kPdlGrid CTAs that follows one of at most kPdlGrid CTAs
// on the same host thread.  Such a predecessor runs in a single wave, so the
// early-launched grid only takes SM slots that the predecessor leaves idle,
// while the launch latency of the chains of small kernels of the coarse
// levels is hidden.
constexpr long long kPdlGrid = 2 * 148;
inline int pdl_mode() {
  static const int m = [] {
    const char* v = std::getenv("H3D_PDL");
    if (v && v[0] == '1') return 1;
    if (v && v[0] == '0') return 0;
    return 2;
  }();
  return m;
}
inline thread_local long long g_prev_grid = 1LL << 40;

// The next launch of this host thread, of n CTAs: does it start early?
inline bool pdl_early(long long n) {
  const int mode = pdl_mode();
  const bool early = mode == 1 || (mode == 2 && n <= kPdlGrid && g_prev_grid <= kPdlGrid);
  g_prev_grid = n;
  return early;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*k)(KArgs...), bool early, dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                 Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t pdl_launch(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                              Args... args) {
  return launch_kernel(k, pdl_early((long long)grid.x * grid.y * grid.z), grid, block, smem, st, args...);
}

// Never early, in the form without opaque pointers: the sweep and the restriction that
// stage planes by plain loads between barriers, with variable density (88 x 88 x 104
// cells: 291 us a cycle, 345 early; 64^3 176, 199) and on large levels, and sequential
// kernels that run for long on few CTAs.
template <typename... KArgs, typename... Args>
inline cudaError_t plain_launch(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                Args... args) {
  g_prev_grid = (long long)grid.x * grid.y * grid.z;
  return launch_kernel(k, false, grid, block, smem, st, args...);
}

// The two forms of a kernel (see pdl_wait); H3D_BOTH(k, a, b): those of k<a, b, EARLY>.
template <typename... KArgs>
struct KernelPair {
  void (*plain)(KArgs...);
  void (*early)(KArgs...);
};
template <typename... KArgs>
KernelPair(void (*)(KArgs...), void (*)(KArgs...)) -> KernelPair<KArgs...>;
#define H3D_BOTH(k, ...) KernelPair{k<__VA_ARGS__, false>, k<__VA_ARGS__, true>}

template <typename... KArgs, typename... Args>
inline cudaError_t pdl_launch(KernelPair<KArgs...> k, dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                              Args... args) {
  const bool early = pdl_early((long long)grid.x * grid.y * grid.z);
  return launch_kernel(early ? k.early : k.plain, early, grid, block, smem, st, args...);
}

template <typename... KArgs>
inline cudaError_t kernel_smem(KernelPair<KArgs...> k, int bytes) {
  cudaError_t e = cudaFuncSetAttribute(k.plain, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return e != cudaSuccess ? e : cudaFuncSetAttribute(k.early, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

__device__ __forceinline__ int find_block(const int* __restrict__ start, int nb, int cta) {
  int lo = 0, hi = nb;  // start[lo] <= cta < start[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (__ldg(start + mid) <= cta) lo = mid;
    else hi = mid;
  }
  return lo;
}

template <typename T>
struct Coef {
  T aw, ae, as, an, ab, at;
};

// Face coefficients of interior cell (x,y,z) (mgsolver.for:186-205).
template <typename T, bool VAR>
__device__ __forceinline__ Coef<T> cell_coef(const BlkLev& B, int x, int y, int z, long long i, const T* fx,
                                             const T* fy, const T* fz) {
  Coef<T> c;
  if (VAR) {
    c.aw = fx[i - 1];
    c.ae = fx[i];
    c.as = fy[i - B.sx];
    c.an = fy[i];
    c.ab = fz[i - B.sxy];
    c.at = fz[i];
  } else {
    const T ax = (T)B.ax, ay = (T)B.ay, az = (T)B.az;
    const int ph = B.phys;
    c.aw = (x == 1 && (ph & 1)) ? T(0) : ax;
    c.ae = (x == B.nx && (ph & 2)) ? T(0) : ax;
    c.as = (y == 1 && (ph & 4)) ? T(0) : ay;
    c.an = (y == B.ny && (ph & 8)) ? T(0) : ay;
    c.ab = (z == 1 && (ph & 16)) ? T(0) : az;
    c.at = (z == B.nz && (ph & 32)) ? T(0) : az;
  }
  return c;
}

template <typename T>
__device__ __forceinline__ T coef_ap(const Coef<T>& c) {
  return -(c.aw + c.ae + c.as + c.an + c.ab + c.at);  // -1.0*(...), mgsolver.for:207-210
}

// Gauss-Seidel update division: IEEE division in FP64 (the reference's
// arithmetic); the FP32 inner solve uses the 2-ulp reciprocal division.
__device__ __forceinline__ double gs_div(double a, double b) { return a / b; }
__device__ __forceinline__ float gs_div(float a, float b) { return __fdividef(a, b); }

// Over-relaxed red-black update of the FP32 inner solve: x + om (gs - x), om
// the handle's over-relaxation factor (1: Gauss-Seidel up to rounding).  The
// FP64 sweeps keep the reference's update.
__device__ __forceinline__ float sorf(float old, float gs, float om) { return fmaf(om, gs - old, old); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

template <typename T>
__device__ __forceinline__ void cp_async_word(T* s, const T* g) {
  const unsigned a = smem_u32(s);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(a), "l"(g), "n"(sizeof(T)) : "memory");
}

// First 128-byte boundary of the dynamic shared memory, by pointer arithmetic
// on the shared array itself so that accesses through it stay shared-memory
// instructions (a round trip through an integer would make them generic).
__device__ __forceinline__ unsigned char* smem_base128(unsigned char* raw) {
  return raw + ((128u - (smem_u32(raw) & 127u)) & 127u);
}

// ---------------------------------------------------------------------------
template <int NT>
__device__ __forceinline__ void block_reduce4(double a0, double a1, double a2, double a3, double* out) {
  __shared__ double sh[4][NT / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
    a2 = fmax(a2, __shfl_xor_sync(0xffffffffu, a2, o));
    a3 += __shfl_xor_sync(0xffffffffu, a3, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { sh[0][w] = a0; sh[1][w] = a1; sh[2][w] = a2; sh[3][w] = a3; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
    for (int q = 0; q < NT / 32; ++q) { s0 += sh[0][q]; s1 += sh[1][q]; s2 = fmax(s2, sh[2][q]); s3 += sh[3][q]; }
    out[0] = s0; out[1] = s1; out[2] = s2; out[3] = s3;
  }
}

// Exact division by a known divisor: a / b correctly rounded, as the IEEE
// division the reference's update uses, from y = RN(1/b): q = RN(a y) is at most two
// units off, one residual step q + (a - b q) y makes it faithful, a second one
// correctly rounded (P. Markstein, Computation of elementary functions on the IBM
// RISC System/6000 processor, 1990).  The residuals are exact while nothing
// under- or overflows: other operands take the division itself.  Five
// multiply-adds where the division is a subroutine.
__device__ __forceinline__ bool div_range(double v) {
  return ((unsigned)(__double2hiint(v) >> 20) & 0x7ffu) - 523u < 1000u;  // 2^-500 <= |v| < 2^500
}
__device__ __forceinline__ double div_known(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-b, q, a), y, q);
  q = fma(fma(-b, q, a), y, q);
  return __builtin_expect(div_range(a) && div_range(b), 1) ? q : a / b;
}

}  // namespace h3d
