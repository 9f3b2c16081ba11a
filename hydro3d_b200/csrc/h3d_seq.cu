// Sequentially ordered solvers on the device: Stone's SIP (sipsol.for).  Their
// recurrences run as wavefronts; a block is one thread-block cluster.
#include <cooperative_groups.h>

#include <algorithm>

#include "h3d_device.cuh"
#include "h3d_kernels.cuh"

namespace h3d {

namespace cg = cooperative_groups;

namespace {

// ---------------------------------------------------------------------------
// Stone's strongly implicit procedure (sipsol.for:2-205, ifi = 44), the
// reference's alternative pressure solver, on level 1 with the constant
// coefficients pressure_1sweep builds (press.for:407-438: the same values as
// coeff's level 1).  The LU factors and both substitutions are recurrences
// over the predecessors (x-1, y-1, z-1) (successors for the backward pass), so
// hyperplanes x+y+z = d are the wavefronts, every value the one the
// reference's k, i, j loops compute, in its operand order.
//
// What bounds them is the chain of nx+ny+nz-2 dependent steps of each pass,
// so a step is made short: thread (y, z) marches along x, step d its cell
// x = d-y-z; the three predecessors are the values that it and the threads
// (y-1, z), (y, z-1) computed one step earlier, exchanged through shared
// memory (two buffers, one barrier a step); the factors of the next steps are
// copied kAhead steps ahead into shared memory (cp.async;
// register prefetches of several steps share scoreboards and wait for the
// newest).  The factor and residual arrays are
// laid out for those loads: cell (x, y, z) of a block at (z*(nx+ny-1) + x+y)*ny
// + y, so that the threads of one z read consecutive addresses.
//
// The rows of a block are spread over a cluster of at most eight CTAs, a slab
// of z each.  Steps run in phases of kPhase steps between two cluster
// barriers, CTA c one phase behind CTA c-1 (forward), whose last row of z it
// reads from a ring that CTA c-1 writes into its shared memory.
//
// 48x32x40 blocks (118 steps a pass): one CTA per block with a barrier a step,
// reading everything from global memory at the point of use, took 859 us a
// sweep (3.6 us a step); four such blocks, 100 sweeps with their residuals, stop
// tests and projection steps: 76.5 ms then, 14.8 ms now (20.9 ms with register
// prefetches).
constexpr int kPhase = 8, kRing = 4 * kPhase, kAhead = 4;
constexpr int kSipThreads = 512, kSipMaxCtas = 8, kSipMaxSmem = 200 * 1024;

struct SipLU {
  double *lb, *lw, *ls, *lpr, *un, *ue, *ut, *res;
};

// Position of interior cell (x, y, z) in the skewed arrays.
struct SipSkew {
  long long off;
  int ny, e;
  __device__ __forceinline__ SipSkew(const BlkLev& B, long long o) : off(o), ny(B.ny), e(B.nx + B.ny - 1) {}
  __device__ __forceinline__ long long at(int x, int y, int z) const {
    return off + ((long long)z * e + x + y) * ny + y;
  }
};

template <typename T>
__device__ __forceinline__ void cp_async_word(T* s, const T* g) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(s);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(a), "l"(g), "n"(sizeof(T)) : "memory");
}

// One CTA's share of a march over `steps` hyperplanes: step(d, k) for its
// active ones, in ascending (FWD) or descending order, a CTA barrier after
// each, a cluster barrier after every phase.  prefetch(d, k) starts a thread's
// copies for step d into its slot k, kAhead steps before they are read.
template <bool FWD, typename Prefetch, typename Step>
__device__ __forceinline__ void sip_march(int steps, int rank, int nranks, Prefetch&& prefetch, Step&& step) {
  const int nblk = (steps + kPhase - 1) / kPhase;
  const int lag = FWD ? rank : nranks - 1 - rank;
#pragma unroll
  for (int k = 0; k < kAhead; ++k) {
    prefetch(FWD ? k : steps - 1 - k, k);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  for (int p = 0; p < nblk + nranks - 1; ++p) {
    const int blk = p - lag;
    if (blk >= 0 && blk < nblk) {
#pragma unroll
      for (int k = 0; k < kPhase; ++k) {
        const int t = blk * kPhase + k;
        if (t < steps) {
          asm volatile("cp.async.wait_group %0;\n" ::"n"(kAhead - 1) : "memory");
          step(FWD ? t : steps - 1 - t, k % kAhead);
          const int tn = t + kAhead;
          prefetch(FWD ? tn : steps - 1 - tn, k % kAhead);
          asm volatile("cp.async.commit_group;\n" ::: "memory");
          __syncthreads();
        }
      }
    }
    if (nranks > 1) cg::this_cluster().sync();
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Shared memory of a march of NV values a cell: the two step buffers
// [2][rows of z][ny + 2] (column 0 and ny + 1 stay zero) and the ring
// [kRing][ny] the neighbouring CTA writes.
struct SipSmem {
  double* cur;
  double* ring;
  int pitch, rows, plane;
};

__device__ __forceinline__ SipSmem sip_smem(double* base, int rows, int ny) {
  SipSmem s;
  s.pitch = ny + 2;
  s.rows = rows;
  s.plane = rows * s.pitch;
  s.cur = base;
  s.ring = base + 2 * s.plane;
  return s;
}

__device__ __forceinline__ void sip_clear(double* base, long long n) {
  for (long long q = threadIdx.x; q < n; q += blockDim.x) base[q] = 0.0;
}

// LU factors (sipsol.for:77-105).
__global__ void __launch_bounds__(kSipThreads) k_sip_factor_c(const BlkLev* __restrict__ bls,
                                                            const long long* __restrict__ offs, SipLU lu) {
  extern __shared__ double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int nr = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const BlkLev B = bls[blockIdx.x / nr];
  const SipSkew S(B, offs[blockIdx.x / nr]);
  pdl_trigger();
  pdl_wait();
  const double alfa = 0.92, small = 1e-20;  // sipsol.for:32-33
  const int nx = B.nx, ny = B.ny, nz = B.nz;
  const int hz = (nz + nr - 1) / nr, z0 = min(nz, rank * hz), z1 = min(nz, z0 + hz);
  const int nrow = (z1 - z0) * ny;
  const long long part = 2LL * hz * (ny + 2) + (long long)kRing * ny;
  SipSmem un = sip_smem(sm, hz, ny), ue = sip_smem(sm + part, hz, ny), ut = sip_smem(sm + 2 * part, hz, ny);
  sip_clear(sm, 3 * part);
  __syncthreads();
  if (nr > 1) cl.sync();
  double* next = rank + 1 < nr ? cl.map_shared_rank(sm, rank + 1) : nullptr;
  const long long ring = 2LL * hz * (ny + 2);
  sip_march<true>(
      nx + ny + nz - 2, rank, nr, [](int, int) {},
      [&](int d, int) {
        const int w = (d & 1) * un.plane, r = un.plane - w;
        for (int q = threadIdx.x; q < nrow; q += blockDim.x) {
          const int zl = q / ny, y = q - zl * ny, z = z0 + zl, x = d - y - z;
          if (x < 0 || x >= nx) continue;
          const int o = zl * un.pitch + y + 1;
          const double unw = un.cur[r + o], uew = ue.cur[r + o], utw = ut.cur[r + o];
          const double uns = un.cur[r + o - 1], ues = ue.cur[r + o - 1], uts = ut.cur[r + o - 1];
          double unb, ueb, utb;
          if (zl > 0) {
            unb = un.cur[r + o - un.pitch];
            ueb = ue.cur[r + o - un.pitch];
            utb = ut.cur[r + o - un.pitch];
          } else {
            const int h = ((d - 1) & (kRing - 1)) * ny + y;
            unb = un.ring[h];
            ueb = ue.ring[h];
            utb = ut.ring[h];
          }
          const Coef<double> c = cell_coef<double, false>(B, x + 1, y + 1, z + 1, 0, nullptr, nullptr, nullptr);
          const double ap = coef_ap(c);
          const double lb = c.ab / (1. + alfa * (unb + ueb));
          const double lw = c.aw / (1. + alfa * (unw + utw));
          const double ls = c.as / (1. + alfa * (ues + uts));
          const double p1 = alfa * (lb * unb + lw * unw);
          const double p2 = alfa * (lb * ueb + ls * ues);
          const double p3 = alfa * (lw * utw + ls * uts);
          const double lpr = 1. / (ap + p1 + p2 + p3 - lb * utb - lw * uew - ls * uns + small);
          const double vn = (c.an - p1) * lpr, ve = (c.ae - p2) * lpr, vt = (c.at - p3) * lpr;
          const long long i = S.at(x, y, z);
          lu.lb[i] = lb;
          lu.lw[i] = lw;
          lu.ls[i] = ls;
          lu.lpr[i] = lpr;
          lu.un[i] = vn;
          lu.ue[i] = ve;
          lu.ut[i] = vt;
          un.cur[w + o] = vn;
          ue.cur[w + o] = ve;
          ut.cur[w + o] = vt;
          if (next && z == z1 - 1) {
            const long long h = ring + (long long)(d & (kRing - 1)) * ny + y;
            next[h] = vn;
            next[part + h] = ve;
            next[2 * part + h] = vt;
          }
        }
      });
}

// Forward and backward substitution of one sweep (sipsol.for:159-175) on res.
// ONE: at most one row (y, z) a thread; otherwise the rows of a step are
// looped over and loaded at the point of use.
template <bool ONE>
__global__ void __launch_bounds__(kSipThreads) k_sip_subst(const BlkLev* __restrict__ bls,
                                                           const long long* __restrict__ offs, SipLU lu) {
  extern __shared__ double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int nr = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const BlkLev B = bls[blockIdx.x / nr];
  const SipSkew S(B, offs[blockIdx.x / nr]);
  pdl_trigger();
  const int nx = B.nx, ny = B.ny, nz = B.nz, steps = nx + ny + nz - 2;
  const int hz = (nz + nr - 1) / nr, z0 = min(nz, rank * hz), z1 = min(nz, z0 + hz);
  const int nrow = (z1 - z0) * ny;
  const long long part = 2LL * hz * (ny + 2) + (long long)kRing * ny;
  const SipSmem v = sip_smem(sm, hz, ny);
  const long long ring = 2LL * hz * (ny + 2);
  // the thread's row (ONE)
  const bool has = (int)threadIdx.x < nrow;
  const int tz = has ? (int)threadIdx.x / ny : 0, ty = has ? (int)threadIdx.x - tz * ny : 0;
  const long long row = S.at(0, ty, z0 + tz);
  const int to = tz * v.pitch + ty + 1, tx = ty + z0 + tz;  // x = d - tx
  // its operands of the next kAhead steps: word j of slot k at pf[(5k + j) * kSipThreads]
  double* pf = sm + part + threadIdx.x;
  auto F = [&](int k, int j) -> double& { return pf[(5 * k + j) * kSipThreads]; };
  pdl_wait();

  // forward: res = (res - lb*res(z-1) - lw*res(x-1) - ls*res(y-1)) * lpr
  sip_clear(sm, part);
  __syncthreads();
  if (nr > 1) cl.sync();
  {
    double* next = rank + 1 < nr ? cl.map_shared_rank(sm, rank + 1) : nullptr;
    sip_march<true>(
        steps, rank, nr,
        [&](int d, int k) {
          const int x = d - tx;
          if (ONE && has && x >= 0 && x < nx) {
            const long long i = row + (long long)x * ny;
            cp_async_word(&F(k, 0), lu.res + i);
            cp_async_word(&F(k, 1), lu.lb + i);
            cp_async_word(&F(k, 2), lu.lw + i);
            cp_async_word(&F(k, 3), lu.ls + i);
            cp_async_word(&F(k, 4), lu.lpr + i);
          }
        },
        [&](int d, int k) {
          const int w = (d & 1) * v.plane, r = v.plane - w;
          if (ONE) {
            const int x = d - tx;
            if (has && x >= 0 && x < nx) {
              const double b = tz > 0 ? v.cur[r + to - v.pitch] : v.ring[((d - 1) & (kRing - 1)) * ny + ty];
              const double n =
                  (F(k, 0) - F(k, 1) * b - F(k, 2) * v.cur[r + to] - F(k, 3) * v.cur[r + to - 1]) * F(k, 4);
              v.cur[w + to] = n;
              lu.res[row + (long long)x * ny] = n;
              if (next && z0 + tz == z1 - 1) next[ring + (long long)(d & (kRing - 1)) * ny + ty] = n;
            }
          } else {
            for (int q = threadIdx.x; q < nrow; q += blockDim.x) {
              const int zl = q / ny, y = q - zl * ny, x = d - y - z0 - zl;
              if (x < 0 || x >= nx) continue;
              const int o = zl * v.pitch + y + 1;
              const long long i = S.at(x, y, z0 + zl);
              const double b = zl > 0 ? v.cur[r + o - v.pitch] : v.ring[((d - 1) & (kRing - 1)) * ny + y];
              const double n =
                  (lu.res[i] - lu.lb[i] * b - lu.lw[i] * v.cur[r + o] - lu.ls[i] * v.cur[r + o - 1]) * lu.lpr[i];
              v.cur[w + o] = n;
              lu.res[i] = n;
              if (next && z0 + zl == z1 - 1) next[ring + (long long)(d & (kRing - 1)) * ny + y] = n;
            }
          }
        });
  }

  // backward: res = res - un*res(y+1) - ue*res(x+1) - ut*res(z+1)
  sip_clear(sm, part);
  __syncthreads();
  if (nr > 1) cl.sync();
  {
    double* next = rank > 0 ? cl.map_shared_rank(sm, rank - 1) : nullptr;
    sip_march<false>(
        steps, rank, nr,
        [&](int d, int k) {
          const int x = d - tx;
          if (ONE && has && x >= 0 && x < nx) {
            const long long i = row + (long long)x * ny;
            cp_async_word(&F(k, 0), lu.res + i);
            cp_async_word(&F(k, 1), lu.un + i);
            cp_async_word(&F(k, 2), lu.ue + i);
            cp_async_word(&F(k, 3), lu.ut + i);
          }
        },
        [&](int d, int k) {
          const int w = (d & 1) * v.plane, r = v.plane - w;
          if (ONE) {
            const int x = d - tx;
            if (has && x >= 0 && x < nx) {
              const double t = z0 + tz < z1 - 1 ? v.cur[r + to + v.pitch] : v.ring[((d + 1) & (kRing - 1)) * ny + ty];
              const double n = F(k, 0) - F(k, 1) * v.cur[r + to + 1] - F(k, 2) * v.cur[r + to] - F(k, 3) * t;
              v.cur[w + to] = n;
              lu.res[row + (long long)x * ny] = n;
              if (next && tz == 0) next[ring + (long long)(d & (kRing - 1)) * ny + ty] = n;
            }
          } else {
            for (int q = threadIdx.x; q < nrow; q += blockDim.x) {
              const int zl = q / ny, y = q - zl * ny, x = d - y - z0 - zl;
              if (x < 0 || x >= nx) continue;
              const int o = zl * v.pitch + y + 1;
              const long long i = S.at(x, y, z0 + zl);
              const double t = z0 + zl < z1 - 1 ? v.cur[r + o + v.pitch] : v.ring[((d + 1) & (kRing - 1)) * ny + y];
              const double n = lu.res[i] - lu.un[i] * v.cur[r + o + 1] - lu.ue[i] * v.cur[r + o] - lu.ut[i] * t;
              v.cur[w + o] = n;
              lu.res[i] = n;
              if (next && zl == 0) next[ring + (long long)(d & (kRing - 1)) * ny + y] = n;
            }
          }
        });
  }
}

// The interior cell (x, y, z from 0) of this thread, 256 cells a CTA.
__device__ __forceinline__ bool sip_cell(const BlkLev* __restrict__ bls, const int* __restrict__ cta_start, int nb,
                                         int* b, int* x, int* y, int* z) {
  *b = find_block(cta_start, nb, blockIdx.x);
  const int nx = bls[*b].nx, ny = bls[*b].ny, nz = bls[*b].nz;
  const int c = (blockIdx.x - cta_start[*b]) * blockDim.x + threadIdx.x;
  if (c >= nx * ny * nz) return false;
  *x = c % nx;
  *y = (c / nx) % ny;
  *z = c / (nx * ny);
  return true;
}

// Residual of every block (sipsol.for:146-157) into the skewed res, and the
// CTA's sum |res| in a fixed order into partials[4 * cta].
__global__ void __launch_bounds__(256) k_sip_residual(const BlkLev* __restrict__ bls,
                                                      const long long* __restrict__ offs,
                                                      const int* __restrict__ cta_start, int nb,
                                                      const double* __restrict__ fi_all,
                                                      const double* __restrict__ su_all, double* __restrict__ res,
                                                      double* __restrict__ partials) {
  pdl_trigger();
  pdl_wait();
  __shared__ double red[8];
  int b, x, y, z;
  double acc = 0.0;
  if (sip_cell(bls, cta_start, nb, &b, &x, &y, &z)) {
    const BlkLev& B = bls[b];
    const SipSkew S(B, offs[b]);
    const long long sj = B.sx, sk = B.sxy;
    const long long q = B.off + (z + 1) * sk + (y + 1) * sj + x + 1;
    const double* fi = fi_all;
    const Coef<double> c = cell_coef<double, false>(B, x + 1, y + 1, z + 1, q, nullptr, nullptr, nullptr);
    const double r = (su_all[q] - coef_ap(c) * fi[q] - c.an * fi[q + sj] - c.as * fi[q - sj] - c.ae * fi[q + 1] -
                      c.aw * fi[q - 1] - c.ab * fi[q - sk] - c.at * fi[q + sk]);
    res[S.at(x, y, z)] = r;
    acc = fabs(r);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += red[w];
    partials[4 * blockIdx.x] = s;
    partials[4 * blockIdx.x + 1] = 0.0;
    partials[4 * blockIdx.x + 2] = 0.0;
    partials[4 * blockIdx.x + 3] = 0.0;
  }
}

// fi = fi + res (sipsol.for:176).
__global__ void __launch_bounds__(256) k_sip_correct(const BlkLev* __restrict__ bls, const long long* __restrict__ offs,
                                                     const int* __restrict__ cta_start, int nb,
                                                     double* __restrict__ fi, const double* __restrict__ res) {
  pdl_trigger();
  pdl_wait();
  int b, x, y, z;
  if (!sip_cell(bls, cta_start, nb, &b, &x, &y, &z)) return;
  const BlkLev& B = bls[b];
  const SipSkew S(B, offs[b]);
  const long long q = B.off + (z + 1) * B.sxy + (y + 1) * (long long)B.sx + x + 1;
  fi[q] = fi[q] + res[S.at(x, y, z)];
}

// nb clusters of `ctas` CTAs (no programmatic dependent launch, nor for the kernel after them).
template <typename K, typename... Args>
cudaError_t cluster_launch(K k, int nb, int ctas, int threads, int smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nb * ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)ctas;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  g_prev_grid = 1LL << 40;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

}  // namespace

// CTAs of a block's cluster: 256 rows (y, z) each, up to the portable eight.
// fits: the step buffers of the factors, the largest, fit shared memory (blocks
// of 128x128 rows do, 160x160 do not: those keep one CTA per block and global
// memory, k_sip_sweep).
SipPlan sip_plan(const std::vector<BlkLev>& bl) {
  SipPlan P;
  int rows = 1, nz = 1, ny = 1;
  for (const auto& B : bl) {
    rows = std::max(rows, B.ny * B.nz);
    nz = std::max(nz, B.nz);
    ny = std::max(ny, B.ny);
  }
  P.ctas = std::max(1, std::min(std::min(kSipMaxCtas, nz), (rows + 255) / 256));
  const int hz = (nz + P.ctas - 1) / P.ctas;
  P.one = hz * ny <= kSipThreads;
  const long long words = 2LL * hz * (ny + 2) + (long long)kRing * ny;
  P.fits = 3 * 8 * words <= kSipMaxSmem;
  P.smem_factor = P.fits ? (int)(3 * 8 * words) : 0;
  P.smem_subst = P.fits ? (int)(8 * words) + (P.one ? 5 * kAhead * kSipThreads * 8 : 0) : 0;
  return P;
}

// The shared-memory limit of the kernels (once per device, before any launch).
cudaError_t init_seq_attributes() {
  const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(k_sip_factor_c, a, kSipMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sip_subst<true>, a, kSipMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sip_subst<false>, a, kSipMaxSmem);
  return e;
}

cudaError_t launch_sip_factor_c(const SipPlan& P, const BlkLev* bl, const long long* offs, int nb, SipArrays a,
                              cudaStream_t st) {
  if (nb <= 0) return cudaSuccess;
  SipLU lu{a.lb, a.lw, a.ls, a.lpr, a.un, a.ue, a.ut, a.res};
  return cluster_launch(k_sip_factor_c, nb, P.ctas, kSipThreads, P.smem_factor, st, bl, offs, lu);
}

cudaError_t launch_sip_sweep_c(const SipPlan& P, const BlkLev* bl, const long long* offs, CellTab interior, SipArrays a,
                             double* fi, const double* su, double* partials, cudaStream_t st) {
  if (interior.nb <= 0) return cudaSuccess;
  SipLU lu{a.lb, a.lw, a.ls, a.lpr, a.un, a.ue, a.ut, a.res};
  pdl_launch(k_sip_residual, interior.ncta, 256, 0, st, bl, offs, interior.cta_start, interior.nb, fi, su, a.res,
             partials);
  const int nb = interior.nb;
  cudaError_t e = P.one ? cluster_launch(k_sip_subst<true>, nb, P.ctas, kSipThreads, P.smem_subst, st, bl, offs, lu)
                        : cluster_launch(k_sip_subst<false>, nb, P.ctas, kSipThreads, P.smem_subst, st, bl, offs, lu);
  if (e != cudaSuccess) return e;
  pdl_launch(k_sip_correct, interior.ncta, 256, 0, st, bl, offs, interior.cta_start, interior.nb, fi, a.res);
  return cudaGetLastError();
}

}  // namespace h3d
