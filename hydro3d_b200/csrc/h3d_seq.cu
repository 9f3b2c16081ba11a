// Sequentially ordered solvers on the device: Stone's SIP (sipsol.for) and the
// line-TDMA sweep (mgsolver.for:434-549).  Their recurrences run as wavefronts,
// a block by one CTA or one thread-block cluster.
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

// Position of interior cell (x, y, z) in the skewed arrays.
struct SipSkew {
  long long off;
  int ny, e;
  __device__ __forceinline__ SipSkew(const BlkLev& B, long long o) : off(o), ny(B.ny), e(B.nx + B.ny - 1) {}
  __device__ __forceinline__ long long at(int x, int y, int z) const {
    return off + ((long long)z * e + x + y) * ny + y;
  }
};

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
                                                            const long long* __restrict__ offs, SipArrays lu) {
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
                                                           const long long* __restrict__ offs, SipArrays lu) {
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
template <bool EARLY>
__global__ void __launch_bounds__(256) k_sip_residual(const BlkLev* __restrict__ bls,
                                                      const long long* __restrict__ offs,
                                                      const int* __restrict__ cta_start, int nb,
                                                      const double* __restrict__ fi_all,
                                                      const double* __restrict__ su_all, double* __restrict__ res,
                                                      double* __restrict__ partials) {
  pdl_trigger();
  pdl_wait<EARLY>(fi_all, su_all);
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
template <bool EARLY>
__global__ void __launch_bounds__(256) k_sip_correct(const BlkLev* __restrict__ bls, const long long* __restrict__ offs,
                                                     const int* __restrict__ cta_start, int nb,
                                                     double* __restrict__ fi, const double* __restrict__ res) {
  pdl_trigger();
  pdl_wait<EARLY>(fi, res);
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

namespace {

// ---------------------------------------------------------------------------
// Line-TDMA sweep of a level (mgrelax, mg_itrsch = 2, mgsolver.for:434-549),
// constant coefficients: j-lines, then i-lines, then k-lines of every block,
// every value the reference's, in its operand order.  A line (u, v) (u, v the
// two indices across it) follows (u-1, v) and (u, v-1), so the lines of an
// anti-diagonal u + v are independent: one thread a line forms the right-hand
// sides t(s) from the four cross neighbours and runs the recurrences c(s) =
// (t(s) - lo c(s-1)) apr(s) and phi(s) = c(s) - a(s) phi(s+1).  apr(s) = 1/(ap - lo a(s-1)) and a(s) =
// hi apr(s) depend on the line only through the walls beside it: they are
// tabulated per axis for the 16 combinations of "first / last u" and "first /
// last v", which takes the division out of the chain.
//
// The chain of (diagonals) x (5 FP64 operations a cell of a line) bounds the
// sweep, so its operands are in shared memory: whole small blocks (k_tdma_s), or the
// diagonals around the current one, copied by the other warps while the chains
// run (k_tdma_g).  For the latter every pass is preceded by a rearrangement of
// the level, by the whole chip, into rows d = u + v of (s, u), where the data
// of a diagonal are contiguous.
//
// Four 32x32x48 blocks, FP64 solve of 21 cycles: 327-345 ms with one thread a line
// reading global memory at the point of use and the division in the chain
// (k_tdma), 43 ms now (150 us a pass of 79 diagonals of 32-cell lines).
constexpr int kTdmaThreads = 256, kTdmaMaxSmem = 227 * 1024;

template <int AXIS>
struct LineAxes {  // (u, v, s) of AXIS: 0 lines along x, 1 along y, 2 along z
  static constexpr int US = AXIS == 0 ? 1 : 0, VS = AXIS == 2 ? 1 : 2, SS = AXIS;
};

template <int AXIS>
__device__ __forceinline__ int ext_of(const BlkLev& B, int a) {
  return a == 0 ? B.nx : a == 1 ? B.ny : B.nz;
}

// Wall-aware face coefficients along the three axes of a line cell.
template <typename T, int AXIS>
struct LineCoef {
  T au, av, as;
  bool ulo, uhi, vlo, vhi, slo, shi;
  __device__ __forceinline__ explicit LineCoef(const BlkLev& B) {
    const T a[3] = {(T)B.ax, (T)B.ay, (T)B.az};
    using L = LineAxes<AXIS>;
    au = a[L::US];
    av = a[L::VS];
    as = a[L::SS];
    ulo = B.phys >> (2 * L::US) & 1;
    uhi = B.phys >> (2 * L::US + 1) & 1;
    vlo = B.phys >> (2 * L::VS) & 1;
    vhi = B.phys >> (2 * L::VS + 1) & 1;
    slo = B.phys >> (2 * L::SS) & 1;
    shi = B.phys >> (2 * L::SS + 1) & 1;
  }
};

// Class of a line: bit 0 / 1 first / last u, bit 2 / 3 first / last v.
__device__ __forceinline__ int line_class(int u, int nu, int v, int nv) {
  return (u == 1 ? 1 : 0) | (u == nu ? 2 : 0) | (v == 1 ? 4 : 0) | (v == nv ? 8 : 0);
}

// tab[(s * 16 + class) * 2] = apr(s), a(s), s = 1..n, by threads 0..15.
template <typename T, int AXIS>
__device__ __forceinline__ void line_table(const LineCoef<T, AXIS>& C, int n, T* tab) {
  const int cl = threadIdx.x;
  if (cl >= 16) return;
  const T lu = (cl & 1) && C.ulo ? T(0) : C.au, hu = (cl & 2) && C.uhi ? T(0) : C.au;
  const T lv = (cl & 4) && C.vlo ? T(0) : C.av, hv = (cl & 8) && C.vhi ? T(0) : C.av;
  T aprev = T(0);
  for (int s = 1; s <= n; ++s) {
    const T lo = s == 1 && C.slo ? T(0) : C.as, hi = s == n && C.shi ? T(0) : C.as;
    Coef<T> c;
    c.aw = AXIS == 0 ? lo : lu;
    c.ae = AXIS == 0 ? hi : hu;
    c.as = AXIS == 1 ? lo : AXIS == 0 ? lu : lv;
    c.an = AXIS == 1 ? hi : AXIS == 0 ? hu : hv;
    c.ab = AXIS == 2 ? lo : lv;
    c.at = AXIS == 2 ? hi : hv;
    const T apr = gs_div(T(1), coef_ap(c) - lo * aprev);
    aprev = hi * apr;
    tab[(s * 16 + cl) * 2] = apr;
    tab[(s * 16 + cl) * 2 + 1] = aprev;
  }
}

// t = rhs - the four cross terms in the reference's order (j- and i-lines: the u
// pair first; k-lines: the v pair first).
template <typename T, int AXIS>
__device__ __forceinline__ T line_rhs(T r, T hu, T lu, T hv, T lv, T e, T w, T t, T b) {
  if (AXIS == 2) return r - hv * t - lv * b - hu * e - lu * w;
  return r - hu * e - lu * w - hv * t - lv * b;
}

__device__ __forceinline__ double lds_word(unsigned a, double) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float lds_word(unsigned a, float) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts_word(unsigned a, double v) {
  asm volatile("st.shared.f64 [%0], %1;\n" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void sts_word(unsigned a, float v) {
  asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(a), "f"(v) : "memory");
}

// Shared-memory addresses of position 0 of a line: right-hand side, cross
// neighbours u+1, u-1, v+1, v-1 and the line's own values; st: bytes a position.
struct LineAddr {
  unsigned r, e, w, t, b, c, st;
};

// One line: the right-hand sides t(s) and c(s) = (t(s) - lo c(s-1)) apr(s)
// upwards, c(s) into the line's own places (no other line of the diagonal reads
// them), then out(s, phi(s)) for s = n down to 1.  tab: the line's class in the
// table; c0 and after: the ghosts at both ends.
//
// Groups of eight positions in two sets of registers: the operands of the next
// group are loaded, and its t(s) formed, in the shadow of the current group's
// chain, never past the line.  FP64 operations complete 8 cycles after issue: the
// chain's floor is 24 cycles a position upwards and 16 downwards; with the loads in
// the chain's way (a loop unrolled by the compiler) it takes 52 upwards.
template <typename T, int AXIS, typename Out>
__device__ __forceinline__ void line_solve(const LineAddr& A, unsigned tab, int n, T hu, T lu, T hv, T lv, T lo1,
                                           T lo, T c0, T after, Out&& out) {
  constexpr int G = 8;
  constexpr unsigned TP = 32 * sizeof(T);  // table bytes a position
  const T z = T(0);
  T t[2][G], a[2][G];
  // operands of position s, t(s) in t and apr(s) in ap
  auto rhs_at = [&](unsigned s, T& tt, T& ap) {
    const unsigned o = s * A.st;
    const T r = lds_word(A.r + o, z), e = lds_word(A.e + o, z), w = lds_word(A.w + o, z), q = lds_word(A.t + o, z),
            b = lds_word(A.b + o, z);
    ap = lds_word(tab + s * TP, z);
    tt = line_rhs<T, AXIS>(r, hu, lu, hv, lv, e, w, q, b);
  };
  const int groups = n / G, head = n % G;
  T c = c0, l = lo1;
  for (int s = 1; s <= head; ++s) {  // the remainder first
    rhs_at(s, t[0][0], a[0][0]);
    c = (t[0][0] - l * c) * a[0][0];
    l = lo;
    sts_word(A.c + s * A.st, c);
  }
  auto load = [&](int h, int s) {
#pragma unroll
    for (int k = 0; k < G; ++k) rhs_at(s + k, t[h][k], a[h][k]);
  };
  auto chain = [&](int h, int s) {
#pragma unroll
    for (int k = 0; k < G; ++k) {
      c = (t[h][k] - l * c) * a[h][k];
      l = lo;
      sts_word(A.c + (s + k) * A.st, c);
    }
  };
  if (groups > 0) {
    int s = head + 1;
    load(0, s);
    for (int left = groups - 1;; s += 2 * G) {
      if (left > 0) load(1, s + G);
      chain(0, s);
      if (left-- == 0) break;
      if (left > 0) load(0, s + 2 * G);
      chain(1, s + G);
      if (left-- == 0) break;
    }
  }
  T x = after;
  auto loadb = [&](int h, int s) {
#pragma unroll
    for (int k = 0; k < G; ++k) {
      t[h][k] = lds_word(A.c + (s - k) * A.st, z);
      a[h][k] = lds_word(tab + (s - k) * TP + (unsigned)sizeof(T), z);
    }
  };
  auto back = [&](int h, int s) {
#pragma unroll
    for (int k = 0; k < G; ++k) {
      x = t[h][k] - a[h][k] * x;
      out(s - k, x);
    }
  };
  if (groups > 0) {
    int s = n;
    loadb(0, s);
    for (int left = groups - 1;; s -= 2 * G) {
      if (left > 0) loadb(1, s - G);
      back(0, s);
      if (left-- == 0) break;
      if (left > 0) loadb(0, s - 2 * G);
      back(1, s - G);
      if (left-- == 0) break;
    }
  }
  for (int s = head; s >= 1; --s) {
    x = lds_word(A.c + s * A.st, z) - lds_word(tab + s * TP + (unsigned)sizeof(T), z) * x;
    out(s, x);
  }
}

// ---- whole block in shared memory -----------------------------------------
// Pitches of the block there: rows 3 mod 4 and planes even, so that lanes on a
// diagonal fall into different banks (two-way conflicts for k-lines).
__host__ __device__ inline int tdma_s_sx(int nx) { return ((nx + 2 + 4) / 4) * 4 - 1; }
__host__ __device__ inline int tdma_s_sxy(int nx, int ny) { return (tdma_s_sx(nx) * (ny + 2) + 1) / 2 * 2; }

template <typename T, int AXIS>
__device__ __forceinline__ void tdma_s_pass(const BlkLev& B, T* D, const T* R, T* tab) {
  using L = LineAxes<AXIS>;
  const int sx = tdma_s_sx(B.nx), sxy = tdma_s_sxy(B.nx, B.ny);
  const int ex[3] = {B.nx, B.ny, B.nz}, pt[3] = {1, sx, sxy};
  const int nu = ex[L::US], nv = ex[L::VS], n = ex[L::SS];
  const int pu = pt[L::US], pv = pt[L::VS], ps = pt[L::SS];
  const LineCoef<T, AXIS> C(B);
  line_table<T, AXIS>(C, n, tab);
  const unsigned W = sizeof(T);
  const unsigned aD = (unsigned)__cvta_generic_to_shared(D), aR = (unsigned)__cvta_generic_to_shared(R);
  const unsigned aA = (unsigned)__cvta_generic_to_shared(tab);
  const T z = T(0);
  __syncthreads();
  for (int d = 2; d <= nu + nv; ++d) {
    const int u = max(1, d - nv) + (int)threadIdx.x, v = d - u;
    if (u <= min(nu, d - 1)) {
      const T hu = u == nu && C.uhi ? z : C.au, lu = u == 1 && C.ulo ? z : C.au;
      const T hv = v == nv && C.vhi ? z : C.av, lv = v == 1 && C.vlo ? z : C.av;
      const unsigned o = (u * pu + v * pv) * W, c = aD + o, st = ps * W;
      const LineAddr A{aR + o, c + pu * W, c - pu * W, c + pv * W, c - pv * W, c, st};
      line_solve<T, AXIS>(A, aA + 2 * W * line_class(u, nu, v, nv), n, hu, lu, hv, lv, C.slo ? z : C.as, C.as,
                          lds_word(c, z), lds_word(c + (n + 1) * st, z), [&](int s, T x) { sts_word(c + s * st, x); });
    }
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(kTdmaThreads) k_tdma_s(const BlkLev* __restrict__ bls, const T* __restrict__ src,
                                                         T* __restrict__ dst, const T* __restrict__ rhs, bool zero) {
  extern __shared__ __align__(16) unsigned char tdma_smem[];
  pdl_trigger();
  const BlkLev B = bls[blockIdx.x];
  const int sx = tdma_s_sx(B.nx), sxy = tdma_s_sxy(B.nx, B.ny);
  T* D = reinterpret_cast<T*>(tdma_smem);
  T* R = D + (size_t)sxy * (B.nz + 2);
  T* tab = R + (size_t)sxy * (B.nz + 2);
  pdl_wait(src, rhs);
  const int ex = B.nx + 2, ey = B.ny + 2, ncell = ex * ey * (B.nz + 2);
  for (int q = threadIdx.x; q < ncell; q += blockDim.x) {
    const int x = q % ex, y = (q / ex) % ey, z = q / (ex * ey);
    const long long i = B.off + (long long)z * B.sxy + (long long)y * B.sx + x;
    const int o = z * sxy + y * sx + x;
    if (zero) D[o] = T(0);
    else cp_async_word(D + o, src + i);
    cp_async_word(R + o, rhs + i);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  tdma_s_pass<T, 1>(B, D, R, tab);
  tdma_s_pass<T, 0>(B, D, R, tab);
  tdma_s_pass<T, 2>(B, D, R, tab);
  for (int q = threadIdx.x; q < ncell; q += blockDim.x) {
    const int x = q % ex, y = (q / ex) % ey, z = q / (ex * ey);
    dst[B.off + (long long)z * B.sxy + (long long)y * B.sx + x] = D[z * sxy + y * sx + x];
  }
}

// ---- larger blocks: diagonal rows in global scratch --------------------------
// Words of a block rearranged for AXIS: rows d = u + v (ghosts included: 0 ..
// nu+nv+2) of (s = 0 .. n+1, u = 0 .. nu+1).
__host__ __device__ inline long long tdma_rows(int nu, int nv, int n) {
  return (long long)(nu + nv + 3) * (n + 2) * (nu + 2);
}

template <int AXIS>
__device__ __forceinline__ long long tdma_at(const BlkLev& B, int x, int y, int z) {
  const int u = AXIS == 0 ? y : x, v = AXIS == 2 ? y : z, s = AXIS == 0 ? x : AXIS == 1 ? y : z;
  const int nu = AXIS == 0 ? B.ny : B.nx, n = AXIS == 0 ? B.nx : AXIS == 1 ? B.ny : B.nz;
  return ((long long)(u + v) * (n + 2) + s) * (nu + 2) + u;
}

// Rearranges the iterate and the right-hand side of every block for the pass
// along AXIS: from the level (FROM < 0; zero: the zero iterate) or from the rows of
// the pass along FROM.  256 cells a CTA, ghosts included.
template <typename T, int FROM, int AXIS, bool EARLY>
__global__ void __launch_bounds__(256) k_tdma_rows(const BlkLev* __restrict__ bls, const int* __restrict__ cta_start,
                                                   int nb, const T* __restrict__ src, const T* __restrict__ rhs,
                                                   const T* __restrict__ from, T* __restrict__ to,
                                                   T* __restrict__ rows, const long long* __restrict__ offs,
                                                   bool zero) {
  pdl_trigger();
  pdl_wait<EARLY>(src, rhs, from);
  const int b = find_block(cta_start, nb, blockIdx.x);
  const BlkLev& B = bls[b];
  const int ex = B.nx + 2, ey = B.ny + 2, q = (blockIdx.x - cta_start[b]) * blockDim.x + threadIdx.x;
  if (q >= ex * ey * (B.nz + 2)) return;
  const int x = q % ex, y = (q / ex) % ey, z = q / (ex * ey);
  const long long i = B.off + (long long)z * B.sxy + (long long)y * B.sx + x;
  const long long o = offs[b] + tdma_at<AXIS>(B, x, y, z);
  if (FROM < 0) to[o] = zero ? T(0) : src[i];
  else to[o] = from[offs[b] + tdma_at<FROM < 0 ? 0 : FROM>(B, x, y, z)];
  rows[o] = rhs[i];
}

// The rows of the last pass (along z) back into the level.
template <typename T, bool EARLY>
__global__ void __launch_bounds__(256) k_tdma_level(const BlkLev* __restrict__ bls, const int* __restrict__ cta_start,
                                                    int nb, const T* __restrict__ from, T* __restrict__ dst,
                                                    const long long* __restrict__ offs) {
  pdl_trigger();
  pdl_wait<EARLY>(from);
  const int b = find_block(cta_start, nb, blockIdx.x);
  const BlkLev& B = bls[b];
  const int ex = B.nx + 2, ey = B.ny + 2, q = (blockIdx.x - cta_start[b]) * blockDim.x + threadIdx.x;
  if (q >= ex * ey * (B.nz + 2)) return;
  const int x = q % ex, y = (q / ex) % ey, z = q / (ex * ey);
  dst[B.off + (long long)z * B.sxy + (long long)y * B.sx + x] = from[offs[b] + tdma_at<2>(B, x, y, z)];
}

// One pass, a CTA per block, on the rearranged iterate (in place) and rhs.
template <typename T, int AXIS>
__global__ void __launch_bounds__(kTdmaThreads) k_tdma_g(const BlkLev* __restrict__ bls, T* __restrict__ iter,
                                                         const T* __restrict__ rows,
                                                         const long long* __restrict__ offs, int nbuf) {
  extern __shared__ __align__(16) unsigned char tdma_smem[];
  using L = LineAxes<AXIS>;
  pdl_trigger();
  const BlkLev B = bls[blockIdx.x];
  T* Dk = iter + offs[blockIdx.x];
  const T* Rk = rows + offs[blockIdx.x];
  const int ex[3] = {B.nx, B.ny, B.nz};
  const int nu = ex[L::US], nv = ex[L::VS], n = ex[L::SS], pitch = nu + 2, row = (n + 2) * pitch;
  T* P = reinterpret_cast<T*>(tdma_smem);  // [2][n + 2][pitch]: c and phi of the current and the previous diagonal
  // nbuf (two: copied while the previous diagonal's chains run) times: the rhs of
  // a diagonal's lines, the old values of the next diagonal's, (u+1, v) and
  // (u, v+1), and the ghosts before and after its lines
  T* ops = P + 2 * row;
  const int opw = 2 * row + 2 * pitch;
  T* tab = ops + nbuf * opw;  // [n + 1][16][2]
  const LineCoef<T, AXIS> C(B);
  const int tid = threadIdx.x;
  line_table<T, AXIS>(C, n, tab);
  // copies the operands of diagonal d, by threads t0, t0 + nt, ...; the ghost
  // lines u = 0 and v = 0 that its lines read go to the places of the previous
  // diagonal's buffer that no line of that diagonal uses
  auto stage = [&](int d, int t0, int nt) {
    const T* r = Rk + (long long)d * row;
    const T* o = Dk + (long long)(d + 1) * row;
    const T* b = Dk + (long long)(d - 1) * row;
    const T* e = Dk + (long long)d * row;
    T* prev = P + ((d - 1) & 1) * row;
    T* SR = ops + (d & (nbuf - 1)) * opw;
    T *ST = SR + row, *E0 = ST + row, *E1 = E0 + pitch;
    for (int q = pitch + t0; q < (n + 1) * pitch; q += nt) {
      cp_async_word(SR + q, r + q);
      cp_async_word(ST + q, o + q);
    }
    for (int s = 1 + t0; s <= n; s += nt) {
      cp_async_word(prev + s * pitch, b + s * pitch);
      if (d - 1 <= nu) cp_async_word(prev + s * pitch + d - 1, b + s * pitch + d - 1);
    }
    for (int u = t0; u < pitch; u += nt) {
      cp_async_word(E0 + u, e + u);
      cp_async_word(E1 + u, e + (n + 1) * pitch + u);
    }
  };
  pdl_wait();
  stage(2, tid, blockDim.x);
  const unsigned W = sizeof(T), rowb = row * W, aP = (unsigned)__cvta_generic_to_shared(P);
  const unsigned aA = (unsigned)__cvta_generic_to_shared(tab);
  const T z = T(0);
  const int chain = 32 * ((min(nu, nv) + 31) / 32);  // threads of the warps that have lines
  for (int d = 2; d <= nu + nv; ++d) {
    const unsigned cur = aP + (d & 1) * rowb, prv = aP + ((d + 1) & 1) * rowb;
    const int u = max(1, d - nv) + tid, v = d - u;
    const bool mine = u <= min(nu, d - 1);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    if (nbuf == 2 && d < nu + nv) {
      if (chain >= kTdmaThreads) stage(d + 1, tid, kTdmaThreads);
      else if (tid >= chain) stage(d + 1, tid - chain, kTdmaThreads - chain);
    }
    if (mine) {
      const T hu = u == nu && C.uhi ? z : C.au, lu = u == 1 && C.ulo ? z : C.au;
      const T hv = v == nv && C.vhi ? z : C.av, lv = v == 1 && C.vlo ? z : C.av;
      const T* E0 = ops + (d & (nbuf - 1)) * opw + 2 * row;
      const unsigned c = u * W, aSR = aP + 2 * rowb + (d & (nbuf - 1)) * (unsigned)(opw * W), aST = aSR + rowb;
      const LineAddr A{aSR + c, aST + c + W, prv + c - W, aST + c, prv + c, cur + c, pitch * W};
      T* o = Dk + (long long)d * row + n * pitch + u;  // out() runs from s = n down
      line_solve<T, AXIS>(A, aA + 2 * W * line_class(u, nu, v, nv), n, hu, lu, hv, lv, C.slo ? z : C.as, C.as, E0[u],
                          E0[pitch + u], [&](int s, T x) {
                            sts_word(A.c + s * A.st, x);
                            *o = x;
                            o -= pitch;
                          });
    }
    if (nbuf == 1 && d < nu + nv) {
      __syncthreads();
      stage(d + 1, tid, kTdmaThreads);
    }
  }
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
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tdma_s<double>, a, kTdmaMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tdma_s<float>, a, kTdmaMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tdma_g<double, 0>, a, kTdmaMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tdma_g<double, 1>, a, kTdmaMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tdma_g<double, 2>, a, kTdmaMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tdma_g<float, 0>, a, kTdmaMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tdma_g<float, 1>, a, kTdmaMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tdma_g<float, 2>, a, kTdmaMaxSmem);
  return e;
}

cudaError_t launch_sip_factor_c(const SipPlan& P, const BlkLev* bl, const long long* offs, int nb, SipArrays a,
                              cudaStream_t st) {
  if (nb <= 0) return cudaSuccess;
  return cluster_launch(k_sip_factor_c, nb, P.ctas, kSipThreads, P.smem_factor, st, bl, offs, a);
}

cudaError_t launch_sip_sweep_c(const SipPlan& P, const BlkLev* bl, const long long* offs, CellTab interior, SipArrays a,
                             double* fi, const double* su, double* partials, cudaStream_t st) {
  if (interior.nb <= 0) return cudaSuccess;
  pdl_launch(KernelPair{k_sip_residual<false>, k_sip_residual<true>}, interior.ncta, 256, 0, st, bl, offs, interior.cta_start, interior.nb, fi, su, a.res,
             partials);
  const int nb = interior.nb;
  cudaError_t e = P.one ? cluster_launch(k_sip_subst<true>, nb, P.ctas, kSipThreads, P.smem_subst, st, bl, offs, a)
                        : cluster_launch(k_sip_subst<false>, nb, P.ctas, kSipThreads, P.smem_subst, st, bl, offs, a);
  if (e != cudaSuccess) return e;
  pdl_launch(KernelPair{k_sip_correct<false>, k_sip_correct<true>}, interior.ncta, 256, 0, st, bl, offs, interior.cta_start, interior.nb, fi, a.res);
  return cudaGetLastError();
}

// Which TDMA kernel a level takes: whole blocks in shared memory where they fit
// (16x16x24 cells in FP64), else the diagonals around the current one there
// (78^3 in FP64), a CTA a block, else, and with variable coefficients, one thread a
// line in global memory (k_tdma).
TdmaPlan tdma_plan(const std::vector<BlkLev>& bl, bool var, int word) {
  TdmaPlan P;
  if (var) return P;
  long long whole = 0, diag[2] = {0, 0}, lines = 0;  // words; diag: one and two operand buffers
  for (const auto& B : bl) {
    const long long ex[3] = {B.nx, B.ny, B.nz}, mx = std::max(B.nx, std::max(B.ny, B.nz)) + 2;
    long long own = 0;
    whole = std::max(whole, 2LL * tdma_s_sxy(B.nx, B.ny) * (B.nz + 2) + mx * 32);
    for (int axis = 0; axis < 3; ++axis) {
      const long long nu = axis == 0 ? ex[1] : ex[0], nv = axis == 2 ? ex[1] : ex[2], n = ex[axis];
      for (int k = 0; k < 2; ++k)
        diag[k] = std::max(diag[k], 2 * (n + 2) * (nu + 2) + (k + 1) * (2 * (n + 2) + 2) * (nu + 2) + (n + 1) * 32);
      lines = std::max(lines, std::min(nu, nv));
      own = std::max(own, (tdma_rows((int)nu, (int)nv, (int)n) + 15) / 16 * 16);
    }
    P.offs.push_back(P.words);
    P.words += own;
  }
  if (lines > kTdmaThreads) return P;
  if (whole * word <= kTdmaMaxSmem) {
    P.mode = TdmaPlan::kWhole;
    P.smem = (int)(whole * word);
  } else if (diag[0] * word <= kTdmaMaxSmem) {
    P.mode = TdmaPlan::kDiagonals;
    P.nbuf = diag[1] * word <= kTdmaMaxSmem ? 2 : 1;
    P.smem = (int)(diag[P.nbuf - 1] * word);
  }
  return P;
}

template <typename T>
cudaError_t launch_tdma(const TdmaPlan& P, bool zero, const BlkLev* bl, const long long* offs, CellTab all,
                        const T* src, T* dst, const T* rhs, T* scratch, cudaStream_t st) {
  const int nb = all.nb;
  if (nb <= 0) return cudaSuccess;
  if (P.mode == TdmaPlan::kWhole) {
    pdl_launch(k_tdma_s<T>, nb, kTdmaThreads, (size_t)P.smem, st, bl, src, dst, rhs, zero);
    return cudaGetLastError();
  }
  if (P.mode != TdmaPlan::kDiagonals) return cudaErrorInvalidValue;
  const size_t sm = (size_t)P.smem;
  T *a = scratch, *b = a + P.words, *rows = b + P.words;
  pdl_launch(H3D_BOTH(k_tdma_rows, T, -1, 1), all.ncta, 256, 0, st, bl, all.cta_start, nb, src, rhs, b, a, rows, offs, zero);
  pdl_launch(k_tdma_g<T, 1>, nb, kTdmaThreads, sm, st, bl, a, rows, offs, P.nbuf);
  pdl_launch(H3D_BOTH(k_tdma_rows, T, 1, 0), all.ncta, 256, 0, st, bl, all.cta_start, nb, src, rhs, a, b, rows, offs, zero);
  pdl_launch(k_tdma_g<T, 0>, nb, kTdmaThreads, sm, st, bl, b, rows, offs, P.nbuf);
  pdl_launch(H3D_BOTH(k_tdma_rows, T, 0, 2), all.ncta, 256, 0, st, bl, all.cta_start, nb, src, rhs, b, a, rows, offs, zero);
  pdl_launch(k_tdma_g<T, 2>, nb, kTdmaThreads, sm, st, bl, a, rows, offs, P.nbuf);
  pdl_launch(H3D_BOTH(k_tdma_level, T), all.ncta, 256, 0, st, bl, all.cta_start, nb, a, dst, offs);
  return cudaGetLastError();
}
template cudaError_t launch_tdma<double>(const TdmaPlan&, bool, const BlkLev*, const long long*, CellTab, const double*,
                                         double*, const double*, double*, cudaStream_t);
template cudaError_t launch_tdma<float>(const TdmaPlan&, bool, const BlkLev*, const long long*, CellTab, const float*,
                                        float*, const float*, float*, cudaStream_t);

}  // namespace h3d
