// Coarse levels of the V-cycle: relaxation visits of small levels in one launch
// and the fused coarse end (one CTA, or one thread-block cluster).
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "h3d_device.cuh"
#include "h3d_kernels.cuh"

namespace h3d {

// ---------------------------------------------------------------------------
// Several sweeps of a small level (mgrelax with `sweeps` iterations) in one
// CTA, in place: per sweep the red cells (x+y+z odd), a barrier, the black
// cells, a barrier, then the ghost fill from the level's sweep table (every
// entry reads an interior cell, so the gather is order-free in place), a
// barrier.  Same cell values as the out-of-place sweep + fill kernels: the
// FP64 update keeps the reference's operand order and IEEE division.
// zero: the iterate is known zero; it is cleared (ghosts included) first.
// start[b]: first flat interior index of block b (start[nb] = all cells).
// sb / ss: the block table and those starts, in shared memory.
template <typename T, bool VAR>
__device__ void small_relax(const BlkLev* sb, const int* ss, int nb, T* __restrict__ phi, const T* rhs,
                            const T* __restrict__ fx, const T* __restrict__ fy, const T* __restrict__ fz,
                            const uint32_t* __restrict__ fdst, const uint32_t* __restrict__ fsrc, int nfill,
                            int sweeps, int zero, long long nelems, float om, int rb) {
  const int ncell = ss[nb];
  if (zero) {
    for (long long q = threadIdx.x; q < nelems; q += blockDim.x) phi[q] = T(0);
    __syncthreads();
  }
  for (int it = 0; it < sweeps; ++it) {
    for (int colour = 1; colour >= 0; --colour) {  // red (x+y+z odd) first
      for (int c = threadIdx.x; c < ncell; c += blockDim.x) {
        int b = 0;
        while (b + 1 < nb && ss[b + 1] <= c) ++b;
        const BlkLev& B = sb[b];
        const int local = c - ss[b];
        const int x = 1 + local % B.nx, y = 1 + (local / B.nx) % B.ny, z = 1 + local / (B.nx * B.ny);
        if (((x + y + z) & 1) != colour) continue;
        const long long i = B.off + (long long)z * B.sxy + (long long)y * B.sx + x;
        const Coef<T> cf = cell_coef<T, VAR>(B, x, y, z, i - B.off, VAR ? fx + B.off : nullptr,
                                             VAR ? fy + B.off : nullptr, VAR ? fz + B.off : nullptr);
        const T ap = coef_ap(cf);
        T v = gs_div(rhs[i] - (cf.aw * phi[i - 1] + cf.ae * phi[i + 1] + cf.as * phi[i - B.sx] +
                               cf.an * phi[i + B.sx] + cf.ab * phi[i - B.sxy] + cf.at * phi[i + B.sxy]),
                     ap);
        if constexpr (sizeof(T) == 4) v = sorf(phi[i], v, om);
        phi[i] = v;
      }
      __syncthreads();
      if (rb && colour == 1) {  // red-black order across block faces: the new red cells into the ghosts
        for (int q = threadIdx.x; q < nfill; q += blockDim.x) phi[fdst[q]] = phi[fsrc[q] & kIdxMask];
        __syncthreads();
      }
    }
    for (int q = threadIdx.x; q < nfill; q += blockDim.x) phi[fdst[q]] = phi[fsrc[q] & kIdxMask];
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// One update of a cell of a constant-coefficient level: sum of the neighbours in
// the reference's order (FP64), fused in FP32.
__device__ __forceinline__ double cell_update(const double* p, int sx, int sxy, double ax, double ay, double az,
                                              double r, double ap, double inv, float) {
  return div_known(r - (ax * p[-1] + ax * p[1] + ay * p[-sx] + ay * p[sx] + az * p[-sxy] + az * p[sxy]), ap, inv);
}
__device__ __forceinline__ float cell_update(const float* p, int sx, int sxy, float ax, float ay, float az, float r,
                                             float, float inv, float om) {
  const float s = fmaf(az, p[sxy], fmaf(az, p[-sxy], fmaf(ay, p[sx], fmaf(ay, p[-sx], fmaf(ax, p[1], ax * p[-1])))));
  return sorf(p[0], (r - s) * inv, om);
}

// Relaxation of one block in shared memory (compact layout, constant
// coefficients) with its cells resident in registers: a thread owns K pairs of
// x-neighbours, one red and one black cell each, and keeps their places and
// right-hand sides for all sweeps, so that a colour is six loads, the sum, five
// multiply-adds and a store.  (The table-driven form decoded a cell entry,
// selected six coefficients and divided for every update: 1.2 us a colour of 512
// cells in FP64, 0.25 us here.)  The caller has zeroed the ghosts of physical walls, whose
// faces have a zero coefficient, so all cells use the interior ones.
// rhs_at(x, y, z): right-hand side.  fill(last): after the black cells (ncol 2:
// after each colour), a barrier, the ghosts the next sweep reads, or all of them
// after the last sweep, and a barrier.
// diag: 128 words of shared memory (diagonal and reciprocal by wall faces).
template <typename T, int K, typename Rhs, typename Fill>
__device__ __forceinline__ void relax_resident(const BlkLev& B, T* phi, T* diag, Rhs&& rhs_at, int sweeps, float om,
                                               int ncol, Fill&& fill) {
  const int nx = B.nx, ny = B.ny, nz = B.nz, hx = (nx + 1) / 2, np = hx * ny * nz;
  const int sx = nx + 2, sxy = sx * (ny + 2);
  const T ax = (T)B.ax, ay = (T)B.ay, az = (T)B.az;
  if (threadIdx.x < 64) {
    const int m = threadIdx.x;
    Coef<T> c;
    c.aw = m & 1 ? T(0) : ax;
    c.ae = m & 2 ? T(0) : ax;
    c.as = m & 4 ? T(0) : ay;
    c.an = m & 8 ? T(0) : ay;
    c.ab = m & 16 ? T(0) : az;
    c.at = m & 32 ? T(0) : az;
    diag[2 * m] = coef_ap(c);
    diag[2 * m + 1] = T(1) / coef_ap(c);
  }
  int at[2][K];  // place in phi (24 bits), wall faces above
  T r[2][K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const int p = threadIdx.x + j * blockDim.x;
    const int xp = p % hx, y = (p / hx) % ny + 1, z = p / (hx * ny) + 1;
    const int odd = (1 + y + z) & 1;  // the first cell of the pair is red (x+y+z odd)
    const int m = (y == 1 ? 4 : 0) | (y == ny ? 8 : 0) | (z == 1 ? 16 : 0) | (z == nz ? 32 : 0);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int x = 2 * xp + (c == 0 ? 2 - odd : 1 + odd);
      const bool in = p < np && x <= nx;
      const int w = (m | (x == 1 ? 1 : 0) | (x == nx ? 2 : 0)) & B.phys;
      at[c][j] = in ? (z * sxy + y * sx + x) | w << 24 : -1;
      r[c][j] = in ? rhs_at(x, y, z) : T(0);
    }
  }
  __syncthreads();
  for (int it = 0; it < sweeps; ++it) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      T v[K];
#pragma unroll
      for (int j = 0; j < K; ++j)
        if (at[c][j] >= 0) {
          const int w = at[c][j] >> 24;
          v[j] = cell_update(phi + (at[c][j] & 0xffffff), sx, sxy, ax, ay, az, r[c][j], diag[2 * w], diag[2 * w + 1],
                             om);
        }
#pragma unroll
      for (int j = 0; j < K; ++j)
        if (at[c][j] >= 0) phi[at[c][j] & 0xffffff] = v[j];
      if (c == 1) fill(it + 1 == sweeps);
      else if (ncol == 2) fill(false);
      else __syncthreads();
    }
  }
}

// Pairs a thread needs for a block (relax_resident), or 0: more than four.
__device__ __forceinline__ int resident_pairs(const BlkLev& B) {
  const int np = (B.nx + 1) / 2 * B.ny * B.nz, k = (np + (int)blockDim.x - 1) / (int)blockDim.x;
  return k <= 1 ? 1 : k <= 2 ? 2 : k <= 4 ? 4 : 0;
}

// True for the ghost cell (x, y, z) of a physical wall.
__device__ __forceinline__ bool wall_ghost(const BlkLev& B, int x, int y, int z) {
  const int ph = B.phys;
  return (x == 0 && (ph & 1)) || (x == B.nx + 1 && (ph & 2)) || (y == 0 && (ph & 4)) || (y == B.ny + 1 && (ph & 8)) ||
         (z == 0 && (ph & 16)) || (z == B.nz + 1 && (ph & 32));
}

// All sweeps of one relaxation visit of a level whose ghost fill stays inside
// every block (independent blocks, a single block, periodic wraps onto
// itself): one CTA per block, in place, the cell arithmetic of small_relax;
// fill entries of block b are fstart[b] .. fstart[b+1]-1 (sources in block b).
template <typename T, bool VAR>
__global__ void __launch_bounds__(1024) k_relax_blocks(const BlkLev* __restrict__ bls, const int* __restrict__ fstart,
                                                       T* __restrict__ phi, const T* __restrict__ rhs,
                                                       const T* __restrict__ fx, const T* __restrict__ fy,
                                                       const T* __restrict__ fz, const uint32_t* __restrict__ fdst,
                                                       const uint32_t* __restrict__ fsrc, int sweeps, int zero,
                                                       float om) {
  pdl_trigger();
  const BlkLev B = bls[blockIdx.x];
  const int f0 = fstart[blockIdx.x], f1 = fstart[blockIdx.x + 1];
  pdl_wait(phi, rhs);
  if (zero) {
    const long long n = (long long)(B.nz + 2) * B.sxy;
    for (long long q = threadIdx.x; q < n; q += blockDim.x) phi[B.off + q] = T(0);
    __syncthreads();
  }
  const int ncell = B.nx * B.ny * B.nz;
  for (int it = 0; it < sweeps; ++it) {
    for (int colour = 1; colour >= 0; --colour) {  // red (x+y+z odd) first
      for (int c = threadIdx.x; c < ncell; c += blockDim.x) {
        const int x = 1 + c % B.nx, y = 1 + (c / B.nx) % B.ny, z = 1 + c / (B.nx * B.ny);
        if (((x + y + z) & 1) != colour) continue;
        const long long i = B.off + (long long)z * B.sxy + (long long)y * B.sx + x;
        const Coef<T> cf = cell_coef<T, VAR>(B, x, y, z, i - B.off, VAR ? fx + B.off : nullptr,
                                             VAR ? fy + B.off : nullptr, VAR ? fz + B.off : nullptr);
        const T ap = coef_ap(cf);
        T v = gs_div(rhs[i] - (cf.aw * phi[i - 1] + cf.ae * phi[i + 1] + cf.as * phi[i - B.sx] +
                               cf.an * phi[i + B.sx] + cf.ab * phi[i - B.sxy] + cf.at * phi[i + B.sxy]),
                     ap);
        if constexpr (sizeof(T) == 4) v = sorf(phi[i], v, om);
        phi[i] = v;
      }
      __syncthreads();
    }
    for (int q = f0 + threadIdx.x; q < f1; q += blockDim.x) phi[fdst[q]] = phi[fsrc[q] & kIdxMask];
    __syncthreads();
  }
}

// The same visit with the block in shared memory and its cells in registers
// (constant coefficients, at most 4 x 512 cell pairs a block).  cdst / csrc:
// the block's fill entries in the compact layout, those that a sweep reads first
// (live[b] of them).  27 uneven blocks of up to 16^3 cells, 32 FP64 sweeps: 245
// us from global memory, 67 us here.
constexpr int kResidentThreads = 512;
template <typename T>
__global__ void __launch_bounds__(kResidentThreads) k_relax_resident(
    const BlkLev* __restrict__ bls, const int* __restrict__ fstart, const int* __restrict__ live, T* __restrict__ phi,
    const T* __restrict__ rhs, const uint32_t* __restrict__ cdst, const uint32_t* __restrict__ csrc, int sweeps,
    int zero, float om) {
  extern __shared__ __align__(16) unsigned char block_smem[];
  __shared__ T diag[128];
  pdl_trigger();
  const BlkLev B = bls[blockIdx.x];
  const int f0 = fstart[blockIdx.x], f1 = fstart[blockIdx.x + 1], fl = f0 + live[blockIdx.x];
  T* P = reinterpret_cast<T*>(block_smem);
  const int ex = B.nx + 2, ey = B.ny + 2, n = ex * ey * (B.nz + 2);
  pdl_wait(phi, rhs);
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    const int x = q % ex, y = (q / ex) % ey, z = q / (ex * ey);
    if (zero || wall_ghost(B, x, y, z)) P[q] = T(0);
    else cp_async_word(P + q, phi + B.off + (long long)z * B.sxy + (long long)y * B.sx + x);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");  // (relax_resident meets before the first sweep)
  auto rhs_at = [&](int x, int y, int z) { return rhs[B.off + (long long)z * B.sxy + (long long)y * B.sx + x]; };
  auto fill = [&](bool last) {
    __syncthreads();
    const int e = last ? f1 : fl;
    if (e > f0) {
      for (int q = f0 + threadIdx.x; q < e; q += blockDim.x) P[cdst[q]] = P[csrc[q]];
      __syncthreads();
    }
  };
  const int k = resident_pairs(B);
  if (k == 1) relax_resident<T, 1>(B, P, diag, rhs_at, sweeps, om, 1, fill);
  else if (k == 2) relax_resident<T, 2>(B, P, diag, rhs_at, sweeps, om, 1, fill);
  else relax_resident<T, 4>(B, P, diag, rhs_at, sweeps, om, 1, fill);
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    const int x = q % ex, y = (q / ex) % ey, z = q / (ex * ey);
    phi[B.off + (long long)z * B.sxy + (long long)y * B.sx + x] = P[q];
  }
}

template <typename T, bool VAR>
__global__ void __launch_bounds__(1024) k_relax_small(const BlkLev* __restrict__ bls, const int* __restrict__ start,
                                                      int nb, T* __restrict__ phi, const T* __restrict__ rhs,
                                                      const T* __restrict__ fx, const T* __restrict__ fy,
                                                      const T* __restrict__ fz, const uint32_t* __restrict__ fdst,
                                                      const uint32_t* __restrict__ fsrc, int nfill, int sweeps,
                                                      int zero, long long nelems, float om, int rb) {
  pdl_trigger();
  __shared__ BlkLev sb[kSmallLevelBlocks];
  __shared__ int ss[kSmallLevelBlocks + 1];
  // the block table and cell starts are written once at setup: read them
  // while the predecessor finishes
  for (int b = threadIdx.x; b < nb; b += blockDim.x) sb[b] = bls[b];
  for (int b = threadIdx.x; b <= nb; b += blockDim.x) ss[b] = start[b];
  pdl_wait(phi, rhs);
  __syncthreads();
  small_relax<T, VAR>(sb, ss, nb, phi, rhs, fx, fy, fz, fdst, fsrc, nfill, sweeps, zero, nelems, om, rb);
}

// The fused coarse tail keeps every tail level in shared memory, in a
// compact layout: the iterate as the padded blocks back to back (block b at
// cbl[b].off, pitches nx+2 and (nx+2)(ny+2)), the rhs as the interior cells
// in natural order (block b from cbl[b].pad).  Cells come from per-level
// tables built at setup, one 64-bit entry a cell: compact index (bits 0-23),
// x, y, z (bits 24-31, 32-39, 40-47) and block (bits 48-53); interior
// tables list the red cells (x+y+z odd) first.
struct CellRef {
  int i, x, y, z, b;
};
__device__ __forceinline__ CellRef cell_ref(unsigned long long e) {
  CellRef c;
  c.i = (int)(e & 0xffffffull);
  c.x = (int)((e >> 24) & 0xff);
  c.y = (int)((e >> 32) & 0xff);
  c.z = (int)((e >> 40) & 0xff);
  c.b = (int)((e >> 48) & 0x3f);
  return c;
}
__device__ __forceinline__ int rhs_index(const BlkLev& B, int x, int y, int z) {
  return B.pad + ((z - 1) * B.ny + (y - 1)) * B.nx + (x - 1);
}
__device__ __forceinline__ long long global_index(const BlkLev& G, int x, int y, int z) {
  return G.off + (long long)z * G.sxy + (long long)y * G.sx + x;
}

// The red then the black cells of one in-place sweep of a tail level; same
// cell arithmetic as small_relax.
template <typename T>
__device__ void tail_colours(const BlkLev* cb, const TailLevel& L, T* phi, const T* rhs, int only = -1) {
  for (int colour = 0; colour < 2; ++colour) {  // red (x+y+z odd) first
    if (only >= 0 && colour != only) continue;
    const int k0 = colour ? L.nred : 0, k1 = colour ? L.nint : L.nred;
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
      const CellRef c = cell_ref(L.cells[k]);
      const BlkLev& B = cb[c.b];
      const int i = c.i;
      const Coef<T> cf = cell_coef<T, false>(B, c.x, c.y, c.z, i - B.off, nullptr, nullptr, nullptr);
      const T ap = coef_ap(cf);
      T v = gs_div(rhs[rhs_index(B, c.x, c.y, c.z)] -
                       (cf.aw * phi[i - 1] + cf.ae * phi[i + 1] + cf.as * phi[i - B.sx] +
                        cf.an * phi[i + B.sx] + cf.ab * phi[i - B.sxy] + cf.at * phi[i + B.sxy]),
                   ap);
      if constexpr (sizeof(T) == 4) v = sorf(phi[i], v, L.om);
      phi[i] = v;
    }
    __syncthreads();
  }
}

// `sweeps` in-place red-black sweeps of a tail level, each followed by its
// ghost fill.
template <typename T>
__device__ void tail_relax(const BlkLev* cb, const TailLevel& L, T* phi, const T* rhs, int sweeps) {
  for (int it = 0; it < sweeps; ++it) {
    if (L.rb_global) {  // a fill after each colour: the red-black order across block faces
      for (int colour = 0; colour < 2; ++colour) {
        tail_colours<T>(cb, L, phi, rhs, colour);
        for (int q = threadIdx.x; q < L.nfill; q += blockDim.x) phi[L.fdst[q]] = phi[L.fsrc[q]];
        __syncthreads();
      }
      continue;
    }
    tail_colours<T>(cb, L, phi, rhs);
    for (int q = threadIdx.x; q < L.nfill; q += blockDim.x) phi[L.fdst[q]] = phi[L.fsrc[q]];
    __syncthreads();
  }
}

// mgrestr into a tail level: the same residual sum over the eight children,
// in the same order, as k_restrict; one thread a coarse cell.
template <typename T>
__device__ void tail_restrict(const BlkLev* fb, const BlkLev* cb, const TailLevel& Cl, const T* phi, const T* rhs,
                              T* rhs_c, int zero_fine) {
  for (int k = threadIdx.x; k < Cl.nint; k += blockDim.x) {
    const CellRef cc = cell_ref(Cl.cells[k]);
    const BlkLev& F = fb[cc.b];
    const int X = cc.x, Y = cc.y, Z = cc.z;
    const T* P = phi + F.off;
    T sum = T(0);
#pragma unroll
    for (int dk = 0; dk < 2; ++dk)
#pragma unroll
      for (int dj = 0; dj < 2; ++dj)
#pragma unroll
        for (int di = 0; di < 2; ++di) {
          const int x = 2 * X - 1 + di, y = 2 * Y - 1 + dj, z = 2 * Z - 1 + dk;
          const int i = z * (int)F.sxy + y * F.sx + x;
          const T rv = rhs[rhs_index(F, x, y, z)];
          T r;
          if (zero_fine) {
            r = rv - T(0);
          } else {
            Coef<T> cf = cell_coef<T, false>(F, x, y, z, i, nullptr, nullptr, nullptr);
            const T ap = coef_ap(cf);
            r = rv - (cf.aw * P[i - 1] + cf.ae * P[i + 1] + cf.as * P[i - F.sx] + cf.an * P[i + F.sx] +
                      cf.ab * P[i - F.sxy] + cf.at * P[i + F.sxy] + ap * P[i]);
          }
          sum = (di | dj | dk) ? sum + r : r;
        }
    rhs_c[rhs_index(cb[cc.b], X, Y, Z)] = T(0.125) * sum;
  }
  __syncthreads();
}

// mgcorr + mgbound of cell (x, y, z) (ghosts included) of block F: the value
// k_prolong writes there, reading the old iterate from `old`.
template <typename T>
__device__ __forceinline__ T tail_prolong_value(const BlkLev& F, const BlkLev& C, const T* phi_c, const T* old, int x,
                                                int y, int z, int zero_old) {
  const int ph = F.phys;
  int sx = x, sy = y, sz = z;
  if (x == 0 && (ph & 1)) sx = 1;
  if (x == F.nx + 1 && (ph & 2)) sx = F.nx;
  if (y == 0 && (ph & 4)) sy = 1;
  if (y == F.ny + 1 && (ph & 8)) sy = F.ny;
  if (z == 0 && (ph & 16)) sz = 1;
  if (z == F.nz + 1 && (ph & 32)) sz = F.nz;
  const T wx0 = (sx & 1) ? T(1) : T(3), wx1 = (sx & 1) ? T(3) : T(1);
  const T wy0 = (sy & 1) ? T(1) : T(3), wy1 = (sy & 1) ? T(3) : T(1);
  const T wz0 = (sz & 1) ? T(1) : T(3), wz1 = (sz & 1) ? T(3) : T(1);
  const int cy = C.sx, cz = (int)C.sxy;
  const T* Q = phi_c + C.off + (sz >> 1) * cz + (sy >> 1) * cy + (sx >> 1);
  // term order (di,dj,dk): 000, 010, 001, 011, 100, 110, 101, 111
  T s = (wx0 * wy0 * wz0) * Q[0];
  s = s + (wx0 * wy1 * wz0) * Q[cy];
  s = s + (wx0 * wy0 * wz1) * Q[cz];
  s = s + (wx0 * wy1 * wz1) * Q[cy + cz];
  s = s + (wx1 * wy0 * wz0) * Q[1];
  s = s + (wx1 * wy1 * wz0) * Q[1 + cy];
  s = s + (wx1 * wy0 * wz1) * Q[1 + cz];
  s = s + (wx1 * wy1 * wz1) * Q[1 + cy + cz];
  const T o = zero_old ? T(0) : old[F.off + sz * (int)F.sxy + sy * F.sx + sx];
  return o + s / T(64);
}

// mgcorr + mgbound into a tail level in place: the ghost cells read interior
// and ghost cells of the old iterate, so their new values go to `scratch`
// (one value a ghost-table entry) first; then the interior cells (each reads
// only itself) update in place, then the ghosts are copied back.
template <typename T>
__device__ void tail_prolong(const BlkLev* fb, const BlkLev* cb, const TailLevel& F, const T* phi_c, T* phi,
                             T* scratch, int zero_old) {
  for (int k = threadIdx.x; k < F.nghost; k += blockDim.x) {
    const CellRef c = cell_ref(F.ghosts[k]);
    scratch[k] = tail_prolong_value(fb[c.b], cb[c.b], phi_c, phi, c.x, c.y, c.z, zero_old);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < F.nint; k += blockDim.x) {
    const CellRef c = cell_ref(F.cells[k]);
    phi[c.i] = tail_prolong_value(fb[c.b], cb[c.b], phi_c, phi, c.x, c.y, c.z, zero_old);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < F.nghost; k += blockDim.x) phi[(int)(F.ghosts[k] & 0xffffffull)] = scratch[k];
  __syncthreads();
}

// The rhs of a tail level from global memory (the restriction into the
// first tail level ran outside); eight loads in flight a thread.
template <typename T>
__device__ void tail_load_rhs(const BlkLev* gb, const BlkLev* cb, const TailLevel& L, const T* g, T* rhs) {
  constexpr int U = 8;
  for (int k0 = threadIdx.x; k0 < L.nint; k0 += U * blockDim.x) {
    T v[U];
    int ri[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * blockDim.x;
      ri[u] = -1;
      if (k < L.nint) {
        const CellRef c = cell_ref(L.cells[k]);
        v[u] = g[global_index(gb[c.b], c.x, c.y, c.z)];
        ri[u] = rhs_index(cb[c.b], c.x, c.y, c.z);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (ri[u] >= 0) rhs[ri[u]] = v[u];
  }
  __syncthreads();
}

// A tail level back to global memory: iterate (interior and ghost cells) and rhs.
template <typename T>
__device__ void tail_store(const BlkLev* gb, const BlkLev* cb, const TailLevel& L, const T* phi, const T* rhs,
                           T* __restrict__ gphi, T* __restrict__ grhs) {
  for (int k = threadIdx.x; k < L.nint + L.nghost; k += blockDim.x) {
    const CellRef c = cell_ref(k < L.nint ? L.cells[k] : L.ghosts[k - L.nint]);
    const long long gi = global_index(gb[c.b], c.x, c.y, c.z);
    gphi[gi] = phi[c.i];
    if (k < L.nint) grhs[gi] = rhs[rhs_index(cb[c.b], c.x, c.y, c.z)];
  }
  __syncthreads();
}

// The coarse end of a V-cycle in one CTA, every level in shared memory: the
// relaxations, restrictions, precision conversions and corrections of the
// tail levels run as the ops of a program built on the host, in order, with
// the CTA's barriers between them instead of kernel boundaries; one op loads
// the first tail level's rhs, the last ones store every tail level.
// curmask bit 2l (2l+1) selects the global FP32 (FP64) iterate buffer of
// tail level l.
__global__ void __launch_bounds__(1024) k_coarse_tail(const TailLevel* __restrict__ lv, const TailOp* __restrict__ ops,
                                                      int nops, unsigned curmask) {
  pdl_trigger();
  __shared__ BlkLev fb[kSmallLevelBlocks], cb[kSmallLevelBlocks], gb[kSmallLevelBlocks];
  extern __shared__ unsigned char smem_raw[];
  unsigned char* arena = smem_base128(smem_raw);
  pdl_wait();
  for (int o = 0; o < nops; ++o) {
    const TailOp op = ops[o];
    const TailLevel& F = lv[op.fine];
    const TailLevel& C = lv[op.coarse];
    const int nb = F.nb;
    __syncthreads();  // the previous op is done with the tables
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
      fb[b] = F.cbl[b];
      cb[b] = C.cbl[b];
      gb[b] = F.gbl[b];
    }
    __syncthreads();
    auto at32 = [&](int off) { return reinterpret_cast<float*>(arena + off); };
    auto at64 = [&](int off) { return reinterpret_cast<double*>(arena + off); };
    switch (op.kind) {
      case kTailLoadRhs:
        if (op.f64) tail_load_rhs<double>(gb, fb, F, F.rhs64, at64(F.s_rhs64));
        else tail_load_rhs<float>(gb, fb, F, F.rhs32, at32(F.s_rhs32));
        break;
      case kTailRelax:
        if (op.f64) {
          double* phi = at64(F.s_phi64);
          if (op.zero) {
            for (int q = threadIdx.x; q < F.npad; q += blockDim.x) phi[q] = 0.0;
            __syncthreads();
          }
          tail_relax<double>(fb, F, phi, at64(F.s_rhs64), op.sweeps);
        } else {
          float* phi = at32(F.s_phi32);
          if (op.zero) {
            for (int q = threadIdx.x; q < F.npad; q += blockDim.x) phi[q] = 0.f;
            __syncthreads();
          }
          tail_relax<float>(fb, F, phi, at32(F.s_rhs32), op.sweeps);
        }
        break;
      case kTailRestrict:  // into the coarse rhs of the fine level's precision
        if (op.f64) tail_restrict<double>(fb, cb, C, at64(F.s_phi64), at64(F.s_rhs64), at64(C.s_rhs64), op.zero);
        else tail_restrict<float>(fb, cb, C, at32(F.s_phi32), at32(F.s_rhs32), at32(C.s_rhs32), op.zero);
        break;
      case kTailProlong:
        if (op.f64)
          tail_prolong<double>(fb, cb, F, at64(C.s_phi64), at64(F.s_phi64), at64(op.sweeps), op.zero);
        else
          tail_prolong<float>(fb, cb, F, at32(C.s_phi32), at32(F.s_phi32), at32(op.sweeps), op.zero);
        break;
      case kTailRhsF2D: {  // the coarsest rhs of a mixed solve to FP64
        const float* a = at32(F.s_rhs32);
        double* b = at64(F.s_rhs64);
        for (int q = threadIdx.x; q < F.nint; q += blockDim.x) b[q] = (double)a[q];
        __syncthreads();
        break;
      }
      case kTailPhiD2F: {  // the coarsest iterate of a mixed solve to FP32
        const double* a = at64(F.s_phi64);
        float* b = at32(F.s_phi32);
        for (int q = threadIdx.x; q < F.npad; q += blockDim.x) b[q] = (float)a[q];
        __syncthreads();
        break;
      }
      case kTailStore: {
        const int c32 = (curmask >> (2 * op.fine)) & 1, c64 = (curmask >> (2 * op.fine + 1)) & 1;
        if (F.s_phi32 >= 0) tail_store<float>(gb, fb, F, at32(F.s_phi32), at32(F.s_rhs32), F.phi32[c32], F.rhs32);
        if (F.s_phi64 >= 0) tail_store<double>(gb, fb, F, at64(F.s_phi64), at64(F.s_rhs64), F.phi64[c64], F.rhs64);
        break;
      }
      default:
        break;
    }
  }
}

// ---------------------------------------------------------------------------
// The coarse end of a V-cycle as one thread-block cluster: CTA b holds block
// b of every tail level in its shared memory (compact layout, every block of
// a level the same size) and runs the same op program as k_coarse_tail on
// it.  Restrictions, corrections and conversions only touch the CTA's own
// block; after the colours of a sweep the cluster synchronises, every CTA
// gathers its ghost cells from the other CTAs' shared memory (fill pairs: own
// compact index; source rank << 24 | its compact index), and the cluster
// synchronises again before any interior changes.
//
// Latency bounds it: a program of short ops on a few thousand cells, every
// instruction fetched cold.  So the code is kept small and a cell cheap: cells come
// from 32-bit tables (x, y, z, and the block faces the cell lies on), red before
// black, and right-hand sides are stored in the tables' order; the diagonal and its
// reciprocal come from a table by wall faces, so that an update divides by
// multiply-adds (div_known); all tables are staged by one flat copy while the predecessor
// finishes; a sweep fills the ghosts that the next one reads, the last one all of
// them.  With 64-bit tables decoded through the block records a launch took 67 us for
// 16 blocks of 16^3 .. 2^3 cells and 46 us for one of 16^3 and 8^3 cells in FP64; 58
// (512 threads a CTA) and 34 us (1024) here.
//
// Sweeps of a visit from which its cells go to registers (the 32 of a converged
// coarsest level; two or three sweeps do not repay the extra code).
constexpr int kResidentSweeps = 8;
struct Cell3 {
  int x, y, z, w;  // w: block faces (bit f)
};
__device__ __forceinline__ Cell3 cell3(uint32_t e) {
  return Cell3{(int)(e & 0xff), (int)(e >> 8 & 0xff), (int)(e >> 16 & 0xff), (int)(e >> 24)};
}
__device__ __forceinline__ int compact_at(const BlkLev& B, int x, int y, int z) {
  return (z * (B.ny + 2) + y) * (B.nx + 2) + x;
}
// Place of a cell's right-hand side: the tables list cells in natural order,
// red ones first, and every two neighbours in that order are one of each.
__device__ __forceinline__ int rhs_at(const BlkLev& B, int nred, int x, int y, int z) {
  return ((x + y + z) & 1 ? 0 : nred) + ((((z - 1) * B.ny + (y - 1)) * B.nx + (x - 1)) >> 1);
}

// One colour (0: red) of a sweep.  The ghosts of physical walls are zero, so
// all cells use the interior coefficients.
template <typename T>
__device__ void cluster_colour(const BlkLev& B, const TailLevel& L, T* phi, const T* rhs, const T* diag, int colour) {
  const int sx = B.nx + 2, sxy = sx * (B.ny + 2), k1 = colour ? L.nint : L.nred;
  const T ax = (T)B.ax, ay = (T)B.ay, az = (T)B.az;
  for (int k = (colour ? L.nred : 0) + threadIdx.x; k < k1; k += blockDim.x) {
    const Cell3 c = cell3(L.cells32[k]);
    T* q = phi + compact_at(B, c.x, c.y, c.z);
    const int w = c.w & B.phys;
    *q = cell_update(q, sx, sxy, ax, ay, az, rhs[k], diag[2 * w], diag[2 * w + 1], L.om);
  }
}

// mgrestr into a tail level: the residual sum over the eight children in
// k_restrict's order; one thread a coarse cell.
template <typename T>
__device__ void cluster_restrict(const BlkLev& F, const TailLevel& Fl, const TailLevel& Cl, const T* P, const T* rhs,
                                 T* rhs_c, int zero_fine) {
  const int sx = F.nx + 2, sxy = sx * (F.ny + 2);
  for (int k = threadIdx.x; k < Cl.nint; k += blockDim.x) {
    const Cell3 cc = cell3(Cl.cells32[k]);
    T sum = T(0);
#pragma unroll 1
    for (int d = 0; d < 8; ++d) {
      const int x = 2 * cc.x - 1 + (d & 1), y = 2 * cc.y - 1 + (d >> 1 & 1), z = 2 * cc.z - 1 + (d >> 2);
      T r = rhs[rhs_at(F, Fl.nred, x, y, z)];
      if (!zero_fine) {
        const T* q = P + compact_at(F, x, y, z);
        const Coef<T> cf = cell_coef<T, false>(F, x, y, z, 0, nullptr, nullptr, nullptr);
        r = r - (cf.aw * q[-1] + cf.ae * q[1] + cf.as * q[-sx] + cf.an * q[sx] + cf.ab * q[-sxy] + cf.at * q[sxy] +
                 coef_ap(cf) * q[0]);
      }
      sum = d ? sum + r : r;
    }
    rhs_c[k] = T(0.125) * sum;
  }
  __syncthreads();
}

// mgcorr + mgbound into a tail level in place (see tail_prolong).
template <typename T>
__device__ void cluster_prolong(const BlkLev& F, const BlkLev& C, const TailLevel& L, const T* phi_c, T* phi,
                                T* scratch, int zero_old) {
  for (int k = threadIdx.x; k < L.nghost; k += blockDim.x) {
    const Cell3 c = cell3(L.cells32[L.nint + k]);
    scratch[k] = tail_prolong_value(F, C, phi_c, phi, c.x, c.y, c.z, zero_old);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < L.nint; k += blockDim.x) {
    const Cell3 c = cell3(L.cells32[k]);
    phi[compact_at(F, c.x, c.y, c.z)] = tail_prolong_value(F, C, phi_c, phi, c.x, c.y, c.z, zero_old);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < L.nghost; k += blockDim.x) {
    const Cell3 c = cell3(L.cells32[L.nint + k]);
    phi[compact_at(F, c.x, c.y, c.z)] = scratch[k];
  }
  __syncthreads();
}

// A tail level back to global memory: iterate (interior and ghost cells) and rhs.
template <typename T>
__device__ void cluster_store(const BlkLev& G, const BlkLev& B, const TailLevel& L, const T* phi, const T* rhs,
                              T* __restrict__ gphi, T* __restrict__ grhs) {
  for (int k = threadIdx.x; k < L.nint + L.nghost; k += blockDim.x) {
    const Cell3 c = cell3(L.cells32[k]);
    const long long gi = global_index(G, c.x, c.y, c.z);
    gphi[gi] = phi[compact_at(B, c.x, c.y, c.z)];
    if (k < L.nint) grhs[gi] = rhs[k];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kClusterTailThreads) k_coarse_cluster(const TailLevel* __restrict__ lvg,
                                                                        const TailOp* __restrict__ opsg,
                                                                        const uint4* __restrict__ tables, int nops,
                                                                        int nlev, unsigned curmask) {
  pdl_trigger();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int b = (int)cl.block_rank();
  __shared__ TailLevel lv[kTailMaxLevels];
  __shared__ BlkLev gtab[kTailMaxLevels], ctab[kTailMaxLevels];  // this block per level: global / compact layout
  __shared__ TailOp ops[kClusterTailMaxOps];
  __shared__ double diag64[128];  // diagonal and reciprocal by wall faces
  extern __shared__ unsigned char smem_raw[];
  unsigned char* arena = smem_base128(smem_raw);
  // the program, the level records and this block's tables are setup data: staged
  // while the predecessor finishes
  {
    const int tab0 = lvg[0].s_cells, words = lvg[0].tab_words;
    uint4* dst = reinterpret_cast<uint4*>(arena + tab0);
    for (int q = threadIdx.x; q < words; q += blockDim.x) dst[q] = __ldg(tables + (size_t)b * words + q);
    for (int q = threadIdx.x; q < nops; q += blockDim.x) ops[q] = opsg[q];
    if (threadIdx.x < nlev) {
      TailLevel l = lvg[threadIdx.x];
      l.nfill = __ldg(l.fstart + b + 1) - __ldg(l.fstart + b);
      l.nlive = __ldg(l.flive + b);
      l.cells32 = reinterpret_cast<const uint32_t*>(arena + l.s_cells);
      l.fdst = reinterpret_cast<const uint32_t*>(arena + l.s_fill);
      lv[threadIdx.x] = l;
      const BlkLev G = l.gbl[b];
      gtab[threadIdx.x] = G;
      BlkLev c = G;
      c.off = 0;
      c.sx = G.nx + 2;
      c.sxy = (long long)(G.nx + 2) * (G.ny + 2);
      c.pad = 0;
      ctab[threadIdx.x] = c;
    }
  }
  __syncthreads();
  pdl_wait();
  const bool alone = cl.num_blocks() == 1;
  auto barrier = [&] {
    if (alone) __syncthreads();
    else cl.sync();
  };
  // ghosts of the first n fill pairs from every block's interior
  auto gather = [&](const TailLevel& F, auto* phi, int n) {
    barrier();  // every block's cells are written
    for (int q = threadIdx.x; q < n; q += blockDim.x) {  // (dst, src) pairs of this block
      const uint32_t src = F.fdst[2 * q + 1];
      phi[F.fdst[2 * q]] = cl.map_shared_rank(phi, (int)(src >> 24))[src & 0xffffffu];
    }
    barrier();  // every ghost gathered before any interior changes
  };
  for (int o = 0; o < nops; ++o) {
    const TailOp op = ops[o];
    const TailLevel& F = lv[op.fine];
    const TailLevel& C = lv[op.coarse];
    // this block's tables at the op's levels (staged once; every op ends with
    // a barrier of the CTA or the cluster)
    const BlkLev& gb = gtab[op.fine];
    const BlkLev& fb = ctab[op.fine];
    const BlkLev& cb = ctab[op.coarse];
    auto at32 = [&](int off) { return reinterpret_cast<float*>(arena + off); };
    auto at64 = [&](int off) { return reinterpret_cast<double*>(arena + off); };
    switch (op.kind) {
      case kTailLoadRhs: {
        auto load = [&](const auto* g, auto* rhs) {
#pragma unroll 4
          for (int k = threadIdx.x; k < F.nint; k += blockDim.x) {
            const Cell3 c = cell3(F.cells32[k]);
            rhs[k] = g[global_index(gb, c.x, c.y, c.z)];
          }
        };
        if (op.f64) load(F.rhs64, at64(F.s_rhs64));
        else load(F.rhs32, at32(F.s_rhs32));
        __syncthreads();
        break;
      }
      case kTailRelax: {
        auto relax = [&](auto* phi, const auto* rhs) {
          using T = typename std::remove_pointer<decltype(phi)>::type;
          T* diag = reinterpret_cast<T*>(diag64);
          if (threadIdx.x < 64) {
            Coef<T> c;
            c.aw = threadIdx.x & 1 ? T(0) : (T)fb.ax;
            c.ae = threadIdx.x & 2 ? T(0) : (T)fb.ax;
            c.as = threadIdx.x & 4 ? T(0) : (T)fb.ay;
            c.an = threadIdx.x & 8 ? T(0) : (T)fb.ay;
            c.ab = threadIdx.x & 16 ? T(0) : (T)fb.az;
            c.at = threadIdx.x & 32 ? T(0) : (T)fb.az;
            diag[2 * threadIdx.x] = coef_ap(c);
            diag[2 * threadIdx.x + 1] = T(1) / coef_ap(c);
          }
          if (op.zero) {
            for (int q = threadIdx.x; q < F.npad; q += blockDim.x) phi[q] = T(0);
          } else {
            for (int q = threadIdx.x; q < F.nghost; q += blockDim.x) {
              const Cell3 c = cell3(F.cells32[F.nint + q]);
              if (c.w & fb.phys) phi[compact_at(fb, c.x, c.y, c.z)] = T(0);
            }
          }
          __syncthreads();
          if constexpr (sizeof(T) == 8) {
            // many sweeps (the converged coarsest level): one red and one black cell a
            // thread, kept in registers; a block alone only has the warps with cells meet
            if (op.sweeps >= kResidentSweeps && F.nred <= (int)blockDim.x) {
              const int na = alone ? (F.nred + 31) / 32 * 32 : (int)blockDim.x;
              if ((int)threadIdx.x < na) {
                auto meet = [&] { asm volatile("bar.sync 1, %0;\n" ::"r"(na) : "memory"); };
                const int sx = fb.nx + 2, sxy = sx * (fb.ny + 2);
                int at[2];
                T r[2], ap[2], inv[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                  const int k = threadIdx.x + (c ? F.nred : 0);
                  const bool in = (int)threadIdx.x < F.nred && k < F.nint;
                  const Cell3 q = cell3(F.cells32[in ? k : 0]);
                  at[c] = in ? compact_at(fb, q.x, q.y, q.z) : -1;
                  r[c] = in ? rhs[k] : T(0);
                  ap[c] = diag[2 * (q.w & fb.phys)];
                  inv[c] = diag[2 * (q.w & fb.phys) + 1];
                }
                for (int it = 0; it < op.sweeps; ++it)
#pragma unroll
                  for (int c = 0; c < 2; ++c) {
                    if (at[c] >= 0)
                      phi[at[c]] = cell_update(phi + at[c], sx, sxy, fb.ax, fb.ay, fb.az, r[c], ap[c], inv[c], 1.f);
                    const bool last = c && it + 1 == op.sweeps;
                    const int n = last ? F.nfill : F.any_live && (c || F.rb_global) ? F.nlive : -1;
                    if (!alone && n >= 0) {
                      gather(F, phi, n);
                    } else {
                      meet();
                      for (int q = threadIdx.x; q < n; q += na) phi[F.fdst[2 * q]] = phi[F.fdst[2 * q + 1] & 0xffffffu];
                      if (n > 0) meet();
                    }
                  }
              }
              __syncthreads();
              return;
            }
          }
          for (int it = 0; it < op.sweeps; ++it)
            for (int colour = 0; colour < 2; ++colour) {
              cluster_colour<T>(fb, F, phi, rhs, diag, colour);
              const bool last = colour && it + 1 == op.sweeps;
              // a fill after each colour: the order across block faces; else after the black
              // cells; all ghosts after the last, before that the ones a sweep reads
              if (last) gather(F, phi, F.nfill);
              else if (F.any_live && (colour || F.rb_global)) gather(F, phi, F.nlive);
              else __syncthreads();
            }
        };
        if (op.f64) relax(at64(F.s_phi64), (const double*)at64(F.s_rhs64));
        else relax(at32(F.s_phi32), (const float*)at32(F.s_rhs32));
        break;
      }
      case kTailDense: {  // x = P b over the cells of every block (FP64), then the sweep fill
        double* phi = at64(F.s_phi64);
        const double* rhs = at64(F.s_rhs64);
        if (op.zero) {
          for (int q = threadIdx.x; q < F.npad; q += blockDim.x) phi[q] = 0.0;
        }
        barrier();  // every block's rhs is complete
        const int nper = F.nint, n = F.dense_n;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
        for (int i = warp; i < nper; i += nwarp) {  // a warp per row of this block; lanes split the columns
          const Cell3 c = cell3(F.cells32[i]);
          const int row = ((c.z - 1) * fb.ny + (c.y - 1)) * fb.nx + (c.x - 1);
          const double* Pr = F.dense + (long long)(b * nper + row) * n;
          double s = 0.0;
          for (int j = lane; j < n; j += 32) {
            const double* r = cl.map_shared_rank(rhs, j / nper);
            s += __ldg(Pr + j) * r[j % nper];
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == 0) phi[compact_at(fb, c.x, c.y, c.z)] = s;
        }
        gather(F, phi, F.nfill);
        break;
      }
      case kTailRestrict:
        if (op.f64) cluster_restrict<double>(fb, F, C, at64(F.s_phi64), at64(F.s_rhs64), at64(C.s_rhs64), op.zero);
        else cluster_restrict<float>(fb, F, C, at32(F.s_phi32), at32(F.s_rhs32), at32(C.s_rhs32), op.zero);
        break;
      case kTailProlong:
        if (op.f64) cluster_prolong<double>(fb, cb, F, at64(C.s_phi64), at64(F.s_phi64), at64(op.sweeps), op.zero);
        else cluster_prolong<float>(fb, cb, F, at32(C.s_phi32), at32(F.s_phi32), at32(op.sweeps), op.zero);
        break;
      case kTailRhsF2D: {
        const float* x = at32(F.s_rhs32);
        double* y = at64(F.s_rhs64);
        for (int q = threadIdx.x; q < F.nint; q += blockDim.x) y[q] = (double)x[q];
        __syncthreads();
        break;
      }
      case kTailPhiD2F: {
        const double* x = at64(F.s_phi64);
        float* y = at32(F.s_phi32);
        for (int q = threadIdx.x; q < F.npad; q += blockDim.x) y[q] = (float)x[q];
        __syncthreads();
        break;
      }
      case kTailStore: {
        const int c32 = (curmask >> (2 * op.fine)) & 1, c64 = (curmask >> (2 * op.fine + 1)) & 1;
        if (F.s_phi32 >= 0) cluster_store<float>(gb, fb, F, at32(F.s_phi32), at32(F.s_rhs32), F.phi32[c32], F.rhs32);
        if (F.s_phi64 >= 0) cluster_store<double>(gb, fb, F, at64(F.s_phi64), at64(F.s_rhs64), F.phi64[c64], F.rhs64);
        break;
      }
      default:
        break;
    }
  }
  if (!alone) cl.sync();  // no CTA leaves while another may still read its shared memory
}

cudaError_t coarse_tail_attributes() {
  cudaError_t e = cudaFuncSetAttribute(k_coarse_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmemBytes);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_relax_resident<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmemBytes);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_relax_resident<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmemBytes);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_coarse_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmemBytes);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_coarse_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

static cudaError_t cluster_config(int nb, int threads, int smem_bytes, cudaStream_t st, cudaLaunchConfig_t* cfg,
                                  cudaLaunchAttribute* at) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(nb);
  cfg->blockDim = dim3(threads);
  cfg->dynamicSmemBytes = (size_t)smem_bytes;
  cfg->stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = nb;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg->attrs = at;
  cfg->numAttrs = 1;
  return cudaSuccess;
}

int coarse_cluster_fits(int nb, int threads, int smem_bytes) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  cluster_config(nb, threads, smem_bytes, nullptr, &cfg, at);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k_coarse_cluster, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

cudaError_t launch_coarse_cluster(int nb, int threads, const TailLevel* lv, int nlev, const TailOp* ops, int nops,
                                  const uint4* tables, unsigned curmask, int smem_bytes, cudaStream_t st) {
  if (nops <= 0 || nops > kClusterTailMaxOps || nlev > kTailMaxLevels) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  cluster_config(nb, threads, smem_bytes, st, &cfg, at);
  cfg.numAttrs = pdl_mode() == 0 ? 1 : 2;  // (its tables are staged while the predecessor finishes)
  g_prev_grid = nb;
  return cudaLaunchKernelEx(&cfg, k_coarse_cluster, lv, ops, tables, nops, nlev, curmask);
}

cudaError_t launch_coarse_tail(const TailLevel* lv, const TailOp* ops, int nops, unsigned curmask, int smem_bytes,
                               cudaStream_t st) {
  if (nops <= 0) return cudaSuccess;
  pdl_launch(k_coarse_tail, 1, 1024, (size_t)smem_bytes, st, lv, ops, nops, curmask);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_relax_small(bool var, const BlkLev* bl, const int* start, int nb, T* phi, const T* rhs,
                               const T* fx, const T* fy, const T* fz, const uint32_t* fdst, const uint32_t* fsrc,
                               int nfill, int sweeps, bool zero, long long nelems, float om, bool rb,
                               cudaStream_t st) {
  if (var)
    pdl_launch(k_relax_small<T, true>, 1, 1024, 0, st, bl, start, nb, phi, rhs, fx, fy, fz, fdst, fsrc, nfill, sweeps,
               (int)zero, nelems, om, (int)rb);
  else
    pdl_launch(k_relax_small<T, false>, 1, 1024, 0, st, bl, start, nb, phi, rhs, fx, fy, fz, fdst, fsrc, nfill,
               sweeps, (int)zero, nelems, om, (int)rb);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_relax_blocks(bool var, const BlkLev* bl, int nb, const int* fstart, T* phi, const T* rhs,
                                const T* fx, const T* fy, const T* fz, const uint32_t* fdst, const uint32_t* fsrc,
                                int sweeps, bool zero, float om, cudaStream_t st) {
  if (nb <= 0) return cudaSuccess;
  if (var)
    pdl_launch(k_relax_blocks<T, true>, nb, 1024, 0, st, bl, fstart, phi, rhs, fx, fy, fz, fdst, fsrc, sweeps,
               (int)zero, om);
  else
    pdl_launch(k_relax_blocks<T, false>, nb, 1024, 0, st, bl, fstart, phi, rhs, fx, fy, fz, fdst, fsrc, sweeps,
               (int)zero, om);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_relax_resident(const BlkLev* bl, int nb, const int* fstart, const int* live, T* phi, const T* rhs,
                                  const uint32_t* cdst, const uint32_t* csrc, int smem, int sweeps, bool zero,
                                  float om, cudaStream_t st) {
  if (nb <= 0) return cudaSuccess;
  pdl_launch(k_relax_resident<T>, nb, kResidentThreads, (size_t)smem, st, bl, fstart, live, phi, rhs, cdst, csrc,
             sweeps, (int)zero, om);
  return cudaGetLastError();
}
// Shared memory of launch_relax_resident for these blocks, or 0 where one does not fit it.
int resident_smem(const std::vector<BlkLev>& bl, int word) {
  long long n = 0;
  for (const auto& B : bl) {
    if ((long long)(B.nx + 1) / 2 * B.ny * B.nz > 4 * kResidentThreads) return 0;
    n = std::max(n, (long long)(B.nx + 2) * (B.ny + 2) * (B.nz + 2) * word);
  }
  return n <= kTailSmemBytes ? (int)n : 0;
}
template cudaError_t launch_relax_resident<double>(const BlkLev*, int, const int*, const int*, double*, const double*,
                                                   const uint32_t*, const uint32_t*, int, int, bool, float,
                                                   cudaStream_t);
template cudaError_t launch_relax_resident<float>(const BlkLev*, int, const int*, const int*, float*, const float*,
                                                  const uint32_t*, const uint32_t*, int, int, bool, float,
                                                  cudaStream_t);
template cudaError_t launch_relax_blocks<double>(bool, const BlkLev*, int, const int*, double*, const double*,
                                                 const double*, const double*, const double*, const uint32_t*,
                                                 const uint32_t*, int, bool, float, cudaStream_t);
template cudaError_t launch_relax_blocks<float>(bool, const BlkLev*, int, const int*, float*, const float*,
                                                const float*, const float*, const float*, const uint32_t*,
                                                const uint32_t*, int, bool, float, cudaStream_t);
template cudaError_t launch_relax_small<double>(bool, const BlkLev*, const int*, int, double*, const double*,
                                                const double*, const double*, const double*, const uint32_t*,
                                                const uint32_t*, int, int, bool, long long, float, bool, cudaStream_t);
template cudaError_t launch_relax_small<float>(bool, const BlkLev*, const int*, int, float*, const float*,
                                               const float*, const float*, const float*, const uint32_t*,
                                               const uint32_t*, int, int, bool, long long, float, bool, cudaStream_t);

}  // namespace h3d
