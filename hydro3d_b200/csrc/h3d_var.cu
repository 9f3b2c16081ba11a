// Kernels of the variable-coefficient (L_LSM) operator.
#include <algorithm>
#include <type_traits>

#include "h3d_device.cuh"
#include "h3d_kernels.cuh"

namespace h3d {

namespace {

// ---------------------------------------------------------------------------
// FP64 defect r = b - A p with variable coefficients (newsolv_mg.for:55 as a
// residual, mgrestr's operand order), 44 bytes a cell with an FP32 result.  A thread
// owns a pair of cells of one row and marches z with the iterate of planes
// z-1 .. z+1 and the lower face coefficient in registers; everything else of plane z+1 is
// loaded while plane z is formed.  (A warp a row without the march had one row's
// scattered loads in flight: 206 us on 256^3 cells, 155 us here; the
// correction added at every point of the stencil, before its own pass: 505 us.)
constexpr int kDefectVarThreads = 256;
__device__ __forceinline__ double2 ld2(const double* p) { return *reinterpret_cast<const double2*>(p); }

template <typename TR, bool EARLY>
__global__ void __launch_bounds__(kDefectVarThreads) k_defect_var(
    const BlkLev* __restrict__ bls, const Tile* __restrict__ tiles, int zc, const double* __restrict__ p,
    const double* __restrict__ bvec, TR* __restrict__ rhs_out, double mean_b, double rscale,
    const double* __restrict__ fx, const double* __restrict__ fy, const double* __restrict__ fz,
    double* __restrict__ partials) {
  using R2 = typename std::conditional<sizeof(TR) == 4, float2, double2>::type;
  pdl_trigger();
  const Tile t = tiles[blockIdx.x];
  const BlkLev B = bls[t.b];
  const int H = B.nx >> 1, rows = kDefectVarThreads / H;
  const int row = threadIdx.x / H, y = t.y0 + row;
  const bool in = row < rows && y <= B.ny;
  const int x0 = 1 + 2 * (threadIdx.x - row * H);
  const long long sx = B.sx, sxy = B.sxy;
  const double rsc = rscale < 0.0 ? B.dv : rscale;
  const int zs = t.z0, ze = min(t.z0 + zc - 1, B.nz);
  double rr = 0, bb = 0, rm = 0, rs = 0;
  struct Plane {  // operands of a plane but p itself
    double2 ps, pn, b, fx, fy, fs, fz;
    double pw, pe, fw;
  };
  pdl_wait<EARLY>(p, bvec);
  if (in) {
    const long long r0 = B.off + (long long)y * sx + x0;
    auto load = [&](int z, Plane& q) {
      const long long i = r0 + (long long)z * sxy;
      q.ps = ld2(p + i - sx);
      q.pn = ld2(p + i + sx);
      q.b = ld2(bvec + i);
      q.fx = ld2(fx + i);
      q.fy = ld2(fy + i);
      q.fs = ld2(fy + i - sx);
      q.fz = ld2(fz + i);
      q.pw = p[i - 1];
      q.pe = p[i + 2];
      q.fw = fx[i - 1];
    };
    long long i = r0 + (long long)zs * sxy;
    double2 pb = ld2(p + i - sxy), pc = ld2(p + i), zb = ld2(fz + i - sxy), pt;
    Plane q, n;
    load(zs, q);
    pt = ld2(p + i + sxy);
    for (int z = zs; z <= ze; ++z, i += sxy) {
      double2 ptn = pt;
      if (z < ze) {
        load(z + 1, n);
        ptn = ld2(p + i + 2 * sxy);
      }
      const Coef<double> c0{q.fw, q.fx.x, q.fs.x, q.fy.x, zb.x, q.fz.x};
      const Coef<double> c1{q.fx.x, q.fx.y, q.fs.y, q.fy.y, zb.y, q.fz.y};
      const double a0 = q.b.x - (c0.aw * q.pw + c0.ae * pc.y + c0.as * q.ps.x + c0.an * q.pn.x + c0.ab * pb.x +
                                 c0.at * pt.x + coef_ap(c0) * pc.x);
      const double a1 = q.b.y - (c1.aw * pc.x + c1.ae * q.pe + c1.as * q.ps.y + c1.an * q.pn.y + c1.ab * pb.y +
                                 c1.at * pt.y + coef_ap(c1) * pc.y);
      R2 ro;
      ro.x = (TR)(a0 - mean_b);
      ro.y = (TR)(a1 - mean_b);
      *reinterpret_cast<R2*>(rhs_out + i) = ro;
      rr += a0 * a0;
      rr += a1 * a1;
      bb += q.b.x * q.b.x;
      bb += q.b.y * q.b.y;
      rm = fmax(rm, fmax(fabs(a0), fabs(a1)) * rsc);
      rs += a0;
      rs += a1;
      pb = pc;
      pc = pt;
      pt = ptn;
      zb = q.fz;
      q = n;
    }
  }
  block_reduce4<kDefectVarThreads>(rr, bb, rm, rs, partials + 4 * (size_t)blockIdx.x);
}

}  // namespace

int defect_var_rows(int nx) { return kDefectVarThreads / (nx / 2); }

template <typename TR>
cudaError_t launch_defect_var(const BlkLev* bl, const Tile* tiles, int ntiles, int zc, const double* p,
                              const double* b, TR* rhs_out, double mean_b, double rscale, const double* fx,
                              const double* fy, const double* fz, double* partials, cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  pdl_launch(H3D_BOTH(k_defect_var, TR), ntiles, kDefectVarThreads, 0, st, bl, tiles, zc, p, b, rhs_out, mean_b, rscale, fx,
             fy, fz, partials);
  return cudaGetLastError();
}
template cudaError_t launch_defect_var<float>(const BlkLev*, const Tile*, int, int, const double*, const double*,
                                              float*, double, double, const double*, const double*, const double*,
                                              double*, cudaStream_t);
template cudaError_t launch_defect_var<double>(const BlkLev*, const Tile*, int, int, const double*, const double*,
                                               double*, double, double, const double*, const double*, const double*,
                                               double*, cudaStream_t);

}  // namespace h3d
