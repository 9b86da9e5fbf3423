// k_levelset.cu -- level-set reinitialisation and mask (set_levelset.f:1-199)
// and the FP64 monitor reductions.  Built with --fmad=false: the update
// phi - dt*S*G rounds like the reference.
#include <cmath>

#include "common.cuh"

namespace nse {

#define LD(p, i) __ldg((p) + (i))

// sg = dtau S(phi) on the interior, S = phi / sqrt(phi^2 + epsilon^2) of the
// input field: the factor of every sweep's update (set_levelset.f:80-96), NaN
// where phi is 0.  Sets *big where a value, ghosts included, is kBig or more.
constexpr double kBig = 0x1p600;
__global__ void k_levelset_sign(Dims d, const double* __restrict__ phi, double* sg, double dtau,
                                int* big) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  if (i > d.nx + 1 || j > d.ny + 1) return;
  const double epsilon = 1.0 - 1;  // the reference's PARAMETER(epsilon=1.0d0-1)
  const long c = d.P(i, j, k);
  const double p0 = phi[c];
  if (fabs(p0) >= kBig) *big = 1;
  if (i >= 1 && i <= d.nx && j >= 1 && j <= d.ny && k >= 1 && k <= d.nz)
    sg[c] = dtau * (p0 / sqrt(p0 * p0 + epsilon * epsilon));
}

// n / d from the correctly rounded reciprocal r of d: of the two FMA residual
// corrections the first leaves less than one unit in the last place and the
// second rounds correctly (Markstein, IBM J. Res. Dev. 34 (1990) 111: division
// from a correctly rounded reciprocal).  |n| < 2 kBig and d within 2^+-200, so
// nothing overflows; an n so small that its residual is not exact gives a
// quotient whose square is lost beside the 1 the slope is compared with.
__device__ __forceinline__ double quotient(double n, double d, double r) {
  double q = __dmul_rn(n, r);
  q = __fma_rn(__fma_rn(-q, d, n), r, q);
  return __fma_rn(__fma_rn(-q, d, n), r, q);
}
// max(lo, hi, 0), a NaN counting as 0
__device__ __forceinline__ double upwind(double lo, double hi) {
  const double q = lo > 0.0 ? lo : 0.0;
  return hi > q ? hi : q;
}

// One sweep of set_levelset.f:32-96 into `out` (interior cells), sg =
// dtau S(phi0).  The reference squares the one-sided differences that point
// towards the interface and takes the larger square; here the differences are
// signed towards it and the larger positive one is squared, the same value.
// The ghosts hold the nearest interior value (:107-124), so they are not read: a
// difference across the boundary is 0 (GHOSTS: the first sweep, which reads
// those of the input).  Each thread marches kc cells in z; a z difference
// quotient serves both of its cells (x and y ones are formed by each: the
// reference divides the two x sides by different spacings, and a ridge of
// phi, where both sides count, crosses half of all warps).  *big: a value of
// phi is too large for `quotient` (a sweep that writes one sets it, the
// sweeps after it divide); so do grids with spacings out of its range (!RCP).
// Bound by the latency of each cell's chain, not by memory (ncu at 256x192x256: issue
// 52%, FP64 pipe 37%, DRAM 2.7 TB/s at 45% of the warp slots): the sign factored
// out, five quotients for seven divisions and a square root, and no separate
// ghost pass take a sweep of 256x192x256 from 218 to 101 us (46 us of HBM
// traffic), of 128x96x128 from 30.6 to 13.6, of 64x48x64 from 11.1 to 3.7.
// Small grids are bound by the launches: each sweep starts while the last one
// drains (programmatic dependent launch).
template <bool GHOSTS, bool RCP>
__global__ void __launch_bounds__(256, 4) k_levelset_iter(Dims d, GridDev g, GridRcp rg, int kc,
                                                          const double* __restrict__ sg,
                                                          const double* phi, double* out,
                                                          int flip, int* big) {
  const int i = 1 + blockIdx.x * 32 + threadIdx.x, j = 1 + blockIdx.y * 8 + threadIdx.y;
  const int k0 = 1 + blockIdx.z * kc, k1 = min(d.nz, k0 + kc - 1);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (i > d.nx || j > d.ny) return;
  const long c0 = d.P(i, j, k0);
  const double dxm = LD(g.dx12, i - 1), dxp = LD(g.dx, i), dym = LD(g.dy12, j - 1),
               dyp = LD(g.dy12, j);
  double rxm = 0.0, rxp = 0.0, rym = 0.0, ryp = 0.0;
  if (RCP) {
    rxm = LD(rg.rdx12, i - 1);
    rxp = LD(rg.rdx, i);
    rym = LD(rg.rdy12, j - 1);
    ryp = LD(rg.rdy12, j);
  }
  // neighbours: the cell itself in place of a ghost
  const int xm = GHOSTS || i > 1 ? -1 : 0, xp = GHOSTS || i < d.nx ? 1 : 0;
  const int ym = GHOSTS || j > 1 ? -(int)d.sx : 0, yp = GHOSTS || j < d.ny ? (int)d.sx : 0;
  const double* sp = sg + c0;
  const double* p = phi + c0;
  double* o = out + c0;
  // everything above is older than the previous sweep, phi is its result
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool div = !RCP || *(volatile int*)big;
  double pc = p[0];
  const double pz = p[GHOSTS || k0 > 1 ? -d.sy : 0];
  auto march = [&](auto quot) {
    double qz = quot(pc - pz, LD(g.dz12, k0 - 1), RCP ? LD(rg.rdz12, k0 - 1) : 0.0);
    for (int k = k0; k <= k1; ++k) {
      const double pn = p[GHOSTS || k < d.nz ? d.sy : 0], s = LD(sp, 0);
      // the sign of phi0 (sg carries that of dtau too); where sg is NaN so
      // is the result, whatever the slopes are
      const int neg = (__double2hiint(s) ^ flip) & 0x80000000;
      auto to = [&](double v, int w) {
        return __hiloint2double(__double2hiint(v) ^ w, __double2loint(v));
      };
      const double x = upwind(to(quot(pc - p[xm], dxm, rxm), neg),
                              to(quot(pc - p[xp], dxp, rxp), neg));
      const double y = upwind(to(quot(pc - p[ym], dym, rym), neg),
                              to(quot(pc - p[yp], dyp, ryp), neg));
      const double qn = quot(pn - pc, LD(g.dz12, k), RCP ? LD(rg.rdz12, k) : 0.0);
      const double z = upwind(to(qz, neg), to(qn, neg ^ 0x80000000));
      const double v = pc - s * (sqrt(x * x + y * y + z * z) - 1.0);
      *o = v;
      if (fabs(v) >= kBig) *big = 1;
      qz = qn;
      pc = pn;
      p += d.sy;
      o += d.sy;
      sp += d.sy;
    }
  };
  if (div) march([](double n, double e, double) { return n / e; });
  else march([](double n, double e, double r) { return quotient(n, e, r); });
}

// Neumann ghosts of set_levelset.f:107-124 (z, then y, then x passes): the
// composition gives every ghost the value of the nearest interior cell
__global__ void k_levelset_bc(Dims d, double* phi) {
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  long nA = 2L * (ny + 2) * (nz + 2);
  long nB = 2L * nx * (nz + 2);
  long nC = 2L * nx * ny;
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  int i, j, k;
  if (t < nA) {
    i = (t & 1) ? nx + 1 : 0;
    long r = t >> 1;
    j = (int)(r % (ny + 2));
    k = (int)(r / (ny + 2));
  } else if (t < nA + nB) {
    long r = t - nA;
    j = (r & 1) ? ny + 1 : 0;
    r >>= 1;
    i = 1 + (int)(r % nx);
    k = (int)(r / nx);
  } else if (t < nA + nB + nC) {
    long r = t - nA - nB;
    k = (r & 1) ? nz + 1 : 0;
    r >>= 1;
    i = 1 + (int)(r % nx);
    j = 1 + (int)(r / nx);
  } else {
    return;
  }
  int ci = i < 1 ? 1 : (i > nx ? nx : i);
  int cj = j < 1 ? 1 : (j > ny ? ny : j);
  int ck = k < 1 ? 1 : (k > nz ? nz : k);
  phi[d.P(i, j, k)] = phi[d.P(ci, cj, ck)];
}

// smoothed-Heaviside mask of set_levelset.f:157-170, transition half-width
// width*dx(i) (width = 1 in the reference)
__global__ void k_levelset_mask(Dims d, GridDev g, const double* __restrict__ phi,
                                double* __restrict__ cv, double width) {
  int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
  int j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
  int k = 1 + blockIdx.z;
  if (i > d.nx || j > d.ny) return;
  const double pi = 3.1415926535;
  double ph = LD(phi, d.P(i, j, k));
  double h = width * LD(g.dx, i);
  double v;
  if (ph >= h) v = 1.0;
  else if (ph <= -1.0 * h) v = 0.0;
  else v = (sin(pi * ph / 2.0 / h) + 1.0) / 2.0;
  cv[d.C(i, j, k)] = v;
}

static void interior_grid(const Dims& d, dim3& grid, dim3& block) {
  block = dim3(64, 4, 1);
  grid = dim3((d.nx + 63) / 64, (d.ny + 3) / 4, d.nz);
}

void launch_levelset_sign(const Dims& d, const double* phi, double* sg, double dtau, int* big,
                          cudaStream_t s) {
  dim3 block(32, 8), grid((d.nx + 33) / 32, (d.ny + 9) / 8, d.nz + 2);
  count_launch();
  k_levelset_sign<<<grid, block, 0, s>>>(d, phi, sg, dtau, big);
}
// chained: the launch before this one on the stream is another sweep; rg: the
// reciprocal spacings, null where a spacing is out of the kernel's range
void launch_levelset_iter(const Dims& d, const GridDev& g, const GridRcp* rg, const double* sg,
                          const double* phi, double* phi_new, double dtau, int* big,
                          bool ghosts, bool chained, cudaStream_t s) {
  // cells a thread marches: the z quotient and the x and y spacings are shared
  // by more of them, as long as the chip stays full (us a sweep with 1, 2, 4
  // and 8: 64x48x64 3.7 3.9 4.7 8.2; 81x64x80 6.8 5.9 6.1 9.8; 128x96x128
  // 18.2 14.8 13.6 14.2; 160x128x160 39.6 30.6 26.7 25.3)
  const int kc = d.ncell < 300000 ? 1 : d.ncell < 600000 ? 2 : d.ncell < 2500000 ? 4 : 8;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((d.nx + 31) / 32, (d.ny + 7) / 8, (d.nz + kc - 1) / kc);
  cfg.blockDim = dim3(32, 8);
  cfg.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  const int flip = std::signbit(dtau) ? (int)0x80000000 : 0;
  const GridRcp r = rg ? *rg : GridRcp{};
  count_launch();
#define NSE_LS(G_, RCP_) \
  cudaLaunchKernelEx(&cfg, k_levelset_iter<G_, RCP_>, d, g, r, kc, sg, phi, phi_new, flip, big)
  if (!rg) { if (ghosts) NSE_LS(true, false); else NSE_LS(false, false); }
  else { if (ghosts) NSE_LS(true, true); else NSE_LS(false, true); }
#undef NSE_LS
}
void launch_levelset_bc(const Dims& d, double* phi, cudaStream_t s) {
  long n = 2L * (d.ny + 2) * (d.nz + 2) + 2L * d.nx * (d.nz + 2) + 2L * d.nx * d.ny;
  count_launch();
  k_levelset_bc<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d, phi);
}
void launch_levelset_mask(const Dims& d, const GridDev& g, const double* phi,
                          double* cellvalue1, double width, cudaStream_t s) {
  dim3 grid, block;
  interior_grid(d, grid, block);
  count_launch();
  k_levelset_mask<<<grid, block, 0, s>>>(d, g, phi, cellvalue1, width);
}

// ---------------------------------------------------------------- monitor --
// FP64 reductions over interior cells: [0] max|divu|, [1] sum |u| dx,
// [2] sum |v| dy, [3] sum |w| dz, [4] sum T dx dy dz, [5] non-finite count of
// u, v, w, T.  Two passes (per-block partials, then one block) so the result
// does not depend on scheduling.
template <class DV>
__global__ void k_monitor_partial(Dims d, GridDev g, const double* u, const double* v,
                                  const double* w, const double* T, const DV* divu,
                                  double* part) {
  __shared__ double sh[6][256];
  double acc[6] = {0, 0, 0, 0, 0, 0};
  long n = d.ncell;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long)gridDim.x * blockDim.x) {
    int i = 1 + (int)(t % d.nx);
    long r = t / d.nx;
    int j = 1 + (int)(r % d.ny);
    int k = 1 + (int)(r / d.ny);
    long c = d.P(i, j, k);
    double uu = u[c], vv = v[c], ww = w[c], tt = T[c];
    acc[0] = fmax(acc[0], fabs((double)divu[c]));
    acc[1] += fabs(uu) * g.dx[i];
    acc[2] += fabs(vv) * g.dy[j];
    acc[3] += fabs(ww) * g.dz[k];
    acc[4] += tt * g.dx[i] * g.dy[j] * g.dz[k];
    acc[5] += (isfinite(uu) && isfinite(vv) && isfinite(ww) && isfinite(tt)) ? 0.0 : 1.0;
  }
  for (int q = 0; q < 6; ++q) sh[q][threadIdx.x] = acc[q];
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sh[0][threadIdx.x] = fmax(sh[0][threadIdx.x], sh[0][threadIdx.x + s]);
      for (int q = 1; q < 6; ++q) sh[q][threadIdx.x] += sh[q][threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int q = 0; q < 6; ++q) part[q * gridDim.x + blockIdx.x] = sh[q][0];
}
__global__ void k_monitor_final(const double* part, int nb, double* out) {
  __shared__ double sh[6][256];
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    acc[0] = fmax(acc[0], part[b]);
    for (int q = 1; q < 6; ++q) acc[q] += part[q * nb + b];
  }
  for (int q = 0; q < 6; ++q) sh[q][threadIdx.x] = acc[q];
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sh[0][threadIdx.x] = fmax(sh[0][threadIdx.x], sh[0][threadIdx.x + s]);
      for (int q = 1; q < 6; ++q) sh[q][threadIdx.x] += sh[q][threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int q = 0; q < 6; ++q) out[q] = sh[q][0];
}
// out6 must hold 6 + 6*592 doubles of device memory (partials follow)
template <class DV>
static void monitor(const Dims& d, const GridDev& g, const double* u, const double* v,
                    const double* w, const double* T, const DV* divu, double* out6,
                    cudaStream_t s) {
  const int nb = 592;  // 4 blocks per SM on a 148-SM part
  double* part = out6 + 6;
  count_launch();
  k_monitor_partial<DV><<<nb, 256, 0, s>>>(d, g, u, v, w, T, divu, part);
  count_launch();
  k_monitor_final<<<1, 256, 0, s>>>(part, nb, out6);
}
void launch_monitor(const Dims& d, const GridDev& g, const double* u, const double* v,
                    const double* w, const double* T, const double* divu, double* out6,
                    cudaStream_t s) {
  monitor<double>(d, g, u, v, w, T, divu, out6, s);
}
// mixed-precision form: divu stored in FP32 (the reductions stay FP64)
void launch_monitor_f32(const Dims& d, const GridDev& g, const double* u, const double* v,
                        const double* w, const double* T, const float* divu, double* out6,
                        cudaStream_t s) {
  monitor<float>(d, g, u, v, w, T, divu, out6, s);
}

}  // namespace nse
