// calculate_dispfield (disp_fields.c:502-1049) on the GPU: the Jeans tables
// FG_Disp_r, FG_DispZ, FG_DispPhi, FG_Vstream and, for velocity structure 3,
// FG_tilted_*.
//
// The reference's solvers march sequentially (outer radius to centre, top
// row to mid-plane), but every density, anisotropy, tilt factor and force
// they evaluate depends only on the grid point, never on the running
// solution.  So each part splits into a wide kernel that evaluates all of
// those coefficients in parallel and a narrow kernel that runs the
// recurrence in the reference's order with the coefficients it would have
// computed:
//  * spherical Jeans (disp_fields.c:512-570): coefficients of the 50 Heun
//    steps of all N+1 radial intervals (k_sph_coef), then one thread per type
//    runs the steps (k_sph_march), then the division by the density;
//  * axisymmetric f(E, Lz) (disp_fields.c:575-729): the integrand at the 51
//    points of every z interval of every column (k_axi_points), the
//    trapezoids of every interval in the reference's order (k_axi_sums), one
//    thread per column adds the intervals up (k_axi_march), then the division
//    by the density and DispPhi / Vstream per grid point (k_axi_stream);
//  * tilted f(E, Lz, I3) (disp_fields.c:733-1044): the coefficients of the
//    100 method-of-lines substeps of every row (k_tilt_coef), then one CTA
//    steps the rows (k_tilt_march); then the tilted tables and the VER_1_1
//    streaming velocity per grid point.
// The spherical and axisymmetric parts of all types and the tilted
// coefficients run on a second stream beside the tilted march, the call's
// longest chain.
// Every expression keeps the reference's operation order and the file is
// built with --fmad=false, so the tables are bit-identical to the CPU
// restatement with gmath.h's functions.  The grid radii
// FG_Rmin (FG_Fac^j - 1) come from the C library's pow on the host.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "context.cuh"
#include "galic_gpu.h"
#include "model.cuh"


using galic_internal::second_stream;

namespace {

constexpr double kPi = 3.14159265358979323846;  // M_PI
constexpr double MIN_DENSITY = 1e-25;           // allvars.h:201
constexpr int SPH_STEPS = 50;                   // disp_fields.c:458
constexpr int AXI_STEPS = 50;                   // disp_fields.c:429
constexpr int TILT_STEPS = 100;                 // disp_fields.c:784
constexpr int NTAB = 8;  // disp_r, dispz, dispphi, vstream, tilted_vz2, tilted_vR2, tilted_vz2_prime, tilted_vR2_prime

struct JeansArgs {
  DevModel M;
  const double *Rg;  // FG_Rmin * (pow(FG_Fac, j) - 1.0), j = 0 .. 2N + 2
  int N, type;
  double HaloStretch, Halo_Mass, Halo_A, Disk_Mass, Disk_H, Disk_Z0, Bulge_Mass, Bulge_A, BulgeStretch;
  double beta, beta_a;  // get_beta_of_type's parameter and scale radius for this type
  double f, kpar;       // DispersionRoverZratio, StreamingVelocityParameter of this type
  double *tab;          // [NTAB][N * N] of this type
};

// the types of a call (blockIdx.y of the kernels that run all of them)
struct JeansTypes {
  JeansArgs t[3];
};

__device__ __forceinline__ double tan_(double x) { return gm_sin(x) / gm_cos(x); }
__device__ __forceinline__ double atan_(double x) { return gm_atan2(x, 1.0); }

// get_density_of_type (disp_fields.c:11-24; halo.c:43-54, disk.c:53-69, bulge.c:39-48)
__device__ double density(const JeansArgs &J, const double *pos)
{
  double rho;
  if(J.type == 1) {
    double r = sqrt(pos[0] * pos[0] + pos[1] * pos[1] + J.HaloStretch * J.HaloStretch * pos[2] * pos[2]);
    const double ra = r + J.Halo_A;
    rho = J.HaloStretch * J.Halo_Mass / (2 * kPi) * J.Halo_A / (r + 1.0e-6 * J.Halo_A) / (ra * ra * ra);
  } else if(J.type == 2) {
    if(!(J.Disk_Mass > 0)) return 0;
    double R = sqrt(pos[0] * pos[0] + pos[1] * pos[1]);
    double z = pos[2];
    const double s = 2 / (gm_exp(z / J.Disk_Z0) + gm_exp(-z / J.Disk_Z0));
    rho = J.Disk_Mass / (4 * kPi * J.Disk_H * J.Disk_H * J.Disk_Z0) * gm_exp(-R / J.Disk_H) * (s * s);
  } else {
    double r = sqrt(pos[0] * pos[0] + pos[1] * pos[1] + pos[2] * pos[2]);
    const double ra = r + J.Bulge_A;
    rho = J.BulgeStretch * J.Bulge_Mass / (2 * kPi) * J.Bulge_Mass / (r + 1.0e-6 * J.Bulge_A) / (ra * ra * ra);
  }
  if(gm_fabs(rho) < MIN_DENSITY) rho = 0;
  return rho;
}

// get_beta_of_type (disp_fields.c:26-60)
__device__ __forceinline__ double beta_of(const JeansArgs &J, const double *pos)
{
  double beta = J.beta;
  if(J.type != 2 && beta >= 1) {
    double r = sqrt(pos[0] * pos[0] + pos[1] * pos[1] + pos[2] * pos[2]);
    double dlogrhodr = -1.0 - 3.0 * r / (r + J.beta_a);
    beta = -0.15 - 0.20 * dlogrhodr;
  }
  return beta;
}

// forcegrid_get_acceleration (grid.c:122-197)
__device__ __forceinline__ void fg_acc(const JeansArgs &J, const LogConsts &L, const double *pos, double *acc)
{
  FgCoord c = fg_coord(J.M, L, pos);
  forcegrid_acc(J.M, c, pos, acc);
}

__device__ __forceinline__ double tilt_den(double f, double alpha)
{
  const double c = gm_cos(alpha), s = gm_sin(alpha);
  return c * c - f * (s * s) + (1.0 + f) / 2.0 * gm_sin(2 * alpha) * tan_(2 * alpha);
}

// h_factor (disp_fields.c:1051-1077)
__device__ double h_factor(const JeansArgs &J, double R, double z)
{
  double fac;
  if(R <= 1.0e-12 * z || R == 0)
    fac = 0;
  else {
    double alpha = atan_(z / R);
    fac = ((J.f - 1) / 2 * tan_(2 * alpha)) / tilt_den(J.f, alpha);
  }
  return fac;
}

__device__ __forceinline__ double *table(const JeansArgs &J, int w) { return J.tab + (size_t) w * J.N * J.N; }

// ---------------------------------------------------------------- spherical

struct SphCoef {
  double a0, c0, a1, c1, dr;
  int flag;  // 2: Heun step, 1: Euler step, 0: no change (disp_fields.c:488-496)
};

// interval m: 0 is [R(N+2) -> R(N)], m >= 1 is [R(j+1) -> R(j)] with j = N - m
__global__ void k_sph_coef(const __grid_constant__ JeansTypes T, SphCoef *coef)
{
  const JeansArgs &J = T.t[blockIdx.y];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if(t >= (J.N + 1) * SPH_STEPS) return;
  const int m = t / SPH_STEPS, i = t - m * SPH_STEPS;
  const int N = J.N;
  const double rstart = (m == 0) ? J.Rg[N + 2] : J.Rg[N - m + 1];
  const double rend = (m == 0) ? J.Rg[N] : J.Rg[N - m];
  const LogConsts L = make_log_consts(J.M);
  // integrate_spherical_jeans_beta (disp_fields.c:456-499), step i
  double dr = (rend - rstart) / SPH_STEPS;
  double r0 = rstart + i * dr;
  double r1 = rstart + (i + 1) * dr;
  double pos0[3] = {r0, 0, 0};
  double pos1[3] = {r1, 0, 0};
  double beta0 = beta_of(J, pos0);
  double beta1 = beta_of(J, pos1);
  double acc[3];
  double dens0 = density(J, pos0);
  fg_acc(J, L, pos0, acc);
  double acc0 = acc[0];
  double dens1 = density(J, pos1);
  fg_acc(J, L, pos1, acc);
  double acc1 = acc[0];
  SphCoef c;
  c.a0 = dens0 * acc0;
  c.c0 = 2 * beta0 / r0;
  c.a1 = dens1 * acc1;
  c.c1 = 2 * beta1 / r1;
  c.dr = dr;
  c.flag = (r1 > gm_fabs(dr) && r0 > gm_fabs(dr)) ? 2 : (r0 > gm_fabs(dr) ? 1 : 0);
  coef[(size_t) blockIdx.y * (N + 1) * SPH_STEPS + t] = c;
}

// One thread per type runs the recurrence, a radial interval at a time; the
// rest of its warp sorts out the interval's kind beforehand and the other
// warps stage the next chunk of coefficients in shared memory meanwhile.  The
// loads of a step do not depend on the step before it, so the unrolled loops
// run them ahead.  All steps Heun steps without anisotropy (c0 = c1 = 0): the
// products with y are zeros, and one addition a step is left of the chain; all
// Heun steps: nine dependent operations of 8 cycles; otherwise with the
// selection of disp_fields.c:488-496.  12 850 steps at N = 256: 1.55 ms ->
// 0.28 ms without and 0.55 ms with anisotropy.
constexpr int SPH_CHUNK = 4 * SPH_STEPS;

__global__ void __launch_bounds__(256) k_sph_march(const __grid_constant__ JeansTypes T, const SphCoef *all)
{
  __shared__ SphCoef buf[2][SPH_CHUNK];
  const JeansArgs &J = T.t[blockIdx.y];
  const int total = (J.N + 1) * SPH_STEPS;
  const SphCoef *coef = all + (size_t) blockIdx.y * total;
  double *disp_r = table(J, 0);
  for(int t = threadIdx.x; t < SPH_CHUNK && t < total; t += blockDim.x) buf[0][t] = coef[t];
  __syncthreads();
  double y = 0.0;
  int b = 0;
  for(int c0 = 0; c0 < total; c0 += SPH_CHUNK, b ^= 1) {
    const int n1 = c0 + SPH_CHUNK;
    if(threadIdx.x >= 32) {
      for(int t = threadIdx.x - 32; t < SPH_CHUNK && n1 + t < total; t += blockDim.x - 32) buf[b ^ 1][t] = coef[n1 + t];
    } else {
      for(int m = c0 / SPH_STEPS, u = 0; u < SPH_CHUNK && c0 + u < total; m++, u += SPH_STEPS) {
        const SphCoef *c = buf[b] + u;
        bool heun = true, plain = true;
        for(int t = threadIdx.x; t < SPH_STEPS; t += 32) {
          heun = heun && c[t].flag == 2;
          plain = plain && c[t].c0 == 0 && c[t].c1 == 0 && gm_fabs(c[t].a0) < 0x1p+500 &&
                  gm_fabs(c[t].a1) < 0x1p+500 && gm_fabs(c[t].dr) < 0x1p+400;
        }
        heun = __all_sync(0xffffffffu, heun);
        plain = __all_sync(0xffffffffu, plain);
        if(threadIdx.x) continue;
        // (within these bounds y and ypred stay finite throughout the interval:
        // a zero times infinity would be NaN)
        if(heun && plain && gm_fabs(y) < 0x1p+1000) {
#pragma unroll 10
          for(int t = 0; t < SPH_STEPS; t++) y += c[t].dr * 0.5 * (c[t].a0 + c[t].a1);
        } else if(heun) {
#pragma unroll 10
          for(int t = 0; t < SPH_STEPS; t++) {
            const double k0 = c[t].a0 - c[t].c0 * y;
            const double ypred = y + c[t].dr * k0;
            y += c[t].dr * 0.5 * (k0 + (c[t].a1 - c[t].c1 * ypred));
          }
        } else {
          for(int t = 0; t < SPH_STEPS; t++) {
            const double k0 = c[t].a0 - c[t].c0 * y;
            const double ypred = y + c[t].dr * k0;
            if(c[t].flag == 2)
              y += c[t].dr * 0.5 * (k0 + (c[t].a1 - c[t].c1 * ypred));
            else if(c[t].flag == 1)
              y = ypred;
          }
        }
        if(m >= 1) disp_r[J.N - m] = y;
      }
    }
    __syncthreads();
  }
}

__global__ void k_sph_divide(const __grid_constant__ JeansTypes T)
{
  const JeansArgs &J = T.t[blockIdx.y];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if(j >= J.N) return;
  double *disp_r = table(J, 0);
  double pos[3] = {J.Rg[j], 0, 0};
  double dens = density(J, pos);
  if(dens > 0)
    disp_r[j] /= dens;
  else
    disp_r[j] = 0;
}

// ---------------------------------------------------------------- axisymmetric

// interval m of column j: 0 is [R(N), R(2N)], m >= 1 is [R(k), R(k+1)] with k = N - m
__device__ __forceinline__ void axi_interval(const JeansArgs &J, int m, double *zstart, double *zend)
{
  const int N = J.N;
  *zstart = (m == 0) ? J.Rg[N] : J.Rg[N - m];
  *zend = (m == 0) ? J.Rg[2 * N] : J.Rg[N - m + 1];
}

// the force grid's radial coordinate of every column at y = 0 (fg_coord's
// expression)
__global__ void k_columns(const __grid_constant__ JeansTypes T, double *jd)
{
  const JeansArgs &J = T.t[0];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if(j >= J.N) return;
  const double pos[3] = {J.Rg[j], 0, 0};
  jd[j] = fg_coord(J.M, make_log_consts(J.M), pos).jdbl;
}

// acc[2] of fg_acc at (R, 0, z), z >= 0, given the column's coordinate: the
// azimuth's atan2, sincos and the radial force are not needed
__device__ __forceinline__ double fg_accz(const JeansArgs &J, const LogConsts &L, double jdbl, double R, double z)
{
  const DevModel &M = J.M;
  const int N = M.FG_Nbin;
  const double pos[3] = {R, 0, z};
  double acc[3] = {0, 0, 0};
  if(M.tabulated) {
    const double idbl = gm_log(gm_fabs(z) / M.FG_Rmin + 1.0) / L.lfg;
    if(jdbl < (double) (N - 1) && idbl < (double) (N - 1)) {
      const int jbin = trunc_int(jdbl), ibin = trunc_int(idbl);
      const double jfac = jdbl - jbin, ifac = idbl - ibin;
      const double2 *F = M.fg_acc + ibin * N + jbin;
      acc[2] = F[0].y * (1 - ifac) * (1 - jfac) + F[1].y * (1 - ifac) * jfac + F[N].y * ifac * (1 - jfac) +
               F[N + 1].y * ifac * jfac;
    } else {
      halo_acc(M, pos, acc);
      acc[2] *= M.M200 / M.Halo_Mass;
    }
  }
  if(M.analytic_halo) {
    double h[3];
    halo_acc(M, pos, h);
    acc[2] += h[2];
  }
  if(M.analytic_bulge) {
    double h[3];
    bulge_acc(M, pos, h);
    acc[2] += h[2];
  }
  return acc[2];
}

// integrate_axisymmetric_jeans (disp_fields.c:427-453): the integrand at the
// 51 points zstart + i dz (point i + 1 is the reference's z1 of step i and z0
// of step i + 1: the same expression, the same value).  Y[(i * (N + 1) + m) * N + j]
__global__ void k_axi_points(const __grid_constant__ JeansTypes T, const double *jd, double *Y)
{
  const JeansArgs &J = T.t[blockIdx.y];
  const int N = J.N;
  const long long t = (long long) blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long) N * (N + 1) * (AXI_STEPS + 1);
  if(t >= total) return;
  const int j = (int) (t % N);
  const long long im = t / N;
  const int m = (int) (im % (N + 1));
  const int i = (int) (im / (N + 1));
  double zstart, zend;
  axi_interval(J, m, &zstart, &zend);
  const LogConsts L = make_log_consts(J.M);
  double dz = (zend - zstart) / AXI_STEPS;
  double z = zstart + i * dz;
  double pos[3] = {J.Rg[j], 0, z};
  Y[blockIdx.y * total + t] = -fg_accz(J, L, jd[j], pos[0], z) * density(J, pos);
}

// the trapezoids of every interval, in order: S[m * N + j]
__global__ void k_axi_sums(const __grid_constant__ JeansTypes T, const double *Y, double *S)
{
  const JeansArgs &J = T.t[blockIdx.y];
  const int N = J.N, M = N * (N + 1);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if(t >= M) return;
  double zstart, zend;
  axi_interval(J, t / N, &zstart, &zend);
  const double dz = (zend - zstart) / AXI_STEPS;
  const double *y = Y + (size_t) blockIdx.y * M * (AXI_STEPS + 1) + t;
  double sum = 0, y0 = y[0];
#pragma unroll 10
  for(int i = 1; i <= AXI_STEPS; i++) {
    const double y1 = y[(size_t) i * M];
    sum += 0.5 * (y0 + y1) * dz;
    y0 = y1;
  }
  S[(size_t) blockIdx.y * M + t] = sum;
}

// the running integral of every column, from the top: dispz[k] before its
// division by the density.  (One thread per column summed its 13 000 points
// in turn before: 1.24 ms a type; points, sums and this for both types of a halo + disk now 280 us.)
__global__ void k_axi_march(const __grid_constant__ JeansTypes T, const double *S)
{
  const JeansArgs &J = T.t[blockIdx.y];
  const int j = blockIdx.x * blockDim.x + threadIdx.x, N = J.N;
  if(j >= N) return;
  const double *s = S + (size_t) blockIdx.y * N * (N + 1) + j;
  double *dispz = table(J, 1) + j;
  double integ = s[0];
#pragma unroll 16
  for(int m = 1; m <= N; m++) {
    integ += s[(size_t) m * N];
    dispz[(size_t) (N - m) * N] = integ;
  }
}
__global__ void k_axi_divide(const __grid_constant__ JeansTypes T)
{
  const JeansArgs &J = T.t[blockIdx.y];
  const int t = blockIdx.x * blockDim.x + threadIdx.x, N = J.N;
  if(t >= N * N) return;
  double *dispz = table(J, 1);
  double pos[3] = {J.Rg[t % N], 0, J.Rg[t / N]};
  const double dens = density(J, pos);
  dispz[t] = dens > 0 ? dispz[t] / dens : 0;
}

// disp_fields.c:638-698: DispPhi and Vstream from FG_DispZ
__global__ void k_axi_stream(const __grid_constant__ JeansTypes T)
{
  const JeansArgs &J = T.t[blockIdx.y];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int N = J.N;
  if(t >= N * N) return;
  const int k = t / N, j = t - k * N;
  const double *DispZ = table(J, 1);
  double *DispPhi = table(J, 2), *Vstream = table(J, 3);
  const LogConsts L = make_log_consts(J.M);
  double z = J.Rg[k];
  double R = J.Rg[j];
  double pos[3], acc[3], R1, R2;
  int i1, i2;
  pos[0] = R;
  pos[1] = 0;
  pos[2] = z;
  fg_acc(J, L, pos, acc);
  const int i = k * N + j;
  if(j > 1 && j < N - 1) {
    R1 = J.Rg[j - 1];
    i1 = k * N + j - 1;
    R2 = J.Rg[j + 1];
    i2 = k * N + j + 1;
  } else if(j == 1) {
    R1 = J.Rg[j];
    i1 = k * N + j;
    R2 = J.Rg[j + 1];
    i2 = k * N + j + 1;
  } else if(j == 0) {
    R1 = J.Rg[j + 1];
    i1 = k * N + j + 1;
    R2 = J.Rg[j + 2];
    i2 = k * N + j + 2;
  } else {
    R1 = J.Rg[j - 1];
    i1 = k * N + j - 1;
    R2 = J.Rg[j];
    i2 = k * N + j;
  }
  pos[0] = R1;
  double dens1 = density(J, pos);
  pos[0] = R2;
  double dens2 = density(J, pos);
  double dlog = 0;
  if(dens1 * DispZ[i1] > 0 && dens2 * DispZ[i2] > 0)
    dlog = gm_log((dens2 * DispZ[i2]) / (dens1 * DispZ[i1])) / gm_log(R2 / R1);
  double Vphi2 = DispZ[i] + R * (-acc[0]) + DispZ[i] * dlog;
  if(Vphi2 > 0) {
    double vstr = 0;
    if(Vphi2 >= DispZ[i]) vstr = J.kpar * sqrt((Vphi2 - DispZ[i]));
    DispPhi[i] = Vphi2 - vstr * vstr;
    Vstream[i] = vstr;
  } else {
    DispPhi[i] = 0;
    Vstream[i] = 0;
  }
}

// ---------------------------------------------------------------- tilted

// The coefficients of one substep: three rows of `pitch` doubles, -p = rho a_z, h =
// h_factor(R_j) and hor = h_over_R.  The neighbour column of dqdR is j + 1 or
// j - 1 by the sign of h (disp_fields.c:793-812), and its h is the neighbour's
// own entry.  The pitch is the march kernel's (a constant there, so that a
// batch's loads differ by immediate offsets).
enum { TC_P = 0, TC_H = 1, TC_HOR = 2, TC_ROWS = 3 };

// rows k_hi .. k_lo (all < N - 1) in marching order, substep st, column j
// (disp_fields.c:775-835); coef[(row * TILT_STEPS + st) * TC_ROWS * pitch]
__global__ void k_tilt_coef(const __grid_constant__ JeansArgs J, const double *jd, int k_lo, int k_hi, int pitch,
                            double *coef)
{
  const int N = J.N;
  const long long t = (long long) blockIdx.x * blockDim.x + threadIdx.x;
  if(t >= (long long) TILT_STEPS * N * (k_hi - k_lo + 1)) return;
  const int g = (int) (t / N), j = (int) (t - (long long) g * N);
  const int st = g % TILT_STEPS, k = k_hi - g / TILT_STEPS;
  const LogConsts L = make_log_consts(J.M);
  double z0 = J.Rg[k + 1];
  double z1 = J.Rg[k];
  double dz = (z1 - z0);
  double z = z0 + (dz / TILT_STEPS) * st;
  double R = J.Rg[j];
  const double pos[3] = {R, 0, z};
  const double f = J.f;
  // h_factor and h_over_r (disp_fields.c:1051-1105) share their angle
  double h, hor;
  if(R <= 1.0e-12 * z || R == 0) {
    h = 0;
    hor = (f - 1) / f;
  } else {
    const double alpha = atan_(z / R);
    double s, c, s2, c2;
    gm_sincos(alpha, &s, &c);
    gm_sincos(2 * alpha, &s2, &c2);
    const double t2 = s2 / c2;
    const double den = c * c - f * (s * s) + (1.0 + f) / 2.0 * s2 * t2;  // tilt_den
    h = ((f - 1) / 2 * t2) / den;
    hor = ((f - 1) / 2 * (s / c) * t2) / den;
  }
  double *o = coef + (size_t) g * TC_ROWS * pitch + j;
  o[TC_P * pitch] = -(-density(J, pos) * fg_accz(J, L, jd[j], R, z));
  o[TC_H * pitch] = h;
  o[TC_HOR * pitch] = hor / z;
}

// num / dR by div_by (model.cuh) is the quotient unless the numerator is so
// tiny (or huge) that the remainder rounds: collects the exponent words of the
// numerators (zero, and what is below 2^-1042, passes)
struct TiltRange {
  unsigned lo = 0xffffffffu, hi = 0;
  __device__ __forceinline__ void add(double num)
  {
    const unsigned e = (unsigned) __double2hiint(num) & 0x7fffffffu;
    lo = min(lo, e - 1);
    hi = max(hi, e);
  }
  __device__ __forceinline__ bool plain() const { return lo >= 0x06000000u && hi < 0x79000000u; }  // 2^-927 .. 2^913
};

// One CTA steps rows k_hi .. k_lo (disp_fields.c:775-839); FG_q holds the row
// above on entry.  25 500 dependent substeps at N = 256, each coupled to a
// neighbour column.  A warp carries 32 columns of which it owns the middle 22:
// for TILT_HALO = 5 substeps (20 such batches a row) it takes its neighbours
// from its own lanes (shuffles), losing one valid lane at each end per
// substep, then the CTA exchanges the columns through shared memory.  A lane
// reads the next batch's coefficients into registers during a batch, the
// quotient by the column spacing comes from its reciprocal, and a batch has no
// branch (one whose numerators leave TiltRange or whose neighbours change
// sides is repeated with the general step).  A substep takes about 300 cycles (its
// chain 105; with the coefficient loads 195); a column per thread with a
// barrier and a division per substep took 1150.  Spread over a cluster of 8
// CTAs it took 450: the cluster barrier's memory fence costs more than the
// issue slots it frees.
constexpr int TILT_HALO = 5, TILT_OWN = 32 - 2 * TILT_HALO;
static_assert(TILT_STEPS % (2 * TILT_HALO) == 0, "pairs of batches end with rows");

struct TiltBatch {
  double p[TILT_HALO], h[TILT_HALO], hor[TILT_HALO];
};

template <int MAXT>
__global__ void __launch_bounds__(MAXT) k_tilt_march(const __grid_constant__ JeansArgs J, int k_lo, int k_hi,
                                                     const double *coef, double *FG_q)
{
  constexpr int PITCH = MAXT / 32 * TILT_OWN;
  __shared__ double qb[2][PITCH];
  const int N = J.N, lane = threadIdx.x & 31;
  const int col = (threadIdx.x >> 5) * TILT_OWN - TILT_HALO + lane;
  const bool in = col >= 0 && col < N;
  const bool own = in && lane >= TILT_HALO && lane < 32 - TILT_HALO;
  const int c = min(max(col, 0), N - 1);
  const bool last = c == N - 1, edge = __any_sync(0xffffffffu, last);  // the warp carries the last column
  // spacing to the right and the left neighbour (disp_fields.c:815: R2 - R1)
  const double dRr = J.Rg[min(c + 1, N - 1)] - J.Rg[c], dRl = J.Rg[max(c - 1, 0)] - J.Rg[c];
  double ir = 1.0 / dRr, il = 1.0 / dRl;
  // (opaque: the compiler would divide in the loop, by the selected spacing)
  asm volatile("" : "+d"(ir), "+d"(il));
  const int batches = (k_hi - k_lo + 1) * (TILT_STEPS / TILT_HALO);
  const double *src = coef + c;
  auto load = [&](TiltBatch &t, int i) {
    const double *s = src + (size_t) min(i, batches - 1) * (TILT_HALO * TC_ROWS * PITCH);
#pragma unroll
    for(int u = 0; u < TILT_HALO; u++) {
      t.p[u] = __ldcs(&s[(u * TC_ROWS + TC_P) * PITCH]);
      t.h[u] = __ldcs(&s[(u * TC_ROWS + TC_H) * PITCH]);
      t.hor[u] = __ldcs(&s[(u * TC_ROWS + TC_HOR) * PITCH]);
    }
  };
  double q = FG_q[(size_t) (k_hi + 1) * N + c], step = 0;
  // one batch of t's coefficients; the batch after the next is loaded into t
  auto march = [&](TiltBatch &t, int i, double *turn) {
    // the neighbour's side (disp_fields.c:793-812) nearly always holds for
    // the batch
    const bool right = t.h[0] > 0 || c == 0;
    const int from = right ? lane + 1 : lane - 1;
    const double dR = right ? dRr : dRl, inv = right ? ir : il, q0 = q;
    bool same = true;
    TiltRange range;
#pragma unroll
    for(int u = 0; u < TILT_HALO; u++) {
      same = same && (t.h[u] > 0 || c == 0) == right;
      const double h2 = __shfl_sync(0xffffffffu, t.h[u], from), qn = __shfl_sync(0xffffffffu, q, from);
      const double num = h2 * qn - t.h[u] * q;
      range.add(num);
      const double dqdR = div_by(num, dR, inv) + q * t.hor[u];
      q = q + (t.p[u] - dqdR) * step;
    }
    bool redo = in && !(same && range.plain());
    if(edge) redo = redo || (last && right);  // no neighbour: dqdR = 0
    if(__any_sync(0xffffffffu, redo)) {
      q = q0;
#pragma unroll
      for(int u = 0; u < TILT_HALO; u++) {
        const bool r = t.h[u] > 0 || c == 0;
        const int f = r ? lane + 1 : lane - 1;
        const double h2 = __shfl_sync(0xffffffffu, t.h[u], f), qn = __shfl_sync(0xffffffffu, q, f);
        const double dqdR = (h2 * qn - t.h[u] * q) / (r ? dRr : dRl) + q * t.hor[u];
        q = q + (t.p[u] - (r && last ? 0.0 : dqdR)) * step;
      }
    }
    load(t, i + 2);
    // two turns: a turn's columns are read after its barrier and written
    // again two barriers later
    if(own) turn[c] = q;
    __syncthreads();
    q = turn[c];
  };
  TiltBatch even, odd;
  load(even, 0);
  load(odd, 1);
  for(int k = k_hi, i = 0; k >= k_lo; k--) {
    step = (J.Rg[k] - J.Rg[k + 1]) / TILT_STEPS;  // dz / nsteps
    for(int h = 0; h < TILT_STEPS / (2 * TILT_HALO); h++, i += 2) {
      march(even, i, qb[0]);
      march(odd, i + 1, qb[1]);
    }
    if(own) FG_q[(size_t) k * N + c] = q;
  }
}

// the same for more columns (N <= 1024): a thread per column, the row in two
// shared buffers, one barrier per substep
__global__ void __launch_bounds__(1024) k_tilt_march_wide(const __grid_constant__ JeansArgs J, int k_lo, int k_hi,
                                                          const double *coef, double *FG_q)
{
  __shared__ double qb[2][1024];
  const int N = J.N, j = threadIdx.x;
  const int c = min(j, N - 1);
  const double dRr = J.Rg[min(c + 1, N - 1)] - J.Rg[c], dRl = J.Rg[max(c - 1, 0)] - J.Rg[c];
  double ir = 1.0 / dRr, il = 1.0 / dRl;
  asm volatile("" : "+d"(ir), "+d"(il));
  double q = FG_q[(size_t) (k_hi + 1) * N + c];
  qb[0][j] = q;
  __syncthreads();
  int cur = 0;
  for(int k = k_hi; k >= k_lo; k--) {
    const double step = (J.Rg[k] - J.Rg[k + 1]) / TILT_STEPS;
    for(int st = 0; st < TILT_STEPS; st++, cur ^= 1, coef += TC_ROWS * 1024) {
      const double h1 = coef[TC_H * 1024 + c];
      const bool right = h1 > 0 || c == 0;
      const bool none = h1 > 0 && c == N - 1;
      const int nb = right ? min(c + 1, N - 1) : c - 1;
      const double num = coef[TC_H * 1024 + nb] * qb[cur][nb] - h1 * q;
      const double dR = right ? dRr : dRl;
      TiltRange range;
      range.add(num);
      const double dqdR = (range.plain() ? div_by(num, dR, right ? ir : il) : num / dR) + q * coef[TC_HOR * 1024 + c];
      q = q + (coef[TC_P * 1024 + c] - (none ? 0.0 : dqdR)) * step;
      qb[cur ^ 1][j] = q;
      __syncthreads();
    }
    if(j < N) FG_q[(size_t) k * N + j] = q;
  }
}

// disp_fields.c:849-898: tilted_vz2 = q / rho and the tilted rotation
__global__ void k_tilt_tables(const JeansArgs J, const double *FG_q)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int N = J.N;
  if(t >= N * N) return;
  const int k = t / N, j = t - k * N;
  double *tvz2 = table(J, 4), *tvR2 = table(J, 5), *tvz2p = table(J, 6), *tvR2p = table(J, 7);
  double R = J.Rg[j];
  double z = J.Rg[k];
  double pos[3] = {R, 0, z};
  double dens = density(J, pos);
  const double vz2 = (dens > 0) ? FG_q[t] / dens : 0;
  tvz2[t] = vz2;
  const double f = J.f;
  if(j > 0) {
    double alpha = atan_(z / R);
    const double c = gm_cos(alpha), s = gm_sin(alpha);
    const double den = tilt_den(f, alpha);
    double vrvz = vz2 * ((f - 1) / 2 * tan_(2 * alpha)) / den;
    double vr2 = vz2 * (f * (c * c) - s * s + (1.0 + f) / 2.0 * gm_sin(2 * alpha) * tan_(2 * alpha)) / den;
    double vr2_prime = vr2 * (c * c) + 2 * vrvz * s * c + vz2 * (s * s);
    double vz2_prime = vr2 * (s * s) - 2 * vrvz * s * c + vz2 * (c * c);
    tvR2[t] = vr2;
    tvz2p[t] = vz2_prime;
    tvR2p[t] = vr2_prime;
  } else {
    tvR2[t] = vz2 / f;
    tvz2p[t] = tvR2[t];
    tvR2p[t] = vz2;
  }
}

// disp_fields.c:902-988 (VER_1_1): DispPhi and Vstream from the tilted tables
__global__ void k_tilt_stream(const JeansArgs J)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int N = J.N;
  if(t >= N * N) return;
  const int k = t / N, j = t - k * N;
  const double *tvz2 = table(J, 4), *tvR2 = table(J, 5);
  double *DispPhi = table(J, 2), *Vstream = table(J, 3);
  const LogConsts L = make_log_consts(J.M);
  double z = J.Rg[k];
  double R = J.Rg[j];
  double pos[3] = {R, 0, z}, acc[3];
  double dens = density(J, pos);
  fg_acc(J, L, pos, acc);
  const int i = t;
  double Vphi2 = 0;
  if(dens > 0) {
    int j1 = (0 < j ? j - 1 : j);
    int j2 = (j < N - 1 ? j + 1 : j);
    int i1 = k * N + j1;
    int i2 = k * N + j2;
    double R1 = J.Rg[j1];
    double R2 = J.Rg[j2];
    pos[0] = R1;
    double dens1 = density(J, pos);
    pos[0] = R2;
    double dens2 = density(J, pos);
    Vphi2 = tvR2[i] + R / dens * (dens2 * tvR2[i2] - dens1 * tvR2[i1]) / (R2 - R1) + R * (-acc[0]) +
            R / dens * (dens2 * h_factor(J, R2, z) * tvz2[i2] - dens1 * h_factor(J, R1, z) * tvz2[i1]) / (R2 - R1);
  }
  if(Vphi2 > 0) {
    double vstr = 0;
    if(Vphi2 >= tvR2[i]) vstr = J.kpar * sqrt((Vphi2 - tvR2[i]));
    DispPhi[i] = Vphi2 - vstr * vstr;
    Vstream[i] = vstr;
  } else {
    DispPhi[i] = 0;
    Vstream[i] = 0;
  }
}

// max |x| into *m (bits of a non-negative double, zeroed by the caller)
__global__ void k_abs_max(const double *x, int n, unsigned long long *m)
{
  unsigned long long b = 0;
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double a = gm_fabs(x[i]);
    if(a == a) b = max(b, (unsigned long long) __double_as_longlong(a));  // std::max passes over NaN
  }
  for(int o = 16; o; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
  if((threadIdx.x & 31) == 0 && b) atomicMax(m, b);
}

#define JCK(call)                                                                             \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if(e_ != cudaSuccess) {                                                                   \
      fprintf(stderr, "galic_cuda: %s failed: %s (%s:%d)\n", #call, cudaGetErrorString(e_), __FILE__, \
              __LINE__);                                                                      \
      rc = GALIC_ERR_CUDA;                                                                    \
      goto done;                                                                              \
    }                                                                                         \
  } while(0)

int jfail(galic_ctx *ctx, int st)
{
  if(ctx) ctx->status = st;
  return st;
}

inline int blocks(long long n, int b) { return (int) ((n + b - 1) / b); }

}  // namespace

extern "C" int galic_calculate_dispfield(galic_ctx *ctx, const galic_sample_params_t *sp,
                                         const galic_jeans_params_t *jp, galic_jeans_tables_t *out)
{
  if(!ctx) return GALIC_ERR_INVALID_ARGUMENT;
  if(!sp || !jp) return jfail(ctx, GALIC_ERR_INVALID_ARGUMENT);
  if(!ctx->have_fg) return jfail(ctx, GALIC_ERR_STATE);
  const galic_params_t &p = ctx->prm;
  const int N = p.FG_Nbin;
  if(N < 3 || N > 1024) return jfail(ctx, GALIC_ERR_UNSUPPORTED);
  for(int t = 1; t <= 3; t++)
    if(p.NType[t] > 0 && p.TypeOfVelocityStructure[t] == 3 && jp->DispersionRoverZratio[t] == 0)
      return jfail(ctx, GALIC_ERR_UNSUPPORTED);  // disp_fields.c:743-750 terminate()
  if(cudaSetDevice(ctx->device)) return jfail(ctx, GALIC_ERR_CUDA);
  cudaStream_t s = ctx->stream, s2 = nullptr;
  if(second_stream(ctx) != cudaSuccess) return jfail(ctx, GALIC_ERR_CUDA);
  s2 = ctx->stream2;
  const size_t G = (size_t) N * N;
  int rc = GALIC_OK, launches = 0;
  double *d_Rg = nullptr, *d_tab = nullptr, *d_Y = nullptr, *d_S = nullptr, *d_q = nullptr, *d_tilt = nullptr;
  SphCoef *d_sph = nullptr;
  unsigned long long *d_max = nullptr;
  // rows of tilted coefficients per block: a block's coefficients are made on
  // the second stream while the block before it marches; two blocks within
  // 64 MiB stay in L2 until they are read
  const int pitch = N <= 384 / 32 * TILT_OWN ? 384 / 32 * TILT_OWN : (N <= 768 / 32 * TILT_OWN ? 768 / 32 * TILT_OWN : 1024);
  const size_t row_doubles = (size_t) TILT_STEPS * TC_ROWS * pitch;
  const int tilt_rows = (int) std::max<size_t>(1, std::min<size_t>(N - 1, (32ull << 20) / (row_doubles * sizeof(double))));
  // types whose integrand points are held at once: all of them within 256 MiB
  // (27 MB a type at N = 256, 428 MB at N = 1024)
  const size_t axi_bytes = (size_t) N * (N + 1) * (AXI_STEPS + 1) * sizeof(double);
  const int axi_types = (int) std::max<size_t>(1, std::min<size_t>(3, (256ull << 20) / axi_bytes));
  std::vector<double> Rg(2 * N + 3);
  for(int j = 0; j < 2 * N + 3; j++) Rg[j] = p.FG_Rmin * (std::pow(p.FG_Fac, j) - 1.0);
  bool any_tilt = false;
  int types[3], nt = 0;
  unsigned long long h_max[4][5] = {};
  JeansArgs J{};
  JeansTypes T{};
  J.M = ctx->dm;
  J.N = N;
  J.HaloStretch = p.HaloStretch;
  J.Halo_Mass = p.Halo_Mass;
  J.Halo_A = p.Halo_A;
  J.Disk_Mass = p.Disk_Mass;
  J.Disk_H = sp->Disk_H;
  J.Disk_Z0 = sp->Disk_Z0;
  J.Bulge_Mass = p.Bulge_Mass;
  J.Bulge_A = p.Bulge_A;
  J.BulgeStretch = p.BulgeStretch;
  JCK(cudaMallocAsync((void **) &d_Rg, (Rg.size() + N) * sizeof(double), s));
  JCK(cudaMallocAsync((void **) &d_tab, 4 * NTAB * G * sizeof(double), s));
  JCK(cudaMallocAsync((void **) &d_max, sizeof(h_max), s));
  for(int t = 1; t <= 3; t++) {
    if(p.NType[t] == 0) continue;
    types[nt] = t;
    any_tilt |= p.TypeOfVelocityStructure[t] == 3;
    JeansArgs &A = T.t[nt++] = J;
    A.Rg = d_Rg;
    A.type = t;
    A.f = jp->DispersionRoverZratio[t];
    A.kpar = jp->StreamingVelocityParameter[t];
    A.beta = (t == 1) ? sp->HaloBetaParameter : (t == 3 ? sp->BulgeBetaParameter : 0.0);
    A.beta_a = (t == 1) ? p.Halo_A : p.Bulge_A;
    A.tab = d_tab + (size_t) t * NTAB * G;
  }
  if(nt == 0) goto done;
  JCK(cudaMallocAsync((void **) &d_sph, (size_t) nt * (N + 1) * SPH_STEPS * sizeof(SphCoef), s));
  JCK(cudaMallocAsync((void **) &d_Y, axi_types * axi_bytes, s));
  JCK(cudaMallocAsync((void **) &d_S, (size_t) axi_types * N * (N + 1) * sizeof(double), s));
  if(any_tilt) {
    JCK(cudaMallocAsync((void **) &d_q, G * sizeof(double), s));
    JCK(cudaMallocAsync((void **) &d_tilt, 2 * tilt_rows * row_doubles * sizeof(double), s));
  }
  JCK(cudaMemcpyAsync(d_Rg, Rg.data(), Rg.size() * sizeof(double), cudaMemcpyHostToDevice, s));
  JCK(cudaMemsetAsync(d_tab, 0, 4 * NTAB * G * sizeof(double), s));
  JCK(cudaMemsetAsync(d_max, 0, sizeof(h_max), s));
  {
    double *d_jd = d_Rg + Rg.size();
    k_columns<<<blocks(N, 128), 128, 0, s>>>(T, d_jd);
    launches++;
    // ev2[2]: everything the second stream reads is in place
    JCK(cudaEventRecord(ctx->ev2[2], s));
    JCK(cudaStreamWaitEvent(s2, ctx->ev2[2], 0));
    // spherical and axisymmetric parts (disp_fields.c:512-729), axi_types
    // types at once; queued behind the first block of tilted coefficients
    auto first_parts = [&]() {
      for(int i0 = 0; i0 < nt; i0 += axi_types) {
        const int k = std::min(axi_types, nt - i0);
        JeansTypes P{};
        std::copy(T.t + i0, T.t + i0 + k, P.t);
        k_axi_points<<<dim3(blocks((long long) N * (N + 1) * (AXI_STEPS + 1), 256), k), 256, 0, s2>>>(P, d_jd, d_Y);
        k_axi_sums<<<dim3(blocks((long long) N * (N + 1), 128), k), 128, 0, s2>>>(P, d_Y, d_S);
        k_axi_march<<<dim3(blocks(N, 32), k), 32, 0, s2>>>(P, d_S);
        k_axi_divide<<<dim3(blocks((long long) G, 256), k), 256, 0, s2>>>(P);
        k_axi_stream<<<dim3(blocks((long long) G, 256), k), 256, 0, s2>>>(P);
        launches += 5;
      }
    };
    k_sph_coef<<<dim3(blocks((long long) (N + 1) * SPH_STEPS, 256), nt), 256, 0, any_tilt ? s2 : s>>>(T, d_sph);
    if(!any_tilt) {
      // the spherical march is the longest chain: beside the axisymmetric part
      k_sph_march<<<dim3(1, nt), 256, 0, s>>>(T, d_sph);
      k_sph_divide<<<dim3(blocks(N, 256), nt), 256, 0, s>>>(T);
      launches += 3;
      first_parts();
    }
    bool queued = !any_tilt;
    for(int i = 0; i < nt; i++) {
      const JeansArgs &A = T.t[i];
      if(p.TypeOfVelocityStructure[A.type] != 3) continue;
      JCK(cudaMemsetAsync(d_q + (size_t) (N - 1) * N, 0, N * sizeof(double), s));  // the top row is 0
      int block = 0;
      for(int k_hi = N - 2; k_hi >= 0; k_hi -= tilt_rows, block++) {
        const int k_lo = std::max(0, k_hi - tilt_rows + 1);
        const long long n = (long long) (k_hi - k_lo + 1) * TILT_STEPS * N;
        double *cf = d_tilt + (size_t) (block & 1) * tilt_rows * row_doubles;
        // ev2[block & 1]: this half's previous block has marched
        if(block >= 2 || i > 0) JCK(cudaStreamWaitEvent(s2, ctx->ev2[block & 1], 0));
        k_tilt_coef<<<blocks(n, 256), 256, 0, s2>>>(A, d_jd, k_lo, k_hi, pitch, cf);
        JCK(cudaEventRecord(ctx->ev2[3 + (block & 1)], s2));
        JCK(cudaStreamWaitEvent(s, ctx->ev2[3 + (block & 1)], 0));
        const int threads = (N + TILT_OWN - 1) / TILT_OWN * 32;
        if(pitch == 384 / 32 * TILT_OWN)
          k_tilt_march<384><<<1, threads, 0, s>>>(A, k_lo, k_hi, cf, d_q);
        else if(pitch == 768 / 32 * TILT_OWN)
          k_tilt_march<768><<<1, threads, 0, s>>>(A, k_lo, k_hi, cf, d_q);
        else
          k_tilt_march_wide<<<1, (N + 31) / 32 * 32, 0, s>>>(A, k_lo, k_hi, cf, d_q);
        JCK(cudaEventRecord(ctx->ev2[block & 1], s));
        launches += 2;
        if(!queued) {
          k_sph_march<<<dim3(1, nt), 256, 0, s2>>>(T, d_sph);
          k_sph_divide<<<dim3(blocks(N, 256), nt), 256, 0, s2>>>(T);
          launches += 3;
          first_parts();
          queued = true;
        }
      }
      // the axisymmetric DispPhi and Vstream of the type come first
      JCK(cudaEventRecord(ctx->ev2[2], s2));
      JCK(cudaStreamWaitEvent(s, ctx->ev2[2], 0));
      k_tilt_tables<<<blocks((long long) G, 256), 256, 0, s>>>(A, d_q);
      k_tilt_stream<<<blocks((long long) G, 256), 256, 0, s>>>(A);
      launches += 2;
    }
    JCK(cudaEventRecord(ctx->ev2[2], s2));
    JCK(cudaStreamWaitEvent(s, ctx->ev2[2], 0));
    JCK(cudaGetLastError());
    // install into the context (as galic_set_vstream / galic_set_dispersion
    // would), device to device, and copy out
    for(int i = 0; i < nt; i++) {
      const int t = types[i];
      const double *D = d_tab + (size_t) t * NTAB * G;
      const int src[5] = {0, 1, 2, 7, 6};  // galic_set_dispersion's order of the tables
      for(int w = 0; w < 5; w++) {
        if(!ctx->d_disp[t][w]) JCK(cudaMallocAsync((void **) &ctx->d_disp[t][w], G * sizeof(double), s));
        JCK(cudaMemcpyAsync(ctx->d_disp[t][w], D + src[w] * G, G * sizeof(double), cudaMemcpyDeviceToDevice, s));
        k_abs_max<<<std::min(blocks((long long) G, 256), 148), 256, 0, s>>>(D + src[w] * G, w == 0 ? N : (int) G,
                                                                            d_max + 5 * t + w);
        launches++;
      }
      JCK(cudaMemcpyAsync(ctx->d_vstream[t], D + 3 * G, G * sizeof(double), cudaMemcpyDeviceToDevice, s));
    }
    JCK(cudaMemcpyAsync(h_max, d_max, sizeof(h_max), cudaMemcpyDeviceToHost, s));
    for(int i = 0; i < nt; i++) {
      const int t = types[i];
      const double *D = d_tab + (size_t) t * NTAB * G;
      ctx->h_vstream[t].resize(G);
      JCK(cudaMemcpyAsync(ctx->h_vstream[t].data(), D + 3 * G, G * sizeof(double), cudaMemcpyDeviceToHost, s));
      if(!out) continue;
      double *dst[NTAB] = {out[t].disp_r,     out[t].dispz,      out[t].dispphi,          out[t].vstream,
                           out[t].tilted_vz2, out[t].tilted_vR2, out[t].tilted_vz2_prime, out[t].tilted_vR2_prime};
      for(int w = 0; w < NTAB; w++)
        if(dst[w]) JCK(cudaMemcpyAsync(dst[w], D + w * G, G * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    JCK(cudaStreamSynchronize(s));
  }
done:
  if(rc != GALIC_OK) cudaStreamSynchronize(s2);
  if(d_Rg) cudaFreeAsync(d_Rg, s);
  if(d_tab) cudaFreeAsync(d_tab, s);
  if(d_sph) cudaFreeAsync(d_sph, s);
  if(d_Y) cudaFreeAsync(d_Y, s);
  if(d_S) cudaFreeAsync(d_S, s);
  if(d_q) cudaFreeAsync(d_q, s);
  if(d_tilt) cudaFreeAsync(d_tilt, s);
  if(d_max) cudaFreeAsync(d_max, s);
  if(rc != GALIC_OK) {
    cudaStreamSynchronize(s);
    return jfail(ctx, rc);
  }
  ctx->last_launches = launches;
  for(int i = 0; i < nt; i++) {
    const int t = types[i];
    const std::vector<double> &v = ctx->h_vstream[t];
    // only +0.0 everywhere allows skipping the lookup
    ctx->dm.vstream_zero[t] =
        std::all_of(v.begin(), v.end(), [](double x) { return x == 0 && !std::signbit(x); }) ? 1 : 0;
    for(int w = 0; w < 5; w++) memcpy(&ctx->disp_max[t][w], &h_max[t][w], sizeof(double));
    ctx->have_disp[t] = true;
    ctx->generation++;
    ctx->tab32_dirty = true;
  }
  return jfail(ctx, GALIC_OK);
}
