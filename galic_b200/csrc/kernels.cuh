// Launch wrappers shared by the C-ABI layer (api.cu) and the kernel files.
#ifndef GALIC_KERNELS_CUH
#define GALIC_KERNELS_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "fixedpoint.cuh"
#include "galic_gpu.h"
#include "model.cuh"

// field order of the per-orbit grids: the argument order of
// produce_orbit_response_field_mod (orbit_response.c:155-157): m, r, t, q, p
enum { F_M = 0, F_R = 1, F_T = 2, F_Q = 3, F_P = 4, NF_ORBIT = 5 };
// committed per-type grids, in galic_grid_id order
enum { NG_COMMITTED = 10 };
// threads per CTA of the persistent orbit kernels
#define CALC_ALL_BLOCK_FP64 128
#define CALC_ALL_BLOCK_FP32 128
#ifndef GALIC_FP64_MIN_BLOCKS
// 3 CTAs of 128 threads per SM (158 registers, none spilled) run the halo +
// disk pass in 300 ms; 4 CTAs (128 registers, 110 bytes spilled) take 363 ms and
// 2 CTAs 302 ms: past 2 warps per scheduler the L1 data stage, the issue slots
// and the FP64 pipe (64, 58 and 43 % busy at 2.4e5 orbits) share the limit
#define GALIC_FP64_MIN_BLOCKS 3
#endif
#ifndef GALIC_FP32_MIN_BLOCKS
// 5 CTAs per SM (96 registers, 20 bytes spilled; 5 x 31 KiB of queues) ran the
// FP32 pass 2 % faster than 4 (105 registers); 6 (80 registers, spills) 18 %
// slower
#define GALIC_FP32_MIN_BLOCKS 5
#endif
// target stacks per type: DGs_MassTarget, EGs_MassTarget, EGs_EgyTarget_{r,t,p,q}
enum { T_DGM = 0, T_EGM = 1, T_R = 2, T_T = 3, T_P = 4, T_Q = 5, NT_TARGET = 6 };

struct OrbitBatch {
  int count;
  const double *pos, *vel;    // count x 3
  const double *mass, *timespan;
  const int *type;
  double *grids;              // count x NF_ORBIT x DG_Ngrid (zeroed by the caller)
  double *tall;               // count
  int *norbit;                // count
  long long *steps;           // count
  double *egy_err;            // count
  int *status;                // count
  int with_egy;               // produce_orbit_response_field_mod (1) or _field (0)
};

struct CalcAllArgs {
  int n;                      // orbits of this launch: order[first + k * stride], k < n
  int first = 0, stride = 1;
  const double *pos, *vel, *mass, *tint;
  const int *type;
  const int *order;           // processing order (longest first)
  int *next;                  // work counter (orbits taken after the lanes' first), zeroed by the caller
  FxWord *fx;                 // [4][NG_COMMITTED][Ngrid] (the time-averaged five of a type as FxNode[Ngrid])
  const int *shift;           // [4][NG_COMMITTED]
  int *orbits;                // per particle
  unsigned long long *steps_total;
  double *max_egy_err;        // max relative energy error (as ordered bits)
  int *status;                // worst OrbitStatus seen
};

constexpr int FIT_TERMS = 9;

struct FitArgs {
  int L;                      // DG_MaxLevel == EG_MaxLevel
  int Ngrid, Nstack;
  const double *committed;    // [4][10][Ngrid]
  double *stacks;             // [4][10][Nstack]
  double *values;             // [4][9][Nstack]: node values of the committed merit terms (fit_fp64.cu:k_fit)
  const double *targets;      // [4][6][Nstack]
  const double *dgs_distance; // [Nstack]
  double *fit;                // [4][7]
  double *raw;                // [4][5]
  unsigned *arrived;          // [4], 0 between whole fits
  int *firstrun;              // [4]
  double thr_d[4], thr_e[4], MType[4];
  int present[4], tovs[4];
  double R200_20, LowerDispLimit;
};

void launch_orbits_dense(const DevModel &M, const OrbitBatch &b, cudaStream_t s);
// the same orbits in the FP32 form (orbit_fp32.cu), with egy fields
void launch_orbits_dense_fp32(const DevModel &M64, const float4 *const quad[4], const float *cellsize32,
                              const OrbitBatch &b, cudaStream_t s);
void launch_scale_dense(const DevModel &M, const OrbitBatch &b, cudaStream_t s);
int launch_calc_all_fp64(const DevModel &M, const CalcAllArgs &a, int grid, int block, cudaStream_t s);
// particles first, first + stride, ... below n
void launch_instantaneous(const DevModel &M, int n, const double *pos, const double *vel, const double *mass,
                          const int *type, double *vdisp, FxWord *fx, const int *shift, int Ngrid, cudaStream_t s,
                          int first = 0, int stride = 1);
// grids first .. first + per - 1 of each of `sets` sets of NG_COMMITTED
void launch_fx_finalize(const FxWord *fx, const int *shift, double *committed, int sets, int first, int per, int Ngrid,
                        int form, cudaStream_t s);
// hist: a second place for the fit ([4][7]), or null; terms first .. first +
// count - 1 of FIT_TERMS only: the fit follows with the launch that completes them
int launch_global_fit(const FitArgs &f, cudaStream_t s, double *hist = nullptr, int first = 0, int count = FIT_TERMS);
int calc_all_occupancy(int block);
int calc_all_fp32_occupancy(int block);
int launch_calc_all_fp32(const DevModel &M64, const float4 *const quad[4], const float *cellsize32,
                         const CalcAllArgs &a, int grid, int block, cudaStream_t s);

#ifdef __CUDACC__
// The first orbit of a lane in a persistent grid: orbit lane * (warps of the
// grid) + warp, so that consecutive orbits of the processing order start in
// different warps.  The end of a pass is set by its longest orbits, and a step
// takes a warp longer the more of its lanes are at work (cell changes,
// drains): started 32 to a warp, 2e4 halo orbits took 17.2 ms (FP64), spread
// over the warps 14.5 ms, and 1e5 orbits 20.8 and 18.9 ms.  (More warps than
// the orbits fill, a few lanes each, ran no faster and kept other streams'
// kernels off the GPU: six concurrent jobs 84 ms against 62 ms.)  Later orbits
// come from a counter: the next is number 32 * warps + count.
struct FirstOrbit {
  int index;  // of this lane
  int lanes;  // orbits handed out this way
  __device__ __forceinline__ FirstOrbit()
  {
    const int warps = (int) (gridDim.x * blockDim.x) >> 5;
    lanes = 32 * warps;
    index = (int) (threadIdx.x & 31) * warps + (int) ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  }
};

// Orbits of a dense launch, one thread per orbit (-1: none), spread like
// FirstOrbit over at least DENSE_WARPS warps where there are that many orbits:
// such a launch lasts as long as its longest orbits, and those take longer in
// full warps.  Measured with the warps filled, with at least 592, 888 and 1184
// of them (ms): one repetition of 401 particles (802 orbits, halo + disk, level
// 7, FP32) 13.7, 8.7, 8.7, 8.8; of 101 (halo, level 6, FP64) 7.8, 6.2, 6.2, 6.2;
// the construction of 6e4 composite particles with two windows of 1608
// particles (FP32) 45.0, 41.5, 42.0, 41.1; six served jobs 56, 53, 53, 53.
// Two FP64 windows at once would rather have fewer: of 4020 particles (halo +
// disk, level 6) 16.8, 16.3, 20.0, 21.0.
constexpr int DENSE_WARPS = 888;
__device__ __forceinline__ int dense_orbit(int count)
{
  const int k = FirstOrbit().index;
  return k < count ? k : -1;
}
inline int dense_grid(int count, int block)
{
  const int full = (count + 31) / 32;
  const int warps = count < DENSE_WARPS ? count : (full > DENSE_WARPS ? full : DENSE_WARPS);
  return (warps + block / 32 - 1) / (block / 32);
}

// Orbits are processed longest first: a pass ends with its last orbits, and as
// a lane takes the next orbit when its own ends, a long orbit started late
// leaves the GPU to a few lanes (in the order used before, by type and
// increasing radius, the far, long orbits of each type came last).  The steps
// of an orbit of TorbitFac periods rank like r^(1/4) (1.1 - v / v_esc): rank
// correlation 0.84 to 0.99 with the counted steps over the halos, disks and
// bulges of the synthetic models (radius alone 0.27 to 0.96).  The class is
// that estimate in steps of a quarter octave, 0 the longest.  A pass's results
// do not depend on the order.  1e5 halo orbits 23.9 -> 20.8 ms (FP64), 1.2e6
// halo + disk orbits 309 -> 306 ms, an ensemble of 12 halos 41.0 -> 37.3 ms.
__device__ __forceinline__ unsigned orbit_length_class(const double *p, const double *v, double vesc, double *r2)
{
  *r2 = p[0] * p[0] + p[1] * p[1] + p[2] * p[2];
  const double u = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) / vesc;
  const float est = sqrtf(sqrtf((float) sqrt(*r2))) * fmaxf(1.1f - (float) u, 1e-3f);  // fmaxf: 1e-3 for NaN too
  const float b = est > 0.f ? 4.f * log2f(est) + 127.f : 0.f;
  return 255u - (unsigned) fminf(fmaxf(b, 0.f), 255.f);
}
#endif

// ---- ensemble of models in one persistent FP32 launch (orbit_fp32.cu)
#define GALIC_ENSEMBLE_MAX 64
struct EnsembleLaunch {
  int nmodels;
  int offset[GALIC_ENSEMBLE_MAX + 1];  // prefix sums of the models' orbit counts
  DevModel dm[GALIC_ENSEMBLE_MAX];
  const float4 *quad[GALIC_ENSEMBLE_MAX][4];
  const float *cellsize32[GALIC_ENSEMBLE_MAX];
  const void *members;  // device array of ensemble_member_bytes() per model
  int *next;
  FxWord *fx;           // [models * 4][NG_COMMITTED][Ngrid]
  const int *shift;     // [models * 4][NG_COMMITTED]
  unsigned long long *steps;
  double *maxerr;
  int *status;
};
int ensemble_variant_count();
int ensemble_variant(int v, int *block, int *min_blocks);
int ensemble_occupancy(int v);
size_t ensemble_member_bytes();
void ensemble_fill_member(void *dst, const DevModel &dm, const double *pos, const double *vel, const double *mass,
                          const double *tint, const int *type, const int *order, int *orbits);
cudaError_t launch_ensemble_fp32(const EnsembleLaunch &L, int v, int grid, cudaStream_t s);

#endif
