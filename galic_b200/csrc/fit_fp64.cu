// Merit function and optimisation repetition (built with --fmad=false).
//
//  k_fit          calc_global_fit (main.c:251-362), one CTA per type and term
//  k_propose      the proposal part of optimize (main.c:365-441)
//  k_eval_terms   the nine stack terms of eval_fit_mod (main.c:1021-1217)
//  k_accept       their combination, the accept branch of optimize
//                 (main.c:468-507) and the accepted positions in order
//  k_commit       the _delta accumulation (main.c:477-486), add_to_energy_grid
//                 of the accepted particles (main.c:488-498) and
//                 commit_updates (main.c:818-835): per bin, the accepted
//                 particles' new - old values are summed in particle order,
//                 as the reference's sequential loop does, then added to the
//                 committed grid.
//
// A repetition's commit is a chain of these kernels on one stream, each a few
// microseconds long, and the next repetition waits for it: latency is what it
// costs.
#include <cuda_runtime.h>

#include "galic_gpu.h"
#include "grng.h"
#include "kernels.cuh"
#include "rep.cuh"
#include "stack.cuh"

namespace {

// The nine terms of the merit function.  0: density (main.c:1033-1047); 1-4:
// the time-averaged dispersions r, t, q, p (main.c:1052-1120); 5-8: the
// instantaneous ones r, t, p, q (main.c:1125-1176).
enum { NTERM = FIT_TERMS };
__device__ __constant__ const int kTermGrid[NTERM] = {GALIC_GRID_MASS_S, GALIC_GRID_R_S, GALIC_GRID_T_S,
                                                      GALIC_GRID_Q_S,    GALIC_GRID_P_S, GALIC_GRID_R_I,
                                                      GALIC_GRID_T_I,    GALIC_GRID_P_I, GALIC_GRID_Q_I};
__device__ __constant__ const int kTermTarget[NTERM] = {T_DGM, T_R, T_T, T_Q, T_P, T_R, T_T, T_P, T_Q};

// KIND 0: term 0, 1: terms 1-4, 2: terms 5-8
template <int KIND>
struct TermLeaf {
  const double *d2, *r2, *dist;
  double R200_20, lowdisp;
  __device__ __forceinline__ TermLeaf(const FitArgs &f, int type, int term)
  {
    const double *tg = f.targets + (size_t) type * NT_TARGET * f.Nstack;
    d2 = tg + (size_t) kTermTarget[term] * f.Nstack;
    r2 = KIND == 2 ? tg + (size_t) T_EGM * f.Nstack : d2;
    dist = f.dgs_distance;
    R200_20 = f.R200_20;
    lowdisp = f.LowerDispLimit;
  }
  __device__ __forceinline__ double operator()(int node, double d1, double r1) const
  {
    return stack_leaf(d1, d2[node], r1, KIND ? r2[node] : 0.0, KIND == 2 ? 0.0 : dist[node], KIND == 0 ? 0 : 3 - KIND,
                      KIND == 1, R200_20, lowdisp);
  }
};

// from_stacks: the finest level is the stacks' (the values of their nodes are
// wanted for k_eval_terms, nothing else changes)
template <int KIND>
__device__ __forceinline__ double fit_term(const FitArgs &f, int type, int term, bool from_stacks,
                                           Pyramid<1, KIND == 2> &sm)
{
  const int L = f.L, N = 1 << L, Ns = f.Nstack, off = stack_off(L);
  double *stacks = f.stacks + (size_t) type * NG_COMMITTED * Ns;
  double *stk = stacks + (size_t) kTermGrid[term] * Ns, *mstk = stacks + (size_t) GALIC_GRID_MASS_I * Ns;
  const double *grids = f.committed + (size_t) type * NG_COMMITTED * f.Ngrid;
  const double *fine = from_stacks ? stk + off : grids + (size_t) kTermGrid[term] * f.Ngrid;
  const double *mfine = from_stacks ? mstk + off : grids + (size_t) GALIC_GRID_MASS_I * f.Ngrid;
  double *val = f.values + ((size_t) type * NTERM + term) * Ns;
  const TermLeaf<KIND> leaf(f, type, term);
  auto children = [&](int g, double (&x)[1][4], double (&m)[4]) {
    const int at[4] = {g, g + 1, g + N, g + N + 1};
#pragma unroll
    for(int q = 0; q < 4; q++) {
      x[0][q] = fine[at[q]];
      if(KIND == 2) m[q] = mfine[at[q]];
    }
    if(!from_stacks)
#pragma unroll
      for(int q = 0; q < 4; q++) {
        stk[off + at[q]] = x[0][q];
        if(KIND == 2 && term == 5) mstk[off + at[q]] = m[q];
      }
    return 1u;
  };
  auto keep = [&](int node, double d, double v, double r) {
    val[node] = v;
    if(!from_stacks) {
      stk[node] = d;
      if(KIND == 2 && term == 5) mstk[node] = r;
    }
  };
  auto keep_leaf = [&](int node, double v) { val[node] = v; };
  double root[1];
  pyramid_cta<1, KIND == 2>(sm, L, children, [](int) { return 0.0; }, leaf,
                            f.targets + ((size_t) type * NT_TARGET + T_DGM) * Ns, KIND == 2 ? f.thr_e[type] : f.thr_d[type],
                            keep, keep_leaf, root);
  return root[0];
}

__device__ __forceinline__ void fit_final(const FitArgs &f, int type)
{
  const volatile double *raw = f.raw + type * 5;
  const double *tg = f.targets + (size_t) type * NT_TARGET * f.Nstack;
  double S = raw[0];
  S *= 1.0 / tg[T_DGM * f.Nstack + 0];
  double sr = raw[1], st = raw[2], sp = raw[3], sq = raw[4];
  double count;
  if(f.tovs[type] == 0 || f.tovs[type] == 1) {
    count = 3.0;
    sq = 0;
  } else
    count = 4.0;
  double *o = f.fit + type * 7;
  double srel = o[5];
  if(f.firstrun[type] == 0) {
    srel = S / ((sr + st + sp + sq) / count);
    f.firstrun[type] = 1;
  }
  o[0] = S;
  o[1] = sr * srel;
  o[2] = st * srel;
  o[3] = sp * srel;
  o[4] = sq * srel;
  o[5] = srel;
  o[6] = count;
}

// One CTA per (type, term): smooths the term's stack, evaluates its misfit and
// leaves both, node by node (f.stacks, f.values); the CTA of a type that ends
// last forms the type's fit.  The three kernels it replaces (smooth, misfit on
// a whole stack in shared memory, final) took 32 us at level 6, with 21 us more
// for the committed instantaneous terms; it takes 15 us (cold caches).
__global__ void __launch_bounds__(1024) k_fit(const __grid_constant__ FitArgs f, int first, int count,
                                              bool from_stacks, double *hist)
{
  __shared__ union {
    Pyramid<1, false> a;
    Pyramid<1, true> b;
  } sm;
  const int type = (int) blockIdx.x / count, term = first + (int) blockIdx.x % count;
  if(type < 1 || !f.present[type]) {
    if(hist && term == 0 && threadIdx.x < 7) hist[type * 7 + threadIdx.x] = f.fit[type * 7 + threadIdx.x];
    return;
  }
  const double v = term == 0 ? fit_term<0>(f, type, term, from_stacks, sm.a)
                             : (term < 5 ? fit_term<1>(f, type, term, from_stacks, sm.a)
                                         : fit_term<2>(f, type, term, from_stacks, sm.b));
  if(threadIdx.x || from_stacks) return;
  // raw[type][w]: w = 0 S, 1 Sdisp_r, 2 Sdisp_t, 3 Sdisp_p, 4 Sdisp_q
  if(term == 0 || term >= 5) {
    *(volatile double *) &f.raw[type * 5 + (term ? term - 4 : 0)] = v;
    __threadfence();
    if(atomicInc(&f.arrived[type], 4) == 4) {  // (wraps to 0)
      __threadfence();
      fit_final(f, type);
      if(hist)
        for(int j = 0; j < 7; j++) hist[type * 7 + j] = f.fit[type * 7 + j];
    }
  }
}

// ---------------------------------------------------------------- optimize

__global__ void k_propose(DevModel M, RepArgs R)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if(k >= R.count) return;
  LogConsts L = make_log_consts(M);
  const int n = R.idx[k];
  const int type = R.p_type[n];
  const int tovs = M.tovs[type];
  const double *pos = &R.p_pos[3 * n];
  grng_t g;
  // repetition k / per_rep of a window of repetitions draws from its own serial
  grng_init(&g, R.seed, (uint32_t) n, R.rep_serial + (uint32_t) (R.per_rep > 0 ? k / R.per_rep : 0));
  (void) grng_uniform(&g);  // dir_rnd (main.c:370)
  double phi = gm_atan2(pos[1], pos[0]);
  double Rv[3], Tv[3], Qv[3];
  if(tovs == 2) {
    double c = gm_cos(phi), s = gm_sin(phi);
    Rv[0] = c; Rv[1] = s; Rv[2] = 0;
    Tv[0] = -s; Tv[1] = c; Tv[2] = 0;
    Qv[0] = 0; Qv[1] = 0; Qv[2] = 1;
  } else {
    double theta = gm_acos(pos[2] / sqrt(pos[0] * pos[0] + pos[1] * pos[1] + pos[2] * pos[2]));
    double st = gm_sin(theta), ct = gm_cos(theta), sp = gm_sin(phi), cp = gm_cos(phi);
    Rv[0] = st * cp; Rv[1] = st * sp; Rv[2] = ct;
    Tv[0] = -ct * cp; Tv[1] = -ct * sp; Tv[2] = st;
    Qv[0] = -sp; Qv[1] = cp; Qv[2] = 0;
  }
  const double *tg = &R.p_targets[4 * n];
  double sigma_r = sqrt(tg[0]), sigma_t = sqrt(tg[1]), sigma_p = sqrt(tg[2]);
  double vstr = vstream_at(M, fg_coord(M, L, pos), type);
  double v_new[3], v2_new;
  int iter = 0, st_code = 0;
  do {
    double vr_new = grng_gaussian(&g, sigma_r);
    double vt_new = grng_gaussian(&g, sigma_t);
    double vq_new = vstr + grng_gaussian(&g, sigma_p);
    for(int j = 0; j < 3; j++) v_new[j] = vr_new * Rv[j] + vt_new * Tv[j] + vq_new * Qv[j];
    v2_new = v_new[0] * v_new[0] + v_new[1] * v_new[1] + v_new[2] * v_new[2];
    iter++;
    if(iter > 100000) {  // main.c:432-433
      st_code = GALIC_ERR_REJECTION_CAP;
      break;
    }
  } while(sqrt(v2_new) >= M.MaxVelInUnitsVesc * R.p_vesc[n]);
  if(st_code) atomicMax(R.status, st_code);
  // what the trial would change in the energy grid (add_to_energy_grid)
  disp_components(M, L, type, pos, v_new, &R.try_disp[4 * k]);
  R.inst_cell[k] = energy_cell(M, L, pos);
  for(int j = 0; j < 3; j++) {
    R.vel_try[3 * k + j] = v_new[j];
    R.b_pos[3 * (2 * k) + j] = pos[j];
    R.b_pos[3 * (2 * k + 1) + j] = pos[j];
    R.b_vel[3 * (2 * k) + j] = R.p_vel[3 * n + j];
    R.b_vel[3 * (2 * k + 1) + j] = v_new[j];
  }
  R.b_mass[2 * k] = R.b_mass[2 * k + 1] = R.p_mass[n];
  R.b_time[2 * k] = R.b_time[2 * k + 1] = R.p_tint[n];
  R.b_type[2 * k] = R.b_type[2 * k + 1] = type;
}

// The stack terms of eval_fit_mod, to R.F[(2k + which) * NTERM + term]; which
// 0 = F_base, 1 = F_try.  What it needs is the old and trial orbits' grids once
// (10 x 2^2L doubles per particle); what an orbit leaves as it was keeps its
// committed value (f.values), so only the part of the grid that an orbit
// crosses costs leaf terms with their divisions.  One CTA per particle and term
// evaluates both sums from one read of the grids.
//   The base evaluation's instantaneous terms are not evaluated per particle:
// its velocity is the particle's own, whose projections are the committed ones
// (p_vdisp was computed from p_vel by the same disp_components), so the change
// it adds to the energy grid is exactly zero and the term is its type's
// committed misfit (f.values' root).  The trial's instantaneous terms change
// four finest nodes, at most four per level: four lanes climb the levels.
// 101 particles at level 6: 103 -> 33 us (cold caches), beside 12 and 4 -> 9 us
// for the acceptance and the list, 78 -> 14 us for the commit: a construction with
// 100 such repetitions 54 -> 41.5 ms.
constexpr int EVAL_BLOCK = 256;

// the trial's instantaneous term a (0-3: r, t, p, q) of particle k, on four
// neighbouring lanes: lane q = 2 dz + dR follows the corner (iz + dz, iR + dR)
__device__ __forceinline__ void eval_inst_term(const RepArgs &R, const FitArgs &f, int k, int a, bool act)
{
  const int lane = threadIdx.x & 31, q = lane & 3, quad = lane & ~3;
  const int n = R.idx[k], type = R.p_type[n];
  const int L = f.L, Ns = f.Nstack;
  const double *stk = f.stacks + ((size_t) type * NG_COMMITTED + kTermGrid[5 + a]) * Ns;
  const double *ms = f.stacks + ((size_t) type * NG_COMMITTED + GALIC_GRID_MASS_I) * Ns;
  const double *val = f.values + ((size_t) type * NTERM + 5 + a) * Ns;
  const TermLeaf<2> leaf(f, type, 5 + a);
  const double thr = f.thr_e[type];
  // add_to_energy_grid: vr2 *= mass etc. (main.c:885-888); order r, t, p, q
  const double dv = (R.try_disp[4 * k + a] - R.p_vdisp[4 * n + a]) * R.p_mass[n];
  const Cell cc = R.inst_cell[k];
  const double w = q == 0 ? (1 - cc.fR) * (1 - cc.fz)
                          : (q == 1 ? (cc.fR) * (1 - cc.fz) : (q == 2 ? (1 - cc.fR) * (cc.fz) : (cc.fR) * (cc.fz)));
  const int dz = q >> 1, dR = q & 1;
  // the two rows and columns that the corners' nodes have at this level
  int z0 = cc.iz, z1 = cc.iz + 1, r0 = cc.iR, r1 = cc.iR + 1;
  int node = stack_off(L) + ((dz ? z1 : z0) << L) + (dR ? r1 : r0);
  double d = stk[node] + w * dv;
  double v = leaf(node, d, ms[node]);
  for(int l = L - 1; l >= 0; l--) {
    const int pz = (dz ? z1 : z0) >> 1, pr = (dR ? r1 : r0) >> 1, cn = 2 << l;
    double cd[4], cv[4];
#pragma unroll
    for(int c = 0; c < 4; c++) {
      const int z = 2 * pz + (c >> 1), r = 2 * pr + (c & 1), at = stack_off(l + 1) + z * cn + r;
      const int iz = z == z0 ? 0 : (z == z1 ? 1 : -1), ir = r == r0 ? 0 : (r == r1 ? 1 : -1);
      const int src = quad + (iz > 0 ? 2 : 0) + (ir > 0 ? 1 : 0);
      const double sd = __shfl_sync(0xffffffffu, d, src), sv = __shfl_sync(0xffffffffu, v, src);
      const bool own = iz >= 0 && ir >= 0;
      cd[c] = own ? sd : stk[at];
      cv[c] = own ? sv : val[at];
    }
    node = stack_off(l) + (pz << l) + pr;
    const double m = ms[node];
    d = cd[0] + cd[2] + cd[1] + cd[3];
    if(m < thr) {
      v = leaf(node, d, m);
    } else {
      v = cv[0];
      v += cv[1];
      v += cv[2];
      v += cv[3];
    }
    z0 >>= 1, z1 >>= 1, r0 >>= 1, r1 >>= 1;
  }
  if(act && q == 0) R.F[(2 * k + 1) * NTERM + 5 + a] = v;
}

template <int KIND>
__device__ __forceinline__ void eval_orbit_term(const RepArgs &R, const FitArgs &f, int k, int term,
                                                Pyramid<2, false> &sm)
{
  const int n = R.idx[k], type = R.p_type[n];
  const int L = f.L, N = 1 << L, G = f.Ngrid, Ns = f.Nstack;
  // orbit fields m, r, t, q, p, as the terms
  const double *gold = R.grids + ((size_t) (2 * k) * NF_ORBIT + term) * G;
  const double *gnew = gold + (size_t) NF_ORBIT * G;
  // the orbit grids are stored unscaled: x mass/tall on the fly, the
  // operation k_scale_dense would have applied
  const double fo = R.b_mass[2 * k] / R.b_tall[2 * k], fn = R.b_mass[2 * k + 1] / R.b_tall[2 * k + 1];
  const double *c = f.stacks + ((size_t) type * NG_COMMITTED + kTermGrid[term]) * Ns + stack_off(L);
  const double *val = f.values + ((size_t) type * NTERM + term) * Ns;
  const TermLeaf<KIND> leaf(f, type, term);
  // committed + new - old
  auto children = [&](int g, double (&x)[2][4], double (&)[4]) {
    unsigned changed = 0;
#pragma unroll
    for(int z = 0; z < 2; z++) {
      const double2 o = *(const double2 *) &gold[g + z * N], w = *(const double2 *) &gnew[g + z * N];
      const double c0 = c[g + z * N], c1 = c[g + z * N + 1];
      x[0][2 * z] = c0 + o.x * fo - o.x * fo;
      x[0][2 * z + 1] = c1 + o.y * fo - o.y * fo;
      x[1][2 * z] = c0 + w.x * fn - o.x * fo;
      x[1][2 * z + 1] = c1 + w.y * fn - o.y * fo;
      changed |= (x[0][2 * z] != c0 || x[0][2 * z + 1] != c1 ? 1u : 0u) |
                 (x[1][2 * z] != c0 || x[1][2 * z + 1] != c1 ? 2u : 0u);
    }
    return changed;
  };
  double root[2];
  pyramid_cta<2, false>(sm, L, children, [&](int node) { return val[node]; }, leaf,
                        f.targets + ((size_t) type * NT_TARGET + T_DGM) * Ns, f.thr_d[type],
                        [](int, double, double, double) {}, [](int, double) {}, root);
  if(threadIdx.x == 0) {
    R.F[(2 * k) * NTERM + term] = root[0];
    R.F[(2 * k + 1) * NTERM + term] = root[1];
  }
}

// the first inst_blocks CTAs: the instantaneous terms
__global__ void __launch_bounds__(EVAL_BLOCK, 3)
    k_eval_terms(const __grid_constant__ RepArgs R, const __grid_constant__ FitArgs f, int inst_blocks)
{
  __shared__ Pyramid<2, false> sm;
  if((int) blockIdx.x < inst_blocks) {
    const int item = (int) (blockIdx.x * (EVAL_BLOCK / 4) + (threadIdx.x >> 2));
    const bool act = item < 4 * R.count;
    eval_inst_term(R, f, act ? item >> 2 : 0, act ? item & 3 : 0, act);
    return;
  }
  const int j = (int) blockIdx.x - inst_blocks, k = j / 5, term = j % 5;
  if(term == 0) eval_orbit_term<0>(R, f, k, term, sm);
  else eval_orbit_term<1>(R, f, k, term, sm);
}

// F of eval_fit_mod from its nine stack terms t[] (main.c:1047, 1120, 1195-1212)
__device__ __forceinline__ double combine_terms(const DevModel &M, const RepArgs &R, const FitArgs &f, int type,
                                                const double *t)
{
  const double MT = f.MType[type];
  double value = t[0];
  value *= 1.0 / MT;
  const double value_rs = t[1] / MT, value_ts = t[2] / MT, value_qs = t[3] / MT, value_ps = t[4] / MT;
  double value_r = t[5], value_t = t[6], value_p = t[7], value_q = t[8];
  if(M.tovs[type] == 0 || type == 2) value_q = 0;  // main.c:1195
  const double *fit = f.fit + type * 7;
  return value + fit[5] / fit[6] * (value_r + value_t + value_p + value_q) +
         (R.fac_rs[type] * value_rs + R.fac_ts[type] * value_ts + R.fac_ps[type] * value_ps +
          R.fac_qs[type] * value_qs) /
             4;
}

// Accepts and lists the accepted positions of each type in increasing order
// (one CTA, in rounds of its threads); k_commit loops over these instead of over
// every position.
__global__ void __launch_bounds__(1024) k_accept(const __grid_constant__ DevModel M, const __grid_constant__ RepArgs R,
                                                 const __grid_constant__ FitArgs f)
{
  __shared__ int warp_sum[3][32];
  int listed[3] = {0, 0, 0};  // accepted so far, types 1 to 3
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for(int k0 = 0; k0 < R.count; k0 += blockDim.x) {
    const int k = k0 + threadIdx.x;
    const bool act = k < R.count;
    int type = 0;
    bool acc = false;
    if(act) {
      const int n = R.idx[k];
      type = R.p_type[n];
      double tb[NTERM];
      for(int j = 0; j < 5; j++) tb[j] = R.F[(2 * k) * NTERM + j];
      for(int j = 0; j < 4; j++) tb[5 + j] = f.values[((size_t) type * NTERM + 5 + j) * f.Nstack];
      const double F_base = combine_terms(M, R, f, type, tb);
      const double F_try = combine_terms(M, R, f, type, &R.F[(2 * k + 1) * NTERM]);
      acc = F_try < F_base;  // main.c:468
      // mass/tall of the old and trial orbits (orbit_response.c:477-486) for
      // the commit, which reads the unscaled orbit grids
      R.fac[2 * k] = R.b_mass[2 * k] / R.b_tall[2 * k];
      R.fac[2 * k + 1] = R.b_mass[2 * k + 1] / R.b_tall[2 * k + 1];
      R.p_orbits[n] = R.b_norbit[2 * k + (acc ? 1 : 0)];  // main.c:460 writes the old orbit's count
      if(acc) {
        for(int j = 0; j < 3; j++) R.p_vel[3 * n + j] = R.vel_try[3 * k + j];
        double *vd = &R.p_vdisp[4 * n];
        const double mass = R.p_mass[n];
        for(int j = 0; j < 4; j++) {
          const double d = R.try_disp[4 * k + j];
          R.inst_v[4 * k + j] = (d - vd[j]) * mass;
          vd[j] = d;
        }
      }
    }
    int before[3];
#pragma unroll
    for(int t = 0; t < 3; t++) {
      const unsigned tried = __ballot_sync(0xffffffffu, act && type == t + 1),
                     m = __ballot_sync(0xffffffffu, acc && type == t + 1);
      before[t] = __popc(m & ((1u << lane) - 1));
      if(lane == 0) {
        warp_sum[t][wid] = __popc(m);
        if(tried) atomicAdd(&R.tries[t + 1], (unsigned long long) __popc(tried));
        if(m) atomicAdd(&R.changes[t + 1], (unsigned long long) __popc(m));
      }
    }
    __syncthreads();
#pragma unroll
    for(int t = 0; t < 3; t++) {
      int at = listed[t] + before[t];
      for(int w = 0; w < (int) (blockDim.x >> 5); w++) {
        if(w < wid) at += warp_sum[t][w];
        listed[t] += warp_sum[t][w];
      }
      if(acc && type == t + 1) R.acc_list[(size_t) t * R.count + at] = k;
    }
    __syncthreads();
  }
  if(threadIdx.x < 3) R.acc_n[threadIdx.x] = listed[threadIdx.x];
}

// Adds the accepted particles' changes to the committed grids, one thread per
// bin.  blockIdx.y = 6 (type - 1) + field: fields 0 to 4 the orbits', new - old;
// 5 the energy grid's four.  A thread's sum is a chain in particle order, so
// the accepted list is staged in shared memory and eight particles' values are
// on their way at a time (the grids were read once by the evaluation and mostly
// come from L2).
constexpr int COMMIT_BLOCK = 128, COMMIT_LIST = 256;

__global__ void __launch_bounds__(COMMIT_BLOCK) k_commit(const __grid_constant__ RepArgs R,
                                                         const __grid_constant__ FitArgs f)
{
  __shared__ int s_k[COMMIT_LIST];
  __shared__ double s_a[COMMIT_LIST], s_b[COMMIT_LIST];
  __shared__ double s_v[COMMIT_LIST][4];
  const int type = blockIdx.y / 6 + 1, fld = blockIdx.y % 6;
  if(!f.present[type]) return;
  const int G = f.Ngrid, Nb = 1 << f.L;
  const int na = R.acc_n[type - 1];
  const int *list = R.acc_list + (size_t) (type - 1) * R.count;
  const int i = blockIdx.x * COMMIT_BLOCK + threadIdx.x;
  double *dst = (double *) f.committed + (size_t) type * NG_COMMITTED * G + i;
  double delta[4] = {0, 0, 0, 0};
  for(int j0 = 0; j0 < na; j0 += COMMIT_LIST) {
    const int nj = min(COMMIT_LIST, na - j0);
    __syncthreads();
    for(int j = threadIdx.x; j < nj; j += COMMIT_BLOCK) {
      const int k = list[j0 + j];
      if(fld < 5) {
        // unscaled orbit grids: x mass/tall as k_scale_dense would (the
        // factors k_accept stored, the same divisions)
        s_k[j] = k;
        s_a[j] = R.fac[2 * k];
        s_b[j] = R.fac[2 * k + 1];
      } else {
        const Cell c = R.inst_cell[k];
        s_k[j] = c.iz * Nb + c.iR;
        s_a[j] = c.fR;
        s_b[j] = c.fz;
        // inst_v holds (vr2, vt2, vp2, vq2) differences times mass
        for(int a = 0; a < 4; a++) s_v[j][a] = R.inst_v[4 * k + a];
      }
    }
    __syncthreads();
    if(i >= G) continue;
    if(fld < 5) {
      const double *base = R.grids + (size_t) fld * G + i;
      const size_t orbit = (size_t) NF_ORBIT * G;
      int j = 0;
      for(; j + 8 <= nj; j += 8) {
        double o[8], w[8];
#pragma unroll
        for(int u = 0; u < 8; u++) {
          const double *g = base + (size_t) (2 * s_k[j + u]) * orbit;
          o[u] = g[0];
          w[u] = g[orbit];
        }
#pragma unroll
        for(int u = 0; u < 8; u++) delta[0] += w[u] * s_b[j + u] - o[u] * s_a[j + u];
      }
      for(; j < nj; j++) {
        const double *g = base + (size_t) (2 * s_k[j]) * orbit;
        delta[0] += g[orbit] * s_b[j] - g[0] * s_a[j];
      }
    } else {
      for(int j = 0; j < nj; j++) {
        const int at = i - s_k[j];
        const double fR = s_a[j], fz = s_b[j];
        double w;
        if(at == 0) w = (1 - fR) * (1 - fz);
        else if(at == 1) w = (fR) * (1 - fz);
        else if(at == Nb) w = (1 - fR) * (fz);
        else if(at == Nb + 1) w = (fR) * (fz);
        else continue;
#pragma unroll
        for(int a = 0; a < 4; a++) delta[a] += w * s_v[j][a];
      }
    }
  }
  if(i >= G) return;
  if(fld < 5) {
    // orbit fields m,r,t,q,p map to committed MASS_S, R_S, T_S, Q_S, P_S
    dst[(size_t) fld * G] += delta[0];
  } else {
#pragma unroll
    for(int a = 0; a < 4; a++) dst[(size_t) kTermGrid[5 + a] * G] += delta[a];
  }
}

}  // namespace

int launch_global_fit(const FitArgs &f, cudaStream_t s, double *hist, int first, int count)
{
  k_fit<<<4 * count, 1024, 0, s>>>(f, first, count, false, hist);
  return 1;
}

int launch_rep_orbits(const DevModel &M, const RepArgs &R, const OrbitBatch &b, cudaStream_t s,
                      const float4 *const *quad32, const float *cellsize32)
{
  const int count = R.count;
  k_propose<<<(count + 63) / 64, 64, 0, s>>>(M, R);
  cudaMemsetAsync(b.grids, 0, (size_t) b.count * NF_ORBIT * M.DG_Ngrid * sizeof(double), s);
  if(quad32)
    launch_orbits_dense_fp32(M, quad32, cellsize32, b, s);
  else
    launch_orbits_dense(M, b, s);
  // the grids stay unscaled: the merit and commit kernels multiply by
  // mass/tall where they read them (one pass over the grids less)
  return 2;
}

int launch_rep_values(const FitArgs &f, cudaStream_t s)
{
  k_fit<<<4 * NTERM, 1024, 0, s>>>(f, 0, NTERM, true, nullptr);
  return 1;
}

int launch_rep_commit(const DevModel &M, const RepArgs &R, const FitArgs &f, cudaStream_t s, double *hist)
{
  const int count = R.count, inst_blocks = (4 * count + EVAL_BLOCK / 4 - 1) / (EVAL_BLOCK / 4);
  k_eval_terms<<<inst_blocks + 5 * count, EVAL_BLOCK, 0, s>>>(R, f, inst_blocks);
  k_accept<<<1, count < 1024 ? (count + 31) / 32 * 32 : 1024, 0, s>>>(M, R, f);
  k_commit<<<dim3((f.Ngrid + COMMIT_BLOCK - 1) / COMMIT_BLOCK, 18), COMMIT_BLOCK, 0, s>>>(R, f);
  return 3 + launch_global_fit(f, s, hist);
}

RepArgs rep_slice(const RepArgs &R, int first, int count, int G)
{
  RepArgs S = R;
  S.count = count;
  S.per_rep = 0;
  S.idx = R.idx + first;
  S.b_pos = R.b_pos + 3 * (size_t) (2 * first);
  S.b_vel = R.b_vel + 3 * (size_t) (2 * first);
  S.b_mass = R.b_mass + 2 * (size_t) first;
  S.b_time = R.b_time + 2 * (size_t) first;
  S.b_type = R.b_type + 2 * (size_t) first;
  S.b_norbit = R.b_norbit + 2 * (size_t) first;
  S.b_tall = R.b_tall + 2 * (size_t) first;
  S.fac = R.fac + 2 * (size_t) first;
  S.grids = R.grids + (size_t) (2 * first) * NF_ORBIT * G;
  S.vel_try = R.vel_try + 3 * (size_t) first;
  S.F = R.F + 2 * (size_t) NTERM * first;
  S.acc_list = R.acc_list + 3 * (size_t) first;
  S.acc_n = R.acc_n + 3 * (size_t) (first / count);
  S.try_disp = R.try_disp + 4 * (size_t) first;
  S.inst_v = R.inst_v + 4 * (size_t) first;
  S.inst_cell = R.inst_cell + first;
  return S;
}

int launch_rep(const DevModel &M, const RepArgs &R, const FitArgs &f, const OrbitBatch &b, cudaStream_t s,
               const float4 *const *quad32, const float *cellsize32)
{
  const int launches = launch_rep_orbits(M, R, b, s, quad32, cellsize32);
  return launches + launch_rep_values(f, s) + launch_rep_commit(M, R, f, s, nullptr);
}
