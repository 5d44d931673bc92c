// FP64 orbit-response kernels (built with --fmad=false).
//
//  k_orbits_dense   produce_orbit_response_field[_mod] (orbit_response.c:33-491)
//                   with reference semantics: one thread per orbit, dense
//                   per-orbit grids accumulated in the reference's order.
//  k_scale_dense    the mass/tall normalisation (orbit_response.c:475-486).
//  k_calc_all_fp64  calc_all_response_fields (main.c:151-231): persistent
//                   threads pull orbits from a work counter; deposits of
//                   consecutive steps are summed per grid node in registers
//                   and flushed as exact fixed-point atomics into the
//                   per-type grids when their node leaves the orbit's cell.
//  k_instantaneous  calc_disp_components_for_particle + add_to_energy_grid
//                   (main.c:226-229).
//  k_fx_finalize    fixed-point words -> FP64 committed grids.
#include <cuda_runtime.h>

#include "flush.cuh"
#include "kernels.cuh"

namespace {

// the weights of a half step for cell c's nodes in slot order (products in
// the order of orbit_response.c:277-320)
__device__ __forceinline__ void slot_weights(const Cell &c, double hdt, double w[4])
{
  const bool oz = c.iz & 1, orr = c.iR & 1;
  const double z0 = oz ? c.fz : 1 - c.fz, z1 = oz ? 1 - c.fz : c.fz;
  const double r0 = orr ? c.fR : 1 - c.fR, r1 = orr ? 1 - c.fR : c.fR;
  w[0] = hdt * r0 * z0;
  w[1] = hdt * r1 * z0;
  w[2] = hdt * r0 * z1;
  w[3] = hdt * r1 * z1;
}

// The orbit's own dense grids [NF_ORBIT][G] in global memory.  The bins of
// the cell the orbit is in are held in registers, by slot: a deposit adds to
// them in the reference's order per bin (bin += value); when the orbit moves
// to another cell, enter() stores the bins whose node leaves and loads those
// of the nodes that come in, and finish() stores the last cell's.  Each
// orbit's grids are its own, so every bin receives the reference's sequence of
// roundings.  enter() is called before the step's projections, so that they
// cover the loads.
struct DenseSink {
  double *grid;
  int G, Nb;
  int with_egy;
  bool held = false;
  SlotNodes node;  // the held cell's nodes
  double c[4][5];
  __device__ __forceinline__ void store_slots(const bool which[4])
  {
#pragma unroll
    for(int k = 0; k < 4; k++) {
      if(!which[k]) continue;
      double *g = grid + node.index(k, Nb);
      g[F_M * G] = c[k][0];
      if(with_egy) {
        g[F_R * G] = c[k][1];
        g[F_T * G] = c[k][2];
        g[F_Q * G] = c[k][3];
        g[F_P * G] = c[k][4];
      }
    }
  }
  __device__ __forceinline__ void enter(int iR, int iz)
  {
    const SlotNodes next(iR, iz);
    bool out[4];
    node.leaving(next, out);
    if(held) store_slots(out);
    held = true;
    node = next;
#pragma unroll
    for(int k = 0; k < 4; k++) {
      if(!out[k]) continue;
      const double *g = grid + node.index(k, Nb);
      c[k][0] = g[F_M * G];
      if(with_egy) {
        c[k][1] = g[F_R * G];
        c[k][2] = g[F_T * G];
        c[k][3] = g[F_Q * G];
        c[k][4] = g[F_P * G];
      }
    }
  }
  __device__ __forceinline__ void add(const Cell &cell, double hdt, double next_hdt, const Proj &p)
  {
    double w[4], n[4];
    slot_weights(cell, hdt, w);
    slot_weights(cell, next_hdt, n);
#pragma unroll
    for(int k = 0; k < 4; k++) {
      c[k][0] = c[k][0] + w[k] + n[k];
      if(with_egy) {
        c[k][1] = c[k][1] + w[k] * p.vr2 + n[k] * p.vr2;
        c[k][2] = c[k][2] + w[k] * p.vt2 + n[k] * p.vt2;
        c[k][3] = c[k][3] + w[k] * p.vq2 + n[k] * p.vq2;
        c[k][4] = c[k][4] + w[k] * p.vp2 + n[k] * p.vp2;
      }
    }
  }
  __device__ __forceinline__ void add(const Cell &cell, double hdt, const Proj &p)
  {
    double w[4];
    slot_weights(cell, hdt, w);
#pragma unroll
    for(int k = 0; k < 4; k++) {
      c[k][0] = c[k][0] + w[k];
      if(with_egy) {
        c[k][1] = c[k][1] + w[k] * p.vr2;
        c[k][2] = c[k][2] + w[k] * p.vt2;
        c[k][3] = c[k][3] + w[k] * p.vq2;
        c[k][4] = c[k][4] + w[k] * p.vp2;
      }
    }
  }
  __device__ __forceinline__ void finish()
  {
    const bool all[4] = {true, true, true, true};
    if(held) store_slots(all);
  }
};

__global__ void k_orbits_dense(const __grid_constant__ DevModel M, OrbitBatch b)
{
  const int k = dense_orbit(b.count);
  if(k < 0) return;
  LogConsts L = step_log_consts(M);
  const size_t G = (size_t) M.DG_Ngrid;
  DenseSink sink;
  sink.grid = b.grids + (size_t) k * NF_ORBIT * G;
  sink.G = (int) G;
  sink.Nb = M.DG_Nbin;
  sink.with_egy = b.with_egy;
  OrbitState s;
  orbit_begin(M, L, s, &b.pos[3 * k], &b.vel[3 * k], b.timespan[k], b.type[k], b.with_egy != 0, sink);
  while(orbit_step(M, L, s, b.with_egy != 0, sink)) {
  }
  sink.finish();
  b.tall[k] = s.tall;
  b.norbit[k] = s.norbit;
  b.steps[k] = s.steps;
  b.status[k] = s.status;
  b.egy_err[k] = s.status == ORBIT_OK ? orbit_energy_error(M, L, s) : -1.0;
}

// grids[k][f][i] *= mass[k] / tall[k]
__global__ void k_scale_dense(OrbitBatch b, int G)
{
  const size_t per = (size_t) NF_ORBIT * G;
  const size_t total = per * b.count;
  for(size_t idx = blockIdx.x * (size_t) blockDim.x + threadIdx.x; idx < total; idx += (size_t) gridDim.x * blockDim.x) {
    int k = (int) (idx / per);
    int f = (int) ((idx - k * per) / G);
    if(!b.with_egy && f != F_M) continue;
    double fac = b.mass[k] / b.tall[k];
    b.grids[idx] *= fac;
  }
}

// Node sink of the batched path.  The deposits of consecutive steps are
// summed per grid NODE in FP64 registers, by slot (see SlotNodes).  Only the
// slots whose node leaves are parked, as records {node index, 5 sums}, in the
// lane's column of the warp's queue; the warp drains all lanes' records
// together (flush.cuh:warp_drain_nodes), each value scaled by mass/Tint and added
// as an exact two-word fixed-point pair (order independent).
template <int PER>
struct NodeSink64 {
  WarpQueue64<PER> *q;
  int lane, Nb;
  int cnt;  // records parked in this lane's column since the last drain
  SlotNodes node;  // the current cell's nodes
  double a[4][5];
  // fac x 2^(shift - 24) of the mass and the energy fields (exact scalings)
  __device__ __forceinline__ void set_orbit(int gbase, double scale_m, double scale_e)
  {
    q->gbase[lane] = gbase;
    q->scale[0][lane] = scale_m;
    q->scale[1][lane] = scale_e;
#pragma unroll
    for(int s = 0; s < 4; s++)
#pragma unroll
      for(int f = 0; f < 5; f++) a[s][f] = 0.0;
  }
  // parks the slots in out that hold a deposit (a node without mass has none)
  __device__ __forceinline__ void park_masked(const bool out[4])
  {
    // straight-line code for every lane of the warp: some lane of 32 changes
    // cell on nearly every step
#pragma unroll
    for(int s = 0; s < 4; s++) {
      if(out[s] && a[s][0] != 0.0) {
        q->base[cnt][lane] = (unsigned short) node.index(s, Nb);
#pragma unroll
        for(int f = 0; f < 5; f++) q->val[cnt][f][lane] = a[s][f];
        cnt++;
      }
    }
  }
  __device__ __forceinline__ void park()
  {
    const bool all[4] = {true, true, true, true};
    park_masked(all);
  }
  __device__ __forceinline__ void enter(int iR, int iz)
  {
    const SlotNodes next(iR, iz);
    if(next.z[0] == node.z[0] && next.z[1] == node.z[1] && next.r[0] == node.r[0] && next.r[1] == node.r[1]) return;
    bool out[4];
    node.leaving(next, out);
    park_masked(out);
#pragma unroll
    for(int s = 0; s < 4; s++)
      if(out[s]) {
#pragma unroll
        for(int f = 0; f < 5; f++) a[s][f] = 0.0;
      }
    node = next;
  }
  // the node sums are this form's own partial sums (the reference adds
  // every product to the grid bin in turn): fused, one rounding per term
  __device__ __forceinline__ void add(const Cell &cell, double hdt, double next_hdt, const Proj &p)
  {
    double w[4], n[4];
    slot_weights(cell, hdt, w);
    slot_weights(cell, next_hdt, n);
#pragma unroll
    for(int k = 0; k < 4; k++) {
      a[k][0] = a[k][0] + w[k] + n[k];
      a[k][1] = fma(n[k], p.vr2, fma(w[k], p.vr2, a[k][1]));
      a[k][2] = fma(n[k], p.vt2, fma(w[k], p.vt2, a[k][2]));
      a[k][3] = fma(n[k], p.vq2, fma(w[k], p.vq2, a[k][3]));
      a[k][4] = fma(n[k], p.vp2, fma(w[k], p.vp2, a[k][4]));
    }
  }
  __device__ __forceinline__ void add(const Cell &cell, double hdt, const Proj &p)
  {
    double w[4];
    slot_weights(cell, hdt, w);
#pragma unroll
    for(int k = 0; k < 4; k++) {
      a[k][0] = a[k][0] + w[k];
      a[k][1] = fma(w[k], p.vr2, a[k][1]);
      a[k][2] = fma(w[k], p.vt2, a[k][2]);
      a[k][3] = fma(w[k], p.vq2, a[k][3]);
      a[k][4] = fma(w[k], p.vp2, a[k][4]);
    }
  }
};

__device__ __forceinline__ void atomic_max_nonneg(double *addr, double v)
{
  // non-negative doubles order like their bit patterns
  if(!(v >= 0)) return;
  atomicMax((unsigned long long *) addr, (unsigned long long) __double_as_longlong(v));
}

enum LaneState { LANE_ACTIVE = 0, LANE_FINISH = 1, LANE_DONE = 2, LANE_START = 3 };

// records per lane of the FP64 queue (FP64 sums: 40 B per record and lane)
constexpr int kPer64 = 8;

template <int MINB>
__global__ void __launch_bounds__(CALC_ALL_BLOCK_FP64, MINB) k_calc_all_fp64(const __grid_constant__ DevModel M, CalcAllArgs A)
{
  __shared__ WarpQueue64<kPer64> queues[CALC_ALL_BLOCK_FP64 / 32];
  // the CTA's step count, largest energy error (as bits: non-negative
  // doubles order like them) and worst status, added to at each orbit's end
  // instead of being held in every thread's registers
  __shared__ unsigned long long cta_steps, cta_err_bits;
  __shared__ int cta_status;
  if(threadIdx.x == 0) {
    cta_steps = 0;
    cta_err_bits = 0;
    cta_status = 0;
  }
  __syncthreads();
  LogConsts L = step_log_consts(M);
  const int G = M.DG_Ngrid;
  OrbitState s;
  NodeSink64<kPer64> sink;
  sink.q = &queues[threadIdx.x >> 5];
  sink.lane = threadIdx.x & 31;
  sink.Nb = M.DG_Nbin;
  sink.cnt = 0;
  int p = -1;

  // starts orbit number k of this launch on this lane; false when there is none
  const FirstOrbit first;
  auto fetch = [&](int k) -> bool {
    if(k >= A.n) {
      p = -1;
      return false;
    }
    k = A.first + k * A.stride;
    p = A.order ? A.order[k] : k;
    const int type = A.type[p];
    const double fac = A.mass[p] / A.tint[p];
    sink.set_orbit(2 * type * G, ldexp(fac, A.shift[type * NG_COMMITTED + GALIC_GRID_MASS_S] - 24),
                   ldexp(fac, A.shift[type * NG_COMMITTED + GALIC_GRID_R_S] - 24));
    orbit_begin(M, L, s, &A.pos[3 * p], &A.vel[3 * p], A.tint[p], type, true, sink);
    return true;
  };

  int state = fetch(first.index) ? LANE_ACTIVE : LANE_DONE;
  for(;;) {
    const bool all_done = !__any_sync(0xffffffffu, state != LANE_DONE);
    // records take the orbit's grid set and scale from the lane's queue
    // header: a lane's records are drained before it starts the next orbit
    if(queue32_due<kPer64>(sink.cnt) ||
       __any_sync(0xffffffffu, (all_done || state == LANE_START) && sink.cnt > 0))
      warp_drain_nodes(*sink.q, (FxNode *) A.fx, sink.cnt);
    if(all_done) break;
    if(state == LANE_ACTIVE) {
      if(!orbit_step(M, L, s, true, sink)) state = LANE_FINISH;
    } else if(state == LANE_FINISH) {
      sink.park();
      A.orbits[p] = s.norbit;
      atomicAdd(&cta_steps, (unsigned long long) s.steps);
      if(s.status != ORBIT_OK)
        atomicMax(&cta_status, s.status);
      else {
        const double e = orbit_energy_error_from(M, L, s, &A.pos[3 * p], &A.vel[3 * p]);
        if(e >= 0) atomicMax(&cta_err_bits, (unsigned long long) __double_as_longlong(e));
      }
      state = LANE_START;
    } else if(state == LANE_START) {
      state = fetch(first.lanes + atomicAdd(A.next, 1)) ? LANE_ACTIVE : LANE_DONE;
    }
  }
  __syncthreads();
  if(threadIdx.x == 0) {
    if(cta_steps) atomicAdd(A.steps_total, cta_steps);
    atomic_max_nonneg(A.max_egy_err, __longlong_as_double((long long) cta_err_bits));
    if(cta_status) atomicMax(A.status, cta_status);
  }
}

// main.c:226-229 for every particle: vdisp = projections of the current
// velocity; the instantaneous energy grids get mass and mass * v^2
__global__ void k_instantaneous(DevModel M, int n, int first, int stride, const double *pos, const double *vel,
                                const double *mass, const int *type, double *vdisp, FxWord *fx, const int *shift,
                                int Ngrid)
{
  int k = first + (blockIdx.x * blockDim.x + threadIdx.x) * stride;
  if(k >= n) return;
  LogConsts L = step_log_consts(M);
  int t = type[k];
  double d[4];
  disp_components(M, L, t, &pos[3 * k], &vel[3 * k], d);
  for(int j = 0; j < 4; j++) vdisp[4 * k + j] = d[j];
  // add_to_energy_grid (main.c:877-917)
  Cell c = energy_cell(M, L, &pos[3 * k]);
  const int Nb = 1 << M.EG_L;
  double m = mass[k];
  double vr2 = d[0] * m, vt2 = d[1] * m, vp2 = d[2] * m, vq2 = d[3] * m;
  const int cells[4] = {c.iz * Nb + c.iR, c.iz * Nb + c.iR + 1, (c.iz + 1) * Nb + c.iR, (c.iz + 1) * Nb + c.iR + 1};
  const double w[4] = {(1 - c.fR) * (1 - c.fz), (c.fR) * (1 - c.fz), (1 - c.fR) * (c.fz), (c.fR) * (c.fz)};
  FxWord *g = fx + (size_t) t * NG_COMMITTED * Ngrid;
  const int *sh = shift + t * NG_COMMITTED;
  for(int j = 0; j < 4; j++) {
    fx_add(&g[(size_t) GALIC_GRID_MASS_I * Ngrid + cells[j]], w[j] * m, sh[GALIC_GRID_MASS_I]);
    fx_add(&g[(size_t) GALIC_GRID_R_I * Ngrid + cells[j]], w[j] * vr2, sh[GALIC_GRID_R_I]);
    fx_add(&g[(size_t) GALIC_GRID_T_I * Ngrid + cells[j]], w[j] * vt2, sh[GALIC_GRID_T_I]);
    fx_add(&g[(size_t) GALIC_GRID_P_I * Ngrid + cells[j]], w[j] * vp2, sh[GALIC_GRID_P_I]);
    fx_add(&g[(size_t) GALIC_GRID_Q_I * Ngrid + cells[j]], w[j] * vq2, sh[GALIC_GRID_Q_I]);
  }
}

// The time-averaged half of every set holds FxNode words (one_word: the FP32
// form's single words), the instantaneous half word pairs grid by grid.
// The grids first .. first + per - 1 of each of the sets.
__global__ void k_fx_finalize(const FxWord *fx, const int *shift, double *out, int sets, int first, int per, int Ngrid,
                              bool one_word)
{
  const size_t total = (size_t) sets * per * Ngrid;
  for(size_t j = blockIdx.x * (size_t) blockDim.x + threadIdx.x; j < total; j += (size_t) gridDim.x * blockDim.x) {
    const int set = (int) (j / Ngrid) / per, f = first + (int) (j / Ngrid) % per, g = set * NG_COMMITTED + f;
    const size_t i = (size_t) g * Ngrid + j % Ngrid;
    FxWord w;
    if(f < NF_ORBIT) {
      // (a set's first five grids are half of its NG_COMMITTED)
      const FxNode *n = (const FxNode *) fx + (size_t) set * 2 * Ngrid + j % Ngrid;
      w.hi = n->hi[f];
      w.lo = one_word ? 0 : n->lo[f];
    } else
      w = fx[i];
    out[i] = fx_value(w, shift[g]);
  }
}

}  // namespace

void launch_orbits_dense(const DevModel &M, const OrbitBatch &b, cudaStream_t s)
{
  int block = 64;
  const int grid = dense_grid(b.count, block);
  if(b.count > 0) k_orbits_dense<<<grid, block, 0, s>>>(M, b);
}

void launch_scale_dense(const DevModel &M, const OrbitBatch &b, cudaStream_t s)
{
  size_t total = (size_t) NF_ORBIT * M.DG_Ngrid * b.count;
  int grid = (int) ((total + 255) / 256);
  if(grid > 148 * 16) grid = 148 * 16;
  if(grid > 0) k_scale_dense<<<grid, 256, 0, s>>>(b, M.DG_Ngrid);
}

int calc_all_occupancy(int block)
{
  int blocks = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_calc_all_fp64<GALIC_FP64_MIN_BLOCKS>, block, 0);
  return blocks;
}

int launch_calc_all_fp64(const DevModel &M, const CalcAllArgs &a, int grid, int block, cudaStream_t s)
{
  k_calc_all_fp64<GALIC_FP64_MIN_BLOCKS><<<grid, block, 0, s>>>(M, a);
  return 1;
}

void launch_instantaneous(const DevModel &M, int n, const double *pos, const double *vel, const double *mass,
                          const int *type, double *vdisp, FxWord *fx, const int *shift, int Ngrid, cudaStream_t s,
                          int first, int stride)
{
  if(n <= first || stride < 1) return;
  const int count = (n - first + stride - 1) / stride;
  k_instantaneous<<<(count + 127) / 128, 128, 0, s>>>(M, n, first, stride, pos, vel, mass, type, vdisp, fx, shift,
                                                      Ngrid);
}

void launch_fx_finalize(const FxWord *fx, const int *shift, double *committed, int sets, int first, int per, int Ngrid,
                        int form, cudaStream_t s)
{
  size_t total = (size_t) sets * per * Ngrid;
  int grid = (int) ((total + 255) / 256);
  if(grid > 148 * 8) grid = 148 * 8;
  k_fx_finalize<<<grid, 256, 0, s>>>(fx, shift, committed, sets, first, per, Ngrid, form == GALIC_FORM_FP32);
}
