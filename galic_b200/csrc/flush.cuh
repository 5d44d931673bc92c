// Warp-cooperative flush of node sums into the fixed-point grids.
//
// Each lane of the batched orbit kernels sums the deposits of consecutive
// steps per grid node in registers.  When a node leaves its cell, the lane
// parks one record (the node's index and its five sums) in its own column of
// the warp's queue (no reservation atomic).  A lane parks at most 4 records
// per loop iteration (one cell's nodes), so the warp drains before any lane
// could pass PER; the drain takes all lanes' records together, so that the
// global atomics run on full warps.  PER is chosen per block size so that the
// queues fit the static shared memory.
#ifndef GALIC_FLUSH_CUH
#define GALIC_FLUSH_CUH

#include "fixedpoint.cuh"
#include "kernels.cuh"

// true when some lane could not park another cell's nodes
template <int PER>
__device__ __forceinline__ bool queue32_due(int cnt)
{
  return __any_sync(0xffffffffu, cnt > PER - 4);
}

// ---------------------------------------------------------------- FP32 sums

template <int PER_>
struct WarpQueue32 {
  static constexpr int PER = PER_;
  static_assert(PER_ * 32 <= 256, "list entries are bytes");
  float val[PER][5][33];         // the node's five sums (33: the five lanes of a record read distinct banks)
  float scale[2][32];            // per lane: {mass field, energy fields} fixed-point factors
  int gbase[32];                 // per lane: first node of its orbit's grid set
  unsigned short base[PER][32];  // the node's index in its grid
  unsigned char list[PER * 32];  // drain: the parked records, slot * 32 + lane
};

// records per lane of a block of BLOCK threads
__host__ __device__ constexpr int queue32_per(int block) { return block <= 128 ? 8 : (block <= 192 ? 7 : 5); }

// Every value is scaled by 2^(shift-24) mass/Tint (one FP32 factor per field
// class, formed when the orbit starts) and rounded to one signed 64-bit word.
// shift - 24 is chosen so that no bin can overflow 2^62; the FP32 rounding of
// the scaled value (2^-24 relative) is far inside the FP32 form's tolerance.
//
// The words are stored node by node (fixedpoint.cuh:FxNode32), and a record
// is handed to five neighbouring lanes, one field each (six records at a
// time, lanes 30 and 31 idle): one atomic instruction then covers runs of
// five consecutive words, 2-3 sectors a record.  L2 executes atomics by
// sector (a B200 does 1.85e11 /s of random isolated words, 4 to 5e11 words/s
// in runs of five).  With a record per lane and field-major grids, five
// isolated words a record, the halo + disk pass of 1.2e6 orbits (4.8e9
// orbit-steps, 1.3 records each) ran 156 ms; so it runs 141 ms (126 ms
// without the atomics, 95 ms without the drain).
//
// All 32 lanes call this at the same point of the loop with their record
// counts; cnt is 0 on return.
template <int PER>
__device__ __forceinline__ void warp_drain32(WarpQueue32<PER> &q, FxNode32 *fx, int &cnt)
{
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int incl = cnt;
#pragma unroll
  for(int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, o);
    if(lane >= o) incl += y;
  }
  const int at = incl - cnt;
#pragma unroll
  for(int k = 0; k < PER; k++)
    if(k < cnt) q.list[at + k] = (unsigned char) (k * 32 + lane);
  __syncwarp();
  const int total = __shfl_sync(FULL, incl, 31);
  const int grp = lane / 5, f = lane - 5 * grp;
  for(int r = lane < 30 ? grp : total; r < total; r += 6) {
    const int e = q.list[r], k = e >> 5, l = e & 31;
    const long long X = __float2ll_rn(q.val[k][f][l] * q.scale[f ? 1 : 0][l]);
    if(X) atomicAdd(&fx[q.gbase[l] + q.base[k][l]].w[f], (unsigned long long) X);
  }
  __syncwarp();
  cnt = 0;
}

// ---------------------------------------------------------------- FP64 sums

template <int PER_>
struct WarpQueue64 {
  static constexpr int PER = PER_;
  int base[PER][32];       // the node's index in its grid (field f of the orbit's set: gbase + f * Ngrid + base)
  double val[PER][5][32];  // the node's five sums
  int off[32];             // drain: first compacted record of each lane
  int gbase[32];           // per lane: first word of its orbit's grid set
  double scale[2][32];     // per lane: {mass field, energy fields} fixed-point factors
};

// Every value v = sum x mass/Tint is added as the two-word fixed-point pair
// of fixedpoint.cuh:fx_add (resolution 2^-S, two integer atomics), so the bins
// carry the full FP64 resolution whatever the headroom of the field's range.
// The lane header holds mass/Tint x 2^(S-24) per field class (scale), which
// gives the pair of fx_add(v, S) bit for bit: the power-of-two factor is
// exact.  A record per lane here: its five conversions overlap.  Five lanes
// per record with node-major words, as above, ran 584 ms against 378 ms (the
// conversions become a serial chain per round; 475 ms with four rounds
// unrolled), a record per lane with node-major pairs 440 ms (the lanes of one
// atomic instruction then touch 32 lines).
template <int PER>
__device__ __forceinline__ void warp_drain64(WarpQueue64<PER> &q, FxWord *fx, int G, int &cnt)
{
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int incl = cnt;
#pragma unroll
  for(int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, o);
    if(lane >= o) incl += y;
  }
  const int total = __shfl_sync(FULL, incl, 31);
  q.off[lane] = incl - cnt;
  __syncwarp();
  for(int r = lane; r < total; r += 32) {
    // the lane L whose records hold r: the last L with off[L] <= r
    int L = 0;
#pragma unroll
    for(int step = 16; step; step >>= 1)
      if(q.off[L + step] <= r) L += step;
    const int k = r - q.off[L];
    const int b = q.gbase[L] + q.base[k][L];
    const double sm = q.scale[0][L], se = q.scale[1][L];
#pragma unroll
    for(int f = 0; f < 5; f++) fx_add_scaled(&fx[b + f * G], q.val[k][f][L] * (f == 0 ? sm : se));
  }
  __syncwarp();
  cnt = 0;
}

#endif
