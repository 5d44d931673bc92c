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
//
// A drain hands each record to five neighbouring lanes, one field each (six
// records a round, lanes 30 and 31 idle).  A node's words are contiguous
// (fixedpoint.cuh:FxNode), so one atomic instruction covers runs of five words,
// two sectors a record: L2 executes atomics by sector (a B200 does 1.85e11 /s
// of random isolated words, 4 to 5e11 words/s in runs of five), and the L1
// passes them on by sector too.  Measured on the halo + disk pass (1.2e6
// orbits, 4.8e9 orbit-steps, 1.3 records each), orbit kernel: FP32 156 ms with
// a record per lane and a grid per field, 141 ms so (126 ms without the
// atomics, 95 ms without the drain); FP64 324 and 300 ms (its L1 data stage
// 69 % and 58 % busy).  Other forms, FP64: ten lanes a record, one word each,
// 391 ms (half the conversions are redundant); two or four rounds unrolled 385
// and 323 ms; a record per lane, staged in shared memory and added by the copy
// engine's bulk reductions, 344 ms (the engine adds 6.2e10 records/s, but each
// lane's command and its proxy fence hold up the warp).
#ifndef GALIC_FLUSH_CUH
#define GALIC_FLUSH_CUH

#include "fixedpoint.cuh"
#include "kernels.cuh"
#include "levels.h"

// The four nodes of a cell by parity: node (z, r) lives in slot
// ((z & 1) << 1) | (r & 1), so that when an orbit moves to a neighbouring cell
// the nodes the two cells share keep their slots.
struct SlotNodes {
  int z[2], r[2];  // the even and the odd node along each axis
  __device__ __forceinline__ SlotNodes() : z{-1, -1}, r{-1, -1} {}
  __device__ __forceinline__ SlotNodes(int iR, int iz) : z{(iz + 1) & ~1, iz | 1}, r{(iR + 1) & ~1, iR | 1} {}
  __device__ __forceinline__ int index(int slot, int Nb) const { return z[slot >> 1] * Nb + r[slot & 1]; }
  // out[slot]: the slot's node is not one of `next`
  __device__ __forceinline__ void leaving(const SlotNodes &next, bool out[4]) const
  {
    const bool lz[2] = {z[0] != next.z[0], z[1] != next.z[1]}, lr[2] = {r[0] != next.r[0], r[1] != next.r[1]};
#pragma unroll
    for(int k = 0; k < 4; k++) out[k] = lz[k >> 1] || lr[k & 1];
  }
};

// T: the type of the sums (float, double)
template <int PER_, class T>
struct WarpQueueT {
  static constexpr int PER = PER_;
  static_assert(PER_ * 32 <= 256, "list entries are bytes");
  static_assert(1 << (2 * GALIC_MAX_LEVEL) <= 1 << 16, "node indices are 16 bits");
  T val[PER][5][33];             // the node's five sums (33: the five lanes of a record read distinct banks)
  T scale[2][32];                // per lane: {mass field, energy fields} fixed-point factors
  int gbase[32];                 // per lane: first node of its orbit's grid set
  unsigned short base[PER][32];  // the node's index in its grid
  unsigned char list[PER * 32];  // drain: the parked records, slot * 32 + lane
};
template <int PER>
using WarpQueue32 = WarpQueueT<PER, float>;
template <int PER>
using WarpQueue64 = WarpQueueT<PER, double>;

// records per lane of a block of BLOCK threads (FP32 sums)
__host__ __device__ constexpr int queue32_per(int block) { return block <= 128 ? 8 : (block <= 192 ? 7 : 5); }

// true when some lane could not park another cell's nodes
template <int PER>
__device__ __forceinline__ bool queue32_due(int cnt)
{
  return __any_sync(0xffffffffu, cnt > PER - 4);
}

// FP32 sums: value x 2^(shift-24) (the orbit's mass/Tint and the field's
// fixed-point scale folded into one FP32 factor per field class when the
// orbit starts) rounded to one signed 64-bit word.  shift - 24 is chosen so
// that no bin can overflow 2^62; the FP32 rounding of the scaled value (2^-24
// relative) is far inside the FP32 form's tolerance.
__device__ __forceinline__ void add_field(FxNode *n, int f, float t)
{
  const long long X = __float2ll_rn(t);
  if(X) atomicAdd(&n->hi[f], (unsigned long long) X);
}
// FP64 sums: the two-word pair of v = sum x mass/Tint (resolution 2^-S), so
// that the bins carry the full FP64 resolution whatever the headroom of the
// field's range.  The factor is mass/Tint x 2^(S-24), whose power of two is
// exact, so the pair is fx_split(v, S)'s bit for bit.
__device__ __forceinline__ void add_field(FxNode *n, int f, double t)
{
  long long H;
  unsigned long long L;
  fx_split_scaled(t, &H, &L);
  atomicAdd(&n->hi[f], (unsigned long long) H);
  atomicAdd(&n->lo[f], L);
}

// all 32 lanes call this at the same point of the loop with their record
// counts; cnt is 0 on return
template <int PER, class T>
__device__ __forceinline__ void warp_drain_nodes(WarpQueueT<PER, T> &q, FxNode *fx, int &cnt)
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
    add_field(&fx[q.gbase[l] + q.base[k][l]], f, q.val[k][f][l] * q.scale[f ? 1 : 0][l]);
  }
  __syncwarp();
  cnt = 0;
}

#endif
