// Device bytes of a context's arrays, for the admission of jobs (server.cpp).
// Kept in step with galic_ctx_create, galic_set_particles, ensure_tab32 and
// ensure_*_scratch (api.cu); tests/test_serving.py compares the sum with what
// the allocator hands out.
#ifndef GALIC_FOOTPRINT_H
#define GALIC_FOOTPRINT_H

#include <algorithm>
#include <cstddef>

namespace galic_footprint {

// FG_Pot and the two forces, three streaming velocities, three FP32 tables of
// four float4, per force-grid cell
constexpr size_t PER_CELL = 8 + 16 + 3 * 8 + 3 * 64;
// DG_CellSize in both precisions, [4][10] committed values and fixed-point
// word pairs, per response-grid bin
constexpr size_t PER_BIN = 8 + 4 + 4 * 10 * 8 + 4 * 10 * 16;
// distance, [4][6] targets, [4][10] stacks, [4][9] node values, per stack node
constexpr size_t PER_NODE = 8 + 4 * 6 * 8 + 4 * 10 * 8 + 4 * 9 * 8;
// pos, vel, mass, Tint, v_esc, targets, dispersions, type, orbits, order
constexpr size_t PER_PARTICLE = 24 + 24 + 3 * 8 + 32 + 32 + 3 * 4;
// while the order is made: keys and indices, and the sort's copies of them
constexpr size_t ORDER_PER_PARTICLE = 3 * 8 + 2 * 4;
// one orbit of a window beside its grids: start, mass, time span, tall, energy
// error, type, orbits, status, steps
constexpr size_t PER_ORBIT = 24 + 24 + 4 * 8 + 3 * 4 + 8;
// an optimised particle beside its two orbits: index, 3 list entries, 3 list
// lengths, projections and velocity of the trial, 2 x 9 merit terms, 2
// factors, change of the energy grid and its cell
constexpr size_t PER_TRIAL = 4 + 12 + 12 + 32 + 24 + 144 + 16 + 32 + 24;

constexpr size_t bins(int level) { return (size_t) 1 << (2 * level); }

inline size_t context(int fg_nbin, int level)
{
  return (size_t) fg_nbin * fg_nbin * PER_CELL + bins(level) * PER_BIN + (4 * bins(level) - 1) / 3 * PER_NODE;
}
// `trials` optimised particles with five FP64 grids per orbit
inline size_t window(size_t trials, int level)
{
  return trials * (2 * (5 * 8 * bins(level) + PER_ORBIT) + PER_TRIAL);
}
// n particles, and the larger of what their ordering and their repetitions
// need (the ordering's arrays are free before the first repetition)
inline size_t particles(size_t n, size_t repetitions) { return n * PER_PARTICLE + std::max(n * ORDER_PER_PARTICLE, repetitions); }

}  // namespace galic_footprint

#endif
