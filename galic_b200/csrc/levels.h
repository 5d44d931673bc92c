// The finest response grid: 128 x 128 bins.
#ifndef GALIC_LEVELS_H
#define GALIC_LEVELS_H

// What is sized for it: the merit pyramid's shared memory and its Z order
// (stack.cuh), a sampled map's whole stack in one CTA's shared memory
// (sampling.cu: 171 of 227 KiB), the 16-bit node index of a queue record
// (flush.cuh), the fixed array of the allocation-free entry point
// (noalloc_fp64.cu).
constexpr int GALIC_MAX_LEVEL = 7;

#endif
