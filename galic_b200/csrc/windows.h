// Whether galic_optimize_reps runs the orbits of two windows at once (host).
#ifndef GALIC_WINDOWS_H
#define GALIC_WINDOWS_H

#include <cstddef>

// A window's orbit launch lasts as long as its longest orbit: while two
// windows leave the GPU room, their orbits run at once, on a stream each.
// largest: particles of the largest window (two orbits each).  Two windows of
// a halo + disk, their orbits one after the other and at once (ms, B200): 2010
// particles a window 27.8 and 17.4 (FP32, level 7), 22.7 and 15.6 (FP64, level
// 6); 4020 particles 35.6 and 25.0, 26.2 and 20.1.  It still gains somewhat
// above the line and ends doing so below 20 000: eight windows of 10 050
// 123.6 and 110.7, of 20 100 169.6 and 172.5 (FP64, level 6).
constexpr int PAIRED_WINDOW_MAX = 4096;
inline bool windows_paired(size_t windows, int largest) { return windows > 1 && largest <= PAIRED_WINDOW_MAX; }

#endif
