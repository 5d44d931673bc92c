// CTA-cooperative versions of GALIC's stack routines.
//
// A stack holds a quadtree pyramid of a 2^L x 2^L grid; level l starts at
// STACKOFFSET(l,0,0) = (4^l - 1)/3 (allvars.h:160).
//
// stack_smooth_cta: smooth_stack (grid.c:1247-1265) of a whole stack in shared
//                   memory (L = 7: 21845 doubles, 171 KiB), level by level,
//                   same summation order.
// pyramid_cta:      smoothing and calc_stack_difference[_mod]
//                   (grid.c:1086-1151).  The reference recurses from the root
//                   and stops at a node when l == maxlevel or
//                   ref1[node] < thresh.  Evaluated bottom up instead: every
//                   node gets either its leaf term or the sum of its four
//                   children's values in the recursion's order
//                   ((c(2i,2j) + c(2i,2j+1)) + c(2i+1,2j)) + c(2i+1,2j+1),
//                   which gives the recursion's result bit for bit.
#ifndef GALIC_STACK_CUH
#define GALIC_STACK_CUH

#include "levels.h"

__host__ __device__ constexpr int stack_off(int l) { return ((1 << (2 * l)) - 1) / 3; }

__device__ __forceinline__ void stack_smooth_cta(double *s, int L)
{
  for(int l = L - 1; l >= 0; l--) {
    const int n = 1 << l, base = stack_off(l), cb = stack_off(l + 1), cn = n << 1;
    for(int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
      int i = idx >> l, j = idx & (n - 1);
      s[base + idx] = s[cb + (2 * i) * cn + 2 * j] + s[cb + (2 * i + 1) * cn + 2 * j] +
                      s[cb + (2 * i) * cn + 2 * j + 1] + s[cb + (2 * i + 1) * cn + 2 * j + 1];
    }
    __syncthreads();
  }
}

// leaf term; mode 0 = calc_stack_difference, 1 = calc_stack_difference_mod
__device__ __forceinline__ double stack_leaf(double d1, double d2, double r1, double r2, double dist, int flag,
                                             int mod, double R200_20, double lowdisp)
{
  if(mod && flag == 2) {
    if(r2 > 0) return fabs(d1 - d2) * (r1 / r2) / (dist < R200_20 ? dist : R200_20);
    return 0;
  }
  if(flag) {
    if(r1 > 0 && r2 > 0) {
      double q2 = d2 / r2;
      return fabs(d1 / r1 - q2) / (q2 > lowdisp ? q2 : lowdisp);
    }
    return 0;
  }
  return fabs(d1 - d2) / (dist < R200_20 ? dist : R200_20);
}

// Smoothing and misfit of W stacks at once, bottom up and without a stored
// stack.  Thread m takes the m-th node of level L - 1 in Z order with its four
// finest values, so a warp's lanes 4q .. 4q + 3 are the children of one node of
// level L - 2, and its 16-lane halves those of one of level L - 3: these levels
// go by shuffles, only the levels above go through shared memory (341 nodes at
// L = 7) and one warp finishes them.  The level-by-level form it replaces kept
// 43 to 171 KiB of stack in shared memory and met at a barrier after each of
// 2 L levels.  Orders of summation as in smooth_stack and the recursion.
//
//   children(g, x, m)  the finest values x[W][4] of the nodes g, g + 1, g + 2^L,
//                      g + 2^L + 1 (MASS: and the reference masses m[4]);
//                      returns the set of the W stacks that differ from the one
//                      with known node values
//   known(node)        these known values of the recursion at a node: an
//                      unchanged subtree's value is not computed again
//   leaf(node, d1, r1) leaf term
//   ref1               reference mass stack (MASS: summed from m instead)
//   keep(node, d1, v, r1), keep_leaf(node, v)
//                      called for the first stack's nodes: of the levels above the
//                      finest, and of the finest whose leaf terms are summed
template <int W, bool MASS>
struct Pyramid {
  static constexpr int NODES = stack_off(GALIC_MAX_LEVEL - 2);  // levels 0 .. L - 3
  double d[W][NODES], v[W][NODES], r[NODES];
};

static_assert(2 * (GALIC_MAX_LEVEL - 1) <= 12, "the nodes of level L - 1 in Z order");
__device__ __forceinline__ int z_order_half(int m)  // the even bits of m (12 bits)
{
  m &= 0x555;
  m = (m | (m >> 1)) & 0x333;
  m = (m | (m >> 2)) & 0x30f;
  return (m | (m >> 4)) & 0x3f;
}

template <int W, bool MASS, class Children, class Known, class Leaf, class Keep, class KeepLeaf>
__device__ __forceinline__ void pyramid_cta(Pyramid<W, MASS> &sm, int L, const Children &children, const Known &known,
                                            const Leaf &leaf, const double *ref1, double thresh, const Keep &keep,
                                            const KeepLeaf &keep_leaf, double *root)
{
  const int lane = threadIdx.x & 31;
  const int n1 = 1 << (L - 1), n2 = n1 * n1;
  const int b0 = stack_off(L), b1 = stack_off(L - 1), b2 = L >= 2 ? stack_off(L - 2) : 0,
            b3 = L >= 3 ? stack_off(L - 3) : 0;
  if(!MASS)
    for(int t = threadIdx.x; t < b3; t += blockDim.x) sm.r[t] = ref1[t];
  // d1 of a node from its children's, held by lanes c, c + s, c + 2s, c + 3s
  auto gather_d = [&](double x, int c, int s) {
    return __shfl_sync(0xffffffffu, x, c) + __shfl_sync(0xffffffffu, x, c + 2 * s) +
           __shfl_sync(0xffffffffu, x, c + s) + __shfl_sync(0xffffffffu, x, c + 3 * s);
  };
  auto gather_v = [&](double x, int c, int s) {
    double v = __shfl_sync(0xffffffffu, x, c);
    v += __shfl_sync(0xffffffffu, x, c + s);
    v += __shfl_sync(0xffffffffu, x, c + 2 * s);
    v += __shfl_sync(0xffffffffu, x, c + 3 * s);
    return v;
  };
  for(int m0 = threadIdx.x & ~31; m0 < n2; m0 += blockDim.x) {
    const bool act = m0 + lane < n2;
    const int m = act ? m0 + lane : 0;
    const int j = z_order_half(m), i = z_order_half(m >> 1);
    const int node1 = b1 + i * n1 + j, node2 = b2 + (i >> 1) * (n1 >> 1) + (j >> 1),
              node3 = b3 + (i >> 2) * (n1 >> 2) + (j >> 2);
    const int g = (2 * i) * (2 * n1) + 2 * j;
    double r1 = MASS ? 0.0 : ref1[node1], r2 = MASS || L < 2 ? 0.0 : ref1[node2], r3 = MASS || L < 3 ? 0.0 : ref1[node3];
    double x[W][4], mq[4], d[W], v[W];
    const unsigned changed = children(g, x, mq);
    if(MASS) r1 = mq[0] + mq[2] + mq[1] + mq[3];
#pragma unroll
    for(int w = 0; w < W; w++) {
      d[w] = x[w][0] + x[w][2] + x[w][1] + x[w][3];
      if(!(changed >> w & 1)) {
        v[w] = known(node1);
      } else if(r1 < thresh) {
        v[w] = leaf(node1, d[w], r1);
      } else {
        const int f[4] = {b0 + g, b0 + g + 1, b0 + g + 2 * n1, b0 + g + 2 * n1 + 1};
        double lv[4];
#pragma unroll
        for(int q = 0; q < 4; q++) lv[q] = leaf(f[q], x[w][q], MASS ? mq[q] : ref1[f[q]]);
        if(act && w == 0)
          for(int q = 0; q < 4; q++) keep_leaf(f[q], lv[q]);
        v[w] = lv[0];
        v[w] += lv[1];
        v[w] += lv[2];
        v[w] += lv[3];
      }
    }
    if(act) keep(node1, d[0], v[0], r1);
    if(L >= 2) {
      if(MASS) r2 = gather_d(r1, lane & ~3, 1);
#pragma unroll
      for(int w = 0; w < W; w++) {
        const double sum = gather_v(v[w], lane & ~3, 1);
        d[w] = gather_d(d[w], lane & ~3, 1);
        v[w] = r2 < thresh ? leaf(node2, d[w], r2) : sum;
      }
      if(act && (lane & 3) == 0) keep(node2, d[0], v[0], r2);
    }
    if(L >= 3) {
      if(MASS) r3 = gather_d(r2, lane & ~15, 4);
#pragma unroll
      for(int w = 0; w < W; w++) {
        const double sum = gather_v(v[w], lane & ~15, 4);
        d[w] = gather_d(d[w], lane & ~15, 4);
        v[w] = r3 < thresh ? leaf(node3, d[w], r3) : sum;
      }
      if(act && (lane & 15) == 0) keep(node3, d[0], v[0], r3);
    }
    if(act && (lane & 15) == 0) {
      const int at = L >= 3 ? node3 : 0;
#pragma unroll
      for(int w = 0; w < W; w++) {
        sm.d[w][at] = d[w];
        sm.v[w][at] = v[w];
      }
      if(MASS) sm.r[at] = r3;
    }
  }
  __syncthreads();
  if(threadIdx.x < 32)
    for(int l = L - 4; l >= 0; l--) {
      const int n = 1 << l, base = stack_off(l), cb = stack_off(l + 1), cn = n << 1;
      for(int t = lane; t < n * n * W; t += 32) {
        const int w = t >> (2 * l), idx = t & (n * n - 1), i = idx >> l, j = idx & (n - 1);
        const int c = cb + (2 * i) * cn + 2 * j;
        const double *cd = sm.d[w], *cv = sm.v[w];
        const double dn = cd[c] + cd[c + cn] + cd[c + 1] + cd[c + cn + 1];
        const double rn = MASS ? sm.r[c] + sm.r[c + cn] + sm.r[c + 1] + sm.r[c + cn + 1] : sm.r[base + idx];
        double vn = cv[c];
        vn += cv[c + 1];
        vn += cv[c + cn];
        vn += cv[c + cn + 1];
        if(rn < thresh) vn = leaf(base + idx, dn, rn);
        sm.d[w][base + idx] = dn;
        sm.v[w][base + idx] = vn;
        if(MASS) sm.r[base + idx] = rn;
        if(w == 0) keep(base + idx, dn, vn, rn);
      }
      __syncwarp();
    }
#pragma unroll
  for(int w = 0; w < W; w++) root[w] = sm.v[w][0];  // (valid in the first warp)
}

#endif
