"""The orbit step's branch-free arithmetic (galic_b200/csrc/stepmath.cuh) equals the general functions bit for bit.

The kernels take it for operands in its stated ranges and the general
functions otherwise; the per-orbit parity tests cover whole orbits, these the
functions themselves (random operands, quotients and roots next to rounding
boundaries, table and octant edges) and orbits whose operands leave the ranges."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from galic_b200 import Context, synth
from oracle_lib import Oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include "gmath.h"
#include "stepmath.cuh"
__global__ void k_cmp(int n, const double *a, const double *b, int what, unsigned *bad)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= n) return;
  const double x = a[i], y = b[i];
  bool ok = true;
  unsigned ones = 0;  // operands the functions refuse
  if(what == 0) ok = step_div(x, y, ones) == x / y || step_ones(ones);
  if(what == 1) ok = step_sqrt(x) == sqrt(x);
  if(what == 2) ok = step_log(x) == gm_log(x);
  if(what == 3) {
    double s, c, s0, c0;
    step_direction(x, y, &s, &c, ones);
    gm_sincos(gm_atan2(x, y), &s0, &c0);
    ok = (s == s0 && c == c0) || step_ones(ones);
  }
  if(what == 4) {
    const StepFloor f = step_floor(x);
    ok = f.i == (int) x && f.d == (double) (int) x;
  }
  if(!ok) atomicAdd(bad, 1u);
}
__global__ void k_rcp32(unsigned *bad)
{
  const unsigned long long stride = (unsigned long long) gridDim.x * blockDim.x;
  for(unsigned long long u = blockIdx.x * (unsigned long long) blockDim.x + threadIdx.x; u < (1ULL << 32); u += stride) {
    const float x = __uint_as_float((unsigned) u), a = step_rcp32(x), b = __frcp_rn(x);
    if(__float_as_uint(a) != __float_as_uint(b) && (a == a || b == b)) atomicAdd(bad, 1u);
  }
}
extern "C" int compare_rcp32(void)
{
  unsigned *bad, h = 0;
  if(cudaMalloc(&bad, 4)) return -1;
  cudaMemset(bad, 0, 4);
  k_rcp32<<<148 * 8, 256>>>(bad);
  if(cudaMemcpy(&h, bad, 4, cudaMemcpyDeviceToHost)) return -1;
  cudaFree(bad);
  return (int) h;
}
extern "C" int compare(int n, const double *a, const double *b, int what)
{
  double *da, *db;
  unsigned *bad, h = 0;
  if(cudaMalloc(&da, n * 8) || cudaMalloc(&db, n * 8) || cudaMalloc(&bad, 4)) return -1;
  cudaMemcpy(da, a, n * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, n * 8, cudaMemcpyHostToDevice);
  cudaMemset(bad, 0, 4);
  k_cmp<<<(n + 255) / 256, 256>>>(n, da, db, what, bad);
  if(cudaMemcpy(&h, bad, 4, cudaMemcpyDeviceToHost)) return -1;
  cudaFree(da); cudaFree(db); cudaFree(bad);
  return (int) h;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("step")
    (d / "t.cu").write_text(SRC)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "--fmad=false", "-ftz=true", "-shared", "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "galic_b200", "csrc"),
                    str(d / "t.cu"), "-o", str(d / "libt.so")], check=True)
    return C.CDLL(str(d / "libt.so"))


def _significands(rng, n):
    """Random significands in [1, 2), a quarter of them next to 1 or 2."""
    m = 1.0 + rng.integers(0, 1 << 52, n) * 2.0 ** -52
    k = n // 8
    m[:k] = 1.0 + rng.integers(0, 16, k) * 2.0 ** -52
    m[k:2 * k] = 2.0 - (1 + rng.integers(0, 16, k)) * 2.0 ** -52
    return rng.permutation(m)


def _operands(what, rng, n):
    scale = np.ldexp(1.0, rng.integers(-100, 100, n))
    a, b = _significands(rng, n) * scale, _significands(rng, n) * np.ldexp(1.0, rng.integers(-100, 100, n))
    sign = rng.choice([-1.0, 1.0], n)
    if what == 0:  # half of the quotients within a few ulp of a rounding boundary
        q = _significands(rng, n)
        near = np.asarray([float(x) for x in (b.astype(np.longdouble) * (q.astype(np.longdouble) + 2.0 ** -53))])
        return np.where(rng.random(n) < 0.5, near * (1 + rng.integers(-2, 3, n) * 2.0 ** -52), a) * sign, b
    if what == 1:
        q = _significands(rng, n).astype(np.longdouble) + np.longdouble(2.0 ** -53)
        near = (q * q).astype(np.float64) * (1 + rng.integers(-2, 3, n) * 2.0 ** -52)
        return np.where(rng.random(n) < 0.5, near * np.ldexp(1.0, 2 * rng.integers(-50, 50, n)), a * a), b
    if what == 2:  # table edges (1 + j / 128 and their midpoints) among them
        edge = 1.0 + rng.integers(0, 512, n) / 256.0 * (1 + rng.integers(-2, 3, n) * 2.0 ** -52)
        return np.maximum(np.where(rng.random(n) < 0.3, edge, _significands(rng, n) * np.ldexp(1.0, rng.integers(0, 300, n))), 1.0), b
    if what == 3:  # all octants, ratios next to the table's k / 16 among them, tiny angles
        ratio = rng.integers(1, 17, n) / 16.0 * (1 + rng.integers(-2, 3, n) * 2.0 ** -52)
        x = b * rng.choice([-1.0, 1.0], n)
        y = np.where(rng.random(n) < 0.5, np.abs(x) * ratio, np.abs(x) * np.exp(rng.uniform(-40, 40, n)))
        y = np.clip(y, 2.0 ** -99, 2.0 ** 99) * sign
        swap = rng.random(n) < 0.5
        return np.where(swap, x, y), np.where(swap, y, x)
    return rng.choice([0.0, 1.0], n) * rng.integers(0, 2 ** 31 - 1, n) + rng.choice([0.0, 0.5, 2.0 ** -52], n), b


@pytest.mark.gpu
@pytest.mark.parametrize("what", [0, 1, 2, 3, 4], ids=["div", "sqrt", "log", "direction", "floor"])
def test_step_functions_equal_the_general_ones(lib, what):
    a, b = _operands(what, np.random.default_rng(what), 4_000_000)
    a, b = np.ascontiguousarray(a, dtype=np.float64), np.ascontiguousarray(b, dtype=np.float64)
    P = C.POINTER(C.c_double)
    assert lib.compare(len(a), a.ctypes.data_as(P), b.ctypes.data_as(P), what) == 0


@pytest.mark.gpu
def test_step_rcp32_equals_the_rounded_reciprocal_everywhere(lib):
    assert lib.compare_rcp32() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("shape", ["halo", "halo_disk"])
def test_orbits_outside_the_step_ranges_equal_the_oracle(shape):
    """Planar, axial, cold and nearly planar orbits, one beyond the force grid: every bin, the time and the orbit count."""
    m = synth.config_halo(n=32, level=5, seed=3) if shape == "halo" else synth.config_halo_disk(24, 8, level=5, seed=3)
    o = Oracle(m.params, use_libm=False)
    o.load_model(m)
    x, v = m.pos[0], m.vel[0]
    far = 3.0 * m.meta["rmax"] * x / np.linalg.norm(x)
    starts = [(x * [1, 1, 0], v * [1, 1, 0]), (x * [0, 1, 1], v * [0, 1, 1]), (x, v * 0), (x * [1, 1, 1e-40], v * [1, 1, 0]),
              (x * [1, 1e-35, 1], v * [1, 1e-200, 1]), (far, v)]
    with Context(m.params) as ctx:
        ctx.load_model(m)
        for t in {int(k) for k in m.ptype}:
            for p, w in starts:
                got = ctx.produce_orbit_response_field_mod(p, w, m.mass[0], m.tint[0], t)
                want = o.orbit_mod(np.ascontiguousarray(p), np.ascontiguousarray(w), m.mass[0], m.tint[0], t)
                assert got[0] == want[0] and got[1] == want[1]
                for a, b in zip(got[2:], want[2:7]):
                    assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.gpu
def test_infinite_projections_stay_infinite():
    """A start so close to the axis that R underflows to 0: the tangential projections are infinite, and so are the
    oracle's bins of the first half step; every bin, the time and the orbit count."""
    m = synth.config_halo_disk(24, 8, level=5, seed=3)
    o = Oracle(m.params, use_libm=False)
    o.load_model(m)
    start = np.array([1e-200, 2e-200, m.pos[0][2]])
    with Context(m.params) as ctx:
        ctx.load_model(m)
        for t in (1, 2):
            got = ctx.produce_orbit_response_field_mod(start, m.vel[0], m.mass[0], m.tint[0], t)
            want = o.orbit_mod(start, np.ascontiguousarray(m.vel[0]), m.mass[0], m.tint[0], t)
            assert any(np.isinf(b).any() for b in want[2:7])
            assert got[0] == want[0] and got[1] == want[1]
            for a, b in zip(got[2:], want[2:7]):
                assert np.array_equal(a, b, equal_nan=True)


BITS_SRC = r'''
#include "gmath.h"
#include "stepmath.cuh"
__device__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
__global__ void k_bits(int n, const double *a, const double *b, int what, unsigned *bad)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= n) return;
  const double x = a[i], y = b[i];
  bool ok = true;
  unsigned ones = 0;  // operands the functions refuse
  if(what == 0) {
    const double q = step_div(x, y, ones);
    ok = same(q, x == 0 && y > 0 ? 0.0 : x / y) || step_ones(ones);
  }
  if(what == 1) ok = same(step_sqrt(x), sqrt(x));
  if(what == 2) ok = same(step_log(x), gm_log(x));
  if(what == 3) {
    double s, c, s0, c0;
    step_direction(x, y, &s, &c, ones);
    gm_sincos(gm_atan2(x, y), &s0, &c0);
    ok = (same(s, s0) && same(c, c0)) || step_ones(ones);
  }
  if(!ok) atomicAdd(bad, 1u);
}
extern "C" int compare_bits(int n, const double *a, const double *b, int what)
{
  double *da, *db;
  unsigned *bad, h = 0;
  if(cudaMalloc(&da, n * 8) || cudaMalloc(&db, n * 8) || cudaMalloc(&bad, 4)) return -1;
  cudaMemcpy(da, a, n * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, n * 8, cudaMemcpyHostToDevice);
  cudaMemset(bad, 0, 4);
  k_bits<<<(n + 255) / 256, 256>>>(n, da, db, what, bad);
  if(cudaMemcpy(&h, bad, 4, cudaMemcpyDeviceToHost)) return -1;
  cudaFree(da); cudaFree(db); cudaFree(bad);
  return (int) h;
}
'''


def _whole_range(what, rng, n):
    """Operands over all of the header's stated ranges, their ends among them."""
    sign = rng.choice([-1.0, 1.0], n)
    pick = lambda lo, hi: np.where(rng.random(n) < 0.05, rng.choice([lo, hi], n), rng.integers(lo, hi + 1, n))
    if what == 0:
        eb = pick(-500, 500)
        b = np.where(eb == 500, 2.0 ** 500, np.ldexp(_significands(rng, n), eb))
        ea = pick(-960, 959)
        ea = np.clip(ea, eb - 958, eb + 958)  # the quotient's exponent is ea - eb or one less
        a = np.ldexp(_significands(rng, n), np.clip(ea, -960, 959))
        # squares of cancelled sums, as the projections have them, over sums of squares
        x, y, u, v = (np.ldexp(_significands(rng, n), rng.integers(-100, 100, n)) for _ in range(4))
        d = x * y - (x * y) * (1 + rng.integers(-3, 4, n) * 2.0 ** -52)
        kind = rng.random(n)
        a = np.where(kind < 0.2, d * d, np.where(kind < 0.25, 0.0, a))
        b = np.where(kind < 0.2, x * x + y * y, b)
        return a * sign, np.where(rng.random(n) < 0.5, b, -b)
    if what == 1:
        return np.where(rng.random(n) < 0.02, rng.choice([2.0 ** -900, 2.0 ** 900], n),
                        np.ldexp(_significands(rng, n), pick(-900, 899))), np.ones(n)
    if what == 2:
        return np.ldexp(_significands(rng, n), pick(0, 999)), np.ones(n)
    return np.ldexp(_significands(rng, n), pick(-100, 99)) * sign, np.ldexp(_significands(rng, n), pick(-100, 99)) * \
        rng.choice([-1.0, 1.0], n)


@pytest.mark.gpu
@pytest.mark.parametrize("what", [0, 1, 2, 3], ids=["div", "sqrt", "log", "direction"])
def test_step_functions_equal_the_general_ones_over_their_ranges(tmp_path_factory, what):
    d = tmp_path_factory.mktemp("bits")
    (d / "t.cu").write_text(BITS_SRC)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "--fmad=false", "-shared", "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "galic_b200", "csrc"),
                    str(d / "t.cu"), "-o", str(d / "libt.so")], check=True)
    a, b = _whole_range(what, np.random.default_rng(40 + what), 4_000_000)
    a, b = np.ascontiguousarray(a, dtype=np.float64), np.ascontiguousarray(b, dtype=np.float64)
    if what == 0:  # nothing outside the stated range
        nz = a != 0
        q = np.abs(a[nz] / b[nz])
        assert 2.0 ** -500 <= np.abs(b).min() and np.abs(b).max() <= 2.0 ** 500
        assert 2.0 ** -960 <= np.abs(a[nz]).min() and 2.0 ** -960 <= q.min() and q.max() <= 2.0 ** 960
    P = C.POINTER(C.c_double)
    assert C.CDLL(str(d / "libt.so")).compare_bits(len(a), a.ctypes.data_as(P), b.ctypes.data_as(P), what) == 0
