"""Windows of optimisation repetitions (galic_optimize_reps): the loop body of
main.c:94-100 run `reps` times, with the old and trial orbits of a window of
repetitions integrated in one launch and the repetitions then evaluated,
accepted and committed in order.

* The result equals `reps` calls of galic_optimize_rep bit for bit, in both
  forms, whether the work runs as one window or many (window_bytes), and
  when the particle sequence wraps so that a particle is optimised twice
  (the window ends before the repeat).
* Against the restatement (oracle/galic_oracle.c) repeating its single
  repetition, main.c:120-146's cycling through a permutation: the same
  velocities, counters, orbit counts and merit values.
"""
import numpy as np
import pytest

from galic_b200 import GALIC_FORM_FP32, GALIC_FORM_FP64, Context, GalicError, synth
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu

FIT_TOL = 1e-10
FIT_ATOL = 1e-14


def cycling_lists(n, count, reps, seed):
    """optimize_some_particles (main.c:120-146): count particles per repetition
    taken in permutation order, wrapping around at the end."""
    perm = np.random.default_rng(seed).permutation(n)
    pos = (np.arange(reps * count) % n)
    return perm[pos].reshape(reps, count).astype(np.int32)


def state(ctx, present):
    vel, orbits, vdisp = ctx.particles()
    resp = np.stack([ctx.response(t, w) for t in present for w in range(10)])
    return vel, orbits, vdisp, resp, ctx.fit(), ctx.counters()


@pytest.mark.parametrize("form", [GALIC_FORM_FP64, GALIC_FORM_FP32], ids=["fp64", "fp32"])
def test_windows_equal_sequential_repetitions(form):
    m = synth.config_halo_disk(n_halo=1500, n_disk=500, level=6, seed=51)
    present = (1, 2)
    lists = cycling_lists(m.n, 90, 30, 3)  # 2700 slots over 2000 particles: wraps once
    results = []
    for mode in ("sequential", "one_call", "small_windows"):
        with Context(m.params) as ctx:
            ctx.load_model(m)
            ctx.calc_all_response_fields(form)
            if mode == "sequential":
                for r in range(len(lists)):
                    ctx.optimize_rep(lists[r], 99, 1000 + r, form)
            elif mode == "one_call":
                ctx.optimize_reps(lists, 99, 1000, form)
            else:
                # about three repetitions per window
                ctx.optimize_reps(lists, 99, 1000, form, window_bytes=3 * 90 * 2 * 5 * 4096 * 8 + 1)
            results.append(state(ctx, present))
    a = results[0]
    assert a[5][1].sum() > 0  # some proposals accepted
    for b in results[1:]:
        for x, y in zip(a[:5], b[:5]):
            assert np.array_equal(x, y)
        assert np.array_equal(a[5][0], b[5][0]) and np.array_equal(a[5][1], b[5][1])


def test_windows_match_oracle_repetitions():
    m = synth.config_composite(n_halo=600, n_disk=300, n_bulge=200, level=5, seed=52)
    present = (1, 2, 3)
    lists = cycling_lists(m.n, 40, 40, 4)  # wraps once
    o = Oracle(m.params, use_libm=False)
    o.load_model(m)
    assert o.calc_all() == 0
    for r in range(len(lists)):
        assert o.optimize_rep(lists[r], 7, 50 + r) == 0
    with Context(m.params) as ctx:
        ctx.load_model(m)
        ctx.calc_all_response_fields()
        ctx.optimize_reps(lists, 7, 50)
        vel, orbits, vdisp = ctx.particles()
        ov, oo, od = o.particles()
        assert np.array_equal(vel, ov)
        assert np.array_equal(orbits, oo)
        assert np.array_equal(vdisp, od)
        tr, ch = ctx.counters()
        otr, och = o.counters()
        assert np.array_equal(tr, otr) and np.array_equal(ch, och)
        f, g = ctx.fit()[list(present), :5], o.fit()[list(present), :5]
        assert np.all(np.abs(f - g) <= FIT_TOL * np.abs(g) + FIT_ATOL)


def test_invalid_windows_rejected():
    m = synth.config_halo(n=64, level=5, seed=53)
    with Context(m.params) as ctx:
        ctx.load_model(m)
        with pytest.raises(GalicError) as e:
            ctx.optimize_reps(np.array([[1, 2]]), 1, 0)  # before any response
        assert e.value.status == 9
        ctx.calc_all_response_fields()
        for bad in ([[1, 1]], [[0, 1], [-1, 2]], [[0, 64]]):
            with pytest.raises(GalicError) as e:
                ctx.optimize_reps(np.array(bad), 1, 0)
            assert e.value.status == 1
        ctx.optimize_reps(np.zeros((3, 0), dtype=np.int32), 1, 0)


def test_windows_report_the_fit_after_every_repetition():
    """fits=True returns the galic_get_fit values after each repetition: the
    same as reading the fit after each galic_optimize_rep call."""
    m = synth.config_halo_disk(n_halo=800, n_disk=300, level=5, seed=54)
    lists = cycling_lists(m.n, 60, 25, 5)
    want = []
    with Context(m.params) as ctx:
        ctx.load_model(m)
        ctx.calc_all_response_fields()
        for r in range(len(lists)):
            ctx.optimize_rep(lists[r], 3, 10 + r)
            want.append(ctx.fit())
    with Context(m.params) as ctx:
        ctx.load_model(m)
        ctx.calc_all_response_fields()
        got = ctx.optimize_reps(lists, 3, 10, window_bytes=4 * 60 * 2 * 5 * 1024 * 8 + 1, fits=True)
    assert got.shape == (len(lists), 4, 7)
    assert np.array_equal(got, np.stack(want), equal_nan=True)


def misfit(d1, d2, r1, r2, level, thresh, low):
    """calc_stack_difference with flag 1 (grid.c:1086-1151) of finest grids, bottom up."""
    def children(a):
        return a[0::2, 0::2], a[0::2, 1::2], a[1::2, 0::2], a[1::2, 1::2]

    def leaf(d1, d2, r1, r2):
        with np.errstate(all="ignore"):
            q2 = d2 / r2
            v = np.abs(d1 / r1 - q2) / np.where(q2 > low, q2, low)
        return np.where((r1 > 0) & (r2 > 0), v, 0.0)

    off = lambda l: (4 ** l - 1) // 3
    at = lambda stack, l: stack[off(l):off(l + 1)].reshape(2 ** l, 2 ** l)
    v = leaf(d1, at(d2, level), r1, at(r2, level))
    for l in range(level - 1, -1, -1):
        c = [children(x) for x in (d1, r1)]
        d1, r1 = [((x[0] + x[2]) + x[1]) + x[3] for x in c]
        x = children(v)
        v = np.where(r1 < thresh, leaf(d1, at(d2, l), r1, at(r2, l)), ((x[0] + x[1]) + x[2]) + x[3])
    return float(v[0, 0])


@pytest.mark.parametrize("level", [1, 2, 3, 4, 5, 7])
def test_fit_at_every_depth_of_the_pyramid(level):
    """The merit takes the lowest three levels by shuffles and the rest through
    shared memory: the instantaneous terms of the committed grids restated here, at
    depths where one or the other is missing, and repetitions as single calls and
    as windows."""
    from galic_b200 import sampling
    m = synth.config_composite(n_halo=300, n_disk=150, n_bulge=100, level=level, seed=57)
    p = m.params
    N = 2 ** level
    with Context(p) as ctx:
        states = []
        lists = np.arange(540, dtype=np.int32).reshape(6, 90)
        for windows in (False, True):
            ctx.load_model(m)
            ctx.calc_all_response_fields(GALIC_FORM_FP64)
            if windows:
                hist = ctx.optimize_reps(lists, 11, 70, GALIC_FORM_FP64, fits=True)
            else:
                each = []
                for r in range(len(lists)):
                    ctx.optimize_rep(lists[r], 11, 70 + r)
                    each.append(ctx.fit())
            states.append(state(ctx, (1, 2, 3))[:5])
        for x, y in zip(*states):
            assert np.array_equal(x, y)
        assert np.array_equal(hist, np.array(each))
        fit = ctx.fit()
        for t in (1, 2, 3):
            grid = {w: ctx.response(t, w).reshape(N, N) for w in range(10)}
            tg = sampling.get_targets(ctx, t)
            thr = p.MinParticlesPerBinForDispersionMeasurement * p.MType[t] / p.NType[t]
            count = 3 if p.TypeOfVelocityStructure[t] in (0, 1) else 4
            for k in range(count):  # r, t, p, q
                v = misfit(grid[6 + k], tg[2 + k], grid[5], tg[1], level, thr, p.LowerDispLimit)
                assert abs(fit[t][1 + k] - v * fit[t][5]) <= 1e-12 * abs(v * fit[t][5]), (t, k)


def short_orbits(n_halo, n_disk, level, seed):
    """A halo + disk whose orbits take a few dozen steps."""
    m = synth.config_halo_disk(n_halo=n_halo, n_disk=n_disk, level=level, seed=seed)
    m.tint = m.tint * 0.05
    return m


@pytest.mark.parametrize("form", [GALIC_FORM_FP64, GALIC_FORM_FP32], ids=["fp64", "fp32"])
def test_large_windows_equal_sequential_repetitions(form):
    """Three windows of 4500 particles each, more than run two at a time, the second with particles of the first."""
    m = short_orbits(6000, 1000, 4, 58)
    lists = cycling_lists(m.n, 1500, 9, 6)  # slots 7000 on repeat those from slot 0
    results = []
    for windows in (False, True):
        with Context(m.params) as ctx:
            ctx.load_model(m)
            ctx.calc_all_response_fields(form)
            if windows:
                ctx.optimize_reps(lists, 5, 30, form, window_bytes=3 * 1500 * 2 * (5 * 256 * 8 + 128))
            else:
                for r in range(len(lists)):
                    ctx.optimize_rep(lists[r], 5, 30 + r, form)
            results.append(state(ctx, (1, 2)))
    for x, y in zip(*results):
        assert np.array_equal(np.asarray(x), np.asarray(y), equal_nan=True)
    assert results[0][5][1].sum() > 0


@pytest.mark.parametrize("count", [2467, 14501])
def test_many_particles_in_one_repetition(count):
    """More particles than the acceptance's CTA has threads, more acceptances of a type than the commit stages at
    once and (14501) more orbits than the spread launch has lanes: the committed grids restated, addition by
    addition in particle order, from the accepted particles' single orbits, and the repetition as a window."""
    m = short_orbits(13001, 3000, 3, 59)
    idx = np.random.default_rng(7).permutation(m.n)[:count].astype(np.int32)
    with Context(m.params) as ctx:
        ctx.load_model(m)
        ctx.calc_all_response_fields(GALIC_FORM_FP64)
        before = {t: [ctx.response(t, w) for w in range(10)] for t in (1, 2)}
        vel0, orbits0, vdisp0 = ctx.particles()
        ctx.optimize_rep(idx, 8, 3)
        vel1, orbits1, vdisp1, _, _, (tries, changes) = first = state(ctx, (1, 2))
        after = {t: [ctx.response(t, w) for w in range(10)] for t in (1, 2)}
        took = np.any(vel0 != vel1, axis=1)
        assert not took[np.setdiff1d(np.arange(m.n), idx)].any()
        for t in (1, 2):
            assert tries[t] == np.sum(m.ptype[idx] == t) and changes[t] == np.sum(took & (m.ptype == t))
        assert changes[1] > 256 and (count < 10000 or changes[2] > 256)
        for t in (1, 2):
            delta = np.zeros((5, 64))
            for k in idx[(m.ptype[idx] == t) & took[idx]]:
                old = ctx.produce_orbit_response_field_mod(m.pos[k], vel0[k], m.mass[k], m.tint[k], t)
                new = ctx.produce_orbit_response_field_mod(m.pos[k], vel1[k], m.mass[k], m.tint[k], t)
                delta += np.stack(new[2:]) - np.stack(old[2:])
                assert orbits1[k] == new[1]
            for w in range(5):
                assert np.array_equal(after[t][w], before[t][w] + delta[w]), (t, w)
            assert np.array_equal(after[t][5], before[t][5])
            # the energy grid: every change of the projections lands on the four nodes of a cell with weights that
            # sum to one, so the grids' sums change by the particles' changes
            sel = took & (m.ptype == t)
            dv = (vdisp1[sel] - vdisp0[sel]) * m.mass[sel][:, None]
            for a in range(4):  # r, t, p, q
                got = np.sum(after[t][6 + a]) - np.sum(before[t][6 + a])
                scale = np.sum(np.abs(dv[:, a])) + np.sum(np.abs(before[t][6 + a]))
                # sums of at most 14501 terms of either sign, each rounded once
                assert abs(got - np.sum(dv[:, a])) <= 14501 * 2.0 ** -53 * 4 * scale, (t, a)
    with Context(m.params) as ctx:
        ctx.load_model(m)
        ctx.calc_all_response_fields(GALIC_FORM_FP64)
        ctx.optimize_reps(idx[None], 8, 3)
        for x, y in zip(first, state(ctx, (1, 2))):
            assert np.array_equal(np.asarray(x), np.asarray(y), equal_nan=True)
