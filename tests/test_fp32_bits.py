"""The FP32 form's bits: its file is compiled with contraction on, so a sum of products whose roundings are not
spelled out may change with the code around it, unseen by the tolerance tests.  Digests of the response grids of a
pass and of the state after two repetitions (particles drawn uniformly on the fixtures' tables), B200."""
import hashlib
import os

import numpy as np
import pytest

import golden_lib
from galic_b200 import GALIC_FORM_FP32, Context

pytestmark = pytest.mark.gpu

# (grids of the pass, grids and velocities after the repetitions)
DIGESTS = {
    "composite": ("286fa344b892d8d3", "0b51e97f89d1ebf8"),
    "halo_disk": ("969d13bb5ab13640", "ee517551fdbe5608"),
    "halo_analytic": ("82ca5361cb4c6c55", "9cbb50d3912ba48a"),
}


def digest(arrays):
    return hashlib.sha256(b"".join(np.ascontiguousarray(a).tobytes() for a in arrays)).hexdigest()[:16]


@pytest.mark.parametrize("shape", sorted(DIGESTS))
def test_fp32_pass_and_repetitions_keep_their_bits(shape):
    ins, _ = golden_lib.load(os.path.join(golden_lib.HERE, "golden", shape + ".npz"))
    m = golden_lib.model(ins)
    types = [t for t in (1, 2, 3) if m.params.NType[t] > 0]
    n = 1500
    rng = np.random.default_rng(20)
    # short orbits that move nearly as the streaming velocity does: the first deposits weigh most, and the
    # difference to the streaming velocity shows its rounding
    pos = rng.uniform(-12.0, 12.0, (n, 3)) * [1.0, 1.0, 0.1]
    ptype = np.asarray(types, dtype=np.int32)[rng.integers(0, len(types), n)]
    p = m.params
    lines = p.FG_Rmin * (p.FG_Fac ** np.arange(p.FG_Nbin) - 1.0)
    R = np.sqrt(pos[:, 0] ** 2 + pos[:, 1] ** 2)
    at = np.searchsorted(lines, np.abs(pos[:, 2])) * p.FG_Nbin + np.searchsorted(lines, R)
    vphi = np.array([np.asarray(m.vstream[t]).reshape(-1)[k] for t, k in zip(ptype, at)])
    vel = np.stack([-pos[:, 1], pos[:, 0], 0 * R], axis=1) * (vphi / R)[:, None] + rng.uniform(-5.0, 5.0, (n, 3))
    mass, tint, vesc = np.full(n, 1.0 / 64), rng.uniform(0.001, 0.02, n), np.full(n, 1000.0)
    targets = rng.uniform(5000.0, 20000.0, (n, 4))
    with Context(m.params) as ctx:
        ctx.load_model(m)
        ctx.set_particles(pos, vel, mass, tint, vesc, ptype, targets)
        ctx.calc_all_response_fields(GALIC_FORM_FP32)
        passed = digest([ctx.response(t, w) for t in types for w in range(10)])
        ctx.optimize_reps(rng.permutation(n)[:600].reshape(2, 300).astype(np.int32), 9, 0, GALIC_FORM_FP32)
        after = digest([ctx.response(t, w) for t in types for w in range(10)] + [ctx.particles()[0]])
    assert (passed, after) == DIGESTS[shape]
