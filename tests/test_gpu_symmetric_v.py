"""The FP64 pp ladder over the symmetric half of V: row tiles with blocks beside the diagonal, K
segments that start on, inside and past the diagonal block, hole counts on both sides of the
limit, and a stored V that is symmetric in some channels only.

Tolerances are those of the parity tests: energies to 1e-12 relative of the oracle's, amplitudes
to 1e-13, t2Diff_pphh to 1e-12 of its largest element.
"""
import ctypes

import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDSolver, System, solver as solver_mod
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

SYSTEMS = [  # largest strict pp counts 196, 184, 382 and 362
    dict(r_s=1.0, n_shells=13, n_particle_shells=2),
    dict(r_s=1.0, n_shells=13, n_particle_shells=3),
    dict(r_s=0.8, n_shells=19, n_particle_shells=2),
    dict(r_s=1.2, n_shells=19, n_particle_shells=4),
]


def skew(s, every):
    """Adds a part to every `every`-th channel's V_pppp that is antisymmetric in both pairs but not
    symmetric under their exchange."""
    dims, pairs = s.chan_dims(), s.array("pp_map").reshape(-1, 2)
    rng, off = np.random.default_rng(7), 0
    for ch, (pp, hh) in enumerate(dims[:, :2]):
        p = pairs[off:off + pp].astype(np.int64)
        off += pp
        if not hh or ch % every:
            continue
        lo, hi = p.min(1), p.max(1)
        sign = np.sign(p[:, 1] - p[:, 0]).astype(float)
        _, k = np.unique(lo << 32 | hi, return_inverse=True)
        m = rng.uniform(-1e-3, 1e-3, (k.max() + 1, k.max() + 1))
        v = np.ctypeslib.as_array(
            ctypes.cast(s.problem.contents.v_pppp[ch], ctypes.POINTER(ctypes.c_double)), (pp, pp))
        v += sign[:, None] * sign[None, :] * m[k[:, None], k[None, :]]


@pytest.mark.parametrize("every", [0, 1, 3])
@pytest.mark.parametrize("kw", SYSTEMS)
def test_steps_match_oracle(kw, every):
    with System.electron_gas(**kw) as s:
        if every:
            skew(s, every)
        with CCDSolver(s) as sol:
            o = Oracle(s)
            for mul in (1, 4, 64):
                sol.set_schedule(thin_split_mul=mul, wide_split_mul=mul)
                e_ref, e = o.step(0.5), sol.step(0.5)
                assert abs(e - e_ref) <= 1e-12 * abs(e_ref)
                d_ref, d = (x.chain(solver_mod.CHAIN_DIFF_PPHH) for x in (o, sol))
                assert np.max(np.abs(d - d_ref)) <= 1e-12 * np.max(np.abs(d_ref))
            np.testing.assert_allclose(sol.t2(), o.t2(), rtol=0, atol=1e-13)
            o.close()
