"""V blocks from the host that lack a symmetry which the iteration does not rely on, against the
oracle: V_hpph of a modified channel and of its transpose with nothing in common, and a V_hhhh whose
rows are not antisymmetric.  (The amplitudes stay antisymmetric: the four ring terms are
antisymmetrised, and T X sums over both orders of the rows' pair.)

Tolerances are those of the parity tests: energies to 1e-12 relative, amplitudes to 1e-13.
"""
import ctypes

import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDSolver, System
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

SYSTEMS = [
    ("pairing", dict(xi=1.0, g=0.4, n_pair_states=9, n_particles=8)),
    ("inf_matter", dict(density=0.16, tz_max=2, n_shells=4, n_particle_shells=1)),
    ("electron_gas", dict(r_s=1.0, n_shells=8, n_particle_shells=2)),
    ("electron_gas", dict(r_s=1.3, n_shells=7, n_particle_shells=4)),
]


def block(pointers, ch, shape):
    return np.ctypeslib.as_array(ctypes.cast(pointers[ch], ctypes.POINTER(ctypes.c_double)), shape)


def perturb(s, what, rng):
    dims, mod = s.chan_dims(), s.array("chan_mod_dims").reshape(-1, 4)
    p = s.problem.contents
    if what in ("v_hpph", "both"):
        for ch, (_, _, hp, ph) in enumerate(mod):
            if ph and hp:
                v = block(p.v_hpph_mod, ch, (hp, ph))
                v += 0.2 * np.max(np.abs(v)) * rng.uniform(-1, 1, v.shape)
    if what in ("v_hhhh", "both"):
        pairs, off = s.array("hh_map").reshape(-1, 2), 0
        for ch, (pp, hh) in enumerate(dims[:, :2]):
            q = pairs[off:off + hh].astype(np.int64)
            off += hh
            if not (pp and hh):
                continue
            lo, hi = q.min(1), q.max(1)
            sign = np.sign(q[:, 1] - q[:, 0])
            _, k = np.unique(lo << 32 | hi, return_inverse=True)
            m = rng.uniform(-1, 1, (k.max() + 1, k.max() + 1))
            v = block(p.v_hhhh, ch, (hh, hh))
            # Symmetric under k <-> l of the row, antisymmetric under i <-> j of the column.
            v += 0.3 * np.max(np.abs(v)) * m[k[:, None], k[None, :]] * sign[None, :]


@pytest.mark.parametrize("what", ["v_hpph", "v_hhhh", "both"])
@pytest.mark.parametrize("path", ["fused", "tables"])
@pytest.mark.parametrize("kind,kw", SYSTEMS)
def test_steps_match_oracle(kind, kw, path, what):
    with getattr(System, kind)(**kw) as s:
        perturb(s, what, np.random.default_rng(11))
        with CCDSolver(s, path=path) as sol:
            o = Oracle(s)
            for _ in range(3):
                e_ref, e = o.step(0.5), sol.step(0.5)
                assert abs(e - e_ref) <= 1e-12 * abs(e_ref)
                np.testing.assert_allclose(sol.t2(), o.t2(), rtol=0, atol=1e-13)
            o.close()
