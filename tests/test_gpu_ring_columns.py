"""The wide ring units on both sides of the rule that gives them all of T' or their columns alone
(more than 296 units): 16-row paddings 48 and 64 of the modified channels (80 is in the full-size
solves).

Tolerances are those of the parity tests: energies to 1e-12 relative of the oracle's, amplitudes
to 1e-13.
"""
import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDSolver, System
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,kw", [
    ("electron_gas", dict(r_s=1.0, n_shells=20, n_particle_shells=4)),
    ("electron_gas", dict(r_s=1.0, n_shells=21, n_particle_shells=4)),  # 322 units
    ("inf_matter", dict(density=0.08, tz_max=1, n_shells=20, n_particle_shells=5)),  # 382
])
def test_steps_match_oracle(kind, kw):
    with getattr(System, kind)(**kw) as s, CCDSolver(s) as sol:
        o = Oracle(s)
        for _ in range(3):
            e_ref, e = o.step(0.5), sol.step(0.5)
            assert abs(e - e_ref) <= 1e-12 * abs(e_ref)
        np.testing.assert_allclose(sol.t2(), o.t2(), rtol=0, atol=1e-13)
        o.close()
