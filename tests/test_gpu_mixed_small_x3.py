"""Three bf16 terms per operand in mixed iterations of small systems (T X in the tensor-core ladder)
and just past the limit, at their own precision.

An operand of three terms leaves a remainder of 2^-26 of the element, so the FP32 accumulation is
what is left: by a replay of the sums on random operands of these sizes up to 3e-7 of the largest
element of D, and 2.3e-6 or more where the third terms of either operand are missing.  The bound of
2e-6 lies between.
"""
import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDSolver, System, solver as solver_mod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,kw", [
    ("pairing", dict(xi=1.0, g=0.37, n_pair_states=4, n_particles=4)),
    ("pairing", dict(xi=1.0, g=0.37, n_pair_states=12, n_particles=4)),   # 100 rows
    ("pairing", dict(xi=1.0, g=0.23, n_pair_states=12, n_particles=12)),  # 72 hole pairs: 3 chunks
    ("pairing", dict(xi=1.0, g=0.37, n_pair_states=14, n_particles=2)),   # 169 rows
    ("electron_gas", dict(r_s=1.0, n_shells=7, n_particle_shells=3)),
    ("inf_matter", dict(density=0.08, tz_max=1, n_shells=4, n_particle_shells=2)),
])
def test_step_matches_fp64(kind, kw):
    with getattr(System, kind)(**kw) as s, CCDSolver(s) as a:
        with CCDSolver(s, precision="mixed_bf16x3") as b:
            for _ in range(3):
                a.step(0.5)
            b.set_t2(a.t2())
            for _ in range(2):  # the second reads the images that the first iteration wrote
                a.step(0.5)
                b.step(0.5)
                da, db = (x.chain(solver_mod.CHAIN_DIFF_PPHH) for x in (a, b))
                assert np.max(np.abs(da - db)) <= 2e-6 * np.max(np.abs(da))
