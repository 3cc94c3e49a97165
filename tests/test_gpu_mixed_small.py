"""Mixed iterations of systems whose channels are all one row tile of the tensor-core ladder (at most
128 strict particle pairs), where it does T X too: one to three 32-deep chunks of hole pairs, and
a system just past the limit.

Each operand is two bf16 terms (remainder 2^-18 of the element) and one product of second terms is
left out: an element of D is off by at most 3 * 2^-18 = 1.2e-5 of the sum of its products' sizes;
3e-5 of the largest element leaves a factor for that sum.
"""
import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDSolver, System, solver as solver_mod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,kw", [
    ("pairing", dict(xi=1.0, g=0.5, n_pair_states=4, n_particles=4)),
    ("pairing", dict(xi=1.0, g=0.4, n_pair_states=12, n_particles=4)),   # 100 rows
    ("pairing", dict(xi=1.0, g=0.3, n_pair_states=12, n_particles=12)),  # 72 hole pairs: 3 chunks
    ("pairing", dict(xi=1.0, g=0.4, n_pair_states=14, n_particles=2)),   # 169 rows
    ("electron_gas", dict(r_s=1.0, n_shells=7, n_particle_shells=3)),
])
@pytest.mark.parametrize("precision", ["mixed_bf16", "mixed_bf16x3"])
def test_step_matches_fp64(kind, kw, precision):
    with getattr(System, kind)(**kw) as s, CCDSolver(s) as a, CCDSolver(s, precision=precision) as b:
        for _ in range(3):
            a.step(0.5)
        b.set_t2(a.t2())
        for _ in range(2):  # the second reads the images that the first iteration wrote
            a.step(0.5)
            b.step(0.5)
            da, db = (x.chain(solver_mod.CHAIN_DIFF_PPHH) for x in (a, b))
            assert np.max(np.abs(da - db)) <= 3e-5 * np.max(np.abs(da))


def test_mixed_energy_is_the_fp64_one():
    with System.pairing(xi=1.0, g=-0.38, n_pair_states=9, n_particles=4) as s:
        with CCDSolver(s) as a, CCDSolver(s, precision="mixed_bf16") as b:
            ea, eb = a.solve(tol=1e-10).e_corr, b.solve(tol=1e-10).e_corr
            assert abs(ea - eb) <= 1e-9 * abs(ea)
