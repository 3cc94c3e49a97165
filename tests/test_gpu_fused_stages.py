"""Stage entry points on a handle of the fused path (its problem carries the three-body V blocks):
whatever the handle did before, they work from its current amplitudes, and the fused iterations,
reads and mixed-precision images that follow work from theirs.

Energies agree with the oracle's to 1e-12 relative, amplitudes to 1e-13 (the parity tests' bounds);
a handle that was used before agrees with a fresh one bit for bit.
"""
import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDSolver, System, solver as solver_mod
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

KW = dict(r_s=1.0, n_shells=7, n_particle_shells=3)
PRECISIONS = ["fp64", "mixed_bf16", "mixed_bf16x3"]
CHAINS = [solver_mod.CHAIN_T2, solver_mod.CHAIN_T2_OLD, solver_mod.CHAIN_OLD_PHHP,
          solver_mod.CHAIN_DIFF_PPHH]


def stages(sol, mixing=0.5):
    sol.calc_t2diff_p2_p1hh()
    sol.calc_t2diff_h2pp_h1()
    sol.calc_t2diff_phhp()
    sol.calc_t2diff_pphh()
    sol.map_from_distributed()
    e = sol.calc_t2_pphh(mixing)
    sol.map_to_distributed()
    return e


def record(sol):
    out = [stages(sol), stages(sol, 0.6)]
    out += [sol.t2()] + [sol.chain(c) for c in CHAINS]
    out += [sol.step(0.5), sol.t2(), stages(sol), sol.step(0.5), sol.t2()]
    return out


BEFORE = {
    "solve": lambda sol: (sol.solve(tol=1e-6), sol.t2()),
    "steps": lambda sol: ([sol.step(0.5) for _ in range(3)], sol.chain(solver_mod.CHAIN_T2)),
    "stages": lambda sol: [stages(sol) for _ in range(2)],
    "set_t2": lambda sol: (sol.mbpt2(init_t2=True), sol.set_t2(2.0 * sol.t2())),
}


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("before", list(BEFORE))
def test_after_reset_as_a_fresh_handle(before, precision):
    with System.electron_gas(**KW) as s:
        with CCDSolver(s, precision=precision) as sol:
            want = record(sol)
        with CCDSolver(s, precision=precision) as sol:
            BEFORE[before](sol)
            sol.reset()
            got = record(sol)
        for a, b in zip(want, got):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("before", list(BEFORE))
def test_go_on_from_the_current_amplitudes(before, precision):
    """As a handle that was given the same amplitudes."""
    with System.electron_gas(**KW) as s:
        with CCDSolver(s, precision=precision) as a, CCDSolver(s, precision=precision) as b:
            BEFORE[before](a)
            b.set_t2(a.t2())
            for x, y in zip(record(a), record(b)):
                np.testing.assert_array_equal(x, y)


def test_scatter_without_an_assembly_keeps_the_amplitudes():
    with System.electron_gas(**KW) as s, CCDSolver(s) as sol:
        for _ in range(3):
            sol.step(0.5)
        t2 = sol.t2()
        sol.map_to_distributed()
        np.testing.assert_array_equal(sol.t2(), t2)
        sol.reset()
        sol.map_to_distributed()
        assert not np.any(sol.t2())


@pytest.mark.parametrize("precision", PRECISIONS)
def test_iterations_match_oracle(precision):
    """Stage iterations are FP64 at every precision; a mixed step between them is within its own
    bound (3e-5 of two bf16 terms, on amplitudes of an iteration that mixes in half of them)."""
    with System.electron_gas(**KW) as s, CCDSolver(s, precision=precision) as sol:
        o = Oracle(s)
        sol.step(0.5)
        sol.reset()
        for _ in range(3):
            e_ref, e = o.step(0.5), stages(sol)
            assert abs(e - e_ref) <= 1e-12 * abs(e_ref)
            np.testing.assert_allclose(sol.t2(), o.t2(), rtol=0, atol=1e-13)
        e_ref, e = o.step(0.5), sol.step(0.5)
        bound = 1e-12 if precision == "fp64" else 3e-5
        assert abs(e - e_ref) <= bound * abs(e_ref)
        t2 = o.t2()
        atol = 1e-13 if precision == "fp64" else 3e-5 * np.max(np.abs(t2))
        np.testing.assert_allclose(sol.t2(), t2, rtol=0, atol=atol)
        o.close()
