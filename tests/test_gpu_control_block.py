"""The host's copy of the control block is only read back after calls that change it: whatever a
handle did before, a call gives what a fresh handle gives, bit for bit."""
import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDGPUError, CCDSolver, System

pytestmark = pytest.mark.gpu

KW = dict(r_s=1.0, n_shells=7, n_particle_shells=3)


def stages(sol, mixing):
    sol.calc_t2diff_p2_p1hh()
    sol.calc_t2diff_h2pp_h1()
    sol.calc_t2diff_phhp()
    sol.calc_t2diff_pphh()
    sol.map_from_distributed()
    e = sol.calc_t2_pphh(mixing)
    sol.map_to_distributed()
    return e


BEFORE = {
    "nothing": lambda sol: None,
    "solve": lambda sol: sol.solve(tol=1e-3, max_iters=7, mixing=0.3),
    "steps": lambda sol: [sol.step(0.7) for _ in range(2)],
    "mbpt2": lambda sol: (sol.step(0.5), sol.mbpt2(init_t2=True)),
    "trace": lambda sol: (sol.trace_arm(1), sol.solve(tol=1e-6), sol.trace_read(), sol.trace_arm(-1)),
    "failed": lambda sol: fail(sol),
}


def fail(sol):
    t2 = np.zeros(sol.n_t2)
    t2[3] = np.nan
    sol.set_t2(t2)
    with pytest.raises(CCDGPUError):
        sol.step(0.5)


def record(sol, path):
    sol.reset()
    out = []
    if path == "tables":
        out += [stages(sol, 0.5), stages(sol, 0.5)]
    out += [sol.step(0.5), sol.mbpt2(), sol.step(0.6)]
    r = sol.solve(tol=1e-7, max_iters=5, mixing=0.5)
    out += [r.e_corr, r.iterations, sol.energy_history()]
    sol.reset()
    out += [sol.t2(), sol.step(0.5), sol.t2()]
    return out


@pytest.mark.parametrize("before", list(BEFORE))
@pytest.mark.parametrize("path,precision", [("fused", "fp64"), ("fused", "mixed_bf16"),
                                            ("tables", "fp64")])
def test_as_a_fresh_handle(before, path, precision):
    with System.electron_gas(**KW) as s:
        with CCDSolver(s, path=path, precision=precision) as sol:
            want = record(sol, path)
        with CCDSolver(s, path=path, precision=precision) as sol:
            BEFORE[before](sol)
            got = record(sol, path)
        for a, b in zip(want, got):
            np.testing.assert_array_equal(a, b)
