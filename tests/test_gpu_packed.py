"""The fused path's packed amplitudes (one element of t_ab,ij = -t_ab,ji = -t_ba,ij = t_ba,ji) at
the edges of their tiles: channels without quads (one hole pair, i = j), one to many strict hole
pairs, fewer rows than a tile, and both isospins.

Tolerances are those of the parity tests: energies to 1e-12 relative of the oracle's, amplitudes
to 1e-13, t2Diff_pphh to 1e-12 of its largest element.
"""
import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDGPUError, CCDSolver, System, solver as solver_mod
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

SYSTEMS = [
    ("pairing", dict(xi=1.0, g=-0.7, n_pair_states=3, n_particles=2)),
    ("pairing", dict(xi=1.0, g=0.4, n_pair_states=9, n_particles=8)),
    ("inf_matter", dict(density=0.08, tz_max=1, n_shells=3, n_particle_shells=1)),
    ("inf_matter", dict(density=0.16, tz_max=2, n_shells=4, n_particle_shells=1)),
    ("electron_gas", dict(r_s=1.0, n_shells=8, n_particle_shells=2)),
    ("electron_gas", dict(r_s=0.7, n_shells=6, n_particle_shells=3)),
    ("electron_gas", dict(r_s=1.3, n_shells=7, n_particle_shells=4)),
]


@pytest.mark.parametrize("path", ["fused", "tables"])
@pytest.mark.parametrize("kind,kw", SYSTEMS)
def test_steps_match_oracle_at_tile_edges(kind, kw, path):
    with getattr(System, kind)(**kw) as s, CCDSolver(s, path=path) as sol:
        o = Oracle(s)
        for _ in range(3):
            e_ref, e = o.step(0.5), sol.step(0.5)
            assert abs(e - e_ref) <= 1e-12 * abs(e_ref)
            d_ref, d = (x.chain(solver_mod.CHAIN_DIFF_PPHH) for x in (o, sol))
            assert np.max(np.abs(d - d_ref)) <= 1e-12 * max(np.max(np.abs(d_ref)), 1e-300)
        t2 = o.t2()
        np.testing.assert_allclose(sol.t2(), t2, rtol=0, atol=1e-13)
        # A restart from those amplitudes goes on as the oracle does.
        with CCDSolver(s, path=path) as again:
            again.set_t2(t2)
            np.testing.assert_array_equal(again.t2(), t2)
            e_ref, e = o.step(0.5), again.step(0.5)
            assert abs(e - e_ref) <= 1e-12 * abs(e_ref)
            np.testing.assert_allclose(again.t2(), o.t2(), rtol=0, atol=1e-13)
        o.close()


def test_diff_is_readable_after_reset():
    kind, kw = SYSTEMS[4]
    with getattr(System, kind)(**kw) as s, CCDSolver(s) as a, CCDSolver(s) as b:
        for _ in range(2):
            a.step(0.5)
            b.step(0.5)
        b.reset()
        assert not np.any(b.t2())
        np.testing.assert_array_equal(a.chain(solver_mod.CHAIN_DIFF_PPHH),
                                      b.chain(solver_mod.CHAIN_DIFF_PPHH))


@pytest.mark.parametrize("precision", ["fp64", "mixed_bf16"])
def test_non_finite_amplitude_anywhere_is_reported(precision):
    """Also where the packed layout keeps no element: a > b, i > j, a = b, i = j."""
    kind, kw = SYSTEMS[5]
    with getattr(System, kind)(**kw) as s, CCDSolver(s, precision=precision) as sol:
        n = sol.n_t2
        for at in (0, 1, n // 3, n // 2, n - 1):
            t2 = np.zeros(n)
            t2[at] = np.inf if at % 2 else np.nan
            sol.set_t2(t2)
            with pytest.raises(CCDGPUError) as ei:
                sol.step(0.5)
            assert ei.value.status == -5
            sol.reset()
        assert np.isfinite(sol.step(0.5))


def test_mixed_solve_repeats_from_its_own_result():
    """A mixed solve that starts from polished amplitudes uses their image, not an older one."""
    kind, kw = SYSTEMS[4]
    with getattr(System, kind)(**kw) as s, CCDSolver(s, precision="mixed_bf16") as sol:
        r1 = sol.solve(tol=1e-12)
        t1 = sol.t2()
        r2 = sol.solve(tol=1e-12)
        assert r2.iterations < r1.iterations
        assert abs(r2.e_corr - r1.e_corr) <= 1e-10 * abs(r1.e_corr)
        np.testing.assert_allclose(sol.t2(), t1, rtol=0, atol=1e-10)
