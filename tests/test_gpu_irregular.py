"""Table path and stage calls on amplitudes and host V blocks without the antisymmetry in (a, b) or in
(i, j) that the packed kernels rely on, against the oracle: channels with and without strict hole
pairs, V_pppp in one and in several row tiles, stored whole and by its symmetry, and generated.

Tolerances are those of the parity tests: amplitudes to 1e-13, t2Diff_pphh to 1e-12 of its largest
element.
"""
import ctypes

import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDSolver, System, solver as solver_mod
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

SYSTEMS = [
    ("pairing", dict(xi=1.0, g=0.4, n_pair_states=7, n_particles=4)),
    ("inf_matter", dict(density=0.16, tz_max=2, n_shells=4, n_particle_shells=1)),
    ("electron_gas", dict(r_s=1.3, n_shells=7, n_particle_shells=4)),
    ("electron_gas", dict(r_s=1.0, n_shells=13, n_particle_shells=2)),
]


def channels(s):
    """(channel, pp, hh, exchanged pp pair, exchanged hh pair, t2 offset) of the active channels."""
    pp_map = s.array("pp_map").reshape(-1, 2).astype(int)
    hh_map = s.array("hh_map").reshape(-1, 2).astype(int)

    def exchanged(q):
        at = {tuple(x): k for k, x in enumerate(q)}
        return np.array([at[(y, x)] for x, y in q], int)

    op = oh = ot = 0
    for ch, (pp, hh) in enumerate(s.chan_dims()[:, :2].astype(int)):
        if pp and hh:
            yield ch, pp, hh, exchanged(pp_map[op:op + pp]), exchanged(hh_map[oh:oh + hh]), ot
            ot += pp * hh
        op += pp
        oh += hh


def amplitudes(s, what, rng):
    t2 = np.zeros(s.t2_size())
    for _, pp, hh, ba, ji, at in channels(s):
        t = rng.uniform(-0.05, 0.05, (pp, hh))
        if what != "any" and what != "ij":
            t -= t[:, ji]
        if what != "any" and what != "ab":
            t -= t[ba, :]
        t2[at:at + pp * hh] = t.ravel()
    return t2


def perturb(s, what, rng):
    def block(pointers, ch, shape):
        return np.ctypeslib.as_array(
            ctypes.cast(pointers[ch], ctypes.POINTER(ctypes.c_double)), shape)

    p = s.problem.contents
    for ch, pp, hh, ba, ji, _ in channels(s):
        if what == "v_hhhh":
            v = block(p.v_hhhh, ch, (hh, hh))
            v += 0.2 * np.max(np.abs(v)) * rng.uniform(-1, 1, v.shape)
        elif what:
            v = block(p.v_hhpp, ch, (hh, pp))
            m = 0.2 * np.max(np.abs(v)) * rng.uniform(-1, 1, v.shape)
            v += m - m[:, ba] if what == "v_hhpp_ij" else m - m[ji, :] if what == "v_hhpp_ab" else m


def stages(sol):
    sol.calc_t2diff_p2_p1hh()
    sol.calc_t2diff_h2pp_h1()
    sol.calc_t2diff_phhp()
    sol.calc_t2diff_pphh()
    sol.map_from_distributed()
    sol.calc_t2_pphh(0.5)
    sol.map_to_distributed()


def check(sol, o, count=3, how=lambda sol: sol.step(0.5)):
    for _ in range(count):
        o.step(0.5)
        how(sol)
        d_ref, d = (x.chain(solver_mod.CHAIN_DIFF_PPHH) for x in (o, sol))
        assert np.max(np.abs(d - d_ref)) <= 1e-12 * max(np.max(np.abs(d_ref)), 1e-300)
        np.testing.assert_allclose(sol.t2(), o.t2(), rtol=0, atol=1e-13)


@pytest.mark.parametrize("v_mode", ["stored", "on_the_fly"])
@pytest.mark.parametrize("what", ["ij", "ab", "any"])
@pytest.mark.parametrize("kind,kw", SYSTEMS)
def test_amplitudes(kind, kw, what, v_mode):
    with getattr(System, kind)(**kw) as s, CCDSolver(s, path="tables", v_mode=v_mode) as sol:
        o, t2 = Oracle(s), amplitudes(s, what, np.random.default_rng(5))
        o.set_t2(t2)
        sol.set_t2(t2)
        check(sol, o)
        # ... and back to the packed kernels, with nothing left behind.
        t2 = amplitudes(s, "", np.random.default_rng(6))
        for x in (o, sol):
            x.reset()
            x.set_t2(t2)
        check(sol, o, 2)
        o.close()


@pytest.mark.parametrize("what", ["v_hhhh", "v_hhpp_ij", "v_hhpp_ab", "v_hhpp"])
@pytest.mark.parametrize("kind,kw", SYSTEMS)
def test_host_v(kind, kw, what):
    with getattr(System, kind)(**kw) as s:
        perturb(s, what, np.random.default_rng(8))
        with CCDSolver(s, path="tables") as sol:
            o = Oracle(s)
            check(sol, o)
            o.close()


@pytest.mark.parametrize("what,v", [("ij", None), ("any", None), ("", "v_hhpp_ij"), ("", "v_hhhh")])
@pytest.mark.parametrize("precision", ["fp64", "mixed_bf16"])
def test_stage_calls_on_a_fused_handle(what, v, precision):
    kind, kw = SYSTEMS[2]
    with getattr(System, kind)(**kw) as s:
        perturb(s, v, np.random.default_rng(9))
        with CCDSolver(s, precision=precision) as sol:
            o, t2 = Oracle(s), amplitudes(s, what, np.random.default_rng(5))
            o.set_t2(t2)
            sol.set_t2(t2)
            check(sol, o, 2, stages)
            o.close()


@pytest.mark.parametrize("kind,kw", SYSTEMS + [
    ("inf_matter", dict(density=0.08, tz_max=1, n_shells=6, n_particle_shells=3))])
def test_the_models_own_v_is_regular(kind, kw):
    """The models' blocks take the packed kernels (more than the two launches of the other path), also
    from amplitudes that an iteration's rounding has left."""
    launches = []
    with getattr(System, kind)(**kw) as s:
        for v_mode in ("stored", "on_the_fly"):
            with CCDSolver(s, path="tables", v_mode=v_mode) as sol:
                for _ in range(2):
                    sol.step(0.5)
                sol.set_t2(sol.t2())
                before = sol.profile()["launches"]
                sol.calc_t2diff_pphh()
                launches.append(sol.profile()["launches"] - before)
    assert launches[0] == launches[1] > 2
