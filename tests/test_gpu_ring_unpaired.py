"""Fused handles whose modified channels are not pairs of transposed channels in the order of the ph'
and hp' lists: a channel whose rows are shared out over two, lists in another order than the tables'
rows and columns, lists of which some are missing, and none; against the oracle.

Tolerances are those of the parity tests: energies to 1e-12 relative, amplitudes to 1e-13.
"""
import ctypes

import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDSolver, System, _native
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

SYSTEMS = [
    ("inf_matter", dict(density=0.08, tz_max=1, n_shells=4, n_particle_shells=2)),
    ("electron_gas", dict(r_s=1.3, n_shells=7, n_particle_shells=4)),
]
PD = ctypes.POINTER(ctypes.c_double)


def split(p, keep):
    """Every fifth modified channel's rows from the middle on go to an empty channel slot."""
    dims = p.chan_mod_dims
    free = [c for c in range(p.n_channels) if not (dims[c].ph and dims[c].hp)]
    used = [c for c in range(p.n_channels) if dims[c].ph > 1 and dims[c].hp][::5]
    moved = {}
    for c, slot in zip(used, free):
        ph, hp, r = dims[c].ph, dims[c].hp, dims[c].ph // 2
        v = np.ctypeslib.as_array(p.v_hpph_mod[c], (hp, ph))
        parts = [np.ascontiguousarray(v[:, :r]), np.ascontiguousarray(v[:, r:])]
        keep += parts
        p.v_hpph_mod[c], p.v_hpph_mod[slot] = (x.ctypes.data_as(PD) for x in parts)
        p.v_hphp_mod[slot] = p.v_hphp_mod[c]
        maps = p.chan_mod_maps
        maps[slot].hp = maps[c].hp
        maps[slot].ph = ctypes.cast(
            ctypes.addressof(maps[c].ph.contents) + r * ctypes.sizeof(_native.Pair),
            ctypes.POINTER(_native.Pair))
        dims[c].ph, dims[slot].ph, dims[slot].hp = r, ph - r, hp
        moved[c] = slot, r
    assert len(moved) >= 3
    for k in range(4, 8):
        for c in range(p.n_channels):
            n = p.chan_dims[c].pp * p.chan_dims[c].hh
            if not n:
                continue
            t = np.ctypeslib.as_array(ctypes.cast(p.maps[k][c], ctypes.POINTER(ctypes.c_uint64)),
                                      (n, 3))
            for m, (slot, r) in moved.items():
                at = (t[:, 0] == m) & (t[:, 1] >= r)
                t[at, 0] = slot
                t[at, 1] -= np.uint64(r)


def reorder(p, keep):
    rng = np.random.default_rng(4)
    for c in range(p.n_channels):
        for kind in ("ph", "hp"):
            n, at = getattr(p.chan_mod_dims[c], kind), getattr(p.chan_mod_maps[c], kind)
            if n and at:
                q = np.ctypeslib.as_array(ctypes.cast(at, ctypes.POINTER(ctypes.c_uint64)), (n, 2))
                q[:] = q[rng.permutation(n)]


def drop_some(p, keep):
    for c in range(0, p.n_channels, 3):
        p.chan_mod_maps[c].ph = None


def drop_all(p, keep):
    p.chan_mod_maps = None


def spoil(p, keep):
    for c in range(p.n_channels):
        if p.chan_mod_dims[c].ph and p.chan_mod_dims[c].hp:
            p.chan_mod_maps[c].ph[0].p = 1 << 40
            return


@pytest.mark.parametrize("precision", ["fp64", "mixed_bf16"])
@pytest.mark.parametrize("change", [split, reorder, drop_some, drop_all, spoil])
@pytest.mark.parametrize("kind,kw", SYSTEMS)
def test_fused_matches_oracle(kind, kw, change, precision):
    keep = []
    with getattr(System, kind)(**kw) as s:
        p = s.problem.contents
        change(p, keep)
        o = Oracle(s)
        with CCDSolver(s, precision=precision) as sol:
            if precision == "fp64":
                for _ in range(3):
                    e_ref, e = o.step(0.5), sol.step(0.5)
                    assert abs(e - e_ref) <= 1e-12 * abs(e_ref)
                    np.testing.assert_allclose(sol.t2(), o.t2(), rtol=0, atol=1e-13)
                o.reset()
                sol.reset()
            e_ref = o.solve(tol=1e-11, max_iters=60, mixing=0.5)[0]
            r = sol.solve(tol=1e-11, max_iters=60, mixing=0.5)
            assert abs(r.e_corr - e_ref) <= 1e-10 * abs(e_ref)
        o.close()
