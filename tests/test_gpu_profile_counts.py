"""The work that the kernel profile counts for the one-body class is that of what it times: the sums
over the pairs that hold each orbital, and T X."""
import numpy as np
import pytest

from coupled_cluster_doubles_b200 import CCDSolver, System

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,precision,with_tx", [
    (dict(r_s=1.0, n_shells=9, n_particle_shells=3), "fp64", True),
    (dict(r_s=1.0, n_shells=16, n_particle_shells=3), "mixed_bf16", True),   # 230 rows
    (dict(r_s=1.0, n_shells=7, n_particle_shells=3), "mixed_bf16", False),   # T X in the ladder
])
def test_onebody_class(kw, precision, with_tx):
    with System.electron_gas(**kw) as s, CCDSolver(s, precision=precision) as sol:
        flops, byts, pairs, op, oh = 0, 0, 0, 0, 0
        pp, hh = (s.array(k).reshape(-1, 2) for k in ("pp_map", "hh_map"))
        for n, m in s.chan_dims()[:, :2].astype(int):
            pk = int((pp[op:op + n, 0] < pp[op:op + n, 1]).sum())
            hk = int((hh[oh:oh + m, 0] < hh[oh:oh + m, 1]).sum())
            op, oh = op + n, oh + m
            if n and m:
                pairs += 2 * pk + 2 * hk  # an entry for each of a pair's orbitals
            if with_tx and pk and hk:
                flops += 2 * pk * hk * hk
                byts += 16 * pk * hk + 8 * hk * hk
        byts += 16 * s.n_sp + 12 * pairs
        _, f, b = sol.kernel_profile(reps=2)["onebody"]
        assert f == flops
        assert b == byts
        assert (f > 0) == with_tx
        e = sol.step(0.5)
        sol.reset()
        assert sol.step(0.5) == e  # nothing of the iteration's state was changed
