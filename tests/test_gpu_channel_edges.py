"""The allocation-free channel entry point at the edges of its tiles: 64-row slices of the pp
index (one slice has no separate sum), 16-row blocks, 16-deep K steps split over the warps,
8-column tiles, and the widest channels.

Tolerance, element by element: a sum of n products in any order is off by at most n 2^-53 of the
sum of the magnitudes, so with X and D each a chain of such sums the bound is
2 (pp + hh + 8) 2^-53 (|V| |T| + |T| (|V_hhhh| + |V_hhpp| |T|)) against an extended-precision
evaluation.
"""
import ctypes

import numpy as np
import pytest

from coupled_cluster_doubles_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pp", [1, 15, 16, 17, 63, 64, 65, 129, 257])
@pytest.mark.parametrize("hh", [1, 7, 8, 9, 16, 17, 33, 41, 72])
def test_channel_ladder_at_tile_edges(pp, hh):
    import torch

    rng = np.random.default_rng(1000 * pp + hh)
    v4, x4 = rng.standard_normal((pp, pp)), rng.standard_normal((hh, pp))
    h4, t2 = rng.standard_normal((hh, hh)), rng.standard_normal((pp, hh))
    dev = [torch.from_numpy(a).cuda() for a in (v4, x4, h4, t2)]
    out = torch.full((pp, hh), float("nan"), dtype=torch.float64, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = _native.gpu_lib().ccdgpu_calc_channel_t2diff_pphh_noalloc(
        *(a.data_ptr() for a in dev), out.data_ptr(), pp, hh, stream)
    assert rc == 0
    wide = np.longdouble
    t = t2.astype(wide)
    ref = wide(0.5) * (t @ (h4 + wide(0.5) * (x4.astype(wide) @ t)) + v4.astype(wide) @ t)
    size = np.abs(v4) @ np.abs(t2) + np.abs(t2) @ (np.abs(h4) + np.abs(x4) @ np.abs(t2))
    assert np.all(np.abs(out.cpu().numpy() - ref) <= 2 * (pp + hh + 8) * 2.0 ** -53 * size)
