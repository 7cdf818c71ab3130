"""The automatic number of plane chunks, seen in the scratch that a sweep asks for (no GPU work)."""
import ctypes

import numpy as np
import pytest


def _scratch(H, W, n_src, r, top_k, n):
    from py_ortho_b200 import _lib as L
    geo, cam, planes = np.zeros((n_src, 18)), np.zeros(18), np.ones(n, np.float32)
    geo[:, 12] = cam[12] = 1.0
    a = L.SweepArgs()
    a.H, a.W, a.n_src, a.r, a.top_k, a.i1 = H, W, n_src, r, top_k, n
    a.ref = a.mu = a.sd = a.best = a.prev = a.s_prev_best = a.s_next_best = a.idx = 256      # never read
    for k in range(n_src):
        a.src[k], a.src_h[k], a.src_w[k] = 256, H, W
    a.geo, a.ref_cam = geo.ctypes.data, cam.ctypes.data
    a.hyp.kind, a.hyp.n, a.hyp.planes = L.HYP_PLANES, n, planes.ctypes.data
    return L.load().mvs_sweep_scratch_bytes(ctypes.addressof(a))


@pytest.mark.parametrize("r", range(8))
def test_chunks_are_planned_for_the_lists_that_the_kernel_keeps(r):
    """The list has min(top_k, sources) entries: a larger top_k plans the same launch."""
    sizes = [(H, W, n) for H, W in ((48, 64), (240, 320), (480, 640), (700, 900)) for n in (16, 64, 128)]
    plans = [_scratch(H, W, 2, r, 2, n) for H, W, n in sizes]
    assert max(plans) > 0
    for k in (3, 9):
        assert [_scratch(H, W, 2, r, k, n) for H, W, n in sizes] == plans
