"""The height sweep's entry points at the edges of what they accept."""
import ctypes

import pytest


def _eval_args(L, W, r, H=8, D=1):
    a = L.HeightEvalArgs()
    a.V, a.D, a.H, a.W, a.r, a.topk, a.gsd = 2, D, H, W, r, 1, 1.0
    a.cams = a.Z = a.cxs = a.cys = a.valid = a.score = 256          # never read: the size query only
    for k in range(2):
        a.img[k], a.img_h[k], a.img_w[k] = 256, 4, 4
    return a


@pytest.mark.parametrize("W,r,fits", [(774, 0, True), (775, 0, False), (521, 8, True), (522, 8, False), (1, 6383, True),
                                      (1, 6384, False), (1500, 3, False), (9, 2**30, False), (9, 2**31 - 20, False),
                                      (9, 2**31 - 16, False), (1000, 2**31 - 8, False), (1, 2**31 - 1, False)])
def test_the_fused_evaluation_takes_what_its_window_means_fit(W, r, fits):
    """(32 + 2 r + 1) (W + 1) doubles within 200 KB, also for radii whose double passes 2^31."""
    from py_ortho_b200 import _lib as L
    a = _eval_args(L, W, r)
    need = L.load().mvs_height_eval_scratch_bytes(ctypes.addressof(a))
    assert fits == ((32 + 2 * r + 1) * (W + 1) * 8 <= 200 * 1024)
    assert (need > 0) == fits
