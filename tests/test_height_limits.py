"""The height sweep's entry points at the edges of what they accept."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import same_bits


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


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(1, 2**31 - 2), (2**31 - 2, 1)])
def test_refinement_steps_on_the_largest_grids(H, W):
    """Within 256 cells of 2^31 (8.6 GB an array), checked in pieces."""
    from py_ortho_b200 import _lib as L
    lib, sh, n = L.load(), L.stream_handle(), H * W
    z = torch.rand(n // 2, device="cuda")
    up, out = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    off = torch.tensor([0.25], device="cuda")
    hc, wc = (1, W // 2) if H == 1 else (H // 2, 1)
    L.check(lib.mvs_height_stack(H, W, hc, wc, z.data_ptr(), 1, off.data_ptr(), up.data_ptr(), out.data_ptr(), sh))
    for o in (0, n // 4 * 2, n - 600):
        want = z[o // 2:o // 2 + 300].repeat_interleave(2)
        assert torch.equal(up[o:o + 600], want) and torch.equal(out[o:o + 600], want + 0.25)
    # a single score is its own best: up + offs[0]
    L.check(lib.mvs_height_pick(H, W, 1, up.data_ptr(), up.data_ptr(), off.data_ptr(), 0.0, 1, 1.0, out.data_ptr(), sh))
    assert torch.equal(out[-600:], up[-600:] + 0.25) and torch.equal(out[:600], up[:600] + 0.25)
    L.check(lib.mvs_median3(H, W, up.data_ptr(), out.data_ptr(), sh))
    for o in (0, n - 600):
        v = up[o:o + 600]
        lo, hi = torch.cat([v[:1], v[:-1]]), torch.cat([v[1:], v[-1:]])
        want = torch.sort(torch.stack([lo, v, hi]), dim=0).values[1]       # three equal rows (columns): the middle of 3
        s = slice(0, 599) if o == 0 else slice(1, 600)
        assert torch.equal(out[o:o + 600][s], want[s])


@pytest.mark.gpu
@pytest.mark.parametrize("W,r", [(656, 3), (775, 0), (1024, 3), (1025, 3), (1500, 3)])
def test_the_score_of_a_grid_too_wide_for_the_fused_evaluation(W, r):
    """The fused call refuses it and writes nothing; its parts give, away from the crop's border, the fused
    score of the grid's first 600 columns."""
    from py_ortho_b200 import _lib as L, height as Hs
    from test_height_routes_gpu import _sweep
    H, C, V = 20, 600, 3
    sw = _sweep(V, W, H, Hs.DenseOptions(window=r, min_texture=0.5), 5)
    sw.t.X0, sw.t.Y0 = -14.0, 7.0                            # the views see the first columns
    Z = torch.rand((2, H, W), device="cuda") * 6
    outs = [torch.full((V, 2, H, W), 77, dtype=torch.uint8, device="cuda"), torch.full((2, H, W), 7.5, device="cuda")]
    a = _eval_args(L, W, r, H, 2)
    cams, img = np.zeros((2, 18)), sw.views[0].pyr[0]
    a.cams, a.Z, a.valid, a.score = cams.ctypes.data, Z.data_ptr(), outs[0].data_ptr(), outs[1].data_ptr()
    a.cxs, a.cys = (t.data_ptr() for t in sw._centres(H, W, 0.7))
    for k in range(2):
        a.img[k], a.img_h[k], a.img_w[k] = img.data_ptr(), int(img.shape[0]), int(img.shape[1])
    ws = torch.empty(1 << 24, dtype=torch.uint8, device="cuda")
    assert L.load().mvs_height_eval(ctypes.addressof(a), ws.data_ptr(), ws.numel(), L.stream_handle()) == L.ERR_UNSUPPORTED
    torch.cuda.synchronize()
    assert (outs[0] == 77).all() and (outs[1] == 7.5).all()
    got = sw.score(Z, 0, 0.7, detail=True)
    crop = _eval_args(L, C, r, H, 2)
    assert L.load().mvs_height_eval_scratch_bytes(ctypes.addressof(crop)) > 0
    want = sw.score(Z[:, :, :C].contiguous(), 0, 0.7, detail=True)
    assert 0 < int(got[2].sum()) < got[2].numel() and (r == 0 or got[0].std() > 0)
    for x, y in zip(got, want):
        assert same_bits(x[..., :C - r].cpu().numpy(), y[..., :C - r].cpu().numpy())
