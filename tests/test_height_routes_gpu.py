"""The height sweep's fused kernels against its separate ones and the oracle, bit for bit: the score
evaluation, the 8-direction aggregation at every register layout, the refinement's stack, choice and
median; and the staged host copies."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _sweep(V, PW, PH, opt, seed):
    """A tile of V random views whose footprints cover most of it."""
    from py_ortho_b200 import height as Hs
    rng = np.random.default_rng(seed)
    views = []
    for k in range(V):
        h, w = int(rng.integers(60, 90)), int(rng.integers(70, 100))
        R = np.diag([1.0, -1.0, -1.0]) + rng.normal(0, 0.01, (3, 3))
        C = np.array([rng.uniform(-4, 4), rng.uniform(-4, 4), 40.0])
        img = rng.uniform(0, 255, (h, w, 1)).astype(np.float32)
        views.append(Hs._View([torch.from_numpy(img).cuda()], None, R, C, 1.4 * w, 0.01 if k else 0.0, 0.0, 0.0,
                              (w - 1) / 2, (h - 1) / 2))
    t = Hs._Tile(0, 0, PW, PH, 0, -0.35 * PW, 0.35 * PH, PW, PH, list(range(V)))
    return Hs._TileSweep(t, views, opt, 0.7, torch.device("cuda"))


@pytest.mark.parametrize("V,D,H,W,r", [(2, 1, 1, 1, 0), (2, 3, 31, 33, 1), (6, 5, 32, 64, 3), (3, 2, 65, 257, 3),
                                       (7, 1, 40, 300, 5), (4, 9, 46, 46, 2), (2, 1, 5, 600, 7)])
def test_fused_score_equals_its_parts(V, D, H, W, r):
    from py_ortho_b200 import height as Hs
    sw = _sweep(V, W, H, Hs.DenseOptions(window=r, min_texture=0.5), V * 100 + W)
    rng = np.random.default_rng(D)
    Z = torch.from_numpy(rng.uniform(0, 6, (D, H, W)).astype(np.float32)).cuda()
    score, st, val, ref = sw.score(Z, 0, 0.7, detail=True)
    parts = [torch.empty_like(score), torch.empty_like(st), torch.empty((D, H, W), dtype=torch.int32, device="cuda"),
             torch.empty_like(val)]
    sw._score_parts(Z, 0, 0.7, parts[0], parts[1], parts[2], parts[3], *sw._centres(H, W, 0.7))
    assert torch.equal(val, parts[3]) and torch.equal(ref, parts[2].to(torch.int64))
    assert same_bits(score.cpu().numpy(), parts[0].cpu().numpy()) and same_bits(st.cpu().numpy(), parts[1].cpu().numpy())


def test_score_of_a_grid_too_wide_for_the_fused_means():
    from py_ortho_b200 import height as Hs
    sw = _sweep(2, 1500, 9, Hs.DenseOptions(window=3), 5)
    Z = torch.zeros((1, 9, 1500), device="cuda")
    assert torch.isfinite(sw.score(Z, 0, 0.7)).all()


@pytest.mark.parametrize("D,H,W", [(1, 1, 1), (1, 7, 5), (2, 9, 1), (31, 12, 17), (32, 5, 40), (33, 23, 8), (64, 6, 6),
                                   (65, 11, 13), (129, 7, 9), (256, 5, 6), (257, 4, 5)])
def test_sgm_at_every_layout(D, H, W):
    from py_ortho_b200 import height as Hs
    rng = np.random.default_rng(D)
    cost = rng.uniform(0, 2, (D, H, W)).astype(np.float32)
    got = Hs.sgm(torch.from_numpy(cost).cuda(), 0.05, 0.6).cpu().numpy()
    assert same_bits(got, O.sgm(cost, np.float32(0.05), np.float32(0.6)))


@pytest.mark.parametrize("D,H,W", [(1, 5, 9), (33, 21, 34), (256, 7, 12)])
def test_sgm_one_direction_at_a_time(D, H, W):
    """With room for one volume of scratch only."""
    from py_ortho_b200 import _lib as L
    cost = np.random.default_rng(D + 1).uniform(0, 2, (D, H, W)).astype(np.float32)
    c = torch.from_numpy(cost).cuda()
    agg, ws = torch.empty_like(c), torch.empty_like(c)
    L.check(L.load().mvs_sgm_ws(D, H, W, c.data_ptr(), 0.05, 0.6, agg.data_ptr(), ws.data_ptr(), 4 * c.numel(),
                                L.stream_handle()))
    assert same_bits(agg.cpu().numpy(), O.sgm(cost, np.float32(0.05), np.float32(0.6)))


@pytest.mark.parametrize("hc,wc,HH,WW,level", [(1, 1, 2, 1, 0), (5, 7, 10, 14, 0), (5, 7, 9, 13, 1), (6, 4, 13, 9, 0),
                                               (23, 40, 46, 79, 1)])
def test_refinement_steps(hc, wc, HH, WW, level):
    """Stack, choice and median against the NumPy expressions (float32, one rounding per operation)."""
    from py_ortho_b200 import _lib as L, height as Hs
    rng = np.random.default_rng(hc + WW)
    Zc = rng.uniform(0, 9, (hc, wc)).astype(np.float32)
    K, cell = 9, np.float32(0.7)
    offs = (np.arange(-4, 5) * 0.7).astype(np.float32)
    up = np.pad(np.repeat(np.repeat(Zc, 2, 0), 2, 1)[:HH, :WW], ((0, max(0, HH - 2 * hc)), (0, max(0, WW - 2 * wc))), mode="edge")
    sc = rng.uniform(-0.2, 0.9, (K, HH, WW)).astype(np.float32)
    sc[:, 0, 0] = 0.1
    sc[3:5, -1, -1] = 0.95                                   # a tie: the first one
    t = [torch.from_numpy(a).cuda() for a in (Zc, offs, sc)]
    g_up, g_st, g_out = (torch.empty(s, device="cuda") for s in ((HH, WW), (K, HH, WW), (HH, WW)))
    sh = L.stream_handle()
    L.check(L.load().mvs_height_stack(HH, WW, hc, wc, t[0].data_ptr(), K, t[1].data_ptr(), g_up.data_ptr(), g_st.data_ptr(), sh))
    L.check(L.load().mvs_height_pick(HH, WW, K, t[2].data_ptr(), g_up.data_ptr(), t[1].data_ptr(), 0.2, int(level == 0),
                                     float(cell), g_out.data_ptr(), sh))
    assert same_bits(g_up.cpu().numpy(), up) and same_bits(g_st.cpu().numpy(), up[None] + offs[:, None, None])
    bi = sc.argmax(0)
    pick = lambda i: np.take_along_axis(sc, i[None], 0)[0]
    bi = np.where(pick(bi) < np.float32(0.2), 4, bi)
    frac = np.zeros((HH, WW), np.float32)
    if level == 0:
        lo, hi = pick(np.clip(bi - 1, 0, K - 1)), pick(np.clip(bi + 1, 0, K - 1))
        den = lo - np.float32(2) * pick(bi) + hi
        ok = (den < np.float32(-1e-6)) & (bi > 0) & (bi < K - 1)
        frac = np.where(ok, np.clip(np.float32(0.5) * (lo - hi) / np.where(ok, den, np.float32(-1)), -0.5, 0.5), 0).astype(np.float32)
    want = up + offs[bi] + frac * cell
    assert same_bits(g_out.cpu().numpy(), want)
    p = np.pad(want, 1, mode="edge")
    med = np.sort(np.stack([p[y:y + HH, x:x + WW] for y in range(3) for x in range(3)]), axis=0)[4]
    assert same_bits(Hs._median3(g_out).cpu().numpy(), med)


@pytest.mark.parametrize("n,dtype", [(1, np.float32), (1 << 20, np.float32), ((1 << 21) + 3, np.float32),
                                     (5_000_001, np.float32), (9_000_001, np.bool_)])
def test_staged_copies(n, dtype):
    """Around one piece, two and an uneven number of pieces; on another stream."""
    from py_ortho_b200 import staging
    rng = np.random.default_rng(n)
    a = rng.integers(0, 2, n).astype(dtype) if dtype is np.bool_ else rng.normal(0, 1, n).astype(dtype)
    with torch.cuda.stream(torch.cuda.Stream()):
        t = staging.to_device(a, torch.device("cuda", 0))
        back = staging.to_host(t)
    assert np.array_equal(back, a) and back.dtype == a.dtype


@pytest.mark.parametrize("stride,rows", [(1, 1 << 24), (2, 700), (3, 1)])
def test_fusion_in_groups_and_with_other_colours(stride, rows, monkeypatch):
    """The fused points of a small flight do not depend on how views are grouped; colours of another
    type come through the picking route with the same points."""
    from py_ortho_b200 import views as V
    rng = np.random.default_rng(stride)
    H, W, n = 37, 52, 4
    cams = [SimpleNamespace(R=np.diag([1.0, -1.0, -1.0]), C=np.array([2.0 * k, 0.5 * k, 40.0]), f=60.0, k1=0.0, k2=0.0,
                            k3=0.0, cx=(W - 1) / 2, cy=(H - 1) / 2, w=W, h=H) for k in range(n)]
    maps = {k: np.where(rng.random((H, W)) < 0.05, np.nan, 40 + rng.normal(0, 0.02, (H, W))).astype(np.float32) for k in range(n)}
    nbrs = {k: [j for j in range(n) if j != k] for k in range(n)}
    tols = {k: {j: 0.01 for j in nbrs[k]} for k in nbrs}
    rgbs = {k: rng.integers(0, 256, (H, W, 3)).astype(np.uint8) for k in range(n)}
    want = O.fuse(list(range(n)), maps, cams, nbrs, tols, 1.5, 2, stride, rgbs)
    monkeypatch.setattr(V, "FUSE_GROUP_ROWS", rows)
    xyz, cols, nv, owner, _ = V.fuse(range(n), maps, cams, nbrs, tols, 1.5, 2, stride, rgbs)
    assert same_bits(xyz.cpu().numpy(), want[0]) and np.array_equal(cols.cpu().numpy(), want[1])
    assert np.array_equal(nv.cpu().numpy(), want[2]) and np.array_equal(owner.cpu().numpy(), want[3])
    grey = {k: v.astype(np.float32) for k, v in rgbs.items()}
    x2, c2, n2, o2, _ = V.fuse(range(n), maps, cams, nbrs, tols, 1.5, 2, stride, grey)
    assert torch.equal(x2, xyz) and torch.equal(n2, nv) and torch.equal(o2, owner)
    assert c2.dtype == torch.float32 and torch.equal(c2.to(torch.uint8), cols)
