"""The routes that a sweep takes by where its sources land and by the size of its image, against the
oracle and against each other. Tolerances are the plane path's (tests_support)."""
import dataclasses

import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import oracle as O
from tests_support import check_parity, gap_of

pytestmark = pytest.mark.gpu


def _dev(a, dt=torch.float32):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dt)


def _moved(cam, dx=0.0, dy=0.0, z=None):
    C = np.array(cam.C, np.float64) + np.array([dx, dy, 0.0])
    if z is not None:
        C[2] = z
    return dataclasses.replace(cam, C=C)


@pytest.mark.parametrize("dx,dy,z", [(18.0, 0.0, None), (-34.0, 3.0, None), (0.0, 400.0, None), (7.0, -26.0, None),
                                     (0.0, 0.0, 8.0), (0.0, 0.0, -40.0)])
def test_sources_out_of_view(dx, dy, z):
    """Sources that see part of the view, none of it, or lie between or beyond the planes (some or
    all of the points behind them): tiles whose halo maps wholly outside a source skip it."""
    from py_ortho_b200 import dense, scene as S
    sc = S.make_scene("c1", seed=6, width=200, height=120)
    ref = sc.grey(sc.ref)
    srcs = [sc.grey(s) for s in sc.srcs]
    cams = [_moved(sc.src_cams[0], dx, dy, z), sc.src_cams[1], _moved(sc.src_cams[2], -dx, dy, z), sc.src_cams[3]]
    planes, r = S.plane_list(35.0, 55.0, 12), 3
    mu, sd = O.ref_stats(ref, r)
    geo = S.geo_rows(sc.ref_cam, cams)
    hyp = dense.Hypotheses.planes_inv(planes)
    st = dense.sweep(_dev(ref), _dev(mu), _dev(sd), None, [_dev(s) for s in srcs], geo, hyp, r, 2,
                     ref_cam=sc.ref_cam.row())
    depth = dense.finalize(hyp, st)
    ray = O.rays_world(ref.shape, sc.ref_cam)
    full = O.sweep(ref, srcs, ray, geo, [np.full(ref.shape, p, np.float32) for p in planes], r, 2, keep_scores=True)
    check_parity(st[4].cpu().numpy(), depth.cpu().numpy(), st[0].cpu().numpy(), full["idx"], full["depth"],
                 full["best"], gap_of(full["scores"]), f"moved {dx} {dy} {z}")


@pytest.mark.parametrize("w,h,n", [(33, 9, 3), (64, 32, 7), (65, 33, 40), (200, 150, 2), (640, 480, 13)])
def test_automatic_chunks_keep_the_bits(w, h, n):
    """The automatic number of plane chunks follows from the tiles and the planes; the state is the
    one-chunk state bit for bit, also for continued sweeps."""
    from py_ortho_b200 import dense
    from tests_support import random_sweep_case
    rng = np.random.default_rng(w + n)
    ref, srcs, ray, geo, hyps = random_sweep_case(rng, h, w, 3, n)
    mu, sd = O.ref_stats(ref, 2)
    t = [_dev(a) for a in (ref, mu, sd, ray)]
    s, hyp = [_dev(a) for a in srcs], dense.Hypotheses.maps_(_dev(hyps))
    a = dense.sweep(*t, s, geo, hyp, 2, 2, plane_chunks=1)
    b = dense.sweep(*t, s, geo, hyp, 2, 2)
    for x, y in zip(a, b):
        assert same_bits(x.cpu().numpy(), y.cpu().numpy())
    a = dense.sweep(*t, s, geo, hyp, 2, 2, state=a, plane_chunks=1)
    b = dense.sweep(*t, s, geo, hyp, 2, 2, state=b)
    for x, y in zip(a, b):
        assert same_bits(x.cpu().numpy(), y.cpu().numpy())


@pytest.mark.parametrize("r", [0, 1, 3, 4, 5, 7])
def test_special_inverse_depths(r):
    """The per-pixel path's inverse depths at the ends of their range, against the oracle's
    per-hypothesis scores (float64 window sums, which track it to ~1e-7; bar: tests_support):
    infinite (depth 0: the reference's own centre as the source sees it), negative, tiny, huge;
    0 and NaN have no valid sample, so every score is -1."""
    from py_ortho_b200 import _lib as L, dense
    from tests_support import SCORE_ABS, random_sweep_case
    rng = np.random.default_rng(40 + r)
    H, W, n = 45, 71, 3
    ref, srcs, ray, geo, _ = random_sweep_case(rng, H, W, n, 2, nan_frac=0.0)
    geo[:, 11] = (0.5, -0.5, 2.0)                  # b_z: in front, behind, in front
    geo[2, 13:16] = 0.0                            # one pinhole source
    base = rng.uniform(0.02, 0.2, (H, W)).astype(np.float32)
    special = [base, np.full_like(base, np.inf), np.full_like(base, -np.inf), -base, np.full_like(base, 1e-30),
               np.full_like(base, 1e30), np.zeros_like(base), np.full_like(base, np.nan)]
    mixed = np.stack(special)[rng.integers(0, len(special) - 2, (H, W)), np.arange(H)[:, None], np.arange(W)[None]]
    mu, sd = O.ref_stats(ref, r)
    t = [_dev(a) for a in (ref, mu, sd, ray)]
    s = [_dev(a) for a in srcs]
    for k, inv in enumerate(special + [mixed]):
        st = dense.sweep(*t, s, geo, dense.Hypotheses.maps_(_dev(inv[None])), r, 2, precision=L.PREC_FP64_SUMS)
        got = st[1].cpu().numpy()
        if k in (6, 7):
            assert np.all(got == -1.0), k
            continue
        full = O.sweep(ref, srcs, ray, geo, [np.ascontiguousarray(inv)], r, 2, keep_scores=True)
        assert np.abs(got - full["scores"][0]).max() <= SCORE_ABS, k


@pytest.mark.parametrize("h,w", [(1, 1), (3, 200), (31, 33), (32, 64), (65, 129), (130, 31), (257, 300)])
def test_window_statistics_at_tile_edges(h, w):
    """The window mean and deviation bit for bit against the oracle: sizes around the 32-row /
    32-column steps, radii inside and beyond the row pass's ring (15), windows larger than the image,
    NaN and infinite pixels."""
    from py_ortho_b200 import fast
    rng = np.random.default_rng(h * 1000 + w)
    a = rng.normal(0, 1, (h, w)).astype(np.float32)
    b = a.copy()
    b[rng.random((h, w)) < 0.01] = np.nan
    b[h // 2, w // 2] = np.inf
    for img in (a, b):
        with np.errstate(invalid="ignore"):
            for r in (0, 1, 5, 14, 15, 16, 40):
                mu, sd = O.ref_stats(img, r)
                gm, gs = fast.ref_stats(img, r)
                nan = np.isnan(mu), np.isnan(sd)
                assert np.array_equal(np.isnan(gm), nan[0]) and np.array_equal(np.isnan(gs), nan[1]), r
                assert same_bits(gm[~nan[0]], mu[~nan[0]]) and same_bits(gs[~nan[1]], sd[~nan[1]]), r
                assert same_bits(fast.box_zero_mean(img, r)[~nan[0]], mu[~nan[0]]), r
