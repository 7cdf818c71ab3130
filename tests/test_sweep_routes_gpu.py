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
