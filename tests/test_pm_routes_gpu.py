"""The float64 PatchMatch's short cuts against the oracle, bit for bit: window corners that prove a
source inside or outside (pinhole and distorted sources, regular and irregular ray grids), the
geometric bound that skips a candidate's windows (values inside and beyond its range), windows at the
image border, masked reference and source pixels."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["pinhole", "distorted", "irregular", "bright", "outside"])
@pytest.mark.parametrize("n_src,r,step,top_k", [(4, 4, 2, 2), (7, 3, 1, 3)])
def test_pm_fp64_short_cuts_bit_exact_vs_oracle(kind, n_src, r, step, top_k):
    from py_ortho_b200 import dense, scene as S
    W, H = 88, 66
    sc = S.make_scene("c2", seed=17, width=W, height=H)
    rng = np.random.default_rng(n_src * 10 + r)
    ref = sc.grey(sc.ref).astype(np.float32)
    srcs = [sc.grey(s).astype(np.float32) for s in sc.srcs[:n_src]]
    ref[rng.random(ref.shape) < 0.003] = np.nan
    srcs[1][20:24, 30:40] = np.nan
    ray = O.rays_world((H, W), sc.ref_cam)
    par = np.array([c.row() for c in sc.src_cams[:n_src]], np.float64)
    if kind == "distorted":
        par[:, 13:16] = (-0.08, 0.03, -0.01)
    elif kind == "irregular":
        ray = (ray + rng.normal(0, 2e-3, ray.shape)).astype(np.float32)
    elif kind == "bright":
        ref, srcs = ref * np.float32(40), [s * np.float32(40) for s in srcs]
    elif kind == "outside":
        par[0, 9] += 400.0
        par[2, 10] -= 60.0
    depth = (sc.depth_true * (1 + rng.normal(0, 0.01, (H, W)))).astype(np.float32)
    depth[rng.random((H, W)) < 0.05] = np.nan
    normal = S.tilted_normals(H, W, 2)
    active = (rng.random((H, W)) < 0.6).astype(np.uint8)
    deps = [None if k == 1 else np.where(rng.random(s.shape) < 0.05, np.nan, 75.0 + rng.normal(0, 2, s.shape))
            .astype(np.float32) for k, s in enumerate(srcs)]
    args = (r, step, top_k, 0.5, 0.02, 2, 55.0, 95.0, 77)
    a = [depth.copy(), normal.copy(), np.zeros((H, W), np.float32)]
    b = [depth.copy(), normal.copy(), np.zeros((H, W), np.float32)]
    ca = dense.pm_refine(ref, ray, sc.ref_cam.C, srcs, deps, par, *a, active, *args)
    cb = O.pm_refine(ref, ray, sc.ref_cam.C, srcs, deps, par, *b, active, *args)
    assert ca == cb > 0
    for x, y in zip(a, b):
        assert same_bits(x, y)


@pytest.mark.parametrize("W,H,n_src,r,step", [(160, 120, 4, 2, 1), (120, 90, 8, 6, 2)])
def test_pm_fp32_refinement_at_other_windows(W, H, n_src, r, step):
    """The float32 mode's window layouts beside test_pm_gpu's (5 samples a side at step 1, 7 at step
    2), by the mode's own statement: same draws as float64, depth within 0.1 % on 99.9 % of pixels."""
    from py_ortho_b200 import dense
    from test_pm_gpu import _rendered_pm_case
    ref, srcs, ray, Cr, par, depth, normal = _rendered_pm_case(W, H, n_src, seed=3)
    out = []
    for prec in ("fp32", "fp64"):
        st = [depth.copy(), normal.copy(), np.zeros((H, W), np.float32)]
        dense.pm_refine(ref, ray, Cr, srcs, [None] * n_src, par, *st, np.ones((H, W), np.uint8), r, step, 2, 0.0, 0.02,
                        2, float(Cr[2]) - 30.0, float(Cr[2]) + 5.0, 99, precision=prec)
        out.append(st[0].astype(np.float64))
    assert np.array_equal(np.isfinite(out[0]), np.isfinite(out[1]))
    fin = np.isfinite(out[1])
    assert (np.abs(out[0] - out[1])[fin] / out[1][fin] <= 1e-3).mean() >= 0.999
