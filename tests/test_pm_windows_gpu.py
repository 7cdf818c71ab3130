"""PatchMatch windows far larger than the image, and steps far larger than the window, against the
oracle: window positions, the bound on the rays' bend and the shared memory sizes do not wrap."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(seed=17, W=30, H=22, n_src=3):
    from py_ortho_b200 import scene as S
    sc = S.make_scene("c2", seed=seed, width=W, height=H)
    rng = np.random.default_rng(seed)
    ref = sc.grey(sc.ref).astype(np.float32)
    srcs = [sc.grey(s).astype(np.float32) for s in sc.srcs[:n_src]]
    ray = O.rays_world((H, W), sc.ref_cam)
    par = np.array([c.row() for c in sc.src_cams[:n_src]], np.float64)
    depth = (sc.depth_true * (1 + rng.normal(0, 0.01, (H, W)))).astype(np.float32)
    return ref, srcs, ray, sc.ref_cam.C, par, depth, S.tilted_normals(H, W, 2), np.ones((H, W), np.uint8)


def _refine(fn, r, step, **kw):
    ref, srcs, ray, Cr, par, depth, normal, act = _case()
    st = [depth, normal, np.zeros_like(depth)]
    n = fn(ref, ray, Cr, srcs, [None] * 3, par, *st, act, r, step, 2, 0.0, 0.02, 2, 55.0, 95.0, 77, **kw)
    return n, st


# (50000, 5): every fifth pixel of the image is a sample; r r passes 2^31. Steps near 2^31: no sample, or
# the centre alone
@pytest.mark.parametrize("r,step", [(50000, 5), (46340, 46340), (40, 3), (5, 2**31 - 1), (1, 2**31 - 2), (0, 2**31 - 1),
                                    (2**30 - 1, 2**30 - 1), (2**30 + 5, 2**30)])
def test_large_windows_and_steps_bit_exact_vs_oracle(r, step):
    from py_ortho_b200 import dense
    na, a = _refine(dense.pm_refine, r, step)
    nb, b = _refine(O.pm_refine, r, step)
    assert na == nb
    for x, y in zip(a, b):
        assert same_bits(x, y)


@pytest.mark.parametrize("r,step", [(2**30 + 5, 2**30), (2**30 - 1, 2**30 - 1)])
def test_float32_windows_whose_positions_are_not_ints_run_in_float64(r, step):
    from py_ortho_b200 import dense
    na, a = _refine(dense.pm_refine, r, step, precision="fp32")
    nb, b = _refine(dense.pm_refine, r, step)
    assert na == nb
    for x, y in zip(a, b):
        assert same_bits(x, y)


@pytest.mark.parametrize("r,step,precision,error", [(2**30, 2**30, "fp64", ValueError), (2**31 - 1, 1, "fp64", ValueError),
                                                    (2**31 - 1, 2**31 - 1, "fp32", ValueError),
                                                    (60, 1, "fp32", RuntimeError), (1 << 20, 1, "fp32", RuntimeError)])
def test_windows_that_are_refused(r, step, precision, error):
    """A step past the window's last offset that is no int; float32 windows above a block's shared memory
    (121 samples a side, and 2^21 + 1, whose square wraps)."""
    from py_ortho_b200 import dense
    with pytest.raises(error):
        _refine(dense.pm_refine, r, step, precision=precision)


@pytest.mark.parametrize("r,step,length,bend", [(3, 1, 1.0, 0.0), (3, 1, 1e5, 3e-4), (12, 4, 1e-3, 0.0), (12, 4, 1e3, 3e-4),
                                               (30, 10, 1e5, 0.0)])
def test_planes_seen_edge_on_bit_exact_vs_oracle(r, step, length, bend):
    """Normals of any length, nearly perpendicular to their rays, on straight and on irregular ray grids: the
    proofs that a window lies inside or outside a source hold where the plane's terms cancel. Every candidate
    is outside the depth range, so the score map is the current planes' photo term."""
    from py_ortho_b200 import dense, scene as S
    W, H = 64, 48
    sc = S.make_scene("c2", seed=5, width=W, height=H)
    rng = np.random.default_rng(r + int(np.log10(length)) + int(bend * 1e5))
    ref = sc.grey(sc.ref).astype(np.float32)
    srcs = [sc.grey(s).astype(np.float32) for s in sc.srcs[:6]]
    par = np.array([c.row() for c in sc.src_cams[:6]], np.float64)
    ray = (O.rays_world((H, W), sc.ref_cam) + rng.normal(0, 1, (3, H, W)) * bend).astype(np.float32)
    u = ray / np.linalg.norm(ray, axis=0)
    t = np.cross(u, rng.normal(0, 1, (3, H, W)), axis=0)
    t /= np.linalg.norm(t, axis=0)
    eps = 10.0 ** rng.uniform(-5, -1, (H, W))
    normal = ((t - eps * u) * length).astype(np.float32)
    depth = (sc.depth_true * (1 + rng.normal(0, 0.01, (H, W)))).astype(np.float32)
    act = np.ones((H, W), np.uint8)
    out = []
    for fn in (dense.pm_refine, O.pm_refine):
        st = [depth.copy(), normal.copy(), np.zeros((H, W), np.float32)]
        assert fn(ref, ray, sc.ref_cam.C, srcs, [None] * 6, par, *st, act, r, step, 3, 0.0, 0.02, 1, 1e9, 1e9 + 1, 5) == 0
        out.append(st[2])
    assert same_bits(*out)
