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
