"""Calls whose scratch cannot come from torch's allocator - no room, a stream that is not torch's, a
stream being captured - give the bits of the plain route."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from conftest import golden, same_bits
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_room(monkeypatch):
    """torch.empty refuses flat byte arrays (what scratch is) above `limit` bytes; the refused sizes."""
    state = SimpleNamespace(limit=0, refused=[])
    empty = torch.empty

    def limited(*a, **kw):
        if kw.get("dtype") is torch.uint8 and len(a) == 1 and isinstance(a[0], int) and a[0] > state.limit:
            state.refused.append(a[0])
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*a, **kw)

    def on(limit=0):
        state.limit = limit
        monkeypatch.setattr(torch, "empty", limited)
        return state
    yield on
    monkeypatch.undo()


def _depth_map():
    from py_ortho_b200 import densify as Dn
    z = golden("depth_map.npz")
    f, cx, cy, w, h = z["intr"]
    rec = SimpleNamespace(intr=[SimpleNamespace(f=f, cx=cx, cy=cy, width=int(w), height=int(h))],
                          cam_group=np.zeros(len(z["C"]), np.int32), X=z["X"], C=z["C"], R=z["R"],
                          obs_cam=z["obs_cam"], obs_pt=z["obs_pt"])
    greys = [((z[f"img{k}"].astype(np.float32) - np.float32(128)) / np.float32(64)).astype(np.float32)
             for k in range(len(z["C"]))]
    opt = Dn.DepthOptions()
    opt.window, opt.num_depths = int(z["opt"][0]), int(z["opt"][1])
    return Dn.depth_map(0, [1, 2, 3, 4], rec, lambda k: (greys[k], None, Dn._Cam(
        z["R"][k], z["C"][k], float(f), 0.0, 0.0, float(cx), float(cy), int(w), int(h))), opt)


def test_a_depth_map_without_room_for_scratch(no_room):
    """The tie-point band and the three sweeps."""
    want = _depth_map()
    state = no_room()
    got = _depth_map()
    assert len(state.refused) >= 2
    for a, b in zip(got, want):
        assert same_bits(a, b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_patchmatch_without_room_for_scratch(precision, no_room):
    from py_ortho_b200 import dense
    from test_pm_gpu import _rendered_pm_case
    ref, srcs, ray, Cr, par, depth, normal = _rendered_pm_case(64, 48, 4, seed=3)
    act = np.ones((48, 64), np.uint8)

    def refine():
        st = [depth.copy(), normal.copy(), np.zeros_like(depth)]
        return [dense.pm_refine(ref, ray, Cr, srcs, [None] * 4, par, *st, act, 2, 1, 2, 0.0, 0.02, 2, 0.1, 1e4, 7,
                                precision=precision)] + st
    want = refine()
    state = no_room()
    got = refine()
    assert len(state.refused) == 1 and got[0] == want[0] > 0
    for a, b in zip(got[1:], want[1:]):
        assert same_bits(a, b)


def _sweep_case():
    from py_ortho_b200 import dense
    from tests_support import random_sweep_case
    h, w, n = 75, 130, 24
    ref, srcs, ray, geo, hyps = random_sweep_case(np.random.default_rng(5), h, w, 3, n)
    mu, sd = O.ref_stats(ref, 2)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    args = [up(a) for a in (ref, mu, sd, ray)] + [[up(a) for a in srcs], geo, dense.Hypotheses.maps_(up(hyps)), 2, 2]

    def reset(state):
        for t in state[:4]:
            t.fill_(-2.0)
        state[4].fill_(-1)
    return args, dense.new_state(h, w), reset


def test_a_sweep_on_a_stream_that_is_not_torch_s():
    from py_ortho_b200 import dense
    args, state, reset = _sweep_case()
    want = [t.clone() for t in dense.sweep(*args, state=state)]
    reset(state)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    dense.sweep(*args, state=state, stream=SimpleNamespace(cuda_stream=s.cuda_stream))
    s.synchronize()
    for a, b in zip(state, want):
        assert torch.equal(a, b)


def test_a_captured_sweep():
    """Captured, the sweep's chunk records are allocated by the graph; replays give the plain call's state."""
    from py_ortho_b200 import _lib as L, dense
    args, state, reset = _sweep_case()
    want = [t.clone() for t in dense.sweep(*args, state=state)]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        dense.sweep(*args, state=state)
    for _ in range(3):
        reset(state)
        g.replay()
        torch.cuda.synchronize()
        for a, b in zip(state, want):
            assert torch.equal(a, b)
    assert L.last_error() == ""


@pytest.mark.parametrize("D,H,W", [(33, 21, 34), (256, 7, 12)])
def test_sgm_without_room_for_eight_volumes(D, H, W, no_room):
    from py_ortho_b200 import height as Hs
    cost = np.random.default_rng(D).uniform(0, 2, (D, H, W)).astype(np.float32)
    state = no_room(4 * D * H * W)
    got = Hs.sgm(torch.from_numpy(cost).cuda(), 0.05, 0.6).cpu().numpy()
    assert state.refused == [32 * D * H * W]
    assert same_bits(got, O.sgm(cost, np.float32(0.05), np.float32(0.6)))
