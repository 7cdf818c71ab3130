"""Point fusion's arguments in every accepted form: the points, colours and order of the plain call."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _flight(n=5, H=37, W=52, seed=0):
    """n overlapping views of a plane with noise; (maps, cams, nbrs, tols, rgbs)."""
    rng = np.random.default_rng(seed)
    cams = [SimpleNamespace(R=np.diag([1.0, -1.0, -1.0]), C=np.array([2.0 * k, 0.5 * k, 40.0]), f=60.0, k1=0.0, k2=0.0,
                            k3=0.0, cx=(W - 1) / 2, cy=(H - 1) / 2, w=W, h=H) for k in range(n)]
    maps = {k: np.where(rng.random((H, W)) < 0.05, np.nan, 40 + rng.normal(0, 0.02, (H, W))).astype(np.float32)
            for k in range(n)}
    nbrs = {k: [j for j in range(n) if j != k] for k in range(n)}
    tols = {k: {j: 0.01 for j in nbrs[k]} for k in nbrs}
    rgbs = {k: rng.integers(0, 256, (H, W, 3)).astype(np.uint8) for k in range(n)}
    return maps, cams, nbrs, tols, rgbs


def _same(got, want):
    assert same_bits(got[0].cpu().numpy(), want[0]) and np.array_equal(got[1].cpu().numpy(), want[1])
    assert np.array_equal(got[2].cpu().numpy(), want[2]) and np.array_equal(got[3].cpu().numpy(), want[3])


def test_an_order_that_can_be_read_once():
    from py_ortho_b200 import views as V
    maps, cams, nbrs, tols, rgbs = _flight()
    want = O.fuse([3, 0, 4, 1, 2], maps, cams, nbrs, tols, 1.5, 2, 2, rgbs)
    assert len(want[0]) > 0
    _same(V.fuse(iter([3, 0, 7, 4, 1, 2]), maps, cams, nbrs, tols, 1.5, 2, 2, rgbs), want)


class _Loading(dict):
    """Colours read from their files on access."""

    def __init__(self, d):
        super().__init__(d)
        self.reads = []

    def __getitem__(self, k):
        self.reads.append(k)
        return super().__getitem__(k)


@pytest.mark.parametrize("rows", [1 << 24, 1])
def test_each_view_s_colours_are_read_once_in_turn(rows, monkeypatch):
    from py_ortho_b200 import views as V
    maps, cams, nbrs, tols, rgbs = _flight(seed=1)
    monkeypatch.setattr(V, "FUSE_GROUP_ROWS", rows)
    lazy = _Loading(rgbs)
    _same(V.fuse(range(5), maps, cams, nbrs, tols, 1.5, 2, 1, lazy), O.fuse(range(5), maps, cams, nbrs, tols, 1.5, 2, 1, rgbs))
    assert lazy.reads == list(range(5))


@pytest.mark.parametrize("rows", [1 << 24, 1])
def test_colours_of_mixed_types(rows, monkeypatch):
    """Views 1 and 3 have float32 colours; view 4 keeps no point (no depth) and has no colours."""
    from py_ortho_b200 import views as V
    maps, cams, nbrs, tols, rgbs = _flight(seed=2)
    monkeypatch.setattr(V, "FUSE_GROUP_ROWS", rows)
    maps[4] = np.full_like(maps[4], np.nan)
    want = O.fuse(range(5), maps, cams, nbrs, tols, 1.5, 2, 1, rgbs)
    mixed = {k: v.astype(np.float32) if k in (1, 3) else v for k, v in rgbs.items() if k != 4}
    mixed[2] = torch.from_numpy(mixed[2]).cuda()
    got = V.fuse(range(5), maps, cams, nbrs, tols, 1.5, 2, 1, mixed)
    assert got[1].dtype == torch.float32
    _same((got[0], got[1].to(torch.uint8), got[2], got[3]), want)
    del mixed[1]
    with pytest.raises(KeyError):
        V.fuse(range(5), maps, cams, nbrs, tols, 1.5, 2, 1, mixed)


@pytest.mark.parametrize("room", [64 << 10, 24 << 10])
def test_without_room_for_every_candidate(room, monkeypatch):
    """Allocations above `room` bytes fail once the first has: 5 x 1924 candidates take 231 KB, one view's 46 KB
    (views one by one), and with less room than that only the kept points' places are taken."""
    from py_ortho_b200 import views as V
    maps, cams, nbrs, tols, rgbs = _flight(seed=3)
    want = O.fuse(range(5), maps, cams, nbrs, tols, 1.5, 2, 1, rgbs)
    empty, refused = torch.empty, []

    def limited(*a, **kw):
        t = empty(*a, **kw)
        # the (candidates, 3) arrays of points; the views' own arrays are flat
        if kw.get("dtype") is torch.float64 and t.ndim == 2 and t.numel() * 8 > room:
            refused.append(t.numel())
            raise torch.cuda.OutOfMemoryError("no room")
        return t
    monkeypatch.setattr(torch, "empty", limited)
    got = V.fuse(iter(range(5)), maps, cams, nbrs, tols, 1.5, 2, 1, rgbs)
    monkeypatch.undo()
    _same(got, want)
    assert len(refused) == (1 if room > 46176 else 6)
    mixed = dict(rgbs)
    mixed[1] = rgbs[1].astype(np.float32)
    monkeypatch.setattr(torch, "empty", limited)
    got = V.fuse(range(5), maps, cams, nbrs, tols, 1.5, 2, 1, mixed)
    monkeypatch.undo()
    assert got[1].dtype == torch.float32
    _same((got[0], got[1].to(torch.uint8), got[2], got[3]), want)


@pytest.mark.parametrize("stride", [36, 37, 52, 53, 2**31 - 60, 2**31 - 1])
def test_strides_around_and_far_beyond_the_image(stride):
    """37 x 52 pixels: from 2 x 2 candidates to the first pixel alone."""
    from py_ortho_b200 import _lib as L, views as V
    maps, cams, nbrs, tols, rgbs = _flight(seed=4)
    for m in maps.values():
        m[0, 0] = 40.0
    want = O.fuse(range(5), maps, cams, nbrs, tols, 1.5, 1, stride, rgbs)
    assert len(want[0]) > 0
    _same(V.fuse(range(5), maps, cams, nbrs, tols, 1.5, 1, stride, rgbs), want)
    assert L.load().mvs_fuse_append_scratch_bytes(37, 52, stride) == 4
