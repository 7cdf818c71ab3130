"""Calls of one kernel from two host threads, each on its own stream, whose shared memory differs: every
call runs and gives its own result."""
import ctypes
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _together(calls, n):
    """calls: functions () -> status, run n times each in threads of their own; the failures."""
    bad, start = [], threading.Barrier(len(calls))

    def loop(call):
        start.wait()
        for _ in range(n):
            s = call()
            if s:
                bad.append(s)
    ts = [threading.Thread(target=loop, args=(c,)) for c in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    return bad


def test_height_evaluations_of_two_grids():
    from py_ortho_b200 import _lib as L
    lib, rng = L.load(), np.random.default_rng(0)
    calls, keep, outs = [], [], []
    for W, r in ((300, 1), (500, 3)):                        # 82 and 156 KB
        s = torch.cuda.Stream()
        H, V, D = 4, 2, 1
        img = torch.from_numpy(rng.uniform(0, 255, (60, 80)).astype(np.float32)).cuda()
        cams = np.tile(np.r_[1.0, 0, 0, 0, -1, 0, 0, 0, -1, 0, 0, 40, 100, 0, 0, 0, 39.5, 29.5], (V, 1))
        Z = torch.from_numpy(rng.uniform(0, 3, (D, H, W)).astype(np.float32)).cuda()
        cxs, cys = torch.linspace(-9, 9, W, device="cuda"), torch.linspace(5, -5, H, device="cuda")
        val, score = torch.empty((V, D, H, W), dtype=torch.uint8, device="cuda"), torch.empty((D, H, W), device="cuda")
        a = L.HeightEvalArgs()
        a.V, a.D, a.H, a.W, a.r, a.topk, a.X0, a.Y0, a.gsd = V, D, H, W, r, 1, -9.0, 5.0, 18.0 / W
        for k in range(V):
            a.img[k], a.img_h[k], a.img_w[k] = img.data_ptr(), 60, 80
        a.cams, a.Z, a.cxs, a.cys = cams.ctypes.data, Z.data_ptr(), cxs.data_ptr(), cys.data_ptr()
        a.full, a.min_texture, a.full_texture, a.valid, a.score = 1.0, 1.0, 10.0, val.data_ptr(), score.data_ptr()
        need = lib.mvs_height_eval_scratch_bytes(ctypes.addressof(a))
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
        keep.append((s, img, cams, Z, cxs, cys, val, a, ws))
        call = lambda a=a, ws=ws, need=need, s=s: lib.mvs_height_eval(ctypes.addressof(a), ws.data_ptr(), need, s.cuda_stream)
        torch.cuda.synchronize()
        assert call() == 0
        torch.cuda.synchronize()
        outs.append((score, score.clone()))
        calls.append(call)
    assert _together(calls, 3000) == []
    for got, want in outs:
        assert torch.equal(got, want)


def test_wide_window_means_of_two_images():
    from py_ortho_b200 import _lib as L
    lib, calls, outs = L.load(), [], []
    for W in (7000, 13000):                                  # 56 and 104 KB
        s = torch.cuda.Stream()
        a = torch.rand((2, W), device="cuda")
        out = torch.empty_like(a)
        call = lambda a=a, W=W, out=out, s=s: lib.mvs_box_zero_mean(2, W, a.data_ptr(), 16, 0, out.data_ptr(), s.cuda_stream)
        torch.cuda.synchronize()
        assert call() == 0
        torch.cuda.synchronize()
        outs.append((out, out.clone()))
        calls.append(call)
    assert _together(calls, 300) == []
    for got, want in outs:
        assert torch.equal(got, want)


def test_float32_patchmatch_of_two_windows():
    from py_ortho_b200 import dense
    from test_pm_gpu import _rendered_pm_case
    ref, srcs, ray, Cr, par, depth, normal = _rendered_pm_case(48, 36, 4, seed=3)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ref, ray, depth, normal, srcs = up(ref), up(ray), up(depth), up(normal), [up(s) for s in srcs]
    act = torch.ones((36, 48), dtype=torch.uint8, device="cuda")

    def refine(r, s):
        with torch.cuda.stream(s):
            d, n, sc = depth.clone(), normal.clone(), torch.zeros_like(depth)
            dense.pm_refine(ref, ray, Cr, srcs, [None] * 4, par, d, n, sc, act, r, 1, 2, 0.0, 0.02, 1, 0.1, 1e4, 7,
                            precision="fp32")
            return d
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    want = [refine(r, s) for r, s in zip((4, 5), streams)]   # 85 and 62 KB of windows, 65 and 95 KB of tiles
    torch.cuda.synchronize()

    def call(k):
        try:
            return 0 if torch.equal(refine((4, 5)[k], streams[k]), want[k]) else 1
        except Exception as e:                               # a refused launch
            return str(e)
    assert _together([lambda: call(0), lambda: call(1)], 300) == []
