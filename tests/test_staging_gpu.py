"""Host arrays of every accepted kind through the staged copies."""
import warnings

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.fixture
def always_warn():
    before = torch.is_warn_always_enabled()
    torch.set_warn_always(True)
    yield
    torch.set_warn_always(before)


@pytest.mark.parametrize("n", [1, 1000, 3 << 20])
@pytest.mark.parametrize("kind", ["array", "read-only", "mapped"])
def test_read_only_arrays_are_copied_without_a_warning(n, kind, always_warn, tmp_path):
    """A decoded image or a mapped file is read-only; torch warns when it wraps one."""
    from py_ortho_b200 import densify, staging
    a = np.random.default_rng(n).normal(0, 1, n).astype(np.float32)
    want = a.copy()
    if kind == "read-only":
        a.flags.writeable = False
    elif kind == "mapped":
        a.tofile(tmp_path / "a")
        a = np.memmap(tmp_path / "a", np.float32, "r")
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        t = staging.to_device(a, DEV)
        u = densify._dev(a.reshape(1, -1))
    t += 1
    assert np.array_equal(u.cpu().numpy()[0], want) and np.array_equal(a, want)
    assert np.array_equal((t - u[0]).cpu().numpy(), (want + np.float32(1)) - want)


def test_without_pinned_memory_the_plain_copy_runs(monkeypatch):
    from py_ortho_b200 import staging
    a = np.random.default_rng(0).normal(0, 1, 5_000_001).astype(np.float32)
    empty, refused = torch.empty, []

    def pageable(*args, **kw):
        if kw.get("pin_memory"):
            refused.append(1)
            raise RuntimeError("CUDA error: out of memory")
        return empty(*args, **kw)
    monkeypatch.setattr(torch, "empty", pageable)
    t = staging.to_device(a, DEV)
    back = staging.to_host(t)
    assert len(refused) == 2 and np.array_equal(back, a)
