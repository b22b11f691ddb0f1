"""Pools that are partly empty (kp_trace): the packets to keep, wherever they lie,
walk as they do in a pool of their own, and the other slots stay as they are.
int64 flux and states: no tolerance."""
import numpy as np
import pytest
import torch

from kratos_polrad_b200 import Mesh, PacketPool, trace
from kratos_polrad_b200.walk import TO_KEEP, TO_RM
from meshcases import CASES

pytestmark = pytest.mark.gpu

LIVE = {"front": lambda k, n: k < n // 9, "back": lambda k, n: k >= n - 7, "every": lambda k, n: k % 13 == 5,
        "none": lambda k, n: k < 0, "all": lambda k, n: k >= 0}


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("live", sorted(LIVE))
@pytest.mark.parametrize("n", [5, 3_001, 57_000, 130_003])
def test_partly_live_pool(n, live, precision):
    dt = torch.float32 if precision == 4 else torch.float64
    mesh = Mesh(next(iter(CASES.values())))
    rng = np.random.default_rng(n)
    lo, hi = np.array(mesh.x_min), np.array(mesh.x_max)
    x = (lo + rng.uniform(0.01, 0.99, (n, 3)) * (hi - lo)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    ib, cell = mesh.locate(x.astype(np.float64))
    steps = np.where(np.arange(n) < n // 3, 200, 3).astype(np.int32)
    keep = LIVE[live](np.arange(n), n)
    T = lambda a, t=None: torch.tensor(a, dtype=t, device="cuda")

    def pool(sel, todo):
        return PacketPool(T(x[sel], dt), T(d[sel], dt), T(cell[sel]), T(ib[sel]),
                          torch.ones(len(x[sel]), dtype=dt, device="cuda"), T(steps[sel]), todo)

    mesh.upload()
    part = pool(slice(None), T(np.where(keep, TO_KEEP, TO_RM), torch.int8))
    before = {k: getattr(part, k).clone() for k in ("x", "cell", "ib", "step", "todo")}
    flux = trace(mesh, part, fx_shift=20)
    own = pool(keep, None)
    want = trace(mesh, own, fx_shift=20) if keep.any() else torch.zeros_like(flux)
    torch.cuda.synchronize()
    assert mesh.status() == 0
    assert torch.equal(flux, want) and bool(flux.any()) == bool(keep.any())
    k = T(keep)
    for name, old in before.items():
        got = getattr(part, name)
        assert torch.equal(got[~k], old[~k]), name
        assert torch.equal(got[k], getattr(own, name)), name
