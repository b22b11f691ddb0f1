"""The pool walk (kp_trace) against the C restatement, bit for bit, where its
short cuts end: quotients from reciprocals (scaled meshes, whose cell volumes
leave the reciprocal's range at one end), directions with zero and with tiny
components, packets on faces, budgets that run out, periodic meshes, one-block
meshes that hand off to themselves, and packet counts around a warp."""
import dataclasses

import numpy as np
import pytest
import torch

from kratos_polrad_b200 import Mesh, PacketPool, trace
from kratos_polrad_b200.mesh import MeshConfig, RefineRegion
from meshcases import AMR_PERIODIC, CASES
from oracle import port

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not port.available(), reason="oracle not built")]

ONE_BLOCK = MeshConfig((0, 0, 0), (1, 1, 1), (8, 8, 8), (8, 8, 8), (True, False, True))
MESHES = dict(CASES, one_block=ONE_BLOCK)


def _scaled(cfg, s):
    t = lambda v: tuple(s * float(a) for a in v)
    return dataclasses.replace(cfg, x_min=t(cfg.x_min), x_max=t(cfg.x_max),
                               refine=[RefineRegion(r.level, t(r.x_min), t(r.x_max))
                                       for r in cfg.refine])


def _packets(mesh, n, ftype, seed, tiny):
    rng = np.random.default_rng(seed)
    lo, hi = np.array(mesh.x_min), np.array(mesh.x_max)
    x = (lo + rng.random((n, 3)) * (hi - lo)).astype(ftype)
    x = np.minimum(x, np.nextafter(hi.astype(ftype), lo.astype(ftype)))
    d = rng.normal(size=(n, 3))
    k = np.arange(n)
    d[k % 7 == 0, 0] = 0.0
    d[k % 11 == 0, 2] = 0.0
    d[k % 17 == 1] *= [1.0, 1e-3, 1e-4]
    if tiny:                                          # beyond the reciprocals' range
        d[k % 3 == 1, 1] = 1e-25 if ftype == np.float32 else 1e-150
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    ib, cell = mesh.locate(x.astype(np.float64))
    xf0, dx0, _, _ = mesh.geometry(4 if ftype == np.float32 else 8)
    on = k % 5 == 0                                   # on the cell's lower y face
    x[on, 1] = (xf0[ib, 1] + cell[:, 1] * dx0[ib, 1]).astype(ftype)[on]
    ib, cell = mesh.locate(x.astype(np.float64))
    steps = np.where(k % 3 == 0, rng.integers(0, 30, n), 2000).astype(np.int32)
    return x, d.astype(ftype), cell, ib, (rng.random(n) + 0.5).astype(ftype), steps


def _check(cfg, precision, n, seed, shift=8, tiny=False, weight=1.0):
    ftype, tdt = (np.float32, torch.float32) if precision == 4 else (np.float64, torch.float64)
    mesh = Mesh(cfg)
    x, d, cell, ib, w, steps = _packets(mesh, n, ftype, seed, tiny)
    w *= ftype(weight)
    o = port.trace(port.Tables.from_mesh(mesh, precision), precision, x, d, cell, ib, w, steps,
                   fx_shift=shift)
    T = lambda a, dt=None: torch.tensor(a, dtype=dt, device="cuda")
    pool = PacketPool(T(x, tdt), T(d, tdt), T(cell), T(ib), T(w, tdt), T(steps))
    flux = trace(mesh, pool, "fixed", shift)
    torch.cuda.synchronize()
    assert mesh.status() == 0
    np.testing.assert_array_equal(pool.x.cpu().numpy().astype(np.float64), o["x"])
    np.testing.assert_array_equal(pool.cell.cpu().numpy(), o["cell"])
    np.testing.assert_array_equal(pool.ib.cpu().numpy(), o["ib"])
    np.testing.assert_array_equal(pool.step.cpu().numpy(), o["step"])
    np.testing.assert_array_equal(pool.todo.cpu().numpy().astype(np.int32), o["todo"])
    if not tiny:          # (a tiny component's distances overflow the int64 deposit, which
        #                    C's conversion leaves undefined: states only)
        assert np.abs(o["flux_fx"]).max() < 2 ** 62
        np.testing.assert_array_equal(flux.cpu().numpy(), o["flux_fx"])


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("name", sorted(MESHES))
@pytest.mark.parametrize("n", [1, 33, 6007])
def test_trace_matches_restatement(name, precision, n):
    _check(MESHES[name], precision, n, seed=n + precision)


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("name", ["amr_box", "amr_periodic"])
def test_trace_tiny_directions(name, precision):
    _check(MESHES[name], precision, 1001, seed=3, tiny=True)


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("log2,shift,weight", [(-23, 0, 2.0 ** -24), (12, 40, 1.0), (25, 60, 1.0)])
def test_trace_scaled_meshes(log2, shift, weight, precision):
    """Cell volumes of 2^-84 (float: beyond the reciprocal's range, so every
    quotient by the volume is a division) to 2^60."""
    _check(_scaled(AMR_PERIODIC, 2.0 ** log2), precision, 2003, seed=5, shift=shift, weight=weight)
