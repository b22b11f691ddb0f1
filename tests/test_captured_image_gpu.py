"""Captured solves with an image and captured gradients, replayed after larger
solves of the same mesh: the queue, the march order and the adjoint's buffers
that the capture was given are still theirs.  int64 tallies: no tolerance."""
import dataclasses

import numpy as np
import pytest
import torch

from kratos_polrad_b200.adjoint import adjoint
from kratos_polrad_b200.mesh import PEEL_ORDER_AUTO, PEEL_ORDER_CELL
from kratos_polrad_b200.transport import TALLY_FLOAT, Tallies, forward
from transport_cases import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [PEEL_ORDER_AUTO, PEEL_ORDER_CELL])
def test_captured_image_survives_a_larger_solve(order):
    mesh, sig, t = case("amr_point")
    mesh.set_sigma(sig)
    mesh.set_peel_order(order)
    t = dataclasses.replace(t, n_packets=6_000, n_record=0)
    want = forward(mesh, t)                          # the queue, before the capture
    got = Tallies(t)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        forward(mesh, t, got)
    for n in (50_000, 300_000):
        forward(mesh, dataclasses.replace(t, n_packets=n))
    fill = torch.full((1 << 28,), 255, dtype=torch.uint8, device="cuda")   # where freed memory would be
    g.replay()
    torch.cuda.synchronize()
    assert mesh.status() == 0 and fill[-1] == 255
    for k in ("mu", "image", "image_batch", "counters"):
        assert torch.equal(getattr(got, k), getattr(want, k)), k


def test_captured_gradient_survives_a_larger_one():
    mesh, sig, t = case("amr_point")
    mesh.set_sigma(sig)
    t = dataclasses.replace(t, n_packets=6_000, n_record=0)
    a = torch.tensor(np.random.default_rng(5).normal(size=(t.image_n, t.image_n, 4)).astype(np.float32),
                     device="cuda")
    want = adjoint(mesh, t, a, 24)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = adjoint(mesh, t, a, 24)
    adjoint(mesh, dataclasses.replace(t, n_packets=300_000), a, 24)
    g.replay()
    torch.cuda.synchronize()
    assert mesh.status() == 0
    for x, y in zip(got, want):
        assert y.abs().sum() > 0 and torch.equal(x, y)


def test_captured_float_flux_before_any_other():
    """The mesh's first float flux, captured and replayed twice: summed in
    double and rounded once per replay, so within 2 * 2^-24 of the fixed-point
    sums, plus those sums' half a unit per segment."""
    mesh, sig, t = case("slab")
    mesh.set_sigma(sig)
    t = dataclasses.replace(t, n_packets=20_000, n_record=0, flux=True, flux_fx_shift=30)
    fx = Tallies(t, n_cells=mesh.n_cells)
    forward(mesh, t, fx)
    forward(mesh, t, fx)
    tf = dataclasses.replace(t, tally_mode=TALLY_FLOAT)
    fl = Tallies(tf, n_cells=mesh.n_cells)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        forward(mesh, tf, fl)
    g.replay()
    g.replay()
    torch.cuda.synchronize()
    assert mesh.status() == 0
    want = fx.flux.double() * fx.flux_scale()
    steps = fx.counts()["steps"]
    assert want.max() > 0
    assert ((fl.flux.double() - want).abs() <= 2 * 2.0 ** -24 * want + steps * 2.0 ** -31).all()
