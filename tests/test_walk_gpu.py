"""The pooled walk (k_walk) against the single-kernel walk of
kp_transport_forward_noalloc, which the oracle pins on small runs: int64
tallies and counters equal, no tolerance.  Packet counts around a warp, and
enough to fill and refill every warp's pool; scheduling batches of every
kind, which must not matter; segment and interaction limits; and a captured
solve, which has to make do with the pool of an earlier, smaller one."""
import dataclasses

import pytest
import torch

from kratos_polrad_b200 import _lib
from kratos_polrad_b200.transport import PHASE_HG_POL, TALLY_FLOAT, Tallies, forward
from test_zz_no_alloc import _noalloc
from transport_cases import case

pytestmark = pytest.mark.gpu

NAMES = ("mu", "image", "image_batch", "counters", "flux")


def _pair(name, **changes):
    mesh, sig, t = case(name)
    t = dataclasses.replace(t, n_record=0, **changes)
    mesh.set_sigma(sig)
    s = torch.cuda.current_stream().cuda_stream
    want = Tallies(t, n_cells=mesh.n_cells)
    _noalloc(mesh, t, want, s)
    return mesh, t, want


def _equal(got, want):
    torch.cuda.synchronize()
    for k in NAMES:
        a, b = getattr(got, k), getattr(want, k)
        if b is not None:
            assert torch.equal(a, b), k


@pytest.mark.parametrize("n", [1, 31, 33, 4097, 700_001])
@pytest.mark.parametrize("name", ["slab", "amr_point", "hg_multi"])
def test_walk_matches_single_kernel(name, n):
    mesh, t, want = _pair(name, n_packets=n, flux=n == 4097)
    got = forward(mesh, t)
    _equal(got, want)
    assert mesh.status() == 0


@pytest.mark.parametrize("lane_batch", [1, 7, 32])
def test_walk_does_not_depend_on_its_batches(lane_batch):
    mesh, t, want = _pair("amr_point", n_packets=400_003, phase=PHASE_HG_POL, hg_g=-0.4, pol_max=0.8)
    _equal(forward(mesh, dataclasses.replace(t, lane_batch=lane_batch)), want)


@pytest.mark.parametrize("limits", [dict(max_steps=1), dict(max_steps=40), dict(max_scatter=1),
                                    dict(max_scatter=3), dict(w_min=0.9)])
def test_walk_limits(limits):
    mesh, t, want = _pair("amr_point", n_packets=20_000, **limits)
    _equal(forward(mesh, t), want)


def test_walk_queue_overflow():
    """Rays that find the queue full are marched by the walk."""
    mesh, t, want = _pair("amr_point", n_packets=30_000)
    _lib.call("kp_mesh_peel_queue_limit", mesh.handle, 40_000)
    _equal(forward(mesh, t), want)


def test_captured_walk_uses_the_pool_there_is():
    mesh, t, want = _pair("slab", n_packets=50_000)
    forward(mesh, dataclasses.replace(t, n_packets=1))       # a pool for one packet
    got = Tallies(t)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        forward(mesh, t, got)
    g.replay()
    _equal(got, want)
    first = case("slab")[0]                                  # captured before any solve
    first.set_sigma(case("slab")[1])
    first.upload()
    again = Tallies(t)
    g2 = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g2):
        forward(first, t, again)
    g2.replay()
    _equal(again, want)


@pytest.mark.parametrize("limit", [dict(), dict(max_steps=40)])
def test_captured_walk_survives_a_larger_solve(limit):
    """A solve captured before the mesh's first one, replayed after a solve
    that outgrew its pool, and captured again at the larger count."""
    mesh, t, want = _pair("slab", n_packets=5_000, **limit)
    big = dataclasses.replace(t, n_packets=700_001)
    got = Tallies(t)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        forward(mesh, t, got)
    want_big = forward(mesh, big)
    g.replay()
    _equal(got, want)
    again = Tallies(big)
    g2 = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g2):
        forward(mesh, big, again)
    forward(mesh, dataclasses.replace(big, n_packets=900_001))
    g2.replay()
    _equal(again, want_big)


@pytest.mark.parametrize("name,n,calls", [("slab", 33, 1), ("amr_point", 50_001, 1), ("hg_multi", 20_000, 3)])
def test_float_flux_is_rounded_once_per_solve(name, n, calls):
    """Float flux with a carry is summed in double and rounded once per call:
    within 2^-24 per call (and the sum of the calls before) of the fixed-point
    sums, plus those sums' half a unit per segment."""
    mesh, sig, t = case(name)
    t = dataclasses.replace(t, n_record=0, n_packets=n, flux=True, flux_fx_shift=30)
    mesh.set_sigma(sig)
    fx = Tallies(t, n_cells=mesh.n_cells)
    tf = dataclasses.replace(t, tally_mode=TALLY_FLOAT)
    fl = Tallies(tf, n_cells=mesh.n_cells)
    for k in range(calls):
        forward(mesh, dataclasses.replace(t, packet_offset=k * n), fx)
        forward(mesh, dataclasses.replace(tf, packet_offset=k * n), fl)
    torch.cuda.synchronize()
    want = fx.flux.double() * fx.flux_scale()
    steps = fx.counts()["steps"]
    assert want.max() > 0
    assert ((fl.flux.double() - want).abs() <= calls * 2.0 ** -24 * want + steps * 2.0 ** -31).all()
