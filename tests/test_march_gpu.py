"""The peel-off march (k_peel) against the C restatement, bit for bit, over
the observers that choose its variants: directions along an axis, in the x-z
plane (no y face is ever crossed) and oblique ones of every sign, on a
periodic three-level mesh with unequal spacings and on a plain AMR box, with
packet counts around a warp's and a block's."""
import dataclasses

import numpy as np
import pytest
import torch

from kratos_polrad_b200.transport import TALLY_FLOAT, forward
from oracle import port
from transport_cases import case, run_oracle, to_device

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not port.available(), reason="oracle not built")]

OBSERVERS = [(0.0, 0.0), (180.0, 0.0), (90.0, 0.0), (47.0, 0.0), (133.0, 0.0), (90.0, 90.0),
             (70.0, 200.0), (110.0, 340.0), (35.0, 120.0)]


@pytest.mark.parametrize("inclination,azimuth", OBSERVERS)
@pytest.mark.parametrize("name,n", [("hg_multi", 257), ("amr_point", 31), ("table", 1000)])
def test_march_matches_oracle(name, n, inclination, azimuth):
    mesh, sig, t = case(name)
    t = dataclasses.replace(t, n_packets=n, n_record=0, inclination_deg=inclination,
                            azimuth_deg=azimuth)
    mesh.set_sigma(sig)
    tal = forward(mesh, to_device(t))
    torch.cuda.synchronize()
    assert mesh.status() == 0
    ref = run_oracle(mesh, sig, t)
    np.testing.assert_array_equal(tal.counters.cpu().numpy(), ref["counters"].astype(np.int64))
    np.testing.assert_array_equal(tal.image.cpu().numpy(), ref["image"])
    np.testing.assert_array_equal(tal.image_batch.cpu().numpy(), ref["image_batch"])


@pytest.mark.parametrize("azimuth", [0.0, 75.0])
def test_march_circular_light(azimuth):
    """Packets that start circularly polarized: V is deposited (light that
    starts without V keeps V = 0, and a zero is not added), in both tally
    modes; float sums within 1e-6 of each entry's I plus the fixed point's
    rounding of at most one half unit per deposit."""
    mesh, sig, t = case("table")
    table = t.packets.copy()
    table["stokes"][:, 2] = np.where(np.arange(len(table)) % 3 == 0, 0.5, -0.25)
    t = dataclasses.replace(t, packets=table, azimuth_deg=azimuth, n_record=0)
    mesh.set_sigma(sig)
    tal = forward(mesh, to_device(t))
    fl = forward(mesh, to_device(dataclasses.replace(t, tally_mode=TALLY_FLOAT)))
    torch.cuda.synchronize()
    ref = run_oracle(mesh, sig, t)
    assert (ref["image"][..., 3] != 0).sum() > 20
    np.testing.assert_array_equal(tal.image.cpu().numpy(), ref["image"])
    np.testing.assert_array_equal(tal.image_batch.cpu().numpy(), ref["image_batch"])
    a = fl.image.cpu().numpy().astype(np.float64)
    b = ref["image"] * 2.0 ** -t.fx_shift
    n_dep = int(ref["counters"][9])
    assert (np.abs(a - b) <= 1e-6 * np.abs(b[..., :1]) + n_dep * 2.0 ** -(t.fx_shift + 1)).all()


@pytest.mark.parametrize("inclination,azimuth", [(60.0, 0.0), (70.0, 200.0)])
def test_march_float_source_pixel(inclination, azimuth):
    """Float tallies at the pixel of a source, where a large share of all rays
    ends: within the final rounding (2^-24) and the carry's own (batches of up
    to 32 rays are one addition: below 2e-7 at this count) of the fixed-point
    sums, plus those sums' rounding of half a unit per deposit."""
    mesh, sig, t = case("amr_point")
    t = dataclasses.replace(t, n_packets=100_001, n_record=0, inclination_deg=inclination,
                            azimuth_deg=azimuth)
    mesh.set_sigma(sig)
    fx = forward(mesh, to_device(t))
    fl = forward(mesh, to_device(dataclasses.replace(t, tally_mode=TALLY_FLOAT)))
    torch.cuda.synchronize()
    b = fx.image.cpu().numpy() * 2.0 ** -t.fx_shift
    a = fl.image.cpu().numpy().astype(np.float64)
    n_dep = int(fx.counters.cpu().numpy()[9])
    assert (np.abs(a - b) <= 3e-7 * np.abs(b[..., :1]) + n_dep * 2.0 ** -(t.fx_shift + 1)).all()


@pytest.mark.parametrize("n", [499_999, 500_000])
def test_march_order_by_packet_count(n):
    """On a mesh of 12 to 32 MB of extinction the order is chosen by the packet
    count: the same int64 tallies as marched as queued, on either side."""
    from kratos_polrad_b200.mesh import Mesh, MeshConfig, PEEL_ORDER_QUEUE
    mesh = Mesh(MeshConfig((0, 0, 0), (1, 1, 1), (160,) * 3, (16,) * 3, (False,) * 3))
    sig = np.empty((mesh.n_cells, 2), np.float32)
    sig[:, 0], sig[:, 1] = 3.0, 0.5
    mesh.set_sigma(sig)
    _, _, t = case("amr_point")
    t = dataclasses.replace(t, n_packets=n, n_record=0, fx_shift=30)
    got = forward(mesh, t)
    mesh.set_peel_order(PEEL_ORDER_QUEUE)
    want = forward(mesh, t)
    torch.cuda.synchronize()
    assert mesh.status() == 0 and want.image.abs().sum() > 0
    assert torch.equal(got.image, want.image) and torch.equal(got.image_batch, want.image_batch)
    assert torch.equal(got.counters, want.counters)
