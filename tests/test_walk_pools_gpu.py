"""Full pools of k_walk, one kernel per kind of solve, bit for bit.

A launch of more than about 4e5 packets gives every warp of the GPU a full
pool and refills it: flights are put back and taken by other lanes, slots are
used again after a birth, interactions come in whole batches.  What a lane
writes to the lists and to the pool is read by other lanes of its warp, in
every kind of walk (with an image, without, with the flux tally, taped,
resumed, the adjoint's two replays).  Each is compared here, at that size,
with a route that has no such pools: the single-kernel walk of
kp_transport_forward_noalloc, one solve for the resumed calls, and for the
gradients the same adjoint in chunks of a few packets per warp.  int64
tallies, counters and records: no tolerance."""
import dataclasses

import numpy as np
import pytest
import torch

from kratos_polrad_b200 import _lib
from kratos_polrad_b200.adjoint import adjoint
from kratos_polrad_b200.transport import Tallies, forward, forward_resume
from test_zz_no_alloc import _noalloc
from transport_cases import case

pytestmark = pytest.mark.gpu

N = 400_003


def _solve_case(name, **changes):
    mesh, sig, t = case(name)
    mesh.set_sigma(sig)
    return mesh, dataclasses.replace(t, **{**dict(n_packets=N, n_record=5000, flux=True,
                                                  flux_fx_shift=24), **changes})


def _same(got, want):
    torch.cuda.synchronize()
    for k in ("mu", "image", "image_batch", "counters", "flux"):
        a, b = getattr(got, k), getattr(want, k)
        if b is not None:
            assert torch.equal(a, b), k
    if got.records is None:
        return
    a, b = got.record_array(), want.record_array()
    for f in a.dtype.names:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)


def _single_kernel(mesh, t):
    want = Tallies(t, n_cells=mesh.n_cells)
    _noalloc(mesh, t, want, torch.cuda.current_stream().cuda_stream)
    return want


@pytest.mark.parametrize("flux", [False, True])
@pytest.mark.parametrize("name", ["slab", "amr_point", "hg_multi"])
def test_full_pools(name, flux):
    mesh, t = _solve_case(name, flux=flux)
    want = _single_kernel(mesh, t)
    _same(forward(mesh, t), want)
    if t.image_n:
        _same(forward(mesh, t, tape=True), want)
    assert mesh.status() == 0


@pytest.mark.parametrize("name,budget", [("slab", 23), ("amr_point", 40), ("hg_multi", 40)])
def test_full_pools_resumed(name, budget):
    mesh, t = _solve_case(name, max_steps=300)
    want = _single_kernel(mesh, t)
    tal, left = forward_resume(mesh, t, budget)
    assert left.shape[0] > N // 10
    rest = dataclasses.replace(t, n_packets=0)
    while left.shape[0] > 0:
        tal, left = forward_resume(mesh, rest, budget, resumed=left.clone(), tallies=tal)
    _same(tal, want)
    assert mesh.status() == 0


@pytest.mark.parametrize("name", ["amr_point", "hg_multi"])
def test_full_pools_gradients(name):
    """One chunk of the whole launch (both replays with full pools), the tape of
    one solve (the second replay), and chunks of 2^16 / 12 packets."""
    mesh, t = _solve_case(name, n_record=0, flux=False)
    a = torch.tensor(np.random.default_rng(3).normal(size=(t.image_n, t.image_n, 4)).astype(np.float32),
                     device="cuda")
    taped = forward(mesh, t, tape=True)
    assert taped.tape_id > 0
    tape = adjoint(mesh, t, a, 24, tape_id=taped.tape_id)
    whole = adjoint(mesh, t, a, 24)
    _lib.call("kp_mesh_peel_queue_limit", mesh.handle, 1 << 16)
    small = adjoint(mesh, t, a, 24)
    torch.cuda.synchronize()
    assert mesh.status() == 0
    for x, y, z in zip(tape, whole, small):
        assert z.abs().sum() > 0
        assert torch.equal(x, z) and torch.equal(y, z)


@pytest.mark.parametrize("n", [95_003, 120_001, 186_000])
@pytest.mark.parametrize("name", ["slab", "amr_point"])
def test_pools_of_no_whole_batch(name, n):
    """Pools of 33 to 63 packets: a whole batch and a part of one are born at
    the start."""
    mesh, t = _solve_case(name, n_packets=n, max_scatter=30)
    _same(forward(mesh, t), _single_kernel(mesh, t))
    assert mesh.status() == 0


def test_pools_of_concurrent_solves():
    """Solves of different meshes in flight on several streams, and from several
    threads, have pools of their own; one mesh after another on a stream shares
    one.  Each as alone."""
    import threading
    made = [_solve_case(name, n_packets=n, n_record=0, flux=False, seed=k)
            for k, (name, n) in enumerate([("slab", 200_000), ("amr_point", 30_000), ("hg_multi", 50_000)] * 3)]
    want = [_single_kernel(mesh, t) for mesh, t in made]
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    got = [Tallies(t) for _, t in made]
    torch.cuda.synchronize()
    for k, (mesh, t) in enumerate(made):
        forward(mesh, t, got[k], stream=streams[k % 3].cuda_stream)
    for g, w in zip(got, want):
        _same(g, w)
    got = [[Tallies(t) for _ in range(5)] for _, t in made]
    torch.cuda.synchronize()

    def work(j):
        for r in range(5):
            for k in range(j, len(made), 3):
                forward(made[k][0], made[k][1], got[k][r], stream=streams[j].cuda_stream)

    threads = [threading.Thread(target=work, args=(j,)) for j in range(3)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for k, w in enumerate(want):
        for g in got[k]:
            _same(g, w)
    for mesh, _ in made:
        assert mesh.status() == 0
