"""The work that a user of this package has it do, as cases to be timed.

Each case names one path through the public entry points and its sizes:

``image``     a solve with a peel-off image (transport.forward) of a dense clump
              on a 2-level AMR mesh: what an observer's picture of a dusty or
              ionised cloud costs, from a quick look of a few thousand packets
              to the full picture of 1e7; with the per-cell path-length flux
              and with float tallies in some
``escape``    a solve without an image: a plane-parallel scattering atmosphere,
              periodic in x and y, escaping Stokes vectors per mu bin
``sources``   a turbulent cloud on a 3-level mesh larger than L2 holds, many
              sources, anisotropic (Henyey-Greenstein) scattering, image
``gradient``  one step of a fit of the coefficients to an observed image:
              TransportImage.apply, a loss on Q and U, its gradients
``resume``    packets with a step budget per call, carried from call to call
              until none is left (a time step of a coupled simulation)
``batch``     many independent small scenes in one launch (a parameter study)
``trace``     the straight walk that fills rad_t::flx, in float or double, on
              a uniform or a refined mesh
``trace_sph`` the same walk on a spherical-polar mesh

Sizes come from scenes.py, the tests and the benchmark's workloads.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from kratos_polrad_b200 import Mesh, PacketPool, problems, scenes, trace
from kratos_polrad_b200.adjoint import TransportImage
from kratos_polrad_b200.batch import Batch
from kratos_polrad_b200.mesh import MeshConfig, RefineRegion
from kratos_polrad_b200.transport import (EMIT_ISOTROPIC, EMIT_UP_UNIFORM, PHASE_HG_POL,
                                          PHASE_RAYLEIGH, SOURCE_PLANE_BASE, SOURCE_POINT,
                                          TALLY_FIXED, TALLY_FLOAT, Source, TransportConfig,
                                          forward, forward_resume)
from kratos_polrad_b200.walk import trace_sph

TWO_PI = 2.0 * math.pi


def listed():
    return [
        # a first look at a set-up: the smallest solve that is made in earnest
        dict(name="image_2k", path="image", root=64, packets=2000, pixels=64, inclination=60.0,
             azimuth=0.0, tally="fixed", flux=False),
        # an interactive picture from an oblique direction, odd sizes
        dict(name="image_300k", path="image", root=96, packets=300007, pixels=100,
             inclination=52.5, azimuth=25.0, tally="fixed", flux=False),
        # the benchmark's picture
        dict(name="image_10m", path="image", root=128, packets=10_000_000, pixels=128,
             inclination=90.0, azimuth=0.0, tally="fixed", flux=False),
        # picture and radiation field of a coupled run, float tallies
        dict(name="image_flux_float_1m", path="image", root=128, packets=1_000_000, pixels=128,
             inclination=60.0, azimuth=0.0, tally="float", flux=True),
        # the scattering atmosphere of the analytic check
        dict(name="escape_1m", path="escape", nx=128, nz=64, tau=10.0, packets=1_000_000, mu=20),
        # the large scene at a picture's packet count
        dict(name="sources_2m", path="sources", root=256, cells=20_000_000, sources=64,
             packets=2_000_000, pixels=256, inclination=60.0, azimuth=0.0),
        # one step of the fit of a 96^3 field
        dict(name="gradient_1m", path="gradient", side=96, packets=1_000_000, pixels=64,
             inclination=60.0, azimuth=0.0, hg=False),
        # a small fit with anisotropic scattering seen obliquely, odd sizes
        dict(name="gradient_40k", path="gradient", side=48, packets=40_009, pixels=37,
             inclination=75.0, azimuth=140.0, hg=True),
        # a coupled run's transport with 256 segments per packet and step
        dict(name="resume_1m", path="resume", root=128, packets=1_000_000, budget=256,
             pixels=128),
        # a parameter study
        dict(name="batch_64", path="batch", scenes=64, packets=60_000),
        # the reference's flux walk, single precision, order-independent flux
        dict(name="trace_f32_2m", path="trace", mesh="clump", side=128, packets=1 << 21,
             precision=4, flux="fixed"),
        # ... and on a uniform mesh in double with float atomics, odd count
        dict(name="trace_f64_300k", path="trace", mesh="uniform", side=64, packets=300_001,
             precision=8, flux="float"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["image"] * 5 + ["escape"] * 2 + ["sources", "gradient", "gradient",
                                                         "resume", "batch", "trace", "trace",
                                                         "trace_sph"])
    view = dict(inclination=rng.choice([90.0, 60.0, rng.uniform(5.0, 175.0)]),
                azimuth=0.0 if rng.random() < 0.5 else rng.uniform(0.0, 360.0))
    if path == "image":
        return dict(path=path, root=16 * rng.randint(3, 8), packets=_log_int(rng, 1000, 5_000_000),
                    pixels=rng.randint(16, 256), tally=rng.choice(["fixed"] * 3 + ["float"]),
                    flux=rng.random() < 0.25, **view)
    if path == "escape":
        return dict(path=path, nx=16 * rng.randint(2, 8), nz=16 * rng.randint(2, 6),
                    tau=round(rng.uniform(0.5, 12.0), 3), packets=_log_int(rng, 1000, 1_500_000),
                    mu=rng.randint(8, 40))
    if path == "sources":
        return dict(path=path, root=128, cells=_log_int(rng, 4_000_000, 12_000_000),
                    sources=rng.randint(1, 64), packets=_log_int(rng, 20_000, 2_000_000),
                    pixels=rng.randint(64, 256), **view)
    if path == "gradient":
        return dict(path=path, side=16 * rng.randint(2, 6), packets=_log_int(rng, 2000, 1_000_000),
                    pixels=rng.randint(16, 96), hg=rng.random() < 0.5, **view)
    if path == "resume":
        return dict(path=path, root=16 * rng.randint(3, 8), packets=_log_int(rng, 2000, 1_000_000),
                    budget=_log_int(rng, 48, 512), pixels=rng.randint(16, 128))
    if path == "batch":
        return dict(path=path, scenes=rng.randint(4, 64), packets=_log_int(rng, 2000, 60_000))
    if path == "trace":
        return dict(path=path, mesh=rng.choice(["uniform", "clump"]), side=16 * rng.randint(3, 8),
                    packets=_log_int(rng, 1000, 1 << 21), precision=rng.choice([4, 8]),
                    flux=rng.choice(["fixed", "float"]))
    return dict(path=path, side=16 * rng.randint(2, 4), packets=_log_int(rng, 1000, 1 << 20),
                precision=rng.choice([4, 8]))


# ---- what the user's program has in hand -----------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _centres(mesh):
    """Cell centres [n_blocks, nz, ny, nx, 3] on the GPU, in cell order."""
    xf0, dx0, _, _ = mesh.geometry(8)
    xf0, dx0 = (torch.from_numpy(a).cuda() for a in (xf0, dx0))
    ax = [xf0[:, a, None] + (torch.arange(mesh.nc[a], device="cuda", dtype=torch.float64) + 0.5)
          * dx0[:, a, None] for a in range(3)]
    shape = (mesh.n_blocks, mesh.nc[2], mesh.nc[1], mesh.nc[0])
    return torch.stack([ax[0][:, None, None, :].expand(shape), ax[1][:, None, :, None].expand(shape),
                        ax[2][:, :, None, None].expand(shape)], -1)


def _lognormal(n, sigma_ln, seed):
    """The density of scenes.lognormal_field, made on the GPU."""
    w = torch.randn((n, n, n), generator=_gen(seed), device="cuda")
    k = torch.fft.fftfreq(n, device="cuda") * n
    kr = torch.fft.rfftfreq(n, device="cuda") * n
    K = torch.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2)
    amp = torch.where(K > 0, K, torch.ones_like(K)) ** (-11.0 / 6.0)
    amp[0, 0, 0] = 0.0
    g = torch.fft.irfftn(torch.fft.rfftn(w) * amp, s=(n, n, n))
    rho = torch.exp(sigma_ln * (g - g.mean()) / g.std())
    return rho / rho.mean()


def _sampled(rho, centres):
    n = rho.shape[0]
    i = (centres * n).long().clamp_(0, n - 1)
    return rho[i[..., 2], i[..., 1], i[..., 0]].reshape(-1)


def _clump(case, seed):
    """The 2-level clump of problems.clump_spec, its coefficients made on the GPU."""
    mesh = Mesh(problems.clump_mesh_config(case["root"]))
    _, _, cfg = problems.clump_spec(case["packets"], seed=seed, image_n=case["pixels"])
    s = 0.1 / (2.0 * math.sqrt(2.0 * math.log(2.0)))
    col = 0.5 + 99.0 * s * math.sqrt(math.pi / 2) * math.erf(0.5 / (s * math.sqrt(2)))
    r2 = ((_centres(mesh) - 0.5) ** 2).sum(-1).reshape(-1)
    ext = (5.0 / col) * (1.0 + 99.0 * torch.exp(-r2 / (2 * s * s)))
    u = torch.rand(mesh.n_cells, generator=_gen(seed), device="cuda", dtype=torch.float64)
    alb = torch.exp(math.log(0.5) + u * (math.log(0.99) - math.log(0.5)))
    mesh.set_sigma(torch.stack([ext * alb, ext * (1.0 - alb)], 1).float().contiguous())
    return mesh, cfg


def _cloud(case, seed):
    """The many-source scene of scenes.large_amr, its density made on the GPU."""
    n, block = case["root"], 16
    rho = _lognormal(n, 1.5, seed)
    nb = n // block
    bmax = rho.reshape(nb, block, nb, block, nb, block).amax(dim=(1, 3, 5)).cpu().numpy()
    order = np.sort(bmax.ravel())[::-1]
    extra = max(0, case["cells"] // block ** 3 - nb ** 3)
    n1 = min(len(order) // 4, max(1, int(extra / 7 * 0.7)))
    n2 = min(max(1, int(extra / 49 * 0.3)), n1 // 2)
    boxes = []
    for level, count in ((1, n1), (2, n2)):
        for kz, ky, kx in zip(*np.nonzero(bmax >= order[max(count, 1) - 1])):
            k = np.array([kx, ky, kz])
            boxes.append(RefineRegion(level, tuple((k + 0.25) / nb), tuple((k + 0.75) / nb)))
    mesh = Mesh(MeshConfig((0, 0, 0), (1, 1, 1), (n,) * 3, (block,) * 3, (False,) * 3, boxes))
    ext = 4.0 * _sampled(rho, _centres(mesh))
    mesh.set_sigma(torch.stack([0.9 * ext, 0.1 * ext], 1).float().contiguous())
    pos = np.random.default_rng(seed).uniform(0.05, 0.95, (case["sources"], 3))
    cfg = TransportConfig(n_packets=case["packets"], seed=seed,
                          sources=[Source(SOURCE_POINT, EMIT_ISOTROPIC, tuple(p)) for p in pos],
                          phase=PHASE_HG_POL, hg_g=0.6, pol_max=0.5, image_n=case["pixels"],
                          inclination_deg=case["inclination"], azimuth_deg=case["azimuth"],
                          image_center=(0.5, 0.5, 0.5), image_half_width=0.75, image_batch_n=64,
                          n_batches=32, w_min=0.01, fx_shift=30)
    return mesh, cfg


def _fit(case, seed):
    """A field to be fitted: the coefficients in hand and the image of the
    field perturbed by 5 %, the target."""
    n = case["side"]
    mesh = Mesh(MeshConfig((0, 0, 0), (1, 1, 1), (n,) * 3, (16,) * 3, (False,) * 3))
    rho = _sampled(_lognormal(n, 1.0, seed), _centres(mesh))
    phase = dict(phase=PHASE_HG_POL, hg_g=0.6, pol_max=0.5) if case["hg"] else \
        dict(phase=PHASE_RAYLEIGH)
    cfg = TransportConfig(n_packets=case["packets"], seed=seed,
                          sources=[Source(SOURCE_POINT, EMIT_ISOTROPIC, (0.5, 0.5, 0.5))],
                          image_n=case["pixels"], inclination_deg=case["inclination"],
                          azimuth_deg=case["azimuth"], image_center=(0.5, 0.5, 0.5),
                          image_half_width=0.75, image_batch_n=8, n_batches=32, w_min=0.01,
                          fx_shift=32, **phase)
    noise = 1.0 + 0.05 * torch.randn(mesh.n_cells, generator=_gen(seed + 1), device="cuda")
    other = 4.0 * rho * noise.clamp_min(0.1)
    mesh.set_sigma(torch.stack([0.9 * other, 0.1 * other], 1).contiguous())
    tal = forward(mesh, cfg)
    target = tal.image.double() * (tal.scale() / cfg.n_packets)
    ext = 4.0 * rho
    return dict(mesh=mesh, cfg=cfg, target=target, sca=(0.9 * ext).requires_grad_(),
                abs=(0.1 * ext).requires_grad_())


def _trace_start(case, seed):
    """Positions in the unit box, directions and weights of a trace, in float_t."""
    g, n = _gen(seed), case["packets"]
    dt = torch.float32 if case["precision"] == 4 else torch.float64
    x = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64).to(dt)
    d = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    d = (d / d.norm(dim=1, keepdim=True)).to(dt)
    w = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) + 0.5).to(dt)
    return x.clamp_(max=1.0 - 1e-6), d, w


def _sph_config(side):
    return MeshConfig((0.5, 0.4, 0.0), (2.5, 2.7, TWO_PI), (side, side, 2 * side), (16, 16, 16),
                      (False, False, True), [RefineRegion(1, (1.0, 1.0, 2.0), (1.6, 1.8, 3.6)),
                                             RefineRegion(2, (1.1, 1.2, 2.5), (1.3, 1.4, 3.0))])


def _located(mesh, x, **start):
    ib, cell = mesh.locate(x.double().cpu().numpy())
    return dict(mesh=mesh, x=x, ib=torch.from_numpy(ib).cuda(), cell=torch.from_numpy(cell).cuda(),
                step=torch.full((len(x),), 4096, dtype=torch.int32, device="cuda"), **start)


def prepare(case, seed):
    path = case["path"]
    if path == "image":
        mesh, cfg = _clump(case, seed)
        cfg = dataclasses.replace(cfg, inclination_deg=case["inclination"],
                                  azimuth_deg=case["azimuth"], flux=case["flux"],
                                  tally_mode=TALLY_FLOAT if case["tally"] == "float" else TALLY_FIXED)
        return dict(path=path, mesh=mesh, cfg=cfg)
    if path == "escape":
        nx, nz = case["nx"], case["nz"]
        mesh = Mesh(MeshConfig((0, 0, 0), (nx, nx, nz), (nx, nx, nz), (16,) * 3,
                               (True, True, False)))
        # a few per cent of structure on the constant density
        u = torch.rand(mesh.n_cells, generator=_gen(seed), device="cuda")
        sca = case["tau"] / nz * (0.97 + 0.06 * u)
        mesh.set_sigma(torch.stack([sca, torch.zeros_like(sca)], 1).contiguous())
        cfg = TransportConfig(n_packets=case["packets"], seed=seed,
                              sources=[Source(SOURCE_PLANE_BASE, EMIT_UP_UNIFORM)],
                              phase=PHASE_RAYLEIGH, n_mu_bins=case["mu"], mu_lo=0.0, mu_hi=1.0,
                              n_batches=32, fx_shift=24)
        return dict(path=path, mesh=mesh, cfg=cfg)
    if path == "sources":
        mesh, cfg = _cloud(case, seed)
        return dict(path=path, mesh=mesh, cfg=cfg)
    if path == "gradient":
        return dict(path=path, **_fit(case, seed))
    if path == "resume":
        mesh, cfg = _clump(case, seed)
        return dict(path=path, mesh=mesh, cfg=cfg, budget=case["budget"])
    if path == "batch":
        made, cfg = scenes.batched_cubes(case["scenes"], packets=(case["packets"] // 10,
                                                                  case["packets"]), seed=seed)
        for mesh, sigma2, _, _, _ in made:
            mesh.set_sigma(sigma2)
        batch = Batch([(mesh, n, k, source) for mesh, _, n, k, source in made])
        batch.autotune(cfg)
        return dict(path=path, batch=batch, cfg=cfg)
    if path == "trace":
        if case["mesh"] == "clump":
            mesh = Mesh(problems.clump_mesh_config(case["side"]))
        else:
            mesh = Mesh(MeshConfig((0, 0, 0), (1, 1, 1), (case["side"],) * 3, (16,) * 3,
                                   (False,) * 3))
        x, d, w = _trace_start(case, seed)
        mesh.upload()
        return dict(path=path, flux=case["flux"], **_located(mesh, x, d=d, w=w))
    mesh = Mesh(_sph_config(case["side"]), spherical=True, r_ratio=1.0)
    u, d, w = _trace_start(case, seed)
    lo = torch.tensor([0.52, 0.515, 0.0], device="cuda", dtype=u.dtype)
    span = torch.tensor([1.96, 2.07, TWO_PI], device="cuda", dtype=u.dtype)
    x = lo + u * span
    st = torch.sin(x[:, 1])
    xc = torch.stack([x[:, 0] * st * torch.cos(x[:, 2]), x[:, 0] * st * torch.sin(x[:, 2]),
                      x[:, 0] * torch.cos(x[:, 1])], 1).contiguous()
    mesh.upload()
    return dict(path=path, xc=xc, **_located(mesh, x, d=d, w=w))


# ---- one pass ----------------------------------------------------------------

def _tallies(t, cfg):
    out = {"counters": t.counters}
    if cfg.image_n:
        out["image"], out["image_batch"] = t.image, t.image_batch
    if cfg.n_mu_bins:
        out["mu"] = t.mu
    if cfg.flux:
        out["flux"] = t.flux
    return out


def run(state):
    path = state["path"]
    if path in ("image", "escape", "sources"):
        return _tallies(forward(state["mesh"], state["cfg"]), state["cfg"])
    if path == "gradient":
        image = TransportImage.apply(state["sca"], state["abs"], state["mesh"], state["cfg"])
        loss = ((image - state["target"])[..., 1:3] ** 2).sum()
        g_sca, g_abs = torch.autograd.grad(loss, (state["sca"], state["abs"]))
        return {"image": image.detach(), "g_sca": g_sca, "g_abs": g_abs}
    if path == "resume":
        mesh, cfg, budget = state["mesh"], state["cfg"], state["budget"]
        tallies, kept = forward_resume(mesh, cfg, budget)
        rest = dataclasses.replace(cfg, n_packets=0)
        while len(kept):
            tallies, kept = forward_resume(mesh, rest, budget, resumed=kept, tallies=tallies)
        return _tallies(tallies, cfg)
    if path == "batch":
        return {"mu": state["batch"].forward(state["cfg"])}
    # the pool is consumed by the walk: the generator's packets are copied into it
    pool = PacketPool(state["x"].clone(), state["d"], state["cell"].clone(), state["ib"].clone(),
                      state["w"], state["step"].clone())
    out = {"x": pool.x, "cell": pool.cell, "ib": pool.ib, "step": pool.step, "todo": pool.todo}
    if path == "trace":
        out["flux"] = trace(state["mesh"], pool, state["flux"])
    else:
        out["xc"] = state["xc"].clone()
        out["flux"] = trace_sph(state["mesh"], pool, out["xc"], fx_shift=16)
    return out


# ---- what a pass cannot do without -------------------------------------------

# Cell segments per packet, averages of the listed scenes at 128 root cells a
# side (they grow with the cells a side), and operations of one: three face
# distances, the optical depth and the move of a walk's segment, one face
# distance and the depth of a segment toward the observer, one interaction.
_WALK, _PEEL, _EVENTS = 165.0, 873.0, 10.0
_WALK_OPS, _PEEL_OPS, _EVENT_OPS = 20.0, 8.0, 300.0


def work(case):
    path, n = case["path"], case["packets"]
    px = 32.0 * case.get("pixels", 0) ** 2
    if path in ("image", "resume"):
        cells = 1.11 * case["root"] ** 3
        per = case["root"] / 128.0
        ops = n * (per * (_WALK * _WALK_OPS + _PEEL * _PEEL_OPS) + _EVENTS * _EVENT_OPS)
        return {"bytes": 8.0 * cells * (2 if case.get("flux") else 1) + px, "flops": ops}
    if path == "escape":
        cells = case["nx"] ** 2 * case["nz"]
        return {"bytes": 8.0 * cells, "flops": n * (2.9 * case["nz"] * _WALK_OPS
                                                   + 1.8 * case["tau"] * _EVENT_OPS)}
    if path == "sources":
        per = case["root"] / 128.0
        return {"bytes": 8.0 * case["cells"] + px,
                "flops": n * (per * (112.0 * _WALK_OPS + 265.0 * _PEEL_OPS) + 2.0 * _EVENT_OPS)}
    if path == "gradient":
        cells, per = case["side"] ** 3, case["side"] / 96.0
        ops = n * (per * (200.0 * _WALK_OPS + 400.0 * _PEEL_OPS) + 6.0 * _EVENT_OPS)
        return {"bytes": 24.0 * cells + px, "flops": 2.0 * ops}
    if path == "batch":
        return {"bytes": case["scenes"] * (8.0 * 51 ** 3 + 32.0 * 32 * 32),
                "flops": case["scenes"] * 0.3 * n * (100.0 * _WALK_OPS + 5.0 * _EVENT_OPS)}
    size = case["precision"]
    packet = 11 * size + 45.0 if path == "trace" else 14 * size + 45.0
    side = case["side"]
    cells = (1.11 if case.get("mesh") == "clump" else 1.0) * side ** 3 * (2 if path == "trace_sph" else 1)
    return {"bytes": n * packet + 8.0 * cells,
            "flops": n * 0.75 * side * (_WALK_OPS if path == "trace" else 120.0)}


# ---- the outputs in 64 bits ----------------------------------------------------

def _uniform_flux(x, d, w, side):
    """w * length / volume per cell of a side^3 grid on the unit box, summed
    over the straight rays from x along d; cells in block order (16^3 blocks,
    x fastest in a block, blocks with z fastest)."""
    flux = torch.zeros(side ** 3, device="cuda", dtype=torch.float64)
    cell = (x * side).long().clamp_(0, side - 1)
    step = torch.where(d > 0, 1, -1)
    nb = side // 16
    for _ in range(3 * side + 3):
        if not len(x):
            break
        face = (cell + (d > 0)).double() / side
        t, axis = torch.where(d != 0, (face - x) / d, torch.full_like(x, 1e300)).min(dim=1)
        t = t.clamp_min(0.0)
        b, c = cell // 16, cell % 16
        flat = ((b[:, 0] * nb + b[:, 1]) * nb + b[:, 2]) * 4096 + c[:, 0] + 16 * (c[:, 1] + 16 * c[:, 2])
        flux.index_add_(0, flat, w * t * side ** 3)
        x = x + t[:, None] * d
        row = torch.arange(len(x), device="cuda")
        cell[row, axis] += step[row, axis]
        inside = ((cell >= 0) & (cell < side)).all(dim=1)
        x, d, w, cell, step = x[inside], d[inside], w[inside], cell[inside], step[inside]
    return flux


def exact(case, seed):
    """The ends of the traces in double (the point where a ray leaves the unit
    box) and their flux on a uniform mesh whose faces are exact in double.
    (In float, and at inexact faces of a block, the reference's walk, which is
    kept bit for bit, steps past a face that rounding put behind it.)  The
    other paths are Monte-Carlo sums over random walks, whose 64-bit value is
    not given by a formula."""
    if case["path"] != "trace" or case["precision"] != 8:
        return None
    x, d, w = (v.double() for v in _trace_start(case, seed))
    t = torch.where(d != 0, ((d > 0).double() - x) / d, torch.full_like(x, 1e300)).min(dim=1).values
    out = {k: None for k in ("cell", "ib", "step", "todo", "flux")}
    out["x"] = x + t[:, None] * d
    side = case["side"]
    if case["mesh"] == "uniform" and case["flux"] == "float" and side & (side - 1) == 0:
        out["flux"] = _uniform_flux(x, d, w, case["side"])
    return out
