"""The work that users of this framework have it do, as measurable cases.

A case is one call (or the few calls that belong together) through the public
entry points: ``runtime.run_steps`` on 2D and 3D programs, the gradient of a
design objective through ``adjoint.simulate``, the checks of an automatically
terminated run, and a batch of requests through ``serve.ServingEngine``.
Scenes are generic: oxide with silicon boxes or layers on a 20 nm grid, CPML or
sponge absorbers, a soft dipole pulse at 1.55 um and x-normal DFT monitors, as
in this repository's workloads and benchmark.  Fields are band-limited noise
(about eight cells per wavelength of the finest structure), so that every cell
is live, as in the middle of a run.
"""

from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch
import torch.utils.checkpoint

from beamz_b200 import adjoint, runtime, serve, workloads
from beamz_b200 import plan as P

RES = 20e-9
OXIDE, SILICON = 2.085, 12.11
F0 = P.LIGHT_SPEED / 1.55e-6
TOTAL_STEPS = 4096  # the clock and the waveforms that a program carries
ETA0 = 376.73


def listed():
    return [
        # A tiny TE scene with conductive silicon, stepped a few steps at a
        # time: an interactive preview.  The smallest call.
        dict(name="te_small", kind="2d", pol="te", shape="83x117", pml=8, material="conductive", monitors=1, freqs=1,
             steps=16),
        # The 2D scene of the benchmark: 400 x 400, 20-cell CPML, one line
        # monitor at three frequencies, one 256-step chunk.
        dict(name="tm_400", kind="2d", pol="tm", shape="400x400", pml=20, material="dielectric", monitors=1, freqs=3,
             steps=256),
        # The smallest 3D request of the serving mix.
        dict(name="box_128", kind="3d", shape="128x128x128", pml=12, material="dielectric", monitors=2, freqs=3,
             wall=False, steps=64),
        # A ragged 3D grid (no extent a multiple of a tile) on a metallic floor.
        dict(name="box_odd", kind="3d", shape="150x203x277", pml=10, material="dielectric", monitors=1, freqs=2,
             wall=True, steps=32),
        # The headline 3D scene: 512 x 512 x 256, 12-cell CPML, four DFT planes
        # at five frequencies.
        dict(name="box_512", kind="3d", shape="256x512x512", pml=12, material="dielectric", monitors=4, freqs=5,
             wall=False, steps=16),
        # A capacity-style grid of layered waveguides, no monitors: the largest.
        dict(name="layers_large", kind="3d", shape="512x640x1024", pml=12, material="layers", monitors=0, freqs=0,
             wall=False, steps=4),
        # Conductive silicon (per-site decay and source on E and H).
        dict(name="conductive", kind="3d", shape="96x192x256", pml=12, material="conductive", monitors=1, freqs=3,
             wall=False, steps=16),
        # A rectilinear grid (derivative metrics on every axis).
        dict(name="rectilinear", kind="3d", shape="128x192x256", pml=12, material="rectilinear", monitors=1, freqs=3,
             wall=False, steps=16),
        # Inverse design in 2D: density -> permittivity -> run -> overlap, and
        # the gradient back (forward and adjoint), 600 x 600 with a 200 x 200
        # design region.
        dict(name="gradient_2d", kind="gradient2d", shape="600x600", pml=20, design="200x200", steps=300),
        # The same in 3D: a 256 x 256 x 128 grid, continuous permittivity (more
        # coefficients than a codebook holds).
        dict(name="gradient_3d", kind="gradient3d", shape="128x256x256", pml=12, design="10x62x62", steps=48),
        # What an automatically terminated run asks between chunks: energy, max
        # |field|, finiteness, the monitors' change and their flux.
        dict(name="checks", kind="checks", shape="192x384x384", pml=12, material="dielectric", monitors=3, freqs=5,
             wall=False, steps=0),
        # A batch of small requests through the serving engine, compile and
        # results included.
        dict(name="serve_mix", kind="serve", shape2="256,416,640,1000", shape3="128x128x128,96x160x192", pml=12,
             monitors=2, freqs=3, steps=300),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["2d", "2d", "2d", "3d", "3d", "3d", "3d", "gradient2d", "gradient3d", "checks", "serve"])
    if kind == "2d":
        ny, nx = _log(rng, 64, 1024), _log(rng, 64, 1024)
        return dict(kind=kind, pol=rng.choice(["tm", "te"]), shape=f"{ny}x{nx}", pml=rng.randint(6, 20),
                    material=rng.choice(["dielectric", "dielectric", "conductive"]), monitors=rng.randint(0, 4),
                    freqs=rng.randint(1, 6), steps=_log(rng, 16, 256))
    if kind == "3d":
        material = rng.choice(["dielectric", "dielectric", "dielectric", "layers", "smooth", "conductive",
                               "rectilinear", "axis_uniform"])
        plain = material in ("dielectric", "layers")
        while True:
            nz, ny, nx = _log(rng, 32, 512), _log(rng, 40, 640), _log(rng, 48, 1024)
            cells = nz * ny * nx
            if cells <= (160e6 if plain else 5e6):  # per-site materials are planned on the host
                break
        steps = max(4, min(64, int(6e8 / cells)))
        return dict(kind=kind, shape=f"{nz}x{ny}x{nx}", pml=rng.randint(5, 13), material=material,
                    monitors=rng.randint(0, 4), freqs=rng.randint(1, 6), wall=rng.random() < 0.3, steps=steps)
    if kind == "gradient2d":
        ny, nx = _log(rng, 200, 640), _log(rng, 200, 640)
        dy, dx = _log(rng, 20, ny - 110), _log(rng, 20, nx - 110)
        return dict(kind=kind, shape=f"{ny}x{nx}", pml=rng.randint(8, 20), design=f"{dy}x{dx}",
                    steps=_log(rng, 100, 300))
    if kind == "gradient3d":
        nz, ny, nx = _log(rng, 64, 128), _log(rng, 96, 256), _log(rng, 96, 256)
        return dict(kind=kind, shape=f"{nz}x{ny}x{nx}", pml=rng.randint(6, 12),
                    design=f"{rng.randint(4, 20)}x{rng.randint(8, ny - 48)}x{rng.randint(8, nx - 48)}",
                    steps=rng.randint(24, 48))
    if kind == "checks":
        return dict(kind=kind, shape=f"{_log(rng, 48, 192)}x{_log(rng, 64, 384)}x{_log(rng, 64, 384)}",
                    pml=rng.randint(6, 12), material="dielectric", monitors=rng.randint(1, 4),
                    freqs=rng.randint(1, 6), wall=rng.random() < 0.3, steps=0)
    side = ",".join(str(_log(rng, 200, 1000)) for _ in range(3))
    vol = ",".join(f"{_log(rng, 48, 128)}x{_log(rng, 64, 160)}x{_log(rng, 64, 192)}" for _ in range(2))
    return dict(kind="serve", shape2=side, shape3=vol, pml=rng.randint(8, 12), monitors=rng.randint(1, 3),
                freqs=rng.randint(1, 4), steps=_log(rng, 120, 300))


# ---- scenes -----------------------------------------------------------------


def _dims(text):
    return tuple(int(v) for v in text.split("x"))


def _dt(ndim, courant):
    return courant * RES / (P.LIGHT_SPEED * math.sqrt(ndim))


def _freqs(n):
    return (np.linspace(0.9, 1.1, n) if n > 1 else np.ones(1)) * F0


@functools.lru_cache(maxsize=8)
def _plane(shape, pml, frac, n_freqs):
    """An x-normal DFT plane over the non-absorbing part; it does not depend on
    the seed, so a program that runs many designs plans it once."""
    nz, ny, nx = shape
    zc = (np.arange(pml, nz - pml) + 0.5) * RES
    yc = (np.arange(pml, ny - pml) + 0.5) * RES
    return P.plane_monitor(shape, RES, "x", frac * nx * RES, zc, yc, _freqs(n_freqs))


@functools.lru_cache(maxsize=64)
def _pulse(dt):
    times = (np.arange(TOTAL_STEPS, dtype=np.float64) + 0.5) * dt
    return P.gaussian_pulse(times, F0, 0.2 * F0, offset=0.5)


def _dipole(component, timing, site, coefficient, dt):
    return P.SourcePlan(component, timing, tuple(int(v) for v in site),
                        np.full((1,) * len(site), coefficient, np.float32), _pulse(dt))


def _boxes(ids, rng, z=None):
    ny, nx = ids.shape[-2:]
    for _ in range(int(rng.integers(8, 17))):
        sy, sx = (int(v) for v in rng.integers(8, max(9, min(100, min(ny, nx) // 2)), size=2))
        y0, x0 = int(rng.integers(0, max(1, ny - sy))), int(rng.integers(0, max(1, nx - sx)))
        ids[(slice(y0, y0 + sy), slice(x0, x0 + sx)) if z is None else (z, slice(y0, y0 + sy), slice(x0, x0 + sx))] = 1


def _layers(ids, rng):
    """Silicon slab waveguides along x with a wandering core."""
    nz, ny, nx = ids.shape
    for zc in range(24, nz - 16, 64):
        for yc in range(32, ny - 24, 96):
            for x in range(0, nx, 16):
                lo = yc - 12 + int(rng.integers(-3, 4))
                ids[zc - 5:zc + 6, lo:lo + 24, x:x + 16] = 1


def _scene_3d(shape, pml, material, monitors, freqs, wall, seed):
    nz, ny, nx = shape
    rng = np.random.default_rng(seed)
    dt = _dt(3, 0.99)
    ids = np.zeros(shape, np.uint8)
    if material == "layers":
        _layers(ids, rng)
    else:
        _boxes(ids, rng, slice(nz // 2 - 5, nz // 2 + 6))
    edges = tuple(e for e in P.ALL_EDGES_3D if not (wall and e == "front"))
    h_terms, e_terms = P.plan_cpml(shape, dt, RES, pml_cells=pml, edges=edges)
    ids = P.extend_into_absorber(ids, P.absorber_edge_counts(shape, pml, edges=edges, resolution=RES))
    table = np.ones(256, np.float32)
    table[0], table[1] = OXIDE, SILICON
    k, j, i = site = (nz // 2, ny // 2, nx // 2)
    eps = float(table[ids[k - 1:k + 1, j, i - 1:i + 1]].mean())
    source = _dipole("Ey", "pre_e", site, -dt / (P.EPS_0 * eps), dt)
    mons = [_plane(shape, pml, f, freqs) for f in (0.2, 0.4, 0.6, 0.8)[:monitors]]
    spec = P.ProgramSpec(shape, dt, RES, voxel_ids=ids, eps_table=table, h_terms=h_terms, e_terms=e_terms,
                         sources=[source], monitors=mons, total_steps=TOTAL_STEPS,
                         metallic_edges=frozenset({"front"}) if wall else frozenset())
    if material == "conductive":
        spec = workloads.conductive(spec)
    elif material in ("rectilinear", "axis_uniform"):
        spec = workloads.graded(spec, material, seed=seed)
    elif material == "smooth":  # a continuous permittivity: one coefficient per site
        eps = torch.as_tensor(table[ids], device="cuda")
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        eps = eps + 0.5 * torch.rand(eps.shape, generator=gen, device="cuda")
        coefs = adjoint.eps_to_coefficients_3d(eps, dt, P.EPS_0)
        spec = adjoint.site_spec(spec, {c: v.cpu().numpy() for c, v in zip(("Ex", "Ey", "Ez"), coefs)})
    return spec


def _line(shape, pol, x, pml, n_freqs):
    """A DFT line along y at column x (the polarization's components)."""
    rows = np.arange(pml, shape[0] - pml)
    idx, w = [], []
    for c in P.COMPONENTS:
        sy, sx = P.component_shape(c, shape, pol)
        idx.append((np.minimum(rows, sy - 1) * sx + min(x, sx - 1)).astype(np.int32)[:, None])
        w.append(np.ones((rows.size, 1), np.float32))
    mask = np.array([1.0 if c in P.active_components(2, pol) else 0.0 for c in P.COMPONENTS], np.float32)
    return P.DftMonitorPlan(np.asarray(_freqs(n_freqs), np.float32), idx, w, mask)


def _scene_2d(shape, pol, pml, material, monitors, freqs, seed):
    ny, nx = shape
    rng = np.random.default_rng(seed)
    dt = _dt(2, 0.7)
    ids = np.zeros(shape, np.uint8)
    _boxes(ids, rng)
    h_terms, e_terms = P.plan_cpml(shape, dt, RES, pml_cells=pml, polarization=pol)
    ids = P.extend_into_absorber(ids, P.absorber_edge_counts(shape, pml, resolution=RES, explicit_thickness=True))
    eps = np.where(ids == 1, np.float32(SILICON), np.float32(OXIDE))
    e_comps = ("Ez",) if pol == "tm" else ("Ex", "Ey")
    h_site = None
    if material == "conductive":
        sigma = np.where(ids == 1, np.float32(4e4), np.float32(0.0))
        e_site, h_site, _eps = P.lossy_site_coefficients_2d(eps, sigma, dt, pol)
    else:
        e_site = {c: (np.float32(1.0), P.e_source_2d(P.site_values_2d(eps, c, pol), dt)) for c in e_comps}
    j, i = site = (ny // 2, int(0.6 * nx) - 6)  # a few cells before the first monitor
    if pol == "tm":
        source = _dipole("Ez", "pre_e", site, -dt / (P.EPS_0 * float(eps[j, i])), dt)
    else:
        source = _dipole("Hz", "h", site, -dt / P.MU_0 / ETA0, dt)
    mons = [_line(shape, pol, int(f * nx), pml, freqs) for f in (0.6, 0.7, 0.8, 0.9)[:monitors]]
    return P.ProgramSpec(shape, dt, RES, polarization=pol, e_site=e_site, h_site=h_site, h_terms=h_terms,
                         e_terms=e_terms, sources=[source], monitors=mons, total_steps=TOTAL_STEPS)


def _spec(case, seed):
    if case["kind"] == "2d":
        return _scene_2d(_dims(case["shape"]), case["pol"], case["pml"], case["material"], case["monitors"],
                         case["freqs"], seed)
    return _scene_3d(_dims(case["shape"]), case["pml"], case["material"], case["monitors"], case["freqs"],
                     case["wall"], seed)


def _fields(spec, seed):
    """Band-limited noise for every active component, E about 1, H about 1/377."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 17)
    out = {}
    for c in P.active_components(spec.ndim, spec.polarization):
        shape = P.component_shape(c, spec.grid_shape, spec.polarization)
        coarse = torch.randn((1, 1, *(max(2, n // 8) for n in shape)), generator=gen, device="cuda")
        mode = "trilinear" if spec.ndim == 3 else "bilinear"
        v = torch.nn.functional.interpolate(coarse, size=shape, mode=mode, align_corners=True)[0, 0]
        out[c] = v if c[0] == "E" else v.mul_(1.0 / ETA0)
    return out


def _requests(case, seed):
    """Specs and step counts of a batch: TM squares and 3D boxes."""
    specs = [_scene_2d((int(n), int(n)), "tm", case["pml"], "dielectric", case["monitors"], case["freqs"], seed + q)
             for q, n in enumerate(case["shape2"].split(","))]
    specs += [_scene_3d(_dims(s), case["pml"], "dielectric", case["monitors"], case["freqs"], False, seed + 50 + q)
              for q, s in enumerate(case["shape3"].split(","))]
    return [(s, case["steps"] + 8 * q - (q % 2)) for q, s in enumerate(specs)]


# ---- gradients --------------------------------------------------------------


def _design(case, seed):
    """A gradient case's spec, box, base permittivity, design voxels, density
    and objective weights.  The dipole sits in the middle of the design and the
    monitor five cells beside it, so that the objective is live early in the
    run.  3D design voxels lie one cell inside the box, whose E sites then hold
    every coefficient that the density moves."""
    shape, d = _dims(case["shape"]), _dims(case["design"])
    gen = torch.Generator(device="cpu").manual_seed(int(seed))
    lo = tuple((n - m) // 2 for n, m in zip(shape, d))
    hi = tuple(a + m for a, m in zip(lo, d))
    site = tuple(a + m // 2 for a, m in zip(lo, d))
    if len(shape) == 2:
        spec = _scene_2d(shape, "tm", case["pml"], "dielectric", 0, 0, seed)
        box, base = (lo, hi), np.full(shape, OXIDE, np.float32)
        mon = _line(shape, "tm", site[1] + 5, case["pml"], 3)
    else:
        spec = _scene_3d(shape, case["pml"], "dielectric", 0, 0, False, seed)
        box, base = (tuple(a - 1 for a in lo), tuple(b + 1 for b in hi)), spec.eps_table[spec.voxel_ids]
        mon = _plane(shape, case["pml"], (site[2] + 5) / shape[2], 3)
    spec = dataclasses.replace(spec, sources=[dataclasses.replace(spec.sources[0], start=site)], monitors=[mon])
    rho = torch.rand(d, generator=gen).cuda()
    weights = torch.randn(mon.points, generator=gen).cuda()
    return spec, box, base, tuple(slice(a, b) for a, b in zip(lo, hi)), rho, weights


def _objective(re, im, weights, ndim):
    """|overlap|^2 of the monitor's middle frequency with a fixed profile."""
    n, c = weights.numel(), P.COMPONENT_INDEX["Ez" if ndim == 2 else "Ey"]
    sl = slice((c * 3 + 1) * n, (c * 3 + 2) * n)
    return (weights * re[sl]).sum() ** 2 + (weights * im[sl]).sum() ** 2


def _gradient_state(case, seed):
    spec, box, base, hot, rho, weights = _design(case, seed)
    eps0 = torch.as_tensor(base, device="cuda")
    if spec.ndim == 3:
        coefs = adjoint.eps_to_coefficients_3d(eps0, spec.dt, P.EPS_0)
        spec = adjoint.site_spec(spec, {c: v.cpu().numpy() for c, v in zip(("Ex", "Ey", "Ez"), coefs)})
    problem = adjoint.AdjointProblem(spec, case["steps"], box)
    return dict(kind="gradient", problem=problem, eps0=eps0, hot=hot, rho=rho.requires_grad_(True), weights=weights,
                spec=spec)


def _run_gradient(s):
    rho, spec = s["rho"], s["spec"]
    rho.grad = None
    eps = s["eps0"].clone()
    eps[s["hot"]] = OXIDE + rho * (SILICON - OXIDE)
    if spec.ndim == 2:
        coefs = [adjoint.eps_to_coefficients_2d(eps, spec.dt, P.EPS_0)]
    else:
        coefs = adjoint.eps_to_coefficients_3d(eps, spec.dt, P.EPS_0)
    re, im = adjoint.simulate(s["problem"], coefs)
    value = _objective(re, im, s["weights"], spec.ndim)
    value.backward()
    return {"value": value.detach(), "gradient": rho.grad, "dft_re": re.detach(), "dft_im": im.detach()}


# ---- the interface ----------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind.startswith("gradient"):
        return _gradient_state(case, seed)
    if kind == "serve":
        batch = _requests(case, seed)
        return dict(kind=kind, engine=serve.ServingEngine(),
                    requests=[serve.Request(r, spec, steps) for r, (spec, steps) in enumerate(batch)])
    spec = _spec(case, seed)
    program = runtime.compile_program(spec, tile="auto", z_chunk="auto")
    state = runtime.initial_state(program, fields=_fields(spec, seed))
    if kind == "checks":
        arena = torch.randn(state.dft_re.shape, generator=torch.Generator(device="cuda").manual_seed(int(seed)),
                            device="cuda")
        state.dft_re.copy_(arena)
        state.dft_im.copy_(arena.flip(0))
        state.dft_w.fill_(100.0)
        # The previous check's arena: the first call records it.
        state.dft_re.mul_(0.9)
        runtime.dft_change(state, program)
        state.dft_re.copy_(arena)
    return dict(kind=kind, program=program, state=state, steps=case["steps"])


def run(s):
    kind = s["kind"]
    if kind == "gradient":
        return _run_gradient(s)
    if kind == "serve":
        results = s["engine"].run(s["requests"])
        return [[r.dft_re, r.dft_im, r.dft_w] for r in results]
    state, program = s["state"], s["program"]
    if kind == "checks":
        d = runtime.field_diagnostics(state, program)
        change, finite = runtime.dft_change(state, program)
        flux = [runtime.monitor_dft_flux(state, program, m, "x", measure=RES * RES)
                for m in range(len(program.spec.monitors))]
        return {"energy": d.energy, "max": d.max_field, "nonfinite": d.nonfinite, "flux": np.stack(flux),
                "finite": bool(finite and d.finite)}
    runtime.run_steps(state, program, s["steps"])
    out = {c: state.field(c) for c in program.active}
    out["psi"] = list(state.psi_h) + list(state.psi_e)
    if program.arena is not None:
        out["dft"] = [state.dft_re, state.dft_im, state.dft_w]
    return out


def _step_work(spec, steps):
    """Bytes of one pass (fields and memories in and out once, material once,
    the DFT arena in and out once) and its arithmetic: per derivative a
    difference and a quotient, per update two products and two sums."""
    act = P.active_components(spec["ndim"], spec["pol"])
    sizes = {c: int(np.prod(P.component_shape(c, spec["shape"], spec["pol"]))) for c in act}
    cells = int(np.prod(spec["shape"]))
    terms = 12 if spec["ndim"] == 3 else 4
    psi = 0
    for a, n in enumerate(spec["shape"]):
        faces = 2 * (2 if spec["ndim"] == 3 else 1)  # terms along the axis, H and E
        psi += faces * 2 * spec["pml"] * (cells // n)
    nbytes = 8 * sum(sizes.values()) + 8 * psi + spec["material"] * cells + 16 * spec["samples"]
    return nbytes, steps * (cells * (2 * terms + 4 * len(act)) + 5 * psi + 4 * spec["samples"])


def _shape_work(shape, pol, pml, material, samples, steps):
    return _step_work(dict(ndim=len(shape), shape=shape, pol=pol, pml=pml, material=material, samples=samples), steps)


def _samples(shape, pml, monitors, freqs):
    """(point, component, frequency) values that the monitors accumulate."""
    if len(shape) == 3:
        return monitors * freqs * 4 * max(0, shape[0] - 2 * pml) * max(0, shape[1] - 2 * pml)
    return monitors * freqs * 3 * max(0, shape[0] - 2 * pml)


def work(case):
    kind = case["kind"]
    if kind == "serve":
        total_b = total_f = 0
        shapes = [(int(n), int(n)) for n in case["shape2"].split(",")] + [_dims(s) for s in case["shape3"].split(",")]
        for q, shape in enumerate(shapes):
            b, f = _shape_work(shape, "tm", case["pml"], 1 if len(shape) == 3 else 4,
                               _samples(shape, case["pml"], case["monitors"], case["freqs"]),
                               case["steps"] + 8 * q - (q % 2))
            total_b, total_f = total_b + b, total_f + f
        return {"bytes": total_b, "flops": total_f}
    shape = _dims(case["shape"])
    if kind == "checks":
        n = _samples(shape, case["pml"], case["monitors"], case["freqs"])
        cells = int(np.prod(shape))
        return {"bytes": 24 * cells + 4 * cells + 16 * n + 8 * n, "flops": 6 * 4 * cells + 20 * n}
    if kind.startswith("gradient"):
        pol = "tm"
        b, f = _shape_work(shape, pol, case["pml"], 12 if len(shape) == 3 else 4, 0, case["steps"])
        return {"bytes": b + 4 * int(np.prod(_dims(case["design"]))), "flops": 2 * f}
    material = {"conductive": 2, "smooth": 12}.get(case["material"], 1) if len(shape) == 3 else (
        16 if case["material"] == "conductive" else 4)
    b, f = _shape_work(shape, case.get("pol", "tm"), case["pml"], material,
                       _samples(shape, case["pml"], case["monitors"], case["freqs"]), case["steps"])
    return {"bytes": b, "flops": f}


def tolerance(case):
    """Four times the distance of the float32 path from float64 (exact): the
    steps' rounding, the float32 clock in the DFT phases (weak fields far from
    the source show it most), and in gradients both, forward and back."""
    if case["kind"] == "serve":
        return {"rel": 1.2e-4}
    if case["kind"].startswith("gradient"):
        return {"rel": 7e-5}
    if case["kind"] == "checks":
        return {"rel": 1e-6}
    return {"rel": 1.5e-5}


# ---- 64-bit answers ---------------------------------------------------------

_AXES = {3: {"z": 0, "y": 1, "x": 2}, 2: {"y": 0, "x": 1}}
_TERMS = {  # component -> ((axis, sign, differentiated component), ...)
    "Hx": (("y", 1, "Ez"), ("z", -1, "Ey")), "Hy": (("z", 1, "Ex"), ("x", -1, "Ez")),
    "Hz": (("x", 1, "Ey"), ("y", -1, "Ex")), "Ex": (("y", 1, "Hz"), ("z", -1, "Hy")),
    "Ey": (("z", 1, "Hx"), ("x", -1, "Hz")), "Ez": (("x", 1, "Hy"), ("y", -1, "Hx")),
}
_EDGES = {"front": ("z", 0), "back": ("z", 1), "bottom": ("y", 0), "top": ("y", 1), "left": ("x", 0), "right": ("x", 1)}


class _Exact:
    """The leapfrog step in float64 with plain tensor operations."""

    def __init__(self, spec, fields=None, sources=None):
        self.spec, self.nd = spec, spec.ndim
        self.axes = _AXES[spec.ndim]
        self.act = P.active_components(spec.ndim, spec.polarization)
        self.shape = {c: P.component_shape(c, spec.grid_shape, spec.polarization) for c in self.act}
        t64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device="cuda")  # noqa: E731
        self.t64 = t64
        self.f = {c: (fields[c].double() if fields is not None
                      else torch.zeros(self.shape[c], dtype=torch.float64, device="cuda")) for c in self.act}
        self.h = {c: tuple(t64(v) for v in hv) for c, hv in spec.h_coefficients().items() if c in self.act}
        self.e = dict(sources) if sources is not None else self._electric()
        self.cpml, self.psi = {}, {}
        for t in list(spec.h_terms) + list(spec.e_terms):
            if t.width:
                axis = next(a for a, n in self.axes.items() if n == t.axis)
                view = [1] * self.nd
                view[t.axis] = -1
                self.cpml[t.component, axis] = (t.axis, t.low, t.high, *(t64(v).reshape(view)
                                                                          for v in (t.a, t.b, t.inv_kappa)))
                self.psi[t.component, axis] = torch.zeros(t.psi_shape(self.shape[t.component]), dtype=torch.float64,
                                                          device="cuda")
        self.metric = None
        if spec.metrics is not None:
            cells = dict(zip(self.axes, spec.grid_shape))
            self.metric = {(w, a): t64(spec.metrics.along(f"{w}_{a}", cells[a] + (w == "h_to_e")))
                           for w in ("e_to_h", "h_to_e") for a in self.axes}
        self.walls = {_EDGES[e] for e in spec.metallic_edges}
        self.src = [(s, t64(s.coeff), np.asarray(s.waveform, np.float64).reshape(-1)) for s in spec.sources]
        self.mon = []
        for m in spec.monitors:
            rows = {c: (torch.as_tensor(np.asarray(m.indices[n]).reshape(m.points, -1).astype(np.int64), device="cuda"),
                        t64(m.weights[n])) for n, c in enumerate(P.COMPONENTS) if m.component_mask[n] and c in self.act}
            zero = torch.zeros((6, len(m.freqs), m.points), dtype=torch.float64, device="cuda")
            self.mon.append([rows, t64(m.freqs), zero, zero.clone(), 0.0])
        self.n = 0

    def _electric(self):
        s = self.spec
        if s.e_site is not None:
            return {c: (self.t64(s.e_site[c][0]), self.t64(s.e_site[c][1])) for c in self.act if c[0] == "E"}
        eps = self.t64(s.eps_table)[torch.as_tensor(s.voxel_ids, device="cuda").long()]
        return {c: (self.t64(1.0), v) for c, v in zip(("Ex", "Ey", "Ez"), exact_coefficients(eps, s.dt))}

    def _deriv(self, comp, axis, v):
        """d/axis of v on comp's support: forward for H, ghost-padded backward for E."""
        a = self.axes[axis]
        n = v.shape[a]
        if comp[0] == "H":
            d = v.narrow(a, 1, n - 1) - v.narrow(a, 0, n - 1)
        else:
            low, high = v.narrow(a, 0, 1), v.narrow(a, n - 1, 1)
            zero = torch.zeros_like(low)
            d = torch.cat([low if (axis, 0) in self.walls else zero, v.narrow(a, 1, n - 1) - v.narrow(a, 0, n - 1),
                           -high if (axis, 1) in self.walls else zero], dim=a)
        if self.metric is None:
            d = d / self.spec.resolution
        else:
            view = [1] * self.nd
            view[a] = -1
            d = d * self.metric["e_to_h" if comp[0] == "H" else "h_to_e", axis].reshape(view)
        if (comp, axis) in self.cpml:
            a, low, high, ca, cb, ck = self.cpml[comp, axis]
            m = d.shape[a]
            slab = torch.cat([d.narrow(a, 0, low), d.narrow(a, m - high, high)], dim=a)
            psi = cb * self.psi[comp, axis] + ca * slab
            self.psi[comp, axis] = psi
            slab = slab * ck + psi
            d = torch.cat([slab.narrow(a, 0, low), d.narrow(a, low, m - low - high), slab.narrow(a, low, high)], dim=a)
        return d

    def _inject(self, timing):
        for s, coeff, wave in self.src:
            if s.timing == timing:
                at = tuple(slice(b, b + n) for b, n in zip(s.start, coeff.shape))
                v = self.f[s.component].clone()
                v[at] = v[at] + coeff * float(wave[min(self.n, wave.size - 1)])
                self.f[s.component] = v

    def _mask(self, comp):
        """PEC: normal H and tangential E vanish on a metallic wall."""
        v = self.f[comp]
        for axis, high in self.walls:
            if (comp[0] == "H") == (comp[1] == axis):
                a = self.axes[axis]
                keep = torch.ones(v.shape[a], dtype=torch.float64, device="cuda")
                keep[-1 if high else 0] = 0.0
                view = [1] * self.nd
                view[a] = -1
                self.f[comp] = self.f[comp] * keep.reshape(view)

    def _update(self, comps):
        for c in comps:
            curl = None
            for axis, sign, other in _TERMS[c]:
                if axis in self.axes and other in self.act:
                    d = self._deriv(c, axis, self.f[other])
                    curl = sign * d if curl is None else (curl + d if sign > 0 else curl - d)
            decay, source = self.h[c] if c[0] == "H" else self.e[c]
            self.f[c] = decay * self.f[c] - source * curl if c[0] == "H" else decay * self.f[c] + source * curl

    def step(self):
        self._inject("pre_e")
        h, e = [c for c in self.act if c[0] == "H"], [c for c in self.act if c[0] == "E"]
        self._update(h)
        self._inject("h")
        for c in h:
            self._mask(c)
        self._update(e)
        self._inject("e")
        for c in e:
            self._mask(c)
        self.n += 1
        t = self.n * float(self.spec.dt)
        for m in self.mon:
            rows, freqs = m[0], m[1]
            phase = 2.0 * math.pi * freqs * t
            sample = torch.stack([(self.f[c].reshape(-1)[rows[c][0]] * rows[c][1]).sum(1) if c in rows
                                  else torch.zeros_like(m[2][0, 0]) for c in P.COMPONENTS])[:, None, :]
            m[2] = m[2] + torch.cos(phase)[None, :, None] * sample
            m[3] = m[3] + torch.sin(phase)[None, :, None] * sample
            m[4] += 1.0

    def arena(self):
        re = torch.cat([m[2].reshape(-1) for m in self.mon]) if self.mon else None
        im = torch.cat([m[3].reshape(-1) for m in self.mon]) if self.mon else None
        w = torch.cat([torch.full((m[1].numel(),), m[4], dtype=torch.float64, device="cuda") for m in self.mon]) \
            if self.mon else None
        return [re, im, w]

    def psi_list(self):
        """The memories in the spec's term order (empty slabs included)."""
        out = []
        for t in list(self.spec.h_terms) + list(self.spec.e_terms):
            axis = next(a for a, n in self.axes.items() if n == t.axis)
            out.append(self.psi[t.component, axis] if t.width
                       else torch.zeros(t.psi_shape(self.shape[t.component]), dtype=torch.float64, device="cuda"))
        return out


def exact_coefficients(eps, dt):
    """dt / (eps0 eps) at the Ex, Ey, Ez sites of a voxel grid: the mean of the
    four voxels that share the edge, indices clipped at the faces."""

    def pair(v, a):
        n = v.shape[a]
        first, last = v.narrow(a, 0, 1), v.narrow(a, n - 1, 1)
        padded = torch.cat([first, v, last], dim=a)
        return 0.5 * (padded.narrow(a, 0, n + 1) + padded.narrow(a, 1, n + 1))

    return [dt / (P.EPS_0 * pair(pair(eps, a), b)) for a, b in ((0, 1), (0, 2), (1, 2))]


def _exact_gradient(case, seed):
    spec, _box, base, hot, rho, weights = _design(case, seed)
    rho, weights = rho.double().requires_grad_(True), weights.double()
    eps = torch.as_tensor(base, device="cuda").double().clone()
    eps[hot] = OXIDE + rho * (SILICON - OXIDE)
    one = torch.ones((), dtype=torch.float64, device="cuda")
    if spec.ndim == 2:
        ny, nx = spec.grid_shape
        rows = torch.arange(ny + 1, device="cuda").clamp(max=ny - 1)
        cols = torch.arange(nx + 1, device="cuda").clamp(max=nx - 1)
        electric = {"Ez": (one, spec.dt / (P.EPS_0 * eps[rows][:, cols]))}
    else:
        electric = {c: (one, v) for c, v in zip(("Ex", "Ey", "Ez"), exact_coefficients(eps, spec.dt))}
    names = list(electric)

    # Steps run in checkpointed blocks, so that the graph of one block at a
    # time is held.
    sim = _Exact(spec, sources=electric)
    keys = list(sim.psi)

    def block(first, count, *flat):
        k = len(sim.act)
        sim.f = dict(zip(sim.act, flat[:k]))
        sim.psi = dict(zip(keys, flat[k:k + len(keys)]))
        sim.mon[0][2], sim.mon[0][3] = flat[k + len(keys):k + len(keys) + 2]
        sim.e = {c: (one, v) for c, v in zip(names, flat[k + len(keys) + 2:])}
        sim.n = first
        for _ in range(count):
            sim.step()
        return (*(sim.f[c] for c in sim.act), *(sim.psi[q] for q in keys), sim.mon[0][2], sim.mon[0][3])

    state = (*(sim.f[c] for c in sim.act), *(sim.psi[q] for q in keys), sim.mon[0][2], sim.mon[0][3])
    coefs = [electric[c][1] for c in names]
    size = 20 if spec.ndim == 2 else 8
    for first in range(0, case["steps"], size):
        state = torch.utils.checkpoint.checkpoint(block, first, min(size, case["steps"] - first), *state, *coefs,
                                                  use_reentrant=False)
    re, im = state[-2].reshape(-1), state[-1].reshape(-1)
    value = _objective(re, im, weights, spec.ndim)
    value.backward()
    return {"value": value.detach(), "gradient": rho.grad, "dft_re": re.detach(), "dft_im": im.detach()}


def _exact_checks(case, seed):
    spec = _spec(case, seed)
    fields = _fields(spec, seed)
    sim = _Exact(spec)
    energy = largest = 0.0
    for c in sim.act:
        v = fields[c].double()
        w = v * v
        if c[0] == "E":
            w = w * (spec.dt / (P.EPS_0 * sim.e[c][1]))
        for a, n in enumerate(spec.grid_shape):  # control volumes: half a cell at the ends of a node axis
            if v.shape[a] == n + 1:
                h = torch.ones(n + 1, dtype=torch.float64, device="cuda")
                h[0] = h[-1] = 0.5
                view = [1, 1, 1]
                view[a] = -1
                w = w * h.reshape(view)
        energy += 0.5 * (P.EPS_0 if c[0] == "E" else P.MU_0) * float(w.sum()) * RES**3
        largest = max(largest, float(v.abs().max()))
    n = sum(6 * len(m.freqs) * m.points for m in spec.monitors)
    arena = torch.randn((n,), generator=torch.Generator(device="cuda").manual_seed(int(seed)), device="cuda")
    re, im = arena.double(), arena.flip(0).double()
    flux, at = [], 0
    for m in spec.monitors:
        nf, q = len(m.freqs), m.points
        v = torch.complex(re[at:at + 6 * nf * q], im[at:at + 6 * nf * q]).reshape(6, nf, q) * (2.0 / 100.0)
        at += 6 * nf * q
        s = (v[1] * v[5].conj() - v[2] * v[4].conj()).real.sum(1)
        flux.append((0.5 * s * RES * RES).cpu().numpy())
    return {"energy": energy, "max": largest, "nonfinite": 0, "flux": np.stack(flux), "finite": True}


def exact(case, seed):
    kind = case["kind"]
    if kind.startswith("gradient"):
        return _exact_gradient(case, seed)
    if kind == "checks":
        return _exact_checks(case, seed)
    if kind == "serve":
        out = []
        for spec, steps in _requests(case, seed):
            sim = _Exact(spec)
            for _ in range(steps):
                sim.step()
            out.append(sim.arena())
        return out
    spec = _spec(case, seed)
    sim = _Exact(spec, _fields(spec, seed))
    for _ in range(case["steps"]):
        sim.step()
    out = dict(sim.f)
    out["psi"] = sim.psi_list()
    if spec.monitors:
        out["dft"] = sim.arena()
    return out
