"""The work a user of this package has it do, as timed cases.

Every case goes through the public Python entry points (``RTE.from_problem``,
``RTE.solve``, ``RTE.render_device``, ``RTE.integrate_to_sensor``,
``gradient.render_differentiable``) on seeded synthetic scenes of the shapes
that the package's own scenes, tests and benchmark use.  A solve runs a fixed
number of iterations (the accuracy is set below what they reach), so that a
pass is always the same work; the counts are those of a solve well on its way
to the accuracies in use (1e-4 and 1e-5 take 5 to 30 iterations).

kinds:
  solve       initialise, iterate, render to device-resident rays
  render      one render of a solved medium to device-resident rays
  sensor      one render of a solved medium through a sensor dict (host arrays)
  gradient    forward and backward of the differentiable render on a solved
              medium: image, d/d(extinction), d/d(albedo)
  retrieval   two optimiser steps: the medium is replaced, re-solved, rendered
              and differentiated, twice
"""
from __future__ import annotations

import numpy as np
import torch

from at3d_gb300.gradient import render_differentiable
from at3d_gb300.medium import henyey_greenstein_legcoef, rayleigh_legcoef
from at3d_gb300.scenes import FIELD_G, FIELD_SSA, VIEW_ZENITHS, cloud_blob, cloud_field, orthographic_views, polarized_blob
from at3d_gb300.solver import RTE
from at3d_gb300 import Species

_SOLACC = 1e-7  # below what the fixed iteration counts reach


def _case(kind, scene, nx, ny, nz, nmu, boundary, iters, npix, views, *, stokes=1, thermal=False, rayleigh=False,
          fraction=0.3, name=None):
    c = dict(kind=kind, scene=scene, nx=nx, ny=ny, nz=nz, nmu=nmu, nphi=2 * nmu, boundary=boundary, iters=iters,
             npix=npix, views=views, stokes=stokes, thermal=thermal, rayleigh=rayleigh, fraction=fraction)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest solve in use (the size of the smoke test and of unit-test scenes): launches and latency
        _case("solve", "blob", 12, 12, 10, 8, "open", 8, 6, 3, rayleigh=True, name="solve_tiny_open"),
        # the plain scalar workload: periodic cloud blob over a Rayleigh atmosphere, every point scattering
        _case("solve", "blob", 32, 32, 24, 8, "periodic", 12, 32, 9, rayleigh=True, name="solve_periodic_32"),
        # the retrieval-sized medium: sparse clouds in clear air, open boundaries
        _case("solve", "field", 64, 64, 32, 8, "open", 12, 64, 9, fraction=0.2, name="solve_open_64"),
        # an odd-sized domain with cloud and a Rayleigh layer (no clear points), intermediate angular resolution
        _case("solve", "field", 45, 37, 29, 12, "open", 10, 23, 5, rayleigh=True, name="solve_odd_open"),
        # the headline workload: one wavelength of the large-eddy-simulation-sized field at 16 x 32 ordinates
        _case("solve", "field", 128, 128, 64, 16, "open", 20, 64, 9, name="solve_open_128"),
        # thermal emission on a large field: few iterations, source at every cloudy point
        _case("solve", "field", 96, 96, 48, 16, "open", 4, 48, 9, thermal=True, name="solve_thermal_96"),
        # I, Q, U on open and on periodic boundaries (polarimetric sensors)
        _case("solve", "polarized", 64, 64, 40, 8, "open", 10, 64, 9, stokes=3, name="solve_polarized_open"),
        _case("solve", "polarized", 64, 64, 40, 8, "periodic", 5, 32, 9, stokes=3, name="solve_polarized_periodic"),
        # images of a solved medium: a nine-view overflight, and one small sensor at a time
        _case("render", "field", 64, 64, 32, 8, "open", 6, 64, 9, fraction=0.2, name="render_views_64"),
        _case("sensor", "blob", 32, 32, 24, 8, "open", 6, 13, 1, rayleigh=True, name="render_sensor_13"),
        # the retrieval's gradient, and whole optimiser steps of a small retrieval
        _case("gradient", "field", 64, 64, 32, 8, "open", 6, 64, 9, fraction=0.2, name="gradient_64"),
        _case("retrieval", "field", 24, 24, 16, 8, "open", 6, 24, 5, fraction=0.3, name="retrieval_24"),
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    """One more case: the kind by its share of use, sizes over their logarithm.  Periodic boundaries cost the most
    per point (the sweep is sequential along each ordinate), so their grids stay smaller."""
    kind = rng.choice(["solve", "solve", "solve", "solve", "render", "sensor", "gradient", "retrieval"])
    boundary = rng.choice(["open", "open", "open", "periodic"])
    stokes = 3 if kind in ("solve", "render", "sensor") and rng.random() < 0.25 else 1
    thermal = kind == "solve" and stokes == 1 and rng.random() < 0.2
    scene = "polarized" if stokes == 3 else rng.choice(["field", "field", "blob"])
    nmu = rng.choice([8, 8, 8, 12, 16] if stokes == 1 and kind not in ("gradient", "retrieval") else [6, 8, 8])
    hi = 32 if kind == "retrieval" else 40 if boundary == "periodic" or stokes == 3 else 96
    nx, ny = _log_int(rng, 10, hi), _log_int(rng, 10, hi)
    nz = _log_int(rng, 9, 48 if boundary == "open" else 32)
    iters = 4 if thermal else rng.randint(4, 12) if kind == "solve" else 6
    npix = _log_int(rng, 5, 24 if kind == "retrieval" else 64)
    views = 1 if kind == "sensor" else rng.randint(1, len(VIEW_ZENITHS))
    return _case(kind, scene, nx, ny, nz, nmu, boundary, iters, npix, views, stokes=stokes, thermal=thermal,
                 rayleigh=scene != "polarized" and rng.random() < 0.4, fraction=round(rng.uniform(0.1, 0.5), 3))


def _problem(case, seed):
    c = case
    grid = dict(nx=c["nx"], ny=c["ny"], nz=c["nz"], boundary=c["boundary"], nmu=c["nmu"], nphi=c["nphi"], solacc=_SOLACC)
    if c["scene"] == "polarized":
        return polarized_blob(seed=seed, **grid)
    if c["scene"] == "blob":
        pb = cloud_blob(seed=seed, **grid)
        if not c["rayleigh"]:
            del pb.species[1]
    else:
        w = seed % len(FIELD_SSA)  # the wavelength of the four-wavelength set
        pb = cloud_field(seed=seed, wavelength_index=w, fraction=c["fraction"], nleg=8 * c["nmu"], **grid)
        if c["rayleigh"]:
            ext = pb.species[0].extinction
            pb.species.append(Species(extinction=np.full_like(ext, 0.01), ssalb=np.ones_like(ext),
                                      legcoef=rayleigh_legcoef(0.86)))
    if c["thermal"]:
        # 11 um: absorbing cloud, 290 K at the ground with a 6.5 K/km lapse rate, warm ground, cold sky
        nx, ny, nz = pb.shape
        pb.species[0].ssalb = (np.asarray(pb.species[0].ssalb, np.float32) * 0.55).astype(np.float32)
        X, _, Z = np.meshgrid(np.arange(nx) * pb.delx, np.arange(ny) * pb.dely, pb.zlevels, indexing="ij")
        pb.temperature = (290.0 - 6.5 * Z + 4.0 * np.sin(2 * np.pi * X / (nx * pb.delx))).astype(np.float32)
        pb.srctype, pb.wavelength, pb.solarflux, pb.skyrad = "T", 11.0, 0.0, 0.0
        pb.ground_temperature, pb.surface_albedo = 295.0, 0.05
    return pb


def _perspective(pb, npix):
    """A small camera above the domain centre: one ray per pixel, directions fanning out over 40 degrees."""
    nx, ny, nz = pb.shape
    a = np.deg2rad(np.linspace(-20.0, 20.0, npix))
    tx, ty = (t.ravel() for t in np.meshgrid(np.tan(a), np.tan(a), indexing="ij"))
    mu = 1.0 / np.sqrt(1.0 + tx * tx + ty * ty)
    phi = np.arctan2(-ty, -tx)
    n = tx.size
    return (np.full(n, 0.5 * nx * pb.delx), np.full(n, 0.5 * ny * pb.dely), np.full(n, float(pb.zlevels[-1]) * 1.25), mu, phi)


def _device(rays):
    return [torch.as_tensor(np.ascontiguousarray(r), dtype=torch.float32 if i < 3 else torch.float64).cuda()
            for i, r in enumerate(rays)]


def prepare(case, seed):
    pb = _problem(case, seed)
    rays = (_perspective(pb, case["npix"]) if case["kind"] == "sensor"
            else orthographic_views(pb, case["npix"], case["npix"], zeniths=VIEW_ZENITHS[:case["views"]]))
    state = {"case": case, "rte": RTE.from_problem(pb), "rays": rays, "nrays": len(rays[0])}
    kind = case["kind"]
    if kind in ("render", "sensor", "gradient"):
        state["rte"].solve(case["iters"], verbose=False)
    if kind in ("solve", "render"):
        state["drays"] = _device(rays)
    elif kind == "sensor":
        state["sensor"] = dict(zip(("ray_x", "ray_y", "ray_z", "ray_mu", "ray_phi"), rays))
    else:
        rng = np.random.default_rng(seed + 1)
        ext, alb = state["rte"].species_properties(0)
        state["noise"] = torch.as_tensor(1.0 + 0.1 * rng.standard_normal(state["nrays"]), dtype=torch.float32).cuda()
        if kind == "gradient":
            state["media"] = [(torch.as_tensor(ext).cuda().requires_grad_(), torch.as_tensor(alb).cuda().requires_grad_())]
            with torch.no_grad():
                image = torch.empty(state["nrays"], dtype=torch.float32, device="cuda")
                _render(state["rte"], _device(rays), image)
            state["measured"] = image * state["noise"]
        else:
            state["media"] = [(torch.as_tensor(ext * f).cuda().requires_grad_(), torch.as_tensor(alb).cuda().requires_grad_())
                              for f in (0.9, 1.1)]
            state["measured"] = 0.3 * state["noise"]
    torch.cuda.synchronize()
    return state


def _render(rte, drays, out):
    rte.render_device(*(t.data_ptr() for t in drays), out.data_ptr(), drays[0].numel(),
                      torch.cuda.current_stream().cuda_stream)


def run(state):
    case, rte = state["case"], state["rte"]
    kind = case["kind"]
    if kind in ("solve", "render"):
        if kind == "solve":
            rte.solve(case["iters"], verbose=False)
        n, nst = state["nrays"], case["stokes"]
        image = torch.empty((n, nst) if nst > 1 else n, dtype=torch.float32, device="cuda")
        _render(rte, state["drays"], image)
        return image
    if kind == "sensor":
        sensor = rte.integrate_to_sensor(dict(state["sensor"]))
        return {k: sensor[k] for k in ("I", "Q", "U") if k in sensor}
    out = []
    for ext, alb in state["media"]:
        ext.grad = alb.grad = None
        image = render_differentiable(rte, ext, alb, state["rays"], maxiter=case["iters"])
        loss = 0.5 * (image - state["measured"]).square().sum()
        loss.backward()
        out.append({"image": image.detach(), "extinction": ext.grad, "albedo": alb.grad})
    return out


def work(case):
    """Bytes: per solution iteration the source, its increment and the radiance series, each read and written once
    where the medium scatters, and the two hemispheric fluxes; per ray its description and radiance; the source and
    the medium once per image.  Operations: per iteration the two transforms in factorised form and the cell
    integral of each point and ordinate; per ray and crossed cell the four new corners' series and the cell integral."""
    c = case
    open_ = 1 if c["boundary"] == "open" else 0
    nx, ny = c["nx"] + 1 + open_, c["ny"] + 1 + open_
    npts = nx * ny * c["nz"]
    nmu, nphi, nst = c["nmu"], c["nphi"], c["stokes"]
    nlm, nang = nmu * nmu, int(1.4 * nmu * nmu)
    scat = 1.0 if c["rayleigh"] or c["scene"] != "field" else min(1.0, 1.1 * c["fraction"])
    it_bytes = 4.0 * npts * (6 * nlm * nst * scat + 2)
    it_flops = npts * nst * (scat * 4.0 * (nlm * nmu + nmu * nphi * nphi) + 40.0 * nang)
    rays = c["views"] * c["npix"] ** 2
    cells = nx + c["nz"]
    img_bytes = rays * (28.0 + 4 * nst) + 4.0 * npts * (nlm * nst * scat + 4)
    img_flops = rays * cells * (4.0 * 2 * nlm * nst * scat + 200.0)
    solves, images = {"solve": (1, 1), "render": (0, 1), "sensor": (0, 1), "gradient": (0, 3), "retrieval": (2, 6)}[c["kind"]]
    grad_bytes = {"gradient": 1, "retrieval": 2}.get(c["kind"], 0) * 4.0 * (npts * (nlm + 2) * scat + 4 * c["nx"] * c["ny"] * c["nz"])
    if c["kind"] == "sensor":  # one small camera reads only what its rays cross
        img_bytes = rays * (28.0 + 4 * nst + cells * 4 * 4.0 * nlm * nst * scat)
    return {"bytes": solves * c["iters"] * it_bytes + images * img_bytes + grad_bytes,
            "flops": solves * c["iters"] * it_flops + images * img_flops}


def exact(case, seed):
    """None: these outputs are whole solutions of the coupled transport problem on 1e3 to 1e6 points and 1e2
    ordinates (or images and derivatives of them); a 64-bit solve in array code takes minutes to hours."""
    return None
