"""The calls whose speed matters: what a user of the sky tracer has it do, through its public Python entry points.

A case is a dict with a "kind":

  render   one image of a resident scene (GpuScene.render / render_xyz / render_device) or of host tables (render)
  sweep    one image per sun elevation, all in one launch (Sweep: a replayed CUDA graph, or a queued batch)
  adjoint  one differentiable render and its gradient (render_film, render_films, torch autograd)
  score    the Oklab score of candidate primary bands over the samples of baked images (score_combos)
  mie      the phase table of one aerosol species (bake_phase)
"""

import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "sky-tracer_gb300") not in sys.path:
    sys.path.insert(0, str(ROOT / "sky-tracer_gb300"))

import sky_cuda  # noqa: E402
from sky_cuda import GpuScene, RenderConfig, adjoint, mie, scoring, sweep  # noqa: E402

DATA = ROOT / "tests" / "golden" / "data"

TRACKING = {"restart": sky_cuda.TRACKING_SEGMENT_RESTART, "carry": sky_cuda.TRACKING_RESIDUAL_CARRY,
            "merged": sky_cuda.TRACKING_MERGED_LAYERS}
PHASE = {"isotropic": sky_cuda.PHASE_ISOTROPIC, "tabulated": sky_cuda.PHASE_TABULATED}
PROJECTION = {"panorama": sky_cuda.PROJECTION_PANORAMA, "lut": sky_cuda.PROJECTION_SKY_VIEW_LUT}

# FP32 work of one chain (camera ray, its scattering vertices with their sun rays, tracking steps), from the event
# counts of the 512x256, 81-wavelength render and the arithmetic of each event in the reference shader.
FLOPS_PER_CHAIN = 800.0


def _render(name, tables, api, width, height, bands, spp, elevation, tracking="merged", phase="tabulated",
            projection="panorama", rr=8):
    return {"name": name, "kind": "render", "tables": tables, "api": api, "width": width, "height": height,
            "bands": bands, "spp": spp, "elevation": elevation, "tracking": tracking, "phase": phase,
            "projection": projection, "rr": rr}


def listed():
    return [
        # the reference's own smoke image with its default settings: a call as small as they come
        _render("smoke-32x16-2spp", "reference", "film", 32, 16, 41, 2, 0.0, "restart", "isotropic", rr=0),
        # a small image, rendered again and again while a scene is set up
        _render("small-64x32-32wl-64spp", "synthetic", "xyz", 64, 32, 32, 64, 10.0),
        # the same image by the drop-in render(scene, config): host tables in, host film out, nothing kept
        _render("one-shot-64x32-32wl-64spp", "synthetic", "once", 64, 32, 32, 64, 10.0),
        # the reference's tables and its default settings (layer by layer tracking, isotropic phase sampling)
        _render("reference-default-128x64-64spp", "reference", "film", 128, 64, 41, 64, 20.0, "restart", "isotropic",
                rr=0),
        # a sky-view LUT of the reference's tables (four aerosol species), as its baking script makes them
        _render("reference-lut-256x256-32spp", "reference", "xyz", 256, 256, 41, 32, 30.0, projection="lut"),
        # one pass of a progressive preview of an odd window: few samples per pixel, all of the image's outputs
        _render("preview-509x251-79wl-3spp", "synthetic", "device", 509, 251, 79, 3, 15.0),
        # the production image
        _render("production-512x256-81wl-256spp", "synthetic", "device", 512, 256, 81, 256, 5.0),
        # LUTs over the day in one launch, the noisy low suns with more samples
        {"name": "sweep-16x128x64-40wl", "kind": "sweep", "api": "graph", "elevations": 16, "width": 128, "height": 64,
         "bands": 40, "spp_low": 64, "spp_high": 512},
        # an image and its gradient with respect to the atmosphere's layers, as a fit to a measured sky takes them
        {"name": "adjoint-128x64-32wl-64spp", "kind": "adjoint", "api": "film", "renders": 1, "width": 128,
         "height": 64, "bands": 32, "spp": 64, "band_params": False, "decorrelate": False, "projection": "panorama"},
        # one step of the fit of four primaries to sixteen elevations
        {"name": "fit-step-16x256x128-4wl-32spp", "kind": "adjoint", "api": "films", "renders": 16, "width": 256,
         "height": 128, "bands": 4, "spp": 32, "band_params": True, "decorrelate": True, "projection": "lut"},
        # candidate sets of four bands scored over ten 256x256 LUTs
        {"name": "score-655360x128", "kind": "score", "bands": 41, "samples": 655360, "combos": 128, "channels": 4},
        # one species of the reference's phase-table bake
        {"name": "mie-waso-41x1024", "kind": "mie", "species": "waso", "bands": 41, "bins": 1024, "radii": 300},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "sweep", "adjoint", "score", "mie"])
    if kind == "render":
        tables = rng.choice(["synthetic", "synthetic", "reference"])
        tracking = rng.choice(["merged", "merged", "restart", "carry"])
        width = _log(rng, 8, 640)
        c = _render("", tables, rng.choice(["film", "xyz", "device", "once"]), width, max(4, width // 2 + rng.randint(-3, 3)),
                    41 if tables == "reference" else _log(rng, 1, 81), _log(rng, 1, 256), rng.uniform(0.0, 80.0),
                    tracking, rng.choice(["tabulated", "tabulated", "isotropic"]),
                    rng.choice(["panorama", "lut"]), rng.choice([0, 8]))
        most = 6e8 if tracking == "merged" else 3e7
        while c["width"] * c["height"] * c["bands"] * c["spp"] > most:
            c["spp" if c["spp"] > 1 else "width"] //= 2
        del c["name"]
        return c
    if kind == "sweep":
        width = _log(rng, 24, 256)
        low = _log(rng, 8, 64)
        c = {"kind": "sweep", "api": rng.choice(["graph", "batch"]), "elevations": rng.randint(3, 16), "width": width,
             "height": max(4, width // 2 + rng.randint(-2, 2)), "bands": _log(rng, 1, 60), "spp_low": low,
             "spp_high": low * rng.randint(2, 12)}
        while c["elevations"] * c["width"] * c["height"] * c["bands"] * c["spp_high"] > 6e8:
            c["spp_low"], c["spp_high"] = max(1, c["spp_low"] // 2), max(2, c["spp_high"] // 2)
            if c["spp_high"] == 2:
                c["bands"] = max(1, c["bands"] // 2)
        return c
    if kind == "adjoint":
        renders = rng.choice([1, 1, rng.randint(2, 16)])
        width = _log(rng, 16, 192)
        c = {"kind": "adjoint", "api": "film" if renders == 1 else "films", "renders": renders, "width": width,
             "height": max(4, width // 2 + rng.randint(-2, 2)), "bands": _log(rng, 1, 40), "spp": _log(rng, 4, 96),
             "band_params": rng.random() < 0.5, "decorrelate": rng.random() < 0.5,
             "projection": rng.choice(["panorama", "lut"])}
        while c["renders"] * c["width"] * c["height"] * c["bands"] * c["spp"] > 6e7 and c["spp"] > 1:
            c["spp"] //= 2
        return c
    if kind == "score":
        samples, combos = _log(rng, 2000, 700000), _log(rng, 1, 256)
        return {"kind": "score", "bands": rng.randint(3, 41), "samples": samples,
                "combos": max(1, min(combos, 90000000 // samples)), "channels": rng.randint(1, 5)}
    return {"kind": "mie", "species": rng.choice(sorted(mie.OPAC_SPECIES)), "bands": rng.randint(1, 41),
            "bins": _log(rng, 64, 1024), "radii": _log(rng, 40, 300)}


def _tables(case, elevation):
    if case.get("tables") == "reference":
        return sky_cuda.load_scene_data(DATA, elevation, 0.0, synthesize_missing_mie_g=0.76)
    return sky_cuda.synthetic_scene(sky_cuda.wavelengths(380.0, 780.0, case["bands"]), DATA,
                                    sun_elevation_deg=elevation)


def _prepare_render(case, rng, seed):
    elevation = case["elevation"] + float(rng.uniform(0.0, 1.0))
    scene = _tables(case, elevation)
    config = RenderConfig(width=case["width"], height=case["height"], spp=case["spp"],
                          seed=int(rng.integers(1, 1 << 62)), sun_elevation_deg=elevation,
                          output_projection=PROJECTION[case["projection"]], phase_sampling=PHASE[case["phase"]],
                          tracking=TRACKING[case["tracking"]], rr_start_depth=case["rr"])
    state = {"case": case, "scene": scene, "config": config}
    if case["api"] != "once":
        state["gpu"] = GpuScene(scene)
    if case["api"] == "device":
        cells, pixels = config.pixels * scene.band_count, config.pixels
        state["out"] = {"cell_sum": torch.zeros(cells, dtype=torch.float64, device="cuda"),
                        "cell_sumsq": torch.zeros(cells, dtype=torch.float64, device="cuda"),
                        "film": torch.zeros(cells, dtype=torch.float32, device="cuda"),
                        "xyz": torch.zeros(pixels * 3, dtype=torch.float64, device="cuda"),
                        "xyz_var": torch.zeros(pixels * 3, dtype=torch.float64, device="cuda"),
                        "rgb": torch.zeros(pixels * 3, dtype=torch.float32, device="cuda"),
                        "status": torch.zeros(1, dtype=torch.int32, device="cuda")}
    return state


def _prepare_sweep(case, rng, seed):
    n = case["elevations"]
    scene = _tables(case, 10.0)
    gpu = GpuScene(scene)
    base = RenderConfig(width=case["width"], height=case["height"], seed=int(rng.integers(1, 1 << 62)),
                        output_projection=sky_cuda.PROJECTION_SKY_VIEW_LUT, phase_sampling=sky_cuda.PHASE_TABULATED,
                        tracking=sky_cuda.TRACKING_MERGED_LAYERS, rr_start_depth=8)
    elevations = sweep.elevation_schedule(n, -4.0, 85.0) + rng.uniform(0.0, 1.0)
    # budgets as the pilot gives them: most where the sun is low, in multiples of a warp's samples where that is less
    fall = np.exp(np.linspace(math.log(case["spp_high"]), math.log(case["spp_low"]), n))
    spp = np.maximum(1, np.round(fall)).astype(int)
    s = sweep.Sweep(gpu, base, elevations, spp)
    if case["api"] == "graph":
        s.capture()
    return {"case": case, "gpu": gpu, "sweep": s}


def _prepare_adjoint(case, rng, seed):
    scene = _tables(case, 10.0)
    gpu = GpuScene(scene)
    config = RenderConfig(width=case["width"], height=case["height"], spp=case["spp"],
                          seed=int(rng.integers(1, 1 << 62)), output_projection=PROJECTION[case["projection"]],
                          phase_sampling=sky_cuda.PHASE_TABULATED, tracking=sky_cuda.TRACKING_MERGED_LAYERS,
                          rr_start_depth=8)
    renderer = adjoint.AdjointRenderer(gpu, config)
    layer = np.concatenate([rng.uniform(0.8, 1.2, renderer.param_count - 2), [0.9, 0.76]])
    band = rng.uniform(0.9, 1.1, (renderer.bands, adjoint.BAND_PARAMS))
    film = (case["renders"], config.rows, config.width, renderer.bands)
    gradient = rng.standard_normal(film).astype(np.float32) / math.prod(film)
    suns = [sky_cuda.sun_from_degrees(float(e), 0.0, scene.sun_angular_radius_rad)[0]
            for e in sweep.elevation_schedule(case["renders"], 2.0, 88.0) + rng.uniform(0.0, 1.0)]
    return {"case": case, "gpu": gpu, "renderer": renderer, "suns": suns,
            "layer": torch.tensor(layer.astype(np.float32), device="cuda", requires_grad=not case["band_params"]),
            "band": torch.tensor(band.astype(np.float32), device="cuda", requires_grad=True)
            if case["band_params"] else None,
            "gradient": torch.tensor(gradient, device="cuda")}


def _prepare_score(case, rng, seed):
    n, bands = case["samples"], case["bands"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    # smooth spectra over a few decades of brightness, as the pixels of baked skies have them
    lam = torch.linspace(0.0, 1.0, bands, device="cuda")[:, None]
    bright = torch.exp(torch.randn(n, generator=gen, device="cuda") * 1.2)
    tilt = torch.randn(n, generator=gen, device="cuda")
    hump = torch.rand(n, generator=gen, device="cuda")
    spectra = bright * torch.exp(-0.7 * tilt * (lam - 0.5)) * (1.0 + 0.5 * torch.cos(6.0 * (lam - hump)))
    weights = rng.uniform(0.0, 1.0, (bands, 3)) / bands
    reference = spectra.double().T.cpu().numpy() @ weights
    picks = np.stack([np.sort(rng.permutation(max(bands, case["channels"]))[:case["channels"]] % bands)
                      for _ in range(case["combos"])])
    xyz = rng.uniform(0.0, 1.0, (case["combos"], case["channels"], 3)) / case["channels"]
    return {"case": case, "spectra": spectra.float().contiguous(), "reference": reference,
            "picks": picks.astype(np.uint32), "xyz": xyz.astype(np.float32)}


def _prepare_mie(case, rng, seed):
    d = mie.OPAC_SPECIES[case["species"]]
    lam = np.linspace(380.0, 780.0, case["bands"]) + rng.uniform(0.0, 1.0)
    index = rng.uniform(1.4, 1.6) + np.linspace(0.0, 0.02, case["bands"]) + 1j * rng.uniform(0.001, 0.02)
    dist = mie.MieDistribution(d.r_mode_um, d.sigma_g, d.r_min_um, d.r_max_um, case["radii"])
    return {"case": case, "dist": dist, "lam": lam, "index": index}


_PREPARE = {"render": _prepare_render, "sweep": _prepare_sweep, "adjoint": _prepare_adjoint, "score": _prepare_score,
            "mie": _prepare_mie}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, np.random.default_rng(int(seed)), seed)


def run(state):
    case = state["case"]
    if case["kind"] == "render":
        if case["api"] == "once":
            return sky_cuda.render(state["scene"], state["config"]).values
        if case["api"] == "film":
            return state["gpu"].render(state["config"])[0].values
        if case["api"] == "xyz":
            film, xyz, var, _ = state["gpu"].render_xyz(state["config"])
            return {"film": film.values, "xyz": xyz, "xyz_var": var}
        out = state["out"]
        state["gpu"].render_device(state["config"], {k: t.data_ptr() for k, t in out.items()},
                                   torch.cuda.current_stream().cuda_stream)
        return out
    if case["kind"] == "sweep":
        s, stream = state["sweep"], torch.cuda.current_stream().cuda_stream
        if case["api"] == "graph":
            s.replay(stream)
        else:
            s.launch(stream)
        return [{"cell_sum": o.cell_sum, "xyz": o.xyz, "xyz_var": o.xyz_var} for o in s.out] + [s.status]
    if case["kind"] == "adjoint":
        layer, band, renderer = state["layer"], state["band"], state["renderer"]
        if case["api"] == "film":
            film = adjoint.render_film(renderer, layer, band, sun=state["suns"][0], decorrelate=case["decorrelate"])[None]
        else:
            film = adjoint.render_films(renderer, layer, band, state["suns"], decorrelate=case["decorrelate"])
        wanted = band if case["band_params"] else layer
        return film, torch.autograd.grad(film, wanted, state["gradient"])[0]
    if case["kind"] == "score":
        scores = scoring.score_combos(state["spectra"], state["reference"], state["picks"], state["xyz"])
        return {f: np.array([s[f] for s in scores]) for f in scoring.FIELDS}
    phase, optics = mie.bake_phase(state["dist"], state["lam"], state["index"], case["bins"])
    return {"phase": phase, **optics}


def work(case):
    if case["kind"] in ("render", "sweep", "adjoint"):
        pixels = case["width"] * case["height"]
        if case["kind"] == "render":
            chains, out = pixels * case["bands"] * case["spp"], pixels * (4 * case["bands"] + 48)
        elif case["kind"] == "sweep":
            spp = np.exp(np.linspace(math.log(case["spp_high"]), math.log(case["spp_low"]), case["elevations"])).mean()
            chains = case["elevations"] * pixels * case["bands"] * float(spp)
            out = case["elevations"] * pixels * (8 * case["bands"] + 48)
        else:  # the film out and its gradient in; the gradient retraces the chains that carry radiance
            chains = 2 * case["renders"] * pixels * case["bands"] * case["spp"]
            out = 8 * case["renders"] * pixels * case["bands"]
        return {"bytes": out + 10000 * case["bands"], "flops": FLOPS_PER_CHAIN * chains}
    if case["kind"] == "score":
        distances = case["samples"] * case["combos"]
        return {"bytes": case["samples"] * (4 * case["bands"] + 24), "flops": distances * (6 * case["channels"] + 45)}
    # the series of a sphere of size parameter x has about x + 4 x^(1/3) + 2 terms: each some 120 operations for its
    # coefficients and 16 for every angle
    d = mie.OPAC_SPECIES[case["species"]]
    x = 2 * math.pi * np.geomspace(d.r_min_um, d.r_max_um, case["radii"]) / 0.55
    terms = case["bands"] * float(np.sum(x + 4.05 * x ** (1 / 3) + 2))
    return {"bytes": 8 * case["bands"] * (case["bins"] + 6), "flops": terms * (120 + 16 * case["bins"])}


def _exact_score(state):
    """Oklab distances of the rebuilt XYZ in 64 bits: mean, RMS and the sorted distances' elements round((n - 1) q)."""
    m1 = torch.tensor([[0.8189330101, 0.3618667424, -0.1288597137], [0.0329845436, 0.9293118715, 0.0361456387],
                       [0.0482003018, 0.2643662691, 0.6338517070]], dtype=torch.float64, device="cuda")
    m2 = torch.tensor([[0.2104542553, 0.7936177850, -0.0040720468], [1.9779984951, -2.4285922050, 0.4505937099],
                       [0.0259040371, 0.7827717662, -0.8086757660]], dtype=torch.float64, device="cuda")

    def lab(xyz):
        lms = xyz @ m1.T
        return (torch.sign(lms) * lms.abs() ** (1.0 / 3.0)) @ m2.T

    reference = torch.tensor(state["reference"], device="cuda")
    n = reference.shape[0]

    def at(q):
        return int(math.floor((n - 1) * q + 0.5))

    scale = max(float(torch.sort(reference[:, 1]).values[at(0.99)]), 1e-12)
    target, rows = lab(reference / scale), []
    for picks, xyz in zip(state["picks"].astype(np.int64), state["xyz"]):
        rebuilt = state["spectra"][torch.tensor(picks, device="cuda")].double().T @ torch.tensor(xyz, device="cuda").double()
        d = torch.sort((lab(rebuilt / scale) - target).norm(dim=1)).values
        rms, mean = float((d * d).mean().sqrt()), float(d.mean())
        q = [float(d[at(p)]) for p in (0.5, 0.9, 0.95, 0.99, 1.0)]
        rows.append([mean, rms, *q, rms + 0.25 * q[2], n])
    columns = dict(zip(scoring.FIELDS, np.array(rows).T))
    columns["finite"] = None
    return columns


def _exact_mie(state, bins):
    """The Mie series (Bohren and Huffman 1983, appendix A) of every sphere in 64 bits, averaged over the radii."""
    dist, lam = state["dist"], state["lam"] * 1e-3
    r = np.geomspace(dist.r_min_um, dist.r_max_um, dist.radii)
    w = np.exp(-np.log(r / dist.r_mode_um) ** 2 / (2.0 * math.log(dist.sigma_g) ** 2))
    w = torch.tensor(w / w.sum(), device="cuda")
    u = (torch.arange(bins, dtype=torch.float64, device="cuda") + 0.5) / bins
    mu = 1.0 - 2.0 * u ** 3
    area = torch.tensor(np.pi * r * r, device="cuda") * w
    phase, optics = [], []
    for wavelength, index in zip(lam, state["index"]):
        k = 2.0 * math.pi / wavelength
        x = torch.tensor(k * r, device="cuda")
        terms = torch.floor(x + 4.05 * x ** (1.0 / 3.0) + 2.0)
        most = int(terms.max())
        mx = x * complex(index)
        start = max(most, int(mx.abs().max())) + 16
        d = torch.zeros_like(mx)
        ds = [None] * (start + 1)
        for n in range(start, 0, -1):
            t = n / mx
            d = t - 1.0 / (d + t)
            ds[n - 1] = d
        psi0, psi1, chi0, chi1 = torch.cos(x), torch.sin(x), -torch.sin(x), torch.cos(x)
        xi1 = torch.complex(psi1, -chi1)
        pi0, pi1 = torch.zeros_like(mu)[None], torch.ones_like(mu)[None]
        s1 = torch.zeros((len(r), bins), dtype=torch.complex128, device="cuda")
        s2 = torch.zeros_like(s1)
        sca, ext, asym = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)
        before = None
        for n in range(1, most + 1):
            psi, chi = (2 * n - 1) * psi1 / x - psi0, (2 * n - 1) * chi1 / x - chi0
            xi = torch.complex(psi, -chi)
            ta, tb = ds[n] / complex(index) + n / x, ds[n] * complex(index) + n / x
            on = n <= terms
            a = torch.where(on, (psi * ta - psi1) / (ta * xi - xi1), 0.0)
            b = torch.where(on, (psi * tb - psi1) / (tb * xi - xi1), 0.0)
            sca += (2 * n + 1) * (a.abs() ** 2 + b.abs() ** 2)
            ext += (2 * n + 1) * (a + b).real
            asym += (2 * n + 1) / (n * (n + 1)) * (a * b.conj()).real
            if before is not None:
                asym += (n - 1) * (n + 1) / n * (before[0] * a.conj() + before[1] * b.conj()).real
            before = (a, b)
            f = (2 * n + 1) / (n * (n + 1))
            tau = n * mu * pi1 - (n + 1) * pi0
            m = int((terms >= n).sum())  # the larger spheres are the last ones
            s1[-m:] += f * (a[-m:, None] * pi1 + b[-m:, None] * tau)
            s2[-m:] += f * (a[-m:, None] * tau + b[-m:, None] * pi1)
            pi0, pi1 = pi1, ((2 * n + 1) * mu * pi1 - (n + 1) * pi0) / n
            psi0, psi1, chi0, chi1 = psi1, psi, chi1, chi
            xi1 = torch.complex(psi1, -chi1)
        q_sca, q_ext = 2.0 * sca / x ** 2, 2.0 * ext / x ** 2
        total, g = (area * q_sca).sum(), (area * 4.0 * asym / x ** 2).sum()
        intensity = (w[:, None] * (s1.abs() ** 2 + s2.abs() ** 2)).sum(0) / (2.0 * k * k)
        phase.append((intensity / total).cpu().numpy())
        optics.append((float(total), float((area * q_ext).sum()), float(g / total)))
    optics = np.array(optics).T
    return {"phase": np.array(phase), "sigma_sca_um2": optics[0], "sigma_ext_um2": optics[1], "g": optics[2]}


def exact(case, seed):
    # an image is a sum over random paths: in 64 bits the same random numbers take other paths
    if case["kind"] == "score":
        return _exact_score(prepare(case, seed))
    if case["kind"] == "mie":
        return _exact_mie(prepare(case, seed), case["bins"])
    return None
