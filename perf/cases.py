"""Timing cases of the framework's main paths, through its public Python API.

listed() names the work a program does with this framework: single patterns
(small, ordinary, large, ragged), orientation and molecule batches, a
refinement step, a polychromatic pattern, the NUFFT forms, the detector chain
and the reference-facing simulate_shot call on host buffers.  draw() gives
more cases of the same ranges.  exact() restates each result in 64 bits with
plain torch, from the published formulas and coefficients alone.

A case is a dict of plain values: "kind" selects the entry point; lengths are
in nm (molecule radius, wavelength), um (pixels, detector centre) and m
(detector distance).
"""
import math

import numpy as np
import torch

from spsim_b200 import autograd, core, synth
from spsim_b200 import spsim as S


# ----------------------------------------------------------------- the cases

def _case(name, kind, natoms, radius, nx, ny, pixel, distance, wavelength, **more):
    c = dict(name=name, kind=kind, natoms=natoms, radius_nm=radius, nx=nx, ny=ny, pixel_um=pixel, distance_m=distance,
             wavelength_nm=wavelength)
    c.update(more)
    return c


def listed():
    return [
        # the plain workload: one small protein on a small detector, a call a
        # script or an interactive loop makes thousands of times (latency)
        _case("plain_1k", "forward", 1000, 2.5, 256, 256, 75.0, 0.15, 0.25),
        # the precision workload: a large particle on a full detector, pattern
        # and noiseless photons, the ordinary production call
        _case("pattern_50k", "pattern", 50000, 12.0, 1024, 1024, 75.0, 0.1, 0.15),
        # an odd detector panel off the beam axis, rotated, with a B factor,
        # in the fast mode
        _case("panel_7k_fast", "forward", 7001, 5.1, 517, 389, 110.0, 0.13, 0.17, precision="f32_fast", rotated=True,
              B=12.5, center_um=9000.0),
        # many orientations of one particle in one call (simulated datasets,
        # orientation recovery)
        _case("orientations_20k", "batch", 20000, 8.0, 256, 256, 150.0, 0.2, 0.2, npat=128),
        # molecules of uneven sizes, each on its own detector, in one call
        dict(name="uneven_16", kind="uneven", n_mol=16, nmin=500, nmax=60000, mix=1003),
        # one step of a refinement: forward and gradient with respect to
        # positions, occupancies and B factors over a few orientations
        _case("refine_5k", "refine", 5000, 4.0, 512, 512, 75.0, 0.15, 0.25, npat=8),
        # a bandwidth-broadened beam
        _case("spectrum_3k", "spectrum", 3000, 3.2, 320, 300, 100.0, 0.12, 0.2, bandwidth=0.02, samples=5),
        # the plain FP64 kernel (checks, small molecules)
        _case("fp64_2k", "forward", 2000, 3.0, 256, 256, 75.0, 0.15, 0.2, precision="fp64"),
        # the NUFFT structure factor, one pattern and an orientation batch
        _case("nufft_50k", "nufft", 50000, 12.0, 1024, 1024, 75.0, 0.1, 0.15),
        _case("nufft_orient_20k", "nufft_batch", 20000, 8.0, 256, 256, 150.0, 0.2, 0.2, npat=128),
        # the detector chain alone, every output, noise on
        _case("chain_1536", "chain", 0, 0.0, 1536, 1030, 75.0, 0.1, 0.15, binning=1),
        # the reference-facing call with host buffers, chain and noise included
        _case("shot_10k", "shot", 10000, 6.5, 512, 480, 75.0, 0.12, 0.15),
    ]


MOST_TERMS = 1.6e11  # atom.pixel terms of the largest listed case


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _molecule_size(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    density = rng.uniform(7.0, 50.0)  # atoms per nm^3: the workloads' particles
    return n, (3 * n / (4 * math.pi * density)) ** (1.0 / 3.0)


def draw(rng):
    kind = rng.choice(["forward", "forward", "pattern", "batch", "uneven", "refine", "spectrum", "nufft", "nufft_batch",
                       "chain", "shot"])
    if kind == "uneven":
        return dict(kind=kind, n_mol=rng.randrange(3, 13), nmin=500, nmax=_log_int(rng, 4000, 60000),
                    mix=rng.randrange(1, 10 ** 6))
    atoms = {"forward": (200, 50000), "pattern": (2000, 50000), "batch": (500, 20000), "refine": (300, 5000),
             "spectrum": (300, 8000), "nufft": (2000, 50000), "nufft_batch": (2000, 20000), "chain": (1, 1),
             "shot": (500, 20000)}[kind]
    side = {"forward": (64, 1024), "pattern": (256, 1024), "batch": (96, 320), "refine": (96, 512),
            "spectrum": (96, 400), "nufft": (128, 1024), "nufft_batch": (96, 320), "chain": (200, 1536),
            "shot": (96, 720)}[kind]
    n, radius = _molecule_size(rng, *atoms)
    nx, ny = _log_int(rng, *side), _log_int(rng, *side)
    if rng.random() < 0.5:  # square, a multiple of four
        nx = ny = max(4, nx // 4 * 4)
    c = dict(kind=kind, natoms=n, radius_nm=radius, nx=nx, ny=ny, pixel_um=rng.choice([75.0, 110.0, 150.0]),
             distance_m=round(rng.uniform(0.1, 0.2), 3), wavelength_nm=round(rng.uniform(0.1, 0.3), 4))
    if kind in ("batch", "refine", "nufft_batch"):
        most = {"batch": 128, "refine": 8, "nufft_batch": 128}[kind]
        c["npat"] = max(1, min(_log_int(rng, 2, most), int(MOST_TERMS / (float(n) * nx * ny))))
    if kind in ("forward", "batch"):
        c["precision"] = rng.choice(["f32", "f32", "f32", "f32_fast"])
        if kind == "forward" and float(n) * nx * ny < 1e9 and rng.random() < 0.2:
            c["precision"] = "fp64"
    if kind == "forward":
        c["rotated"] = rng.random() < 0.5
        c["B"] = rng.choice([0.0, 0.0, 20.0])
        c["center_um"] = rng.choice([0.0, 0.0, 6000.0])
        c["spherical"] = rng.random() < 0.15
    if kind == "spectrum":
        c["bandwidth"] = rng.choice([0.01, 0.02, 0.1])
        c["samples"] = rng.choice([3, 5, 7])
    if kind == "chain":
        c["binning"] = rng.choice([1, 1, 2, 3])
    return c


# ----------------------------------------------------------------- what a program has in hand

def _det(c):
    """Keyword arguments of a case's detector."""
    return dict(nx=c["nx"], ny=c["ny"], width=c["nx"] * c["pixel_um"] * 1e-6, height=c["ny"] * c["pixel_um"] * 1e-6,
                distance=c["distance_m"], wavelength=c["wavelength_nm"] * 1e-9,
                center_x=c.get("center_um", 0.0) * 1e-6, spherical=bool(c.get("spherical", False)))


def _atoms(c, seed):
    return synth.random_molecule(c["natoms"], c["radius_nm"] * 1e-9, seed)


def _rots(c, seed):
    return synth.haar_rotations(c.get("npat", 1), seed + 7)


def _occ_b(n, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 11))
    return rng.uniform(0.5, 1.0, n).astype(np.float32), rng.uniform(0.0, 30.0, n).astype(np.float32)


def _chain_values(c, seed):
    """Chain parameters of a detector with readout noise (the arguments of core.chain_params)."""
    d = _det(c)
    b = c.get("binning", 1)
    return dict(nx=d["nx"], ny=d["ny"], width=d["width"], height=d["height"], distance=d["distance"],
                pixel_width=c["pixel_um"] * 1e-6, pixel_height=c["pixel_um"] * 1e-6, wavelength=d["wavelength"],
                beam_intensity=1e30, quantum_efficiency=1.0, electron_hole_production_energy=5.8e-19, readout_noise=10.0,
                linear_full_well=2e5, maximum_value=65535.0, exposure_time=1e-3, dark_current=0.0, binning_x=b,
                binning_y=b, polarization=3, seed=1234 + seed)


def _chain_intensity(c, seed):
    """Speckle intensities falling off from the beam: photon means from under one to thousands."""
    g = torch.Generator(device="cuda").manual_seed(seed + 5)
    y = torch.linspace(-1, 1, c["ny"], device="cuda")[:, None]
    x = torch.linspace(-1, 1, c["nx"], device="cuda")[None, :]
    envelope = 10.0 ** (8.0 - 5.0 * torch.sqrt(x * x + y * y))
    speckle = -torch.log(torch.rand(c["ny"], c["nx"], generator=g, device="cuda").clamp_min(1e-6))
    return (envelope * speckle).reshape(-1).float()


def _shifted(pos, seed):
    """Positions displaced by N(0, 0.5 Angstrom): the structure a refinement's data came from."""
    rng = np.random.Generator(np.random.PCG64(seed + 13))
    return (pos.astype(np.float64) + rng.normal(0.0, 0.5e-10, pos.shape)).astype(np.float32)


def _refine_target(c, seed):
    """Poisson counts at a mean of 100 photons per pixel from the displaced structure."""
    Z, pos = _atoms(c, seed)
    occ, b = _occ_b(len(Z), seed)
    q = _q64(_det(c))
    p = torch.as_tensor(_shifted(pos, seed).astype(np.float64), device="cuda")
    I = torch.stack([_amplitude(Z, p, q @ torch.as_tensor(R, device="cuda").T, occ, b).abs().square()
                     for R in _rots(c, seed)])
    g = torch.Generator(device="cuda").manual_seed(seed + 17)
    return torch.poisson((I * (100.0 / I.mean())).float(), generator=g)


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = {"case": c}
    if kind == "uneven":
        st["mols"], st["qsets"] = [], []
        for k, m in enumerate(_uneven(c)):
            Z, pos = synth.random_molecule(m["natoms"], m["radius"], seed * 1000 + k)
            st["mols"].append(core.Molecule(Z, pos))
            st["qsets"].append(core.QSet.from_detector(**m["det"]))
        st["F"] = [torch.empty(q.npix, dtype=torch.complex64, device="cuda") for q in st["qsets"]]
        st["I"] = [torch.empty(q.npix, dtype=torch.float32, device="cuda") for q in st["qsets"]]
        return st
    if kind == "chain":
        st["I"] = _chain_intensity(c, seed)
        st["chain"] = core.chain_params(**_chain_values(c, seed))
        return st
    Z, pos = _atoms(c, seed)
    if kind == "shot":
        opts = S.set_defaults()
        o = opts.contents
        det, exp = o.detector.contents, o.experiment.contents
        d = _det(c)
        det.nx, det.ny, det.nz = d["nx"], d["ny"], 1
        det.width, det.height, det.distance = d["width"], d["height"], d["distance"]
        det.pixel_width = det.pixel_height = c["pixel_um"] * 1e-6
        det.quantum_efficiency, det.electron_hole_production_energy = 1.0, 5.8e-19
        det.readout_noise, det.linear_full_well, det.maximum_value = 10.0, 2e5, 65535.0
        exp.wavelength, exp.beam_intensity, exp.exposure_time = d["wavelength"], 1e32, 1e-3
        o.random_orientation = 0
        o.euler_orientation[0] = o.euler_orientation[1] = o.euler_orientation[2] = 0.0
        o.verbosity_level = 0
        o.random_seed = 99 + seed
        st["opts"], st["mol"] = opts, S.get_molecule_from_atoms(Z, pos)
        return st
    st["qs"] = core.QSet.from_detector(**_det(c))
    n, npat = st["qs"].npix, c.get("npat", 1)
    if kind == "refine":
        occ, b = _occ_b(len(Z), seed)
        st["mol"] = core.Molecule(Z, pos, occ=occ, bfac=b)
        st["rots"] = _rots(c, seed)
        st["pos"] = torch.tensor(pos, device="cuda", requires_grad=True)
        st["occ"] = torch.tensor(occ, device="cuda", requires_grad=True)
        st["bfac"] = torch.tensor(b, device="cuda", requires_grad=True)
        st["counts"] = _refine_target(c, seed)
        return st
    st["mol"] = core.Molecule(Z, pos)
    if kind == "batch":
        st["rots"] = _rots(c, seed)
        st["I"] = torch.empty(npat, n, device="cuda")
        st["rows"] = list(st["I"].unbind(0))
        return st
    if kind == "nufft_batch":
        st["rots"] = _rots(c, seed)
        st["I"] = torch.empty(npat, n, device="cuda")
        return st
    if c.get("rotated"):
        st["rot"] = _rots(c, seed)[0]
    st["F"] = torch.empty(n, dtype=torch.complex64, device="cuda")
    st["I"] = torch.empty(n, device="cuda")
    if kind == "pattern":
        st["chain"] = core.chain_params(**_chain_values(c, seed))
    return st


# ----------------------------------------------------------------- one pass

CHAIN_DETERMINISTIC = ["photons_per_pixel", "noiseless_output"]


def run(st):
    c, kind = st["case"], st["case"]["kind"]
    if kind == "forward":
        return core.forward(st["mol"], st["qs"], rot=st.get("rot"), B=c.get("B", 0.0), precision=c.get("precision", "f32"),
                            F=st["F"], I=st["I"])
    if kind == "pattern":
        F, I = core.forward(st["mol"], st["qs"], F=st["F"], I=st["I"])
        return [F, I, core.detector_chain(st["chain"], I, outputs=CHAIN_DETERMINISTIC)]
    if kind == "batch":
        core.forward_batch(st["mol"], st["qs"], rots=st["rots"], precision=c.get("precision", "f32"), I=st["rows"],
                           want_F=False)
        return st["I"]
    if kind == "uneven":
        return list(core.forward_batch(st["mols"], st["qsets"], F=st["F"], I=st["I"]))
    if kind == "refine":
        for t in (st["pos"], st["occ"], st["bfac"]):
            t.grad = None
        I = autograd.intensity(st["mol"], st["qs"], st["pos"], st["occ"], st["bfac"], rots=st["rots"])
        # the photon scale refitted at every step, the likelihood summed in FP64
        scale = st["counts"].sum(dtype=torch.float64) / I.detach().sum(dtype=torch.float64)
        autograd.poisson_nll(I.double() * scale, st["counts"], eps=1e-6).backward()
        return [I.detach(), st["pos"].grad, st["occ"].grad, st["bfac"].grad]
    if kind == "spectrum":
        return core.forward_spectrum(st["mol"], st["qs"], c["wavelength_nm"] * 1e-9, c["bandwidth"], c["samples"],
                                     F=st["F"], I=st["I"])
    if kind == "nufft":
        return core.forward_nufft(st["mol"], st["qs"], F=st["F"], I=st["I"])
    if kind == "nufft_batch":
        return core.forward_nufft_batch(st["mol"], st["qs"], st["rots"], I=st["I"], want_F=False)[1]
    if kind == "chain":
        return core.detector_chain(st["chain"], st["I"])
    if kind == "shot":
        # the deterministic outputs: the noise streams advance from shot to shot
        shot = S.simulate_shot(st["mol"], st["opts"])
        det, n = st["opts"].contents.detector.contents, c["nx"] * c["ny"]
        out = {"F": S.as_array(shot.contents.F, n), "ints": S.as_array(shot.contents.ints, n),
               "photons": S.as_array(det.photons_per_pixel, n), "noiseless": S.as_array(det.noiseless_output, n)}
        S.free_stuff(shot, st["opts"])
        return out
    raise ValueError(kind)


# ----------------------------------------------------------------- bytes and operations

def _uneven(c):
    return synth.uneven_batch(seed=c["mix"], n_mol=c["n_mol"], nmin=c["nmin"], nmax=c["nmax"])


def work(case):
    """Bytes: atoms (20 B: position, weight, element) and other inputs read once,
    outputs written once.  Operations: of a direct sum 10 per atom.pixel term
    as the sum is defined (three products of the phase, two accumulations);
    of the NUFFT one FFT's over as many points as there are atoms and pixels;
    of the chain 100 per pixel (two Philox draws)."""
    c, kind = case, case["kind"]
    if kind == "uneven":
        terms = pix = atoms = 0
        for m in _uneven(c):
            p = m["det"]["nx"] * m["det"]["ny"]
            terms, pix, atoms = terms + float(p) * m["natoms"], pix + p, atoms + m["natoms"]
        return {"bytes": 20.0 * atoms + 12.0 * pix, "flops": 10.0 * terms}
    n, a, npat = float(c["nx"] * c["ny"]), float(c["natoms"]), c.get("npat", 1)
    if kind == "chain":
        return {"bytes": 4 * n + 20 * n + 8 * n / c.get("binning", 1) ** 2, "flops": 100 * n}
    if kind == "batch":
        return {"bytes": 20 * a + 4 * n * npat, "flops": 10 * a * n * npat}
    if kind == "refine":
        # I and the counts, dL/dI; 12 B positions and 4 B each of occupancies and B in, the same out
        return {"bytes": 40 * a + 12 * n * npat, "flops": 30 * a * n * npat}
    if kind == "spectrum":
        return {"bytes": 20 * a + 12 * n, "flops": 10 * a * n * (c["samples"] | 1)}
    if kind in ("nufft", "nufft_batch"):
        pts = a + n * npat
        return {"bytes": 20 * a + (12 if kind == "nufft" else 4) * n * npat, "flops": 5 * pts * math.log2(pts)}
    per_pixel = {"forward": 12, "pattern": 24, "shot": 12 + 8 + 28}[kind]
    return {"bytes": 20 * a + per_pixel * n, "flops": 10 * a * n}


# ----------------------------------------------------------------- the same in 64 bits

# Four-Gaussian form factors of the CCP4 atomsf.lib table, as floats: a1..a4, b1..b4, c.
FORM_FACTORS = {
    6: (2.31, 1.02, 1.5886, 0.865, 20.8439, 10.2075, 0.5687, 51.6512, 0.2156),
    7: (12.2126, 3.1322, 2.0125, 1.1663, 0.0057, 9.8933, 28.9975, 0.5826, -11.529),
    8: (3.0485, 2.2868, 1.5463, 0.867, 13.2771, 5.7011, 0.3239, 32.9089, 0.2508),
    16: (6.9053, 5.2034, 1.4379, 1.5863, 1.4679, 22.2151, 0.2536, 56.172, 0.8669),
}


def _f32(v):
    return float(np.float32(v))


def _q64(d):
    """Ewald-sphere q of every pixel (1/m), FP64 from the float arguments of the call."""
    nx, ny = d["nx"], d["ny"]
    w, h, dist, lam = (_f32(d[k]) for k in ("width", "height", "distance", "wavelength"))
    cx = _f32(d.get("center_x", 0.0))
    x = torch.arange(nx, dtype=torch.float64, device="cuda")
    y = torch.arange(ny, dtype=torch.float64, device="cuda")
    px = (((x - (nx - 1) / 2.0) / nx) * w - cx)[None, :].expand(ny, nx)
    py = (((y - (ny - 1) / 2.0) / ny) * h)[:, None].expand(ny, nx)
    if d.get("spherical"):
        sx, sy = float(np.float32(w) / np.float32(nx)), float(np.float32(h) / np.float32(ny))
        fx, fy = (2 * math.sin(math.atan(s / dist) / 2) / lam for s in (sx, sy))
        q = torch.stack([fx * px / sx, fy * py / sy, torch.zeros_like(px)], dim=-1)
    else:
        r = torch.sqrt(px * px + py * py + dist * dist)
        q = torch.stack([px / r / lam, py / r / lam, (dist / r - 1.0) / lam], dim=-1)
    return q.reshape(-1, 3)


def _form_factors(elements, q, B):
    s2 = (q * q).sum(1) * 1e-20 / 4
    rows = []
    for z in elements:
        k = [_f32(v) for v in FORM_FACTORS[int(z)]]
        f = k[8] * torch.exp(-B * s2)
        for i in range(4):
            f = f + k[i] * torch.exp(-(k[4 + i] + B) * s2)
        rows.append(f)
    return torch.stack(rows, dim=1), s2  # (pixels, elements)


def _blocks(npix, natoms):
    step = max(1, int(4e7) // max(1, natoms))
    return [(i, min(npix, i + step)) for i in range(0, npix, step)]


def _amplitude(Z, pos, q, occ=None, bfac=None, B=0.0, qscale=1.0, grad=None):
    """F(q) = sum_e f_e sum_j w_j exp(-B_j s^2) exp(-2 pi i q.r_j), complex128.
    With grad(i, j, I) = dL/dI of pixels i..j: also dL/dpos, dL/docc and dL/dB."""
    elements, which = np.unique(Z, return_inverse=True)
    p = torch.as_tensor(pos, dtype=torch.float64, device="cuda")
    n = p.shape[0]
    w = torch.ones(n, dtype=torch.float64, device="cuda") if occ is None else torch.as_tensor(
        occ.astype(np.float64), device="cuda")
    which = torch.as_tensor(which, device="cuda")
    hot = torch.nn.functional.one_hot(which, len(elements)).double()
    b = None if bfac is None else torch.as_tensor(bfac.astype(np.float64), device="cuda")
    F = torch.empty(q.shape[0], dtype=torch.complex128, device="cuda")
    g = None if grad is None else [torch.zeros(n, 3, dtype=torch.float64, device="cuda"),
                                   torch.zeros(n, dtype=torch.float64, device="cuda"),
                                   torch.zeros(n, dtype=torch.float64, device="cuda")]
    for i, j in _blocks(q.shape[0], n):
        qq = q[i:j]
        t = (qq * qscale) @ p.T
        t -= torch.round(t)
        t *= 2 * math.pi
        co, si = torch.cos(t), torch.sin(t)
        ff, s2 = _form_factors(elements, qq, B)
        if b is not None:
            e = torch.exp(-s2[:, None] * b[None, :])
            co *= e
            si *= e
        re = ((co @ (hot * w[:, None])) * ff).sum(1)
        im = -((si @ (hot * w[:, None])) * ff).sum(1)
        F[i:j] = torch.complex(re, im)
        if g is not None:
            # dL/dF of pixel: 2 G conj(F); dF/dw_j = f E e^{-i t}, dF/dr_j = -2 pi i q w_j f E e^{-i t}
            G = grad(i, j, re * re + im * im)
            fj = ff[:, which]
            zr = 2 * G[:, None] * (re[:, None] * co - im[:, None] * si) * fj
            zi = 2 * G[:, None] * (re[:, None] * -si - im[:, None] * co) * fj  # Im(conj(F) f E e^{-it})
            g[0] += (2 * math.pi * w)[:, None] * (zi.T @ qq)
            g[1] += zr.sum(0)
            g[2] -= w * (s2 @ zr)
    return F if g is None else (F, g)


def _chain_exact(v, I):
    """thomson, solid angle, photons and the noiseless output of chain parameters v."""
    f = {k: (_f32(x) if isinstance(x, float) else x) for k, x in v.items()}
    nx, ny = f["nx"], f["ny"]
    x = torch.arange(nx, dtype=torch.float64, device="cuda")
    y = torch.arange(ny, dtype=torch.float64, device="cuda")
    px = (((x - (nx - 1) / 2.0) / nx) * f["width"])[None, :].expand(ny, nx)
    py = (((y - (ny - 1) / 2.0) / ny) * f["height"])[:, None].expand(ny, nx)
    r2 = px * px + py * py
    d2 = f["distance"] ** 2
    cos2 = d2 / (r2 + d2)
    thomson = (2.81794e-15 ** 2 * (1 + cos2) / 2).reshape(-1)  # unpolarised
    solid = (f["pixel_width"] * f["pixel_height"] / d2 * cos2 ** 1.5).reshape(-1)
    return thomson, solid, thomson * solid * I * f["beam_intensity"]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "uneven":
        F = []
        for k, m in enumerate(_uneven(c)):
            Z, pos = synth.random_molecule(m["natoms"], m["radius"], seed * 1000 + k)
            F.append(_amplitude(Z, pos.astype(np.float64), _q64(m["det"])))
        return [F, [f.abs().square() for f in F]]
    if kind == "chain":
        I = _chain_intensity(c, seed).double()
        T, Om, ph = _chain_exact(_chain_values(c, seed), I)
        return {"thomson_correction": T, "solid_angle": Om, "photons_per_pixel": ph}
    Z, pos = _atoms(c, seed)
    p = pos.astype(np.float64)
    q = _q64(_det(c))
    if kind in ("batch", "nufft_batch"):
        return torch.stack([_amplitude(Z, p, q @ torch.as_tensor(R, device="cuda").T).abs().square()
                            for R in _rots(c, seed)])
    if kind == "refine":
        occ, b = _occ_b(len(Z), seed)
        counts = _refine_target(c, seed).double()
        qs = [q @ torch.as_tensor(R, device="cuda").T for R in _rots(c, seed)]
        I = torch.stack([_amplitude(Z, p, qr, occ, b).abs().square() for qr in qs])
        scale = counts.sum() / I.sum()
        total = None
        for n, qr in zip(counts, qs):
            g = _amplitude(Z, p, qr, occ, b, grad=lambda i, j, v: scale * (1 - n[i:j] / (v * scale + 1e-6)))[1]
            total = g if total is None else [t + x for t, x in zip(total, g)]
        return [I] + total
    if kind == "spectrum":
        lam, bw, ns = _f32(c["wavelength_nm"] * 1e-9), _f32(c["bandwidth"]), c["samples"] | 1
        lj = [lam * (1 - bw / 2) + j / (ns - 1) * lam * bw for j in range(ns)]
        wt = [math.exp(-(((v - lam) / (lam * bw / 4)) ** 2) / 2) for v in lj]
        F = sum(w / sum(wt) * _amplitude(Z, p, q, qscale=lam / v) for w, v in zip(wt, lj))
        return [F, F.abs().square()]
    if kind == "shot":
        q = q.float().double()  # the reference's float HKL list
        F = _amplitude(Z, p, q)
        return {"F": F.cpu().numpy(), "ints": F.abs().square().cpu().numpy()}
    if c.get("rotated"):
        q = q @ torch.as_tensor(_rots(c, seed)[0], device="cuda").T
    F = _amplitude(Z, p, q, B=_f32(c.get("B", 0.0)))
    I = F.abs().square()
    if kind == "pattern":
        return [F, I, {"photons_per_pixel": _chain_exact(_chain_values(c, seed), I)[2]}]
    return [F, I]
