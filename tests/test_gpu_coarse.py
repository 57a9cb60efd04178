"""Forwards on coarse grids of nodes against the FP64 oracle, at the FP32
tolerance of the sum on every pixel (floored maximum relative |F|^2 error 1e-5,
L2 1e-6; tests/test_gpu_sf.py): tile edges of the interpolation's 8 x 8
fragments, detectors off the beam axis, wide and spherical ones, every weight
and B factor, and the calls that must not take the grids."""
import numpy as np
import pytest
import torch

from conftest import intensity_errors
from oracle import oracle as O
from spsim_b200 import core, spsim as S, synth

pytestmark = pytest.mark.gpu

TOL = (1e-5, 1e-6)


def _det(nx, ny, pixel=150e-6, distance=0.2, wavelength=0.2e-9, **kw):
    return dict(nx=nx, ny=ny, width=nx * pixel, height=ny * pixel, distance=distance, wavelength=wavelength, **kw)


def _q(d):
    return O.hkl_detector(d["nx"], d["ny"], d["width"], d["height"], d["distance"], d["wavelength"],
                          center_x=d.get("center_x", 0.0), center_y=d.get("center_y", 0.0),
                          spherical=d.get("spherical", False))


def _check(F, I, Z, pos, q, **kw):
    F64, I64 = O.structure_factor(Z, pos.astype(np.float64), q, **kw)
    e_max, e_l2 = intensity_errors(I.cpu().numpy(), I64)
    assert e_max < TOL[0] and e_l2 < TOL[1], (e_max, e_l2)
    if F is not None:
        assert np.abs(F.cpu().numpy() - F64).max() < 1e-5 * np.abs(F64).max()


def _on_grid(yes=True):
    terms = core.last_forward_stats()[0]
    assert (core.last_terms_evaluated() < terms) == yes


@pytest.mark.parametrize("nx,ny", [(64, 250), (127, 130), (129, 95), (200, 61), (257, 256), (1000, 17)])
@pytest.mark.parametrize("precision", ["f32", "f32_fast", "fp64"])
def test_ragged_detectors(cuda, nx, ny, precision):
    Z, pos = synth.random_molecule(3000, 3.0e-9, 201)
    pos += np.float32(5e-9)  # a centre phase
    d = _det(nx, ny)
    R = synth.haar_rotations(1, 202)[0]
    F, I = core.forward(core.Molecule(Z, pos), core.QSet.from_detector(**d), rot=R, B=7.5, precision=precision)
    _on_grid()
    _check(F, I, Z, pos, _q(d) @ R.T, B=7.5)


@pytest.mark.parametrize("kw", [dict(center_x=0.012), dict(spherical=True), dict(distance=0.012),
                                dict(wavelength=0.06e-9), dict(pixel=2e-3, distance=0.5)],
                         ids=["off_axis", "spherical", "wide_angle", "hard_x_rays", "large_pixels"])
def test_geometries(cuda, kw):
    # wide_angle: pixels to 0.9 detector distances off the axis, form factors
    # falling over their whole range; hard_x_rays: phases up to ~0.1 cycle per pixel
    Z, pos = synth.random_molecule(2500, 2.8e-9, 203)
    d = _det(144, 140, **kw)
    F, I = core.forward(core.Molecule(Z, pos), core.QSet.from_detector(**d))
    _on_grid()
    _check(F, I, Z, pos, _q(d))


def test_panel_off_the_beam_axis(cuda):
    # no bright pixels near the beam: the FP32 terms' own noise reaches 1.5e-5 of
    # the dimmest intensities with the sum on every pixel, which bounds the grid's
    Z, pos = synth.random_molecule(2500, 2.8e-9, 203)
    d = _det(144, 140, center_x=-0.05, center_y=0.03)
    q, qs, mol = _q(d), core.QSet.from_detector(**d), core.Molecule(Z, pos)
    _, I64 = O.structure_factor(Z, pos.astype(np.float64), q)
    _, I = core.forward(mol, qs)
    _on_grid()
    try:
        core.set_variant(128, 8, 4)
        _, Ip = core.forward(mol, qs)
        _on_grid(False)
    finally:
        core.set_variant(-1)
    got, bound = (intensity_errors(v.cpu().numpy(), I64) for v in (I, Ip))
    assert got[0] <= max(TOL[0], bound[0]) and got[1] <= max(TOL[1], bound[1]), (got, bound)


def test_weights_and_b_factors(cuda):
    Z, pos = synth.random_molecule(2000, 2.5e-9, 204)
    Z[::7] = 0
    Z[::11] = 19  # potassium: the widest form factor of common elements
    rng = np.random.Generator(np.random.PCG64(205))
    occ = rng.uniform(-0.5, 1.0, len(Z)).astype(np.float32)
    b = rng.uniform(0.0, 60.0, len(Z)).astype(np.float32)
    d = _det(130, 140, distance=0.05)
    q, qs = _q(d), core.QSet.from_detector(**d)
    for occ_, b_, B in ((occ, None, 0.0), (occ, b, 0.0), (None, b, 12.0)):
        F, I = core.forward(core.Molecule(Z, pos, occ=occ_, bfac=b_), qs, B=B)
        _on_grid()
        _check(F, I, Z, pos, q, occ=occ_, bfac=b_, B=B)


def test_b_factors_rewritten_beyond_the_grids_limit(cuda):
    # the limit is 2 * 20 + 100 = 140 A^2: on either side of it, and back, in a
    # batch of orientations with a molecule that stays within it
    Z, pos = synth.random_molecule(1500, 2.5e-9, 206)
    rng = np.random.Generator(np.random.PCG64(207))
    b0 = rng.uniform(0.0, 20.0, len(Z)).astype(np.float32)
    b0[0] = 20.0
    d = _det(128, 120, distance=0.03)
    q, qs = _q(d), core.QSet.from_detector(**d)
    mol, other = core.Molecule(Z, pos, bfac=b0), core.Molecule(Z, pos, bfac=b0)
    R = synth.haar_rotations(2, 208)
    p = torch.from_numpy(pos).cuda()
    for top in (100.0, 3000.0, 139.0):
        b = b0.copy()
        b[5:400:9] = top
        mol.update_device(p, bfac=torch.from_numpy(b).cuda())
        F, I = core.forward_batch([other, mol], [qs, qs], rots=R)
        _on_grid()
        for k, bk in enumerate((b0, b)):
            _check(F[k], I[k], Z, pos, q @ R[k].T, bfac=bk)


@pytest.mark.parametrize("B,nodes", [(20.0, True), (60.0, True), (100.0, True), (180.0, True), (200.0, False)])
def test_amplitudes_that_fall_far(cuda, B, nodes):
    # amplitudes that fall by e^-2 to e^-17 along an axis, e^-4 to e^-33 to the
    # corners: the dim pixels keep their own accuracy beside the bright ones.  A
    # ring's rms error against its rms amplitude: the FP32 weight's exponent, up
    # to 33 / ln 2 = 48, rounds to 48 * 2^-24 * ln 2 = 2e-6
    Z, pos = synth.random_molecule(3000, 3.0e-9, 214)
    b = np.full(len(Z), B, np.float32)
    d = _det(400, 400, pixel=192e-6, distance=0.06, wavelength=0.1e-9)
    q, qs, mol = _q(d), core.QSet.from_detector(**d), core.Molecule(Z, pos, bfac=b)
    F, _ = core.forward(mol, qs)
    _on_grid(nodes)
    F64, I64 = O.structure_factor(Z, pos.astype(np.float64), q, bfac=b)
    s2 = (q * q).sum(1)
    ring = np.minimum(6 * s2 / s2.max(), 5).astype(int)
    err = np.abs(F.cpu().numpy() - F64) ** 2
    for k in range(6):
        assert np.sqrt(err[ring == k].mean() / I64[ring == k].mean()) < 2e-6, k
    # the gradient of a loss that weighs every pixel's logarithm alike
    g = (np.random.Generator(np.random.PCG64(215)).normal(size=len(q)) / (I64 + 1e-12 * I64.max())).astype(np.float32)
    grads = core.adjoint(mol, qs, torch.from_numpy(F64.astype(np.complex64)).cuda(), torch.from_numpy(g).cuda())
    exact = O.structure_factor_vjp(Z, pos.astype(np.float64), q, g.astype(np.float64), bfac=b)
    for ours, e in zip(grads, exact):
        assert _rel(ours.cpu().numpy(), e) < 1e-5


def test_fp64_at_its_own_tolerance(cuda):
    # 2e-7 floored maximum, 1e-7 L2: the float32 outputs' rounding; weights, B factors, a wide detector
    Z, pos = synth.random_molecule(1500, 2.5e-9, 212)
    rng = np.random.Generator(np.random.PCG64(213))
    occ = rng.uniform(-0.5, 1.0, len(Z)).astype(np.float32)
    b = rng.uniform(0.0, 60.0, len(Z)).astype(np.float32)
    for d in (_det(130, 141), _det(128, 97, distance=0.02), _det(100, 120, spherical=True)):
        q, qs = _q(d), core.QSet.from_detector(**d)
        for b_, B in ((None, 0.0), (b, 6.0)):
            F, I = core.forward(core.Molecule(Z, pos, occ=occ, bfac=b_), qs, B=B, precision="fp64")
            _on_grid()
            F64, I64 = O.structure_factor(Z, pos.astype(np.float64), q, occ=occ, bfac=b_, B=B)
            e_max, e_l2 = intensity_errors(I.cpu().numpy(), I64)
            assert e_max < 2e-7 and e_l2 < 1e-7, (e_max, e_l2)
            assert np.linalg.norm(F.cpu().numpy() - F64) < 1e-7 * np.linalg.norm(F64)


@pytest.mark.parametrize("natoms,precision,update,tile", [(400, "f32", False, 64), (6000, "f32", False, 256),
                                                          (6000, "f32_fast", False, 256), (6000, "f32", True, 128),
                                                          (6000, "fp64", False, 128)])
def test_the_node_kernel_that_ran(cuda, natoms, precision, update, tile):
    Z, pos = synth.random_molecule(natoms, 3.6e-9, 216)
    d = _det(256, 250)
    mol, qs = core.Molecule(Z, pos), core.QSet.from_detector(**d)
    if update:
        mol.update_device(torch.from_numpy(pos).cuda())
    core.forward(mol, qs, precision=precision)
    assert core.last_node_tile() == tile
    core.forward(mol, core.QSet.from_list(qs.q()[:5000]), precision=precision)
    assert core.last_node_tile() == 0


def test_general_matrices_and_spectrum(cuda):
    Z, pos = synth.random_molecule(2500, 2.6e-9, 209)
    d = _det(132, 136)
    q, qs, mol = _q(d), core.QSet.from_detector(**d), core.Molecule(Z, pos)
    R = synth.haar_rotations(1, 210)[0] @ np.diag([1.0, 1.3, 0.8])  # not a rotation: it stretches q
    F, I = core.forward(mol, qs, rot=R)
    _on_grid()
    # the oracle takes form factors at |R q|, the library's at |q|: point atoms compare the sum
    point = core.Molecule(Z, pos, delta_atoms=True)
    F, I = core.forward(point, qs, rot=R)
    _on_grid()
    u = q @ R.T
    F64 = np.exp(-2j * np.pi * (u @ pos.astype(np.float64).T)).sum(1)
    e_max, e_l2 = intensity_errors(I.cpu().numpy(), np.abs(F64) ** 2)
    assert e_max < TOL[0] and e_l2 < TOL[1], (e_max, e_l2)
    F, I = core.forward_spectrum(mol, qs, d["wavelength"], 0.1, 4)
    _on_grid()
    _, I64 = O.structure_factor_spectrum(Z, pos.astype(np.float64), q, d["wavelength"], 0.1, 4)
    e_max, e_l2 = intensity_errors(I.cpu().numpy(), I64)
    assert e_max < TOL[0] and e_l2 < TOL[1], (e_max, e_l2)


def test_calls_that_stay_on_every_pixel(cuda):
    Z, pos = synth.random_molecule(4000, 3.0e-9, 211)
    mol = core.Molecule(Z, pos)
    d = _det(128, 128)
    qs = core.QSet.from_detector(**d)
    cases = [(core.QSet.from_list(qs.q()), "fp64"), (core.QSet.from_list(qs.q()), "f32"), (core.QSet.from_detector(**_det(15, 2000)), "f32"),
             (core.QSet.from_detector(**_det(128, 128, pixel=1e-3, distance=0.05)), "f32"),  # 64 mm at 50 mm
             (core.QSet.from_detector(**_det(128, 128, wavelength=0.01e-9)), "f32")]  # undersampled
    for q, precision in cases:
        F, I = core.forward(mol, q, precision=precision)
        _on_grid(False)
        _, I64 = O.structure_factor(Z, pos.astype(np.float64), q.q().astype(np.float64))
        assert np.abs(I.cpu().numpy() - I64).max() < 1e-4 * I64.max()
    # a batch with one such pattern runs on every pixel as a whole
    core.forward_batch([mol, mol], [qs, cases[2][0]])
    _on_grid(False)
    # no atoms: zeros
    _, I = core.forward(core.Molecule(np.zeros(5, np.int32), pos[:5]), qs)
    assert not I.any()


def _cells_case(shape, n, seed):
    """Atoms of a ball, a rod, a sheet and two far balls, which leave cells empty, single and uneven."""
    Z, pos = synth.random_molecule(n, 8.2e-9, seed)
    if shape == "rod":
        pos = pos * np.float32([0.2, 0.15, 1.0])
    elif shape == "sheet":
        pos = pos * np.float32([1.0, 0.04, 0.9])
    elif shape == "pair":
        pos = pos * np.float32(0.4) + np.float32([5e-9, 0, 0]) * np.sign(pos[:, :1])
    return Z, (pos + np.float32([4e-9, -1e-9, 2e-9])).astype(np.float32)


@pytest.mark.parametrize("shape", ["ball", "rod", "sheet", "pair"])
@pytest.mark.parametrize("precision", ["f32", "fp64"])
@pytest.mark.parametrize("det", [dict(center_x=0.007), dict(spherical=True)], ids=["off_axis", "spherical"])
def test_cells(cuda, shape, precision, det):
    # sums cell by cell: far fewer terms than on the patterns' own nodes, which a
    # molecule whose positions were rewritten on the device still takes
    Z, pos = _cells_case(shape, 12001, 221)
    rng = np.random.Generator(np.random.PCG64(222))
    occ = rng.uniform(-0.5, 1.0, len(Z)).astype(np.float32)
    b = rng.uniform(0.0, 40.0, len(Z)).astype(np.float32)
    d = _det(141, 118, pixel=280e-6, wavelength=0.13e-9, **det)
    q, qs, R = _q(d), core.QSet.from_detector(**d), synth.haar_rotations(96, 223)
    mol = core.Molecule(Z, pos, occ=occ, bfac=b)
    F = torch.empty(len(R), d["ny"] * d["nx"], dtype=torch.complex64, device="cuda")
    I = torch.empty(len(R), d["ny"] * d["nx"], device="cuda")
    core.forward_batch([mol] * len(R), [qs] * len(R), rots=R, precision=precision, F=list(F), I=list(I), B=5.0)
    terms = core.last_terms_evaluated()
    for k in (0, 57, 95):
        F64, I64 = O.structure_factor(Z, pos.astype(np.float64), q @ R[k].T, occ=occ, bfac=b, B=5.0)
        e_max, e_l2 = intensity_errors(I[k].cpu().numpy(), I64)
        tol = TOL if precision == "f32" else (2e-7, 1e-7)
        assert e_max < tol[0] and e_l2 < tol[1], (k, e_max, e_l2)
        assert np.linalg.norm(F[k].cpu().numpy().reshape(F64.shape) - F64) < tol[1] * np.linalg.norm(F64)
    # rotations of the next call go into the same plan
    core.forward_batch([mol] * len(R), [qs] * len(R), rots=R[::-1].copy(), precision=precision, F=list(F), I=list(I), B=5.0)
    assert core.last_terms_evaluated() == terms
    F64, I64 = O.structure_factor(Z, pos.astype(np.float64), q @ R[95].T, occ=occ, bfac=b, B=5.0)
    assert intensity_errors(I[0].cpu().numpy(), I64)[1] < 1e-6
    if precision == "f32":
        moved = core.Molecule(Z, pos, occ=occ, bfac=b)
        moved.update_device(torch.from_numpy(pos).cuda())
        core.forward_batch([moved] * len(R), [qs] * len(R), rots=R, F=None, I=list(I), want_F=False, B=5.0)
        assert core.last_terms_evaluated() > 1.3 * terms


def test_cells_of_a_spectrum_and_of_uneven_molecules(cuda):
    Z, pos = synth.random_molecule(30000, 9.0e-9, 224)
    d = _det(256, 250, pixel=75e-6)
    q, mol, qs = _q(d), core.Molecule(Z, pos), core.QSet.from_detector(**d)
    F, I = core.forward(mol, qs)
    whole = core.last_terms_evaluated()
    _check(F, I, Z, pos, q)
    F, I = core.forward_spectrum(mol, qs, d["wavelength"], 0.05, 4)
    assert core.last_terms_evaluated() < 6 * whole
    pick = np.arange(0, len(q), 97)  # the oracle on every 97th pixel
    _, I64 = O.structure_factor_spectrum(Z, pos.astype(np.float64), q[pick], d["wavelength"], 0.05, 4)
    e_max, e_l2 = intensity_errors(I.cpu().numpy().reshape(-1)[pick], I64)
    assert e_max < TOL[0] and e_l2 < TOL[1], (e_max, e_l2)
    # molecules with and without cells in one call
    Zs, ps = synth.random_molecule(700, 1.5e-9, 225)
    small = core.Molecule(Zs, ps)
    Fs, Is = core.forward_batch([small, mol, small], [qs] * 3)
    _check(Fs[1], Is[1], Z, pos, q)
    for k in (0, 2):
        _check(Fs[k], Is[k], Zs, ps, q)


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("nx,ny", [(96, 70), (129, 65), (61, 200)])
@pytest.mark.parametrize("precision", ["f32", "f32_fast"])
@pytest.mark.parametrize("with_b", [False, True])
def test_adjoint(cuda, nx, ny, precision, with_b):
    # the gradient through the nodes against the oracle's vector-Jacobian
    # product, at the adjoint's tolerance (1e-4 relative L2): an odd number of
    # patterns, elements whose segments share a block, a centre phase, global B
    Z, pos = synth.random_molecule(1403, 2.4e-9, 221)
    pos += np.float32(4e-9)
    rng = np.random.Generator(np.random.PCG64(222))
    occ = rng.uniform(0.5, 1.0, len(Z)).astype(np.float32)
    b = rng.uniform(0.0, 30.0, len(Z)).astype(np.float32) if with_b else None
    B = 0.0 if with_b else 9.0
    d = _det(nx, ny)
    R = synth.haar_rotations(3, 223)
    q = np.concatenate([_q(d) @ r.T for r in R])
    g = rng.normal(size=q.shape[0]).astype(np.float32)
    mol, qs = core.Molecule(Z, pos, occ=occ, bfac=b), core.QSet.from_detector(**d)
    F, _ = core.forward_batch([mol] * 3, [qs] * 3, rots=R, B=B, precision=precision)
    dpos, docc, dB = core.adjoint(mol, qs, torch.cat(F), torch.from_numpy(g).cuda(), rots=R, B=B, precision=precision)
    # the oracle's gradient has no global B: the same factor on every atom
    ball = np.full(len(Z), B, np.float32) if b is None else b
    dp, do, db = O.structure_factor_vjp(Z, pos.astype(np.float64), q, g.astype(np.float64), occ=occ, bfac=ball)
    assert _rel(dpos.cpu().numpy(), dp) < 1e-4
    assert _rel(docc.cpu().numpy(), do) < 1e-4
    if with_b:
        assert _rel(dB.cpu().numpy(), db) < 1e-4


def test_adjoint_of_b_factors_beyond_the_grids_limit(cuda):
    Z, pos = synth.random_molecule(1500, 2.5e-9, 224)
    rng = np.random.Generator(np.random.PCG64(225))
    b0 = rng.uniform(0.0, 20.0, len(Z)).astype(np.float32)
    d = _det(128, 120, distance=0.03)
    q, qs = _q(d), core.QSet.from_detector(**d)
    mol = core.Molecule(Z, pos, bfac=b0)
    g = rng.normal(size=q.shape[0]).astype(np.float32)
    for top in (90.0, 2500.0, 60.0):
        b = b0.copy()
        b[3:300:7] = top
        mol.update_device(torch.from_numpy(pos).cuda(), bfac=torch.from_numpy(b).cuda())
        F, _ = core.forward(mol, qs)
        dpos, docc, dB = core.adjoint(mol, qs, F, torch.from_numpy(g).cuda())
        dp, do, db = O.structure_factor_vjp(Z, pos.astype(np.float64), q, g.astype(np.float64), bfac=b)
        assert _rel(dpos.cpu().numpy(), dp) < 1e-4
        assert _rel(docc.cpu().numpy(), do) < 1e-4
        assert _rel(dB.cpu().numpy(), db) < 1e-4


@pytest.mark.parametrize("eps", [1e-3, 1e-6, 1e-8, 1e-12])
@pytest.mark.parametrize("elements", [(6, 8), (6, 7, 8, 16), (1, 6, 7, 8, 16, 26)], ids=["2", "4", "6"])
def test_nufft_at_the_nodes(cuda, eps, elements):
    # 2^16 pixels: the NUFFT's stencils at the nodes of the detector's grid, two
    # and four element slots a cell and two groups, narrow and wide stencils, one
    # rotated pattern and a batch, with a global B and a centre phase; tolerances
    # of the NUFFT against the sum (relative L2 max(3 eps, 2e-7), maximum
    # max(30 eps, 2e-6) of the largest amplitude)
    _, pos = synth.random_molecule(2000, 2.6e-9, 231)
    pos += np.float32(6e-9)
    Z = np.random.Generator(np.random.PCG64(232)).choice(elements, len(pos)).astype(np.int32)
    d = _det(250, 263)
    R = synth.haar_rotations(2, 233)
    mol, qs = core.Molecule(Z, pos), core.QSet.from_detector(**d)
    F1, I1 = core.forward_nufft(mol, qs, rot=R[0], B=5.0, eps=eps)
    F2, I2 = core.forward_nufft_batch(mol, qs, R, B=5.0, eps=eps)
    core.synchronize()
    for F, I, r in ((F1, I1, R[0]), (F2[0], I2[0], R[0]), (F2[1], I2[1], R[1])):
        F64, I64 = O.structure_factor(Z, pos.astype(np.float64), _q(d) @ r.T, B=5.0)
        dF = np.abs(F.cpu().numpy() - F64)
        assert np.linalg.norm(dF) < max(3 * eps, 2e-7) * np.linalg.norm(F64)
        assert dF.max() < max(30 * eps, 2e-6) * np.abs(F64).max()
        assert np.abs(I.cpu().numpy() - I64).max() < max(60 * eps, 4e-6) * I64.max()


@pytest.mark.parametrize("nx,ny,chunks,kw", [
    (400, 371, 1, dict()), (399, 357, 3, dict(b_factor=9.0)), (512, 300, 1, dict(spherical=1)),
    (420, 401, 4, dict(center_x=0.011, center_y=-0.004)), (400, 380, 1, dict(distance=0.05)),
    (450, 444, 2, dict(spherical=1, b_factor=4.0))],
    ids=["one_pass", "chunks_b", "spherical", "off_axis", "wide", "spherical_chunks"])
@pytest.mark.parametrize("fast", [False, True], ids=["f32", "f32_fast"])
def test_simulate_shot_on_the_nodes(cuda, tmp_path, monkeypatch, nx, ny, chunks, kw, fast):
    # the pattern is that of the shot's own float HKL list (its rounding is some
    # 1e-5 of the amplitudes, two orders beyond the bounds here): the oracle on it
    monkeypatch.chdir(tmp_path)
    Z, pos = synth.random_molecule(9000, 6.0e-9, 231)
    pos += np.float32(3e-9)
    opts = S.set_defaults()
    o = opts.contents
    det, exp = o.detector.contents, o.experiment.contents
    det.nx, det.ny, det.nz = nx, ny, 1
    det.pixel_width = det.pixel_height = 75e-6
    det.width, det.height = nx * det.pixel_width, ny * det.pixel_height
    det.distance = kw.get("distance", 0.15)
    det.center_x, det.center_y, det.spherical = kw.get("center_x", 0.0), kw.get("center_y", 0.0), kw.get("spherical", 0)
    exp.wavelength = 1.5e-10
    o.b_factor = kw.get("b_factor", 0.0)
    o.verbosity_level = 0
    o.random_orientation = 0
    o.euler_orientation[0], o.euler_orientation[1], o.euler_orientation[2] = 0.4, -0.9, 1.7
    mol = S.get_molecule_from_atoms(Z, pos)
    S.set_precision("f32_fast" if fast else "f32")
    S.set_shot_chunks(chunks)
    try:
        shot = S.simulate_shot(mol, opts)
    finally:
        S.set_shot_chunks(0)
        S.set_precision("f32")
    _on_grid()
    n = nx * ny
    q = S.as_array(shot.contents.HKL_list, 3 * n).reshape(-1, 3).astype(np.float64)
    pick = np.arange(0, n, 7)
    F64, I64 = O.structure_factor(Z, pos.astype(np.float64), q[pick], B=kw.get("b_factor", 0.0))
    e_max, e_l2 = intensity_errors(S.as_array(shot.contents.ints, n)[pick], I64)
    assert e_max < TOL[0] and e_l2 < TOL[1], (e_max, e_l2)
    F = S.as_array(shot.contents.F, n)[pick]
    assert np.linalg.norm(F - F64) < 1e-6 * np.linalg.norm(F64)
    S.free_stuff(shot, opts)
    S.free_mol(mol)


def test_shots_of_new_molecules_make_no_lists_of_cells_that_they_cannot_repay(cuda, tmp_path, monkeypatch):
    # a list takes 0.15 ms and saves some 0.1 ms per shot here: from the second
    # shot of a molecule on; the next molecule takes over the buffer
    monkeypatch.chdir(tmp_path)
    opts = S.set_defaults()
    o = opts.contents
    det, exp = o.detector.contents, o.experiment.contents
    det.nx, det.ny, det.nz = 512, 480, 1
    det.pixel_width = det.pixel_height = 75e-6
    det.width, det.height, det.distance = 512 * 75e-6, 480 * 75e-6, 0.12
    exp.wavelength = 1.5e-10
    o.verbosity_level = 0
    o.random_orientation = 0
    o.euler_orientation[0] = o.euler_orientation[1] = o.euler_orientation[2] = 0.0
    S.set_shot_chunks(1)
    try:
        for seed in (241, 242):
            Z, pos = synth.random_molecule(20000, 8.0e-9, seed)
            mol = S.get_molecule_from_atoms(Z, pos)
            terms, F = [], []
            for _ in range(3):
                shot = S.simulate_shot(mol, opts)
                _on_grid()
                terms.append(core.last_terms_evaluated())
                F.append(S.as_array(shot.contents.F, 512 * 480).copy())
                S.free_stuff(shot, opts)
            S.free_mol(mol)
            assert terms[0] > terms[1] == terms[2]
            for f in F[1:]:
                assert np.linalg.norm(f - F[0]) < 2e-7 * np.linalg.norm(F[0])
    finally:
        S.set_shot_chunks(0)
