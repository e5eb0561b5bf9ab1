"""GPU parity: every stage of the CUDA path against the FP64 oracle (or an FP64 numpy
statement of the same operation), the whole job against the oracle and the reference's
own golden outputs, and full-size (512 / 1024 molecules) properties.  All calls go
through the C ABI (libcalcir.so via ctypes)."""
import os
import subprocess

import numpy as np
import pytest

from conftest import GOLDEN_CASES, golden_params, load_golden
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SPEC_TOL = 1e-4    # relative L2 per spectrum, plain FP32 path vs FP64 oracle
HBAR = 5.308837367


def make_params(lib, prm, **extra):
    keys = {k: prm[k] for k in ("ntcfpoints", "nsamples", "sampleEvery", "omegaStep", "nchrom_mol", "nzeros",
                                "map", "dt", "t1", "avef", "beginTime", "omegaStart", "omegaStop")}
    model = "tip4p2005" if prm["imodel"] else "tip4p"
    species = ["H2O", "HOD/D2O", "HOD/H2O", "D2O"][prm["ispecies"]]
    keys.update(extra)
    return lib.default_params(model=model, species=species, **keys)


def near_cutoff(xyz, box, prm, eps=2e-5):
    """Chromophores with some O(m)..H(n) distance within eps of the field cutoff: FP32 and
    FP64 may disagree on including that molecule."""
    mol, n, Hpos, _, _ = O.chromophores(xyz, box, prm["natom_mol"], prm["nchrom_mol"])
    r = np.linalg.norm(O.min_image(mol[None, :, 0, :] - Hpos[:, None, :], np.asarray(box, float)), axis=2)
    return np.any(np.abs(r - O.CUTOFF) < eps, axis=1)


@pytest.mark.parametrize("case", GOLDEN_CASES)
def test_build_hamiltonian(lib, case):
    meta, _ = load_golden(case)
    prm = golden_params(meta)
    xyz, box = lib.synth_trajectory(meta["nmol"], 4, seed=meta["seed"])
    with lib.Engine(make_params(lib, prm), xyz.shape[1]) as eng:
        H, E, dip, pol = eng.build_hamiltonian(xyz, box)
    for f in range(4):
        Eo, Ho, dipo, polo = O.frame(xyz[f], box, prm)
        ok = ~near_cutoff(xyz[f], box, prm)
        np.testing.assert_allclose(E[f][ok], Eo[ok], rtol=2e-5, atol=2e-7)
        sel = np.ix_(ok, ok)
        assert np.array_equal(H[f], H[f].T), "H must be exactly symmetric"
        np.testing.assert_allclose(H[f][sel], Ho[sel], rtol=1e-4, atol=2e-3)
        np.testing.assert_allclose(dip[f][:, ok], dipo[:, ok], rtol=1e-4, atol=1e-6)
        np.testing.assert_allclose(pol[f][:, ok], polo[:, ok], rtol=1e-4, atol=1e-6)


def _sym(rng, n, scale=1000.0):
    a = rng.standard_normal((n, n))
    return ((a + a.T) * (scale / np.sqrt(8 * n))).astype(np.float32)


def _check_eig(A, w, V, tol_scale=1.0):
    A64 = A.astype(np.float64)
    n = A.shape[0]
    nrm = max(np.abs(np.linalg.eigvalsh(A64)).max(), 1e-30)
    wref = np.linalg.eigvalsh(A64)
    assert np.all(np.diff(w) >= 0), "eigenvalues must ascend"
    assert np.abs(w - wref).max() <= 2e-6 * tol_scale * nrm * max(1.0, np.sqrt(n) / 4)
    V64 = V.astype(np.float64)
    assert np.abs(V64.T @ V64 - np.eye(n)).max() <= 2e-6 * tol_scale * max(1.0, np.sqrt(n))
    assert np.abs(A64 @ V64 - V64 * w[None, :]).max() <= 4e-6 * tol_scale * nrm * max(1.0, np.sqrt(n) / 4)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 17, 64, 127, 128, 256, 257, 301, 432, 513, 686, 1023, 1024, 2048])
def test_eigh_random(lib, n):
    rng = np.random.default_rng(n)
    nmat = 3 if n <= 1024 else 1
    A = np.stack([_sym(rng, n) for _ in range(nmat)])
    with lib.Engine(lib.default_params(species="H2O"), 8) as eng:
        w, V = eng.eigh(A)
    for m in range(nmat):
        _check_eig(A[m], w[m], V[m])


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_eigh_rejects_non_finite_host_matrices(lib, bad):
    """A NaN or infinity in a host matrix is an error before any GPU work (the host check of
    cir_eigh); the context stays usable."""
    from calcir_gb300 import CirError
    rng = np.random.default_rng(3)
    A = np.stack([_sym(rng, 40) for _ in range(2)])
    A[1, 7, 3] = A[1, 3, 7] = bad
    with lib.Engine(lib.default_params(species="H2O"), 8) as eng:
        with pytest.raises(CirError, match="NaN or Inf"):
            eng.eigh(A)
        w, V = eng.eigh(A[:1])
    _check_eig(A[0], w[0], V[0])


@pytest.mark.parametrize("n", [96, 302])
def test_eigh_special_matrices(lib, n):
    """Zero, scaled identity, exact ties, a rank-one perturbation, diagonal, and a
    tridiagonal with exact zeros (96: unblocked tridiagonalisation; 302: blocked, with a
    padded leading dimension)."""
    rng = np.random.default_rng(5)
    cases = [np.zeros((n, n), np.float32), np.eye(n, dtype=np.float32) * 3.0,
             np.diag(np.repeat(np.arange(n // 8 + 1, dtype=np.float32), 8)[:n]),   # exact ties
             (np.eye(n) + np.outer(np.ones(n), np.ones(n)) / n).astype(np.float32),   # degenerate
             np.diag(rng.standard_normal(n).astype(np.float32)) * 500]
    t = np.zeros((n, n), np.float32)                                          # tridiagonal with zeros
    t[np.arange(n - 1), np.arange(1, n)] = t[np.arange(1, n), np.arange(n - 1)] = (np.arange(n - 1) % 5 != 0) * 7.0
    t += np.diag(np.linspace(-300, 300, n).astype(np.float32))
    cases.append(t)
    with lib.Engine(lib.default_params(species="H2O"), 8) as eng:
        w, V = eng.eigh(np.stack(cases))
    for m, A in enumerate(cases):
        _check_eig(A, w[m], V[m])


@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
@pytest.mark.parametrize("n", [300, 1024])
def test_eigh_clustered_spectrum(lib, n, precision):
    """Eigenvalues in tight clusters (members 1e-4 apart, 1e-7 of the norm, up to 24 per
    cluster): every merge deflates long runs of consecutive close pairs by Givens rotations,
    which it applies to U as chains with one carried value per column.  The eigenpairs meet
    the bounds of the random matrices."""
    rng = np.random.default_rng(n + 11)
    lam = []
    while len(lam) < n:
        c = rng.uniform(-1000.0, 1000.0)
        lam.extend(c + 1e-4 * np.arange(min(int(rng.integers(1, 25)), n - len(lam))))
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * np.asarray(lam)) @ Q.T
    A = ((A + A.T) / 2).astype(np.float32)
    with lib.Engine(lib.default_params(species="H2O", precision=precision), 8) as eng:
        w, V = eng.eigh(A[None])
    _check_eig(A, w[0], V[0])


def test_propagate(lib):
    rng = np.random.default_rng(1)
    n, nprop, dt = 200, 3, 0.010
    A = np.stack([_sym(rng, n) for _ in range(nprop)])
    F = (rng.standard_normal((nprop, n, n)) + 1j * rng.standard_normal((nprop, n, n))).astype(np.complex64)
    with lib.Engine(lib.default_params(species="H2O"), 8) as eng:
        w, V = eng.eigh(A)
        out = eng.propagate(V, w, np.float32(dt), F)
    for m in range(nprop):
        V64 = V[m].astype(np.float64)
        ph = np.exp(1j * w[m].astype(np.float64) * np.float32(dt) / HBAR)
        ref = (V64 * ph[None, :]) @ (V64.T @ F[m].astype(np.complex128))
        assert O.rel_l2(out[m], ref) < 3e-6


def test_tcf_terms_and_spectral_density(lib):
    meta, _ = load_golden("small_h2o")
    prm = golden_params(meta)
    xyz, box = lib.synth_trajectory(meta["nmol"], 2, seed=meta["seed"])
    E0, H0, d0, p0 = O.frame(xyz[0], box, prm)
    E1, H1, d1, p1 = O.frame(xyz[1], box, prm)
    rng = np.random.default_rng(3)
    n = H0.shape[0]
    F = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
    with lib.Engine(make_params(lib, prm), xyz.shape[1]) as eng:
        got = eng.tcf_terms(F.astype(np.complex64), d0.astype(np.float32), p0.astype(np.float32),
                            d1.astype(np.float32), p1.astype(np.float32))
        psi = (F.astype(np.complex64).astype(np.complex128) @ np.vstack([d0, p0]).astype(np.float32).T.astype(np.float64)).T
        ref = O.tcf_terms(psi, np.vstack([d1, p1]).astype(np.float32).astype(np.float64))
        for g, r in zip(got, ref):
            assert abs(g - r) <= 1e-5 * (abs(r) + 1e-3)
        lam, V = np.linalg.eigh(H0)
        Sw = eng.spectral_density(V.astype(np.float32), lam.astype(np.float32), d0.astype(np.float32))
    omega = prm["omegaStart"] + prm["omegaStep"] * np.arange(len(Sw))
    Mv = V.T @ d0.T
    g = HBAR / (np.float32(prm["t1"]) * 2.0)
    dw = omega[:, None] - (lam[None, :] + np.float32(prm["avef"]))
    ref = np.sum(np.sum(Mv * Mv, 1)[None, :] * g / (dw * dw + g * g) / O.PI, 1)
    assert O.rel_l2(Sw, ref) < 1e-5


@pytest.mark.parametrize("nzeros", [0, 1, 2, 97, 500, 25600])
def test_lineshape_fft(lib, nzeros):
    rng = np.random.default_rng(nzeros)
    ntcf = 150
    p = lib.default_params(species="H2O", ntcfpoints=ntcf, nzeros=nzeros, omegaStart=2000, omegaStop=5000,
                           avef=3415.0)
    tcf = (rng.standard_normal(ntcf) + 1j * rng.standard_normal(ntcf)) * np.exp(-np.arange(ntcf) / 40)
    prm = {"ntcfpoints": ntcf, "nzeros": nzeros, "dt": 0.010, "avef": 3415.0, "omegaStart": 2000,
           "omegaStop": 5000}
    with lib.Engine(p, 8) as eng:
        om, val = eng.lineshape(tcf)
    om_ref, val_ref = O.lineshape_rows(prm, O.c2r(tcf, ntcf + nzeros))
    np.testing.assert_array_equal(om, om_ref.astype(np.float32))
    assert O.rel_l2(val, val_ref) < 2e-6


def _frames_for(lib, meta):
    prm = golden_params(meta)
    xyz, box = lib.synth_trajectory(meta["nmol"], meta["nframes"], seed=meta["seed"])
    fos = np.array([O.frame_index(prm, meta["frame_dt"], s, k)
                    for s in range(prm["nsamples"]) for k in range(prm["ntcfpoints"])], np.int32)
    return prm, xyz, box, fos


def _compare_run(out, ref, prm, tol, name):
    for k in ("tcf_ir", "tcf_vv", "tcf_vh", "sw", "ls_ir", "ls_vv", "ls_vh"):
        e = O.rel_l2(out[k], ref[k])
        assert e < tol, (name, k, e)
    np.testing.assert_array_equal(out["omega"], np.asarray(ref["omega"], np.float32))
    np.testing.assert_array_equal(out["ls_omega"], np.asarray(ref["ls_omega"], np.float32))
    step = prm["omegaStep"]
    ntot = np.sum(ref["count"])
    assert abs(np.sum(out["pw"]) * step - 1) < 1e-5
    assert np.max(np.abs(np.cumsum(out["pw"]) - np.cumsum(ref["pw"]))) * step <= 4.0 / ntot + 1e-6
    for k in ("rw", "rmw"):
        a, b = np.nan_to_num(out[k] * out["pw"]), np.nan_to_num(ref[k] * ref["pw"])
        assert np.max(np.abs(np.cumsum(a) - np.cumsum(b))) <= 4.0 * np.abs(b).max() + 1e-6 * np.abs(b).sum()


@pytest.mark.parametrize("case", GOLDEN_CASES)
def test_run_matches_oracle_and_reference(lib, case):
    meta, gold = load_golden(case)
    prm, xyz, box, fos = _frames_for(lib, meta)
    with lib.Engine(make_params(lib, prm), xyz.shape[1]) as eng:
        out = eng.run(xyz, box, fos)
        st = eng.stats()
    assert st["kernel_launches"] > 0 and st["frame_steps"] == len(fos)
    assert out["bins_out_of_range"] == 0
    ref = O.run(prm, xyz, [box] * len(xyz), fos)
    _compare_run(out, ref, prm, SPEC_TOL, case)
    # and directly against the reference program's own outputs
    for k, f in (("tcf_ir", "ir"), ("tcf_vv", "vv"), ("tcf_vh", "vh")):
        g = gold[f + "rtcf"][:, 1] + 1j * gold[f + "itcf"][:, 1]
        assert O.rel_l2(out[k], g) < 2 * SPEC_TOL, (case, k)
    for k, f in (("ls_ir", "irls"), ("ls_vv", "vvls"), ("ls_vh", "vhls")):
        assert O.rel_l2(out[k], gold[f][:, 1]) < 2 * SPEC_TOL, (case, k)
        np.testing.assert_array_equal(O.as_printed(out["ls_omega"]), gold[f][:, 0])
    assert O.rel_l2(out["sw"], gold["spdn"][:, 1]) < 2 * SPEC_TOL


def test_run_full_propagation_matches_psi_oracle(lib):
    """The oracle's F-matrix and psi-vector propagations agree; the GPU path carries F."""
    meta, _ = load_golden("multi_d2o_map1")
    prm, xyz, box, fos = _frames_for(lib, meta)
    a = O.run(prm, xyz, [box] * len(xyz), fos, propagate="full")
    b = O.run(prm, xyz, [box] * len(xyz), fos, propagate="psi")
    for k in ("tcf_ir", "tcf_vv", "tcf_vh"):
        assert O.rel_l2(a[k], b[k]) < 1e-12


def test_dropin_executable(lib, tmp_path):
    """calcir input.inp writes the 13 files of the reference, matching its outputs."""
    meta, gold = load_golden("hod_d2o")
    xyz, box = lib.synth_trajectory(meta["nmol"], meta["nframes"], seed=meta["seed"])
    lib.write_traj(str(tmp_path / "traj.cirtrj"), xyz, box, 0.010)
    lines = ["xtcf traj.cirtrj", "outf ref", "natom_mol 4"] + [f"{k} {v}" for k, v in meta["keys"].items()]
    (tmp_path / "input.inp").write_text("\n".join(lines) + "\n")
    r = subprocess.run([lib.EXE_PATH, "input.inp"], cwd=tmp_path, stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    for f in ["irrtcf", "iritcf", "vvrtcf", "vvitcf", "vhrtcf", "vhitcf", "spdn", "Pw", "Rw", "Rmw", "irls",
              "vvls", "vhls"]:
        a = np.loadtxt(tmp_path / f"ref_{f}.dat", ndmin=2)
        assert a.shape == gold[f].shape, f
        np.testing.assert_array_equal(a[:, 0], gold[f][:, 0])
        if f in ("Pw", "Rw", "Rmw"):
            continue
        assert O.rel_l2(a[:, 1], gold[f][:, 1]) < 2 * SPEC_TOL, f
    # the usage message and exit code of calcIR.cu:14-18
    r = subprocess.run([lib.EXE_PATH], stdout=subprocess.PIPE, text=True)
    assert r.returncode != 0 and "Usage" in r.stdout


def test_dropin_executable_reads_xtc(lib, tmp_path):
    """`xtcf traj.xtc` (a GROMACS trajectory, 1/1000 nm precision): the executable's spectra
    equal a run on the frames as decoded, and stay within the quantisation of the
    positions of the uncompressed run."""
    import ctypes as C
    meta, _ = load_golden("hod_d2o")
    xyz, box = lib.synth_trajectory(meta["nmol"], meta["nframes"], seed=meta["seed"])
    b = np.ascontiguousarray(np.broadcast_to(box, (xyz.shape[0], 3)), np.float32)
    t = (0.010 * np.arange(xyz.shape[0])).astype(np.float32)
    from calcir_gb300._lib import check, load
    check(load().cir_xtc_write(str(tmp_path / "traj.xtc").encode(), xyz.shape[1], xyz.shape[0],
                               C.c_void_p(xyz.ctypes.data), C.c_void_p(b.ctypes.data), C.c_void_p(t.ctypes.data),
                               C.c_float(1000.0)))
    lines = ["xtcf traj.xtc", "outf x", "natom_mol 4"] + [f"{k} {v}" for k, v in meta["keys"].items()]
    (tmp_path / "input.inp").write_text("\n".join(lines) + "\n")
    r = subprocess.run([lib.EXE_PATH, "input.inp"], cwd=tmp_path, stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    dec = np.zeros_like(xyz)
    check(load().cir_traj_read(str(tmp_path / "traj.xtc").encode(), 0, xyz.shape[0], C.c_void_p(dec.ctypes.data),
                               None, None))
    assert np.abs(dec - xyz).max() <= 0.5e-3 + 1e-6
    prm, _, _, fos = _frames_for(lib, meta)
    with lib.Engine(make_params(lib, prm), xyz.shape[1]) as eng:
        out = eng.run(dec, box, fos)
    for f, k in (("irrtcf", "tcf_ir"), ("vvrtcf", "tcf_vv"), ("spdn", "sw")):
        a = np.loadtxt(tmp_path / f"x_{f}.dat", ndmin=2)[:, 1]
        ref = out[k].real if k.startswith("tcf") else out[k]
        assert O.rel_l2(a, ref) < 1e-5, f


@pytest.mark.parametrize("nmol", [512, 1024])
def test_full_size_eigen_and_unitarity(lib, nmol):
    """Full-size systems (1024 / 2048 chromophores): eigen-residuals, orthogonality, and
    F stays unitary over propagation steps (a size-independent property)."""
    nf = 6
    xyz, box = lib.synth_trajectory(nmol, nf, seed=21)
    p = lib.default_params(species="H2O", model="tip4p2005", avef=3415.0)
    with lib.Engine(p, xyz.shape[1]) as eng:
        H, E, dip, pol = eng.build_hamiltonian(xyz, box)
        w, V = eng.eigh(H)
        n = H.shape[-1]
        F = np.eye(n, dtype=np.complex64)
        for f in range(1, nf):
            F = eng.propagate(V[f], w[f], np.float32(0.010), F)
    for f in (0, nf - 1):
        _check_eig(H[f], w[f], V[f], tol_scale=2.0)
    F64 = F.astype(np.complex128)
    assert np.abs(F64.conj().T @ F64 - np.eye(n)).max() < 2e-4
    # reference identity at t = 0: IR tcf = sum_a |mu_a|^2 (calcIR.cu:628-647 with F = I)
    Eo, Ho, do, po = O.frame(xyz[0], box, {"natom_mol": 4, "nchrom_mol": 2, "imodel": 1, "ispecies": 0,
                                           "map": 0, "avef": 3415.0})
    np.testing.assert_allclose(np.sum(dip[0].astype(np.float64) ** 2), np.sum(do ** 2), rtol=1e-4)


_FULL_PRM = {"natom_mol": 4, "nchrom_mol": 2, "imodel": 1, "ispecies": 0, "map": 0, "ntcfpoints": 6,
             "nsamples": 2, "sampleEvery": 0.03, "dt": 0.010, "t1": 0.260, "avef": 3415.0, "omegaStart": 1000,
             "omegaStop": 5000, "omegaStep": 1, "nzeros": 2000, "beginTime": 0.0}
_FULL_REF = {}


def _full_case(lib, nmol):
    """nmol molecules, 2 origins x 6 steps, and the oracle's whole job on them (computed once)."""
    if nmol not in _FULL_REF:
        prm = _FULL_PRM
        xyz, box = lib.synth_trajectory(nmol, 10, seed=4)
        fos = np.array([O.frame_index(prm, 0.010, s, k) for s in range(2) for k in range(6)], np.int32)
        _FULL_REF[nmol] = (xyz, box, fos, O.run(prm, xyz, [box] * len(xyz), fos))
    return _FULL_REF[nmol]


@pytest.mark.parametrize("nmol", [512, 1024])
@pytest.mark.parametrize("precision", ["fp32", "bf16x3", "tf32"])
def test_run_full_size_against_oracle(lib, precision, nmol):
    """512 molecules (the full configuration's system, 1024 chromophores) and 1024 molecules
    (2048 chromophores, the largest order of the eigensolver), 2 origins x 6 steps, vs the
    oracle: the plain form within 1e-4 and the mixed forms (tensor-core propagation and
    eigenvector products) within 1e-3 per spectrum."""
    prm = _FULL_PRM
    xyz, box, fos, ref = _full_case(lib, nmol)
    with lib.Engine(make_params(lib, prm, precision=precision), xyz.shape[1]) as eng:
        out = eng.run(xyz, box, fos)
    errs = {k: O.rel_l2(out[k], ref[k]) for k in ("tcf_ir", "tcf_vv", "tcf_vh", "sw", "ls_ir", "ls_vv", "ls_vh")}
    print(f"{2 * nmol} chromophores {precision}:", {k: f"{v:.2e}" for k, v in errs.items()})
    _compare_run(out, ref, prm, SPEC_TOL if precision == "fp32" else MIXED_TOL, f"full{nmol}-" + precision)


def test_run_ten_origins_full_size(lib):
    """Ten time origins of 1024 chromophores (the headline's origin count), 3 steps each: the
    split-BF16 propagation runs each product as two whole waves of 128 x 256 tiles (nine
    origins) and the tenth origin in 128 x 64 tiles.  Against the FP32 form of the same run
    and the oracle; an error confined to the tail origin would still move the origin average
    by a tenth of its size."""
    prm = dict(_FULL_PRM, nsamples=10, ntcfpoints=3, sampleEvery=0.02)
    fos = np.array([O.frame_index(prm, 0.010, s, k) for s in range(10) for k in range(3)], np.int32)
    xyz, box = lib.synth_trajectory(512, int(fos.max()) + 1, seed=6)
    outs = {}
    for precision in ("fp32", "bf16x3"):
        with lib.Engine(make_params(lib, prm, precision=precision), xyz.shape[1]) as eng:
            outs[precision] = eng.run(xyz, box, fos)
    ref = O.run(prm, xyz, [box] * len(xyz), fos)
    for k in ("tcf_ir", "tcf_vv", "tcf_vh", "sw", "ls_ir", "ls_vv", "ls_vh"):
        em, ep = O.rel_l2(outs["bf16x3"][k], ref[k]), O.rel_l2(outs["fp32"][k], ref[k])
        print(f"ten origins {k}: bf16x3 {em:.2e}, fp32 {ep:.2e}")
        assert ep < SPEC_TOL and em < 2e-4, (k, em, ep)


@pytest.mark.parametrize("n", [200, 1024, 2048])
def test_propagate_tensor_core_tf32(lib, n):
    """The tcgen05 TF32 propagation against the FP64 statement of the same step; TF32
    inputs carry 11 significant bits, so the bound is 2e-3 relative."""
    rng = np.random.default_rng(n + 7)
    nprop, dt = 2, 0.010
    A = np.stack([_sym(rng, n) for _ in range(nprop)])
    F = (rng.standard_normal((nprop, n, n)) + 1j * rng.standard_normal((nprop, n, n))).astype(np.complex64)
    with lib.Engine(lib.default_params(species="H2O", precision="tf32"), 8) as eng:
        w, V = eng.eigh(A)
        out = eng.propagate(V, w, np.float32(dt), F)
    for m in range(nprop):
        V64 = V[m].astype(np.float64)
        ph = np.exp(1j * w[m].astype(np.float64) * np.float32(dt) / HBAR)
        ref = (V64 * ph[None, :]) @ (V64.T @ F[m].astype(np.complex128))
        err = O.rel_l2(out[m], ref)
        print(f"tf32 propagation step, n={n}: relative L2 error {err:.2e}")
        assert err < 2e-3, err
        assert err > 1e-7, "tensor-core path produced FP32-exact output: is it running?"


@pytest.mark.parametrize("n", [200, 1024, 2048])
def test_propagate_tensor_core_bf16x3(lib, n):
    """3-pass split-BF16 tcgen05 propagation: about 16 significant bits per operand."""
    rng = np.random.default_rng(n + 11)
    nprop, dt = 2, 0.010
    A = np.stack([_sym(rng, n) for _ in range(nprop)])
    F = (rng.standard_normal((nprop, n, n)) + 1j * rng.standard_normal((nprop, n, n))).astype(np.complex64)
    with lib.Engine(lib.default_params(species="H2O", precision="bf16x3"), 8) as eng:
        w, V = eng.eigh(A)
        out = eng.propagate(V, w, np.float32(dt), F)
    for m in range(nprop):
        V64 = V[m].astype(np.float64)
        ph = np.exp(1j * w[m].astype(np.float64) * np.float32(dt) / HBAR)
        ref = (V64 * ph[None, :]) @ (V64.T @ F[m].astype(np.complex128))
        err = O.rel_l2(out[m], ref)
        print(f"bf16x3 propagation step, n={n}: relative L2 error {err:.2e}")
        assert 1e-8 < err < 5e-5, err


MIXED_TOL = 1e-3   # relative L2 per spectrum for the mixed-precision forms


@pytest.mark.parametrize("precision", ["bf16x3", "tf32"])
@pytest.mark.parametrize("case", ["small_h2o", "multi_d2o_map1"])
def test_run_mixed_precision_forms(lib, case, precision):
    """The tensor-core forms against the FP64 oracle: every IR/Raman spectrum within
    1e-3 relative L2 (the bound the mixed-precision form is held to)."""
    meta, _ = load_golden(case)
    prm, xyz, box, fos = _frames_for(lib, meta)
    with lib.Engine(make_params(lib, prm, precision=precision), xyz.shape[1]) as eng:
        out = eng.run(xyz, box, fos)
    ref = O.run(prm, xyz, [box] * len(xyz), fos)
    errs = {k: O.rel_l2(out[k], ref[k]) for k in ("tcf_ir", "tcf_vv", "tcf_vh", "ls_ir", "ls_vv", "ls_vh", "sw")}
    print(case, precision, {k: f"{v:.2e}" for k, v in errs.items()})
    for k, v in errs.items():
        assert v < MIXED_TOL, (k, v)


# the direct sum's tiles (64 and 256 terms, 64 output pairs) and its remainders, and the
# mixed-radix transform above 40 terms per unit of n's factor sum (n = 4200: 26, 40 * 26 = 1040)
@pytest.mark.parametrize("ntcf,nzeros", [(1, 1), (2, 0), (3, 1), (64, 63), (65, 64), (66, 191), (257, 255), (258, 511),
                                         (322, 4001), (1000, 3200), (2000, 2200)])
def test_lineshape_forms(lib, ntcf, nzeros):
    rng = np.random.default_rng(ntcf + nzeros)
    p = lib.default_params(species="H2O", ntcfpoints=ntcf, nzeros=nzeros, omegaStart=2000, omegaStop=5000, avef=3415.0)
    tcf = (rng.standard_normal(ntcf) + 1j * rng.standard_normal(ntcf)) * np.exp(-np.arange(ntcf) / 40)
    prm = {"ntcfpoints": ntcf, "nzeros": nzeros, "dt": 0.010, "avef": 3415.0, "omegaStart": 2000, "omegaStop": 5000}
    with lib.Engine(p, 8) as eng:
        om, val = eng.lineshape(tcf)
    om_ref, val_ref = O.lineshape_rows(prm, O.c2r(tcf, ntcf + nzeros))
    np.testing.assert_array_equal(om, om_ref.astype(np.float32))
    # four FP32 roundings (the sum, the axis step, the norm and the quotient), 6e-8 each
    assert O.rel_l2(val, val_ref) < 5e-7


# every form of the tridiagonalisation and the edges between them (152 SMs): resident in shared
# memory (n <= 128 in 4 warps for large batches, 8 warps up to 192, up to 256 for a single wave),
# streaming with two blocks per SM or one (n <= 512), one block or a cluster per matrix (n > 512)
@pytest.mark.parametrize("n,nmat", [(4, 305), (33, 3), (128, 305), (129, 2), (192, 2), (193, 153), (256, 2), (256, 153),
                                    (260, 2), (353, 153), (512, 153), (512, 2), (513, 2), (642, 12), (801, 30),
                                    (770, 60), (1025, 2), (1031, 20)])
def test_eigh_forms(lib, n, nmat):
    rng = np.random.default_rng(n + nmat)
    p = lib.default_params(species="H2O")
    base = rng.standard_normal((2, n, n)).astype(np.float32) * 5
    base = base + base.transpose(0, 2, 1)
    base[:, np.arange(n), np.arange(n)] += 150 * rng.standard_normal((2, n)).astype(np.float32)
    A = np.ascontiguousarray(base[np.arange(nmat) % 2])
    with lib.Engine(p, 8) as eng:
        w, V = eng.eigh(A)
    for i in sorted({0, 1, nmat - 1}):
        _check_eig(A[i], w[i], V[i])
    for i in range(2, nmat):      # every matrix of the batch, to the last bit
        assert np.array_equal(w[i], w[i % 2]) and np.array_equal(V[i], V[i % 2])


@pytest.mark.parametrize("nmol,nframes", [(8, 3), (33, 250), (100, 120)])
def test_build_forms(lib, nmol, nframes):
    """A batch (a thread per chromophore, four tiles of H a block) equals its frames built one by
    one (a warp per chromophore, one tile a block) to the last bit."""
    xyz, box = lib.synth_trajectory(nmol, nframes, seed=nmol)
    with lib.Engine(lib.default_params(species="H2O", model="tip4p2005"), 4 * nmol) as eng:
        batch = eng.build_hamiltonian(xyz, box)
        for f in (0, 1, nframes // 2, nframes - 1):
            one = eng.build_hamiltonian(xyz[f:f + 1], box)
            for b, o in zip(batch, one):
                np.testing.assert_array_equal(b[f], o[0])


@pytest.mark.parametrize("nmol,origins", [(27, 2), (33, 150), (41, 240)])
def test_contraction_forms(lib, nmol, origins):
    """The plain contraction with one row of F a warp and four (from 9728 rows), and blocks of 32
    and 64 rows (from 19456), with a ragged last block; the spectral density of many origins."""
    prm = {"natom_mol": 4, "nchrom_mol": 2, "nzeros": 64, "ntcfpoints": 3, "nsamples": origins, "sampleEvery": 0.01,
           "dt": 0.01, "t1": 0.26, "avef": 3415.0, "omegaStart": 2000.0, "omegaStop": 5000.0, "omegaStep": 7,
           "beginTime": 0.0, "map": 0, "imodel": 1, "ispecies": 0}
    xyz, box = lib.synth_trajectory(nmol, origins + 2, seed=3)
    fos = (np.arange(origins)[:, None] + np.arange(3)[None, :]).astype(np.int32).ravel()
    p = lib.default_params(species="H2O", model="tip4p2005", nsamples=origins, ntcfpoints=3, nzeros=64, omegaStep=7,
                           avef=3415.0, omegaStart=2000, omegaStop=5000, sampleEvery=0.01)
    with lib.Engine(p, xyz.shape[1]) as eng:
        out = eng.run(xyz, box, fos)
    ref = O.run(prm, xyz, np.broadcast_to(box, (len(xyz), 3)), fos)
    for k in ("tcf_ir", "tcf_vv", "tcf_vh", "ls_ir", "ls_vv", "ls_vh", "sw"):
        assert O.rel_l2(out[k], ref[k]) < 1e-4, k      # the plain form's bound


@pytest.mark.parametrize("n,batch", [(2, 1), (19, 2), (33, 3), (128, 1), (160, 60), (255, 24), (509, 2), (512, 4), (640, 1)])
def test_propagate_forms(lib, n, batch):
    """The FP32 products on small tiles and on the tensor cores, whole and ragged tiles, rows that
    are and are not 16-byte aligned, against 64 bits: 2^-23 sqrt(n) a product for the sums,
    2^-23 of the phase (at most 8 rad)."""
    rng = np.random.default_rng(n)
    V = np.stack([np.linalg.qr(rng.standard_normal((n, n)))[0] for _ in range(batch)]).astype(np.float32)
    w = rng.uniform(-400, 400, (batch, n)).astype(np.float32)
    F = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))).astype(np.complex64)
    with lib.Engine(lib.default_params(species="H2O", model="tip4p2005"), 12) as eng:
        got = eng.propagate(V, w, 0.1, F)
    V64 = V.astype(np.float64)
    phase = np.exp(1j * w.astype(np.float64) * np.float32(0.1) / HBAR)
    ref = V64 @ (phase[:, :, None] * (V64.swapaxes(1, 2) @ F.astype(np.complex128)))
    assert O.rel_l2(got, ref) < 2.0 ** -23 * (2 * np.sqrt(n) + 8)


@pytest.mark.parametrize("n,batch", [(2, 3), (3, 1), (33, 5), (130, 2), (513, 1)])
def test_unit_eigenvectors(lib, n, batch):
    """The plain form's eigenvectors have length one to the rounding of their elements (2^-24
    each, at most 2^-23 of the squared length, and as much again for the sum that scales them)."""
    A = np.random.default_rng(n).standard_normal((batch, n, n)).astype(np.float32)
    with lib.Engine(lib.default_params(species="H2O", model="tip4p2005"), 12) as eng:
        _, V = eng.eigh(A + A.swapaxes(1, 2))
    assert np.abs((np.asarray(V, np.float64) ** 2).sum(1) - 1).max() < 2.0 ** -22


# the merges of the divide and conquer: one lane a root in blocks of 64 to 512 threads, several
# lanes, clusters of 2 to 8 blocks with one lane and with several; spectra that deflate by small
# components and by close pairs, alone and in chains
@pytest.mark.parametrize("kind", ["pairs", "clusters", "glued", "graded"])
@pytest.mark.parametrize("n,nmat", [(66, 1), (130, 1), (130, 700), (300, 1), (516, 1), (520, 160), (1024, 1), (1100, 1)])
def test_merge_forms(lib, kind, n, nmat):
    rng = np.random.default_rng(n)
    if kind == "glued":           # equal Wilkinson blocks, weakly coupled
        d, e = np.abs(np.arange(n) % 21 - 10.0), np.where(np.arange(n - 1) % 21 == 20, 1e-4, 1.0)
        A = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    else:
        w = {"pairs": np.repeat(rng.standard_normal((n + 1) // 2), 2)[:n], "clusters": np.round(2 * rng.standard_normal(n)),
             "graded": 10.0 ** rng.uniform(-5, 2, n)}[kind]
        Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
        A = (Q * w) @ Q.T
    A = np.broadcast_to(((A + A.T) / 2).astype(np.float32), (nmat, n, n))
    with lib.Engine(lib.default_params(species="H2O"), 8) as eng:
        w, V = eng.eigh(np.ascontiguousarray(A))
    _check_eig(A[0], w[0], V[0])
    for i in range(1, nmat):
        assert np.array_equal(w[i], w[0]) and np.array_equal(V[i], V[0])


@pytest.mark.parametrize("nmol,origins", [(10, 1), (17, 9), (40, 3), (64, 1), (100, 4), (100, 40)])
def test_contraction_in_product(lib, nmol, origins):
    """The correlation terms added by the small products' epilogue (one group of threads up to order
    32, four above; ragged tiles), and by the contraction where the product is large, against the
    oracle."""
    test_contraction_forms(lib, nmol, origins)


@pytest.mark.parametrize("precision,tol", [("fp32", None), ("tf32", 2e-3), ("bf16x3", 5e-5)])
@pytest.mark.parametrize("n,batch", [(129, 60), (250, 40)])
def test_propagate_ragged_tiles(lib, precision, tol, n, batch):
    """More tiles than SMs whose last rows are missing: in every tensor-core product lanes of a warp
    leave the epilogue early, and all have to meet again for the next tile's loads.  Bounds as
    for one step in each form above."""
    rng = np.random.default_rng(n)
    V = np.stack([np.linalg.qr(rng.standard_normal((n, n)))[0] for _ in range(batch)]).astype(np.float32)
    w = rng.uniform(-400, 400, (batch, n)).astype(np.float32)
    F = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))).astype(np.complex64)
    with lib.Engine(lib.default_params(species="H2O", model="tip4p2005", precision=precision), 12) as eng:
        got = eng.propagate(V, w, 0.1, F)
    V64 = V.astype(np.float64)
    phase = np.exp(1j * w.astype(np.float64) * np.float32(0.1) / HBAR)
    ref = V64 @ (phase[:, :, None] * (V64.swapaxes(1, 2) @ F.astype(np.complex128)))
    for b in range(batch):
        assert O.rel_l2(got[b], ref[b]) < (tol or 2.0 ** -23 * (2 * np.sqrt(n) + 8)), b


@pytest.mark.parametrize("n,steps", [(256, 150), (320, 250), (512, 150), (1024, 250)])
def test_propagate_chain_keeps_length(lib, n, steps):
    """A long chain of plain steps neither shrinks nor stretches F: its projection on the same chain in
    64 bits stays at one.  Rounding to nearest leaves no more than 2^-28 of a fixed sign a step
    (1e-6 in 250); sums cut off toward zero lost 2^-23 each (3e-5)."""
    rng = np.random.default_rng(n)
    V = np.linalg.qr(rng.standard_normal((n, n)))[0].astype(np.float32)
    w = rng.uniform(-400, 400, n).astype(np.float32)
    F = np.eye(n, dtype=np.complex64)[None]
    V64 = V.astype(np.float64)
    ph = np.exp(1j * w.astype(np.float64) * np.float32(0.010) / HBAR)[:, None]
    ref = F[0].astype(np.complex128)
    mul = lambda a, z: (a @ z.view(np.float64).reshape(n, 2 * n)).view(np.complex128)
    with lib.Engine(lib.default_params(species="H2O", model="tip4p2005"), 12) as eng:
        for _ in range(steps):
            F = eng.propagate(V[None], w[None], 0.010, F)
            ref = mul(V64, np.ascontiguousarray(ph * mul(np.ascontiguousarray(V64.T), ref)))
    got = F[0].astype(np.complex128)
    drift = np.vdot(ref, got).real / np.vdot(ref, ref).real - 1
    print(f"n={n}, {steps} steps: projection - 1 {drift:.1e}, relative error {O.rel_l2(got, ref):.1e}")
    assert abs(drift) < steps * 2.0 ** -28


@pytest.mark.parametrize("n,batch", [(256, 24), (509, 2), (640, 1)])
def test_propagate_graded(lib, n, batch):
    """Rows and columns of F over nine orders of magnitude: every column is as exact as one of
    equal elements (the bound of test_propagate_forms)."""
    rng = np.random.default_rng(n)
    V = np.stack([np.linalg.qr(rng.standard_normal((n, n)))[0] for _ in range(batch)]).astype(np.float32)
    w = rng.uniform(-400, 400, (batch, n)).astype(np.float32)
    F = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    F = (F * 10.0 ** rng.uniform(-9, 0, (batch, n, 1)) * 10.0 ** rng.uniform(-9, 0, (batch, 1, n))).astype(np.complex64)
    with lib.Engine(lib.default_params(species="H2O", model="tip4p2005"), 12) as eng:
        got = eng.propagate(V, w, 0.1, F)
    V64 = V.astype(np.float64)
    phase = np.exp(1j * w.astype(np.float64) * np.float32(0.1) / HBAR)
    ref = V64 @ (phase[:, :, None] * (V64.swapaxes(1, 2) @ F.astype(np.complex128)))
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < 2.0 ** -23 * (2 * np.sqrt(n) + 8)


@pytest.mark.parametrize("n,batch", [(64, 2), (300, 8), (509, 2)])
@pytest.mark.parametrize("value", [np.inf, 2e38, 4e33, 3e-36, 1e-33, 1e-30])
def test_propagate_range(lib, n, batch, value):
    """A column of F of infinite, very large or very small values beside ordinary ones, in the small
    products and on the tensor cores: infinities come out as FP32 sums give them, the other columns'
    errors stay those of test_propagate_forms, also where BF16 terms would run out of their range."""
    rng = np.random.default_rng(n)
    V = (rng.uniform(0.5, 1.0, (batch, n, n)) / n).astype(np.float32)      # positive: no Inf - Inf, no 0 * Inf
    w = rng.uniform(50, 400, (batch, n)).astype(np.float32)                # phases in the first quadrant
    F = (rng.uniform(0.5, 1.0, (batch, n, n)) + 0.01j).astype(np.complex64)
    j = n // 2
    F[:, :, j] = (value if np.isfinite(value) else 1.0) * rng.uniform(0.5, 1.0, (batch, n))
    if not np.isfinite(value):
        F[:, n - 1, j] = np.inf
    with lib.Engine(lib.default_params(species="H2O", model="tip4p2005"), 12) as eng:
        got = eng.propagate(V, w, 0.010, F)
    keep = [c for c in range(n) if c != j or np.isfinite(value)]
    V64 = V.astype(np.float64)
    phase = np.exp(1j * w.astype(np.float64) * np.float32(0.010) / HBAR)
    F64 = F[:, :, keep].astype(np.complex128)
    ref = V64 @ (phase[:, :, None] * (V64.swapaxes(1, 2) @ F64))
    err = np.linalg.norm(got[:, :, keep] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < 2.0 ** -23 * (2 * np.sqrt(n) + 8)
    if not np.isfinite(value):
        assert np.all(got[:, :, j].real == np.inf) and np.all(got[:, :, j].imag == np.inf)


@pytest.mark.parametrize("n", [64, 100, 200, 300, 600])
@pytest.mark.parametrize("scale", [1e12, 1e17])
def test_eigh_large_matrices(lib, n, scale):
    """Matrices whose squares are in FP32's range but whose cubes are not."""
    A = (_sym(np.random.default_rng(n), n, 1.0) * np.float32(scale)).astype(np.float32)
    with lib.Engine(lib.default_params(species="H2O"), 8) as eng:
        w, V = eng.eigh(A[None])
    _check_eig(A / np.float32(scale), w[0] / np.float32(scale), V[0])


@pytest.mark.parametrize("n", [64, 100, 200, 300, 600])
@pytest.mark.parametrize("coupling", [1e-18, 1e-19])
def test_eigh_weak_couplings(lib, n, coupling):
    """Columns so short that the square of a reflector's scale overflows."""
    A = _sym(np.random.default_rng(n), n, coupling)
    A[np.arange(n), np.arange(n)] = np.arange(1, n + 1)
    with lib.Engine(lib.default_params(species="H2O"), 8) as eng:
        w, V = eng.eigh(A[None])
    _check_eig(A, w[0], V[0])


@pytest.mark.parametrize("n", [40, 129, 400, 1030])
def test_tcf_terms_infinite(lib, n):
    """An infinite dipole gives an infinite IR term, and the other terms as without it (2^-23 sqrt(n)
    for psi and its product with m(t), all terms being positive; five roundings more in VV)."""
    rng = np.random.default_rng(n)
    F = (rng.uniform(0.5, 1, (n, n)) + 1j * rng.uniform(0.5, 1, (n, n))).astype(np.complex64)
    d0, d1 = rng.uniform(0.5, 1, (2, 3, n)).astype(np.float32)
    p0, p1 = rng.uniform(0.5, 1, (2, 6, n)).astype(np.float32)
    d1[1, n // 2] = np.inf
    with lib.Engine(lib.default_params(species="H2O"), 8) as eng:
        out = np.zeros(6)      # (the wrapper's a + 1j b makes a NaN of an infinite b)
        lib.check(eng.lib.cir_tcf_terms(eng.h, n, *[lib.ptr(x) for x in (F.view(np.float32), d0, p0, d1, p1, out)]))
    assert out[0] == np.inf and out[1] == np.inf
    vv, vh = out[2] + 1j * out[3], out[4] + 1j * out[5]
    psi = F.astype(np.complex128) @ p0.astype(np.float64).T          # [n][6]
    P = p1.astype(np.float64) @ psi                                    # [b][a] = m_b . psi_a
    ii, ij = P[0, 0] + P[1, 1] + P[2, 2], P[3, 3] + P[4, 4] + P[5, 5]
    jj = P[:3, :3].sum() - ii
    tol = 2.0 ** -23 * (np.sqrt(n) + 5)
    assert abs(vv - (3 * ii + jj + 4 * ij) / 15) < tol * abs(vv)
    assert abs(vh - (2 * ii - jj + 6 * ij) / 30) < tol * abs(vv)


@pytest.mark.parametrize("start,stop", [(2000, 5000), (3415, 3415), (3000, 3200), (3600, 3700), (6000, 7000), (1, 900)])
def test_lineshape_rows(lib, start, stop):
    """The rows selected, for windows about, beside and beyond the axis, are those of cir_result_sizes."""
    p = lib.default_params(species="H2O", ntcfpoints=150, nzeros=2500, omegaStart=start, omegaStop=stop, avef=3415.0)
    prm = {"ntcfpoints": 150, "nzeros": 2500, "dt": 0.010, "avef": 3415.0, "omegaStart": start, "omegaStop": stop}
    tcf = np.exp(-np.arange(150) / 40.0) * (1 + 1j)
    with lib.Engine(p, 8) as eng:
        om, _ = eng.lineshape(tcf)
    ref, _ = O.lineshape_rows(prm, O.c2r(tcf, 2650))
    assert len(om) == lib.result_sizes(p)[2]
    np.testing.assert_array_equal(om, ref.astype(np.float32))


def test_create_with_very_long_padding(lib):
    """A context for a transform of more than 2^30 points is made without working through them."""
    with lib.Engine(lib.default_params(species="H2O", nzeros=1_900_000_000), 8):
        pass


@pytest.mark.parametrize("n,batch", [(1, 3), (24, 40), (32, 100), (33, 150), (63, 64), (65, 150), (66, 152), (98, 64), (113, 16)])
def test_propagate_tile_forms(lib, n, batch):
    """The products of many small matrices on tiles of 64 and 128, whole and ragged, aligned rows and not."""
    test_propagate_forms(lib, n, batch)


@pytest.mark.parametrize("nmol,origins", [(12, 60), (25, 100), (32, 64), (33, 160), (49, 60)])
def test_contraction_in_tiles(lib, nmol, origins):
    """The correlation terms from tiles of 64, and by their own launch after tiles of 128."""
    test_contraction_forms(lib, nmol, origins)
