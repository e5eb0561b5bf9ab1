"""Performance cases of the framework: the calls its users make, through the public entry points.

A case is one of seven kinds of work:

* ``lineshape``   the transform of a correlation function into a printed spectrum (cir_lineshape)
* ``density``     the spectral density of one diagonalised frame (cir_spectral_density)
* ``hamiltonian`` field, maps, Hamiltonian, dipoles and polarisabilities of frames (cir_build_hamiltonian)
* ``frame``       one time step of a caller's own loop on device buffers: build, diagonalise and
                  propagate F for one or several trajectories (cir_build_hamiltonian, cir_eigh,
                  cir_propagate), in the plain form; the mixed form is measured on whole jobs
* ``run``         a whole job of one trajectory (Engine.run)
* ``multi``       a whole job of many trajectories in boxes of uneven size (Engine.run_multi)
* ``gradient``    a spectrum-mismatch loss and its gradient (Engine.loss_grad)

``exact`` restates the equations in float64 with torch alone: the propagator is applied as the
Taylor series of exp(i H dt / hbar), so it needs no eigendecomposition, and the gradient is
autograd's through the whole chain.
"""
import math

import numpy as np
import torch

import calcir_gb300 as cg
from calcir_gb300._lib import check, ptr

HBAR, PI = 5.308837367, 3.14159265359      # cm^-1 ps, and the constant the spectra are defined with
BOHR, HARTREE = np.float32(18.8973), np.float32(2.1947463e5)
CUTOFF, OM, QH, QM, TDM = (np.float32(x) for x in (0.7831, 0.0150, 0.52, 1.04, 0.067))
DT = 0.010                                   # ps between steps and between frames

# frequency, position, momentum, dipole-derivative and intramolecular maps by (map, species)
MAPS = {
    (0, "H2O"): (3670.2, -3541.7, -152677.0, 0.19285, -1.7261e-5, 1.6466, 5.7692e-4,
                 0.1646, 11.39, 63.41, -1361.0, 27165.0, -1.887),
    (0, "D2O"): (2767.8, -2630.3, -102601.0, 0.16593, -2.0632e-5, 2.0475, 8.9108e-4,
                 0.1646, 11.39, 63.41, -1361.0, 27165.0, -1.887),
    (1, "H2O"): (3732.9, -3519.8, -153520.0, 0.19318, -1.7248e-5, 1.6102, 5.8697e-4,
                 0.1622, 10.381, 137.6, -1360.8, 27171.0, -1.887),
    (1, "D2O"): (2748.2, -2572.2, -102980.0, 0.16598, -2.0752e-5, 1.9813, 9.1419e-4,
                 0.1622, 10.381, 137.6, -1360.8, 27171.0, -1.887),
}
WINDOW = {"H2O": (3415.2, 2000.0, 5000.0), "D2O": (2500.0, 1500.0, 3500.0)}   # avef, omegaStart, omegaStop


def _case(name, kind, **kw):
    c = {"kind": kind, "nmol": 64, "frames": 1, "origins": 1, "points": 150, "zeros": 25600, "precision": "fp32",
         "map": 0, "species": "H2O", "sizes": "", "copies": 1}
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the end of every job and of every refit of a damping time: 150 points padded with 25600 zeros
        _case("lineshape_150", "lineshape"),
        # the density of states of one snapshot of 512 molecules
        _case("density_512", "density", nmol=512),
        # a simulation engine asking for the Hamiltonian of its current frame: the smallest call
        _case("hamiltonian_64", "hamiltonian", nmol=64),
        # a stored trajectory of an uneven box turned into Hamiltonians for a caller's own analysis
        _case("hamiltonian_343x200", "hamiltonian", nmol=343, frames=200),
        # on-the-fly spectroscopy: one frame at a time from inside a simulation's time step
        _case("frame_64_fp32", "frame", nmol=64),
        _case("frame_512_fp32", "frame", nmol=512),
        # the same for the large box
        _case("frame_1024_fp32", "frame", nmol=1024),
        # the default job (one origin, 150 points) of the small box, in the plain drop-in form
        _case("run_64_fp32", "run", nmol=64),
        # a production box in the plain form: 10 origins, the first 20 points
        _case("run_512_fp32", "run", nmol=512, origins=10, points=20),
        # the same box in the mixed form with more origins: the largest batches
        _case("run_512_bf16x3", "run", nmol=512, origins=25, points=24, precision="bf16x3"),
        # replicas of boxes of uneven size in one call
        _case("multi_bf16x3", "multi", sizes="128,216,343,512", copies=16, points=20, precision="bf16x3"),
        # one evaluation of a map refit against measured spectra
        _case("gradient_256", "gradient", nmol=256, origins=4, points=100),
    ]


def draw(rng):
    def logint(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["lineshape", "density", "hamiltonian", "frame", "frame", "run", "run", "run", "multi", "gradient"])
    c = _case(None, kind, map=rng.choice([0, 0, 1]), species=rng.choice(["H2O", "H2O", "H2O", "D2O"]))
    if kind == "lineshape":
        c.update(points=logint(40, 400), zeros=logint(2000, 40000))
    elif kind == "density":
        c.update(nmol=logint(24, 1024))
    elif kind == "hamiltonian":
        c.update(nmol=logint(24, 512))
        c.update(frames=logint(1, max(1, int(200 * (343 / c["nmol"]) ** 2) if c["nmol"] > 343 else 200)))
    elif kind == "frame":
        c.update(nmol=logint(24, 1024))
        c.update(frames=1 if c["nmol"] > 512 else logint(1, max(1, min(64, 8 * (512 // c["nmol"]) ** 2))))
    elif kind == "run":
        c.update(nmol=logint(24, 512), precision=rng.choice(["fp32", "bf16x3"]), origins=rng.randint(1, 16))
        c.update(points=rng.randint(10, 24 if c["nmol"] > 128 or c["precision"] != "fp32" else 150))
    elif kind == "multi":
        sizes = sorted({logint(24, 400) for _ in range(rng.randint(2, 4))})
        c.update(sizes=",".join(str(s) for s in sizes), copies=rng.randint(1, 16), points=rng.randint(10, 20),
                 precision=rng.choice(["fp32", "bf16x3"]))
    else:
        c.update(nmol=logint(24, 256), origins=rng.randint(1, 4), points=rng.randint(20, 100))
    return c


# ---------------------------------------------------------------- inputs

def _params(case):
    avef, lo, hi = WINDOW[case["species"]]
    return dict(model="tip4p2005", species=case["species"], map=case["map"], ntcfpoints=case["points"],
                nsamples=case["origins"], sampleEvery=10 * DT, dt=DT, t1=0.26, avef=avef, omegaStart=lo,
                omegaStop=hi, omegaStep=1, nzeros=case["zeros"])


def _sizes(case):
    if case["kind"] == "multi":
        return [int(s) for s in case["sizes"].split(",") for _ in range(case["copies"])]
    return [case["nmol"]]


def _frames_of_step(case):
    """Origins ten steps apart along one trajectory."""
    return (10 * np.arange(case["origins"])[:, None] + np.arange(case["points"])[None, :]).astype(np.int32).ravel()


def _box(nmol, frames, seed):
    """A synthetic trajectory; the generator gives up on a start where a molecule has no room."""
    for again in range(50):
        try:
            return cg.synth_trajectory(nmol, frames, seed=seed + 10_000_019 * again)
        except cg.CirError:
            pass
    raise RuntimeError("no trajectory of %d molecules from seed %d" % (nmol, seed))


def _trajectories(case, seed):
    """The library's synthetic trajectories: [(xyz (frames, atoms, 3), boxes (frames, 3))], float32."""
    nf = case["frames"] if case["kind"] in ("hamiltonian", "frame") else int(_frames_of_step(case).max()) + 1
    out = []
    for i, nmol in enumerate(_sizes(case)):
        if case["kind"] == "frame":      # the current frames of independent trajectories
            parts = [_box(nmol, 1, 1000 * seed + f + 1) for f in range(nf)]
            xyz, box = np.concatenate([p[0] for p in parts]), parts[0][1]
        else:
            xyz, box = _box(nmol, nf, 1000 * seed + i + 1)
        out.append((xyz, np.tile(np.asarray(box, np.float32), (nf, 1))))
    return out


def _correlation(case, seed):
    """A damped correlation function as a job ends with: decaying, beating, of either sign."""
    rng = np.random.default_rng(seed)
    t = DT * np.arange(case["points"])
    w = rng.normal(0, 150, 40) / HBAR
    a = rng.uniform(0.5, 1.5, 40)
    return (a[None, :] * np.exp(1j * w[None, :] * t[:, None])).sum(1) * np.exp(-t / 0.52)


def _propagated(n, batch, seed):
    """A dense complex F with rows of unit norm, as some hundred steps leave it."""
    g = torch.Generator().manual_seed(seed)
    return torch.view_as_complex(torch.randn(batch, n, n, 2, generator=g) / math.sqrt(2 * n))


def _eigenpairs(case, seed):
    """A frame's eigenpairs: random orthonormal vectors (a product of reflections) and a water band."""
    g = torch.Generator().manual_seed(seed)
    n = 2 * case["nmol"]
    V = torch.eye(n)
    for v in torch.randn(24, n, generator=g):
        V -= torch.outer(V @ v, v) * (2.0 / float(v @ v))
    w = torch.sort(torch.randn(n, generator=g) * 150.0).values
    return V, w, 0.1 * torch.randn(3, n, generator=g)


def _target(case, rows):
    """Measured IR and VV bands (Gaussians) on the printed frequency axis, of the job's own size."""
    avef = WINDOW[case["species"]][0]
    return [(s * case["nmol"] * np.exp(-0.5 * ((rows - avef - d) / w) ** 2)).astype(np.float32)
            for s, d, w in ((4e-6, 20.0, 90.0), (1.2e-3, -60.0, 110.0))]


def _device_engine(case):
    eng = cg.Engine(cg.default_params(**_params(case), precision=case["precision"]), 4 * _sizes(case)[0])
    stream = torch.cuda.Stream()
    eng.set_stream(stream.cuda_stream)
    return eng, stream


def prepare(case, seed):
    kind = case["kind"]
    eng, stream = _device_engine(case)
    s = {"case": case, "eng": eng, "stream": stream}
    n = 2 * case["nmol"]
    if kind == "lineshape":
        s["tcf"] = _correlation(case, seed)
    elif kind == "density":
        V, w, dip = _eigenpairs(case, seed)
        s.update(V=V.T.contiguous().cuda(), w=w.cuda(), dip=dip.cuda())       # column j contiguous
        s["sw"] = torch.zeros(cg.result_sizes(eng.params)[1], device="cuda")
    else:
        traj = _trajectories(case, seed)
        if kind == "multi":
            s["traj"] = [(torch.from_numpy(x).cuda(), torch.from_numpy(b).cuda(), _frames_of_step(case)) for x, b in traj]
        elif kind == "gradient":       # host arrays, as a fitting script holds them
            s.update(xyz=traj[0][0], box=traj[0][1], fos=_frames_of_step(case))
            s["target"] = _target(case, _rows(case)[0])
        else:
            s.update(xyz=torch.from_numpy(traj[0][0]).cuda(), box=torch.from_numpy(traj[0][1]).cuda())
            nf = s["xyz"].shape[0]
            if kind == "run":
                s["fos"] = _frames_of_step(case)
            else:
                s.update(H=torch.empty(nf, n, n, device="cuda"), E=torch.empty(nf, n, device="cuda"),
                         dip=torch.empty(nf, 3, n, device="cuda"), pol=torch.empty(nf, 6, n, device="cuda"))
            if kind == "frame":
                s["F0"] = _propagated(n, nf, seed).cuda()
                s.update(F=torch.empty_like(s["F0"]), w=torch.empty(nf, n, device="cuda"))
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------- one pass

def _spectra(res):
    """A job's outputs.  The correlation functions are sums of float32 products that the library
    hands over in doubles and prints with six digits: they are taken in single precision.  The
    eigenvalue histograms (pw, rw, rmw) are left out: a count per 1 cm^-1 bin is a step function
    of the last bit of every eigenvalue."""
    out = {k: res[k].astype(np.complex64) for k in ("tcf_ir", "tcf_vv", "tcf_vh")}
    out.update({k: res[k] for k in ("sw", "ls_omega", "ls_ir", "ls_vv", "ls_vh")})
    return out


def run(s):
    case, eng, kind = s["case"], s["eng"], s["case"]["kind"]
    lib, h = eng.lib, eng.h
    if kind == "lineshape":
        omega, inten = eng.lineshape(s["tcf"])
        return {"omega": omega, "intensity": inten}
    if kind == "density":
        with torch.cuda.stream(s["stream"]):
            s["sw"].zero_()
        check(lib.cir_spectral_density(h, 2 * case["nmol"], ptr(s["V"]), ptr(s["w"]), ptr(s["dip"]), ptr(s["sw"])))
        return s["sw"]
    if kind == "run":
        return _spectra(eng.run(s["xyz"].data_ptr(), s["box"].data_ptr(), s["fos"], nframes=s["xyz"].shape[0]))
    if kind == "multi":
        # 64 outputs at most: the stacked spectra of all trajectories
        res = [_spectra(r) for r in eng.run_multi(s["traj"])]
        return {k: np.stack([r[k] for r in res]) for k in res[0]}
    if kind == "gradient":
        loss, grad = eng.loss_grad(s["xyz"], s["box"], s["fos"], *s["target"])
        # the coefficients themselves are single precision (cir_set_coeffs)
        return {"loss": np.float32(loss), "grad": grad.astype(np.float32)}
    nf, n = s["xyz"].shape[0], 2 * case["nmol"]
    check(lib.cir_build_hamiltonian(h, nf, ptr(s["xyz"]), ptr(s["box"]), ptr(s["H"]), ptr(s["E"]), ptr(s["dip"]), ptr(s["pol"])))
    if kind == "hamiltonian":
        return {"H": s["H"], "eproj": s["E"], "dip": s["dip"], "pol": s["pol"]}
    # the eigenvectors replace H; their signs and the basis of close pairs are free, F is not
    with torch.cuda.stream(s["stream"]):
        s["F"].copy_(s["F0"])
    check(lib.cir_eigh(h, nf, n, ptr(s["H"]), ptr(s["w"])))
    check(lib.cir_propagate(h, nf, n, ptr(s["H"]), ptr(s["w"]), DT, ptr(s["F"])))
    return {"w": s["w"], "F": s["F"], "dip": s["dip"], "pol": s["pol"]}


# ---------------------------------------------------------------- what one pass cannot do without

def work(case):
    kind, n = case["kind"], 2 * case["nmol"]
    avef, lo, hi = WINDOW[case["species"]]
    nfft, nom = case["points"] + case["zeros"], int(hi - lo) + 1
    spectra = 16.0 * case["points"] * 3 + 4.0 * (5 * nom)
    fft = 5.0 * nfft * math.log2(nfft)
    # per pair of chromophores the coupling (about 40 operations, once by symmetry), per chromophore and
    # molecule the distance test and the field of those inside the cutoff
    def build(n):
        return 20.0 * n * n + 15.0 * n * (n / 2)

    # tridiagonalisation 4/3 n^3, the eigenvectors' back-transformation 2 n^3
    def eig(n):
        return 10.0 / 3.0 * n ** 3

    def prop(n):
        return 8.0 * n ** 3        # V (e^{i L t} (V^T F)), V real, F complex

    if kind == "lineshape":
        return {"bytes": 16.0 * case["points"] + 8.0 * nom, "flops": fft}
    if kind == "density":
        return {"bytes": 4.0 * (n * n + 4 * n + 2 * nom), "flops": 6.0 * n * n + 8.0 * n * nom}
    if kind == "hamiltonian":
        return {"bytes": case["frames"] * 4.0 * (n * n + 6 * n + 10 * n), "flops": case["frames"] * build(n)}
    if kind == "frame":
        return {"bytes": case["frames"] * 4.0 * (6 * n + 4 * n * n + 10 * n),
                "flops": case["frames"] * (build(n) + eig(n) + prop(n))}
    steps = case["origins"] * case["points"]
    if kind == "gradient":         # nine vectors forward, recomputed and backward; two products for dL/dH
        return {"bytes": steps * 24.0 * n,
                "flops": steps * (build(n) * 2 + eig(n) + 3 * 72.0 * n * n + 4.0 * n ** 3) + 2 * fft}
    tot = {"bytes": 0.0, "flops": 0.0}
    for nmol in _sizes(case):
        m = 2 * nmol
        tot["bytes"] += steps * 24.0 * m + spectra
        tot["flops"] += steps * (build(m) + eig(m) + prop(m)) + 3 * fft
    return tot


# ---------------------------------------------------------------- the same results in float64

def _f(x):
    return float(np.float32(x))


def _theta(case):
    return torch.tensor([_f(x) for x in MAPS[case["map"], case["species"]]], dtype=torch.float64, device=_dev())


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _wrap(d, box):
    return d - box * torch.floor(d / box + 0.5)


def _geometry(xyz, box):
    """What does not depend on the maps: field, unit vectors and the dipole-dipole tensor of one frame."""
    x32 = torch.from_numpy(np.ascontiguousarray(xyz)).to(_dev()).reshape(-1, 4, 3)
    b32 = torch.from_numpy(np.ascontiguousarray(box)).to(_dev())
    x, b = x32.double(), b32.double()
    O, Hs, M = x[:, 0], x[:, 1:3], x[:, 3]
    nmol, n = x.shape[0], 2 * x.shape[0]
    H = Hs.reshape(n, 3)
    mol = torch.arange(n, device=x.device) // 2
    u = _wrap(H - O[mol], b)
    u = u / u.norm(dim=1, keepdim=True)
    dM = _wrap(M - O, b)
    M = O + _f(OM) * dM / dM.norm(dim=1, keepdim=True)
    # the O..H cutoff is a decision on the float32 distance
    d32 = x32[:, 0][None, :, :] - x32[:, 1:3].reshape(n, 3)[:, None, :]
    q = d32 / b32
    d32 = d32 - b32 * (torch.sign(q) * torch.floor(q.abs() + 0.5))
    r32 = torch.sqrt((d32[..., 0] * d32[..., 0] + d32[..., 1] * d32[..., 1]) + d32[..., 2] * d32[..., 2])
    inside = (r32 <= torch.tensor(CUTOFF, device=x.device)) & (mol[:, None] != torch.arange(nmol, device=x.device)[None, :])
    E = torch.zeros(n, 3, dtype=torch.float64, device=x.device)
    for site, charge in ((Hs[:, 0], _f(QH)), (Hs[:, 1], _f(QH)), (M, -_f(QM))):
        d = _wrap(H[:, None, :] - site[None, :, :], b) * _f(BOHR)
        r = d.norm(dim=2)
        r = torch.where(inside, r, torch.ones_like(r))
        E += (torch.where(inside, charge / r ** 3, torch.zeros_like(r))[..., None] * d).sum(1)
    E = (E * u).sum(1)
    t = _wrap(O[mol] + _f(TDM) * u, b)
    d = _wrap(t[:, None, :] - t[None, :, :], b)
    r = d.norm(dim=2)
    other = mol[:, None] != mol[None, :]
    r = torch.where(other, r, torch.ones_like(r))
    d = d / r[..., None]
    un, vn = (u[:, None, :] * d).sum(2), (u[None, :, :] * d).sum(2)
    g = torch.where(other, (u @ u.T - 3.0 * un * vn) / (r * _f(BOHR)) ** 3 * _f(HARTREE), torch.zeros_like(r))
    return E, u, g


def _system(case, geo, th):
    """H (about avef), the nine dipole and polarisability rows of one frame."""
    E, u, g = geo
    w = th[0] + th[1] * E + th[2] * E * E
    x, p = th[3] + th[4] * w, th[5] + th[6] * w
    mup = th[7] + th[8] * E + th[9] * E * E
    a = x * mup
    H = g * torch.outer(a, a) + torch.diag(w - _f(WINDOW[case["species"]][0]))
    i = torch.arange(0, E.shape[0], 2, device=E.device)
    intra = (th[10] + th[11] * (E[i] + E[i + 1])) * x[i] * x[i + 1] + th[12] * p[i] * p[i + 1]
    H = H.index_put((i, i + 1), intra).index_put((i + 1, i), intra)
    ux, uy, uz = u[:, 0], u[:, 1], u[:, 2]
    k = _f(4.6)
    m = torch.stack([ux * a, uy * a, uz * a, (k * ux * ux + 1) * x, (k * uy * uy + 1) * x, (k * uz * uz + 1) * x,
                     k * ux * uy * x, k * uy * uz * x, k * uz * ux * x])
    return H, m


def _propagate(H, re, im):
    """exp(i H dt / hbar) (re + i im) by its Taylor series; H (..., n, n), re and im (..., n, k)."""
    tau = _f(DT) / HBAR
    k = re.shape[-1]
    term = torch.cat([re, im], -1)
    total = term
    for m in range(1, 33):
        y = (H @ term) * (tau / m)
        term = torch.cat([-y[..., k:], y[..., :k]], -1)
        total = total + term
    return total[..., :k], total[..., k:]


def _terms(psi, m):
    """IR, VV and VH terms of psi_a = F m_a(0) with m(t); psi (..., n, 9), m (..., 9, n)."""
    c = m.transpose(-1, -2)
    ir = (c[..., :3] * psi[..., :3]).sum((-1, -2))
    ii = (c[..., 3:6] * psi[..., 3:6]).sum((-1, -2))
    ij = (c[..., 6:] * psi[..., 6:]).sum((-1, -2))
    jj = (c[..., 3:6].sum(-1) * psi[..., 3:6].sum(-1)).sum(-1) - ii
    return ir, (3 * ii + jj + 4 * ij) / 15, (2 * ii - jj + 6 * ij) / 30


def _rows(case):
    """The printed rows of a lineshape: frequencies, their places in the transform, the norm."""
    avef, lo, hi = (np.float32(v) for v in WINDOW[case["species"]])
    K, Z = case["points"], case["zeros"]
    n = K + Z
    factor = np.float32(2 * PI * HBAR / float(np.float32(DT) * np.float32(n)))
    i = np.arange(n // 2, n)
    f1 = (-(i - n)).astype(np.float32) * factor + avef
    j = np.arange(0, K + Z // 2)
    f2 = (-j).astype(np.float32) * factor + avef
    keep1, keep2 = f1 <= hi, f2 >= lo
    return (np.concatenate([f1[keep1], f2[keep2]]), np.concatenate([i[keep1], j[keep2]]),
            float(factor * np.float32(n)))


def _transform(case, tcf):
    """Lineshape values of a damped correlation function (torch complex128)."""
    _, at, norm = _rows(case)
    n = case["points"] + case["zeros"]
    X = torch.zeros(n // 2 + 1, dtype=torch.complex128, device=tcf.device)
    keep = min(case["points"], n // 2 + 1)
    X = torch.cat([tcf[:1].real.to(tcf.dtype), tcf[1:keep], X[keep:]])
    y = torch.fft.irfft(X, n) * n
    return y[torch.from_numpy(at).to(y.device)] / norm


def _job(case, xyz, box, th):
    """Damped correlation functions, lineshapes and spectral density of one trajectory's job."""
    S, K = case["origins"], case["points"]
    fos = _frames_of_step(case).reshape(S, K)
    last = {f: int(np.argwhere(fos == f)[:, 1].max()) for f in np.unique(fos)}
    cache, sums, densities = {}, [[], [], []], []
    for k in range(K):
        for f in fos[:, k]:
            if f not in cache:
                cache[f] = _system(case, _geometry(xyz[f], box[f]), th)
        m = torch.stack([cache[f][1] for f in fos[:, k]])
        H = torch.stack([cache[f][0] for f in fos[:, k]])
        if k == 0:
            re, im = m.transpose(-1, -2), torch.zeros_like(m).transpose(-1, -2)
            if case["kind"] != "gradient":
                densities = [_density(case, *torch.linalg.eigh(H[s]), m[s, :3]) for s in range(S)]
        else:
            re, im = _propagate(H, re, im)
        for q, (a, b) in enumerate(zip(_terms(re, m), _terms(im, m))):
            sums[q].append(torch.complex(a.sum(), b.sum()))
        for f in [f for f in cache if last[f] <= k]:
            del cache[f]
    t = torch.arange(K, dtype=torch.float64, device=_dev()) * _f(DT)
    decay = torch.exp(-t / (2 * _f(0.26))) / S
    tcf = [torch.stack(x) * decay for x in sums]
    return tcf, [_transform(case, x) for x in tcf], sum(densities) / S if densities else None


def _density(case, w, V, dip):
    avef, lo, hi = WINDOW[case["species"]]
    gamma = HBAR / (2 * _f(0.26))
    mu2 = ((dip @ V) ** 2).sum(0)
    om = torch.arange(int(hi - lo) + 1, dtype=torch.float64, device=w.device) + _f(lo)
    dw = om[:, None] - (w[None, :] + _f(avef))
    return (mu2 * gamma / (dw * dw + gamma * gamma)).sum(1) / PI


def exact(case, seed):
    kind = case["kind"]
    th = _theta(case)
    if kind == "lineshape":
        tcf = torch.from_numpy(_correlation(case, seed)).to(_dev())
        return {"omega": _rows(case)[0].astype(np.float64), "intensity": _transform(case, tcf)}
    if kind == "density":
        V, w, dip = (x.double().to(_dev()) for x in _eigenpairs(case, seed))
        return _density(case, w, V, dip)
    traj = _trajectories(case, seed)
    if kind in ("hamiltonian", "frame"):
        geo = [_geometry(x, b) for x, b in zip(*traj[0])]
        sysm = [_system(case, g, th) for g in geo]
        m = torch.stack([y for _, y in sysm])
        out = {"dip": m[:, :3], "pol": m[:, 3:]}
        if kind == "hamiltonian":
            return dict(out, H=torch.stack([x for x, _ in sysm]), eproj=torch.stack([g[0] for g in geo]))
        F0 = _propagated(2 * case["nmol"], case["frames"], seed).to(_dev()).to(torch.complex128)
        F = [torch.complex(*_propagate(H, f.real, f.imag)) for (H, _), f in zip(sysm, F0)]
        return dict(out, F=torch.stack(F), w=torch.stack([torch.linalg.eigvalsh(H) for H, _ in sysm]))
    if kind == "gradient":
        th.requires_grad_(True)
        _, ls, _ = _job(case, *traj[0], th)
        want = [torch.from_numpy(t).double().to(_dev()) for t in _target(case, _rows(case)[0])]
        loss = ((ls[0] - want[0]) ** 2).sum() + ((ls[1] - want[1]) ** 2).sum()
        loss.backward()
        return {"loss": loss.detach(), "grad": th.grad}
    jobs = [_job(case, x, b, th) for x, b in traj]
    names = ("ir", "vv", "vh")
    out = {"tcf_" + q: torch.stack([j[0][i] for j in jobs]) for i, q in enumerate(names)}
    out.update({"ls_" + q: torch.stack([j[1][i] for j in jobs]) for i, q in enumerate(names)})
    out["sw"] = torch.stack([j[2] for j in jobs])
    out["ls_omega"] = np.stack([_rows(case)[0].astype(np.float64)] * len(jobs))
    return out if kind == "multi" else {k: v[0] for k, v in out.items()}
