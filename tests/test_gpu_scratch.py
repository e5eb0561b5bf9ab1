"""Calls do not depend on what earlier ones left in the context's scratch: after one on device data
with a NaN (the library checks host arguments only, so such a call runs and its result is NaN or an
error), valid calls give what a fresh context gives."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sym(n, seed):
    a = np.random.default_rng(seed).standard_normal((1, n, n)).astype(np.float32) * 30
    return a + a.transpose(0, 2, 1)


def _eigh(eng, A):
    """cir_eigh on a device copy of A: (status, w, V)."""
    import torch
    from calcir_gb300._lib import ptr
    dA = torch.from_numpy(A).cuda()
    w = torch.empty(A.shape[:2], device="cuda")
    torch.cuda.synchronize()
    rc = eng.lib.cir_eigh(eng.h, A.shape[0], A.shape[1], ptr(dA), ptr(w))
    return rc, w.cpu().numpy(), dA.cpu().numpy()


@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
def test_eigh_after_a_nan(lib, precision):
    p = lib.default_params(species="H2O", precision=precision)
    bad = _sym(600, 1)
    bad[0, 17, 400] = bad[0, 400, 17] = np.nan
    with lib.Engine(p, 8) as eng:
        rc, w, _ = _eigh(eng, bad)
        assert rc != 0 or not np.isfinite(w).all()
        for n in (514, 600, 1024, 1030, 200):
            A = _sym(n, n)
            rc, w, V = _eigh(eng, A)
            with lib.Engine(p, 8) as fresh:
                rc0, w0, V0 = _eigh(fresh, A)
            assert rc == rc0 == 0 and np.isfinite(w0).all() and np.isfinite(V0).all()
            np.testing.assert_array_equal(w, w0)
            np.testing.assert_array_equal(V, V0)


def test_run_after_a_nan(lib):
    import torch
    nmol = 300
    xyz, box = lib.synth_trajectory(nmol, 2, seed=3)
    p = lib.default_params(model="tip4p2005", species="H2O", ntcfpoints=2, nsamples=1, nzeros=200, avef=3415.0)
    bx = torch.from_numpy(np.tile(np.asarray(box, np.float32), (2, 1))).cuda()
    fos = np.arange(2, dtype=np.int32)
    out = []
    for first in (True, False):
        with lib.Engine(p, xyz.shape[1]) as eng:
            for spoil in ((True, False) if first else (False,)):
                x = np.array(xyz)
                if spoil:
                    x[0, 41] = np.nan
                dx = torch.from_numpy(x).cuda()
                torch.cuda.synchronize()
                try:
                    res = eng.run(dx.data_ptr(), bx.data_ptr(), fos, nframes=2)
                except lib.CirError:
                    assert spoil
            out.append(res)
    for k in ("tcf_ir", "tcf_vv", "tcf_vh", "sw", "ls_ir"):
        assert np.isfinite(out[1][k]).all()
        np.testing.assert_allclose(out[0][k], out[1][k], rtol=1e-12, atol=1e-12 * np.abs(out[1][k]).max(), err_msg=k)


def test_noalloc_after_a_nan(lib):
    import torch
    from calcir_gb300._lib import load
    so = load()
    bad = _sym(600, 1)
    bad[0, 17, 400] = bad[0, 400, 17] = np.nan
    got = []
    for A in (_sym(514, 2), bad, _sym(514, 2)):
        dA = torch.from_numpy(A).cuda()
        w = torch.empty(A.shape[:2], device="cuda")
        torch.cuda.synchronize()
        rc = so.cir_eigh_noalloc(1, A.shape[1], C.c_void_p(dA.data_ptr()), C.c_void_p(w.data_ptr()), None)
        got.append((rc, w.cpu().numpy(), dA.cpu().numpy()))
    assert got[0][0] == got[2][0] == 0 and np.isfinite(got[0][1]).all()
    np.testing.assert_array_equal(got[0][1], got[2][1])
    np.testing.assert_array_equal(got[0][2], got[2][2])
