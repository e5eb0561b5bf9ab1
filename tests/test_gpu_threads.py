"""Contexts of one process are independent: one per host thread, of any sizes, at the same time."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _together(jobs, seconds=120):
    """Runs the jobs in a thread each; what they raised."""
    raised = []

    def go(job):
        try:
            job()
        except Exception as x:      # reported by the test
            raised.append(repr(x))
    threads = [threading.Thread(target=go, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join(seconds)
    assert not any(t.is_alive() for t in threads)
    return raised


def test_builds_of_two_sizes_at_once(lib):
    """Small and large boxes built from two threads: each launch has the shared memory that its own size
    needs, whatever the other thread's last launch asked for."""
    import torch
    from calcir_gb300._lib import check, ptr
    data = []
    for nmol in (16, 1000):
        xyz = np.random.default_rng(nmol).uniform(0, 3.1, (1, 4 * nmol, 3)).astype(np.float32)
        n = 2 * nmol
        data.append((nmol, torch.from_numpy(xyz).cuda(), torch.full((1, 3), 3.1, device="cuda"),
                     torch.empty(1, n, n, device="cuda")))
    torch.cuda.synchronize()

    def job(nmol, xyz, box, H):
        def run():
            with lib.Engine(lib.default_params(model="tip4p2005", species="H2O"), 4 * nmol) as eng:
                for i in range(4000):
                    check(eng.lib.cir_build_hamiltonian(eng.h, 1, ptr(xyz), ptr(box), ptr(H), None, None, None))
                    if i % 200 == 0:
                        eng.synchronize()
                eng.synchronize()
        return run
    assert not _together([job(*d) for d in data])


def test_runs_of_many_sizes_at_once(lib):
    sizes = (16, 40, 64, 150)

    def job(nmol):
        xyz, box = lib.synth_trajectory(nmol, 3, seed=nmol)
        fos = np.arange(3, dtype=np.int32)
        bx = np.tile(np.asarray(box, np.float32), (3, 1))

        def run():
            p = lib.default_params(model="tip4p2005", species="H2O", ntcfpoints=3, nsamples=1, nzeros=200, avef=3415.0)
            with lib.Engine(p, 4 * nmol) as eng:
                ref = eng.run(xyz, bx, fos)
                for _ in range(60):
                    got = eng.run(xyz, bx, fos)
                    np.testing.assert_allclose(got["tcf_ir"], ref["tcf_ir"], rtol=1e-9)
        return run
    assert not _together([job(n) for n in sizes])
