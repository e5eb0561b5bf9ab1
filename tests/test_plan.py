"""The batched runners' host-side planning (calcir_gb300/csrc/cir_plan.h), compiled on its own
with the host compiler: chunk lengths against the tridiagonalisation's waves, and the first
part of a chunk's eigensolver batch when it is split over two streams."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
HEADER_DIR = os.path.join(os.path.dirname(HERE), "calcir_gb300", "csrc")

DRIVER = r"""
#include <cstdio>
#include "cir_plan.h"
int main() {
    int K, St, kn, wave, nmat;
    while (std::scanf("%d %d %d %d %d", &K, &St, &kn, &wave, &nmat) == 5)
        std::printf("%d %d\n", cir_plan_chunk(K, St, kn, wave), cir_split_first_part(nmat, wave));
    return 0;
}
"""


@pytest.fixture(scope="module")
def planner():
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    d = tempfile.mkdtemp(prefix="cir_plan_")
    src, exe = os.path.join(d, "plan.cpp"), os.path.join(d, "plan")
    with open(src, "w") as f:
        f.write(DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", HEADER_DIR, src, "-o", exe], check=True)

    def run(cases):
        inp = "".join(f"{K} {St} {kn} {w} {nm}\n" for K, St, kn, w, nm in cases)
        out = subprocess.run([exe], input=inp, capture_output=True, text=True, check=True).stdout.split()
        return [(int(out[2 * i]), int(out[2 * i + 1])) for i in range(len(cases))]
    yield run
    shutil.rmtree(d, ignore_errors=True)


def test_chunks_avoid_nearly_empty_last_waves(planner):
    (kn_a, _), (kn_b, _), (kn_c, _), (kn_d, _) = planner([
        (200, 32, 101, 456, 0),   # order 1024, 32 origins, memory for 101 steps: 101 + 99 (6400 = 7.09 + 6.95 waves)
        (200, 32, 100, 456, 0),   # 100 + 100 would leave two nearly empty waves: the planner still has 2 chunks
        (250, 10, 250, 456, 0),   # the headline job fits in one chunk
        (200, 32, 40, 456, 0),    # five chunks of 40 steps (1280 = 2.81 waves each)
    ])
    assert kn_a == 101
    assert kn_b == 100
    assert kn_c == 250
    assert kn_d == 40


def test_chunk_length_bounds(planner):
    res = planner([(K, St, km, w, 0) for K, St, km, w in [(7, 3, 1, 456, ), (7, 3, 100, 456), (1, 1, 5, 1), (50, 1000, 3, 456)]])
    assert res[0][0] == 1            # kn_max = 1
    assert res[1][0] == 7            # never more than K
    assert res[2][0] == 1
    assert 1 <= res[3][0] <= 3


def test_split_first_part_is_whole_waves_but_the_last(planner):
    res = planner([(1, 1, 1, 456, 2500), (1, 1, 1, 456, 911), (1, 1, 1, 456, 912), (1, 1, 1, 304, 1250)])
    assert res[0][1] == 1824         # 5 whole waves of 456 in 2500: the first 4 on one stream
    assert res[1][1] == 0            # fewer than two waves: one stream
    assert res[2][1] == 456
    assert res[3][1] == 912          # order 2048, two blocks per SM


FORM_DRIVER = r"""
#include <cstdio>
#include "cir_plan.h"
int main() {
    int n, nmat, tuned;
    while (std::scanf("%d %d %d", &n, &nmat, &tuned) == 3)
        std::printf("%d %d\n", (int)cir_tridiag_form(n, nmat, 152), cir_tridiag_limit(tuned, nmat, 152));
    return 0;
}
"""


def test_tridiagonalisation_form(tmp_path):
    """The kernel follows from the order and the number of matrices; what the autotuner found for an
    order limits the blocks per SM of batches of the size it measured, and of no smaller ones."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src, exe = str(tmp_path / "form.cpp"), str(tmp_path / "form")
    with open(src, "w") as f:
        f.write(FORM_DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", HEADER_DIR, src, "-o", exe], check=True)

    def run(cases):
        inp = "".join("%d %d %d\n" % c for c in cases)
        out = subprocess.run([exe], input=inp, capture_output=True, text=True, check=True).stdout.split()
        return [(int(out[2 * i]), int(out[2 * i + 1])) for i in range(len(cases))]
    forms = [((3, 1), 1), ((128, 304), 1), ((128, 305), 0), ((129, 305), 1), ((192, 1000), 1), ((193, 152), 1),
             ((193, 153), 2), ((256, 152), 1), ((257, 152), 3), ((257, 153), 2), ((512, 153), 2), ((512, 152), 3),
             ((513, 1000), 3), ((2048, 1), 3)]
    for tuned in (0, 1, 3):
        for ((n, nmat), form), (got, limit) in zip(forms, run([(n, nmat, tuned) for (n, nmat), _ in forms])):
            assert got == form, (n, nmat, tuned)
            assert limit == (tuned if nmat > 304 else 0)


WIDE_DRIVER = r"""
#include <cstdio>
#include "cir_plan.h"
int main() {
    int nmol, nf;
    while (std::scanf("%d %d", &nmol, &nf) == 2) std::printf("%d\n", cir_build_wide(2 * nmol, nmol, nf, 152) ? 1 : 0);
    return 0;
}
"""


def test_build_form(tmp_path):
    """A warp or a thread per chromophore: the form that measured at least 15% faster (GB300), over box
    sizes and batches, large boxes of few frames among them."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src, exe = str(tmp_path / "wide.cpp"), str(tmp_path / "wide")
    with open(src, "w") as f:
        f.write(WIDE_DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", HEADER_DIR, src, "-o", exe], check=True)
    wide = [(1, 1), (5, 100), (12, 200), (24, 1), (24, 100), (40, 100), (64, 1), (64, 30), (100, 30), (150, 30), (250, 10),
            (343, 1), (343, 10), (512, 4), (700, 1), (700, 4), (1000, 1), (1000, 2)]
    narrow = [(2, 3000), (5, 1000), (12, 1000), (24, 500), (40, 500), (64, 200), (100, 100), (150, 100), (250, 100),
              (343, 30), (343, 200), (512, 30), (700, 10), (1000, 4), (1000, 30)]
    cases = wide + narrow
    out = subprocess.run([exe], input="".join("%d %d\n" % c for c in cases), capture_output=True, text=True,
                         check=True).stdout.split()
    assert [int(x) for x in out] == [1] * len(wide) + [0] * len(narrow)


GEMM_DRIVER = r"""
#include <cstdio>
#include "cir_plan.h"
int main() {
    int M, N, K, b, e, a;
    while (std::scanf("%d %d %d %d %d %d", &M, &N, &K, &b, &e, &a) == 6)
        std::printf("%d\n", (int)cir_gemm_form(M, N, K, b, e, (a & 1) != 0, (a & 2) != 0, 152));
    return 0;
}
"""


def test_product_form(tmp_path):
    """The FP32 product's kernel: the one that measured fastest by 10% or more (GB300), or either of two
    that are level."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src, exe = str(tmp_path / "gemm.cpp"), str(tmp_path / "gemm")
    with open(src, "w") as f:
        f.write(GEMM_DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", HEADER_DIR, src, "-o", exe], check=True)
    small, t64, t128, tc = 0, 1, 2, 3
    # the last number: 3: rows of operands and output start on 16 bytes, 2: the output's alone, 0: neither
    cases = [((128, 256, 128, 1, 1, 3), {small}), ((200, 400, 200, 1, 1, 3), {small}), ((64, 128, 64, 16, 1, 3), {small, t64}),
             ((33, 66, 33, 300, 1, 0), {t64}), ((50, 100, 50, 300, 1, 3), {t64}), ((56, 112, 56, 600, 0, 3), {t64}),
             ((65, 130, 65, 300, 1, 0), {t128, t64}), ((66, 132, 66, 152, 0, 3), {t128, t64}), ((97, 194, 97, 150, 1, 0), {t128}),
             ((128, 256, 128, 300, 1, 3), {tc}), ((256, 512, 256, 16, 1, 3), {tc}), ((1024, 2048, 1024, 1, 1, 3), {tc}),
             ((1024, 2048, 1024, 200, 0, 3), {tc}), ((686, 686, 128, 64, 2, 0), {t64, t128}), ((1024, 1024, 128, 64, 2, 3), {tc}),
             ((432, 432, 128, 64, 2, 3), {tc}), ((343, 686, 128, 16, 2, 0), {t64, t128})]
    inp = "".join("%d %d %d %d %d %d\n" % c for c, _ in cases)
    out = subprocess.run([exe], input=inp, capture_output=True, text=True, check=True).stdout.split()
    for (c, forms), got in zip(cases, out):
        assert int(got) in forms, (c, got)
