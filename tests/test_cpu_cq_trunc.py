"""The client quantizer's float form of the kernels (a fused multiply-add
rounded toward zero, then a truncating conversion, with no test for small
words) equals the oracle's integer restatement of d_CQ_IABS_4 on every lossy
word: a stride-7 sweep of the 2^32 words for two exponents, a stride-97 sweep
for the extremes."""
import os
import subprocess

import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "cq_trunc_check.c")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    from oracle import oracle as O
    lib = O.build()
    exe = str(tmp_path_factory.mktemp("cq") / "cq_trunc_check")
    subprocess.check_call(["gcc", "-O2", "-fopenmp", "-frounding-math", "-ffp-contract=off", "-o", exe, SRC, "-lm",
                           "-L", os.path.dirname(lib), "-lcortado_oracle", "-Wl,-rpath," + os.path.dirname(lib)])
    return exe


@pytest.mark.parametrize("eb_e,stride", [(100, 7), (133, 7), (1, 97), (2, 97), (50, 97), (200, 97), (229, 97),
                                         (230, 97)])
def test_truncating_form_matches_oracle(checker, eb_e, stride):
    r = subprocess.run([checker, str(eb_e), str(stride)], capture_output=True, text=True, timeout=900)
    checked, bad = (int(v) for v in r.stdout.split())
    assert checked > 0
    assert bad == 0 and r.returncode == 0
