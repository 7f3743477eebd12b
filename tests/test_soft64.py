"""Integer forms of the FP64 operations (csrc/soft64.cuh) against the host's IEEE arithmetic:
the header compiled for the host, seeded operands over the exponent range with ties, carries
and operands that the functions must leave to the hardware; every handled result bit for bit."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ceda_demonstrations_gb300", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    out = str(tmp_path_factory.mktemp("soft64") / "soft64_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fsanitize=undefined", "-fno-sanitize-recover",
                    "-I" + CSRC, os.path.join(HERE, "native", "soft64_check.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_integer_forms_are_correctly_rounded(program, seed):
    n = 3000000
    r = subprocess.run([program, str(n), str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    handled = [int(v) for v in r.stdout.split("handled")[1].split("wrong")[0].split()]
    # additions: same signs (a half), near exponents (21 of 27); products and small addends: most
    assert handled[0] > 0.25 * n and handled[1] > 0.7 * n and handled[2] > 0.5 * n, handled
