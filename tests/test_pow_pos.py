"""The power of the double steps (pow_pos.cuh), compiled for the host: its accuracy, the arguments it leaves to pow(),
and its table, recomputed from what its rows are defined as."""
import os
import subprocess
from decimal import Decimal, getcontext

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pow") / "pow_pos")
    subprocess.run(["g++", "-std=gnu++17", "-O2", "-mfma", "-ffp-contract=off", os.path.join(ROOT, "tests", "cpp", "pow_pos.cpp"),
                    "-I", os.path.join(ROOT, "tests", "cpp", "host_cuda"), "-I", os.path.join(ROOT, "umappp_b200", "csrc"),
                    "-lquadmath", "-o", exe], check=True)
    return exe


def out(program, *args):
    r = subprocess.run([program, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    return r.stdout


@pytest.mark.parametrize("seed", [1, 2])
def test_error_is_at_most_that_stated(program, seed):
    assert float(out(program, "errors", str(seed), "400000")) <= 1.01


def test_ends_of_the_range(program):
    out(program, "ends")


def test_table(program):
    getcontext().prec = 60
    log2 = Decimal(2).ln()
    rows = [[Decimal(float.fromhex(x)) for x in line.split()] for line in out(program, "table").split("\n") if line]
    assert len(rows) == 64
    for i, (inv, hi, lo, e2) in enumerate(rows):
        middle = 1 + (Decimal(i) + Decimal("0.5")) / 64
        assert abs(inv * middle - 1) <= Decimal(2) ** -11                 # 1 / c, rounded
        assert (inv * 2 ** 12) % 1 == 0                                   # to 12 bits: the product with a mantissa is short
        for edge in (Decimal(i) / 64, Decimal(i + 1) / 64):
            assert abs((1 + edge) * inv - 1) <= Decimal(2) ** -7          # the polynomial's range
        assert (hi * 2 ** 40) % 1 == 0                                    # k + hi is exact
        want = -inv.ln() / log2
        assert abs(hi - want) <= Decimal(2) ** -41 and abs(hi + lo - want) <= Decimal(2) ** -94
        want = (Decimal(i) / 64 * log2).exp()
        assert abs(e2 - want) <= Decimal(2) ** -53                        # correctly rounded in [1, 2)
