"""The warp's inversion by division steps (csrc/gb_inv_warp.cuh) on the CPU,
the lanes taking turns: the steps alone, without the check and the way out
behind them, give the inverse in both fields, and no signed value overflows (the
program stops at one)."""
import os
import random
import subprocess

import pytest

from conftest import PKG, REPO

FIELDS = {
    "fp": (0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB, 384),
    "fr": (0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001, 256),
}


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("inv") / "inv_warp")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fsanitize=signed-integer-overflow,shift",
                           "-fno-sanitize-recover=all", "-I", os.path.join(PKG, "csrc"), "-o", exe,
                           os.path.join(REPO, "tests", "inv_warp_harness.cpp")])
    return exe


@pytest.mark.parametrize("field", FIELDS)
def test_division_steps(program, field):
    m, bits = FIELDS[field]
    rng = random.Random(field)
    R = 1 << bits
    values = [1, 2, 3, m - 1, m - 2, (m + 1) // 2, R % m, R * R % m, 1 << 30, (1 << 30) - 1, 1 << 31, (1 << 60) + 1,
              m >> 1, m - (1 << 30), (1 << (m.bit_length() - 1)) - 1, 1 << (m.bit_length() - 1)]
    values += [rng.randrange(1, m) for _ in range(12)]
    text = "".join("%s %0*x\n" % (field, bits // 4, v) for v in values)
    out = subprocess.run([program], input=text, capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-500:]
    # Montgomery form in and out: a = x R, result = x^-1 R
    assert [int(w, 16) for w in out.stdout.split()] == [R * R * pow(v, -1, m) % m for v in values]
