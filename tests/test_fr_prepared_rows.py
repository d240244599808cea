"""The generated rows of the Fr product by a prepared constant (csrc/
gb_fr_shoup.cuh), executed on Python integers statement by statement: for
x < 2r and a constant w < r the result is x w mod r and below 2r, at the ends
of both ranges and on random values."""
import os
import random
import re

import pytest

from conftest import PKG

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
M32 = 0xFFFFFFFF


@pytest.fixture(scope="module")
def statements():
    src = open(os.path.join(PKG, "csrc", "gb_fr_shoup.cuh")).read()
    out = []
    for text, outs, ins in re.findall(r'asm\((.*?)\n        : (.*?)\n        : (.*?)\);', src, re.S):
        ops = re.findall(r'\((.*?)\)', outs) + re.findall(r'\((.*?)\)', ins)
        lines = "".join(re.findall(r'"(.*?)"', text, re.S)).replace("\\n\\t", "").split(";")
        out.append((ops, [ln.strip() for ln in lines if ln.strip()]))
    return out


def run(statements, x, w, v):
    env = {"%s[%d]" % (n, k): (val >> (32 * k)) & M32 for n, val in (("x", x), ("w", w), ("v", v)) for k in range(8)}
    for ops, lines in statements:
        carry = None  # no carry crosses a statement
        for line in lines:
            op, rest = line.split(" ", 1)
            dst, *src = [o.strip() for o in rest.split(",")]
            a = [env[ops[int(o[1:])]] if o[0] == "%" else int(o, 0) for o in src]
            kind = op.split(".")
            cin = 0
            if kind[0] in ("madc", "addc", "subc"):
                cin = carry
                assert cin is not None
            if kind[0] in ("mul", "mad", "madc"):
                p = a[0] * a[1]
                t = (p & M32 if kind[1] == "lo" else p >> 32) + (a[2] if len(a) > 2 else 0) + cin
            elif kind[0] in ("add", "addc"):
                t = a[0] + a[1] + cin
            else:
                t = a[0] - a[1] - cin
            env[ops[int(dst[1:])]] = t & M32
            carry = (t >> 32) & 1 if "cc" in kind else None
    return sum(env["z[%d]" % k] << (32 * k) for k in range(8))


EDGES = [0, 1, 2, M32, 1 << 32, (1 << 224) - 1, (1 << 255) - 1, 1 << 255, R - 2, R - 1, R, R + 1, 2 * R - 1]


@pytest.mark.parametrize("w", [e for e in EDGES if e < R])
def test_edges(statements, w):
    for x in EDGES:
        z = run(statements, x, w, (w << 256) // R)
        assert z < 2 * R and (z - x * w) % R == 0


def test_random(statements):
    rng = random.Random(17)
    for _ in range(400):
        x, w = rng.randrange(2 * R), rng.randrange(R)
        z = run(statements, x, w, (w << 256) // R)
        assert z < 2 * R and (z - x * w) % R == 0
