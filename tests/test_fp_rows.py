"""The generated rows of the Fp product and squaring (csrc/gb_fp_rows.cuh),
executed on Python integers statement by statement: a b / 2^384 mod p, fully
reduced, at the ends of the range and on random values."""
import os
import random
import re

import pytest

from conftest import PKG

P = 0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB
M32 = 0xFFFFFFFF
R_INV = pow(1 << 384, -1, P)


def compiled(name):
    """The function's statements as one Python function of the words a and b."""
    src = open(os.path.join(PKG, "csrc", "gb_fp_rows.cuh")).read()
    body = re.search(r"GB_D void %s\(.*?\n\{(.*?)\n\}" % name, src, re.S).group(1)
    py = ["def f(a, b):", " s, h, e, o, f, g, t, r = ([0] * 24 for _ in range(8))", " m = c = br = cc = 0"]
    body = body.replace("#pragma unroll\n", "")
    for text in re.findall(r"\s*(asm\(.*?\);|for \(.*?\) [^;]+;|[^\s;][^;]*;)", body, re.S):
        text = text.strip()
        if text.startswith("uint32_t"):
            continue
        if not text.startswith("asm"):
            loop = re.match(r"for \(int k = (\d+); k ([<>]) (\d+); k(\+\+|--)\) (.*)", text, re.S)
            if loop:
                lo, _, hi, step, text = loop.groups()
                py.append(" for k in range(%s, %s, %d):" % (lo, hi, 1 if step == "++" else -1))
            text = re.sub(r"(0x[0-9a-f]+)u\b", r"\1", text.rstrip(";"))
            text = re.sub(r"__umulhi\((.*?), (.*?)\)", r"(\1 * \2 >> 32)", text)
            text = re.sub(r"__funnelshift_l\((.*?), (.*?), (\d+)\)", r"((\2 << 32 | \1) << \3 >> 32)", text)
            text = re.sub(r"= br \? (.*?) : (.*)", r"= \1 if br else \2", text)
            text = re.sub(r"(.*?) <<= (\d+)", r"\1 = \1 << \2", text)
            dst, val = text.split(" = ", 1)
            py.append((" " if loop else "") + " %s = (%s) & %d" % (dst, val, M32))
            continue
        ops = re.findall(r'"\+?=?&?r"\((.*?)\)', text)
        py.append(" cc = None")  # no carry crosses a statement
        for line in "".join(re.findall(r'"([a-z][^"]*?(?:;|;\\n\\t))"', text)).replace("\\n\\t", "").split(";"):
            if not line.strip():
                continue
            op, rest = line.strip().split(" ", 1)
            dst, *x = [ops[int(v[1:])] if v[0] == "%" else v for v in (w.strip() for w in rest.split(","))]
            kind = op.split(".")
            sign = "-" if kind[0].startswith("sub") else "+"
            if kind[0] in ("mul", "mad", "madc"):
                val = "(%s * %s %s)" % (x[0], x[1], "& %d" % M32 if kind[1] == "lo" else ">> 32")
                val += " + " + x[2] if len(x) > 2 else ""
            else:
                val = "%s %s %s" % (x[0], sign, x[1])
            if kind[0] in ("madc", "addc", "subc"):
                val += " %s cc" % sign
            py.append(" z = " + val)
            py.append(" %s = z & %d" % (dst, M32))
            py.append(" cc = z >> 32 & 1" if "cc" in kind else " cc = None")
    py.append(" return r")
    env = {}
    exec("\n".join(py), env)
    return env["f"]


@pytest.fixture(scope="module")
def rows():
    return compiled("fp_mul_rows"), compiled("fp_sqr_rows")


def words(v):
    return [(v >> (32 * k)) & M32 for k in range(12)]


def value(r):
    return sum(w << (32 * k) for k, w in enumerate(r[:12]))


EDGES = [0, 1, 2, M32, 1 << 32, (1 << 352) - 1, 1 << 380, (1 << 384) % P, P // 2, P - 2, P - 1]


@pytest.mark.parametrize("a", EDGES)
def test_edges(rows, a):
    mul, sqr = rows
    assert value(sqr(words(a), None)) == a * a * R_INV % P
    for b in EDGES:
        assert value(mul(words(a), words(b))) == a * b * R_INV % P


def test_random(rows):
    mul, sqr = rows
    rng = random.Random(23)
    for _ in range(300):
        a, b = rng.randrange(P), rng.randrange(P)
        assert value(mul(words(a), words(b))) == a * b * R_INV % P
        assert value(sqr(words(a), None)) == a * a * R_INV % P
