"""Writes gb_fr_shoup.cuh: the product of an Fr value by a prepared constant.

For a constant w < r kept with v = floor(w 2^256 / r), and any x < 2r (2r is
below 2^256), let q be the upper half of x v and z = x w - q r (Shoup's
modular product by an invariant; Harvey, "Faster arithmetic for
number-theoretic transforms", 2014).  Since x w - (x v / 2^256) r lies in
[0, x r / 2^256) and x / 2^256 < 0.91, z < 1.91 r + (the quotient's error) r:
the result stays in [0, 2r) as long as q is at most x v / 2^256 and more than
x v / 2^256 - 1.09.  So only the upper half of x v is formed: products of
limbs i + j >= 7 whole and the upper words of i + j = 6; what is left out is
below 14 * 2^224, i.e. 2^-28 units of q.  x w and q r are needed mod 2^256
only, and q r is taken as q (2^256 - r) with 2^256 - r = (2^32 - 1) + 0 * 2^32
+ ..., whose two lowest limbs cost additions.  In 32-bit products: 36 + 7
upper words for q, 28 + 8 lower words for x w, 15 + 6 lower words for
q (2^256 - r): 79 full products and 21 half ones, against 120 of the
Montgomery product, and no step depends on the previous one's low word.

Sums are kept in two rows, products at even word offsets in one and at odd
offsets in the other, so that a row of products is one carry chain.

    python gen_fr_shoup.py > gb_fr_shoup.cuh
"""
from gen_rows import chain, emit

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
NEG_R = [((1 << 256) - R) >> (32 * i) & 0xFFFFFFFF for i in range(8)]
assert NEG_R[0] == 0xFFFFFFFF and NEG_R[1] == 0


class Rows:
    """rows of products x[i] * y(j) added at word i + j of `acc`; words at or
    above `top` are dropped"""

    def __init__(self, acc, top):
        self.acc, self.top, self.live = acc, top, set()

    def word(self, w):
        return "%s[%d]" % (self.acc, w)

    def have(self, w):
        return self.word(w) if w in self.live else "#0"

    def row(self, x, i, y, js, upper_only=None):
        ins, carry = [], False

        def put(kind, w, j, keep_carry):
            nonlocal carry
            a, xi = self.have(w), "%s[%d]" % (x, i)
            if not carry and a == "#0":
                ins.append(("mul.%s.u32" % kind, self.word(w), xi, y(j)))
            else:
                op = ("madc" if carry else "mad") + "." + kind + (".cc" if keep_carry else "") + ".u32"
                ins.append((op, self.word(w), xi, y(j), a))
                carry = keep_carry
            self.live.add(w)

        words = []
        if upper_only is not None:
            words.append(("hi", i + upper_only + 1, upper_only))
        for j in js:
            words.append(("lo", i + j, j))
            if i + j + 1 < self.top:
                words.append(("hi", i + j + 1, j))
        for n, (kind, w, j) in enumerate(words):
            last = n + 1 == len(words)
            # an upper word added to an empty one cannot carry
            put(kind, w, j, not (w + 1 == self.top or (last and kind == "hi" and self.have(w) == "#0")))
        if carry:
            w = words[-1][1] + 1
            ins.append(("addc.u32", self.word(w), self.have(w), "#0"))
            self.live.add(w)
        return emit(ins) if ins else ""


def body():
    out = ""
    even, odd = Rows("a", 16), Rows("c", 16)
    v = lambda j: "v[%d]" % j  # noqa: E731
    for i in range(8):
        out += odd.row("x", i, v, [j for j in range(8) if i + j >= 7 and (i + j) % 2])
        out += even.row("x", i, v, [j for j in range(8) if i + j >= 8 and (i + j) % 2 == 0], 6 - i if i < 7 else None)
    q = ["q[%d]" % k for k in range(8)]
    out += chain("add", q, ["a[%d]" % (8 + k) for k in range(8)], ["c[%d]" % (8 + k) for k in range(8)],
                 [("add.cc.u32", "drop", "a[7]", "c[7]")])
    even, odd = Rows("b", 8), Rows("d", 8)
    w, m = lambda j: "w[%d]" % j, lambda j: "#0x%08x" % NEG_R[j]  # noqa: E731
    for x, y, j0 in (("x", w, 0), ("q", m, 2)):
        for i in range(8):
            out += even.row(x, i, y, [j for j in range(j0, 8) if i + j <= 7 and (i + j) % 2 == 0])
            out += odd.row(x, i, y, [j for j in range(j0, 8) if i + j <= 7 and (i + j) % 2])
    b = ["b[%d]" % k for k in range(8)]
    out += chain("add", b[1:], b[1:], ["d[%d]" % k for k in range(1, 8)])
    out += chain("add", b[1:], b[1:], q[:7])
    out += chain("sub", ["z[%d]" % k for k in range(8)], b, q)
    return out


if __name__ == "__main__":
    print("// Generated by gen_fr_shoup.py: do not edit.")
    print("// z = x w - q r, q = (upper half of x v) for x < 2r, w < r, v = floor(w 2^256 / r):")
    print("// z < 2r and z = x w mod r.")
    print("#pragma once")
    print("#include <stdint.h>")
    print("#if defined(__CUDA_ARCH__)")
    print("namespace gb {")
    print("__device__ __forceinline__ void fr_mul_prepared(uint32_t *z, const uint32_t *x, const uint32_t *w,\n"
          "                                                const uint32_t *v)\n{")
    print("    uint32_t a[16], c[16], b[8], d[8], q[8], drop;")
    print(body().rstrip("\n"))
    print("}\n}  // namespace gb")
    print("#endif")
