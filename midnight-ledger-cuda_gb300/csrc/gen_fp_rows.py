"""Writes gb_fp_rows.cuh: the Fp Montgomery product and squaring as rows of
32-bit multiply-adds, each row one carry chain.

A running value V is held as two rows of words, V = E + 2^32 O: products of
even-indexed multiplicand words go to E, of odd-indexed ones to O, so a row of
six products fills twelve words without overlap.  A step adds a b_i, then m p
with m = -E_0 / p mod 2^32, which clears E_0, and divides by 2^32.  The
division moves no words: E / 2^32 = E_1 + 2^32 (E_2, E_3, ...), so the next
step's E is O with E_1 added at its lowest word, its O is E from word 2 on,
and the carry of that one addition enters the next O row's chain as its
carry-in.  (Adding E / 2^32 to O instead costs 13 carry additions a step, each
2 cycles a warp beside 4 for a 32 x 32 product.)

Bounds, for a, b < p < 2^381: V < 2p after a step, so O < 2^350; before the
division V < 2^414, so E fits 13 words and O 12.

The squaring forms a^2 first (66 cross products, doubled, and 12 squares) and
then reduces its lower half by the same steps without the a b_i rows, adding
the upper half at the end.

    python gen_fp_rows.py > gb_fp_rows.cuh
"""
from gen_rows import chain, emit

P = 0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB
N = 12
PW = ["#0x%08x" % ((P >> (32 * i)) & 0xFFFFFFFF) for i in range(N)]
INV = (-pow(P, -1, 1 << 32)) % (1 << 32)


def words(name, n):
    return ["%s[%d]" % (name, i) for i in range(n)]


def row(dst, x, y, add, head=(), top=None):
    """dst = add + x * y over the words of the six x's: one chain; `head` goes
    before it and leaves its carry-in; `top` takes the carry out as (dst, add)"""
    ins = list(head)
    for k in range(N // 2):
        last = k == N // 2 - 1 and top is None
        ins.append((("madc" if ins else "mad") + ".lo.cc.u32", dst[2 * k], x[k], y, add[2 * k]))
        ins.append(("madc.hi" + (".u32" if last else ".cc.u32"), dst[2 * k + 1], x[k], y, add[2 * k + 1]))
    if top is not None:
        ins.append(("addc.u32", top[0], top[1], "#0"))
    return emit(ins)


def products(dst, x, y):
    return "".join("    %s = %s * %s;\n    %s = __umulhi(%s, %s);\n" % (dst[2 * k], x[k], y, dst[2 * k + 1], x[k], y)
                   for k in range(N // 2))


def shifted(O, E):
    """the words that follow a division by 2^32: (E's, less E_1 at word 0; O's)"""
    return O, E[2:N + 1] + ["#0"]


def finish(E, O, extra):
    out = chain("add", words("r", N), O, E[1:])
    if extra:
        out += chain("add", words("r", N), words("r", N), extra)
    t = words("t", N)
    ins = [(("sub" if k == 0 else "subc") + ".cc.u32", t[k], "r[%d]" % k, PW[k]) for k in range(N)]
    out += emit(ins + [("subc.u32", "br", "#0", "#0")])
    return out + "#pragma unroll\n    for (int k = 0; k < 12; k++) r[k] = br ? r[k] : t[k];\n"


def mul():
    a = words("a", N)
    E, O, F, G = words("e", N + 1), words("o", N), words("f", N + 1), words("g", N)
    out = ("GB_D void fp_mul_rows(uint32_t *r, const uint32_t *a, const uint32_t *b)\n{\n"
           "    uint32_t e[13], o[12], f[13], g[12], t[12], m, br;\n")
    for i in range(N):
        b = "b[%d]" % i
        if i == 0:
            out += products(E, a[0::2], b) + products(O, a[1::2], b) + "    e[12] = 0;\n"
        else:
            e_add, o_add = shifted(O, E)
            out += row(G, a[1::2], b, o_add, head=[("add.cc.u32", F[0], O[0], E[1])])
            out += row(F, a[0::2], b, [F[0]] + e_add[1:], top=(F[N], "#0"))
            E, F, O, G = F, E, G, O
        out += "    m = %s * 0x%08xu;\n" % (E[0], INV)
        out += row(E, PW[0::2], "m", E, top=(E[N], E[N])) + row(O, PW[1::2], "m", O)
    return out + finish(E, O, None) + "}\n"


def sqr():
    a, t, h = words("a", N), words("s", 2 * N), words("h", 2 * N)
    out = ("GB_D void fp_sqr_rows(uint32_t *r, const uint32_t *a)\n{\n"
           "    uint32_t s[24], h[24], e[13], o[12], f[13], g[12], t[12], m, c, br;\n")
    live = {0: set(), 1: set()}
    for i in range(N - 1):  # cross products a_i a_j, j > i: even offsets in s, odd ones in h
        for par, acc in ((1, h), (0, t)):
            js, f = [j for j in range(i + 1, N) if (i + j) % 2 == par], live[par]
            ins, carry = [], False
            for j in js:
                w = i + j
                if w not in f and not carry:
                    ins += [("mul.lo.u32", acc[w], a[i], a[j]), ("mul.hi.u32", acc[w + 1], a[i], a[j])]
                else:
                    ins.append((("madc" if carry else "mad") + ".lo.cc.u32", acc[w], a[i], a[j],
                                acc[w] if w in f else "#0"))
                    carry = not (j == js[-1] and w + 1 not in f)  # an upper word added to nothing cannot carry
                    ins.append(("madc.hi" + (".cc" if carry else "") + ".u32", acc[w + 1], a[i], a[j],
                                acc[w + 1] if w + 1 in f else "#0"))
                f |= {w, w + 1}
            if carry:
                w = i + js[-1] + 2
                ins.append(("addc.u32", acc[w], acc[w] if w in f else "#0", "#0"))
                f.add(w)
            if ins:
                out += emit(ins)
    pick = lambda acc, par, k: acc[k] if k in live[par] else "#0"  # noqa: E731
    out += chain("add", t[1:23], [pick(t, 0, k) for k in range(1, 23)], [pick(h, 1, k) for k in range(1, 23)])
    out += ("    s[23] = s[22] >> 31;\n#pragma unroll\n"
            "    for (int k = 22; k > 1; k--) s[k] = __funnelshift_l(s[k - 1], s[k], 1);\n    s[1] <<= 1;\n")
    ins = [("mul.lo.u32", t[0], a[0], a[0]), ("mad.hi.cc.u32", t[1], a[0], a[0], t[1])]
    for i in range(1, N):
        ins.append(("madc.lo.cc.u32", t[2 * i], a[i], a[i], t[2 * i]))
        ins.append(("madc.hi" + ("" if i == N - 1 else ".cc") + ".u32", t[2 * i + 1], a[i], a[i], t[2 * i + 1]))
    out += emit(ins)
    E, O, F, G = words("e", N + 1), words("o", N), words("f", N + 1), words("g", N)
    for i in range(N):
        if i == 0:
            out += "    m = s[0] * 0x%08xu;\n" % INV
            out += row(E, PW[0::2], "m", t[:N], top=(E[N], "#0")) + products(O, [w[1:] + "u" for w in PW[1::2]], "m")
            continue
        e_add, o_add = shifted(O, E)
        out += emit([("add.cc.u32", F[0], O[0], E[1]), ("addc.u32", "c", "#0", "#0")])
        out += "    m = %s * 0x%08xu;\n" % (F[0], INV)
        # c + 2^32 - 1 carries exactly when c = 1
        out += row(G, PW[1::2], "m", o_add, head=[("add.cc.u32", "c", "c", "#0xffffffff")])
        out += row(F, PW[0::2], "m", [F[0]] + e_add[1:], top=(F[N], "#0"))
        E, F, O, G = F, E, G, O
    return out + finish(E, O, t[N:]) + "}\n"


if __name__ == "__main__":
    print("// Generated by gen_fp_rows.py: do not edit.")
    print("// r = a b / 2^384 mod p and r = a^2 / 2^384 mod p, fully reduced, for a, b < p.")
    print("#pragma once")
    print("#include <stdint.h>")
    print("#if defined(__CUDA_ARCH__)")
    print("namespace gb {")
    print(mul())
    print(sqr().rstrip("\n"))
    print("}  // namespace gb")
    print("#endif")
