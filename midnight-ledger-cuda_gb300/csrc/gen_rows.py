"""Inline-PTX statements for the generated field products: a carry chain is
one asm statement, so no carry crosses a statement."""


def emit(ins):
    """one asm statement for the (opcode, destination, sources...) list;
    operands are C lvalues, '#...' immediates"""
    outs, ins_only, read_first, written = [], [], set(), set()
    for _, d, *_ in ins:
        if d not in outs:
            outs.append(d)
    for _, d, *src in ins:
        for o in src:
            if o[0] == "#":
                continue
            if o in outs:
                if o not in written:
                    read_first.add(o)
            elif o not in ins_only:
                ins_only.append(o)
        written.add(d)
    num = {o: "%%%d" % i for i, o in enumerate(outs + ins_only)}
    text = "\\n\\t\"\n        \"".join(
        op + " " + ", ".join(o[1:] if o[0] == "#" else num[o] for o in ops) + ";" for op, *ops in ins)
    res = ", ".join('"%s"(%s)' % ("+r" if o in read_first else "=&r", o) for o in outs)
    arg = ", ".join('"r"(%s)' % o for o in ins_only)
    return '    asm("%s"\n        : %s\n        : %s);\n' % (text, res, arg)


def chain(op, dst, a, b, head=()):
    n = len(dst)
    return emit(list(head) + [(op + ("" if k == 0 and not head else "c") + (".u32" if k == n - 1 else ".cc.u32"),
                               dst[k], a[k], b[k]) for k in range(n)])
