// Generated by gen_fp_rows.py: do not edit.
// r = a b / 2^384 mod p and r = a^2 / 2^384 mod p, fully reduced, for a, b < p.
#pragma once
#include <stdint.h>
#if defined(__CUDA_ARCH__)
namespace gb {
GB_D void fp_mul_rows(uint32_t *r, const uint32_t *a, const uint32_t *b)
{
    uint32_t e[13], o[12], f[13], g[12], t[12], m, br;
    e[0] = a[0] * b[0];
    e[1] = __umulhi(a[0], b[0]);
    e[2] = a[2] * b[0];
    e[3] = __umulhi(a[2], b[0]);
    e[4] = a[4] * b[0];
    e[5] = __umulhi(a[4], b[0]);
    e[6] = a[6] * b[0];
    e[7] = __umulhi(a[6], b[0]);
    e[8] = a[8] * b[0];
    e[9] = __umulhi(a[8], b[0]);
    e[10] = a[10] * b[0];
    e[11] = __umulhi(a[10], b[0]);
    o[0] = a[1] * b[0];
    o[1] = __umulhi(a[1], b[0]);
    o[2] = a[3] * b[0];
    o[3] = __umulhi(a[3], b[0]);
    o[4] = a[5] * b[0];
    o[5] = __umulhi(a[5], b[0]);
    o[6] = a[7] * b[0];
    o[7] = __umulhi(a[7], b[0]);
    o[8] = a[9] * b[0];
    o[9] = __umulhi(a[9], b[0]);
    o[10] = a[11] * b[0];
    o[11] = __umulhi(a[11], b[0]);
    e[12] = 0;
    m = e[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(f[0]), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(o[0]), "r"(e[1]), "r"(a[1]), "r"(b[1]), "r"(e[2]), "r"(e[3]), "r"(a[3]), "r"(e[4]), "r"(e[5]), "r"(a[5]), "r"(e[6]), "r"(e[7]), "r"(a[7]), "r"(e[8]), "r"(e[9]), "r"(a[9]), "r"(e[10]), "r"(e[11]), "r"(a[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(a[0]), "r"(b[1]), "r"(o[1]), "r"(a[2]), "r"(o[2]), "r"(o[3]), "r"(a[4]), "r"(o[4]), "r"(o[5]), "r"(a[6]), "r"(o[6]), "r"(o[7]), "r"(a[8]), "r"(o[8]), "r"(o[9]), "r"(a[10]), "r"(o[10]), "r"(o[11]));
    m = f[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(f[0]), "+r"(f[1]), "+r"(f[2]), "+r"(f[3]), "+r"(f[4]), "+r"(f[5]), "+r"(f[6]), "+r"(f[7]), "+r"(f[8]), "+r"(f[9]), "+r"(f[10]), "+r"(f[11]), "+r"(f[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(g[0]), "+r"(g[1]), "+r"(g[2]), "+r"(g[3]), "+r"(g[4]), "+r"(g[5]), "+r"(g[6]), "+r"(g[7]), "+r"(g[8]), "+r"(g[9]), "+r"(g[10]), "+r"(g[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(e[0]), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(g[0]), "r"(f[1]), "r"(a[1]), "r"(b[2]), "r"(f[2]), "r"(f[3]), "r"(a[3]), "r"(f[4]), "r"(f[5]), "r"(a[5]), "r"(f[6]), "r"(f[7]), "r"(a[7]), "r"(f[8]), "r"(f[9]), "r"(a[9]), "r"(f[10]), "r"(f[11]), "r"(a[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(a[0]), "r"(b[2]), "r"(g[1]), "r"(a[2]), "r"(g[2]), "r"(g[3]), "r"(a[4]), "r"(g[4]), "r"(g[5]), "r"(a[6]), "r"(g[6]), "r"(g[7]), "r"(a[8]), "r"(g[8]), "r"(g[9]), "r"(a[10]), "r"(g[10]), "r"(g[11]));
    m = e[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(f[0]), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(o[0]), "r"(e[1]), "r"(a[1]), "r"(b[3]), "r"(e[2]), "r"(e[3]), "r"(a[3]), "r"(e[4]), "r"(e[5]), "r"(a[5]), "r"(e[6]), "r"(e[7]), "r"(a[7]), "r"(e[8]), "r"(e[9]), "r"(a[9]), "r"(e[10]), "r"(e[11]), "r"(a[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(a[0]), "r"(b[3]), "r"(o[1]), "r"(a[2]), "r"(o[2]), "r"(o[3]), "r"(a[4]), "r"(o[4]), "r"(o[5]), "r"(a[6]), "r"(o[6]), "r"(o[7]), "r"(a[8]), "r"(o[8]), "r"(o[9]), "r"(a[10]), "r"(o[10]), "r"(o[11]));
    m = f[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(f[0]), "+r"(f[1]), "+r"(f[2]), "+r"(f[3]), "+r"(f[4]), "+r"(f[5]), "+r"(f[6]), "+r"(f[7]), "+r"(f[8]), "+r"(f[9]), "+r"(f[10]), "+r"(f[11]), "+r"(f[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(g[0]), "+r"(g[1]), "+r"(g[2]), "+r"(g[3]), "+r"(g[4]), "+r"(g[5]), "+r"(g[6]), "+r"(g[7]), "+r"(g[8]), "+r"(g[9]), "+r"(g[10]), "+r"(g[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(e[0]), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(g[0]), "r"(f[1]), "r"(a[1]), "r"(b[4]), "r"(f[2]), "r"(f[3]), "r"(a[3]), "r"(f[4]), "r"(f[5]), "r"(a[5]), "r"(f[6]), "r"(f[7]), "r"(a[7]), "r"(f[8]), "r"(f[9]), "r"(a[9]), "r"(f[10]), "r"(f[11]), "r"(a[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(a[0]), "r"(b[4]), "r"(g[1]), "r"(a[2]), "r"(g[2]), "r"(g[3]), "r"(a[4]), "r"(g[4]), "r"(g[5]), "r"(a[6]), "r"(g[6]), "r"(g[7]), "r"(a[8]), "r"(g[8]), "r"(g[9]), "r"(a[10]), "r"(g[10]), "r"(g[11]));
    m = e[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(f[0]), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(o[0]), "r"(e[1]), "r"(a[1]), "r"(b[5]), "r"(e[2]), "r"(e[3]), "r"(a[3]), "r"(e[4]), "r"(e[5]), "r"(a[5]), "r"(e[6]), "r"(e[7]), "r"(a[7]), "r"(e[8]), "r"(e[9]), "r"(a[9]), "r"(e[10]), "r"(e[11]), "r"(a[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(a[0]), "r"(b[5]), "r"(o[1]), "r"(a[2]), "r"(o[2]), "r"(o[3]), "r"(a[4]), "r"(o[4]), "r"(o[5]), "r"(a[6]), "r"(o[6]), "r"(o[7]), "r"(a[8]), "r"(o[8]), "r"(o[9]), "r"(a[10]), "r"(o[10]), "r"(o[11]));
    m = f[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(f[0]), "+r"(f[1]), "+r"(f[2]), "+r"(f[3]), "+r"(f[4]), "+r"(f[5]), "+r"(f[6]), "+r"(f[7]), "+r"(f[8]), "+r"(f[9]), "+r"(f[10]), "+r"(f[11]), "+r"(f[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(g[0]), "+r"(g[1]), "+r"(g[2]), "+r"(g[3]), "+r"(g[4]), "+r"(g[5]), "+r"(g[6]), "+r"(g[7]), "+r"(g[8]), "+r"(g[9]), "+r"(g[10]), "+r"(g[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(e[0]), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(g[0]), "r"(f[1]), "r"(a[1]), "r"(b[6]), "r"(f[2]), "r"(f[3]), "r"(a[3]), "r"(f[4]), "r"(f[5]), "r"(a[5]), "r"(f[6]), "r"(f[7]), "r"(a[7]), "r"(f[8]), "r"(f[9]), "r"(a[9]), "r"(f[10]), "r"(f[11]), "r"(a[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(a[0]), "r"(b[6]), "r"(g[1]), "r"(a[2]), "r"(g[2]), "r"(g[3]), "r"(a[4]), "r"(g[4]), "r"(g[5]), "r"(a[6]), "r"(g[6]), "r"(g[7]), "r"(a[8]), "r"(g[8]), "r"(g[9]), "r"(a[10]), "r"(g[10]), "r"(g[11]));
    m = e[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(f[0]), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(o[0]), "r"(e[1]), "r"(a[1]), "r"(b[7]), "r"(e[2]), "r"(e[3]), "r"(a[3]), "r"(e[4]), "r"(e[5]), "r"(a[5]), "r"(e[6]), "r"(e[7]), "r"(a[7]), "r"(e[8]), "r"(e[9]), "r"(a[9]), "r"(e[10]), "r"(e[11]), "r"(a[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(a[0]), "r"(b[7]), "r"(o[1]), "r"(a[2]), "r"(o[2]), "r"(o[3]), "r"(a[4]), "r"(o[4]), "r"(o[5]), "r"(a[6]), "r"(o[6]), "r"(o[7]), "r"(a[8]), "r"(o[8]), "r"(o[9]), "r"(a[10]), "r"(o[10]), "r"(o[11]));
    m = f[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(f[0]), "+r"(f[1]), "+r"(f[2]), "+r"(f[3]), "+r"(f[4]), "+r"(f[5]), "+r"(f[6]), "+r"(f[7]), "+r"(f[8]), "+r"(f[9]), "+r"(f[10]), "+r"(f[11]), "+r"(f[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(g[0]), "+r"(g[1]), "+r"(g[2]), "+r"(g[3]), "+r"(g[4]), "+r"(g[5]), "+r"(g[6]), "+r"(g[7]), "+r"(g[8]), "+r"(g[9]), "+r"(g[10]), "+r"(g[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(e[0]), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(g[0]), "r"(f[1]), "r"(a[1]), "r"(b[8]), "r"(f[2]), "r"(f[3]), "r"(a[3]), "r"(f[4]), "r"(f[5]), "r"(a[5]), "r"(f[6]), "r"(f[7]), "r"(a[7]), "r"(f[8]), "r"(f[9]), "r"(a[9]), "r"(f[10]), "r"(f[11]), "r"(a[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(a[0]), "r"(b[8]), "r"(g[1]), "r"(a[2]), "r"(g[2]), "r"(g[3]), "r"(a[4]), "r"(g[4]), "r"(g[5]), "r"(a[6]), "r"(g[6]), "r"(g[7]), "r"(a[8]), "r"(g[8]), "r"(g[9]), "r"(a[10]), "r"(g[10]), "r"(g[11]));
    m = e[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(f[0]), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(o[0]), "r"(e[1]), "r"(a[1]), "r"(b[9]), "r"(e[2]), "r"(e[3]), "r"(a[3]), "r"(e[4]), "r"(e[5]), "r"(a[5]), "r"(e[6]), "r"(e[7]), "r"(a[7]), "r"(e[8]), "r"(e[9]), "r"(a[9]), "r"(e[10]), "r"(e[11]), "r"(a[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(a[0]), "r"(b[9]), "r"(o[1]), "r"(a[2]), "r"(o[2]), "r"(o[3]), "r"(a[4]), "r"(o[4]), "r"(o[5]), "r"(a[6]), "r"(o[6]), "r"(o[7]), "r"(a[8]), "r"(o[8]), "r"(o[9]), "r"(a[10]), "r"(o[10]), "r"(o[11]));
    m = f[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(f[0]), "+r"(f[1]), "+r"(f[2]), "+r"(f[3]), "+r"(f[4]), "+r"(f[5]), "+r"(f[6]), "+r"(f[7]), "+r"(f[8]), "+r"(f[9]), "+r"(f[10]), "+r"(f[11]), "+r"(f[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(g[0]), "+r"(g[1]), "+r"(g[2]), "+r"(g[3]), "+r"(g[4]), "+r"(g[5]), "+r"(g[6]), "+r"(g[7]), "+r"(g[8]), "+r"(g[9]), "+r"(g[10]), "+r"(g[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(e[0]), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(g[0]), "r"(f[1]), "r"(a[1]), "r"(b[10]), "r"(f[2]), "r"(f[3]), "r"(a[3]), "r"(f[4]), "r"(f[5]), "r"(a[5]), "r"(f[6]), "r"(f[7]), "r"(a[7]), "r"(f[8]), "r"(f[9]), "r"(a[9]), "r"(f[10]), "r"(f[11]), "r"(a[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(a[0]), "r"(b[10]), "r"(g[1]), "r"(a[2]), "r"(g[2]), "r"(g[3]), "r"(a[4]), "r"(g[4]), "r"(g[5]), "r"(a[6]), "r"(g[6]), "r"(g[7]), "r"(a[8]), "r"(g[8]), "r"(g[9]), "r"(a[10]), "r"(g[10]), "r"(g[11]));
    m = e[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11])
        : "r"(m));
    asm("add.cc.u32 %0, %13, %14;\n\t"
        "madc.lo.cc.u32 %1, %15, %16, %17;\n\t"
        "madc.hi.cc.u32 %2, %15, %16, %18;\n\t"
        "madc.lo.cc.u32 %3, %19, %16, %20;\n\t"
        "madc.hi.cc.u32 %4, %19, %16, %21;\n\t"
        "madc.lo.cc.u32 %5, %22, %16, %23;\n\t"
        "madc.hi.cc.u32 %6, %22, %16, %24;\n\t"
        "madc.lo.cc.u32 %7, %25, %16, %26;\n\t"
        "madc.hi.cc.u32 %8, %25, %16, %27;\n\t"
        "madc.lo.cc.u32 %9, %28, %16, %29;\n\t"
        "madc.hi.cc.u32 %10, %28, %16, %30;\n\t"
        "madc.lo.cc.u32 %11, %31, %16, %32;\n\t"
        "madc.hi.u32 %12, %31, %16, 0;"
        : "=&r"(f[0]), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(o[0]), "r"(e[1]), "r"(a[1]), "r"(b[11]), "r"(e[2]), "r"(e[3]), "r"(a[3]), "r"(e[4]), "r"(e[5]), "r"(a[5]), "r"(e[6]), "r"(e[7]), "r"(a[7]), "r"(e[8]), "r"(e[9]), "r"(a[9]), "r"(e[10]), "r"(e[11]), "r"(a[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, %13, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %14, %15;\n\t"
        "madc.lo.cc.u32 %2, %16, %14, %17;\n\t"
        "madc.hi.cc.u32 %3, %16, %14, %18;\n\t"
        "madc.lo.cc.u32 %4, %19, %14, %20;\n\t"
        "madc.hi.cc.u32 %5, %19, %14, %21;\n\t"
        "madc.lo.cc.u32 %6, %22, %14, %23;\n\t"
        "madc.hi.cc.u32 %7, %22, %14, %24;\n\t"
        "madc.lo.cc.u32 %8, %25, %14, %26;\n\t"
        "madc.hi.cc.u32 %9, %25, %14, %27;\n\t"
        "madc.lo.cc.u32 %10, %28, %14, %29;\n\t"
        "madc.hi.cc.u32 %11, %28, %14, %30;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(a[0]), "r"(b[11]), "r"(o[1]), "r"(a[2]), "r"(o[2]), "r"(o[3]), "r"(a[4]), "r"(o[4]), "r"(o[5]), "r"(a[6]), "r"(o[6]), "r"(o[7]), "r"(a[8]), "r"(o[8]), "r"(o[9]), "r"(a[10]), "r"(o[10]), "r"(o[11]));
    m = f[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %10;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : "+r"(f[0]), "+r"(f[1]), "+r"(f[2]), "+r"(f[3]), "+r"(f[4]), "+r"(f[5]), "+r"(f[6]), "+r"(f[7]), "+r"(f[8]), "+r"(f[9]), "+r"(f[10]), "+r"(f[11]), "+r"(f[12])
        : "r"(m));
    asm("mad.lo.cc.u32 %0, 0xb9feffff, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xb9feffff, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, 0x1eabfffe, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, 0x1eabfffe, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, 0x6730d2a0, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, 0x6730d2a0, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, 0x64774b84, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, 0x64774b84, %12, %7;\n\t"
        "madc.lo.cc.u32 %8, 0x4b1ba7b6, %12, %8;\n\t"
        "madc.hi.cc.u32 %9, 0x4b1ba7b6, %12, %9;\n\t"
        "madc.lo.cc.u32 %10, 0x1a0111ea, %12, %10;\n\t"
        "madc.hi.u32 %11, 0x1a0111ea, %12, %11;"
        : "+r"(g[0]), "+r"(g[1]), "+r"(g[2]), "+r"(g[3]), "+r"(g[4]), "+r"(g[5]), "+r"(g[6]), "+r"(g[7]), "+r"(g[8]), "+r"(g[9]), "+r"(g[10]), "+r"(g[11])
        : "r"(m));
    asm("add.cc.u32 %0, %12, %13;\n\t"
        "addc.cc.u32 %1, %14, %15;\n\t"
        "addc.cc.u32 %2, %16, %17;\n\t"
        "addc.cc.u32 %3, %18, %19;\n\t"
        "addc.cc.u32 %4, %20, %21;\n\t"
        "addc.cc.u32 %5, %22, %23;\n\t"
        "addc.cc.u32 %6, %24, %25;\n\t"
        "addc.cc.u32 %7, %26, %27;\n\t"
        "addc.cc.u32 %8, %28, %29;\n\t"
        "addc.cc.u32 %9, %30, %31;\n\t"
        "addc.cc.u32 %10, %32, %33;\n\t"
        "addc.u32 %11, %34, %35;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11])
        : "r"(g[0]), "r"(f[1]), "r"(g[1]), "r"(f[2]), "r"(g[2]), "r"(f[3]), "r"(g[3]), "r"(f[4]), "r"(g[4]), "r"(f[5]), "r"(g[5]), "r"(f[6]), "r"(g[6]), "r"(f[7]), "r"(g[7]), "r"(f[8]), "r"(g[8]), "r"(f[9]), "r"(g[9]), "r"(f[10]), "r"(g[10]), "r"(f[11]), "r"(g[11]), "r"(f[12]));
    asm("sub.cc.u32 %0, %13, 0xffffaaab;\n\t"
        "subc.cc.u32 %1, %14, 0xb9feffff;\n\t"
        "subc.cc.u32 %2, %15, 0xb153ffff;\n\t"
        "subc.cc.u32 %3, %16, 0x1eabfffe;\n\t"
        "subc.cc.u32 %4, %17, 0xf6b0f624;\n\t"
        "subc.cc.u32 %5, %18, 0x6730d2a0;\n\t"
        "subc.cc.u32 %6, %19, 0xf38512bf;\n\t"
        "subc.cc.u32 %7, %20, 0x64774b84;\n\t"
        "subc.cc.u32 %8, %21, 0x434bacd7;\n\t"
        "subc.cc.u32 %9, %22, 0x4b1ba7b6;\n\t"
        "subc.cc.u32 %10, %23, 0x397fe69a;\n\t"
        "subc.cc.u32 %11, %24, 0x1a0111ea;\n\t"
        "subc.u32 %12, 0, 0;"
        : "=&r"(t[0]), "=&r"(t[1]), "=&r"(t[2]), "=&r"(t[3]), "=&r"(t[4]), "=&r"(t[5]), "=&r"(t[6]), "=&r"(t[7]), "=&r"(t[8]), "=&r"(t[9]), "=&r"(t[10]), "=&r"(t[11]), "=&r"(br)
        : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]));
#pragma unroll
    for (int k = 0; k < 12; k++) r[k] = br ? r[k] : t[k];
}

GB_D void fp_sqr_rows(uint32_t *r, const uint32_t *a)
{
    uint32_t s[24], h[24], e[13], o[12], f[13], g[12], t[12], m, c, br;
    asm("mul.lo.u32 %0, %12, %13;\n\t"
        "mul.hi.u32 %1, %12, %13;\n\t"
        "mul.lo.u32 %2, %12, %14;\n\t"
        "mul.hi.u32 %3, %12, %14;\n\t"
        "mul.lo.u32 %4, %12, %15;\n\t"
        "mul.hi.u32 %5, %12, %15;\n\t"
        "mul.lo.u32 %6, %12, %16;\n\t"
        "mul.hi.u32 %7, %12, %16;\n\t"
        "mul.lo.u32 %8, %12, %17;\n\t"
        "mul.hi.u32 %9, %12, %17;\n\t"
        "mul.lo.u32 %10, %12, %18;\n\t"
        "mul.hi.u32 %11, %12, %18;"
        : "=&r"(h[1]), "=&r"(h[2]), "=&r"(h[3]), "=&r"(h[4]), "=&r"(h[5]), "=&r"(h[6]), "=&r"(h[7]), "=&r"(h[8]), "=&r"(h[9]), "=&r"(h[10]), "=&r"(h[11]), "=&r"(h[12])
        : "r"(a[0]), "r"(a[1]), "r"(a[3]), "r"(a[5]), "r"(a[7]), "r"(a[9]), "r"(a[11]));
    asm("mul.lo.u32 %0, %10, %11;\n\t"
        "mul.hi.u32 %1, %10, %11;\n\t"
        "mul.lo.u32 %2, %10, %12;\n\t"
        "mul.hi.u32 %3, %10, %12;\n\t"
        "mul.lo.u32 %4, %10, %13;\n\t"
        "mul.hi.u32 %5, %10, %13;\n\t"
        "mul.lo.u32 %6, %10, %14;\n\t"
        "mul.hi.u32 %7, %10, %14;\n\t"
        "mul.lo.u32 %8, %10, %15;\n\t"
        "mul.hi.u32 %9, %10, %15;"
        : "=&r"(s[2]), "=&r"(s[3]), "=&r"(s[4]), "=&r"(s[5]), "=&r"(s[6]), "=&r"(s[7]), "=&r"(s[8]), "=&r"(s[9]), "=&r"(s[10]), "=&r"(s[11])
        : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(a[8]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %11, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, %11, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, %11, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, %11, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %14, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %14, %5;\n\t"
        "madc.lo.cc.u32 %6, %11, %15, %6;\n\t"
        "madc.hi.cc.u32 %7, %11, %15, %7;\n\t"
        "madc.lo.cc.u32 %8, %11, %16, %8;\n\t"
        "madc.hi.cc.u32 %9, %11, %16, %9;\n\t"
        "addc.u32 %10, 0, 0;"
        : "+r"(h[3]), "+r"(h[4]), "+r"(h[5]), "+r"(h[6]), "+r"(h[7]), "+r"(h[8]), "+r"(h[9]), "+r"(h[10]), "+r"(h[11]), "+r"(h[12]), "=&r"(h[13])
        : "r"(a[1]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(a[8]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %10, %11, %0;\n\t"
        "madc.hi.cc.u32 %1, %10, %11, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, %10, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, %10, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, %10, %14, %6;\n\t"
        "madc.hi.cc.u32 %7, %10, %14, %7;\n\t"
        "madc.lo.cc.u32 %8, %10, %15, 0;\n\t"
        "madc.hi.u32 %9, %10, %15, 0;"
        : "+r"(s[4]), "+r"(s[5]), "+r"(s[6]), "+r"(s[7]), "+r"(s[8]), "+r"(s[9]), "+r"(s[10]), "+r"(s[11]), "=&r"(s[12]), "=&r"(s[13])
        : "r"(a[1]), "r"(a[3]), "r"(a[5]), "r"(a[7]), "r"(a[9]), "r"(a[11]));
    asm("mad.lo.cc.u32 %0, %10, %11, %0;\n\t"
        "madc.hi.cc.u32 %1, %10, %11, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, %10, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, %10, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, %10, %14, %6;\n\t"
        "madc.hi.cc.u32 %7, %10, %14, %7;\n\t"
        "madc.lo.cc.u32 %8, %10, %15, %8;\n\t"
        "madc.hi.u32 %9, %10, %15, 0;"
        : "+r"(h[5]), "+r"(h[6]), "+r"(h[7]), "+r"(h[8]), "+r"(h[9]), "+r"(h[10]), "+r"(h[11]), "+r"(h[12]), "+r"(h[13]), "=&r"(h[14])
        : "r"(a[2]), "r"(a[3]), "r"(a[5]), "r"(a[7]), "r"(a[9]), "r"(a[11]));
    asm("mad.lo.cc.u32 %0, %9, %10, %0;\n\t"
        "madc.hi.cc.u32 %1, %9, %10, %1;\n\t"
        "madc.lo.cc.u32 %2, %9, %11, %2;\n\t"
        "madc.hi.cc.u32 %3, %9, %11, %3;\n\t"
        "madc.lo.cc.u32 %4, %9, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, %9, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, %9, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, %9, %13, %7;\n\t"
        "addc.u32 %8, 0, 0;"
        : "+r"(s[6]), "+r"(s[7]), "+r"(s[8]), "+r"(s[9]), "+r"(s[10]), "+r"(s[11]), "+r"(s[12]), "+r"(s[13]), "=&r"(s[14])
        : "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(a[8]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %9, %10, %0;\n\t"
        "madc.hi.cc.u32 %1, %9, %10, %1;\n\t"
        "madc.lo.cc.u32 %2, %9, %11, %2;\n\t"
        "madc.hi.cc.u32 %3, %9, %11, %3;\n\t"
        "madc.lo.cc.u32 %4, %9, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, %9, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, %9, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, %9, %13, %7;\n\t"
        "addc.u32 %8, 0, 0;"
        : "+r"(h[7]), "+r"(h[8]), "+r"(h[9]), "+r"(h[10]), "+r"(h[11]), "+r"(h[12]), "+r"(h[13]), "+r"(h[14]), "=&r"(h[15])
        : "r"(a[3]), "r"(a[4]), "r"(a[6]), "r"(a[8]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %8, %9, %0;\n\t"
        "madc.hi.cc.u32 %1, %8, %9, %1;\n\t"
        "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
        "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
        "madc.lo.cc.u32 %4, %8, %11, %4;\n\t"
        "madc.hi.cc.u32 %5, %8, %11, %5;\n\t"
        "madc.lo.cc.u32 %6, %8, %12, %6;\n\t"
        "madc.hi.u32 %7, %8, %12, 0;"
        : "+r"(s[8]), "+r"(s[9]), "+r"(s[10]), "+r"(s[11]), "+r"(s[12]), "+r"(s[13]), "+r"(s[14]), "=&r"(s[15])
        : "r"(a[3]), "r"(a[5]), "r"(a[7]), "r"(a[9]), "r"(a[11]));
    asm("mad.lo.cc.u32 %0, %8, %9, %0;\n\t"
        "madc.hi.cc.u32 %1, %8, %9, %1;\n\t"
        "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
        "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
        "madc.lo.cc.u32 %4, %8, %11, %4;\n\t"
        "madc.hi.cc.u32 %5, %8, %11, %5;\n\t"
        "madc.lo.cc.u32 %6, %8, %12, %6;\n\t"
        "madc.hi.u32 %7, %8, %12, 0;"
        : "+r"(h[9]), "+r"(h[10]), "+r"(h[11]), "+r"(h[12]), "+r"(h[13]), "+r"(h[14]), "+r"(h[15]), "=&r"(h[16])
        : "r"(a[4]), "r"(a[5]), "r"(a[7]), "r"(a[9]), "r"(a[11]));
    asm("mad.lo.cc.u32 %0, %7, %8, %0;\n\t"
        "madc.hi.cc.u32 %1, %7, %8, %1;\n\t"
        "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
        "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
        "madc.lo.cc.u32 %4, %7, %10, %4;\n\t"
        "madc.hi.cc.u32 %5, %7, %10, %5;\n\t"
        "addc.u32 %6, 0, 0;"
        : "+r"(s[10]), "+r"(s[11]), "+r"(s[12]), "+r"(s[13]), "+r"(s[14]), "+r"(s[15]), "=&r"(s[16])
        : "r"(a[4]), "r"(a[6]), "r"(a[8]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %7, %8, %0;\n\t"
        "madc.hi.cc.u32 %1, %7, %8, %1;\n\t"
        "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
        "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
        "madc.lo.cc.u32 %4, %7, %10, %4;\n\t"
        "madc.hi.cc.u32 %5, %7, %10, %5;\n\t"
        "addc.u32 %6, 0, 0;"
        : "+r"(h[11]), "+r"(h[12]), "+r"(h[13]), "+r"(h[14]), "+r"(h[15]), "+r"(h[16]), "=&r"(h[17])
        : "r"(a[5]), "r"(a[6]), "r"(a[8]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %6, %7, %0;\n\t"
        "madc.hi.cc.u32 %1, %6, %7, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %8, %2;\n\t"
        "madc.hi.cc.u32 %3, %6, %8, %3;\n\t"
        "madc.lo.cc.u32 %4, %6, %9, %4;\n\t"
        "madc.hi.u32 %5, %6, %9, 0;"
        : "+r"(s[12]), "+r"(s[13]), "+r"(s[14]), "+r"(s[15]), "+r"(s[16]), "=&r"(s[17])
        : "r"(a[5]), "r"(a[7]), "r"(a[9]), "r"(a[11]));
    asm("mad.lo.cc.u32 %0, %6, %7, %0;\n\t"
        "madc.hi.cc.u32 %1, %6, %7, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %8, %2;\n\t"
        "madc.hi.cc.u32 %3, %6, %8, %3;\n\t"
        "madc.lo.cc.u32 %4, %6, %9, %4;\n\t"
        "madc.hi.u32 %5, %6, %9, 0;"
        : "+r"(h[13]), "+r"(h[14]), "+r"(h[15]), "+r"(h[16]), "+r"(h[17]), "=&r"(h[18])
        : "r"(a[6]), "r"(a[7]), "r"(a[9]), "r"(a[11]));
    asm("mad.lo.cc.u32 %0, %5, %6, %0;\n\t"
        "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
        "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
        "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
        "addc.u32 %4, 0, 0;"
        : "+r"(s[14]), "+r"(s[15]), "+r"(s[16]), "+r"(s[17]), "=&r"(s[18])
        : "r"(a[6]), "r"(a[8]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %5, %6, %0;\n\t"
        "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
        "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
        "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
        "addc.u32 %4, 0, 0;"
        : "+r"(h[15]), "+r"(h[16]), "+r"(h[17]), "+r"(h[18]), "=&r"(h[19])
        : "r"(a[7]), "r"(a[8]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %4, %5, %0;\n\t"
        "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
        "madc.lo.cc.u32 %2, %4, %6, %2;\n\t"
        "madc.hi.u32 %3, %4, %6, 0;"
        : "+r"(s[16]), "+r"(s[17]), "+r"(s[18]), "=&r"(s[19])
        : "r"(a[7]), "r"(a[9]), "r"(a[11]));
    asm("mad.lo.cc.u32 %0, %4, %5, %0;\n\t"
        "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
        "madc.lo.cc.u32 %2, %4, %6, %2;\n\t"
        "madc.hi.u32 %3, %4, %6, 0;"
        : "+r"(h[17]), "+r"(h[18]), "+r"(h[19]), "=&r"(h[20])
        : "r"(a[8]), "r"(a[9]), "r"(a[11]));
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32 %2, 0, 0;"
        : "+r"(s[18]), "+r"(s[19]), "=&r"(s[20])
        : "r"(a[8]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32 %2, 0, 0;"
        : "+r"(h[19]), "+r"(h[20]), "=&r"(h[21])
        : "r"(a[9]), "r"(a[10]));
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
        "madc.hi.u32 %1, %2, %3, 0;"
        : "+r"(s[20]), "=&r"(s[21])
        : "r"(a[9]), "r"(a[11]));
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
        "madc.hi.u32 %1, %2, %3, 0;"
        : "+r"(h[21]), "=&r"(h[22])
        : "r"(a[10]), "r"(a[11]));
    asm("add.cc.u32 %0, 0, %22;\n\t"
        "addc.cc.u32 %1, %1, %23;\n\t"
        "addc.cc.u32 %2, %2, %24;\n\t"
        "addc.cc.u32 %3, %3, %25;\n\t"
        "addc.cc.u32 %4, %4, %26;\n\t"
        "addc.cc.u32 %5, %5, %27;\n\t"
        "addc.cc.u32 %6, %6, %28;\n\t"
        "addc.cc.u32 %7, %7, %29;\n\t"
        "addc.cc.u32 %8, %8, %30;\n\t"
        "addc.cc.u32 %9, %9, %31;\n\t"
        "addc.cc.u32 %10, %10, %32;\n\t"
        "addc.cc.u32 %11, %11, %33;\n\t"
        "addc.cc.u32 %12, %12, %34;\n\t"
        "addc.cc.u32 %13, %13, %35;\n\t"
        "addc.cc.u32 %14, %14, %36;\n\t"
        "addc.cc.u32 %15, %15, %37;\n\t"
        "addc.cc.u32 %16, %16, %38;\n\t"
        "addc.cc.u32 %17, %17, %39;\n\t"
        "addc.cc.u32 %18, %18, %40;\n\t"
        "addc.cc.u32 %19, %19, %41;\n\t"
        "addc.cc.u32 %20, %20, %42;\n\t"
        "addc.u32 %21, 0, %43;"
        : "=&r"(s[1]), "+r"(s[2]), "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6]), "+r"(s[7]), "+r"(s[8]), "+r"(s[9]), "+r"(s[10]), "+r"(s[11]), "+r"(s[12]), "+r"(s[13]), "+r"(s[14]), "+r"(s[15]), "+r"(s[16]), "+r"(s[17]), "+r"(s[18]), "+r"(s[19]), "+r"(s[20]), "+r"(s[21]), "=&r"(s[22])
        : "r"(h[1]), "r"(h[2]), "r"(h[3]), "r"(h[4]), "r"(h[5]), "r"(h[6]), "r"(h[7]), "r"(h[8]), "r"(h[9]), "r"(h[10]), "r"(h[11]), "r"(h[12]), "r"(h[13]), "r"(h[14]), "r"(h[15]), "r"(h[16]), "r"(h[17]), "r"(h[18]), "r"(h[19]), "r"(h[20]), "r"(h[21]), "r"(h[22]));
    s[23] = s[22] >> 31;
#pragma unroll
    for (int k = 22; k > 1; k--) s[k] = __funnelshift_l(s[k - 1], s[k], 1);
    s[1] <<= 1;
    asm("mul.lo.u32 %0, %24, %24;\n\t"
        "mad.hi.cc.u32 %1, %24, %24, %1;\n\t"
        "madc.lo.cc.u32 %2, %25, %25, %2;\n\t"
        "madc.hi.cc.u32 %3, %25, %25, %3;\n\t"
        "madc.lo.cc.u32 %4, %26, %26, %4;\n\t"
        "madc.hi.cc.u32 %5, %26, %26, %5;\n\t"
        "madc.lo.cc.u32 %6, %27, %27, %6;\n\t"
        "madc.hi.cc.u32 %7, %27, %27, %7;\n\t"
        "madc.lo.cc.u32 %8, %28, %28, %8;\n\t"
        "madc.hi.cc.u32 %9, %28, %28, %9;\n\t"
        "madc.lo.cc.u32 %10, %29, %29, %10;\n\t"
        "madc.hi.cc.u32 %11, %29, %29, %11;\n\t"
        "madc.lo.cc.u32 %12, %30, %30, %12;\n\t"
        "madc.hi.cc.u32 %13, %30, %30, %13;\n\t"
        "madc.lo.cc.u32 %14, %31, %31, %14;\n\t"
        "madc.hi.cc.u32 %15, %31, %31, %15;\n\t"
        "madc.lo.cc.u32 %16, %32, %32, %16;\n\t"
        "madc.hi.cc.u32 %17, %32, %32, %17;\n\t"
        "madc.lo.cc.u32 %18, %33, %33, %18;\n\t"
        "madc.hi.cc.u32 %19, %33, %33, %19;\n\t"
        "madc.lo.cc.u32 %20, %34, %34, %20;\n\t"
        "madc.hi.cc.u32 %21, %34, %34, %21;\n\t"
        "madc.lo.cc.u32 %22, %35, %35, %22;\n\t"
        "madc.hi.u32 %23, %35, %35, %23;"
        : "=&r"(s[0]), "+r"(s[1]), "+r"(s[2]), "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6]), "+r"(s[7]), "+r"(s[8]), "+r"(s[9]), "+r"(s[10]), "+r"(s[11]), "+r"(s[12]), "+r"(s[13]), "+r"(s[14]), "+r"(s[15]), "+r"(s[16]), "+r"(s[17]), "+r"(s[18]), "+r"(s[19]), "+r"(s[20]), "+r"(s[21]), "+r"(s[22]), "+r"(s[23])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]));
    m = s[0] * 0xfffcfffdu;
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %14;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %15;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %16;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %17;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %18;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %19;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %20;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %21;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %22;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %23;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %24;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %25;\n\t"
        "addc.u32 %12, 0, 0;"
        : "=&r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(m), "r"(s[0]), "r"(s[1]), "r"(s[2]), "r"(s[3]), "r"(s[4]), "r"(s[5]), "r"(s[6]), "r"(s[7]), "r"(s[8]), "r"(s[9]), "r"(s[10]), "r"(s[11]));
    o[0] = 0xb9feffffu * m;
    o[1] = __umulhi(0xb9feffffu, m);
    o[2] = 0x1eabfffeu * m;
    o[3] = __umulhi(0x1eabfffeu, m);
    o[4] = 0x6730d2a0u * m;
    o[5] = __umulhi(0x6730d2a0u, m);
    o[6] = 0x64774b84u * m;
    o[7] = __umulhi(0x64774b84u, m);
    o[8] = 0x4b1ba7b6u * m;
    o[9] = __umulhi(0x4b1ba7b6u, m);
    o[10] = 0x1a0111eau * m;
    o[11] = __umulhi(0x1a0111eau, m);
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(f[0]), "=&r"(c)
        : "r"(o[0]), "r"(e[1]));
    m = f[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(m), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(e[10]), "r"(e[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(m), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(e[0]), "=&r"(c)
        : "r"(g[0]), "r"(f[1]));
    m = e[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(m), "r"(f[2]), "r"(f[3]), "r"(f[4]), "r"(f[5]), "r"(f[6]), "r"(f[7]), "r"(f[8]), "r"(f[9]), "r"(f[10]), "r"(f[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(m), "r"(g[1]), "r"(g[2]), "r"(g[3]), "r"(g[4]), "r"(g[5]), "r"(g[6]), "r"(g[7]), "r"(g[8]), "r"(g[9]), "r"(g[10]), "r"(g[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(f[0]), "=&r"(c)
        : "r"(o[0]), "r"(e[1]));
    m = f[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(m), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(e[10]), "r"(e[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(m), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(e[0]), "=&r"(c)
        : "r"(g[0]), "r"(f[1]));
    m = e[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(m), "r"(f[2]), "r"(f[3]), "r"(f[4]), "r"(f[5]), "r"(f[6]), "r"(f[7]), "r"(f[8]), "r"(f[9]), "r"(f[10]), "r"(f[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(m), "r"(g[1]), "r"(g[2]), "r"(g[3]), "r"(g[4]), "r"(g[5]), "r"(g[6]), "r"(g[7]), "r"(g[8]), "r"(g[9]), "r"(g[10]), "r"(g[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(f[0]), "=&r"(c)
        : "r"(o[0]), "r"(e[1]));
    m = f[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(m), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(e[10]), "r"(e[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(m), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(e[0]), "=&r"(c)
        : "r"(g[0]), "r"(f[1]));
    m = e[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(m), "r"(f[2]), "r"(f[3]), "r"(f[4]), "r"(f[5]), "r"(f[6]), "r"(f[7]), "r"(f[8]), "r"(f[9]), "r"(f[10]), "r"(f[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(m), "r"(g[1]), "r"(g[2]), "r"(g[3]), "r"(g[4]), "r"(g[5]), "r"(g[6]), "r"(g[7]), "r"(g[8]), "r"(g[9]), "r"(g[10]), "r"(g[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(f[0]), "=&r"(c)
        : "r"(o[0]), "r"(e[1]));
    m = f[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(m), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(e[10]), "r"(e[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(m), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(e[0]), "=&r"(c)
        : "r"(g[0]), "r"(f[1]));
    m = e[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(m), "r"(f[2]), "r"(f[3]), "r"(f[4]), "r"(f[5]), "r"(f[6]), "r"(f[7]), "r"(f[8]), "r"(f[9]), "r"(f[10]), "r"(f[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(m), "r"(g[1]), "r"(g[2]), "r"(g[3]), "r"(g[4]), "r"(g[5]), "r"(g[6]), "r"(g[7]), "r"(g[8]), "r"(g[9]), "r"(g[10]), "r"(g[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(f[0]), "=&r"(c)
        : "r"(o[0]), "r"(e[1]));
    m = f[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(m), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(e[10]), "r"(e[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(m), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(e[0]), "=&r"(c)
        : "r"(g[0]), "r"(f[1]));
    m = e[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(o[0]), "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4]), "=&r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "=&r"(o[8]), "=&r"(o[9]), "=&r"(o[10]), "=&r"(o[11])
        : "r"(m), "r"(f[2]), "r"(f[3]), "r"(f[4]), "r"(f[5]), "r"(f[6]), "r"(f[7]), "r"(f[8]), "r"(f[9]), "r"(f[10]), "r"(f[11]), "r"(f[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]), "=&r"(e[7]), "=&r"(e[8]), "=&r"(e[9]), "=&r"(e[10]), "=&r"(e[11]), "=&r"(e[12])
        : "r"(m), "r"(g[1]), "r"(g[2]), "r"(g[3]), "r"(g[4]), "r"(g[5]), "r"(g[6]), "r"(g[7]), "r"(g[8]), "r"(g[9]), "r"(g[10]), "r"(g[11]));
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;"
        : "=&r"(f[0]), "=&r"(c)
        : "r"(o[0]), "r"(e[1]));
    m = f[0] * 0xfffcfffdu;
    asm("add.cc.u32 %0, %0, 0xffffffff;\n\t"
        "madc.lo.cc.u32 %1, 0xb9feffff, %13, %14;\n\t"
        "madc.hi.cc.u32 %2, 0xb9feffff, %13, %15;\n\t"
        "madc.lo.cc.u32 %3, 0x1eabfffe, %13, %16;\n\t"
        "madc.hi.cc.u32 %4, 0x1eabfffe, %13, %17;\n\t"
        "madc.lo.cc.u32 %5, 0x6730d2a0, %13, %18;\n\t"
        "madc.hi.cc.u32 %6, 0x6730d2a0, %13, %19;\n\t"
        "madc.lo.cc.u32 %7, 0x64774b84, %13, %20;\n\t"
        "madc.hi.cc.u32 %8, 0x64774b84, %13, %21;\n\t"
        "madc.lo.cc.u32 %9, 0x4b1ba7b6, %13, %22;\n\t"
        "madc.hi.cc.u32 %10, 0x4b1ba7b6, %13, %23;\n\t"
        "madc.lo.cc.u32 %11, 0x1a0111ea, %13, %24;\n\t"
        "madc.hi.u32 %12, 0x1a0111ea, %13, 0;"
        : "+r"(c), "=&r"(g[0]), "=&r"(g[1]), "=&r"(g[2]), "=&r"(g[3]), "=&r"(g[4]), "=&r"(g[5]), "=&r"(g[6]), "=&r"(g[7]), "=&r"(g[8]), "=&r"(g[9]), "=&r"(g[10]), "=&r"(g[11])
        : "r"(m), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(e[10]), "r"(e[11]), "r"(e[12]));
    asm("mad.lo.cc.u32 %0, 0xffffaaab, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, 0xffffaaab, %13, %14;\n\t"
        "madc.lo.cc.u32 %2, 0xb153ffff, %13, %15;\n\t"
        "madc.hi.cc.u32 %3, 0xb153ffff, %13, %16;\n\t"
        "madc.lo.cc.u32 %4, 0xf6b0f624, %13, %17;\n\t"
        "madc.hi.cc.u32 %5, 0xf6b0f624, %13, %18;\n\t"
        "madc.lo.cc.u32 %6, 0xf38512bf, %13, %19;\n\t"
        "madc.hi.cc.u32 %7, 0xf38512bf, %13, %20;\n\t"
        "madc.lo.cc.u32 %8, 0x434bacd7, %13, %21;\n\t"
        "madc.hi.cc.u32 %9, 0x434bacd7, %13, %22;\n\t"
        "madc.lo.cc.u32 %10, 0x397fe69a, %13, %23;\n\t"
        "madc.hi.cc.u32 %11, 0x397fe69a, %13, %24;\n\t"
        "addc.u32 %12, 0, 0;"
        : "+r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3]), "=&r"(f[4]), "=&r"(f[5]), "=&r"(f[6]), "=&r"(f[7]), "=&r"(f[8]), "=&r"(f[9]), "=&r"(f[10]), "=&r"(f[11]), "=&r"(f[12])
        : "r"(m), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]));
    asm("add.cc.u32 %0, %12, %13;\n\t"
        "addc.cc.u32 %1, %14, %15;\n\t"
        "addc.cc.u32 %2, %16, %17;\n\t"
        "addc.cc.u32 %3, %18, %19;\n\t"
        "addc.cc.u32 %4, %20, %21;\n\t"
        "addc.cc.u32 %5, %22, %23;\n\t"
        "addc.cc.u32 %6, %24, %25;\n\t"
        "addc.cc.u32 %7, %26, %27;\n\t"
        "addc.cc.u32 %8, %28, %29;\n\t"
        "addc.cc.u32 %9, %30, %31;\n\t"
        "addc.cc.u32 %10, %32, %33;\n\t"
        "addc.u32 %11, %34, %35;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11])
        : "r"(g[0]), "r"(f[1]), "r"(g[1]), "r"(f[2]), "r"(g[2]), "r"(f[3]), "r"(g[3]), "r"(f[4]), "r"(g[4]), "r"(f[5]), "r"(g[5]), "r"(f[6]), "r"(g[6]), "r"(f[7]), "r"(g[7]), "r"(f[8]), "r"(g[8]), "r"(f[9]), "r"(g[9]), "r"(f[10]), "r"(g[10]), "r"(f[11]), "r"(g[11]), "r"(f[12]));
    asm("add.cc.u32 %0, %0, %12;\n\t"
        "addc.cc.u32 %1, %1, %13;\n\t"
        "addc.cc.u32 %2, %2, %14;\n\t"
        "addc.cc.u32 %3, %3, %15;\n\t"
        "addc.cc.u32 %4, %4, %16;\n\t"
        "addc.cc.u32 %5, %5, %17;\n\t"
        "addc.cc.u32 %6, %6, %18;\n\t"
        "addc.cc.u32 %7, %7, %19;\n\t"
        "addc.cc.u32 %8, %8, %20;\n\t"
        "addc.cc.u32 %9, %9, %21;\n\t"
        "addc.cc.u32 %10, %10, %22;\n\t"
        "addc.u32 %11, %11, %23;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11])
        : "r"(s[12]), "r"(s[13]), "r"(s[14]), "r"(s[15]), "r"(s[16]), "r"(s[17]), "r"(s[18]), "r"(s[19]), "r"(s[20]), "r"(s[21]), "r"(s[22]), "r"(s[23]));
    asm("sub.cc.u32 %0, %13, 0xffffaaab;\n\t"
        "subc.cc.u32 %1, %14, 0xb9feffff;\n\t"
        "subc.cc.u32 %2, %15, 0xb153ffff;\n\t"
        "subc.cc.u32 %3, %16, 0x1eabfffe;\n\t"
        "subc.cc.u32 %4, %17, 0xf6b0f624;\n\t"
        "subc.cc.u32 %5, %18, 0x6730d2a0;\n\t"
        "subc.cc.u32 %6, %19, 0xf38512bf;\n\t"
        "subc.cc.u32 %7, %20, 0x64774b84;\n\t"
        "subc.cc.u32 %8, %21, 0x434bacd7;\n\t"
        "subc.cc.u32 %9, %22, 0x4b1ba7b6;\n\t"
        "subc.cc.u32 %10, %23, 0x397fe69a;\n\t"
        "subc.cc.u32 %11, %24, 0x1a0111ea;\n\t"
        "subc.u32 %12, 0, 0;"
        : "=&r"(t[0]), "=&r"(t[1]), "=&r"(t[2]), "=&r"(t[3]), "=&r"(t[4]), "=&r"(t[5]), "=&r"(t[6]), "=&r"(t[7]), "=&r"(t[8]), "=&r"(t[9]), "=&r"(t[10]), "=&r"(t[11]), "=&r"(br)
        : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]));
#pragma unroll
    for (int k = 0; k < 12; k++) r[k] = br ? r[k] : t[k];
}
}  // namespace gb
#endif
