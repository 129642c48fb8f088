// Folds over the BLS12-381 scalar field by one challenge: x0 + r x from a table of r.
//
// A fold's multiplier is the same for a whole round, so its multiples come from a table:
// c_i = r 2^(32 i + 64) mod p, i = 0..7 (shared memory, one block-wide set-up a round or item).
// x0 2^64 + sum_i x_i c_i is below 2^64 x0 + 2^35 p, all its products start at word 0 -- rows of
// one even and one odd carry chain, none of them shifted and none waiting for another row's
// reduction -- and two rows of Montgomery reduction divide it by 2^64: 64 + 16 multiply-add
// pairs where a product takes 112, and the addition of x0 comes with them. The result is below
// x0 + p + 2^-29 p: one conditional subtraction, and the rare value still at or above p (its top
// word then is p's) is corrected exactly. Checked on the CPU by
// tests/test_field_lazy_emulated.py. Measured on B200: g(abc + de) at n = 22
// 2.52 -> 2.41 ms.
#pragma once
#include <cstdint>

namespace sc {

// Row i: e and o += x c for the even and the odd words of c (e0..e9 words 0..9, o0..o8 words
// 1..9; the chains' carries go into e8, e9 and o8).
__device__ __forceinline__ void bls_fold_row(uint32_t (&e)[10], uint32_t (&o)[9], const uint32_t x, const uint32_t (&c)[8]) {
  asm("{\n\t"
      "mad.lo.cc.u32 %0, %20, %19, %0;\n\t"
      "madc.hi.cc.u32 %1, %20, %19, %1;\n\t"
      "madc.lo.cc.u32 %2, %22, %19, %2;\n\t"
      "madc.hi.cc.u32 %3, %22, %19, %3;\n\t"
      "madc.lo.cc.u32 %4, %24, %19, %4;\n\t"
      "madc.hi.cc.u32 %5, %24, %19, %5;\n\t"
      "madc.lo.cc.u32 %6, %26, %19, %6;\n\t"
      "madc.hi.cc.u32 %7, %26, %19, %7;\n\t"
      "addc.cc.u32 %8, %8, 0;\n\t"
      "addc.u32 %9, %9, 0;\n\t"
      "mad.lo.cc.u32 %10, %21, %19, %10;\n\t"
      "madc.hi.cc.u32 %11, %21, %19, %11;\n\t"
      "madc.lo.cc.u32 %12, %23, %19, %12;\n\t"
      "madc.hi.cc.u32 %13, %23, %19, %13;\n\t"
      "madc.lo.cc.u32 %14, %25, %19, %14;\n\t"
      "madc.hi.cc.u32 %15, %25, %19, %15;\n\t"
      "madc.lo.cc.u32 %16, %27, %19, %16;\n\t"
      "madc.hi.cc.u32 %17, %27, %19, %17;\n\t"
      "addc.u32 %18, %18, 0;\n\t"
      "}"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]),
        "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(o[8])
      : "r"(x), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]), "r"(c[5]), "r"(c[6]), "r"(c[7]));
}

// r = (e + o 2^32) / 2^64 mod p by two rows of reduction, below 2^256: t = e + o 2^32, then twice
// m = -t_0 (as -1/p = -1 mod 2^32), t = (t + m p) / 2^32.
__device__ __forceinline__ void bls_fold_end(uint32_t (&r)[8], const uint32_t (&e)[10], const uint32_t (&o)[9], const uint32_t (&p)[8]) {
  asm("{\n\t.reg .u32 t0, t1, t2, t3, t4, t5, t6, t7, t8, t9, m;\n\t"
      "mov.u32 t0, %8;\n\t"
      "add.cc.u32 t1, %9, %18;\n\t"
      "addc.cc.u32 t2, %10, %19;\n\t"
      "addc.cc.u32 t3, %11, %20;\n\t"
      "addc.cc.u32 t4, %12, %21;\n\t"
      "addc.cc.u32 t5, %13, %22;\n\t"
      "addc.cc.u32 t6, %14, %23;\n\t"
      "addc.cc.u32 t7, %15, %24;\n\t"
      "addc.cc.u32 t8, %16, %25;\n\t"
      "addc.u32 t9, %17, %26;\n\t"
      "sub.u32 m, 0, t0;\n\t"
      "mad.lo.cc.u32 t0, m, %27, t0;\n\t"
      "madc.hi.cc.u32 t1, m, %27, t1;\n\t"
      "madc.lo.cc.u32 t2, m, %29, t2;\n\t"
      "madc.hi.cc.u32 t3, m, %29, t3;\n\t"
      "madc.lo.cc.u32 t4, m, %31, t4;\n\t"
      "madc.hi.cc.u32 t5, m, %31, t5;\n\t"
      "madc.lo.cc.u32 t6, m, %33, t6;\n\t"
      "madc.hi.cc.u32 t7, m, %33, t7;\n\t"
      "addc.cc.u32 t8, t8, 0;\n\t"
      "addc.u32 t9, t9, 0;\n\t"
      "mad.lo.cc.u32 t1, m, %28, t1;\n\t"
      "madc.hi.cc.u32 t2, m, %28, t2;\n\t"
      "madc.lo.cc.u32 t3, m, %30, t3;\n\t"
      "madc.hi.cc.u32 t4, m, %30, t4;\n\t"
      "madc.lo.cc.u32 t5, m, %32, t5;\n\t"
      "madc.hi.cc.u32 t6, m, %32, t6;\n\t"
      "madc.lo.cc.u32 t7, m, %34, t7;\n\t"
      "madc.hi.cc.u32 t8, m, %34, t8;\n\t"
      "addc.u32 t9, t9, 0;\n\t"
      "sub.u32 m, 0, t1;\n\t"
      "mad.lo.cc.u32 t1, m, %27, t1;\n\t"
      "madc.hi.cc.u32 t2, m, %27, t2;\n\t"
      "madc.lo.cc.u32 t3, m, %29, t3;\n\t"
      "madc.hi.cc.u32 t4, m, %29, t4;\n\t"
      "madc.lo.cc.u32 t5, m, %31, t5;\n\t"
      "madc.hi.cc.u32 t6, m, %31, t6;\n\t"
      "madc.lo.cc.u32 t7, m, %33, t7;\n\t"
      "madc.hi.cc.u32 t8, m, %33, t8;\n\t"
      "addc.u32 t9, t9, 0;\n\t"
      "mad.lo.cc.u32 t2, m, %28, t2;\n\t"
      "madc.hi.cc.u32 t3, m, %28, t3;\n\t"
      "madc.lo.cc.u32 t4, m, %30, t4;\n\t"
      "madc.hi.cc.u32 t5, m, %30, t5;\n\t"
      "madc.lo.cc.u32 t6, m, %32, t6;\n\t"
      "madc.hi.cc.u32 t7, m, %32, t7;\n\t"
      "madc.lo.cc.u32 t8, m, %34, t8;\n\t"
      "madc.hi.u32 t9, m, %34, t9;\n\t"
      "mov.u32 %0, t2;\n\t"
      "mov.u32 %1, t3;\n\t"
      "mov.u32 %2, t4;\n\t"
      "mov.u32 %3, t5;\n\t"
      "mov.u32 %4, t6;\n\t"
      "mov.u32 %5, t7;\n\t"
      "mov.u32 %6, t8;\n\t"
      "mov.u32 %7, t9;\n\t"
      "}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7])
      : "r"(e[0]), "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]),
        "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]),
        "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7]));
}

}  // namespace sc
