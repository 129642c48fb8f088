// Goldilocks sums of products reduced once (p = 2^64 - 2^32 + 1, R = 2^64; field_gold.cuh).
//
// A sum of products is five words: 128 bits and the carries above them. Adding a product costs
// its four multiply-add pairs and five carries, where a reduced product and a lazy addition
// cost 29 instructions; the whole sum is reduced as one product is (the words above 2^128 are
// worth 2^32 - 1 each 2^64). Operands are any words below 2^64; sums of fewer than 2^31
// products. Checked on the CPU by tests/test_field_lazy_emulated.py.
#pragma once
#include <cstdint>

#include "field_gold.cuh"

namespace sc {

// r = x y.
__device__ __forceinline__ void gold_acc_first(uint32_t (&r)[5], const uint32_t (&x)[2], const uint32_t (&y)[2]) {
  asm("{\n\t.reg .u32 t1, t2, t3;\n\t"
      "mul.lo.u32 %0, %5, %7;\n\t"
      "mul.hi.u32 t1, %5, %7;\n\t"
      "mul.lo.u32 t2, %6, %8;\n\t"
      "mul.hi.u32 t3, %6, %8;\n\t"
      "mad.lo.cc.u32 t1, %5, %8, t1;\n\t"
      "madc.hi.cc.u32 t2, %5, %8, t2;\n\t"
      "addc.u32 t3, t3, 0;\n\t"
      "mad.lo.cc.u32 %1, %6, %7, t1;\n\t"
      "madc.hi.cc.u32 %2, %6, %7, t2;\n\t"
      "addc.u32 %3, t3, 0;\n\t"
      "mov.u32 %4, 0;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4])
      : "r"(x[0]), "r"(x[1]), "r"(y[0]), "r"(y[1]));
}

// r = t + x y.
__device__ __forceinline__ void gold_acc_mul(uint32_t (&r)[5], const uint32_t (&t)[5], const uint32_t (&x)[2],
                                             const uint32_t (&y)[2]) {
  asm("{\n\t.reg .u32 t1, t2, t3, t4;\n\t"
      "mad.lo.cc.u32 %0, %10, %12, %5;\n\t"
      "madc.hi.cc.u32 t1, %10, %12, %6;\n\t"
      "madc.lo.cc.u32 t2, %11, %13, %7;\n\t"
      "madc.hi.cc.u32 t3, %11, %13, %8;\n\t"
      "addc.u32 t4, %9, 0;\n\t"
      "mad.lo.cc.u32 t1, %10, %13, t1;\n\t"
      "madc.hi.cc.u32 t2, %10, %13, t2;\n\t"
      "addc.cc.u32 t3, t3, 0;\n\t"
      "addc.u32 t4, t4, 0;\n\t"
      "mad.lo.cc.u32 %1, %11, %12, t1;\n\t"
      "madc.hi.cc.u32 %2, %11, %12, t2;\n\t"
      "addc.cc.u32 %3, t3, 0;\n\t"
      "addc.u32 %4, t4, 0;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4])
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(x[0]), "r"(x[1]), "r"(y[0]), "r"(y[1]));
}

// r = t + x 2^64 (a value among the products).
__device__ __forceinline__ void gold_acc_add(uint32_t (&r)[5], const uint32_t (&t)[5], const uint32_t (&x)[2]) {
  asm("{\n\t"
      "mov.u32 %0, %5;\n\t"
      "mov.u32 %1, %6;\n\t"
      "add.cc.u32 %2, %7, %10;\n\t"
      "addc.cc.u32 %3, %8, %11;\n\t"
      "addc.u32 %4, %9, 0;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4])
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(x[0]), "r"(x[1]));
}

// r = t / 2^64 mod p, any representative below 2^64. With l the low 64 bits and h the rest:
// a = l (1 + 2^32) mod 2^64 (carry e), b = a - (a >> 32) - e < p (gold_mul in field.cuh), and
// t / 2^64 = h - b; h's words above 2^64 come in as eps each, a carry of that as eps once more,
// and a borrow of b as p.
__device__ __forceinline__ void gold_acc_reduce(uint32_t (&r)[2], const uint32_t (&t)[5], const GoldK k) {
  asm("{\n\t.reg .u32 a1, e, b0, b1, h0, h1, c, m;\n\t"
      "add.cc.u32 a1, %2, %3;\n\t"
      "addc.u32 e, 0, 0;\n\t"
      "sub.cc.u32 b0, %2, a1;\n\t"
      "subc.u32 b1, a1, 0;\n\t"
      "sub.cc.u32 b0, b0, e;\n\t"
      "subc.u32 b1, b1, 0;\n\t"
      "mad.lo.cc.u32 h0, %6, %9, %4;\n\t"
      "madc.hi.cc.u32 h1, %6, %9, %5;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "mad.lo.cc.u32 h0, c, %9, h0;\n\t"
      "addc.u32 h1, h1, 0;\n\t"
      "sub.cc.u32 h0, h0, b0;\n\t"
      "subc.cc.u32 h1, h1, b1;\n\t"
      "subc.u32 m, 0, 0;\n\t"
      "mad.lo.cc.u32 %0, m, m, h0;\n\t"
      "madc.lo.u32 %1, m, %7, h1;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1])
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(k.one), "r"(k.zero), "r"(k.eps));
}

// r = p - a for a <= p.
__device__ __forceinline__ void gold_neg(uint32_t (&r)[2], const uint32_t (&a)[2], const GoldK k) {
  asm("{\n\t"
      "sub.cc.u32 %0, %4, %2;\n\t"
      "subc.u32 %1, %5, %3;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1])
      : "r"(a[0]), "r"(a[1]), "r"(k.one), "r"(k.eps));
}

}  // namespace sc
