// 2^127 - 1 arithmetic on any representative below 2^128.
//
// With p = 2^127 - 1, 2^128 = 2 (mod p): a carry out of 128 bits is worth 2 and a borrow -2, so
// sums, differences and products stay in four words with no compare and no select, and a value
// is made canonical (m127_canon) only by a fold, whose result is stored, and by fe_mul; point sums
// leave a thread as any representative and are reduced once a round. R = 2^128 = 2 (mod p), so the
// Montgomery product x y / R = x y / 2: with x y = hi 2^128 + lo it is hi + lo / 2, and
// lo / 2 = (lo >> 1) + (lo & 1) 2^126.
//
// The 256-bit product's words at even positions (i + j even) and at odd ones are two sets of
// carry chains of multiply-adds, merged by one chain of additions: 16 multiply-add pairs, 3
// carries, 7 additions; the reduction is 15 more instructions. Each statement is one asm block
// (the carry flag does not survive between statements); tests/test_field_lazy_emulated.py runs
// them on the CPU against big integers. Measured on B200 against the canonical product in C++
// with 64-bit intermediates, called out of line: a 17-term gate over 2^127 - 1 at n = 16 843 ->
// 684 us, a permutation check 315 -> 278 us, 40 served requests 7.12 -> 6.69 ms.
#pragma once
#include <cstdint>

namespace sc {

// r = x y 2^-128 mod p for any x, y below 2^128; r below 2^128.
__device__ __forceinline__ void m127_mul_lazy(uint32_t (&r)[4], const uint32_t (&x)[4], const uint32_t (&y)[4]) {
  asm("{\n\t.reg .u32 e0, e1, e2, e3, e4, e5, e6, e7, o1, o2, o3, o4, o5, o6, o7, b, c;\n\t"
      // y0
      "mul.lo.u32 e0, %4, %8;\n\t"
      "mul.hi.u32 e1, %4, %8;\n\t"
      "mul.lo.u32 e2, %6, %8;\n\t"
      "mul.hi.u32 e3, %6, %8;\n\t"
      "mul.lo.u32 o1, %5, %8;\n\t"
      "mul.hi.u32 o2, %5, %8;\n\t"
      "mul.lo.u32 o3, %7, %8;\n\t"
      "mul.hi.u32 o4, %7, %8;\n\t"
      // y1
      "mad.lo.cc.u32 e2, %5, %9, e2;\n\t"
      "madc.hi.cc.u32 e3, %5, %9, e3;\n\t"
      "madc.lo.cc.u32 e4, %7, %9, 0;\n\t"
      "madc.hi.u32 e5, %7, %9, 0;\n\t"
      "mad.lo.cc.u32 o1, %4, %9, o1;\n\t"
      "madc.hi.cc.u32 o2, %4, %9, o2;\n\t"
      "madc.lo.cc.u32 o3, %6, %9, o3;\n\t"
      "madc.hi.cc.u32 o4, %6, %9, o4;\n\t"
      "addc.u32 o5, 0, 0;\n\t"
      // y2
      "mad.lo.cc.u32 e2, %4, %10, e2;\n\t"
      "madc.hi.cc.u32 e3, %4, %10, e3;\n\t"
      "madc.lo.cc.u32 e4, %6, %10, e4;\n\t"
      "madc.hi.cc.u32 e5, %6, %10, e5;\n\t"
      "addc.u32 e6, 0, 0;\n\t"
      "mad.lo.cc.u32 o3, %5, %10, o3;\n\t"
      "madc.hi.cc.u32 o4, %5, %10, o4;\n\t"
      "madc.lo.cc.u32 o5, %7, %10, o5;\n\t"
      "madc.hi.u32 o6, %7, %10, 0;\n\t"
      // y3
      "mad.lo.cc.u32 e4, %5, %11, e4;\n\t"
      "madc.hi.cc.u32 e5, %5, %11, e5;\n\t"
      "madc.lo.cc.u32 e6, %7, %11, e6;\n\t"
      "madc.hi.u32 e7, %7, %11, 0;\n\t"
      "mad.lo.cc.u32 o3, %4, %11, o3;\n\t"
      "madc.hi.cc.u32 o4, %4, %11, o4;\n\t"
      "madc.lo.cc.u32 o5, %6, %11, o5;\n\t"
      "madc.hi.cc.u32 o6, %6, %11, o6;\n\t"
      "addc.u32 o7, 0, 0;\n\t"
      // even + odd: lo = (e0, e1, e2, e3), hi = (e4 .. e7)
      "add.cc.u32 e1, e1, o1;\n\t"
      "addc.cc.u32 e2, e2, o2;\n\t"
      "addc.cc.u32 e3, e3, o3;\n\t"
      "addc.cc.u32 e4, e4, o4;\n\t"
      "addc.cc.u32 e5, e5, o5;\n\t"
      "addc.cc.u32 e6, e6, o6;\n\t"
      "addc.u32 e7, e7, o7;\n\t"
      // lo / 2
      "and.b32 b, e0, 1;\n\t"
      "shl.b32 b, b, 30;\n\t"
      "shf.r.wrap.b32 e0, e0, e1, 1;\n\t"
      "shf.r.wrap.b32 e1, e1, e2, 1;\n\t"
      "shf.r.wrap.b32 e2, e2, e3, 1;\n\t"
      "shr.u32 e3, e3, 1;\n\t"
      "add.u32 e3, e3, b;\n\t"
      // hi + lo / 2, the carry worth 2 (the sum is below 2^128 + 2^127 + 2^126: no second carry)
      "add.cc.u32 e0, e0, e4;\n\t"
      "addc.cc.u32 e1, e1, e5;\n\t"
      "addc.cc.u32 e2, e2, e6;\n\t"
      "addc.cc.u32 e3, e3, e7;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "add.u32 c, c, c;\n\t"
      "add.cc.u32 %0, e0, c;\n\t"
      "addc.cc.u32 %1, e1, 0;\n\t"
      "addc.cc.u32 %2, e2, 0;\n\t"
      "addc.u32 %3, e3, 0;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3])
      : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]));
}

// r = a + b for any a, b below 2^128: the carry's 2 is added, and if that carried in turn the
// sum is 0 and 2 is added once more.
__device__ __forceinline__ void m127_add_lazy(uint32_t (&r)[4], const uint32_t (&a)[4], const uint32_t (&b)[4]) {
  asm("{\n\t.reg .u32 s0, s1, s2, s3, c;\n\t"
      "add.cc.u32 s0, %4, %8;\n\t"
      "addc.cc.u32 s1, %5, %9;\n\t"
      "addc.cc.u32 s2, %6, %10;\n\t"
      "addc.cc.u32 s3, %7, %11;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "add.u32 c, c, c;\n\t"
      "add.cc.u32 s0, s0, c;\n\t"
      "addc.cc.u32 %1, s1, 0;\n\t"
      "addc.cc.u32 %2, s2, 0;\n\t"
      "addc.cc.u32 %3, s3, 0;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "add.u32 c, c, c;\n\t"
      "add.u32 %0, s0, c;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]));
}

// r = a - b for any a, b below 2^128: a borrow is worth -2, and so is the borrow of taking that
// away (the difference was 0 or 1; it becomes 2^128 - 2 or - 1, and 2 less does not borrow).
__device__ __forceinline__ void m127_sub_lazy(uint32_t (&r)[4], const uint32_t (&a)[4], const uint32_t (&b)[4]) {
  asm("{\n\t.reg .u32 s0, s1, s2, s3, c;\n\t"
      "sub.cc.u32 s0, %4, %8;\n\t"
      "subc.cc.u32 s1, %5, %9;\n\t"
      "subc.cc.u32 s2, %6, %10;\n\t"
      "subc.cc.u32 s3, %7, %11;\n\t"
      "subc.u32 c, 0, 0;\n\t"
      "and.b32 c, c, 2;\n\t"
      "sub.cc.u32 s0, s0, c;\n\t"
      "subc.cc.u32 %1, s1, 0;\n\t"
      "subc.cc.u32 %2, s2, 0;\n\t"
      "subc.cc.u32 %3, s3, 0;\n\t"
      "subc.u32 c, 0, 0;\n\t"
      "and.b32 c, c, 2;\n\t"
      "sub.u32 %0, s0, c;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]));
}

// The canonical representative of any a below 2^128: t = (a mod 2^127) + (a >> 127) <= p + 1,
// then t - p when t >= p, which is when t + 1 reaches 2^127.
__device__ __forceinline__ void m127_canon(uint32_t (&r)[4], const uint32_t (&a)[4]) {
  asm("{\n\t.reg .u32 t0, t1, t2, t3, u;\n\t"
      "shr.u32 u, %7, 31;\n\t"
      "and.b32 t3, %7, 0x7fffffff;\n\t"
      "add.cc.u32 t0, %4, u;\n\t"
      "addc.cc.u32 t1, %5, 0;\n\t"
      "addc.cc.u32 t2, %6, 0;\n\t"
      "addc.u32 t3, t3, 0;\n\t"
      "add.cc.u32 u, t0, 1;\n\t"
      "addc.cc.u32 u, t1, 0;\n\t"
      "addc.cc.u32 u, t2, 0;\n\t"
      "addc.u32 u, t3, 0;\n\t"
      "shr.u32 u, u, 31;\n\t"
      "add.cc.u32 %0, t0, u;\n\t"
      "addc.cc.u32 %1, t1, 0;\n\t"
      "addc.cc.u32 %2, t2, 0;\n\t"
      "addc.u32 t3, t3, 0;\n\t"
      "and.b32 %3, t3, 0x7fffffff;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]));
}

}  // namespace sc
