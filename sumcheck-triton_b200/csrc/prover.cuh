// The SumCheck round kernel and its finalisation.
//
// One launch per round j does the whole round, with no host round trip:
//
//   1. fold (j >= 1): each thread reads 4 consecutive entries of every table of round j-1
//      (one 128-bit load per limb plane), folds them with r_{j-1} into the pair
//      (T_j[2i], T_j[2i+1]) and writes that pair back (the fold of the previous round,
//      reference field_sumcheck.cu:677-694, fused into this round's read);
//   2. evaluate: extends every table's pair to t = 0..d - 1 (v(t) = v(t-1) + (o - e); reference
//      field_sumcheck.cu:326-348) and evaluates the constraint at each point
//      (field_sumcheck.cu:389-590) and, in the place of point d, its leading coefficient,
//      accumulating d+1 sums per thread (see eval_pair for the exact-arithmetic shortcuts:
//      factors taken in pairs, g(1) from the claim);
//   3. reduce: the point sums are summed word by word as integers -- over the warp, the block
//      (shared memory) and the grid (64-bit atomic adds) -- with no modular arithmetic until
//      the last block to finish (atomic ticket) reads (d + 1) L integers and reduces them
//      mod p: a single-pass grid reduction in place of the reference's log-depth launch tree
//      (field_sumcheck.cu:635-675, :996-1010);
//   4. finalise (last block only): stores g_j(0..d), adds the round's checksum, derives r_j
//      by SHA3 over the round polynomial on the device (field_sumcheck.cu:857-907), and when
//      needed g_j(r_j) (the next round's claim) and, in the last round, the final claim and
//      the folded values f_k(r).
//
// Tables are limb-planar: table k, limb l is the u32 plane at (k * L + l) * len.
// Kernels are templates over the limb count L, the field kind K (a special reduction for
// Goldilocks) and DMAX, the largest degree the launch handles (register arrays of DMAX + 1
// points; the host picks the smallest class >= the expression's degree).
#pragma once
#include <cstdint>
#include <type_traits>

#include "field.cuh"
#include "keccak.cuh"

namespace sc {

constexpr int kMaxVars = 32;
constexpr int kMaxTerms = 32;
constexpr int kMaxFlat = 128;
constexpr int kMaxRounds = 40;

// Copies of a round's grid-wide integer sums: block (or item) i adds to copy i % kSumCopies, so
// that a few hundred blocks finishing together do not queue on the same addresses; the last
// block adds the copies up. One round at a time uses them.
constexpr int kSumCopies = 16;
__host__ __device__ constexpr size_t sums_bytes(int L) { return sizeof(uint64_t) * kSumCopies * kMaxPoints * L; }
// Shared-memory words of the block reduction's scratch: a 64-bit sum per warp, point and limb.
__host__ __device__ constexpr int reduce_scratch_words(int threads, int L) { return (threads / 32) * kMaxPoints * L * 2; }

enum ChallengeMode : int32_t { kChallengeSha3 = 0, kChallengeFixed = 1, kChallengeExplicit = 2 };

// Coefficient handling per term: +1 / -1 are an add / a subtract; other small values an
// addition chain; anything else a product with the coefficient's Montgomery image. The
// scaling is applied once per pair to the first factor (value and difference), not per point.
enum CoeffKind : uint8_t { kCoeffPlus = 0, kCoeffMinus = 1, kCoeffSmall = 2, kCoeffMont = 3 };

// Constants of one field that only the finalisation needs (device memory, per field).
struct FieldConsts {
  uint32_t p[kMaxLimbs];
  uint32_t np;
  uint32_t limbs;
  uint32_t one[kMaxLimbs];                   // R mod p
  uint32_t r2[kMaxLimbs];                    // R^2 mod p
  uint32_t r3[kMaxLimbs];                    // R^3 mod p
  uint32_t kfold[8][kMaxLimbs];              // 2^(64 + 32 i) mod p (fold tables, field.cuh)
  uint32_t pts[kMaxPoints][kMaxLimbs];       // Montgomery image of t = 0..7
  uint32_t kdig[8][kMaxLimbs];               // R^2 2^(32 i) mod p: digest word i
  uint32_t lag[kMaxPoints][kMaxPoints][kMaxLimbs];  // lag[d][t] = 1 / prod_{s<=d, s!=t} (t - s)
};

// A compiled expression for one field (kernel parameter: lives in the constant bank).
struct ExprDev {
  int32_t num_vars;
  int32_t num_terms;
  int32_t degree;
  int32_t pad;
  uint8_t term_len[kMaxTerms];
  uint8_t term_off[kMaxTerms];
  uint8_t flat[kMaxFlat];
  uint8_t coeff_kind[kMaxTerms];
  int32_t coeff_small[kMaxTerms];
  uint32_t coeff_mont[kMaxTerms][kMaxLimbs];
  int32_t shape;                    // Shape the host matched (kShapeGeneric: none)
  uint8_t role[16];                 // shape kernels: table index of each role
};

// Expression shapes with a compile-time evaluator (the host matches the term structure and
// maps tables to roles; any table order and any order of the symmetric factors matches):
//   kShapeZerocheck  F (X1 S1 + X2 S2 + X1 X2 M - X3 S4 + S5)   roles S1 X1 F S2 X2 M S4 X3 S5
//                    evaluated as F (X1 (S1 + M X2) + S2 X2 - S4 X3 + S5): 5 products a point
//                    (the vanilla zerocheck gate, src/zkduel/workloads.py:37-43)
//   kShapeAbcg       G (A B C + D E)                              roles A B C G D E
//                    4 products a point (poly_abcg_plus_deg, workloads.py:32)
enum Shape : int32_t { kShapeGeneric = 0, kShapeZerocheck = 1, kShapeAbcg = 2 };

__host__ __device__ constexpr int shape_tables(int shape) {
  return shape == kShapeZerocheck ? 9 : (shape == kShapeAbcg ? 6 : 0);
}

// Device-detected errors, or-ed into ProofState::status (the host fails the call with
// SC_ERR_DEVICE when it reads a nonzero status):
//   kStatusClaim  a round that evaluated g(1) directly and was given a claim to meet
//                 (RoundArgs::check_claim) found g_j(0) + g_j(1) != the claim -- the tables
//                 are not the ones the recorded rounds were proved on, or the recorded claim
//                 was altered (a resumed transcript's first round checks this).
constexpr uint32_t kStatusClaim = 1u;

// Per-proof device state, all Montgomery limbs (written by the finalisation).
struct ProofState {
  uint32_t* counter;     // block tickets of the running round, reset to 0 after each round
  uint64_t* checksum;    // sum over rounds and points of (i + 1) limb_i
  uint32_t* polys;       // [n][kMaxPoints][L]
  uint32_t* chals;       // [n][L]
  uint32_t* finals;      // [1 + K][L]: g_{n-1}(r_{n-1}), then f_k(r) for every table
  uint32_t* claim0;      // [L]
  uint32_t* status;      // nonzero on a device-detected error: kStatusClaim
  uint32_t* claim;       // [L]: g_{j-1}(r_{j-1}), the claim round j's g(0) + g(1) must meet
};

struct RoundArgs {
  const uint32_t* src;   // T_{j-1} when folding, else T_j
  uint32_t* dst;         // T_j when folding, else unused
  uint64_t src_len;      // entries per plane of src
  uint64_t pairs;        // N_j / 2
  int32_t round;
  int32_t num_rounds;
  int32_t fold;
  int32_t mode;          // ChallengeMode
  int32_t skip1;         // g(1) = claim - g(0) instead of evaluating point 1
  int32_t want_claim;    // store g_j(r_j) for the next round
  uint64_t* sums;        // the grid's integer sums, [kSumCopies][kMaxPoints * L]: zero before
                         // the round, zero again after it
  const FieldConsts* fc;
  ProofState st;
  uint32_t* ext_out;     // non-null: the round's sums g_j(0..d) go here and the round is not
                         // finalised (one rank of a split proof; the commit finalises it)
  const uint32_t* last;  // non-null: T_{n-1} for the last round's f_k(r) (a tail's, in shared memory)
  int32_t check_claim;   // with skip1 == 0: check g_j(0) + g_j(1) against st.claim (kStatusClaim)
  int32_t pad;
};

// Rounds are queued with programmatic stream serialisation: a round's launch and its blocks'
// start overlap the end of the round before, and pdl_begin waits for that round's results
// (before anything it wrote is read), then lets the next round's launch begin. Without the
// launch attribute both are no-ops.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <int L>
__device__ __forceinline__ Fe<L> ld_fe(const uint32_t* p) {
  Fe<L> r;
#pragma unroll
  for (int i = 0; i < L; ++i) r.w[i] = p[i];
  return r;
}

template <int L>
__device__ __forceinline__ Fe<L> ld_fe_cg(const uint32_t* p) {
  Fe<L> r;
#pragma unroll
  for (int i = 0; i < L; ++i) r.w[i] = __ldcg(p + i);
  return r;
}

template <int L>
__device__ __forceinline__ void st_fe(uint32_t* p, const Fe<L>& a) {
#pragma unroll
  for (int i = 0; i < L; ++i) p[i] = a.w[i];
}

// Shared-memory element of thread `tid` in a [slot][limb][thread] array (conflict-free).
template <int L>
__device__ __forceinline__ Fe<L> sm_get(const uint32_t* sm, int slot, int tid, int nthr) {
  Fe<L> r;
#pragma unroll
  for (int l = 0; l < L; ++l) r.w[l] = sm[(slot * L + l) * nthr + tid];
  return r;
}

template <int L>
__device__ __forceinline__ void sm_put(uint32_t* sm, int slot, int tid, int nthr, const Fe<L>& a) {
#pragma unroll
  for (int l = 0; l < L; ++l) sm[(slot * L + l) * nthr + tid] = a.w[l];
}

template <int L, int K>
__device__ __forceinline__ Fe<L> add_or_sub(const Fe<L>& acc, const Fe<L>& x, bool neg, const FieldParams<L, K>& F) {
  return neg ? fe_sub(acc, x, F) : fe_add(acc, x, F);
}

// The generic evaluator over Goldilocks in lazy arithmetic (field.cuh gl_*): stepped values,
// products and point sums are any representatives in [0, 2^64); the values and differences it
// reads are canonical. A thread's point sums leave it as they are: the round's integer sums are
// reduced mod p once (sums_to_points). Measured on B200, the mixed stream's 64-bit group alone,
// when the sums were still made canonical per thread: 5.93 against 6.07 ms.
#ifndef SC_GOLD_LAZY_GENERIC
#define SC_GOLD_LAZY_GENERIC 1
#endif
template <int L, int K>
__host__ __device__ constexpr bool lazy_generic() {
  return L == 2 && K == kFieldGoldilocks && SC_GOLD_LAZY_GENERIC;
}
template <bool LZ, int L, int K>
__device__ __forceinline__ Fe<L> lz_add(const Fe<L>& a, const Fe<L>& b, const FieldParams<L, K>& F) {
  if constexpr (LZ) return gl_add(a, b, gold_k(F));
  else return fa_add(a, b, F);
}
template <bool LZ, int L, int K>  // b canonical
__device__ __forceinline__ Fe<L> lz_add_c(const Fe<L>& a, const Fe<L>& b, const FieldParams<L, K>& F) {
  if constexpr (LZ) return gl_add_c(a, b, gold_k(F));
  else return fa_add(a, b, F);
}
template <bool LZ, int L, int K>
__device__ __forceinline__ Fe<L> lz_sub(const Fe<L>& a, const Fe<L>& b, const FieldParams<L, K>& F) {
  if constexpr (LZ) return gl_sub(a, b, gold_k(F));
  else return fa_sub(a, b, F);
}
template <bool LZ, int L, int K>
__device__ __forceinline__ Fe<L> lz_mul(const Fe<L>& a, const Fe<L>& b, const FieldParams<L, K>& F) {
  if constexpr (LZ) return gl_mul(a, b, gold_k(F));
  else return fa_mul(a, b, F);
}
template <bool LZ, int L, int K>
__device__ __forceinline__ void lz_mul2(Fe<L>& r0, const Fe<L>& a0, const Fe<L>& b0, Fe<L>& r1, const Fe<L>& a1,
                                        const Fe<L>& b1, const FieldParams<L, K>& F) {
  if constexpr (LZ) {
    const Fe<L> x = gl_mul(a0, b0, gold_k(F));
    r1 = gl_mul(a1, b1, gold_k(F));
    r0 = x;
  } else {
    fa_mul2(r0, a0, b0, r1, a1, b1, F);
  }
}
template <bool LZ, int L, int K>
__device__ __forceinline__ Fe<L> lz_add_or_sub(const Fe<L>& acc, const Fe<L>& x, bool neg, const FieldParams<L, K>& F) {
  return neg ? lz_sub<LZ>(acc, x, F) : lz_add<LZ>(acc, x, F);
}

// One pair: acc[t] += expression at point t, for the finite points t (0..d - 1, or 0 and 1 for
// d = 1; 1 skipped when skip1), and acc[DMAX] += its coefficient of t^d (make_point_weights).
// get(k, e, o) gives table k's values at 0 and 1; add(slot, x, neg) adds to a sum.
//
// A term's factors are taken two at a time where that saves products (more than three points):
// the product of two is a quadratic, known from its values at 0 and 1 and its leading
// coefficient (three products) and stepped from point to point by two additions, so each
// further point costs one product for the two factors instead of two. Six factors at six points take
// 21 products instead of 30, four at four points 10 instead of 12.
template <int L, int K, int DMAX, typename Get, typename Add, typename Prod>
__device__ __forceinline__ void eval_pair(const ExprDev& E, Get get, Add add, Prod& prod, bool skip1,
                                          const FieldParams<L, K>& F) {
  constexpr bool LZ = lazy_generic<L, K>();
  const int d = E.degree;
  const int fin = d >= 2 ? d - 1 : 1;  // last finite point
  for (int i = 0; i < E.num_terms; ++i) {
    const int off = E.term_off[i];
    const int len = E.term_len[i];
    const int kind = E.coeff_kind[i];
    const bool full = len == d && d >= 2;
    const bool paired = fin + 1 - (skip1 ? 1 : 0) + (full ? 1 : 0) > 3;  // points the term is needed at
    const bool neg = kind == kCoeffMinus || (kind == kCoeffSmall && E.coeff_small[i] < 0);
    Fe<L> prod0, lead;
    for (int f = 0; f < len;) {
      // this step's factor, or the product of two: v(0), v(1) - v(0), the step's step, and the
      // leading coefficient
      Fe<L> v, v1;
      get(E.flat[off + f], v, v1);
      if (f == 0) {
        if (kind == kCoeffSmall) {
          const int32_t c = E.coeff_small[i];
          const uint32_t m = c < 0 ? static_cast<uint32_t>(-static_cast<int64_t>(c)) : static_cast<uint32_t>(c);
          v = fe_mul_small(v, m, F);
          v1 = fe_mul_small(v1, m, F);
        } else if (kind == kCoeffMont) {
          Fe<L> cm;
#pragma unroll
          for (int l = 0; l < L; ++l) cm.w[l] = E.coeff_mont[i][l];
          fe_mul2(v, v, cm, v1, v1, cm, F);
        }
      }
      Fe<L> li = fe_sub(v1, v, F), df = li, dd = fe_zero<L>();
      const bool two = paired && f + 1 < len;
      if (two) {
        Fe<L> w, w1;
        get(E.flat[off + f + 1], w, w1);
        li = fa_mul(li, fe_sub(w1, w, F), F);
        fa_mul2(v, v, w, v1, v1, w1, F);
        df = fa_sub(v1, v, F);
        dd = fa_add(li, li, F);
      }
      // products two points at a time: the leading coefficient with point 0, then 1 | 2, 3 | ..
      if (f == 0) {
        if (full) lead = li;
        prod0 = v;
      } else if (full) {
        lz_mul2<LZ>(lead, lead, li, prod0, prod0, v, F);
      } else {
        prod0 = lz_mul<LZ>(prod0, v, F);
      }
      auto step = [&]() {
        v = lz_add_c<LZ>(v, df, F);
        if (two) df = fa_add(df, dd, F);
      };
#pragma unroll
      for (int t = 1; t < DMAX; t += 2) {  // t odd, then t + 1
        if (t > fin) break;
        step();
        const Fe<L> va = v;
        const bool odd = !(skip1 && t == 1), even = t + 1 < DMAX && t + 1 <= fin;
        const int u = t + 1 < DMAX ? t + 1 : t;
        if (even) step();
        if (f == 0) {
          prod.set(t, va);
          if (even) prod.set(u, v);
        } else if (odd && even) {
          Fe<L> x, y;
          lz_mul2<LZ>(x, prod.get(t), va, y, prod.get(u), v, F);
          prod.set(t, x);
          prod.set(u, y);
        } else if (odd) {
          prod.set(t, lz_mul<LZ>(prod.get(t), va, F));
        } else if (even) {
          prod.set(u, lz_mul<LZ>(prod.get(u), v, F));
        }
      }
      f += two ? 2 : 1;
    }
    if (full) add(DMAX, lead, neg);
    add(0, prod0, neg);
#pragma unroll
    for (int t = 1; t < DMAX; ++t) {
      if (t > fin) break;
      if (skip1 && t == 1) continue;
      add(t, prod.get(t), neg);
    }
  }
}

// A term's products at points 1..DMAX - 1: in registers, or in this thread's shared-memory slots.
template <int L, int DMAX>
struct RegProducts {
  Fe<L> a[DMAX];
  __device__ __forceinline__ Fe<L> get(int t) const { return a[t]; }
  __device__ __forceinline__ void set(int t, const Fe<L>& x) { a[t] = x; }
};
template <int L>
struct SmProducts {
  uint32_t* sm;
  int tid, nthr;
  __device__ __forceinline__ Fe<L> get(int t) const { return sm_get<L>(sm, t - 1, tid, nthr); }
  __device__ __forceinline__ void set(int t, const Fe<L>& x) { sm_put<L>(sm, t - 1, tid, nthr, x); }
};

// Where the generic evaluator keeps a pair's tables, a term's products and a thread's point sums.
// Fields of up to 4 limbs stage the tables' values in shared memory and hold products and sums
// in registers. At 8 limbs those are 8 words each: the tables are read from memory at every use
// (T_j from L2, where this thread has just written it) and shared memory takes the products and
// sums instead, which leaves 128 registers and 4 blocks an SM up to degree 4. Measured on B200, 64 mixed
// proofs: 4.84 ms, against 4.99 with the products in registers (3 blocks) and 5.10 with the
// tables staged and both in registers; at 4 limbs 40 served requests took 7.18 ms staged, 7.30
// from memory.
__host__ __device__ constexpr bool streamed_tables(int L) { return L >= 8; }

// Shape kernels hold a pair's tables in role order. shape_value is the formula at one point,
// shape_value2 at two points, their products side by side; value(i) and value2(i) give role
// i's value. shape_ends is point 0 and the leading coefficient (from the tables' differences,
// the term of full degree alone).
template <int L, int K, typename V>
__device__ __forceinline__ Fe<L> shape_value(V v, const FieldParams<L, K>& F, std::integral_constant<int, kShapeZerocheck>) {
  const Fe<L> u = fa_add(v(0), fa_mul(v(5), v(4), F), F);  // S1 + M X2
  Fe<L> s = fa_mul(v(1), u, F);                            // X1 (S1 + M X2)
  s = fa_add(s, fa_mul(v(3), v(4), F), F);                 // + S2 X2
  s = fa_sub(s, fa_mul(v(6), v(7), F), F);                 // - S4 X3
  s = fa_add(s, v(8), F);                                  // + S5
  return fa_mul(v(2), s, F);                               // F (...)
}
template <int L, int K, typename V>
__device__ __forceinline__ Fe<L> shape_value(V v, const FieldParams<L, K>& F, std::integral_constant<int, kShapeAbcg>) {
  Fe<L> ab, de;
  fa_mul2(ab, v(0), v(1), de, v(4), v(5), F);
  return fa_mul(v(3), fa_add(fa_mul(ab, v(2), F), de, F), F);
}
template <int L, int K, typename V, typename W>
__device__ __forceinline__ void shape_value2(V v, W w, Fe<L>& x, Fe<L>& y, const FieldParams<L, K>& F,
                                             std::integral_constant<int, kShapeZerocheck> shape) {
  x = shape_value<L, K>(v, F, shape);
  y = shape_value<L, K>(w, F, shape);
}
template <int L, int K, typename V, typename W>
__device__ __forceinline__ void shape_value2(V v, W w, Fe<L>& x, Fe<L>& y, const FieldParams<L, K>& F,
                                             std::integral_constant<int, kShapeAbcg>) {
  Fe<L> p, q;
  fa_mul2(x, v(0), v(1), y, w(0), w(1), F);
  fa_mul2(x, x, v(2), y, y, w(2), F);
  fa_mul2(p, v(4), v(5), q, w(4), w(5), F);
  x = fa_add(x, p, F);
  y = fa_add(y, q, F);
  fa_mul2(x, x, v(3), y, y, w(3), F);
}
template <int L, int K, typename V, typename D>
__device__ __forceinline__ void shape_ends(V v, D d, Fe<L>& x, Fe<L>& lead, const FieldParams<L, K>& F,
                                           std::integral_constant<int, kShapeZerocheck> shape) {
  x = shape_value<L, K>(v, F, shape);
  lead = fa_mul(fa_mul(d(2), d(1), F), fa_mul(d(4), d(5), F), F);  // F X1 X2 M
}
template <int L, int K, typename V, typename D>
__device__ __forceinline__ void shape_ends(V v, D d, Fe<L>& x, Fe<L>& lead, const FieldParams<L, K>& F,
                                           std::integral_constant<int, kShapeAbcg>) {
  fa_mul2(x, v(0), v(1), lead, d(0), d(1), F);
  fa_mul2(x, x, v(2), lead, lead, d(2), F);
  x = fa_add(x, fa_mul(v(4), v(5), F), F);
  fa_mul2(x, x, v(3), lead, lead, d(3), F);  // G (A B C + D E); A B C G
}

// The same formulas in lazy Goldilocks arithmetic, added to a point's sum unreduced
// (field_gold_acc.cuh): one reduction for the bracket, none for its product with the last factor.
// The zerocheck's role 6 (S4) comes negated, so that its product is added.
struct GoldSum {
  uint32_t w[5];
};
__device__ __forceinline__ void shape_add(GoldSum& acc, const Fe<2> (&v)[9], const GoldK k,
                                          std::integral_constant<int, kShapeZerocheck>) {
  uint32_t t[5];
  Fe<2> u, s;
  gold_acc_first(t, v[5].w, v[4].w);  // M X2 + S1
  gold_acc_add(t, t, v[0].w);
  gold_acc_reduce(u.w, t, k);
  gold_acc_first(t, v[1].w, u.w);     // X1 (S1 + M X2) + S2 X2 - S4 X3 + S5
  gold_acc_mul(t, t, v[3].w, v[4].w);
  gold_acc_mul(t, t, v[6].w, v[7].w);
  gold_acc_add(t, t, v[8].w);
  gold_acc_reduce(s.w, t, k);
  gold_acc_mul(acc.w, acc.w, v[2].w, s.w);
}
__device__ __forceinline__ void shape_add(GoldSum& acc, const Fe<2> (&v)[6], const GoldK k,
                                          std::integral_constant<int, kShapeAbcg>) {
  uint32_t t[5];
  Fe<2> s;
  gold_acc_first(t, gl_mul(v[0], v[1], k).w, v[2].w);
  gold_acc_mul(t, t, v[4].w, v[5].w);
  gold_acc_reduce(s.w, t, k);
  gold_acc_mul(acc.w, acc.w, v[3].w, s.w);
}
__device__ __forceinline__ void shape_add_lead(GoldSum& acc, const Fe<2> (&d)[9], const GoldK k,
                                               std::integral_constant<int, kShapeZerocheck>) {
  gold_acc_mul(acc.w, acc.w, gl_mul(d[2], d[1], k).w, gl_mul(d[4], d[5], k).w);
}
__device__ __forceinline__ void shape_add_lead(GoldSum& acc, const Fe<2> (&d)[6], const GoldK k,
                                               std::integral_constant<int, kShapeAbcg>) {
  gold_acc_mul(acc.w, acc.w, gl_mul(d[0], d[1], k).w, gl_mul(d[2], d[3], k).w);
}

// 2-limb Goldilocks shape kernels evaluate their points in lazy arithmetic: the point steps
// add a canonical difference (six ALU instructions, no compare or select), the formula's
// products are summed unreduced, and the point sums are reduced once, after the thread's last
// pair. Folds, stored tables and differences stay canonical. Measured on B200, zerocheck gate
// n = 24: canonical sums 1.65 ms, lazy sums 1.60 ms (both a product reduced at a time, before
// the leading coefficient took the last point); with reduced products 1.27 ms, with products
// summed unreduced 1.18 ms.
#ifndef SC_GOLD_LAZY
#define SC_GOLD_LAZY 1
#endif

// Folds (if fold) and evaluates pairs q = first, first + stride, ... < last, adding the
// point sums into acc. Generic, up to 4 limbs: every table's values at 0 and 1 go to this
// block's [K][L][nthr] shared arrays sv / sd for eval_pair; at 8 limbs the tables are read from
// memory at every use and sv holds the point sums and products (streamed_tables). Shape kernels
// keep values and differences in registers (tables read in role order) and evaluate the shape's
// compile-time formula at each point.
// 2-limb shape kernels issue every load of a pair before its folds and run 2 blocks/SM
// (<= 128 registers for the loaded words): measured on B200, Goldilocks n = 24 went from
// 2.18 ms (loads interleaved with folds, 3 blocks/SM) to 2.01 ms.
#ifndef SC_EARLY_LOADS
#define SC_EARLY_LOADS 1
#endif

// 2-limb Goldilocks shape kernels copy each thread's next pair into shared memory with
// asynchronous copies (cp.async) while the current pair is evaluated, so its loads are in
// flight during the arithmetic instead of before it. One stage per thread, laid out
// [table][limb][thread] (16-byte entries in fold rounds, 8-byte in round 0) after the block
// reduction's scratch; the next pair's copies are issued only after every value of the
// current stage has been consumed by an arithmetic instruction, and each thread waits for its
// own copies alone (cp.async.wait_group), so no block barrier is involved.
#ifndef SC_GOLD_ASYNC
#define SC_GOLD_ASYNC 1
#endif
// The same stage for the 8-limb g(abc + de) shape kernel (96 KB a block of 128 threads, 2 blocks
// an SM) measured slower on B200: plain BLS n = 22 3.37 against 3.25 ms (255 registers with 120
// bytes of spills, against none).
__host__ __device__ constexpr bool shape_async_stage(int L, int K, int shape) {
  return SC_GOLD_ASYNC && L == 2 && K == kFieldGoldilocks && shape != kShapeGeneric && SC_GOLD_SHAPE_FMA &&
         SC_GOLD_LAZY;
}
// Dynamic shared memory (bytes) of a compile-time shape round kernel of `threads` threads.
__host__ __device__ constexpr size_t shape_round_smem_bytes(int L, int K, int shape, int threads) {
  return 4 * (static_cast<size_t>(reduce_scratch_words(threads, L)) +
              (shape_async_stage(L, K, shape) ? static_cast<size_t>(threads) * shape_tables(shape) * L * 4 : 0));
}
__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* gmem_src) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_8(void* smem_dst, const void* gmem_src) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }
#ifndef SC_PAIR_UNROLL
#define SC_PAIR_UNROLL 1
#endif
constexpr int kPairUnroll = SC_PAIR_UNROLL;
template <int L, int K, int DMAX, int SHAPE = kShapeGeneric>
__device__ __forceinline__ void process_pairs(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst,
                                              uint64_t src_len, bool fold,
                                              const Fe<L>& r_prev, const ExprDev& E, uint32_t* sv, uint32_t* sd,
                                              uint64_t first, uint64_t last, uint64_t stride, bool skip1,
                                              Fe<L> (&acc)[DMAX + 1], const FieldParams<L, K>& F,
                                              const uint32_t* fold_table = nullptr) {
  if constexpr (SHAPE != kShapeGeneric && L == 2 && K == kFieldGoldilocks && SC_GOLD_SHAPE_FMA) {
    // the shape kernels' folds and points with every Goldilocks carry on the FMA pipe
    FieldParams<2, kFieldGoldilocksFma> G;
    G.p[0] = F.p[0];
    G.p[1] = F.p[1];
    G.np = F.np;
    process_pairs<L, kFieldGoldilocksFma, DMAX, SHAPE>(src, dst, src_len, fold, r_prev, E, sv, sd, first, last, stride,
                                                        skip1, acc, G);
    return;
  }
  const int tid = threadIdx.x, nthr = blockDim.x;
  constexpr bool kStream = SHAPE == kShapeGeneric && streamed_tables(L);
  if constexpr (kStream) {
#pragma unroll
    for (int t = 0; t <= DMAX; ++t) sm_put<L>(sv, t, tid, nthr, fe_zero<L>());
  }
  GoldSum gsum[DMAX + 1];  // the lazy Goldilocks shapes' point sums
#pragma unroll
  for (int t = 0; t <= DMAX; ++t)
#pragma unroll
    for (int i = 0; i < 5; ++i) gsum[t].w[i] = 0;
  constexpr int NR = SHAPE == kShapeGeneric ? 1 : shape_tables(SHAPE);
  constexpr bool kGoldLazy = SHAPE != kShapeGeneric && L == 2 && K == kFieldGoldilocksFma && SC_GOLD_LAZY;
  constexpr bool kAsync = kGoldLazy && SC_GOLD_ASYNC;
  const int nv = SHAPE == kShapeGeneric ? E.num_vars : NR;
  // kAsync: this thread's stage, after the block reduction's scratch (16-byte aligned)
  uint32_t* const stage = sv + reduce_scratch_words(nthr, L);
  auto issue = [&](uint64_t qn) {  // copies of pair qn into the stage
#pragma unroll
    for (int i = 0; i < NR; ++i)
#pragma unroll
      for (int l = 0; l < L; ++l) {
        const uint32_t* plane = src + (static_cast<uint64_t>(E.role[i]) * L + l) * src_len;
        const int slot = (i * L + l) * nthr + tid;
        if (fold)
          cp_async_16(reinterpret_cast<uint4*>(stage) + slot, reinterpret_cast<const uint4*>(plane) + qn);
        else
          cp_async_8(reinterpret_cast<uint2*>(stage) + slot, reinterpret_cast<const uint2*>(plane) + qn);
      }
    cp_async_commit();
  };
  if constexpr (kAsync) {
    if (first < last) issue(first);
  }
#pragma unroll(SHAPE == kShapeGeneric ? 1 : kPairUnroll)
  for (uint64_t q = first; q < last; q += stride) {
    Fe<L> sh_v[NR], sh_d[NR];
    if constexpr (kAsync) {
      cp_async_wait_all();  // this pair's copies (this thread's own) have landed
      if (fold) {
        const uint64_t dst_len = src_len >> 1;
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          Fe<L> x0, x1, x2, x3;
#pragma unroll
          for (int l = 0; l < L; ++l) {
            const uint4 v = reinterpret_cast<const uint4*>(stage)[(i * L + l) * nthr + tid];
            x0.w[l] = v.x; x1.w[l] = v.y; x2.w[l] = v.z; x3.w[l] = v.w;
          }
          Fe<L> e, o;
          fe_fold2(e, o, x0, x1, x2, x3, r_prev, F);
#pragma unroll
          for (int l = 0; l < L; ++l)
            reinterpret_cast<uint2*>(dst + (static_cast<uint64_t>(E.role[i]) * L + l) * dst_len)[q] = make_uint2(e.w[l], o.w[l]);
          sh_v[i] = e;
          sh_d[i] = o;
        }
        // every value of the stage has been consumed by the folds: the next pair may land
        if (q + stride < last) issue(q + stride);
      } else {
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
          for (int l = 0; l < L; ++l) {
            const uint2 v = reinterpret_cast<const uint2*>(stage)[(i * L + l) * nthr + tid];
            sh_v[i].w[l] = v.x;
            sh_d[i].w[l] = v.y;
          }
        // the next pair is issued after the differences below, which consume every value
      }
    } else
#if SC_EARLY_LOADS
    if constexpr (SHAPE != kShapeGeneric && L <= 2) {
      // every load of the pair first (one 16- or 8-byte load per table and limb plane), then
      // the folds: the loads of a pair are all in flight together
      if (fold) {
        uint4 raw[NR][L];
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
          for (int l = 0; l < L; ++l)
            raw[i][l] = __ldcs(reinterpret_cast<const uint4*>(src + (static_cast<uint64_t>(E.role[i]) * L + l) * src_len) + q);
        const uint64_t dst_len = src_len >> 1;
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          Fe<L> x0, x1, x2, x3;
#pragma unroll
          for (int l = 0; l < L; ++l) {
            x0.w[l] = raw[i][l].x; x1.w[l] = raw[i][l].y; x2.w[l] = raw[i][l].z; x3.w[l] = raw[i][l].w;
          }
          Fe<L> e, o;
          fe_fold2(e, o, x0, x1, x2, x3, r_prev, F);
#pragma unroll
          for (int l = 0; l < L; ++l)
            reinterpret_cast<uint2*>(dst + (static_cast<uint64_t>(E.role[i]) * L + l) * dst_len)[q] = make_uint2(e.w[l], o.w[l]);
          sh_v[i] = e;
          sh_d[i] = o;
        }
      } else {
        uint2 raw[NR][L];
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
          for (int l = 0; l < L; ++l)
            raw[i][l] = __ldcs(reinterpret_cast<const uint2*>(src + (static_cast<uint64_t>(E.role[i]) * L + l) * src_len) + q);
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
          for (int l = 0; l < L; ++l) {
            sh_v[i].w[l] = raw[i][l].x;
            sh_d[i].w[l] = raw[i][l].y;
          }
      }
    } else
#endif
#pragma unroll (SHAPE == kShapeGeneric ? 1 : NR)
    for (int i = 0; i < (kStream && !fold ? 0 : nv); ++i) {
      const int k = SHAPE == kShapeGeneric ? i : E.role[i];
      Fe<L> e, o;
      if (fold) {
        Fe<L> x0, x1, x2, x3;
#pragma unroll
        for (int l = 0; l < L; ++l) {
          const uint4 v = __ldcs(reinterpret_cast<const uint4*>(src + (static_cast<uint64_t>(k) * L + l) * src_len) + q);
          x0.w[l] = v.x; x1.w[l] = v.y; x2.w[l] = v.z; x3.w[l] = v.w;
        }
        fe_fold2(e, o, x0, x1, x2, x3, r_prev, F, fold_table);
        const uint64_t dst_len = src_len >> 1;
#pragma unroll
        for (int l = 0; l < L; ++l)
          reinterpret_cast<uint2*>(dst + (static_cast<uint64_t>(k) * L + l) * dst_len)[q] = make_uint2(e.w[l], o.w[l]);
      } else {
#pragma unroll
        for (int l = 0; l < L; ++l) {
          const uint2 v = __ldcs(reinterpret_cast<const uint2*>(src + (static_cast<uint64_t>(k) * L + l) * src_len) + q);
          e.w[l] = v.x; o.w[l] = v.y;
        }
      }
      if constexpr (SHAPE == kShapeGeneric) {
        if constexpr (!kStream) {
          sm_put<L>(sv, k, tid, nthr, e);
          sm_put<L>(sd, k, tid, nthr, o);
        }
      } else {
        sh_v[i] = e;
        sh_d[i] = o;  // o for now: the difference is formed below
      }
    }
    if constexpr (kStream) {
      SmProducts<L> products{sv + (DMAX + 1) * L * nthr, tid, nthr};
      const uint32_t* const tab = fold ? dst : src;
      const uint64_t len = fold ? src_len >> 1 : src_len;
      eval_pair<L, K, DMAX>(
          E,
          [&](int k, Fe<L>& e, Fe<L>& o) {
#pragma unroll
            for (int l = 0; l < L; ++l) {
              const uint2 w = reinterpret_cast<const uint2*>(tab + (static_cast<uint64_t>(k) * L + l) * len)[q];
              e.w[l] = w.x;
              o.w[l] = w.y;
            }
          },
          [&](int t, const Fe<L>& x, bool neg) {
            sm_put<L>(sv, t, tid, nthr, add_or_sub(sm_get<L>(sv, t, tid, nthr), x, neg, F));
          },
          products, skip1, F);
    } else if constexpr (SHAPE == kShapeGeneric) {
      RegProducts<L, DMAX> products;
      eval_pair<L, K, DMAX>(
          E,
          [&](int k, Fe<L>& e, Fe<L>& o) {
            e = sm_get<L>(sv, k, tid, nthr);
            o = sm_get<L>(sd, k, tid, nthr);
          },
          [&](int t, const Fe<L>& x, bool neg) { acc[t] = lz_add_or_sub<lazy_generic<L, K>()>(acc[t], x, neg, F); },
          products, skip1, F);
    } else if constexpr (kGoldLazy) {
      // as below, in lazy arithmetic: sh_v / sh_d arrive canonical, the differences are
      // canonical, the stepped values and the point sums are any representatives
      constexpr int D = 4;
      static_assert(DMAX == D, "shape kernels evaluate degree-4 shapes");
      const GoldK gk = gold_k(F);
      const std::integral_constant<int, SHAPE> shape{};
      if constexpr (SHAPE == kShapeZerocheck) {
        gold_neg(sh_v[6].w, sh_v[6].w, gk);
        gold_neg(sh_d[6].w, sh_d[6].w, gk);
      }
      shape_add(gsum[0], sh_v, gk, shape);
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const Fe<L> o = sh_d[r];
        sh_d[r] = fe_sub(o, sh_v[r], F);
        sh_v[r] = o;
      }
      if constexpr (kAsync) {
        if (!fold && q + stride < last) issue(q + stride);
      }
      shape_add_lead(gsum[D], sh_d, gk, shape);
      if (!skip1) shape_add(gsum[1], sh_v, gk, shape);
#pragma unroll
      for (int t = 2; t < D; ++t) {
#pragma unroll
        for (int r = 0; r < NR; ++r) sh_v[r] = gl_add_c(sh_v[r], sh_d[r], gk);
        shape_add(gsum[t], sh_v, gk, shape);
      }
    } else {
      // sh_v: the values at 0, sh_d: at 1; then the values at 1 and the differences
      static_assert(DMAX == 4, "shape kernels evaluate degree-4 shapes");
      const std::integral_constant<int, SHAPE> shape{};
      Fe<L> x, y;
      shape_ends<L, K>([&](int i) { return sh_v[i]; }, [&](int i) { return fe_sub(sh_d[i], sh_v[i], F); }, x, y, F, shape);
      acc[0] = fa_add(acc[0], x, F);
      acc[4] = fa_add(acc[4], y, F);
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const Fe<L> o = sh_d[r];
        sh_d[r] = fe_sub(o, sh_v[r], F);
        sh_v[r] = o;
      }
      if (!skip1) acc[1] = fa_add(acc[1], shape_value<L, K>([&](int i) { return sh_v[i]; }, F, shape), F);
      shape_value2<L, K>([&](int i) { return fa_add(sh_v[i], sh_d[i], F); },
                         [&](int i) { return fa_add(fa_add(sh_v[i], sh_d[i], F), sh_d[i], F); }, x, y, F, shape);
      acc[2] = fa_add(acc[2], x, F);
      acc[3] = fa_add(acc[3], y, F);
    }
  }
  if constexpr (kGoldLazy) {
#pragma unroll
    for (int t = 0; t <= DMAX; ++t) gold_acc_reduce(acc[t].w, gsum[t].w, gold_k(F));
  }
  if constexpr (kStream) {
#pragma unroll
    for (int t = 0; t <= DMAX; ++t) acc[t] = sm_get<L>(sv, t, tid, nthr);
  }
  if constexpr (SHAPE == kShapeGeneric) {  // the leading coefficient belongs in slot d
    const int d = E.degree;
#pragma unroll
    for (int t = 2; t < DMAX; ++t)
      if (t == d) acc[t] = acc[DMAX];
  }
}

template <int L>
__device__ __forceinline__ Fe<L> fc_get(const uint32_t* row) {
  return ld_fe<L>(row);
}

// The fold table of r into shared memory (field_bls_fold.cuh); every thread of the block calls.
template <int L, int K>
__device__ __forceinline__ void make_fold_table(const FieldConsts& fc, const Fe<L>& r, const FieldParams<L, K>& F,
                                                uint32_t* table) {
  if (threadIdx.x < 8) st_fe<L>(table + threadIdx.x * L, fe_mul(r, fc_get<L>(fc.kfold[threadIdx.x]), F));
  __syncthreads();
}

// ---- reduction
//
// Point sums are added word by word as integers: a 32-bit word splits into 16-bit halves whose
// warp sums (redux) cannot overflow, and every wider sum is 64 bits. Nothing is reduced mod p
// before the whole round's sum is known, so any representative of a residue may be summed and
// no modular additions run in the tail of a round. Measured on B200 (clocks of one block): the
// shuffle tree of modular additions it replaces took 3.3k at 2 limbs and degree 4, 6.7k at 8
// limbs and degree 4, 17k at 8 limbs and degree 7, and ran twice a round with a loop over the
// blocks' partials in between (6.3k / 10.9k).

// Shared memory of a round's end. msg is the hash message preceded by three zero bytes, so that
// its 21-byte domain string ends on a word and j and the words of g_j follow aligned: message
// word q is the funnel shift of msg[q] and msg[q + 1].
constexpr int kMsgG = 7;  // msg[0..5] the domain string, msg[6] = j, msg[7..] the words of g_j
template <int L>
struct RoundEnd {
  static constexpr int kMsgWords = 34 * ((25 + 4 * kMaxPoints * L) / 136 + 1) + 1;
  uint64_t s[kMaxPoints * L];             // the round's integer sums
  int64_t slot[kMaxPoints * (L + 1)];     // their words
  uint32_t half[kMaxPoints * L * 2];      // a block's sums as 16-bit halves (tail.cuh)
  uint32_t msg[kMsgWords];
  uint32_t r[L];                          // r_j
  __align__(8) uint32_t dig[8];
  int is_last;
  __device__ uint64_t half_sum(int i) const { return half[2 * i] + (static_cast<uint64_t>(half[2 * i + 1]) << 16); }
  __device__ uint32_t* g() { return msg + kMsgG; }  // g_j(t): words g()[t L + l]
};

// This warp's integer sums of acc[0..d] into its row of scratch.
template <int L, int N>
__device__ __forceinline__ void warp_sums(const Fe<L> (&acc)[N], int d, uint32_t* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t* row = reinterpret_cast<uint64_t*>(scratch) + warp * kMaxPoints * L;
  constexpr int NV = (N * L + 31) / 32;
  uint64_t mine[NV];  // lane i keeps the sums of words i, i + 32, ...
#pragma unroll
  for (int v = 0; v < NV; ++v) mine[v] = 0;
#pragma unroll
  for (int t = 0; t < N; ++t) {
    if (t > d) break;
#pragma unroll
    for (int l = 0; l < L; ++l) {
      const uint32_t lo = __reduce_add_sync(0xffffffffu, acc[t].w[l] & 0xffffu);
      const uint32_t hi = __reduce_add_sync(0xffffffffu, acc[t].w[l] >> 16);
      if (lane == (t * L + l) % 32) mine[(t * L + l) / 32] = lo + (static_cast<uint64_t>(hi) << 16);
    }
  }
#pragma unroll
  for (int v = 0; v < NV; ++v)
    if (v * 32 + lane < N * L) row[v * 32 + lane] = mine[v];
}

// After warp_sums and a barrier: the block's sums, into s_sm (alone: the block is the whole
// round) or added to copy `copy` of the round's sums.
template <int L>
__device__ __forceinline__ void block_sums(const uint32_t* scratch, int d, bool alone, uint64_t* s_sm, uint64_t* sums,
                                           uint32_t copy) {
  const int nwarps = blockDim.x >> 5;
  const uint64_t* rows = reinterpret_cast<const uint64_t*>(scratch);
  for (int i = threadIdx.x; i < (d + 1) * L; i += blockDim.x) {
    uint64_t s = 0;
    for (int w = 0; w < nwarps; ++w) s += rows[w * kMaxPoints * L + i];
    if (alone)
      s_sm[i] = s;
    else
      atomicAdd(reinterpret_cast<unsigned long long*>(sums + (copy % kSumCopies) * kMaxPoints * L + i),
                static_cast<unsigned long long>(s));
  }
}

// Block-wide, after the block added its sums (or, alone, put them into end.s): true in the block
// that completes the round (its `parts`-th block or item), with the round's integer sums in
// end.s; every thread calls. Ends with a barrier.
template <int L>
__device__ __forceinline__ bool grid_end(int d, uint32_t parts, uint64_t* sums, uint32_t* counter, RoundEnd<L>& end) {
  if (parts > 1) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) end.is_last = atomicAdd(counter, 1u) == parts - 1;
    __syncthreads();
    if (!end.is_last) return false;
    __threadfence();
    for (int i = threadIdx.x; i < (d + 1) * L; i += blockDim.x) {
      uint64_t v[kSumCopies], s = 0;
#pragma unroll
      for (int c = 0; c < kSumCopies; ++c) v[c] = c < static_cast<int>(parts) ? __ldcg(sums + c * kMaxPoints * L + i) : 0;
#pragma unroll
      for (int c = 0; c < kSumCopies; ++c) {
        s += v[c];
        if (c < static_cast<int>(parts)) sums[c * kMaxPoints * L + i] = 0;
      }
      end.s[i] = s;
    }
    if (threadIdx.x == 0) *counter = 0;
  }
  __syncthreads();
  return true;
}
// After warp_sums: the block's sums to the round's, then grid_end.
template <int L>
__device__ __forceinline__ bool grid_sums(const uint32_t* scratch, int d, uint32_t part, uint32_t parts, uint64_t* sums,
                                          uint32_t* counter, RoundEnd<L>& end) {
  __syncthreads();
  block_sums<L>(scratch, d, parts == 1, end.s, sums, part);
  return grid_end<L>(d, parts, sums, counter, end);
}


// a b R^-1 mod p, fully reduced, for a < p and any b < 2^(32 L).
template <int L, int K>
__device__ __forceinline__ Fe<L> fe_mul_any(const Fe<L>& a, Fe<L> b, const FieldParams<L, K>& F) {
  if constexpr (K == kFieldGoldilocks && L == 2) {
    Fe<2> r;
    gold_mul(r.w, a.w, b.w);  // h < p and b' < p below, whatever b is
    return r;
  } else {
    return fe_mul(a, b, F);  // the rows scan b's words against a: t < a + p throughout; or any operands
  }
}

// The evaluators' points. For degree d >= 2 they evaluate 0, 1, .. d - 1 (1 is left out when
// g(1) comes from the claim) and, in the place of point d, the leading coefficient: every factor's
// value at "infinity" is its difference o - e, so that point needs no stepping and only the
// terms of full degree. The d-th finite difference of a polynomial of degree d is d! times
// its leading coefficient, so g(d) = d! lead - sum_{s < d} (-1)^(d - s) C(d, s) g(s): integer
// weights, applied once a round to the integer sums. Degree 1 evaluates 0 and 1.
struct PointWeights {
  int32_t w[kMaxPoints][kMaxPoints];  // [d][s]: weight of slot s in g(d)
};
constexpr PointWeights make_point_weights() {
  PointWeights P{};
  for (int d = 1; d < kMaxPoints; ++d) {
    int64_t binom = 1, fact = 1;
    for (int s = 0; s < d; ++s) {
      P.w[d][s] = static_cast<int32_t>((d - s) % 2 ? binom : -binom);
      binom = binom * (d - s) / (s + 1);
      fact *= s + 1;
    }
    P.w[d][d] = static_cast<int32_t>(fact);
  }
  P.w[1][0] = 0;  // degree 1: point 1 itself
  return P;
}
static __constant__ PointWeights kPointWeights = make_point_weights();

// Field constants of a round's end, by lane of warp 0 (they depend on nothing else, so a block
// that proves several rounds loads them once).
template <int L>
struct EndConsts {
  Fe<L> con;  // sums_to_points
  Fe<L> dig;  // lanes 0..8 / L - 1: the digest's weights
};
template <int L>
__device__ __forceinline__ EndConsts<L> load_end_consts(const FieldConsts& fc) {
  const int lane = threadIdx.x & 31, part = lane >> 3;
  EndConsts<L> c;
  c.con = fc_get<L>(part == 0 ? fc.one : (part == 1 ? fc.r2 : fc.r3));
  c.dig = lane < 8 / L ? fc_get<L>(fc.kdig[lane * L]) : fe_zero<L>();
  return c;
}

// The round's integer sums (sum(t L + l)) to g_j, into end.g() (warp 0). `claim`, when not null,
// stands in for point 1: g(1) = claim - g(0). Lane t < 8 turns its slot's sums into words; lane
// t then forms g(t) as an integer (point d: the weighted sum of the slots; L words and a signed
// rest) and the rest's words times R^2 (and R^3 at one limb) and the low words times `one` are
// one product each, in lanes t, 8 + t and 16 + t.
template <int L, int K, typename Sum>
__device__ __forceinline__ void sums_to_points(Sum sum, int d, const uint32_t* claim, bool skip1, const Fe<L>& con,
                                               const FieldParams<L, K>& F, RoundEnd<L>& end) {
  int64_t* const slot_sm = end.slot;
  const int lane = threadIdx.x & 31, t = lane & 7, part = lane >> 3;
  Fe<L> cl = fe_zero<L>();
  if (claim && lane == 1) cl = ld_fe_cg<L>(claim);
  if (lane <= d && !(skip1 && lane == 1)) {
    uint64_t c = 0;
#pragma unroll
    for (int l = 0; l < L; ++l) {
      c += sum(lane * L + l);
      slot_sm[lane * (L + 1) + l] = static_cast<int64_t>(c & 0xffffffffu);
      c >>= 32;
    }
    slot_sm[lane * (L + 1) + L] = static_cast<int64_t>(c);
  }
  __syncwarp();
  if (skip1 && lane == 1) {  // claim - g(0); the claim alone is missing from one rank's share
#pragma unroll
    for (int l = 0; l <= L; ++l) slot_sm[(L + 1) + l] = (l < L ? static_cast<int64_t>(cl.w[l < L ? l : 0]) : 0) - slot_sm[l];
  }
  __syncwarp();
  Fe<L> v = fe_zero<L>();
  bool neg = false;
  if (t <= d && part < (L == 1 ? 3 : 2)) {
    int64_t a[L + 1];
#pragma unroll
    for (int l = 0; l <= L; ++l) a[l] = t < d ? slot_sm[t * (L + 1) + l] : 0;
    if (t == d)
      for (int s = 0; s <= d; ++s) {
        const int64_t w = kPointWeights.w[d][s];
#pragma unroll
        for (int l = 0; l <= L; ++l) a[l] += w * slot_sm[s * (L + 1) + l];
      }
    int64_t c = 0;
#pragma unroll
    for (int l = 0; l < L; ++l) {
      c += a[l];
      v.w[l] = static_cast<uint32_t>(c);
      c >>= 32;
    }
    int64_t hi = c + a[L];
    neg = hi < 0;
    if (neg) {  // the absolute value; the sign is applied at the end
      uint64_t k = 1;
#pragma unroll
      for (int l = 0; l < L; ++l) {
        k += static_cast<uint32_t>(~v.w[l]);
        v.w[l] = static_cast<uint32_t>(k);
        k >>= 32;
      }
      hi = static_cast<int64_t>(~static_cast<uint64_t>(hi) + k);
    }
    if (part) {
      v = fe_zero<L>();
      const uint64_t h = static_cast<uint64_t>(hi);
      if constexpr (L == 1) {
        v.w[0] = static_cast<uint32_t>(part == 1 ? h : h >> 32);
      } else {
        v.w[0] = static_cast<uint32_t>(h);
        v.w[1] = static_cast<uint32_t>(h >> 32);
      }
    }
  }
  Fe<L> x = fe_mul_any(con, v, F);
  if constexpr (L == 1) x = fe_add(x, fe_shfl_down(x, 16), F);
  Fe<L> g = fe_add(x, fe_shfl_down(x, 8), F);
  if (neg) g = fe_sub(fe_zero<L>(), g, F);
  if (lane <= d) st_fe<L>(end.g() + lane * L, g);
  __syncwarp();
}

// The transcript's 21-byte domain string behind three zero bytes, as little-endian words.
struct TranscriptDomain {
  uint32_t w[6];
};
constexpr TranscriptDomain make_transcript_domain() {
  const char dom[] = "zkduel:field-sweep:v1";
  TranscriptDomain t{};
  for (int i = 0; i < 21; ++i)
    t.w[(i + 3) / 4] |= static_cast<uint32_t>(static_cast<unsigned char>(dom[i])) << (8 * ((i + 3) % 4));
  return t;
}
static __constant__ TranscriptDomain kTranscriptDomain = make_transcript_domain();

// The parts of round j's hash message that are known before g_j (threads first, first + step, ..).
template <int L>
__device__ __forceinline__ void begin_message(RoundEnd<L>& end, int d, int j, int first, int step) {
  const int past = kMsgG + (d + 1) * L;  // the word after g_j: the padding's first byte
  for (int i = first; i < RoundEnd<L>::kMsgWords; i += step)
    if (i < kMsgG || i >= past)
      end.msg[i] = i < 6 ? kTranscriptDomain.w[i] : (i == 6 ? static_cast<uint32_t>(j) : (i == past ? 6u : 0u));
}

// The end of round j, with g_j complete in end.g() and begin_message done; every thread of the
// block calls, after a barrier. Warp 0 checks the claim, derives r_j (into end.r too, for a caller
// that goes on with the next round in this block, after a barrier of its own) and writes the next
// claim; the next warp, if there is one, stores the round polynomial, the checksum and the claim
// of round 0 meanwhile.
template <int L, int K>
__device__ __forceinline__ void finalize_round(const RoundArgs& A, const ExprDev& E, const FieldParams<L, K>& F,
                                               const EndConsts<L>& consts, RoundEnd<L>& end) {
  const uint32_t* const g_sm = end.g();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d = E.degree;
  const int j = A.round;
  const FieldConsts& fc = *A.fc;
  if (warp == (blockDim.x > 32 ? 1 : 0)) {
    // round polynomial, checksum, the first round's claim
    uint64_t cs = 0;
    for (int i = lane; i < (d + 1) * L; i += 32) {
      const uint32_t w = g_sm[i];
      A.st.polys[(j * kMaxPoints + i / L) * L + i % L] = w;
      cs += static_cast<uint64_t>(i % L + 1) * w;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) cs += __shfl_down_sync(0xffffffffu, cs, off);
    if (lane == 0) {
      *A.st.checksum += cs;
      if (j == 0) st_fe<L>(A.st.claim0, fe_add(ld_fe<L>(g_sm), ld_fe<L>(g_sm + L), F));
    }
  }
  if (warp != 0) return;
  if (A.check_claim && !A.skip1) {  // by the warp that writes the next claim below, and before it does
    if (lane == 0) {
      const Fe<L> s = fe_add(ld_fe<L>(g_sm), ld_fe<L>(g_sm + L), F), c = ld_fe_cg<L>(A.st.claim);
      bool eq = true;
#pragma unroll
      for (int l = 0; l < L; ++l) eq = eq && s.w[l] == c.w[l];
      if (!eq) atomicOr(A.st.status, kStatusClaim);
    }
    __syncwarp();
  }
  const bool last_round = j == A.num_rounds - 1;
  const bool claim = A.want_claim || last_round;
  // What the end of the round reads from global memory, before the hash: the digest's weights
  // (lanes 0..7) and the Lagrange weights (lanes 8..8 + d); T_{n-1} in the last round (lane k).
  constexpr int kParts = 8 / L;  // field-sized pieces of the 256-bit digest
  Fe<L> con = consts.dig;
  if (claim && lane >= 8 && lane <= 8 + d) con = fc_get<L>(fc.lag[d][lane - 8]);
  Fe<L> e = fe_zero<L>(), o = fe_zero<L>();
  if (last_round && lane < E.num_vars) {
    const uint32_t* tab = A.last ? A.last : (A.fold ? A.dst : A.src);  // T_{n-1}: 2 entries per plane
#pragma unroll
    for (int l = 0; l < L; ++l) {
      e.w[l] = tab[(lane * L + l) * 2 + 0];
      o.w[l] = tab[(lane * L + l) * 2 + 1];
    }
  }
  // challenge r_j; lanes 8 + t: g_j(t) times its Lagrange weight, in the same product
  Fe<L> v = fe_zero<L>();
  if (A.mode == kChallengeSha3) {
    auto word = [&](int q) -> uint32_t { return __funnelshift_l(end.msg[q], end.msg[q + 1], 8); };
    uint32_t lo, hi;
    sha3_256_warp(word, 25 + 4 * (d + 1) * L, lo, hi);
    if (lane < 4) {
      end.dig[2 * lane] = lo;
      end.dig[2 * lane + 1] = hi;
    }
    __syncwarp();
    // digest (little-endian 256-bit D) -> D R mod p = sum_i D_i (R^2 2^(32 L i)) / R
    if (lane < kParts) v = ld_fe<L>(end.dig + lane * L);
  }
  if (claim && lane >= 8 && lane <= 8 + d) v = ld_fe<L>(g_sm + (lane - 8) * L);
  Fe<L> x = fe_mul_any(con, v, F);
  Fe<L> r;
  if (A.mode == kChallengeSha3) {
    Fe<L> y = x;
#pragma unroll
    for (int off = kParts / 2; off > 0; off >>= 1) y = fe_add(y, fe_shfl_down(y, off), F);
    r = fe_shfl(y, 0);
  } else if (A.mode == kChallengeFixed) {
    r = fc_get<L>(fc.one);
  } else {
    r = ld_fe_cg<L>(A.st.chals + j * L);
  }
  if (lane == 0) {
    if (A.mode != kChallengeExplicit) st_fe<L>(A.st.chals + j * L, r);
    st_fe<L>(end.r, r);
  }
  if (!claim) return;
  // g_j(r_j), the next round's claim or the final claim: sum_t w_t prod_{s != t} (r - s), the
  // products of all factors but one by doubling over the lanes of an octet (lane i the factor
  // r - i, or 1): pairs, then quads beside "all but mine" of a quad, then the other quad's.
  const int i8 = lane & 7;
  Fe<L> u = fc_get<L>(fc.one);
  if (i8 <= d) u = fe_sub(r, fc_get<L>(fc.pts[i8]), F);
  const Fe<L> u1 = fe_shfl_xor(u, 1);
  const Fe<L> p2 = fe_mul(u, u1, F);
  const Fe<L> p2o = fe_shfl_xor(p2, 2);
  const Fe<L> p4 = fe_mul(lane < 8 ? p2 : u1, p2o, F);  // lanes 0..7 the quad, 8..15 all but mine of it
  Fe<L> q = p4;
  if (d >= 4) q = fe_mul(p4, fe_shfl(p4, (lane & 3) | (~lane & 4)), F);  // times the other quad (lanes 0..7)
  const bool mine = lane >= 8 && lane <= 8 + d;
  Fe<L> term = fe_mul(q, x, F);
  if (!mine) term = fe_zero<L>();
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) term = fe_add(term, fe_shfl_down(term, off), F);
  if (lane == 8) st_fe<L>(last_round ? A.st.finals : A.st.claim, term);
  // last round: f_k(r) per table
  if (last_round) {
    const Fe<L> f = fe_add(e, fe_mul(r, fe_sub(o, e, F), F), F);
    if (lane < E.num_vars) st_fe<L>(A.st.finals + (1 + lane) * L, f);
  }
}

// The round's integer sums to g_j and its end; every thread of the block calls, after a barrier.
template <int L, int K, typename Sum>
__device__ __forceinline__ void finish_round(const RoundArgs& A, const ExprDev& E, const FieldParams<L, K>& F,
                                             const EndConsts<L>& consts, Sum sum, RoundEnd<L>& end) {
  const int d = E.degree, tid = threadIdx.x, nthr = blockDim.x;
  if (tid < 32)
    sums_to_points<L, K>(sum, d, A.skip1 && !A.ext_out ? A.st.claim : nullptr, A.skip1 != 0, consts.con, F, end);
  if (tid >= 32 || nthr == 32) begin_message<L>(end, d, A.round, nthr == 32 ? tid : tid - 32, nthr == 32 ? 32 : nthr - 32);
  __syncthreads();
  if (A.ext_out) {
    for (int i = tid; i < (d + 1) * L; i += nthr) A.ext_out[i] = end.g()[i];
  } else {
    finalize_round<L, K>(A, E, F, consts, end);
  }
}
template <int L, int K>
__device__ __forceinline__ void finish_round(const RoundArgs& A, const ExprDev& E, const FieldParams<L, K>& F,
                                             RoundEnd<L>& end) {
  finish_round<L, K>(A, E, F, load_end_consts<L>(*A.fc), [&](int i) { return end.s[i]; }, end);
}

// Dynamic shared memory per thread of the generic evaluator: both values of every table, or the
// point sums.
__host__ __device__ constexpr int round_smem_words_per_thread(int K, int L, int dmax) {
  return streamed_tables(L) ? 2 * dmax * L : 2 * K * L;
}

// Launch shape per limb count: 8-limb kernels run 128-thread blocks, smaller fields 256-thread
// blocks. Blocks an SM asked of the compiler at 8 limbs: batch_min_blocks below for the generic
// kernels (SC_L8_MIN_BLOCKS, <= 168 registers, above degree 4), round_min_blocks for the shapes.
__host__ __device__ constexpr int kernel_threads(int L) { return L >= 8 ? 128 : 256; }
#ifndef SC_L8_MIN_BLOCKS
#define SC_L8_MIN_BLOCKS 3
#endif
// 4-limb kernels at 2 blocks/SM (<= 128 registers: 16 warps instead of 8; the degree <= 7
// class spills 36 bytes). Measured on B200 over 4,000 requests of the served stream (2^127 - 1)
// at 80% load: p50 1.34 -> 1.04 ms, p90 13.0 -> 6.6 ms, p99 39-43 -> 23.3 ms; the plain 4-limb
// proofs took the same time either way.
#ifndef SC_L4_MIN_BLOCKS
#define SC_L4_MIN_BLOCKS 2
#endif
// 2-limb generic and batched kernels at 3 blocks/SM (<= 85 registers; 74-80 used, the
// degree <= 7 class spills 4-20 bytes): the 512-proof mixed stream went from 9.89k to 10.16k
// proofs/s (the 64-bit ticks' busy time 31.5 -> 30.0 ms), plain 64-bit proofs the same. At 4
// limbs, 3 blocks/SM spilled 700+ bytes and served p50 went from 1.03 to 1.31 ms.
#ifndef SC_L2_MIN_BLOCKS
#define SC_L2_MIN_BLOCKS 3
#endif
__host__ __device__ constexpr int kernel_min_blocks(int L) {
  return L >= 8 ? SC_L8_MIN_BLOCKS : (L == 4 ? SC_L4_MIN_BLOCKS : (L == 2 ? SC_L2_MIN_BLOCKS : 1));
}
#ifndef SC_SHAPE_MIN_BLOCKS
#define SC_SHAPE_MIN_BLOCKS 2
#endif
// The 1- and 2-limb shape kernels run 2 blocks of 256 threads: at 3 the 2-limb ones spilled
// (zerocheck gate n = 24 1.66 against 1.55 ms with the pair staged in shared memory). The 8-limb
// shape kernels hold every table's value and difference in registers: at 3 blocks
// of 128 threads they spilled; at 2 (no spills) plain BLS n = 22 took 3.28 against 3.37 ms
// with the even/odd product.
#ifndef SC_SHAPE_L8_MIN_BLOCKS
#define SC_SHAPE_L8_MIN_BLOCKS 2
#endif
// The generic kernels, plain and batched, per limb count and degree class: at 8 limbs 4 blocks/SM up to degree 4
// (128 registers), 3 above (shared memory for 7-8 points' products and sums). 5 and 4 blocks
// spilled more than they hid (64 mixed proofs 5.09 ms against 4.84; 3 and 3 blocks 4.99).
__host__ __device__ constexpr int batch_min_blocks(int L, int dmax) {
  return L >= 8 && dmax <= 4 ? 4 : kernel_min_blocks(L);
}
__host__ __device__ constexpr int round_min_blocks(int L, int shape) {
  return (shape != 0 && L <= 2) ? SC_SHAPE_MIN_BLOCKS
                                : ((shape != 0 && L >= 8) ? SC_SHAPE_L8_MIN_BLOCKS : kernel_min_blocks(L));
}

template <int L, int K, int DMAX, int SHAPE = kShapeGeneric>
__global__ void __launch_bounds__(kernel_threads(L), SHAPE ? round_min_blocks(L, SHAPE) : batch_min_blocks(L, DMAX))
    round_kernel(const RoundArgs A, const ExprDev E, const FieldParams<L, K> F) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ RoundEnd<L> end;

  const int tid = threadIdx.x;
  const int nthr = blockDim.x;
  const int d = E.degree;
  uint32_t* sv = smem;                           // [K][L][nthr] values at 0 (or the point sums)
  uint32_t* sd = smem + E.num_vars * L * nthr;   // [K][L][nthr] values at 1

  pdl_begin();
  Fe<L> acc[DMAX + 1];
#pragma unroll
  for (int t = 0; t <= DMAX; ++t) acc[t] = fe_zero<L>();
  Fe<L> r_prev = fe_zero<L>();
  if (A.fold) r_prev = ld_fe_cg<L>(A.st.chals + (A.round - 1) * L);
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * nthr;
  constexpr int kTable = fold_table_words<L, K>();
  __shared__ __align__(16) uint32_t fold_table[kTable ? kTable : 4];
  if constexpr (kTable != 0) {
    if (A.fold) make_fold_table<L, K>(*A.fc, r_prev, F, fold_table);
  }
  process_pairs<L, K, DMAX, SHAPE>(A.src, A.dst, A.src_len, A.fold != 0, r_prev, E, sv, sd,
                                   static_cast<uint64_t>(blockIdx.x) * nthr + tid, A.pairs, stride, A.skip1 != 0, acc, F,
                                   fold_table);

  // the block's integer sums to the grid's; the last block finalises the round
  __syncthreads();
  warp_sums<L, DMAX + 1>(acc, d, smem);
  if (!grid_sums<L>(smem, d, blockIdx.x, gridDim.x, A.sums, A.st.counter, end)) return;
  finish_round<L, K>(A, E, F, end);
}

// ------------------------------------------------------------------------------ resume folds
//
// T_i = T_{i-1} + r_{i-1} (odd - even) and nothing else: the folds that bring a resumed
// proof's tables to the round it continues from (the round kernel folds the last one
// itself). One thread per output pair of one table: a 16-byte load per limb plane in, an
// 8-byte store per plane out, as the round kernel's fused fold. src_len >= 4 entries.
template <int L, int K>
__global__ void __launch_bounds__(256) fold_kernel(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst,
                                                   uint64_t src_len, int num_tables, const uint32_t* r_dev,
                                                   const FieldParams<L, K> F) {
  const uint64_t quads = src_len >> 2;  // output pairs per table
  const uint64_t total = quads * static_cast<uint64_t>(num_tables);
  const uint64_t dst_len = src_len >> 1;
  const Fe<L> r = ld_fe_cg<L>(r_dev);
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint64_t k = i / quads, q = i - k * quads;
    Fe<L> x0, x1, x2, x3;
#pragma unroll
    for (int l = 0; l < L; ++l) {
      const uint4 v = __ldcs(reinterpret_cast<const uint4*>(src + (k * L + l) * src_len) + q);
      x0.w[l] = v.x; x1.w[l] = v.y; x2.w[l] = v.z; x3.w[l] = v.w;
    }
    Fe<L> e, o;
    fe_fold2(e, o, x0, x1, x2, x3, r, F);
#pragma unroll
    for (int l = 0; l < L; ++l) reinterpret_cast<uint2*>(dst + (k * L + l) * dst_len)[q] = make_uint2(e.w[l], o.w[l]);
  }
}

}  // namespace sc
