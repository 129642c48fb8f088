// Small rounds in one block.
//
// A round of a few hundred pairs or fewer is bound by latency: one thread per pair walks
// through every fold, point and term of the expression while most of the GPU has nothing to
// do, and grid-wide sums and a launch cost as much again. Here one block has the round to
// itself and spreads it over all its threads:
//   fold      one (table, entry) of T_j per thread, from T_{j-1} in global memory in the first
//             round and in shared memory afterwards;
//   evaluate  one (pair, point, group of terms) per thread, points 0..d - 1 and the leading
//             coefficient (prover.cuh, make_point_weights), the factors' values formed from
//             T_j in shared memory;
//   sum       16-bit halves of the words as integers, over the warp where its lanes share the
//             point, then in shared memory;
//   finish    prover.cuh, finish_round.
// Rounds follow one another inside the block (a proof's last rounds in one launch, the served
// and batched tails), T_j never leaving shared memory, or a launch holds one round and stores
// T_j for the next; a round of a few thousand pairs is cut into parts of a few dozen, a block
// each, whose sums meet as any round's do (prove_part). Measured on B200, clocks of a late round (a few pairs): 9k at 1 limb (the
// hash 5k of them), 12k at 2, 15k at 4 and 26k at 8 limbs, where the one-thread-a-pair round
// took 16k to 140k, plus its launch.
#pragma once
#include "prover.cuh"

namespace sc {

constexpr int kTailThreads = 512;
__host__ __device__ constexpr int tail_threads(int L) { return L >= 8 ? 256 : kTailThreads; }

// Shared-memory words of a tail that starts with `pairs` pairs: T_j, T_{j+1} beside it.
__host__ __device__ constexpr size_t tail_smem_words(uint64_t pairs, int K, int L) {
  return static_cast<size_t>(3) * pairs * K * L;
}

// The factor's value at this thread's point from its table's entries (e, o): e at 0, o - e for
// the leading coefficient (lead), else o + (point - 1) (o - e).
template <int L, int K>
__device__ __forceinline__ Fe<L> tail_value(const Fe<L>& e, const Fe<L>& o, int point, bool lead,
                                            const FieldParams<L, K>& F) {
  if (!lead && point < 2) return point == 0 ? e : o;
  constexpr bool LZ = lazy_generic<L, K>();
  const Fe<L> d = fe_sub(o, e, F);
  if (lead) return d;
  Fe<L> v = lz_add_c<LZ>(o, d, F);
  for (int t = 2; t < point; ++t) v = lz_add_c<LZ>(v, d, F);
  return v;
}

// P pairs of T_j (P a power of two, the pairs from q0 on) into cur, [table][limb][2 P]: folded
// with r from T_{j-1} -- prev (shared memory, [table][limb][4 P]) or, when null, A.src -- or, in
// round 0, copied from A.src. store: also to A.dst.
template <int L, int K>
__device__ __forceinline__ void tail_fold(const RoundArgs& A, int nv, const FieldParams<L, K>& F, const Fe<L>& r,
                                          uint64_t q0, int lgP, const uint32_t* prev, bool store, uint32_t* cur) {
  const int lg2P = lgP + 1, entries = nv << lg2P;
  for (int i = threadIdx.x; i < entries; i += blockDim.x) {
    const int v = i >> lg2P, x = i & ((1 << lg2P) - 1);
    Fe<L> f;
    if (!A.fold) {
#pragma unroll
      for (int l = 0; l < L; ++l) f.w[l] = __ldcg(A.src + static_cast<uint64_t>(v * L + l) * A.src_len + 2 * q0 + x);
    } else {
      Fe<L> a, b;
#pragma unroll
      for (int l = 0; l < L; ++l) {
        uint2 w;
        if (prev)
          w = reinterpret_cast<const uint2*>(prev + ((v * L + l) << (lg2P + 1)))[x];
        else
          w = __ldcg(reinterpret_cast<const uint2*>(A.src + static_cast<uint64_t>(v * L + l) * A.src_len) + 2 * q0 + x);
        a.w[l] = w.x;
        b.w[l] = w.y;
      }
      f = fe_fold(a, b, r, F);
      if (store) {
#pragma unroll
        for (int l = 0; l < L; ++l) A.dst[static_cast<uint64_t>(v * L + l) * (A.src_len >> 1) + 2 * q0 + x] = f.w[l];
      }
    }
#pragma unroll
    for (int l = 0; l < L; ++l) cur[((v * L + l) << lg2P) + x] = f.w[l];
  }
}

// The point sums of the P pairs in cur, added as 16-bit halves into cnt[(point L + l) 2 + half].
// task = (term group, point, pair), pairs fastest; the groups share the terms out. skip1: point
// 1 is left out.
template <int L, int K>
__device__ __forceinline__ void tail_eval(const ExprDev& E, const FieldParams<L, K>& F, const uint32_t* cur, int lgP,
                                          bool skip1, uint32_t* cnt) {
  constexpr bool LZ = lazy_generic<L, K>();
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31;
  const int d = E.degree, S = d + 1 - (skip1 ? 1 : 0), P = 1 << lgP, lg2P = lgP + 1;
  const uint32_t s_inv = 65536u / S + 1;  // combo / S below, for combo < 2^13
  int G = nthr / (S << lgP);
  G = G < 1 ? 1 : (G > E.num_terms ? E.num_terms : G);
  const int tasks = (G * S) << lgP;
  for (int i = tid; i < ((tasks + 31) & ~31); i += nthr) {
    const bool active = i < tasks;
    const int combo = i >> lgP, q = i & (P - 1);
    const int g = static_cast<int>((combo * s_inv) >> 16);
    int point = combo - g * S;
    if (skip1 && point) ++point;
    const bool lead = point == d && d >= 2;
    Fe<L> sum = fe_zero<L>();
    if (active)
      for (int t = g; t < E.num_terms; t += G) {
        const int off = E.term_off[t], len = E.term_len[t], kind = E.coeff_kind[t];
        if (lead && len < d) continue;
        auto value = [&](int v) {
          Fe<L> e, o;
#pragma unroll
          for (int l = 0; l < L; ++l) {
            const uint2 w = reinterpret_cast<const uint2*>(cur + ((v * L + l) << lg2P))[q];
            e.w[l] = w.x;
            o.w[l] = w.y;
          }
          return tail_value(e, o, point, lead, F);
        };
        Fe<L> prod = value(E.flat[off]);
        bool neg = kind == kCoeffMinus;
        if (kind == kCoeffSmall) {
          const int32_t c = E.coeff_small[t];
          const uint32_t m = c < 0 ? static_cast<uint32_t>(-static_cast<int64_t>(c)) : static_cast<uint32_t>(c);
          Fe<L> base = prod;  // double and add
          prod = fe_zero<L>();
          for (uint32_t k = m; k; k >>= 1) {
            if (k & 1u) prod = lz_add<LZ>(prod, base, F);
            if (k > 1u) base = lz_add<LZ>(base, base, F);
          }
          neg = c < 0;
        } else if (kind == kCoeffMont) {
          Fe<L> cm;
#pragma unroll
          for (int l = 0; l < L; ++l) cm.w[l] = E.coeff_mont[t][l];
          prod = lz_mul<LZ>(prod, cm, F);
        }
        for (int f = 1; f < len; ++f) prod = lz_mul<LZ>(prod, value(E.flat[off + f]), F);
        sum = lz_add_or_sub<LZ>(sum, prod, neg, F);
      }
    // a warp's lanes share the point when P >= 32
    if (P >= 32) {
      uint32_t mine = 0;
#pragma unroll
      for (int l = 0; l < L; ++l) {
        const uint32_t lo = __reduce_add_sync(0xffffffffu, sum.w[l] & 0xffffu);
        const uint32_t hi = __reduce_add_sync(0xffffffffu, sum.w[l] >> 16);
        if (lane == 2 * l) mine = lo;
        if (lane == 2 * l + 1) mine = hi;
      }
      if (lane < 2 * L) atomicAdd(&cnt[point * L * 2 + lane], mine);
    } else if (active) {
#pragma unroll
      for (int l = 0; l < L; ++l) {
        atomicAdd(&cnt[(point * L + l) * 2], sum.w[l] & 0xffffu);
        atomicAdd(&cnt[(point * L + l) * 2 + 1], sum.w[l] >> 16);
      }
    }
  }
}

// Rounds A.round .. A.round + rounds - 1 of a proof by this block; every thread calls, after a
// barrier. A (shared memory) describes the first of them, with A.pairs a power of two, and is
// advanced from round to round; r_ready: end.r holds the challenge its fold needs. smem:
// tail_smem_words(A.pairs, tables, L) words. store: T_j of the last of the rounds also goes to
// A.dst. The first round may take g(1) from the claim or check it (A's flags); the rounds after it
// do neither, whatever their size: point 1 is one more task beside the others here.
template <int L, int K>
__device__ __forceinline__ void prove_tail(RoundArgs& A, const ExprDev& E, const FieldParams<L, K>& F, int rounds,
                                           bool r_ready, bool store, uint32_t* smem, RoundEnd<L>& end) {
  const int tid = threadIdx.x, nthr = blockDim.x, nv = E.num_vars;
  const EndConsts<L> consts = load_end_consts<L>(*A.fc);
  uint32_t* cur = smem;
  uint32_t* nxt = smem + static_cast<size_t>(2) * nv * L * A.pairs;
  for (int k = 0;; ++k) {
    const int lgP = 31 - __clz(static_cast<int>(A.pairs));
    Fe<L> r = fe_zero<L>();
    if (A.fold) r = k == 0 && !r_ready ? ld_fe_cg<L>(A.st.chals + (A.round - 1) * L) : ld_fe<L>(end.r);
    tail_fold<L, K>(A, nv, F, r, 0, lgP, k == 0 ? nullptr : nxt, store && k == rounds - 1, cur);
    for (int i = tid; i < kMaxPoints * L * 2; i += nthr) end.half[i] = 0;
    __syncthreads();
    tail_eval<L, K>(E, F, cur, lgP, A.skip1 != 0, end.half);
    if (tid == 0) A.last = cur;
    __syncthreads();
    finish_round<L, K>(A, E, F, consts, [&](int i) { return end.half_sum(i); }, end);
    if (k == rounds - 1) break;
    __syncthreads();  // the finish read A; r_j is visible to the block
    if (tid == 0) {
      ++A.round;
      A.pairs >>= 1;
      A.fold = 1;
      A.skip1 = A.want_claim = A.check_claim = 0;  // the claim belonged to the first round
    }
    // T_j becomes the source; T_{j+1} goes where T_{j-1} was (the first time: behind T_j)
    uint32_t* const t = cur;
    cur = nxt;
    nxt = t;
    __syncthreads();
  }
}

// P = 2^lgP pairs of a round, from part P on, by this block; `parts` blocks make up the round and the last
// of them ends it. smem: 2 P tables L words.
template <int L, int K>
__device__ __forceinline__ void prove_part(const RoundArgs& A, const ExprDev& E, const FieldParams<L, K>& F, int lgP,
                                           uint32_t part, uint32_t parts, uint32_t* smem, RoundEnd<L>& end) {
  const int tid = threadIdx.x, nthr = blockDim.x, d = E.degree;
  Fe<L> r = fe_zero<L>();
  if (A.fold) r = ld_fe_cg<L>(A.st.chals + (A.round - 1) * L);
  tail_fold<L, K>(A, E.num_vars, F, r, static_cast<uint64_t>(part) << lgP, lgP, nullptr, true, smem);
  for (int i = tid; i < kMaxPoints * L * 2; i += nthr) end.half[i] = 0;
  __syncthreads();
  tail_eval<L, K>(E, F, smem, lgP, A.skip1 != 0, end.half);
  __syncthreads();
  for (int i = tid; i < (d + 1) * L; i += nthr) {
    if (parts == 1)
      end.s[i] = end.half_sum(i);
    else
      atomicAdd(reinterpret_cast<unsigned long long*>(A.sums + (part % kSumCopies) * kMaxPoints * L + i),
                static_cast<unsigned long long>(end.half_sum(i)));
  }
  if (!grid_end<L>(d, parts, A.sums, A.st.counter, end)) return;
  finish_round<L, K>(A, E, F, end);
}

struct TailArgs {
  RoundArgs first;
  int32_t rounds;
  int32_t store;
};

template <int L, int K>
__global__ void __launch_bounds__(tail_threads(L), 1) tail_kernel(const TailArgs T, const ExprDev E, const FieldParams<L, K> F) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ RoundEnd<L> end;
  __shared__ __align__(16) RoundArgs A;
  if (threadIdx.x == 0) A = T.first;
  pdl_begin();
  __syncthreads();
  prove_tail<L, K>(A, E, F, T.rounds, false, T.store != 0, smem, end);
}

// One round over gridDim.x blocks of 2^lgP pairs.
struct PartArgs {
  RoundArgs round;
  int32_t lgP;
  int32_t pad;
};
template <int L, int K>
__global__ void __launch_bounds__(tail_threads(L), 1) part_kernel(const PartArgs T, const ExprDev E, const FieldParams<L, K> F) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ RoundEnd<L> end;
  pdl_begin();
  prove_part<L, K>(T.round, E, F, T.lgP, blockIdx.x, gridDim.x, smem, end);
}

}  // namespace sc
