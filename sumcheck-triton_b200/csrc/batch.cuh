// The batched round kernel: ticks of many proofs' rounds over a device work queue.
#pragma once
#include "tail.cuh"

namespace sc {

// ------------------------------------------------------------------------------ batched
//
// Many independent proofs advance together, one launch per "tick" and degree class: a
// persistent kernel whose blocks pull (proof round, tile of pairs) items from a device work
// queue (an atomic counter over the tick's item list). Every item adds its point sums to
// its round's integer sums; the block that finishes the last item of a proof's round (per-proof
// atomic ticket) reads that round's sums and finalises it -- SHA3 challenge included --
// while the other blocks go on with other proofs' items. A round's items may be spread over
// several ticks (the served prover slices large rounds): the ticket counts to the round's
// item total, whichever tick its last item runs in.
//
// Tail rounds: once a proof's round fits in one item, the block that proves it also proves
// every later round of that proof (tail_rounds of them), one after another with block
// barriers in between -- a few microseconds a round instead of one tick each. Round j + 1
// reads T_j, which this block wrote itself, and r_j, which its warp 0 just derived; as soon as
// the rest fits this block's shared memory, tail.cuh spreads it over all threads.

struct BatchRound {
  RoundArgs args;        // this proof's round (src/dst/len/pairs/round/fold/mode/flags/fc/state)
  const ExprDev* expr;   // this proof's expression
  int32_t first_item;    // this tick's items of the round: [first_item, first_item + num_items)
  int32_t num_items;
  int32_t item_base;     // round-relative index of this tick's first item of the round
  int32_t round_items;   // items of the whole round, over all ticks
  int32_t tail_rounds;   // > 0: the block that finalises this round proves the next tail_rounds too
  uint32_t skip1_min_pairs;  // tail rounds: g(1) from the claim when a round has this many pairs
  uint32_t* fold_a;      // tail rounds: T_i for odd i
  uint32_t* fold_b;      //              T_i for even i >= 2
};

struct BatchItem {
  int32_t round;       // index into the tick's BatchRound array
  int32_t lgP;         // >= 0: a small part of 2^lgP pairs, spread over the block (tail.cuh); -1: not
  uint64_t start;      // pairs [start, start + count)
  uint64_t count;
};

struct BatchTickArgs {
  const BatchRound* rounds;
  const BatchItem* items;  // nullptr: one round, item i = pairs [i tile, (i + 1) tile)
  int32_t num_items;
  int32_t lgP;             // with items nullptr: >= 0 for parts of 2^lgP pairs (BatchItem::lgP)
  uint32_t* head;          // queue counter of this tick (zero before the launch); nullptr:
                           // block b does item b alone (grid = num_items)
  uint64_t tile;           // pairs per item when items is nullptr
  unsigned long long* span;  // non-null (zero before the launch): [0] the complement of the first
                             // block's start, [1] the last one's end (nanoseconds)
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// prove_tail out of line: the tick's own register budget does not see it.
template <int L, int K>
__device__ __noinline__ void batch_tail(RoundArgs* A, const ExprDev* E, const FieldParams<L, K> F, int rounds,
                                        uint32_t* smem, RoundEnd<L>* end) {
  prove_tail<L, K>(*A, *E, F, rounds, true, false, smem, *end);
}

template <int L, int K>
__device__ __noinline__ void batch_part(const RoundArgs* A, const ExprDev* E, const FieldParams<L, K> F, int lgP,
                                        uint32_t part, uint32_t parts, uint32_t* smem, RoundEnd<L>* end) {
  prove_part<L, K>(*A, *E, F, lgP, part, parts, smem, *end);
}

// finish_round out of line, for the same reason.
template <int L, int K>
__device__ __noinline__ void batch_finish(const RoundArgs* A, const ExprDev* E, const FieldParams<L, K> F, RoundEnd<L>* end) {
  finish_round<L, K>(*A, *E, F, *end);
}

template <int L, int K, int DMAX>
__global__ void __launch_bounds__(kernel_threads(L), batch_min_blocks(L, DMAX))
    batch_round_kernel(const BatchTickArgs T, const FieldParams<L, K> F) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ RoundEnd<L> end;
  __shared__ __align__(16) ExprDev E;
  __shared__ __align__(16) BatchRound R;
  __shared__ const ExprDev* cur_expr;
  __shared__ int item_sm;

  const int tid = threadIdx.x, nthr = blockDim.x;
  uint32_t dyn_bytes;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
  const uint32_t* table_of = nullptr;  // the challenge the fold table is of
  if (tid == 0) cur_expr = nullptr;
  pdl_begin();
  if (T.span && tid == 0) atomicMax(T.span, ~global_ns());
  for (int pass = 0;; ++pass) {
    __syncthreads();
    if (tid == 0)
      item_sm = T.head ? static_cast<int>(atomicAdd(T.head, 1u)) : (pass == 0 ? static_cast<int>(blockIdx.x) : T.num_items);
    __syncthreads();
    const int it = item_sm;
    if (it >= T.num_items) break;
    BatchItem I;
    if (T.items) {
      I = T.items[it];
    } else {
      I.round = 0;
      I.lgP = T.lgP;
      I.start = static_cast<uint64_t>(it) * T.tile;
    }
    if (tid == 0) R = T.rounds[I.round];
    __syncthreads();
    if (!T.items) I.count = R.args.pairs - I.start < T.tile ? R.args.pairs - I.start : T.tile;
    if (R.expr != cur_expr) {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(R.expr);
      uint32_t* dst = reinterpret_cast<uint32_t*>(&E);
      for (int i = tid; i < static_cast<int>(sizeof(ExprDev) / 4); i += nthr) dst[i] = src[i];
      __syncthreads();
      if (tid == 0) cur_expr = R.expr;
    }
    const int d = E.degree;
    uint32_t* sv = smem;
    uint32_t* sd = smem + E.num_vars * L * nthr;
    // k = 0: this item of the proof's round; k >= 1: the proof's tail rounds (only in the
    // block that finalised round k - 1; R.args then describes round R.args.round)
    if (I.lgP >= 0) {
      batch_part<L, K>(&R.args, &E, F, I.lgP, static_cast<uint32_t>(R.item_base + (it - R.first_item)),
                       static_cast<uint32_t>(R.round_items), smem, &end);
      continue;
    }
    for (int k = 0;; ++k) {
      if (k > 0 && tail_smem_words(R.args.pairs, E.num_vars, L) * 4 <= dyn_bytes) {
        batch_tail<L, K>(&R.args, &E, F, R.tail_rounds - k + 1, smem, &end);
        break;
      }
      Fe<L> acc[DMAX + 1];
#pragma unroll
      for (int t = 0; t <= DMAX; ++t) acc[t] = fe_zero<L>();
      Fe<L> r_prev = fe_zero<L>();
      if (R.args.fold) r_prev = k == 0 ? ld_fe_cg<L>(R.args.st.chals + (R.args.round - 1) * L) : ld_fe<L>(end.r);
      const uint64_t q0 = k == 0 ? I.start : 0, q1 = k == 0 ? I.start + I.count : R.args.pairs;
      constexpr int kTable = fold_table_words<L, K>();
      __shared__ __align__(16) uint32_t fold_table[kTable ? kTable : 4];
      if constexpr (kTable != 0) {
        const uint32_t* const r_at = R.args.st.chals + (R.args.round - 1) * L;  // one table for a round's items
        if (R.args.fold && r_at != table_of) {
          make_fold_table<L, K>(*R.args.fc, r_prev, F, fold_table);
          table_of = r_at;
        }
      }
      process_pairs<L, K, DMAX>(R.args.src, R.args.dst, R.args.src_len, R.args.fold != 0, r_prev, E, sv, sd, q0 + tid,
                                q1, nthr, R.args.skip1 != 0, acc, F, fold_table);
      __syncthreads();
      warp_sums<L, DMAX + 1>(acc, d, smem);
      const uint32_t part = k == 0 ? static_cast<uint32_t>(R.item_base + (it - R.first_item)) : 0;
      const uint32_t parts = k == 0 ? static_cast<uint32_t>(R.round_items) : 1;
      if (!grid_sums<L>(smem, d, part, parts, R.args.sums, R.args.st.counter, end)) break;
      batch_finish<L, K>(&R.args, &E, F, &end);
      if (k == R.tail_rounds) break;
      __syncthreads();  // the finalisation read R.args; r_j and T_j are visible to the block
      if (tid == 0) {   // round j + 1 of the same proof
        RoundArgs& A = R.args;
        const int j = A.round + 1;
        if (j >= 2) A.src = A.dst;  // T_j (round 1 folds the tables themselves)
        A.dst = (j & 1) ? R.fold_a : R.fold_b;
        A.round = j;
        A.pairs >>= 1;
        A.src_len = A.pairs * 4;
        A.fold = 1;
        A.skip1 = A.pairs >= R.skip1_min_pairs ? 1 : 0;
        A.want_claim = (j + 1 < A.num_rounds && (A.pairs >> 1) >= R.skip1_min_pairs) ? 1 : 0;
        A.check_claim = 0;
      }
      __syncthreads();
    }
  }
  if (T.span && tid == 0) atomicMax(T.span + 1, global_ns());
}

}  // namespace sc
