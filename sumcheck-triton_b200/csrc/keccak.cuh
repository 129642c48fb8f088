// SHA3-256 on the device, computed by one warp.
//
// Written from FIPS 202 (SHA-3 Standard, NIST 2015): Keccak-f[1600] is 24 rounds of
// theta, rho, pi, chi, iota on a 5x5 array of 64-bit lanes; SHA3-256 absorbs 136-byte
// blocks (rate 1088 bits) after padding the message with 0x06 ... 0x80.
//
// Layout: lane i < 25 of the warp holds state word A[x + 5y] (x = i % 5, y = i / 5).
// Column parities, the pi permutation and chi's neighbours are warp shuffles, so the state
// never leaves registers and costs each thread two registers. The rho offsets and round
// constants are computed at compile time from the standard's own definitions (section
// 3.2.2: offsets (t + 1)(t + 2)/2 along the (x, y) -> (y, 2x + 3y) walk; section 3.2.5: the
// rc LFSR), not typed in.
#pragma once
#include <cstdint>

namespace sc {

struct KeccakConsts {
  uint32_t rot[25];
  uint64_t rc[24];
};

constexpr bool keccak_rc_bit(int t) {
  // FIPS 202 Algorithm 5. Bit k of r is R[k]; R starts as 10000000 (R[0] = 1).
  if (t % 255 == 0) return true;
  unsigned r = 1;
  for (int i = 1; i <= t % 255; ++i) {
    r <<= 1;                     // R = 0 || R, so R[8] is the old R[7]
    if (r & 0x100) r ^= 0x171;   // R[0], R[4], R[5], R[6] ^= R[8]; clears R[8]
    r &= 0xFF;                   // Trunc_8
  }
  return (r & 1) != 0;
}

constexpr KeccakConsts make_keccak_consts() {
  KeccakConsts k{};
  k.rot[0] = 0;
  int x = 1, y = 0;
  for (int t = 0; t < 24; ++t) {
    k.rot[x + 5 * y] = static_cast<uint32_t>(((t + 1) * (t + 2) / 2) % 64);
    int nx = y, ny = (2 * x + 3 * y) % 5;
    x = nx;
    y = ny;
  }
  for (int ir = 0; ir < 24; ++ir) {
    uint64_t rc = 0;
    for (int j = 0; j <= 6; ++j) {
      if (keccak_rc_bit(j + 7 * ir)) rc |= uint64_t{1} << ((1 << j) - 1);
    }
    k.rc[ir] = rc;
  }
  return k;
}

static __constant__ KeccakConsts kKeccak = make_keccak_consts();

// Keccak-f[1600] on the warp-distributed state: lane i < 25 holds word A[i % 5, i / 5] as
// (lo, hi). All 32 lanes must call; lanes 25..31 carry values nothing reads.
//
// The permutation is one dependent chain, so its time is the latency of the exchanges between
// lanes. A round has three: the column parities, the neighbour columns' parities (theta), and
// one for pi and chi together -- chi's two neighbours are read straight from the rotated words
// they come from, instead of a pi exchange followed by a chi exchange. Words are two 32-bit
// registers: the per-lane rotation is a swap and two funnel shifts. Two rounds a loop pass
// (24 unrolled rounds would be fetched anew at every round's end). Measured on B200, one warp:
// 4530 clocks, against 5205 with four exchanges and 64-bit shifts. Exchanging through shared
// memory (4970-5340), and theta in one exchange of ten words (5060), were slower.
__device__ __forceinline__ void keccak_f1600_warp(uint32_t& lo, uint32_t& hi, int lane) {
  constexpr unsigned kAll = 0xffffffffu;
  const int x = lane % 5, y = (lane / 5) % 5;
  const int row = 5 * y;
  const uint32_t rot = lane < 25 ? kKeccak.rot[lane] : 0u;
  const bool swap = rot >= 32;
  const uint32_t s = rot & 31;
  const int x1 = (x + 1) % 5, x2 = (x + 2) % 5, xm = (x + 4) % 5;
  const int c1 = x + 5 * ((y + 1) % 5), c2 = x + 5 * ((y + 2) % 5), c3 = x + 5 * ((y + 3) % 5), c4 = x + 5 * ((y + 4) % 5);
  // pi (FIPS 202 3.2.3): A'[x, y] = A[(x + 3y) mod 5, x]
  const int p0 = (x + 3 * y) % 5 + 5 * x, p1 = (x1 + 3 * y) % 5 + 5 * x1, p2 = (x2 + 3 * y) % 5 + 5 * x2;
  const uint32_t iota = lane == 0 ? ~0u : 0u;
#pragma unroll 2
  for (int ir = 0; ir < 24; ++ir) {
    const uint64_t rc = kKeccak.rc[ir];
    const uint32_t rc_lo = static_cast<uint32_t>(rc) & iota, rc_hi = static_cast<uint32_t>(rc >> 32) & iota;
    // theta
    uint32_t cl = lo ^ __shfl_sync(kAll, lo, c1) ^ __shfl_sync(kAll, lo, c2);
    uint32_t ch = hi ^ __shfl_sync(kAll, hi, c1) ^ __shfl_sync(kAll, hi, c2);
    cl = cl ^ __shfl_sync(kAll, lo, c3) ^ __shfl_sync(kAll, lo, c4);
    ch = ch ^ __shfl_sync(kAll, hi, c3) ^ __shfl_sync(kAll, hi, c4);
    const uint32_t ml = __shfl_sync(kAll, cl, xm + row), mh = __shfl_sync(kAll, ch, xm + row);
    const uint32_t ul = __shfl_sync(kAll, cl, x1 + row), uh = __shfl_sync(kAll, ch, x1 + row);
    lo ^= ml ^ __funnelshift_l(uh, ul, 1);
    hi ^= mh ^ __funnelshift_l(ul, uh, 1);
    // rho
    const uint32_t s0 = swap ? hi : lo, s1 = swap ? lo : hi;
    const uint32_t rl = __funnelshift_l(s1, s0, s), rh = __funnelshift_l(s0, s1, s);
    // pi and chi, then iota
    const uint32_t b0l = __shfl_sync(kAll, rl, p0), b0h = __shfl_sync(kAll, rh, p0);
    const uint32_t b1l = __shfl_sync(kAll, rl, p1), b1h = __shfl_sync(kAll, rh, p1);
    const uint32_t b2l = __shfl_sync(kAll, rl, p2), b2h = __shfl_sync(kAll, rh, p2);
    lo = (b0l ^ (~b1l & b2l)) ^ rc_lo;
    hi = (b0h ^ (~b1h & b2h)) ^ rc_hi;
  }
}

// SHA3-256 by one warp (every lane calls). word(q) is the message's 32-bit little-endian word
// q, with the padding's 0x06 after the last byte and zeros beyond; len its length in bytes.
// digest: lanes 0..3 get 64-bit word `lane` of the digest as (lo, hi); the others' are unused.
template <typename Word>
__device__ __forceinline__ void sha3_256_warp(Word word, int len, uint32_t& lo, uint32_t& hi) {
  const int lane = threadIdx.x & 31;
  constexpr int kRate = 136;
  const int nblocks = len / kRate + 1;
  lo = hi = 0;
  for (int b = 0; b < nblocks; ++b) {
    if (lane < kRate / 8) {
      const int q = b * (kRate / 4) + 2 * lane;
      lo ^= word(q);
      hi ^= word(q + 1);
      if (b == nblocks - 1 && lane == kRate / 8 - 1) hi ^= 0x80000000u;
    }
    keccak_f1600_warp(lo, hi, lane);
  }
}

}  // namespace sc
