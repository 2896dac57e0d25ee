// Sort positions from one bitmap over the values of a field.
//
// The sort position of an extremum is the number of distinct smaller
// critical-point values in its quantization bin.  Floats of one binade have
// 2^23 codes, so one bit per code (with counts) takes 1.4 MB a binade, and a field whose
// values reach from eb to 2^k eb needs k of them per sign, however many
// critical points it has.  So:
//   1. the encoder (or rank_bits_pairs_kernel, from a pair list) sets the bit
//      of every critical point's value: atomics without a return value, into
//      a few tens of MB that stay in L2;
//   2. two passes over the touched range give every 96 bits the number of set
//      bits before them;
//   3. the lowest code of every bin is found by bisection (a bin is a monotone
//      function of the value), and its prefix count kept in a table;
//   4. an extremum's position is its own prefix count less its bin's.
// No record is moved, and nothing is sorted: the bucket ranking (tsz_sort.cu),
// which this replaces for fields, reads or writes each pair six times and
// falls back to sorting for the wide bins next to zero.  512^3 field, 34.5 M
// critical points: 650 us (and 1030 in the encoder that writes the pairs)
// against 141 (and 1110 in the one that sets the bits: L2 atomics); 1800 x 3600
// field, 1.5 M around zero: 486 (54) against 67 (73).  What bounds it: the
// random 32-byte sector that every extremum reads (95 of the 141 us).
//
// Values nearer to zero than 2^-6 eb (two bins share them) are kept aside and
// sorted, all zeros as one of them (a field of small integers, us, buckets /
// each zero aside / so: 300 x 400 126 / 193 / 123, 160 x 170 x 180 520 / 636 /
// 226); values from 2^30 eb on, more than kSideCap aside, or more than
// kMaxBins bins are left to the bucket ranking, which takes the codes that the
// encoder leaves beside the bits (from a pair list, the pairs).  Such fields,
// in buckets alone / encoded a second time for pairs / from the codes:
//   512^3 of zero mean, bound 1/50 of its deviation       6.29 / 6.55 / 5.2 ms
//   512^3 with seven eighths below the bound              78.0 / 78.9 / 33.8
//   512^3 in 10 M bins                                    5.38 / 5.74 / 5.0
//   1800 x 3600 noise below the bound                     3.30 / 3.41 / 2.2
// (most of it from the gather of the buckets that are radix-sorted, which had
// one CTA a bucket).  A field with bits for all values pays nothing for the
// saddles' codes that measures: compression of 512^3 929 / 930 us.
#pragma once
#include "tsz_common.cuh"

namespace tsz {

constexpr unsigned kRbBits = 96;           // bits of a 16-byte unit; its first word is the prefix count
constexpr unsigned kRbBelow = 6, kRbAbove = 30;   // binades below and above eb
constexpr unsigned kSideCap = 4096;
constexpr unsigned kRankSmall = 2048;      // lists that one CTA sorts
constexpr unsigned kMaxBins = 1u << 22;

// Pairs from which bits are set for them, which is a launch and a wait of its
// own.  Ranking a list (us, bits / buckets): values spread over many bins,
// 16384 pairs 67 / 60, 32768 75 / 60, 65536 77 / 63, 131072 83 / 87, 1 M
// 104 / 147; a thousand and more in a bin, 16384 70 / 72, 32768 75 / 97, 65536
// 79 / 186, 131072 82 / 429.
constexpr unsigned long long kRankBitsMin = 1ull << 16;
// Values of a field from which the encoder sets them, for nothing in launches or
// waits, in a workspace that has the bitmap; fewer are not worth it.  Compression
// of 2D noise (us, bits from the encoder / pairs in buckets): 8100 values 106 /
// 118, 16384 102 / 117, 32761 108 / 118, with a thousand points in a bin 104 /
// 118, 104 / 122, 104 / 163; of a smooth field, whose few points one CTA sorts
// either way, 74.4 / 75.0, 70.0 / 69.9, 69.3 / 70.3.
constexpr unsigned long long kRankBitsFieldMin = 1ull << 14;
// Values from which a workspace gets the bitmap for it (118 MB; 0.25 ms, once).
// Below, one that has met a field of more points than one CTA sorts has it.
constexpr unsigned long long kRankBitsAlways = 1ull << 18;
constexpr unsigned kRbUnits = (unsigned)((2ull * (kRbBelow + kRbAbove) << 23) / kRbBits) + 2u;

struct RankBits {
  unsigned *bits;      // kRbUnits x 4 words, zero between calls
  unsigned rz, rh;     // magnitudes (float bits) [rz, rh) have a bit
  uint2 *side;         // {code, extremum index or ~0} of the values below rz
  uint2 *first;        // the first kRankSmall pairs of an encoder launch: a field with no more needs no scan
  unsigned *stat;      // zeroed: [0] largest ~code, [1] largest code, [2] values aside (but zeros), [3] out of
                       // range, [4] zeros among them, [5] their position
};

constexpr unsigned kZeroCode = 0x80000000u;   // of +0 and -0
// what a thread has seen: the bits will not do; a zero
enum : unsigned { kRbFull = 1u, kRbZero = 2u };

// bit of a value code, by value: the negative half, then the positive one;
// false when the value has none
__host__ __device__ __forceinline__ bool rb_index(unsigned rz, unsigned rh, unsigned code, unsigned *idx) {
  const bool pos = code >> 31;
  const unsigned mag = (pos ? code : ~code) & 0x7FFFFFFFu;
  *idx = pos ? (rh - rz) + (mag - rz) : rh - 1u - mag;
  return mag - rz < rh - rz;
}

// Keeps a value without a bit aside.  Zeros, of which a masked or quantized
// field is full, leave a mark only.  Of the others, the lanes that are here
// together take their places with one atomic, and a thread that has seen that
// the bits will not do takes none: in a field that lies near zero every value
// comes here.
__device__ __forceinline__ void rb_aside(const RankBits &rb, unsigned code, unsigned ext, unsigned &seen) {
  const unsigned mag = ((code >> 31) ? code : ~code) & 0x7FFFFFFFu;
  if (code == kZeroCode) {
    if (!(seen & kRbZero)) rb.stat[4] = 1u;
    seen |= kRbZero;
    return;
  }
  if (seen & kRbFull) return;
  if (mag >= rb.rh) {
    rb.stat[3] = 1u;
    seen |= kRbFull;
    return;
  }
  const unsigned m = __activemask(), lane = threadIdx.x & 31u, first = (unsigned)__ffs((int)m) - 1u;
  unsigned k = 0;
  if (lane == first) k = atomicAdd(rb.stat + 2, (unsigned)__popc(m));
  k = __shfl_sync(m, k, (int)first);
  if (k + (unsigned)__popc(m) > kSideCap) seen |= kRbFull;
  k += (unsigned)__popc(m & ((1u << lane) - 1u));
  if (k < kSideCap) rb.side[k] = make_uint2(code, ext);
}

__device__ __forceinline__ void rb_set(const RankBits &rb, unsigned code, unsigned ext, unsigned &seen) {
  unsigned idx;
  if (rb_index(rb.rz, rb.rh, code, &idx)) {
    const unsigned q = idx / kRbBits, r = idx - q * kRbBits;
    atomicOr(rb.bits + 4u * q + 1u + (r >> 5), 1u << (r & 31u));
  } else {
    rb_aside(rb, code, ext, seen);
  }
}

// largest ~code and code of a thread's values into the statistics (all lanes)
__device__ __forceinline__ void rb_extent(const RankBits &rb, unsigned ncode, unsigned code) {
  ncode = __reduce_max_sync(0xffffffffu, ncode);
  code = __reduce_max_sync(0xffffffffu, code);
  if ((threadIdx.x & 31) == 0 && (ncode | code)) {
    atomicMax(rb.stat, ncode);
    atomicMax(rb.stat + 1, code);
  }
}

}  // namespace tsz
