// Fused topology encoder for blockSize 64, the block size of the reference's
// benchmark configurations: classification of every point (4 neighbours in
// 2D, 6 in 3D), quantization, deltas, bit packing with the 2-bit type tags,
// the critical-point pairs for the rank stage, and the decoupled look-back
// that places every tile in the stream -- one pass over the field.
//
// Same stream bytes as the general octet encoder (tsz_codec2.cuh) and the
// reference (SZp/src/szp_cuda_topology_3d.cu:832-1059,
// SZp/src/szp_cuda_topology.cu:532-772); it differs in how the work maps onto
// the machine:
//   * thread t of a CTA owns elements 8t .. 8t+7 of a 2048-element tile, so a
//     warp reads 1 KB of the field with two 16-byte loads per lane and eight
//     lanes form one codec block;
//   * the +-1 neighbours come from the adjacent lanes (shuffles), and each
//     edge along the row is compared once for both of its points;
//   * the two other axes are folded into max / min masks one axis at a time,
//     so that only one neighbour octet pair is live, and comparisons are sign
//     bits of differences (FMA pipe) pushed into masks;
//   * index arithmetic is per octet (one coordinate split), never per point;
//   * the CTA keeps two tile images and runs one tile behind, and a warp of
//     its own claims tiles and looks back while the others work.
//
// What bounds it (512^3 field, abs eb 1e-4, B200): instruction issue, with the
// ALU pipe 65 % busy (4.2 warp instructions per element, of which
// classification 0.9).  Its time there, the extrema's codes and the values'
// bits included, by what it was brought down with:
//   1110 us  look-back by all warps behind the write-out, 64 registers
//    994     look-back by a ninth warp beside the front half, which knows full
//            blocks; claiming a tile ahead instead of just before its front
//            half costs 350 (every look-back behind the tile waits for it)
//    894     56 registers: four CTAs per SM instead of three
//    772     descriptors as one 16-byte word: one load in the look-back
//    712     comparisons on the FMA pipe, 32-bit coordinate split
//
// The same kernel without the classification encodes integers (with the types
// of a byte array, or none) and quantized fields, in place of the octet encoder
// with its look-back in line: plain field of 60 M floats 575 -> 463 us for
// encoding and decoding, double field of 256^3 217 -> 184, topology of 512^3
// (its sort positions) 977 -> 941.  Five CTAs per SM (40 registers, spills)
// measure the same.
#include "tsz_codec2.cuh"
#include "tsz_enc64.h"
#include "tsz_ops.h"
#include "tsz_runtime.h"

namespace tsz {

constexpr int kE64Threads = 256;                 // the threads that own elements
constexpr int kE64Warps = kE64Threads / 32;
constexpr int kE64Cta = kE64Threads + 32;        // and one warp for tile claims and look-backs
constexpr int kE64Tile = 8 * kE64Threads;        // elements per tile
constexpr int kE64Blocks = kE64Tile / 64;        // codec blocks per tile
constexpr unsigned kE64BlockMax = 289;           // block_bytes(64, 33, tags): a safe bound
constexpr unsigned kE64Img = (kE64Blocks * kE64BlockMax + 64u + 15u) & ~15u;
// staged critical points, one per element at most: pairs, or codes (extrema
// from the front, saddles from the back)
__host__ __device__ constexpr unsigned e64_part(bool bits) { return kE64Img + kE64Tile * (bits ? 4u : 8u); }
// the same of a kernel for mode, whose points are staged only where it classifies
__host__ __device__ constexpr unsigned e64_part(int mode, bool bits) {
  return mode == kEncClassify ? e64_part(bits) : kE64Img;
}

struct E64Sh {
  unsigned wb[kE64Warps], wc[kE64Warps];         // block bytes and (extrema << 16 | points) of each warp
  unsigned long long gbyte, gcnt;                // the tile's place, from the look-back
  unsigned tile_bytes, tile_cps, tile_ext;
  unsigned boff[kE64Blocks];
};

// barrier of the warps that own elements
__device__ __forceinline__ void e64_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// the claim of a tile, from the ninth warp to the others
__device__ __forceinline__ void e64_claim_post() { asm volatile("bar.arrive 2, 288;" ::: "memory"); }
__device__ __forceinline__ void e64_claim_wait() { asm volatile("bar.sync 2, 288;" ::: "memory"); }

// Shifts the sign bit of f into the low end of mask.
__device__ __forceinline__ unsigned push_sign(float f, unsigned mask) {
  return __funnelshift_l(__float_as_uint(f), mask, 1);
}
// x with -0 as +0 (NaN stays NaN)
__device__ __forceinline__ float plus_zero(float x) { return __fadd_rn(x, 0.0f); }
// float_code of a value that is not -0
__device__ __forceinline__ unsigned value_code(float x) {
  const unsigned b = __float_as_uint(x);
  return b ^ ((unsigned)((int)b >> 31) | 0x80000000u);
}

// Masks are built from the sign bits of differences: with no -0 among the
// values, a - b is negative exactly when a < b (a denormal difference is not
// flushed, equal values give +0, and NaN, which a comparison with NaN and
// inf - inf give, has a clear sign bit).  A comparison is then one addition on
// the FMA pipe and one shift, where compare, select and combine are three
// instructions on the ALU pipe, which bounds this kernel.  Element 0 is the
// highest bit of a mask.

// hi / lo masks of one axis: bit 7 - t set when c[t] is above (below) both of
// its neighbours at -off and +off.  c > max.NaN(m, p) is exactly
// (c > m && c > p), NaN operands included.
__device__ __forceinline__ void e64_axis(const float *__restrict__ d, long long i0, long long off, unsigned inter,
                                         bool vec, const float (&c)[8], unsigned &hi, unsigned &lo) {
  float m[8], p[8];
  if (vec) {
    const float4 *pm = reinterpret_cast<const float4 *>(d + i0 - off);
    const float4 *pp = reinterpret_cast<const float4 *>(d + i0 + off);
    const float4 a0 = __ldg(pm), a1 = __ldg(pm + 1), b0 = __ldg(pp), b1 = __ldg(pp + 1);
    m[0] = a0.x; m[1] = a0.y; m[2] = a0.z; m[3] = a0.w; m[4] = a1.x; m[5] = a1.y; m[6] = a1.z; m[7] = a1.w;
    p[0] = b0.x; p[1] = b0.y; p[2] = b0.z; p[3] = b0.w; p[4] = b1.x; p[5] = b1.y; p[6] = b1.z; p[7] = b1.w;
  } else {
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const bool in = (inter >> (7 - t)) & 1u;
      m[t] = in ? __ldg(d + i0 + t - off) : 0.f;
      p[t] = in ? __ldg(d + i0 + t + off) : 0.f;
    }
  }
  unsigned h = 0, w = 0;
#pragma unroll
  for (int t = 0; t < 8; t++) {
    h = push_sign(__fsub_rn(plus_zero(fmax_nan(m[t], p[t])), c[t]), h);
    w = push_sign(__fsub_rn(c[t], fmin_nan(m[t], p[t])), w);
  }
  hi = h;
  lo = w;
}

// (q, r) = divmod(i, d) of a 32-bit index: fdivmod's product in two 32 x 32
// multiplications
__device__ __forceinline__ unsigned divmod32(unsigned i, unsigned d, unsigned long long m, unsigned &r) {
  const unsigned long long t = (unsigned long long)i * (unsigned)m;
  const unsigned long long u = (unsigned long long)i * (unsigned)(m >> 32) + (t >> 32);
  const unsigned q = m ? (unsigned)(u >> 32) : i;
  r = i - q * d;
  return q;
}

// Front half of a tile: load, classify, quantize, pack into img, stage the
// critical points, publish the tile's aggregate.  The 256 threads that own
// elements call it.  FULL: every block of the tile has 64 elements, so the only
// position without a delta is a block's last.  The modes without
// classification take integers as they are or quantize only, and their tags,
// where they have any, from a byte per element.
template <int MODE, bool D3, bool BITS, bool FULL>
__device__ __forceinline__ void e64_front(const Enc64Args &a, long long tile, bool small, unsigned char *img, void *stage,
                                          E64Sh &sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int l = lane & 7, bi = tid >> 3;
  const long long n = (long long)a.n;
  const long long i0 = tile * kE64Tile + 8 * tid;   // local index of the octet
  const long long g0 = (long long)a.base + i0;       // its global index
  const long long bstart = tile * kE64Tile + 64 * bi;
  const int len = FULL ? 64 : (bstart >= n ? 0 : (n - bstart >= 64 ? 64 : (int)(n - bstart)));
  const int e0 = 8 * l;
  const int nv = FULL ? 8 : (len - e0 < 0 ? 0 : (len - e0 > 8 ? 8 : len - e0));

  // ---- values of the octet ----
  constexpr bool kTags = mode_tags(MODE), kFloats = MODE == kEncClassify || MODE == kEncQuant;
  float x[8];
  int q[8];
  unsigned tags = 0, cpm = 0, exm = 0;
  if (!kFloats) {
    if (nv == 8) {
      const int4 *pi = reinterpret_cast<const int4 *>(a.ints + i0);
      const int4 u = __ldg(pi), v = __ldg(pi + 1);
      q[0] = u.x; q[1] = u.y; q[2] = u.z; q[3] = u.w; q[4] = v.x; q[5] = v.y; q[6] = v.z; q[7] = v.w;
    } else {
#pragma unroll
      for (int t = 0; t < 8; t++) q[t] = t < nv ? __ldg(a.ints + i0 + t) : 0;
    }
    if (kTags && nv > 0) {
      // element t from bits 2t of the types to the t-th field from the top
      const unsigned ty = __brev(load_type_octet(a.types, i0, nv)) >> 16;
      tags = ((ty & 0x5555u) << 1) | ((ty >> 1) & 0x5555u);
    }
  } else if (nv == 8) {
    const float4 *px = reinterpret_cast<const float4 *>(a.data + g0);
    const float4 u = __ldg(px), v = __ldg(px + 1);
    x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
  } else {
#pragma unroll
    for (int t = 0; t < 8; t++) x[t] = t < nv ? __ldg(a.data + g0 + t) : 0.f;
  }
  if constexpr (MODE == kEncClassify) {
  // -0 as +0: the same quantized value, value code and comparisons
#pragma unroll
  for (int t = 0; t < 8; t++) x[t] = plus_zero(x[t]);

  // ---- interior mask (element 0 in bit 7): one coordinate split per octet ----
  unsigned inter = 0;
  bool wrap = false;
  if (small) {
    if (nv > 0) {
      unsigned r, z0, y, xx = 0;
      const unsigned d3 = (unsigned)a.g.d3;
      if (D3) {
        xx = divmod32((unsigned)g0, (unsigned)a.g.plane, a.g.m_plane, r);
        y = divmod32(r, d3, a.g.m_d3, z0);
      } else {
        y = divmod32((unsigned)g0, d3, a.g.m_d3, z0);
      }
      if (z0 + 7u < d3) {
        // a row's first and last columns, and its first and last rows and planes, are boundary
        const bool row_in = y - 1u < (unsigned)a.g.d2 - 2u && (!D3 || xx - 1u < (unsigned)a.g.d1 - 2u);
        inter = row_in ? (z0 ? 0xffu : 0x7fu) & (z0 + 8u == d3 ? 0xfeu : 0xffu) : 0u;
        if (!FULL) inter &= 0xff00u >> nv;
      } else {
        wrap = true;   // the octet crosses a row
        if (FULL && d3 > 8u) {
          // columns z0 .. d3-1 of a row, then 0 .. of the next
          const unsigned k = d3 - z0;                     // 1 .. 7
          const bool plane_in = !D3 || xx - 1u < (unsigned)a.g.d1 - 2u;
          if (plane_in && y - 1u < (unsigned)a.g.d2 - 2u) inter = ((1u << k) - 1u) >> 1;
          // (y + 2 < d2, not y < d2 - 2: one row a plane must not wrap)
          if (plane_in && y + 2u < (unsigned)a.g.d2) inter |= 0xffu & ~((2u << k) - 1u);
          inter = __brev(inter) >> 24;
        } else {
          inter = __brev(octet_interior(g0, nv, a.g)) >> 24;
        }
      }
    }
  } else if (nv > 0) {
    long long r, z0, y, xx = 0;
    if (D3) {
      xx = fdivmod(g0, a.g.plane, a.g.m_plane, r);
      y = fdivmod(r, a.g.d3, a.g.m_d3, z0);
    } else {
      y = fdivmod(g0, a.g.d3, a.g.m_d3, z0);
    }
    if (z0 + 7 < a.g.d3) {
      const bool row_in = y >= 1 && y <= a.g.d2 - 2 && (!D3 || (xx >= 1 && xx <= a.g.d1 - 2));
      if (row_in) {
        const long long lo = 1 - z0, hi = a.g.d3 - 2 - z0;
        const int ulo = lo > 0 ? (int)lo : 0, uhi = hi < 7 ? (int)hi : 7;
        if (ulo <= uhi) inter = ((2u << uhi) - 1u) & ~((1u << ulo) - 1u);
      }
      inter = __brev(inter & ((nv >= 8) ? 0xffu : ((1u << nv) - 1u))) >> 24;
    } else {
      wrap = true;
      inter = __brev(octet_interior(g0, nv, a.g)) >> 24;
    }
  }

  // ---- classification ----
  // +-1 along the row: the adjacent lanes' values (the warp covers 256
  // consecutive elements); the warp's end lanes load their outer neighbour
  float prev = __shfl_up_sync(0xffffffffu, x[7], 1);
  float next = __shfl_down_sync(0xffffffffu, x[0], 1);
  if (lane == 0 && (inter & 0x80u)) prev = plus_zero(__ldg(a.data + g0 - 1));
  if (lane == 31 && (inter & 1u)) next = plus_zero(__ldg(a.data + g0 + 8));
  if (__any_sync(0xffffffffu, inter != 0u)) {
    // edge j (0..8) joins element j-1 and j (element -1 = prev, 8 = next): bit 8 - j
    unsigned gt = 0, lt = 0;
    float cl = prev;
#pragma unroll
    for (int t = 0; t < 9; t++) {
      const float cr = t < 8 ? x[t < 8 ? t : 0] : next;
      lt = push_sign(__fsub_rn(cl, cr), lt);
      gt = push_sign(__fsub_rn(cr, cl), gt);
      cl = cr;
    }
    const unsigned hz = (lt >> 1) & gt, lz = (gt >> 1) & lt;
    unsigned ha = 0, la = 0, hb = 0, lb = 0;
    if (inter) {
      // vector loads when the octet lies in one row and the offset keeps the
      // 16-byte alignment; per-element loads otherwise
      const long long oa = D3 ? a.g.plane : a.g.d3;
      e64_axis(a.data, g0, oa, inter, !wrap && (oa & 3) == 0, x, ha, la);
      if (D3) e64_axis(a.data, g0, a.g.d3, inter, !wrap && (a.g.d3 & 3) == 0, x, hb, lb);
    }
    unsigned mx, mn, sd;
    if (D3) {
      mx = ha & hb & hz;
      mn = la & lb & lz & ~mx;
      sd = (ha | hb | hz) & (la | lb | lz) & ~mx & ~mn;
    } else {
      // rows are the vertical axis, the row direction the horizontal one
      mx = ha & hz;
      mn = la & lz & ~mx;
      sd = ((la & hz) | (ha & lz)) & ~mx & ~mn;
    }
    mx &= inter;
    mn &= inter;
    sd &= inter;
    cpm = mx | mn | sd;
    exm = mx | mn;
    // 2-bit types: maximum 01, minimum 10, saddle 11 (element 0 in the top two bits)
    tags = spread2(mx | sd) | (spread2(mn | sd) << 1);
  }
  }

  // ---- quantization and deltas ----
  if (kFloats) {
#pragma unroll
    for (int t = 0; t < 8; t++) q[t] = t < nv ? quantize(x[t], a.inv) : 0;
  }
  const int qn = __shfl_down_sync(0xffffffffu, q[0], 1, 8);
  const int cnt = len > 0 ? len - 1 : 0;
  unsigned sign = 0, maxm = 0, mags[8];
#pragma unroll
  for (int t = 0; t < 8; t++) {
    int d = (int)((unsigned)((t < 7) ? q[t + 1] : qn) - (unsigned)q[t]);
    if (FULL ? (t == 7 && l == 7) : e0 + t >= cnt) d = 0;
    sign = __funnelshift_l((unsigned)d, sign, 1);    // delta e0 + t at bit 7 - t
    mags[t] = (unsigned)(d < 0 ? 0u - (unsigned)d : (unsigned)d);
    maxm = mags[t] > maxm ? mags[t] : maxm;
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    const unsigned u = __shfl_xor_sync(0xffffffffu, maxm, o, 8);
    maxm = u > maxm ? u : maxm;
  }
  // below 2^16 log2f is off by less than its distance from the next integer
  const unsigned bc = maxm < 65536u ? 32u - (unsigned)__clz((int)maxm) : bitcount(maxm);
  const unsigned bbytes = FULL ? (kTags ? 21u : 5u) + (bc ? 8u + ((bc * 63u + 7u) >> 3) : 0u)
                               : (len ? block_bytes((unsigned)len, bc, kTags) : 0u);

  // ---- tile scans: block bytes, and points with extrema above them ----
  unsigned boff, cpo, exo;
  {
    // the eight lanes of a block hold its bytes: a scan over the warp's blocks
    unsigned ib = bbytes, u = __shfl_up_sync(0xffffffffu, ib, 8);
    if (lane >= 8) ib += u;
    u = __shfl_up_sync(0xffffffffu, ib, 16);
    if (lane >= 16) ib += u;
    const unsigned c = (unsigned)__popc(cpm) | ((unsigned)__popc(exm) << 16);
    unsigned ic = c;
    if (MODE == kEncClassify) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        u = __shfl_up_sync(0xffffffffu, ic, o);
        if (lane >= o) ic += u;
      }
    }
    if (lane == 31) { sh.wb[warp] = ib; sh.wc[warp] = ic; }
    // also the point after which every thread has left the image's last write-out
    e64_sync();
    unsigned sb = sh.wb[lane & 7], sc = sh.wc[lane & 7];
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const unsigned ub = __shfl_up_sync(0xffffffffu, sb, o, 8), uc = __shfl_up_sync(0xffffffffu, sc, o, 8);
      if ((lane & 7) >= o) { sb += ub; sc += uc; }
    }
    const unsigned tb = __shfl_sync(0xffffffffu, sb, 7), tc = __shfl_sync(0xffffffffu, sc, 7);
    unsigned pb = __shfl_sync(0xffffffffu, sb, (warp + 7) & 7), pc = __shfl_sync(0xffffffffu, sc, (warp + 7) & 7);
    if (warp == 0) { pb = 0u; pc = 0u; }
    boff = pb + ib - bbytes;
    pc += ic - c;
    cpo = pc & 0xffffu;
    exo = pc >> 16;
    if (tid == 0) {
      sh.tile_bytes = tb;
      sh.tile_cps = tc & 0xffffu;
      sh.tile_ext = tc >> 16;
      publish_aggregate(a.desc, tile, tb, ((unsigned long long)(tc & 0xffffu) << 32) | (tc >> 16));
    }
  }
  if (l == 0) sh.boff[bi] = boff;

  // ---- critical points, staged ----
  if (MODE == kEncClassify && cpm) {
    if (BITS) {
      unsigned *st = static_cast<unsigned *>(stage);
      unsigned ei = exo, si = kE64Tile - 1u - (cpo - exo);
#pragma unroll
      for (int t = 0; t < 8; t++) {
        if ((cpm >> (7 - t)) & 1u) {
          const bool ext = (exm >> (7 - t)) & 1u;
          st[ext ? ei : si] = value_code(x[t]);
          if (ext) ei++; else si--;
        }
      }
    } else {
      uint2 *st = static_cast<uint2 *>(stage);
      unsigned ci = cpo, ei = exo;
#pragma unroll
      for (int t = 0; t < 8; t++) {
        if ((cpm >> (7 - t)) & 1u) {
          const bool ext = (exm >> (7 - t)) & 1u;
          st[ci++] = make_uint2(value_code(x[t]), ext ? ei : kNoExtremum);
          ei += ext ? 1u : 0u;
        }
      }
    }
  }

  // ---- pack the octet into the tile image ----
  if (FULL || nv > 0) {
    unsigned p = boff;
    if (l == 0) {
      const unsigned an = (unsigned)q[0];
      img[p] = (unsigned char)an;
      img[p + 1] = (unsigned char)(an >> 8);
      img[p + 2] = (unsigned char)(an >> 16);
      img[p + 3] = (unsigned char)(an >> 24);
      if (FULL || len > 1) img[p + 4] = (unsigned char)bc;
    }
    p += 4;
    if (FULL || len > 1) {
      p += 1;
      if (bc) {
        const unsigned sbytes = FULL ? 8u : (unsigned)(cnt + 7) / 8u;
        const unsigned ucnt = FULL ? 63u : (unsigned)cnt;
        const bool has_d = FULL || e0 < cnt;
        if (has_d) img[p + l] = (unsigned char)sign;
        p += sbytes;
        const unsigned fb = bc >> 3, rem = bc & 7u;
        if (has_d) {
          if (fb == 1) {
#pragma unroll
            for (int t = 0; t < 8; t++)
              if (FULL ? (t < 7 || l < 7) : e0 + t < cnt)
                img[p + (unsigned)(e0 + t)] = (unsigned char)(mags[t] >> rem);
          } else if (fb >= 2) {
#pragma unroll
            for (int t = 0; t < 8; t++) {
              if (e0 + t < (int)ucnt) {
                unsigned v = mags[t] >> rem;
                const unsigned o = p + (unsigned)(e0 + t) * fb;
                for (unsigned u = 0; u < fb; u++) { img[o + u] = (unsigned char)v; v >>= 8; }
              }
            }
          }
        }
        p += fb * ucnt;
        if (rem) {
          // a full block's 63 fields leave less than a byte unused: 8 rem bytes
          const unsigned rbytes = FULL ? 8u * rem : (rem * ucnt - 1u) / 8u + 1u;
          if (has_d) {
            // the octet's 8 rem bits, left-aligned in hi:lo: exactly rem bytes at byte l * rem
            const unsigned mask = (1u << rem) - 1u;
            unsigned h = mags[0] & mask, w = mags[4] & mask;
#pragma unroll
            for (int t = 1; t < 4; t++) {
              h = (h << rem) | (mags[t] & mask);
              w = (w << rem) | (mags[4 + t] & mask);
            }
            const unsigned up = 32u - 4u * rem;      // 4 .. 28
            h <<= up;
            w <<= up;
            const unsigned hi = h | (w >> (4u * rem)), lo = w << (32u - 4u * rem);
            const unsigned ob = p + (unsigned)l * rem, room = FULL ? rem : (rbytes > (unsigned)l * rem ? min(rem, rbytes - (unsigned)l * rem) : 0u);
#pragma unroll
            for (unsigned u = 0; u < 7; u++)
              if (u < room) img[ob + u] = (unsigned char)(u < 4 ? hi >> (24u - 8u * u) : lo >> (56u - 8u * u));
          }
          p += rbytes;
        }
      }
    }
    // tag byte j: elements 4j .. 4j+3, element 4j in the top two bits
    const unsigned tb = ((unsigned)len + 3u) / 4u;
    if (kTags && (FULL || 2u * l < tb)) img[p + 2 * l] = (unsigned char)(tags >> 8);
    if (kTags && (FULL || 2u * l + 1u < tb)) img[p + 2 * l + 1] = (unsigned char)tags;
  }
}

// Look-back of a tile by one warp, four predecessors per lane and round.
// Publishes the inclusive prefix.
__device__ __forceinline__ Prefix e64_lookback(TileDesc *desc, long long t, unsigned long long agg_bytes,
                                               unsigned long long agg_cnt, int *err, int spin_limit) {
  const int lane = threadIdx.x & 31;
  const int limit = spin_limit > 0 ? spin_limit : kSpinLimit;
  Prefix ex{0ull, 0ull};
  if (t > 0) {
    bool timed_out = false, found = false;
    for (long long base = t - 1; !found; base -= 128) {
      unsigned long long st[4], ct[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const long long idx = base - 32 * u - lane;
        st[u] = 2ull << kStatShift;
        ct[u] = 0;
        if (idx >= 0) desc_read(desc + idx, st[u], ct[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const long long idx = base - 32 * u - lane;
        if (!found) {
          int spins = 0;
          while ((st[u] >> kStatShift) == 0ull) {
            if (++spins > limit) { timed_out = true; break; }
            __nanosleep(spins < 64 ? 32 : 256);
            desc_read(desc + idx, st[u], ct[u]);
          }
          unsigned long long flag = st[u] >> kStatShift;
          if (flag == 0ull) flag = 2ull;   // timed out: an empty inclusive value
          const unsigned m = __ballot_sync(0xffffffffu, flag == 2ull);
          const int first = m ? __ffs(m) - 1 : 32;
          if (lane <= first) {
            ex.bytes += st[u] & kByteMask;
            ex.cnt += ct[u];
          }
          found = m != 0u;
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ex.bytes += __shfl_xor_sync(0xffffffffu, ex.bytes, o);
      ex.cnt += __shfl_xor_sync(0xffffffffu, ex.cnt, o);
    }
    if (timed_out) atomicExch(err, kErrLookbackTimeout);
  }
  if (lane == 0) desc_publish(desc + t, 2ull, ex.bytes + agg_bytes, ex.cnt + agg_cnt);
  return ex;
}

// Back half of a tile, its place known: block index, write-out of the image
// and of the staged critical points.  The threads that own elements call it.
template <bool BITS>
__device__ __forceinline__ void e64_back(const Enc64Args &a, long long tile, const unsigned char *img,
                                         const void *stage, const E64Sh &sh, unsigned &nmax, unsigned &cmax,
                                         unsigned &seen) {
  const int tid = threadIdx.x;
  const long long n = (long long)a.n;
  const long long nblocks = (n + 63) / 64;
  const unsigned tile_bytes = sh.tile_bytes;
  const unsigned long long G0 = sh.gbyte;
  const bool fits = (G0 + tile_bytes) <= a.out_cap;
  if (!fits && tid == 0) atomicExch(a.err, kErrOutputOverflow);
  if (a.blk_off && tid < kE64Blocks) {
    const long long b = tile * kE64Blocks + tid;
    if (b < nblocks) a.blk_off[b] = G0 + sh.boff[tid];
  }
  // write-out: aligned 16-byte stores in the middle
  if (fits && tile_bytes) {
    const uint32_t *imgw = reinterpret_cast<const uint32_t *>(img);
    unsigned char *dst = a.out + G0;
    unsigned head = (unsigned)((16u - (unsigned)(reinterpret_cast<uintptr_t>(dst) & 15u)) & 15u);
    if (head > tile_bytes) head = tile_bytes;
    if ((unsigned)tid < head) dst[tid] = img[tid];
    const unsigned nq = (tile_bytes - head) >> 4;
    const unsigned shb = 8u * (head & 3u);
    const unsigned w0 = head >> 2;
    uint4 *dq = reinterpret_cast<uint4 *>(dst + head);
    for (unsigned qd = tid; qd < nq; qd += kE64Threads) {
      const unsigned wi = w0 + 4u * qd;
      uint4 v;
      if (shb) {
        v.x = __funnelshift_r(imgw[wi], imgw[wi + 1], shb);
        v.y = __funnelshift_r(imgw[wi + 1], imgw[wi + 2], shb);
        v.z = __funnelshift_r(imgw[wi + 2], imgw[wi + 3], shb);
        v.w = __funnelshift_r(imgw[wi + 3], imgw[wi + 4], shb);
      } else {
        v.x = imgw[wi]; v.y = imgw[wi + 1]; v.z = imgw[wi + 2]; v.w = imgw[wi + 3];
      }
      dq[qd] = v;
    }
    const unsigned t0b = head + 16u * nq;
    if (t0b + tid < tile_bytes) dst[t0b + tid] = img[t0b + tid];
  }
  const unsigned long long cb = sh.gcnt >> 32, eb0 = sh.gcnt & 0xffffffffull;
  const unsigned ntc = sh.tile_cps, nte = sh.tile_ext;
  if (BITS) {
    // every value's bit; the codes of the extrema, and those of the saddles, in
    // raster order: what the bucket ranking takes where the bits do not do
    if (cb + ntc > a.cp_cap) {
      if (tid == 0) atomicExch(a.err, kErrCapacity);
    } else {
      const unsigned *st = static_cast<const unsigned *>(stage);
      unsigned *eo = a.code_out + eb0, *so = a.code_out + a.cp_cap + (cb - eb0) - nte;
      const bool head = cb < kRankSmall;
      for (unsigned k = tid; k < ntc; k += kE64Threads) {
        const bool is_ext = k < nte;
        const unsigned code = st[is_ext ? k : kE64Tile - 1u + nte - k];
        const unsigned ext = is_ext ? (unsigned)eb0 + k : kNoExtremum;
        rb_set(a.rb, code, ext, seen);
        if (head && cb + k < kRankSmall) a.rb.first[cb + k] = make_uint2(code, ext);
        nmax = max(nmax, ~code);
        cmax = max(cmax, code);
        (is_ext ? eo : so)[k] = code;
      }
    }
  } else {
    // critical-point pairs in raster order
    const uint2 *st = static_cast<const uint2 *>(stage);
    uint2 *cp = a.cp_out;
    for (unsigned k = tid; k < ntc; k += kE64Threads) {
      if (cb + k < a.cp_cap) {
        uint2 pr = st[k];
        if (pr.y != kNoExtremum) pr.y += (unsigned)eb0;
        cp[cb + k] = pr;
      }
    }
    if (tid == 0 && cb + ntc > a.cp_cap) atomicExch(a.err, kErrCapacity);
  }
}

// The ninth warp's part of a tile: its place, and the totals after the last one.
__device__ __forceinline__ void e64_place(const Enc64Args &a, long long tile, E64Sh &sh) {
  const unsigned tb = sh.tile_bytes, tc = sh.tile_cps, te = sh.tile_ext;
  const Prefix pf = e64_lookback(a.desc, tile, tb, ((unsigned long long)tc << 32) | te, a.err, a.spin_limit);
  if ((threadIdx.x & 31) == 0) {
    sh.gbyte = pf.bytes;
    sh.gcnt = pf.cnt;
    if (tile == ((long long)a.n + kE64Tile - 1) / kE64Tile - 1 && a.total) {
      a.total[0] = pf.bytes + tb;
      a.total[1] = (pf.cnt >> 32) + tc;
      a.total[2] = (pf.cnt & 0xffffffffull) + te;
    }
  }
}

// Persistent CTAs claim tiles in order.  Eight warps own the elements and keep
// two images: they run one tile behind (the front half of tile k, whose
// aggregate is published in it, then the write-out of tile k-1).  A ninth warp
// claims the tiles and looks back for tile k-1 while the others are in the
// front half of tile k.
// A look-back waits for the aggregates of earlier tiles only, and a tile's
// aggregate waits, through its CTA's barrier, for look-backs of earlier tiles
// only, so the waits cannot form a cycle.
template <int MODE, bool D3, bool BITS>
__global__ void __launch_bounds__(kE64Cta, 4) enc64_kernel(Enc64Args a) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  __shared__ E64Sh sh[2];
  __shared__ long long s_claim[2];
  constexpr unsigned kPart = e64_part(MODE, BITS);
  const long long ntiles = ((long long)a.n + kE64Tile - 1) / kE64Tile;
  const long long nfull = (long long)a.n / kE64Tile;
  const long long tend = a.tile_hi ? (long long)a.tile_hi : ntiles;
  const bool owner = threadIdx.x < kE64Threads;
  // flat indices and extents of the field in 32 bits
  const bool small = a.g.d1 * a.g.plane < (1ll << 32);
  long long prev = -1;
  int cur = 0;
  unsigned nmax = 0, cmax = 0, seen = 0;
  while (true) {
    // claimed only now (while the other warps write the last tile out), not a
    // tile ahead: every look-back behind a claimed tile waits for its front half
    long long tile;
    if (owner) {
      e64_claim_wait();
      tile = s_claim[cur];
    } else {
      tile = 0;
      if (threadIdx.x == kE64Threads) tile = (long long)a.tile_lo + (long long)atomicAdd(a.tile_ctr, 1u);
      tile = __shfl_sync(0xffffffffu, tile, 0);
      if (threadIdx.x == kE64Threads) s_claim[cur] = tile;
      __syncwarp();
      e64_claim_post();
    }
    const bool more = tile < tend;
    if (owner) {
      unsigned char *part = smem_dyn + (size_t)cur * kPart;
      if (more) {
        if (tile < nfull) e64_front<MODE, D3, BITS, true>(a, tile, small, part, part + kE64Img, sh[cur]);
        else e64_front<MODE, D3, BITS, false>(a, tile, small, part, part + kE64Img, sh[cur]);
      }
    } else {
      if (prev >= 0) e64_place(a, prev, sh[cur ^ 1]);
    }
    __syncthreads();
    if (owner && prev >= 0) {
      const unsigned char *pp = smem_dyn + (size_t)(cur ^ 1) * kPart;
      e64_back<BITS>(a, prev, pp, pp + kE64Img, sh[cur ^ 1], nmax, cmax, seen);
    }
    if (!more) break;
    prev = tile;
    cur ^= 1;
  }
  if (BITS && owner) rb_extent(a.rb, nmax, cmax);
}

// The fields of a batch.  The ninth warp maps a claim to its field (the claims
// of a CTA only move forward) and leaves the field's arguments in shared
// memory, three tiles' worth: the tile being claimed, the one before it and
// the one that is still written out.
__global__ void __launch_bounds__(kE64Cta, 4)
enc64_batch_kernel(const EncArgs *__restrict__ fields, const unsigned long long *__restrict__ tstart,
                   const unsigned *__restrict__ nfields_dev, unsigned *queue) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  __shared__ E64Sh sh[2];
  __shared__ Enc64Args s_args[3];
  __shared__ long long s_claim[3];
  constexpr unsigned kPart = e64_part(false);
  const int nf = (int)*nfields_dev;
  const unsigned long long total = tstart[nf];
  const bool owner = threadIdx.x < kE64Threads;
  const int lane = threadIdx.x & 31;
  int field = 0, have[3] = {-1, -1, -1};
  bool pending = false;
  unsigned unused0 = 0, unused1 = 0, unused2 = 0;
  for (int it = 0, cur = 0, slot = 0;; it++, cur ^= 1) {
    const int before = slot == 0 ? 2 : slot - 1;
    if (owner) {
      e64_claim_wait();
    } else {
      unsigned long long t = 0;
      if (lane == 0) t = atomicAdd(queue, 1u);
      t = __shfl_sync(0xffffffffu, t, 0);
      if (t < total) {
        // the last field that starts at or before t, 32 fields a step from the last claim's
        while (true) {
          const int i = field + 1 + lane;
          const unsigned m = __ballot_sync(0xffffffffu, i < nf && tstart[i < nf ? i : nf] <= t);
          field += __popc(m);      // starts ascend: the set lanes are the first ones
          if (m != 0xffffffffu) break;
        }
        if (lane == 0) {
          if (have[slot] != field) {
            const EncArgs &e = fields[field];
            Enc64Args &a = s_args[slot];
            a.data = e.data;
            a.n = e.n;
            a.inv = e.inv;
            a.g = e.g;
            a.out = e.out;
            a.out_cap = e.out_cap;
            a.blk_off = e.blk_off;
            a.desc = e.desc;
            a.err = e.err;
            a.total = e.total;
            a.cp_out = reinterpret_cast<uint2 *>(e.cp_out);
            a.cp_cap = e.cp_cap;
            a.spin_limit = 0;
            a.base = 0;
          }
          s_claim[slot] = (long long)(t - tstart[field]);
        }
#pragma unroll
        for (int k = 0; k < 3; k++)
          if (k == slot) have[k] = field;
      } else if (lane == 0) {
        s_claim[slot] = -1;
      }
      __syncwarp();
      e64_claim_post();
    }
    const long long tile = s_claim[slot];
    if (owner) {
      if (tile >= 0) {
        const Enc64Args &a = s_args[slot];
        const bool small = a.g.d1 * a.g.plane < (1ll << 32), full = tile < (long long)(a.n / kE64Tile);
        unsigned char *part = smem_dyn + (size_t)cur * kPart;
        if (a.g.nd == 3) {
          if (full) e64_front<kEncClassify, true, false, true>(a, tile, small, part, part + kE64Img, sh[cur]);
          else e64_front<kEncClassify, true, false, false>(a, tile, small, part, part + kE64Img, sh[cur]);
        } else {
          if (full) e64_front<kEncClassify, false, false, true>(a, tile, small, part, part + kE64Img, sh[cur]);
          else e64_front<kEncClassify, false, false, false>(a, tile, small, part, part + kE64Img, sh[cur]);
        }
      }
    } else if (pending) {
      e64_place(s_args[before], s_claim[before], sh[cur ^ 1]);
    }
    __syncthreads();
    if (owner && pending) {
      const unsigned char *pp = smem_dyn + (size_t)(cur ^ 1) * kPart;
      e64_back<false>(s_args[before], s_claim[before], pp, pp + kE64Img, sh[cur ^ 1], unused0, unused1,
                      unused2);
    }
    if (tile < 0) break;
    pending = true;
    slot = slot == 2 ? 0 : slot + 1;
  }
}

cudaError_t enc64_batch_prepare(int *per_sm) {
  const int smem = 2 * (int)e64_part(false);
  cudaError_t e = cudaFuncSetAttribute(enc64_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, enc64_batch_kernel, kE64Cta, smem);
  return e;
}

cudaError_t launch_enc64_batch(const EncArgs *fields, const unsigned long long *tstart, const unsigned *nfields_dev,
                               unsigned *queue, cudaStream_t s, int grid) {
  enc64_batch_kernel<<<grid, kE64Cta, 2 * e64_part(false), s>>>(fields, tstart, nfields_dev, queue);
  return cudaGetLastError();
}

unsigned long long enc64_tiles(unsigned long long n) { return (n + kE64Tile - 1) / kE64Tile; }

static cudaError_t launch_enc64(int mode, const Enc64Args &a, cudaStream_t s, int sm_count) {
  const size_t smem = 2 * (size_t)e64_part(mode, a.code_out != nullptr);
  const bool d3 = a.g.nd == 3;
  auto k = mode == kEncInts       ? enc64_kernel<kEncInts, false, false>
           : mode == kEncIntTypes ? enc64_kernel<kEncIntTypes, false, false>
           : mode == kEncQuant    ? enc64_kernel<kEncQuant, false, false>
           : a.code_out           ? (d3 ? enc64_kernel<kEncClassify, true, true> : enc64_kernel<kEncClassify, false, true>)
                                  : (d3 ? enc64_kernel<kEncClassify, true, false> : enc64_kernel<kEncClassify, false, false>);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kE64Cta, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  const unsigned long long ntiles = enc64_tiles(a.n);
  const unsigned long long hi = a.tile_hi ? a.tile_hi : ntiles;
  const unsigned long long span = hi > a.tile_lo ? hi - a.tile_lo : 0;
  unsigned long long grid = (unsigned long long)sm_count * per_sm;
  if (grid > span) grid = span;
  if (grid < 1) grid = 1;
  k<<<(unsigned)grid, kE64Cta, smem, s>>>(a);
  return cudaGetLastError();
}

// Bounded-wait check of the look-back: a two-tile field encoded from tile 1
// on, so tile 0 never publishes and tile 1's look-back must give up after
// spin_limit polls, report kErrLookbackTimeout and finish its write-out (at
// offset 0 of the output, inside its capacity).
int selftest_lookback(int spin_limit, int *status, float *ms) {
  const unsigned long long n = 2 * kE64Tile;
  const size_t cap = 2 * kE64Img;
  unsigned char *buf = nullptr;
  const size_t bytes = n * 4 + cap + 2 * sizeof(TileDesc) + kE64Tile * sizeof(uint2) + 256;
  if (cuda_fail(cudaMalloc(&buf, bytes), "cudaMalloc")) return -1;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int rc = -1;
  if (!cuda_fail(cudaMemset(buf, 0, bytes), "memset") && !cuda_fail(cudaEventCreate(&e0), "event") &&
      !cuda_fail(cudaEventCreate(&e1), "event")) {
    Enc64Args a{};
    a.data = reinterpret_cast<const float *>(buf);
    a.n = n;
    a.inv = 1.0e3;
    a.g = make_geom(2, 64, (long long)n / 64, 1);
    a.out = buf + n * 4;
    a.out_cap = cap;
    a.desc = reinterpret_cast<TileDesc *>(buf + n * 4 + cap);
    a.cp_out = reinterpret_cast<uint2 *>(buf + n * 4 + cap + 2 * sizeof(TileDesc));
    a.cp_cap = kE64Tile;
    unsigned long long *w = reinterpret_cast<unsigned long long *>(buf + bytes - 64);
    a.tile_ctr = reinterpret_cast<unsigned *>(w);
    a.err = reinterpret_cast<int *>(w + 1);
    a.total = w + 2;
    a.tile_lo = 1;
    a.tile_hi = 2;
    a.spin_limit = spin_limit;
    cudaEventRecord(e0, 0);
    const cudaError_t le = launch_enc64(kEncClassify, a, 0, 1);
    cudaEventRecord(e1, 0);
    int h = 0;
    if (!cuda_fail(le, "probe launch") && !cuda_fail(cudaMemcpy(&h, a.err, 4, cudaMemcpyDeviceToHost), "D2H")) {
      cudaEventElapsedTime(ms, e0, e1);
      *status = h;
      rc = 0;
    }
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFree(buf);
  return rc;
}

bool enc64_applies(const EncArgs &a, int mode) {
  if (a.B != 64 || a.out == nullptr || enc_tile_blocks(64) != kE64Blocks) return false;
  const void *in = a.data;
  if (mode == kEncClassify) {
    if (a.cp_mode != kCpPairs && a.cp_mode != kCpBits) return false;
  } else if (mode == kEncInts || mode == kEncIntTypes) {
    in = a.ints;
  } else if (mode != kEncQuant) {
    return false;
  }
  return (reinterpret_cast<uintptr_t>(in) & 15) == 0;
}

cudaError_t launch_enc64_args(const Enc64Args &a, cudaStream_t s, int sm_count) {
  return launch_enc64(kEncClassify, a, s, sm_count);
}

cudaError_t launch_enc64_from(int mode, const EncArgs &e, cudaStream_t s, int sm_count) {
  Enc64Args a{};
  a.data = e.data;
  a.n = e.n;
  a.inv = e.inv;
  a.g = e.g;
  a.out = e.out;
  a.out_cap = e.out_cap;
  a.blk_off = e.blk_off;
  a.desc = e.desc;
  a.tile_ctr = e.tile_ctr;
  a.tile_lo = e.tile_lo;
  a.tile_hi = e.tile_hi;
  a.err = e.err;
  a.total = e.total;
  if (e.cp_mode == kCpBits) {
    a.code_out = reinterpret_cast<unsigned *>(e.cp_out);
    a.rb = e.rb;
  } else {
    a.cp_out = reinterpret_cast<uint2 *>(e.cp_out);
  }
  a.cp_cap = e.cp_cap;
  a.spin_limit = 0;
  a.ints = e.ints;
  a.types = e.types;
  return launch_enc64(mode, a, s, sm_count);
}

}  // namespace tsz

using namespace tsz;

extern "C" SZP_B200_API int szp_b200_selftest_bounded_wait(int which, int spin_limit, int *status, float *ms) {
  clear_error();
  if (!status || !ms) { set_error("szp_b200_selftest_bounded_wait: null argument"); return -1; }
  if (spin_limit < 1 || spin_limit > (1 << 20)) {
    set_error("szp_b200_selftest_bounded_wait: spin_limit must lie in [1, 2^20]");
    return -1;
  }
  *status = 0;
  *ms = 0.f;
  if (which == 0) return selftest_lookback(spin_limit, status, ms);
  if (which == 1) return selftest_grid_barrier(spin_limit, status, ms);
  set_error("szp_b200_selftest_bounded_wait: which must be 0 (look-back) or 1 (grid barrier)");
  return -1;
}
