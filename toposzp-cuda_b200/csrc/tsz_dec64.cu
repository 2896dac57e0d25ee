// Block decoder for blockSize 64 (topology, sort-position and plain streams).
//
// Same values as the octet decoder (tsz_codec2.cuh; SZp/src/
// szp_cuda_decompress.cu:673-741), which is bound by instruction issue: 92
// instructions per element, at 1.9 TB/s.  Eight lanes decode a block, eight
// values each, as there; what is left out or cheaper:
//   * a value past a block's last delta is decoded from whatever follows it and
//     goes nowhere (it could only reach elements that do not exist), so no value
//     has a bound check of its own;
//   * the remainder fields of an octet are a 64-bit big-endian window, four
//     fields in each of two words, moved to the top by a multiply;
//   * a block's offsets, length, bit count and checks are worked out by one
//     lane of the CTA's first warp, not by the eight that decode it, and a CTA
//     of full blocks has no length of its own anywhere (512^3: 316 -> 262 us
//     for the stage, ALU pipe 76 % busy before);
//   * signs multiply: q[t + 1] = q[t] + magnitude * (+1 or -1), one multiply-add
//     per value on the FMA pipe, which also is the octet's prefix sum;
//   * blocks with full magnitude bytes beyond one take the byte loop.
#include "tsz_codec.h"
#include "tsz_codec2.cuh"

namespace tsz {

// Sixteen CTAs of 128 threads per SM (32 registers): a CTA waits for its image
// and for its blocks' fields with nothing of its own to do meanwhile.  Decode
// stage of 512^3: 223 us; 260 with 6 x 256 threads (40 registers), 231 with
// 8 x 256, 245 with 12 x 128, 261 with 32 x 64; 275 when 16 CTAs per SM loop
// over the tiles (spills).
constexpr int kD64Threads = 128;
constexpr int kD64Blocks = kD64Threads / 8;

// The image of a CTA's blocks.  Twice what its sixteen blocks can take: an
// index of the caller's may leave bytes between blocks, as many as the octet
// decoder's tile of 32 blocks has room for.  The sixteen CTAs of an SM hold
// 170 KB so, and take as long as with half of it (512^3: 1340 against 1339 us).
constexpr unsigned kD64ImgBlocks = 32;
__host__ __device__ constexpr unsigned d64_img_bytes(bool tags) {
  return (kD64ImgBlocks * (tags ? 289u : 273u) + 64u + 15u) & ~15u;
}

// the 8 bytes at image position p, as two little-endian words
__device__ __forceinline__ void ld_window(const unsigned *imgw, unsigned p, unsigned &lo, unsigned &hi) {
  const unsigned wi = p >> 2, sh = 8u * (p & 3u);
  const unsigned a = imgw[wi], b = imgw[wi + 1], c = imgw[wi + 2];
  lo = __funnelshift_r(a, b, sh);
  hi = __funnelshift_r(b, c, sh);
}

// x >> n for n <= 32 (zero at 32)
__device__ __forceinline__ unsigned shr_clamp(unsigned x, unsigned n) {
  unsigned r;
  asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
  return r;
}

constexpr unsigned kD64Ok = 0x10000u;

// A block as its warp of the CTA found it: x: image position of its block, y:
// anchor, z: image position of its types, w: bit count, kD64Ok.
// FULL: the block has 64 elements.
template <bool TAGS, bool FULL>
__device__ __forceinline__ unsigned d64_octet(const DecArgs &a, const unsigned char *img, const uint4 &h,
                                              long long base, int len, int l) {
  const unsigned *imgw = reinterpret_cast<const unsigned *>(img);
  const bool ok = (h.w & kD64Ok) != 0;
  const unsigned bc = h.w & 0xffu;
  const int e0 = 8 * l;
  const int nv = FULL ? 8 : (len - e0 < 0 ? 0 : (len - e0 > 8 ? 8 : len - e0));
  const unsigned cnt = FULL ? 63u : (len > 0 ? (unsigned)len - 1u : 0u);
  // q[t]: sum of the octet's deltas before element t; q[8]: of all of them
  int q[9];
#pragma unroll
  for (int t = 0; t < 9; t++) q[t] = 0;
  if (ok && bc && (FULL || (unsigned)e0 < cnt)) {
    const unsigned p = h.x + 5u, sbytes = (cnt + 7u) >> 3;
    const unsigned neg = (unsigned)img[p + l] << 24;     // sign of delta e0 + t at bit 31 - t
    const unsigned mag = p + sbytes, fb = bc >> 3, rem = bc & 7u;
    // rem bytes at byte l rem of the remainder section, most significant bits
    // first: fields 0 .. 3 on top of w0, 4 .. 7 of w1 (28 bits or fewer each)
    unsigned rl, rh;
    ld_window(imgw, mag + fb * cnt + (unsigned)l * rem, rl, rh);
    const unsigned w0 = __byte_perm(rl, 0u, 0x0123);
    const unsigned w1 = __funnelshift_l(__byte_perm(rh, 0u, 0x0123), w0, 4u * rem);
    const unsigned down = 32u - rem, up = 1u << rem;     // no field when rem is 0: a shift by 32
    const unsigned ups[4] = {1u, up, up * up, up * up * up};
    if (fb <= 1) {
      unsigned fl = 0, fh = 0;
      if (fb) ld_window(imgw, mag + (unsigned)e0, fl, fh);
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const unsigned full = __byte_perm(t < 4 ? fl : fh, 0u, 0x4440u + (unsigned)(t & 3));
        const unsigned m = full * up + shr_clamp((t < 4 ? w0 : w1) * ups[t & 3], down);
        q[t + 1] = (int)(m * (unsigned)(((int)(neg << t) >> 31) | 1) + (unsigned)q[t]);
      }
    } else {
#pragma unroll
      for (int t = 0; t < 8; t++) {
        unsigned full = 0;
        if ((unsigned)(e0 + t) < cnt) {
          const unsigned o = mag + (unsigned)(e0 + t) * fb;
          for (unsigned u = 0; u < fb; u++) full |= (unsigned)img[o + u] << (8u * u);
        }
        const unsigned m = full * up + shr_clamp((t < 4 ? w0 : w1) * ups[t & 3], down);
        q[t + 1] = (int)(m * (unsigned)(((int)(neg << t) >> 31) | 1) + (unsigned)q[t]);
      }
    }
  }
  // exclusive scan of the octet sums over the block's lanes
  int inc = q[8];
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o, 8);
    if (l >= o) inc = (int)((unsigned)inc + (unsigned)u);
  }
  if (!ok || nv == 0) return 0u;
  const int v0 = (int)(h.y + (unsigned)inc - (unsigned)q[8]);
#pragma unroll
  for (int t = 0; t < 8; t++) q[t] = (int)((unsigned)q[t] + (unsigned)v0);
  const long long i0 = base + e0;
  if (a.out_f) {
    float f[8];
#pragma unroll
    for (int t = 0; t < 8; t++) f[t] = __fmul_rn((float)q[t], a.eb);
    // i0 is a multiple of 8: the array's alignment decides
    if (nv == 8 && ((reinterpret_cast<uintptr_t>(a.out_f) & 15) == 0)) {
      reinterpret_cast<float4 *>(a.out_f + i0)[0] = make_float4(f[0], f[1], f[2], f[3]);
      reinterpret_cast<float4 *>(a.out_f + i0)[1] = make_float4(f[4], f[5], f[6], f[7]);
    } else {
#pragma unroll
      for (int t = 0; t < 8; t++) if (t < nv) a.out_f[i0 + t] = f[t];
    }
  }
  if (!TAGS && a.out_i) {
    if (nv == 8 && ((reinterpret_cast<uintptr_t>(a.out_i) & 15) == 0)) {
      reinterpret_cast<int4 *>(a.out_i + i0)[0] = make_int4(q[0], q[1], q[2], q[3]);
      reinterpret_cast<int4 *>(a.out_i + i0)[1] = make_int4(q[4], q[5], q[6], q[7]);
    } else {
#pragma unroll
      for (int t = 0; t < 8; t++) if (t < nv) a.out_i[i0 + t] = q[t];
    }
  }
  if (!TAGS) return 0u;
  const unsigned tb = FULL ? 16u : ((unsigned)len + 3u) / 4u;
  // element 0 in the top two of 16 bits; elements past nv as regular points
  unsigned tg = ((FULL || 2u * l < tb) ? (unsigned)img[h.z + 2 * l] << 8 : 0u) |
                ((FULL || 2u * l + 1u < tb) ? (unsigned)img[h.z + 2 * l + 1] : 0u);
  if (!FULL && nv < 8) tg &= 0xffffu << (16 - 2 * nv);
  if (a.pl_lo) {
    // element t to bit t: low bits compacted in the lower half, high bits in
    // the upper, element 0 on top; all reversed
    unsigned x = (tg & 0x5555u) | ((tg & 0xaaaau) << 15);
    x = (x | (x >> 1)) & 0x33333333u;
    x = (x | (x >> 2)) & 0x0f0f0f0fu;
    x = __brev((x | (x >> 4)) & 0x00ff00ffu);
    const long long o = i0 >> 3;
    a.pl_lo[o] = (unsigned char)(x >> 24);
    a.pl_hi[o] = (unsigned char)(x >> 8);
    // the rest of the planes' last word
    if (!FULL && i0 + 8 >= (long long)a.n)
      for (long long k = o + 1; k & 3; k++) a.pl_lo[k] = a.pl_hi[k] = 0;
  }
  if (a.fn_u8) {
    if (nv == 8 && ((reinterpret_cast<uintptr_t>(a.fn_u8) & 7) == 0)) {
      // four two-bit fields of a byte, most significant first, to four bytes
      unsigned w[2];
#pragma unroll
      for (int hf = 0; hf < 2; hf++) {
        const unsigned x = hf ? tg & 0xffu : tg >> 8;
        const unsigned y = (x | (x << 12)) & 0x000f000fu;        // low nibble, high nibble << 16
        const unsigned z = (y | (y << 6)) & 0x03030303u;         // fields 3, 2 (low to high byte), 1, 0
        w[hf] = __byte_perm(z, 0u, 0x0123);
      }
      *reinterpret_cast<uint2 *>(a.fn_u8 + i0) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
      for (int t = 0; t < 8; t++) if (t < nv) a.fn_u8[i0 + t] = (unsigned char)((tg >> (14 - 2 * t)) & 3u);
    }
  }
  if (a.fn_i) {
#pragma unroll
    for (int t = 0; t < 8; t++) if (t < nv) a.fn_i[i0 + t] = (int)((tg >> (14 - 2 * t)) & 3u);
  }
  return (unsigned)__popc((tg ^ (tg >> 1)) & 0x5555u);   // types 01 and 10
}

template <bool TAGS>
__global__ void __launch_bounds__(kD64Threads, 16) decode64_kernel(DecArgs a) {
  __shared__ __align__(16) unsigned char img[d64_img_bytes(TAGS) + 32];
  __shared__ uint4 s_hd[kD64Blocks];
  const int tid = threadIdx.x, l = tid & 7, bi = tid >> 3;
  const long long n = (long long)a.n;
  const long long nblocks = (n + 63) / 64;
  const long long b0 = (long long)blockIdx.x * kD64Blocks;
  const int nb = (int)((nblocks - b0) < kD64Blocks ? (nblocks - b0) : kD64Blocks);
  // the image holds the payload bytes from the 16-byte boundary at or below
  // payload + lo: img[ib + k] is payload[lo + k]
  const unsigned long long lo = a.blk_off[b0];
  const unsigned long long end = b0 + nb < nblocks ? a.blk_off[b0 + nb] : a.payload_len;
  const unsigned long long hi = end > a.payload_len ? a.payload_len : end;
  unsigned long long o0 = 0, o1 = 0;
  if (tid < nb) {
    o0 = a.blk_off[b0 + tid];
    o1 = b0 + tid + 1 < nblocks ? a.blk_off[b0 + tid + 1] : a.payload_len;
  }
  if (lo > hi || hi - lo > d64_img_bytes(TAGS) - 48u) {
    if (tid == 0) atomicExch(a.err, kErrMalformed);
    return;
  }
  const unsigned ib = (unsigned)(reinterpret_cast<uintptr_t>(a.payload + lo) & 15u);
  {
    // addresses as integers: the aligned start may precede the payload
    const uintptr_t pb = reinterpret_cast<uintptr_t>(a.payload), pe = pb + a.payload_len;
    const uintptr_t g16 = pb + lo - ib;
    const unsigned nq = (ib + (unsigned)(hi - lo) + 15u) >> 4;
    // 16-byte pieces inside the payload: all but perhaps the first and the last
    const unsigned q_lo = lo < ib ? 1u : 0u;
    const unsigned q_hi = g16 + 16ull * nq <= pe ? nq : nq - 1u;
    uint4 *imgq = reinterpret_cast<uint4 *>(img);
    for (unsigned q = tid; q < nq; q += kD64Threads) {
      const uintptr_t src = g16 + 16u * q;
      uint4 v;
      if (q >= q_lo && q < q_hi) {
        v = __ldg(reinterpret_cast<const uint4 *>(src));
      } else {
        unsigned w4[4] = {0u, 0u, 0u, 0u};
#pragma unroll 1
        for (int t = 0; t < 16; t++)
          if (src + t >= pb && src + t < pe)
            w4[t >> 2] |= (unsigned)(*reinterpret_cast<const unsigned char *>(src + t)) << (8 * (t & 3));
        v = make_uint4(w4[0], w4[1], w4[2], w4[3]);
      }
      imgq[q] = v;
    }
  }
  __syncthreads();
  // a lane a block: the blocks' fields and checks, once and not once a lane of
  // the eight that decode it
  if (tid < kD64Blocks) {
    uint4 h = make_uint4(0u, 0u, 0u, 0u);
    if (tid < nb) {
      const long long left = n - (b0 + tid) * 64;
      const unsigned len = left < 64 ? (unsigned)left : 64u;
      // (no sum of an offset, which may be anything in a caller's index)
      bool ok = !(o0 < lo || o0 > hi || hi - o0 < 4 || o1 < o0 || o1 > end);
      if (ok) {
        h.x = (unsigned)(o0 - lo) + ib;
        const unsigned bend = (unsigned)((o1 < hi ? o1 : hi) - lo) + ib;
        unsigned w0, w1;
        ld_window(reinterpret_cast<const unsigned *>(img), h.x, w0, w1);
        h.y = w0;
        const unsigned bc = len > 1u && h.x + 4 < bend ? w1 & 0xffu : 0u;
        const unsigned bytes = bc > 32u ? 0u : block_bytes_layout(len, bc, TAGS, a.cpu_layout != 0);
        ok = bc <= 32u && h.x + bytes <= bend;
        h.z = h.x + bytes - (len + 3u) / 4u;
        h.w = bc | (ok ? kD64Ok : 0u);
      }
      if (!ok) atomicExch(a.err, kErrMalformed);
    }
    s_hd[tid] = h;
  }
  __syncthreads();
  const uint4 h = s_hd[bi];
  const long long base = (b0 + bi) * 64;
  unsigned n_ext;
  if ((b0 + kD64Blocks) * 64 <= n) {
    n_ext = d64_octet<TAGS, true>(a, img, h, base, 64, l);
  } else {
    const int len = bi < nb ? (int)((n - base) < 64 ? (n - base) : 64) : 0;
    n_ext = d64_octet<TAGS, false>(a, img, h, base, len, l);
  }
  if (TAGS && a.ext_count) {
    // one atomic per CTA: every CTA adds to the same word
    __shared__ unsigned s_ext[kD64Threads / 32];
    n_ext = __reduce_add_sync(0xffffffffu, n_ext);
    if ((tid & 31) == 0) s_ext[tid >> 5] = n_ext;
    __syncthreads();
    if (tid == 0) {
      unsigned tot = 0;
#pragma unroll
      for (int w = 0; w < kD64Threads / 32; w++) tot += s_ext[w];
      if (tot) atomicAdd(a.ext_count, (unsigned long long)tot);
    }
  }
}

cudaError_t launch_decode64(bool tags, const DecArgs &a, cudaStream_t s) {
  const unsigned long long nb = (a.n + 63) / 64;
  if (nb == 0) return cudaSuccess;
  const unsigned grid = (unsigned)((nb + kD64Blocks - 1) / kD64Blocks);
  if (tags) decode64_kernel<true><<<grid, kD64Threads, 0, s>>>(a);
  else decode64_kernel<false><<<grid, kD64Threads, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace tsz
