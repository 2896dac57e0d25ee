// Block decoder for blockSize 64 (topology, sort-position and plain streams).
//
// Same values as the octet decoder (tsz_codec2.cuh; SZp/src/
// szp_cuda_decompress.cu:673-741), which is bound by instruction issue: 92
// instructions per element, at 1.9 TB/s.  Eight lanes decode a block, eight
// values each, as there; what is left out or cheaper:
//   * a value past a block's last delta is decoded from whatever follows it and
//     goes nowhere (it could only reach elements that do not exist), so no value
//     has a bound check of its own;
//   * the remainder fields of an octet are a 64-bit big-endian window, shifted
//     left by one field a value;
//   * signs multiply: q[t + 1] = q[t] + magnitude * (+1 or -1), one multiply-add
//     per value on the FMA pipe, which also is the octet's prefix sum;
//   * blocks with full magnitude bytes beyond one take the byte loop.
#include "tsz_codec.h"
#include "tsz_codec2.cuh"

namespace tsz {

constexpr int kD64Threads = 256;
constexpr int kD64Blocks = kD64Threads / 8;

__host__ __device__ constexpr unsigned d64_img_bytes(bool tags) {
  return ((unsigned)kD64Blocks * (tags ? 289u : 273u) + 64u + 15u) & ~15u;
}

// the 8 bytes at image position p, as two little-endian words
__device__ __forceinline__ void ld_window(const unsigned *imgw, unsigned p, unsigned &lo, unsigned &hi) {
  const unsigned wi = p >> 2, sh = 8u * (p & 3u);
  const unsigned a = imgw[wi], b = imgw[wi + 1], c = imgw[wi + 2];
  lo = __funnelshift_r(a, b, sh);
  hi = __funnelshift_r(b, c, sh);
}

template <bool TAGS>
__global__ void __launch_bounds__(kD64Threads, 6) decode64_kernel(DecArgs a) {
  __shared__ __align__(16) unsigned char img[d64_img_bytes(TAGS) + 32];
  __shared__ unsigned long long s_off[kD64Blocks + 1];
  const int tid = threadIdx.x, l = tid & 7, bi = tid >> 3;
  const long long n = (long long)a.n;
  const long long nblocks = (n + 63) / 64;
  const long long b0 = (long long)blockIdx.x * kD64Blocks;
  const int nb = (int)((nblocks - b0) < kD64Blocks ? (nblocks - b0) : kD64Blocks);
  if (tid <= nb) s_off[tid] = b0 + tid < nblocks ? a.blk_off[b0 + tid] : a.payload_len;
  __syncthreads();
  // the image holds the payload bytes from the 16-byte boundary at or below
  // payload + lo: img[ib + k] is payload[lo + k]
  const unsigned long long lo = s_off[0];
  unsigned long long hi = s_off[nb];
  if (hi > a.payload_len) hi = a.payload_len;
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
    uint4 *imgq = reinterpret_cast<uint4 *>(img);
    for (unsigned q = tid; q < nq; q += kD64Threads) {
      const uintptr_t src = g16 + 16u * q;
      uint4 v;
      if (src >= pb && src + 16 <= pe) {
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
  const unsigned *imgw = reinterpret_cast<const unsigned *>(img);
  const bool have = bi < nb;
  const long long base = (b0 + bi) * 64;
  const int len = have ? (int)((n - base) < 64 ? (n - base) : 64) : 0;
  const int e0 = 8 * l;
  const int nv = len - e0 < 0 ? 0 : (len - e0 > 8 ? 8 : len - e0);
  bool ok = have;
  unsigned start = 0, bend = 0;
  if (ok) {
    const unsigned long long o0 = s_off[bi], o1 = s_off[bi + 1];
    if (o0 < lo || o0 + 4 > hi || o1 < o0 || o1 > s_off[nb]) ok = false;
    start = (unsigned)(o0 - lo) + ib;
    bend = (unsigned)((o1 < hi ? o1 : hi) - lo) + ib;
  }
  unsigned bc = 0;
  int anchor = 0;
  if (ok) {
    unsigned w0, w1;
    ld_window(imgw, start, w0, w1);
    anchor = (int)w0;
    if (len > 1) bc = start + 4 < bend ? w1 & 0xffu : 0u;
    if (bc > 32u || start + block_bytes_layout((unsigned)len, bc, TAGS, a.cpu_layout != 0) > bend) ok = false;
  }
  if (have && !ok && l == 0) atomicExch(a.err, kErrMalformed);
  const unsigned cnt = len > 0 ? (unsigned)len - 1u : 0u;
  // q[t]: sum of the octet's deltas before element t; q[8]: of all of them
  int q[9];
#pragma unroll
  for (int t = 0; t < 9; t++) q[t] = 0;
  if (ok && bc && (unsigned)e0 < cnt) {
    const unsigned p = start + 5u, sbytes = (cnt + 7u) >> 3;
    const unsigned neg = (unsigned)img[p + l] << 24;     // sign of delta e0 + t at bit 31 - t
    const unsigned mag = p + sbytes, fb = bc >> 3, rem = bc & 7u;
    // rem bytes at byte l rem of the remainder section, most significant bits first
    unsigned rl, rh;
    ld_window(imgw, mag + fb * cnt + (unsigned)l * rem, rl, rh);
    unsigned wh = __byte_perm(rl, 0u, 0x0123), wl = __byte_perm(rh, 0u, 0x0123);
    const unsigned down = 31u - rem;                     // a field is (wh >> 1) >> down: nothing when rem is 0
    unsigned fl = 0, fh = 0;
    if (fb == 1) ld_window(imgw, mag + (unsigned)e0, fl, fh);
    const unsigned up = 1u << rem;
    if (fb <= 1) {
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const unsigned full = __byte_perm(fl, fh, 0x4440u + (unsigned)t) & 0xffu;
        const unsigned m = full * up + ((wh >> 1) >> down);
        wh = __funnelshift_l(wl, wh, rem);
        wl <<= rem;
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
        const unsigned m = full * up + ((wh >> 1) >> down);
        wh = __funnelshift_l(wl, wh, rem);
        wl <<= rem;
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
  const int v0 = (int)((unsigned)anchor + (unsigned)inc - (unsigned)q[8]);
  unsigned n_ext = 0;
  if (ok && nv > 0) {
#pragma unroll
    for (int t = 0; t < 8; t++) q[t] = (int)((unsigned)q[t] + (unsigned)v0);
    const long long i0 = base + e0;
    if (a.out_f) {
      float f[8];
#pragma unroll
      for (int t = 0; t < 8; t++) f[t] = __fmul_rn((float)q[t], a.eb);
      if (nv == 8 && ((reinterpret_cast<uintptr_t>(a.out_f + i0) & 15) == 0)) {
        reinterpret_cast<float4 *>(a.out_f + i0)[0] = make_float4(f[0], f[1], f[2], f[3]);
        reinterpret_cast<float4 *>(a.out_f + i0)[1] = make_float4(f[4], f[5], f[6], f[7]);
      } else {
#pragma unroll
        for (int t = 0; t < 8; t++) if (t < nv) a.out_f[i0 + t] = f[t];
      }
    }
    if (!TAGS && a.out_i) {
      if (nv == 8 && ((reinterpret_cast<uintptr_t>(a.out_i + i0) & 15) == 0)) {
        reinterpret_cast<int4 *>(a.out_i + i0)[0] = make_int4(q[0], q[1], q[2], q[3]);
        reinterpret_cast<int4 *>(a.out_i + i0)[1] = make_int4(q[4], q[5], q[6], q[7]);
      } else {
#pragma unroll
        for (int t = 0; t < 8; t++) if (t < nv) a.out_i[i0 + t] = q[t];
      }
    }
    if (TAGS) {
      const unsigned tb = ((unsigned)len + 3u) / 4u;
      const unsigned tsec = start + block_bytes_layout((unsigned)len, bc, true, a.cpu_layout != 0) - tb;
      // element 0 in the top two of 16 bits; elements past nv as regular points
      unsigned tg = (2u * l < tb ? (unsigned)img[tsec + 2 * l] << 8 : 0u) |
                    (2u * l + 1u < tb ? (unsigned)img[tsec + 2 * l + 1] : 0u);
      if (nv < 8) tg &= 0xffffu << (16 - 2 * nv);
      n_ext = (unsigned)__popc((tg ^ (tg >> 1)) & 0x5555u);   // types 01 and 10
      if (a.pl_lo) {
        // element t to bit t: the compacted fields, element 0 on top, reversed
        const long long o = i0 >> 3;
        a.pl_lo[o] = (unsigned char)(__brev(compact2(tg)) >> 24);
        a.pl_hi[o] = (unsigned char)(__brev(compact2(tg >> 1)) >> 24);
        // the rest of the planes' last word
        if (i0 + 8 >= n)
          for (long long k = o + 1; k & 3; k++) a.pl_lo[k] = a.pl_hi[k] = 0;
      }
      if (a.fn_u8) {
        if (nv == 8 && ((reinterpret_cast<uintptr_t>(a.fn_u8 + i0) & 7) == 0)) {
          // four two-bit fields of a byte, most significant first, to four bytes
          unsigned w[2];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const unsigned x = h ? tg & 0xffu : tg >> 8;
            const unsigned y = (x | (x << 12)) & 0x000f000fu;        // low nibble, high nibble << 16
            const unsigned z = (y | (y << 6)) & 0x03030303u;         // fields 3, 2 (low to high byte), 1, 0
            w[h] = __byte_perm(z, 0u, 0x0123);
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
    }
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
