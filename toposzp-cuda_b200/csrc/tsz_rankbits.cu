// Sort positions from a bitmap over the values of a field (tsz_rankbits.cuh).
#include "tsz_rankbits.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "tsz_codec2.cuh"
#include "tsz_ops.h"

namespace tsz {

// Sorts 2048 keys of a 1024-thread CTA, keys 2t and 2t + 1 in thread t
// (bitonic, over the first P, a power of two of at least 64; the rest are at
// their largest value).  Exchanges within 64 keys are register shuffles; only
// those further apart go through shared memory (15 of 66 at P = 2048), which
// takes 5 us where barriers at every step took 25.
__device__ __forceinline__ void sort_keys_2048(unsigned long long (&v)[2], unsigned P, unsigned long long *sm) {
  const unsigned t = threadIdx.x;
  for (unsigned k = 2; k <= P; k <<= 1) {
    for (unsigned j = k >> 1; j > 0; j >>= 1) {
      if (j >= 64) {
        sm[2 * t] = v[0];
        sm[2 * t + 1] = v[1];
        __syncthreads();
        const unsigned long long o[2] = {sm[(2 * t) ^ j], sm[(2 * t + 1) ^ j]};
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const unsigned e = 2 * t + u;
          const bool keep_min = ((e & j) == 0) == ((e & k) == 0);
          v[u] = (v[u] < o[u]) == keep_min ? v[u] : o[u];
        }
      } else if (j >= 2) {
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const unsigned e = 2 * t + u;
          const unsigned long long o = __shfl_xor_sync(0xffffffffu, v[u], j >> 1);
          const bool keep_min = ((e & j) == 0) == ((e & k) == 0);
          v[u] = (v[u] < o) == keep_min ? v[u] : o;
        }
      } else {
        const bool up = ((2 * t) & k) == 0;
        if ((v[0] > v[1]) == up) {
          const unsigned long long x = v[0];
          v[0] = v[1];
          v[1] = x;
        }
      }
    }
  }
}

// ---- 1. bits of a pair list ------------------------------------------------
__global__ void __launch_bounds__(256)
rank_bits_pairs_kernel(const uint2 *__restrict__ pairs, unsigned long long K, RankBits rb) {
  unsigned nmax = 0, cmax = 0;
  unsigned seen = 0;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < K; k += stride) {
    const uint2 p = pairs[k];
    rb_set(rb, p.x, p.y, seen);
    nmax = max(nmax, ~p.x);
    cmax = max(cmax, p.x);
  }
  rb_extent(rb, nmax, cmax);
}

// ---- 2. prefix counts ------------------------------------------------------
// Counts of tiles of 2048 units (32 KB), then prefixes: every CTA sums the
// counts of the tiles before its own (at most 3300, L2 hits) and scans its
// tile.  The touched range stays in L2 between the two, which take 7 + 11 us
// for the 27 MB of a field of one sign and 10 + 16 us for 46 MB of two; one
// launch with decoupled look-back took 30 us for the latter.
constexpr int kRbPer = 8;
constexpr int kRbTile = kRbPer * kThreads;

__device__ __forceinline__ unsigned unit_count(const uint4 &a) {
  return (unsigned)(__popc(a.y) + __popc(a.z) + __popc(a.w));
}

__device__ __forceinline__ void load_units(const unsigned *__restrict__ bits, unsigned u0, unsigned u1,
                                           unsigned (&c)[kRbPer]) {
  uint4 v[kRbPer];
#pragma unroll
  for (int r = 0; r < kRbPer; r++) {
    const unsigned u = u0 + r * kThreads + threadIdx.x;
    v[r] = u < u1 ? reinterpret_cast<const uint4 *>(bits)[u] : make_uint4(0u, 0u, 0u, 0u);
  }
#pragma unroll
  for (int r = 0; r < kRbPer; r++) c[r] = unit_count(v[r]);
}

__global__ void __launch_bounds__(kThreads)
rank_bits_count_kernel(const unsigned *__restrict__ bits, unsigned u0, unsigned u1, unsigned *__restrict__ cnt) {
  __shared__ unsigned s_w[kWarps];
  unsigned c[kRbPer], t = 0;
  load_units(bits, u0 + blockIdx.x * kRbTile, u1, c);
#pragma unroll
  for (int r = 0; r < kRbPer; r++) t += c[r];
  t = __reduce_add_sync(0xffffffffu, t);
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned s = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) s += s_w[w];
    cnt[blockIdx.x] = s;
  }
}

__global__ void __launch_bounds__(kThreads)
rank_bits_prefix_kernel(unsigned *__restrict__ bits, unsigned u0, unsigned u1, const unsigned *__restrict__ cnt) {
  __shared__ unsigned long long s_w64[2][kWarps];
  __shared__ unsigned s_w[kWarps];
  unsigned c[kRbPer], before = 0;
  load_units(bits, u0 + blockIdx.x * kRbTile, u1, c);
  for (unsigned t = threadIdx.x; t < blockIdx.x; t += kThreads) before += __ldg(cnt + t);
  before = __reduce_add_sync(0xffffffffu, before);
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = before;
  // eight rounds of 256 consecutive units; their counts (at most 96 x 256 =
  // 24576 a round) scanned four rounds at a time in 16-bit fields
  unsigned long long ex[2], tot[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    unsigned long long v = 0;
#pragma unroll
    for (int r = 0; r < 4; r++) v |= (unsigned long long)c[4 * h + r] << (16 * r);
    ex[h] = cta_excl_scan64<kWarps>(v, s_w64[h], &tot[h]);
  }
  unsigned base = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) base += s_w[w];
#pragma unroll
  for (int r = 0; r < kRbPer; r++) {
    const unsigned u = u0 + blockIdx.x * kRbTile + r * kThreads + threadIdx.x;
    if (u < u1) bits[4ull * u] = base + (unsigned)((ex[r >> 2] >> (16 * (r & 3))) & 0xffffull);
    base += (unsigned)((tot[r >> 2] >> (16 * (r & 3))) & 0xffffull);
  }
}

// set bits before bit idx, which lies in a scanned unit
__device__ __forceinline__ unsigned rb_prefix(const unsigned *__restrict__ bits, unsigned idx) {
  const unsigned q = idx / kRbBits, r = idx - q * kRbBits;
  const uint4 a = __ldg(reinterpret_cast<const uint4 *>(bits) + q);
  // bits below r: of the unit's words, the ones before r's word whole
  const unsigned low = (1u << (r & 31u)) - 1u;
  const unsigned w1 = r >= 32u ? ~0u : low, w2 = r >= 64u ? ~0u : (r >= 32u ? low : 0u), w3 = r >= 64u ? low : 0u;
  return a.x + (unsigned)(__popc(a.y & w1) + __popc(a.z & w2) + __popc(a.w & w3));
}

// ---- 3. prefix count of every bin's lowest code ----------------------------
struct RbRange {
  unsigned rz, rh;
  unsigned lo, hi;     // bits [lo, hi) hold every set one
  int b0;              // bin of the smallest value
  unsigned nbins;
  float eb;
  double inv;
};

__device__ __forceinline__ unsigned rb_code(const RbRange &g, unsigned idx) {
  const unsigned S = g.rh - g.rz;
  return idx < S ? ~((g.rh - 1u - idx) | 0x80000000u) : ((idx - S + g.rz) | 0x80000000u);
}

// set bits before bit idx, lo <= idx <= hi
__device__ __forceinline__ unsigned rb_prefix_at(const unsigned *__restrict__ bits, const RbRange &g, unsigned idx) {
  if (g.hi <= g.lo) return 0u;
  if (idx < g.hi) return rb_prefix(bits, idx);
  const unsigned c = rb_prefix(bits, g.hi - 1u), q = (g.hi - 1u) / kRbBits, r = g.hi - 1u - q * kRbBits;
  return c + ((__ldg(bits + 4ull * q + 1u + (r >> 5)) >> (r & 31u)) & 1u);
}

__global__ void rank_bits_bins_kernel(const unsigned *__restrict__ bits, RbRange g, unsigned *__restrict__ binp) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.nbins) return;
  const int bin = g.b0 + (int)i;
  // first bit whose bin is not below this one
  unsigned lo = g.lo, hi = g.hi;
  while (lo < hi) {
    const unsigned mid = lo + ((hi - lo) >> 1);
    if (quant_bin(code_float(rb_code(g, mid)), g.eb, g.inv) < bin) lo = mid + 1u; else hi = mid;
  }
  binp[i] = rb_prefix_at(bits, g, lo);
}

// ---- 3b. the values aside (bins 0 and 1), sorted by one CTA ----------------
// A value of bin 0 comes after the bin's set bits, all negative; one of bin 1
// before them, so the distinct ones of bin 1 are added to that bin's positions
// (its table entry less their number).  A key of its own for the zeros (zero:
// there are some), whose position goes to *zero_pos.
__global__ void __launch_bounds__(1024)
rank_bits_side_kernel(const unsigned *__restrict__ bits, RbRange g, const uint2 *__restrict__ side, unsigned nside,
                      bool zero, unsigned *__restrict__ binp, int *__restrict__ out, unsigned *__restrict__ zero_pos) {
  const unsigned cnt = nside + (zero ? 1u : 0u);
  auto load = [&](unsigned i) {
    if (i >= cnt) return ~0ull;
    if (i == nside) return ((unsigned long long)kZeroCode << 32) | kNoExtremum;
    const uint2 v = side[i];
    return ((unsigned long long)v.x << 32) | v.y;
  };
  __shared__ unsigned long long key[kSideCap];
  __shared__ unsigned s_w[32];
  unsigned P = 64;
  while (P < cnt) P <<= 1;
  if (P <= 2048) {
    unsigned long long v2[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      v2[u] = load(2u * threadIdx.x + u);
    }
    sort_keys_2048(v2, P, key);
    key[2u * threadIdx.x] = v2[0];
    key[2u * threadIdx.x + 1u] = v2[1];
    __syncthreads();
  } else {
    for (unsigned i = threadIdx.x; i < P; i += blockDim.x)
      key[i] = load(i);
    __syncthreads();
    for (unsigned k = 2; k <= P; k <<= 1)
      for (unsigned j = k >> 1; j > 0; j >>= 1) {
        for (unsigned i = threadIdx.x; i < P; i += blockDim.x) {
          const unsigned x = i ^ j;
          if (x > i) {
            const unsigned long long a = key[i], b = key[x];
            if ((a > b) == ((i & k) == 0)) { key[i] = b; key[x] = a; }
          }
        }
        __syncthreads();
      }
  }
  // first occurrences before each value, and those of bin 0 among them
  const unsigned per = (cnt + blockDim.x - 1) / blockDim.x;
  const unsigned i0 = threadIdx.x * per, i1 = min(i0 + per, cnt);
  auto bin_of = [&](unsigned i) { return quant_bin(code_float((unsigned)(key[i] >> 32)), g.eb, g.inv); };
  unsigned d = 0, d0 = 0;
  for (unsigned i = i0; i < i1; i++)
    if (i == 0 || (key[i] >> 32) != (key[i - 1] >> 32)) { d++; d0 += bin_of(i) <= 0 ? 1u : 0u; }
  // at most 4096 of each: one scan of both
  const unsigned v = d | (d0 << 16);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) s_w[warp] = inc;
  __syncthreads();
  unsigned pre = inc - v, tot = 0;
  for (int w = 0; w < 32; w++) {
    if (w < warp) pre += s_w[w];
    tot += s_w[w];
  }
  const unsigned D0 = tot >> 16, D1 = (tot & 0xffffu) - D0;
  // set bits of bin 0
  const unsigned S = g.rh - g.rz;
  unsigned base0 = 0;
  if (g.b0 <= 0 && 0 - (long long)g.b0 < (long long)g.nbins)
    base0 = rb_prefix_at(bits, g, min(max(S, g.lo), g.hi)) - binp[0 - g.b0];
  unsigned run = pre & 0xffffu;   // distinct values before the thread's first
  for (unsigned i = i0; i < i1; i++) {
    if (i == 0 || (key[i] >> 32) != (key[i - 1] >> 32)) run++;
    const unsigned e = (unsigned)key[i], pos = bin_of(i) <= 0 ? base0 + run - 1u : run - 1u - D0;
    if (e != kNoExtremum) out[e] = (int)pos;
    if ((unsigned)(key[i] >> 32) == kZeroCode) *zero_pos = pos;
  }
  __syncthreads();
  if (threadIdx.x == 0 && D1 && g.b0 <= 1 && 1 - (long long)g.b0 < (long long)g.nbins) binp[1 - g.b0] -= D1;
}

// ---- 4. positions ----------------------------------------------------------
__device__ __forceinline__ int rb_rank(const unsigned *__restrict__ bits, const RbRange &g,
                                       const unsigned *__restrict__ binp, unsigned code, unsigned idx) {
  const int bin = quant_bin(code_float(code), g.eb, g.inv);
  return (int)(rb_prefix(bits, idx) - __ldg(binp + (unsigned)(bin - g.b0)));
}

// codes[e] of the extrema in raster order; four per thread (the loads of their
// sectors in flight together)
__global__ void __launch_bounds__(256)
rank_bits_codes_kernel(const unsigned *__restrict__ codes, unsigned long long E, const unsigned *__restrict__ bits,
                       RbRange g, const unsigned *__restrict__ binp, const unsigned *__restrict__ zero_pos,
                       int *__restrict__ out) {
  const unsigned long long e0 = 4ull * ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x);
  if (e0 >= E) return;
  if (e0 + 4 <= E) {
    const uint4 c = __ldg(reinterpret_cast<const uint4 *>(codes + e0));
    const unsigned cc[4] = {c.x, c.y, c.z, c.w};
    int r[4];
    bool in[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      unsigned idx;
      in[k] = rb_index(g.rz, g.rh, cc[k], &idx);
      r[k] = in[k] ? rb_rank(bits, g, binp, cc[k], idx) : 0;
    }
    if (in[0] && in[1] && in[2] && in[3]) {
      *reinterpret_cast<int4 *>(out + e0) = make_int4(r[0], r[1], r[2], r[3]);
    } else {
      // values aside have their positions already, but the zeros
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (in[k]) out[e0 + k] = r[k];
        else if (cc[k] == kZeroCode) out[e0 + k] = (int)*zero_pos;
      }
    }
  } else {
    for (unsigned long long e = e0; e < E; e++) {
      unsigned idx;
      const unsigned c = codes[e];
      if (rb_index(g.rz, g.rh, c, &idx)) out[e] = rb_rank(bits, g, binp, c, idx);
      else if (c == kZeroCode) out[e] = (int)*zero_pos;
    }
  }
}

__global__ void __launch_bounds__(256)
rank_bits_pair_out_kernel(const uint2 *__restrict__ pairs, unsigned long long K, const unsigned *__restrict__ bits,
                          RbRange g, const unsigned *__restrict__ binp, const unsigned *__restrict__ zero_pos,
                          int *__restrict__ out) {
  const unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  const uint2 p = pairs[k];
  unsigned idx;
  if (p.y == kNoExtremum) return;
  if (rb_index(g.rz, g.rh, p.x, &idx)) out[p.y] = rb_rank(bits, g, binp, p.x, idx);
  else if (p.x == kZeroCode) out[p.y] = (int)*zero_pos;
}

// ---- host ------------------------------------------------------------------
static int host_bin(unsigned code, float eb, double inv) {
  volatile float s = code_float(code) + eb;     // float addition first, as quant_bin
  return (int)((double)s * inv);                // below 2^31: magnitudes are below 2^30 eb
}

static size_t rb_bytes() { return (size_t)kRbUnits * 16; }

// The workspace's allocation: the bits, the values aside and the first pairs,
// the bins' prefix counts and the tiles' counts.
struct RbStore {
  size_t side, first, bins, cnt, bytes;
  RbStore() {
    side = rb_bytes();
    first = side + kSideCap * sizeof(uint2);
    bins = first + kRankSmall * sizeof(uint2);
    cnt = bins + (size_t)kMaxBins * 4;
    bytes = cnt + ((size_t)kRbUnits / kRbTile + 2) * 4;
  }
};

size_t rank_bits_bytes() { return RbStore().bytes; }

// Whether the workspace has the bitmap, or could get it.  It is optional (the
// bucket ranking gives the same positions without it): no room for it is no
// error, and is remembered, so that later calls do not try again.
bool rank_bits_reserve(szp_b200_ctx *ctx) {
  if (ctx->rank_bits) return true;
  if (ctx->rank_bits_no_room) return false;
  void *p = nullptr;
  if (cudaMalloc(&p, rank_bits_bytes()) != cudaSuccess) {
    cudaGetLastError();
    ctx->rank_bits_no_room = true;
    return false;
  }
  ctx->rank_bits = static_cast<unsigned *>(p);
  ctx->rank_bits_dirty = true;
  return true;
}

bool rank_bits_begin(szp_b200_ctx *ctx, float eb, RankBits *rb) {
  int e = 0;
  if (!(eb > 0.f) || !std::isfinite(eb)) return false;
  std::frexp(eb, &e);
  e -= 1;                                        // 2^e <= eb
  const float z = std::ldexp(1.0f, e - (int)kRbBelow);
  float h = e + (int)kRbAbove > 127 ? INFINITY : std::ldexp(1.0f, e + (int)kRbAbove);
  unsigned zb, hb;
  memcpy(&zb, &z, 4);
  memcpy(&hb, &h, 4);
  if (zb == 0) zb = 1;
  if (hb <= zb || 2ull * (hb - zb) / kRbBits + 2 > kRbUnits) return false;
  if (!rank_bits_reserve(ctx)) return false;
  const RbStore at;
  unsigned char *base = reinterpret_cast<unsigned char *>(ctx->rank_bits);
  rb->bits = ctx->rank_bits;
  rb->rz = zb;
  rb->rh = hb;
  rb->side = reinterpret_cast<uint2 *>(base + at.side);
  rb->first = reinterpret_cast<uint2 *>(base + at.first);
  rb->stat = reinterpret_cast<unsigned *>(ctx->d_words + kRbStatWord);
  cudaStream_t s = ctx->stream;
  if (ctx->rank_bits_dirty && cuda_fail(cudaMemsetAsync(ctx->rank_bits, 0, rb_bytes(), s), "memset")) return false;
  // from here until the bits are cleared again
  ctx->rank_bits_dirty = true;
  return true;
}

// bits below a code's: its own place, or that of the gap it lies in
static unsigned rb_place(const RankBits &rb, unsigned code, bool *in) {
  const unsigned S = rb.rh - rb.rz, mag = ((code >> 31) ? code : ~code) & 0x7FFFFFFFu;
  unsigned idx;
  *in = rb_index(rb.rz, rb.rh, code, &idx);
  return *in ? idx : (mag < rb.rz ? S : ((code >> 31) ? 2u * S : 0u));
}

int rank_bits_finish(szp_b200_ctx *ctx, const RankBits &rb, const unsigned *h_stat, float eb, const unsigned *d_codes,
                     const uint2 *d_pairs, unsigned long long K, unsigned long long E, int *d_sp) {
  if (!d_pairs && K <= kRankSmall) return rank_small(ctx, rb.first, K, eb, d_sp, &rb);
  const unsigned cmin = ~h_stat[0], cmax = h_stat[1];
  RbRange g;
  g.rz = rb.rz;
  g.rh = rb.rh;
  g.eb = eb;
  g.inv = 1.0 / (double)eb;
  // the bits that may be set are those between the smallest and the largest value's
  bool in;
  const unsigned lo = rb_place(rb, cmin, &in), top = rb_place(rb, cmax, &in), hi = in ? top + 1u : top;
  g.lo = lo;
  g.hi = hi;
  cudaStream_t s = ctx->stream;
  const unsigned s0 = lo / kRbBits, s1 = hi > lo ? (hi - 1u) / kRbBits + 1u : s0;
  const bool zero = h_stat[4] != 0u;
  bool apply = !h_stat[3] && h_stat[2] + (zero ? 1u : 0u) <= kSideCap;
  if (apply) {
    g.b0 = host_bin(cmin, eb, g.inv);
    const long long nb = (long long)host_bin(cmax, eb, g.inv) - g.b0 + 1;
    apply = nb >= 1 && nb <= (long long)kMaxBins;
    g.nbins = (unsigned)nb;
  }
  if (E && apply) {
    const RbStore at;
    unsigned char *base = reinterpret_cast<unsigned char *>(ctx->rank_bits);
    unsigned *binp = reinterpret_cast<unsigned *>(base + at.bins), *cnt = reinterpret_cast<unsigned *>(base + at.cnt);
    const unsigned ntiles = (s1 - s0 + kRbTile - 1) / kRbTile;
    if (ntiles) {
      rank_bits_count_kernel<<<ntiles, kThreads, 0, s>>>(rb.bits, s0, s1, cnt);
      rank_bits_prefix_kernel<<<ntiles, kThreads, 0, s>>>(rb.bits, s0, s1, cnt);
      ctx->launches += 2;
    }
    rank_bits_bins_kernel<<<(g.nbins + 127) / 128, 128, 0, s>>>(rb.bits, g, binp);
    ctx->launches += 1;
    unsigned *zero_pos = rb.stat + 5;
    if (h_stat[2] || zero) {
      rank_bits_side_kernel<<<1, 1024, 0, s>>>(rb.bits, g, rb.side, h_stat[2], zero, binp, d_sp, zero_pos);
      ctx->launches += 1;
    }
    if (d_codes)
      rank_bits_codes_kernel<<<(unsigned)((E + 1023) / 1024), 256, 0, s>>>(d_codes, E, rb.bits, g, binp,
                                                                              zero_pos, d_sp);
    else
      rank_bits_pair_out_kernel<<<(unsigned)((K + 255) / 256), 256, 0, s>>>(d_pairs, K, rb.bits, g, binp,
                                                                                 zero_pos, d_sp);
    ctx->launches += 1;
    if (cuda_fail(cudaGetLastError(), "rank kernels")) return -1;
  }
  // the words that were set, for the next call
  if (s1 > s0 && cuda_fail(cudaMemsetAsync(rb.bits + 4ull * s0, 0, 16ull * (s1 - s0), s), "memset")) return -1;
  ctx->rank_bits_dirty = false;
  return apply ? 0 : 1;
}

int rank_bits_from_pairs(szp_b200_ctx *ctx, const uint2 *d_pairs, unsigned long long K, unsigned long long E, float eb,
                         int *d_sp) {
  RankBits rb;
  if (!rank_bits_begin(ctx, eb, &rb)) return 1;
  cudaStream_t s = ctx->stream;
  const unsigned grid = (unsigned)std::min<unsigned long long>((K + 1023) / 1024, (unsigned long long)ctx->sm_count * 8);
  if (cuda_fail(cudaMemsetAsync(rb.stat, 0, 32, s), "memset")) return -1;
  rank_bits_pairs_kernel<<<grid, 256, 0, s>>>(d_pairs, K, rb);
  ctx->launches += 1;
  unsigned *h_stat = reinterpret_cast<unsigned *>(ctx->h_words + kRbStatWord);
  if (cuda_fail(cudaGetLastError(), "rank kernels") ||
      cuda_fail(cudaMemcpyAsync(h_stat, rb.stat, 32, cudaMemcpyDeviceToHost, s), "D2H") ||
      cuda_fail(cudaStreamSynchronize(s), "rank"))
    return -1;
  return rank_bits_finish(ctx, rb, h_stat, eb, nullptr, d_pairs, K, E, d_sp);
}

// ---- up to 2048 pairs: sorted by one CTA -----------------------------------
constexpr int kSmallThreads = 1024;
static_assert(kRankSmall == 2 * kSmallThreads, "two items per thread");

// with fields: CTA f takes fields[f] of a batch
__global__ void __launch_bounds__(kSmallThreads)
rank_small_kernel(const uint2 *__restrict__ pairs, unsigned K, float eb, double inv, int *__restrict__ out,
                  RankBits rb, const SmallField *__restrict__ fields) {
  if (fields) {
    const SmallField f = fields[blockIdx.x];
    pairs += f.pairs_off;
    K = f.K;
    eb = f.eb;
    inv = 1.0 / (double)eb;
    out += f.ebase;
  }
  __shared__ unsigned long long key[kRankSmall];
  __shared__ unsigned s_w[kSmallThreads / 32];
  unsigned P = 64;
  while (P < K) P <<= 1;
  unsigned long long v2[2];
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const unsigned i = 2u * threadIdx.x + u;
    const uint2 p = i < K ? pairs[i] : make_uint2(~0u, ~0u);
    v2[u] = ((unsigned long long)p.x << 32) | p.y;
    unsigned idx;
    if (rb.bits && i < K && rb_index(rb.rz, rb.rh, p.x, &idx)) {
      const unsigned q = idx / kRbBits;
      rb.bits[4u * q + 1u + ((idx - q * kRbBits) >> 5)] = 0u;
    }
  }
  sort_keys_2048(v2, P, key);
  key[2u * threadIdx.x] = v2[0];
  key[2u * threadIdx.x + 1u] = v2[1];
  __syncthreads();
  // D: distinct codes up to item i; H: the D of its bin's first item (a bin is
  // a monotone function of the code); its position is D - H
  const unsigned i0 = 2u * threadIdx.x;
  unsigned D[2], H[2];
  unsigned nc[2], nb[2];
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const unsigned i = i0 + u;
    nc[u] = nb[u] = 0;
    if (i < K) {
      const unsigned c = (unsigned)(key[i] >> 32), b = i ? (unsigned)(key[i - 1] >> 32) : 0u;
      nc[u] = i == 0 || c != b;
      nb[u] = i == 0 || quant_bin(code_float(c), eb, inv) != quant_bin(code_float(b), eb, inv);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned v = nc[0] + nc[1], inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned x = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += x;
  }
  if (lane == 31) s_w[warp] = inc;
  __syncthreads();
  unsigned pre = inc - v;
  for (int w = 0; w < warp; w++) pre += s_w[w];
  D[0] = pre + nc[0];
  D[1] = D[0] + nc[1];
  __syncthreads();
  unsigned m = max(nb[0] ? D[0] : 0u, nb[1] ? D[1] : 0u), hi = m;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned x = __shfl_up_sync(0xffffffffu, hi, o);
    if (lane >= o) hi = max(hi, x);
  }
  if (lane == 31) s_w[warp] = hi;
  unsigned before = __shfl_up_sync(0xffffffffu, hi, 1);
  if (lane == 0) before = 0u;
  __syncthreads();
  for (int w = 0; w < warp; w++) before = max(before, s_w[w]);
  H[0] = nb[0] ? D[0] : before;
  H[1] = nb[1] ? D[1] : H[0];
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const unsigned e = i0 + u < K ? (unsigned)key[i0 + u] : kNoExtremum;
    if (e != kNoExtremum) out[e] = (int)(D[u] - H[u]);
  }
}

int rank_small(szp_b200_ctx *ctx, const uint2 *d_pairs, unsigned long long K, float eb, int *d_sp,
               const RankBits *rb) {
  rank_small_kernel<<<1, kSmallThreads, 0, ctx->stream>>>(d_pairs, (unsigned)K, eb, 1.0 / (double)eb, d_sp,
                                                          rb ? *rb : RankBits{}, nullptr);
  if (rb) ctx->rank_bits_dirty = false;
  ctx->launches += 1;
  return cuda_fail(cudaGetLastError(), "rank kernel") ? -1 : 0;
}

int rank_small_fields(szp_b200_ctx *ctx, const uint2 *d_pairs, const SmallField *d_fields, unsigned count, int *d_sp) {
  rank_small_kernel<<<count, kSmallThreads, 0, ctx->stream>>>(d_pairs, 0, 1.0f, 1.0, d_sp, RankBits{}, d_fields);
  ctx->launches += 1;
  return cuda_fail(cudaGetLastError(), "rank kernel") ? -1 : 0;
}

}  // namespace tsz
