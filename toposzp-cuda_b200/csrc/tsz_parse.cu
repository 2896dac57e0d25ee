// Block offsets of a compressed stream, found on the device from the stream
// bytes alone.
//
// The streams carry no block index: a block's length follows from its bit
// count byte, so block k+1 starts where block k ends and the reference finds
// the offsets with one serial walk (SZp/src/szp_cuda_decompress.cu:233-328
// and its thread-count detection, :400-418).  Here the payload is cut into
// segments of kSegBytes that are walked side by side.  A block that starts in
// segment j-1 ends less than M bytes into segment j (M = largest valid
// block), so the first block start in segment j, its entry, lies in
// [jS, jS + M).
//
// Checked guess (parse_guess_kernel).  Walks from wrong places meet bit count
// bytes above 32, or fall in step with the true walk, within a few blocks.  So
// one warp per segment starts a walk at each of the M possible block starts
// some blocks ahead of its segment; when all walks that are left at the
// segment agree on one entry, it walks the segment from there and a
// decoupled look-back gives the index of its first block.  Each segment
// compares its entry with the exit of the one before, and segment 0 starts at
// offset 0, so a parse in which no comparison fails and which reaches its last
// block is the serial walk's, exactly.  Otherwise (a guess that is not unique,
// as in fields of constant blocks, or a stream that is not valid) the exact
// parse below runs over it; its launches return at once when it need not.
//
// Exact parse (parse_seg_kernel, parse_write_kernel):
//   1. For every segment and every entry, one thread walks the blocks that
//      start inside the segment and records (blocks started, exit entry into
//      the next segment): the segment's transfer function F.
//   2. Functions are composed a group at a time.  The CTA that finishes last
//      in a group composes it, level by level up to one function, inside the
//      same launch.  Beside the group's function it stores, for each member
//      and each entry of the group, the composition of the members before it
//      (the prefix functions P), so no pass back down the levels is needed.
//   3. One CTA per segment finds its true entry and first block index with
//      one load per level (P of its groups, from entry 0 at the top), walks
//      its blocks and writes their offsets; the one that reaches block nb-1
//      sizes it with its own element count and records the payload length.
// Validation matches the reference's single-chunk check: every bit count is
// at most 32 and the last block ends inside min(buffer, validation bound).
// A walk that meets a bit count above 32 or the buffer end stops ("stuck");
// such a chain is reported as a failed parse unless it is past block nb-1.
//
// What bounds it: the serial chain of a segment's walk, so all walks run on a
// copy of the segment in shared memory and segments are short.  Kernel times
// on B200, against the walk of every entry of 16 KB segments in global memory
// and composition passes of their own, which this replaces:
//   87 MB stream of the plain codec (960 K blocks)        520 -> 135 us
//   5.4 + 2.4 MB streams of a 1800 x 3600 field            720 ->  50 us
// (settled by the guess).  Where the guess fails the exact parse adds 290 us
// on the 87 MB stream.

#include <algorithm>

#include "tsz_common.cuh"
#include "tsz_lookback.cuh"
#include "tsz_ops.h"
#include "tsz_runtime.h"

namespace tsz {

// Segments of the exact parse: about 70 blocks of 64 values a walk.  Halving
// them halves the chain but doubles the function tables (4 B per entry, 281
// entries at blockSize 64).
constexpr unsigned kSegBytes = 8192;
constexpr unsigned kSegStage = kSegBytes + 48;   // staged bytes: the segment, the byte after p + 4, alignment
constexpr int kMaxLevels = 16;
constexpr int kExitBits = 13;                    // M <= 4229 (the plain codec's blockSize 1025)
constexpr unsigned kStuck = (1u << kExitBits) - 1u;   // exit entry of a walk that stopped
// blocks a segment may start (blockSize >= 2: at least 5 bytes each)
constexpr unsigned kSegList = kSegBytes / 5 + 2;

struct ParseGeom {
  const unsigned char *p;      // payload (after the 8-byte offset table)
  unsigned long long len;      // payload bytes present in the buffer
  int B;
  bool tags;
  unsigned full_tag;           // tag bytes of a full block
  unsigned M;                  // largest valid block (bit count 32)
  bool cpu;                    // OpenMP layout: one-element blocks carry a bit-count byte
};

// The levels of the composition.  Level 0 items are the segments; level l+1
// items are the groups of G level-l items; the top level has one item.  All
// values are (blocks << kExitBits) | exit entry.
struct ParseTree {
  int levels;                                // L: items cnt[0] .. cnt[L-1], cnt[L-1] == 1
  int lgG;                                   // G = 2^lgG members a group
  bool staged;                               // a group's segment functions fit the CTA's shared memory
  unsigned cnt[kMaxLevels];
  unsigned *f0, *p0;                         // F and P of the segments (one array when staged); at
                                             // most 32 x 8 KB / 5 B blocks in a group: 32 bits hold both
  unsigned long long *f[kMaxLevels];         // l >= 1: F of the level-l items
  unsigned long long *p[kMaxLevels];         // and their P
  unsigned *done[kMaxLevels];                // l >= 1: finished members of each level-l item (zeroed)
};

// Length of a full block (B >= 2 elements) from its bit count byte; 0 =
// invalid.  mag_bytes(n, bc) is ceil(n bc / 8), so a step of a walk is one
// load and a few integer operations (a table of lengths would be a second
// load behind it: 150 cycles a block instead of 100).
struct BlockLen {
  unsigned base, sign, cnt;
  __device__ explicit BlockLen(const ParseGeom &g)
      : base(5u + g.full_tag), sign(base + (unsigned)((g.B - 2) >> 3) + 1u), cnt((unsigned)g.B - 1u) {}
  __device__ __forceinline__ unsigned operator()(unsigned bc) const {
    const unsigned len = bc ? sign + ((bc * cnt + 7u) >> 3) : base;
    return bc <= 32u ? len : 0u;
  }
};

// Payload bytes [s0, s0 + bytes) that exist, into buf; returns the place of
// byte s0 in buf.  16-byte loads wherever all 16 bytes are inside the payload.
__device__ __forceinline__ unsigned stage_segment(const ParseGeom &g, unsigned long long s0, unsigned char *buf,
                                                  unsigned bytes = kSegBytes + 5u) {
  const unsigned char *a = g.p + s0;
  const unsigned lead = (unsigned)(reinterpret_cast<uintptr_t>(a) & 15u);
  const unsigned long long rest = g.len - s0;
  const unsigned want = (unsigned)(rest < bytes ? rest : bytes) + lead;
  const unsigned nq = (want + 15u) >> 4;
  const unsigned char *al = a - lead;
  constexpr unsigned kU = 4;   // chunks in flight per thread
  for (unsigned q0 = threadIdx.x; q0 < nq; q0 += kU * blockDim.x) {
    uint4 v[kU];
#pragma unroll
    for (unsigned u = 0; u < kU; u++) {
      const unsigned o = 16u * (q0 + u * blockDim.x);
      // from the second chunk on, and for s0 > 0 from the first, no byte lies before the payload
      if ((s0 || o >= lead) && o + 16u <= want) v[u] = __ldg(reinterpret_cast<const uint4 *>(al + o));
    }
#pragma unroll
    for (unsigned u = 0; u < kU; u++) {
      const unsigned o = 16u * (q0 + u * blockDim.x);
      if (o >= want) continue;
      if (!((s0 || o >= lead) && o + 16u <= want)) {
        unsigned w[4] = {0u, 0u, 0u, 0u};
        for (unsigned k = 0; k < 16; k++)
          if ((s0 || o + k >= lead) && o + k < want) w[k >> 2] |= (unsigned)__ldg(al + o + k) << (8u * (k & 3u));
        v[u] = make_uint4(w[0], w[1], w[2], w[3]);
      }
      *reinterpret_cast<uint4 *>(buf + o) = v[u];
    }
  }
  return lead;
}

// Composition of one group of level-l items into the level-(l+1) item grp,
// by all threads of the CTA: entry e runs through the members, and the prefix
// before each member goes to P.  The functions of the segments go through
// shared memory first where they fit (sm), so that a step of the chain costs
// a shared load and not an L2 round trip: level 0 has most of the groups.
__device__ void compose_group(const ParseTree &t, int l, unsigned grp, unsigned M, unsigned *sm) {
  const unsigned i0 = grp << t.lgG, m = min(1u << t.lgG, t.cnt[l] - i0);
  unsigned long long *dst = t.f[l + 1] + (size_t)grp * M;
  if (l == 0) {
    const unsigned *src = t.f0 + (size_t)i0 * M;
    unsigned *pre = t.p0 + (size_t)i0 * M;
    if (t.staged) {
      for (unsigned w = threadIdx.x; w < m * M; w += blockDim.x) sm[w] = __ldcg(src + w);
      __syncthreads();
    }
    for (unsigned e = threadIdx.x; e < M; e += blockDim.x) {
      unsigned c = 0, x = e;
      for (unsigned k = 0; k < m; k++) {
        if (k) pre[k * M + e] = (c << kExitBits) | x;
        if (x != kStuck) {
          const unsigned v = t.staged ? sm[k * M + x] : __ldcg(src + k * M + x);
          c += v >> kExitBits;
          x = v & kStuck;
        }
      }
      dst[e] = ((unsigned long long)c << kExitBits) | x;
    }
  } else {
    const unsigned long long *src = t.f[l] + (size_t)i0 * M;
    unsigned long long *pre = t.p[l] + (size_t)i0 * M;
    for (unsigned e = threadIdx.x; e < M; e += blockDim.x) {
      unsigned long long c = 0;
      unsigned x = e;
      for (unsigned k = 0; k < m; k++) {
        if (k) pre[(size_t)k * M + e] = (c << kExitBits) | x;
        if (x != kStuck) {
          const unsigned long long v = __ldcg(src + (size_t)k * M + x);
          c += v >> kExitBits;
          x = (unsigned)(v & kStuck);
        }
      }
      dst[e] = (c << kExitBits) | x;
    }
  }
}

// Outcome of the guess and what it shares between segments.
struct ParseGuess {
  TileDesc *desc;        // per tile, zeroed: count of blocks; pad[0] = exit entry
  unsigned *words;       // zeroed: [0] tile ticket, [1] a guess failed, [2] look-back status
  unsigned unit;         // segment bytes (a multiple of 16, above 4 M)
  unsigned list;         // entries of a warp's list: blocks of a segment, or M
};

// whether the guess settled the parse (the exact parse then has nothing to do)
__device__ __forceinline__ bool parse_settled(const ParseGuess &u, const unsigned long long *status) {
  return u.words && u.words[1] == 0u && u.words[2] == 0u && status[0] != 0ull;
}

// 1 + 2. transfer functions of the segments, composed up to the top level.
__global__ void parse_seg_kernel(ParseGeom g, ParseTree t, ParseGuess u, unsigned long long *status) {
  extern __shared__ __align__(16) unsigned char psm[];
  __shared__ unsigned s_last, s_skip;
  if (threadIdx.x == 0) {
    s_skip = parse_settled(u, status);
    // a length that a failed guess recorded does not count; every CTA, of this
    // launch and the next, that reads the words before or after this comes to
    // the same answer
    if (!s_skip && blockIdx.x == 0) {
      u.words[1] = 1u;
      status[0] = 0ull;
    }
  }
  __syncthreads();
  if (s_skip) return;
  const BlockLen lens(g);
  for (unsigned j = blockIdx.x; j < t.cnt[0]; j += gridDim.x) {
    const unsigned long long s0 = (unsigned long long)j * kSegBytes;
    __syncthreads();
    const unsigned lead = stage_segment(g, s0, psm);
    __syncthreads();
    const unsigned char *buf = psm + lead;
    // a bit count byte at or past the buffer end stops the walk
    const unsigned long long rest = g.len - s0;
    const unsigned lim = (unsigned)(rest < kSegBytes + 5u ? rest : kSegBytes + 5u);
    for (unsigned e = threadIdx.x; e < g.M; e += blockDim.x) {
      unsigned p = e, c = 0, x = kStuck;
      while (true) {
        if (p >= kSegBytes) { x = p - kSegBytes; break; }
        if (p + 4u >= lim) break;
        const unsigned len = lens(buf[p + 4u]);
        if (!len) break;
        c++;
        p += len;
      }
      t.f0[(size_t)j * g.M + e] = (c << kExitBits) | x;
    }
    // the last member of a group composes it, and so on up
    unsigned item = j;
    for (int l = 0; l + 1 < t.levels; l++) {
      __threadfence();
      __syncthreads();
      const unsigned grp = item >> t.lgG;
      if (threadIdx.x == 0) {
        const unsigned members = min(1u << t.lgG, t.cnt[l] - (grp << t.lgG));
        s_last = atomicAdd(&t.done[l + 1][grp], 1u) == members - 1u;
      }
      __syncthreads();
      if (!s_last) break;
      __threadfence();
      compose_group(t, l, grp, g.M, reinterpret_cast<unsigned *>(psm));
      item = grp;
    }
  }
}

// 3. offsets of the blocks that start in each segment
struct ParseOut {
  unsigned long long *offs;          // [nb]
  unsigned long long *status;        // [0] payload length + 1 once block nb-1 is sized, [1] error
  unsigned long long n;              // elements (when n_dev is null)
  const unsigned long long *n_dev;   // elements, read on the device (optional)
  unsigned long long maxc;           // validation bound of the whole stream (when n_dev is null)
  bool ref_bound;                    // also bound by the reference's 8n+1024 / 4n+4 limit
};

// element count, block count and validation bound of a parse
struct ParseDims {
  unsigned long long n, nb, nlast, lim;
  __device__ ParseDims(const ParseGeom &g, const ParseOut &o) {
    n = o.n_dev ? *o.n_dev : o.n;
    nb = (n + g.B - 1) / g.B;
    nlast = n ? n - (nb - 1) * g.B : 0;
    const unsigned long long maxc =
        !o.ref_bound ? ~0ull : (o.n_dev ? (g.tags ? 8ull * n + 1024ull : 4ull * n + 4ull) : o.maxc);
    // validation bound in payload coordinates (the offset table is 8 bytes)
    lim = maxc > 8 ? (maxc - 8 < g.len ? maxc - 8 : g.len) : 0;
  }
};

// end of the last block (nlast elements), at payload offset p with its bit
// count byte *bcp; 0 and *err (1: no bit count byte, 2: invalid) on failure
__device__ __forceinline__ unsigned long long last_block_end(const ParseGeom &g, const ParseDims &d,
                                                             unsigned long long p, const unsigned char *bcp,
                                                             unsigned long long *err) {
  if (d.nlast <= 1) return p + 4 + (g.cpu ? 1 : 0) + (g.tags ? 1 : 0);
  if (p + 4 >= d.lim) { *err = 1; return 0; }
  const unsigned bc = *bcp;
  if (bc > 32u) { *err = 2; return 0; }
  return p + block_bytes((unsigned)d.nlast, bc, g.tags);
}

constexpr int kWriteThreads = 64;

__global__ void __launch_bounds__(kWriteThreads)
parse_write_kernel(ParseGeom g, ParseTree t, ParseOut o, ParseGuess u) {
  __shared__ __align__(16) unsigned char raw[kSegStage];
  __shared__ unsigned short list[kSegList];
  __shared__ unsigned s_cnt, s_skip;
  if (threadIdx.x == 0) s_skip = parse_settled(u, o.status);
  __syncthreads();
  if (s_skip) return;
  const ParseDims d(g, o);
  if (d.n == 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0) o.status[0] = 1;     // empty stream: nothing to walk
    return;
  }
  const BlockLen lens(g);
  for (unsigned j = blockIdx.x; j < t.cnt[0]; j += gridDim.x) {
    const unsigned long long s0 = (unsigned long long)j * kSegBytes;
    // true entry and first block: the prefixes of this segment's groups
    unsigned x = 0;
    unsigned long long idx0 = 0;
    for (int l = t.levels - 2; l >= 0; l--) {              // the top level is one item, entered at 0
      const unsigned item = j >> (l * t.lgG);
      if (x == kStuck || (item & ((1u << t.lgG) - 1u)) == 0) continue;   // a first member: entered as its group
      const unsigned long long v = l == 0 ? (unsigned long long)t.p0[(size_t)j * g.M + x]
                                          : t.p[l][(size_t)item * g.M + x];
      idx0 += v >> kExitBits;
      x = (unsigned)(v & kStuck);
    }
    if (x == kStuck || idx0 >= d.nb) return;               // and so are all segments after this one
    __syncthreads();
    const unsigned lead = stage_segment(g, s0, raw);
    __syncthreads();
    const unsigned char *buf = raw + lead;
    if (threadIdx.x == 0) {
      const unsigned long long left = d.nb - idx0;         // blocks from idx0 on, the last one included
      const unsigned long long rl = d.lim > s0 ? d.lim - s0 : 0;
      const unsigned rlim = (unsigned)(rl < kSegBytes + 5u ? rl : kSegBytes + 5u);
      const unsigned full = (unsigned)(left - 1 < kSegList ? left - 1 : kSegList);   // full blocks to walk
      unsigned p = x, c = 0;
      unsigned long long err = 0;
      while (p < kSegBytes && c < full) {
        list[c++] = (unsigned short)p;
        if (p + 4u >= rlim) { err = 1; break; }
        const unsigned len = lens(buf[p + 4u]);
        if (!len) { err = 2; break; }
        p += len;
      }
      if (!err && p < kSegBytes && idx0 + c == d.nb - 1) {
        // the last block, with its own element count
        list[c++] = (unsigned short)p;
        const unsigned long long q = last_block_end(g, d, s0 + p, buf + p + 4u, &err);
        if (q > d.lim) err = 3;
        else if (q) o.status[0] = q + 1;
      }
      if (err) atomicExch(o.status + 1, err);
      s_cnt = c;
    }
    __syncthreads();
    for (unsigned k = threadIdx.x; k < s_cnt; k += kWriteThreads) o.offs[idx0 + k] = s0 + list[k];
  }
}

// The checked guess.  A CTA of NW warps takes a tile of NW segments of `unit`
// bytes, staged with the two segments before it; tiles are claimed in order (a
// look-back only waits for tiles held by running CTAs).  Each warp finds the
// entry of its segment, then the lanes of one warp walk the segments side by
// side (one lane per warp took twice as long: its instructions fill a whole
// warp's issue slots).  What counts is the length of the serial walks: 2 KB
// segments (19 to 40 blocks of ordinary fields) with walks from one segment
// ahead, which on fields of every kind left one entry in all but one in a
// thousand cases (1 KB ahead: in three of four).  Where they did not, the
// entry is the exit of the segment before it, one more walk; the first
// segment of a tile starts its walks from two segments ahead instead.
constexpr unsigned kNoEntry = 0xFFFFFFFFu;

// Stages the payload bytes [s0, s0 + bytes) as block lengths: tab[lead + k] is
// the length of a full block whose bit count byte is byte s0 + k (0: invalid,
// or past the payload's end), and a walk's step is p += tab[p + 4], one load
// and one add.  Returns lead.  (A step that loads the byte and works its
// length out takes three times as long; converting every byte costs the CTA
// about 1 K issue slots per scheduler.)
__device__ __forceinline__ unsigned stage_steps(const ParseGeom &g, unsigned long long s0, unsigned bytes,
                                                const BlockLen &lens, unsigned short *tab) {
  const unsigned char *a = g.p + s0;
  const unsigned lead = (unsigned)(reinterpret_cast<uintptr_t>(a) & 15u);
  const unsigned long long rest = g.len > s0 ? g.len - s0 : 0ull;
  const unsigned have = (unsigned)(rest < bytes ? rest : bytes) + lead;    // staged bytes that exist
  const unsigned nq = (bytes + lead + 15u) >> 4;
  const unsigned char *al = a - lead;
  constexpr unsigned kU = 2;   // chunks in flight per thread
  for (unsigned q0 = threadIdx.x; q0 < nq; q0 += kU * blockDim.x) {
    uint4 v[kU];
#pragma unroll
    for (unsigned u = 0; u < kU; u++) {
      const unsigned o = 16u * (q0 + u * blockDim.x);
      v[u] = make_uint4(~0u, ~0u, ~0u, ~0u);
      // from the second chunk on, and for s0 > 0 from the first, no byte lies before the payload
      if ((s0 || o >= lead) && o + 16u <= have) {
        v[u] = __ldg(reinterpret_cast<const uint4 *>(al + o));
      } else if (o < have) {
        unsigned w[4] = {~0u, ~0u, ~0u, ~0u};
#pragma unroll 1
        for (unsigned k = 0; k < 16; k++)
          if ((s0 || o + k >= lead) && o + k < have)
            w[k >> 2] ^= (unsigned)(__ldg(al + o + k) ^ 0xffu) << (8u * (k & 3u));
        v[u] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
#pragma unroll
    for (unsigned u = 0; u < kU; u++) {
      const unsigned q = q0 + u * blockDim.x;
      if (q >= nq) continue;
      const unsigned in[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
      unsigned out[8];
#pragma unroll
      for (unsigned k = 0; k < 8; k++)
        out[k] = lens((in[k >> 1] >> (16u * (k & 1u))) & 0xffu) |
                 (lens((in[k >> 1] >> (16u * (k & 1u) + 8u)) & 0xffu) << 16);
      reinterpret_cast<uint4 *>(tab)[2 * q] = make_uint4(out[0], out[1], out[2], out[3]);
      reinterpret_cast<uint4 *>(tab)[2 * q + 1] = make_uint4(out[4], out[5], out[6], out[7]);
    }
  }
  return lead;
}

// Walks from the block starts e < M up to place dist (step: the table at the
// first start's bit count byte): the distance past it at which all that do not
// stop leave, or kNoEntry where none arrives or two leave in different places.
// All lanes of a warp.  Most starts have an invalid bit count byte; the rest
// go through `keep` to the lanes, a new one whenever a lane's walk ends.
// Of blocks of zeros every start is valid and no walk meets another: a look
// every 16 rounds ends it once two places differ, or after `rounds` of them.
__device__ __forceinline__ unsigned warm_walks(const unsigned short *step, unsigned dist, unsigned M, unsigned rounds,
                                               unsigned short *keep) {
  const unsigned lane = threadIdx.x & 31;
  unsigned kept = 0;
#pragma unroll 2
  for (unsigned e0 = 0; e0 < M; e0 += 32) {
    const unsigned e = e0 + lane;
    const bool c = e < M && step[e] != 0;
    const unsigned m = __ballot_sync(0xffffffffu, c);
    if (c) keep[kept + __popc(m & ((1u << lane) - 1u))] = (unsigned short)e;
    kept += (unsigned)__popc(m);
  }
  __syncwarp();
  unsigned lo = kNoEntry, hi = 0u;
  unsigned next = 32, p = lane < kept ? keep[lane] : kNoEntry;
  bool open = false;
  for (unsigned r = 1; __any_sync(0xffffffffu, p != kNoEntry); r++) {
    // four blocks between refills; a walk that stops stays where it is
    unsigned last = p;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      last = p;
      if (p < dist) p += step[p];
    }
    if (p != kNoEntry) {
      if (p >= dist) {
        lo = min(lo, p - dist);
        hi = max(hi, p - dist);
        p = kNoEntry;
      } else if (p == last) {
        p = kNoEntry;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, p == kNoEntry);
    const unsigned mine = next + __popc(m & ((1u << lane) - 1u));
    if (p == kNoEntry && mine < kept) p = keep[mine];
    next += (unsigned)__popc(m);
    if ((r & 15u) == 0u) {
      const unsigned l = __reduce_min_sync(0xffffffffu, lo);
      open = r >= rounds || (l != kNoEntry && l != __reduce_max_sync(0xffffffffu, hi));
      if (open) break;
    }
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  __syncwarp();
  return open || lo != hi ? kNoEntry : lo;
}

// State of a tile between its two halves.
template <int NW>
struct GuessTile {
  unsigned tile, total;
  unsigned entry[NW], exit[NW], cnt[NW], off[NW];
};

// Back half of a tile: look-back, entries checked, offsets written.
template <int NW>
__device__ __forceinline__ void guess_back(const ParseGeom &g, const ParseOut &o, const ParseGuess &u,
                                           const ParseDims &d, const GuessTile<NW> &s, const unsigned short *lists) {
  const unsigned w = threadIdx.x >> 5, lane = threadIdx.x & 31, tile = s.tile;
  const Prefix pf = lookback_cta<NW>(u.desc, tile, s.total, 0ull, reinterpret_cast<int *>(u.words + 2));
  if (threadIdx.x < NW) {
    const unsigned k = threadIdx.x;
    __threadfence();   // thread 0 has read the descriptor of the tile before
    // a segment that holds a block of the stream starts where the one before it ended
    const unsigned before = k ? s.exit[k - 1] : (tile ? (unsigned)ld_relaxed_u64(u.desc[tile - 1].pad) : 0u);
    if (pf.bytes + s.off[k] < d.nb && s.entry[k] != before) u.words[1] = 1u;
  }
  const unsigned long long s0 = ((unsigned long long)tile * NW + w) * u.unit, idx0 = pf.bytes + s.off[w];
  const unsigned short *list = lists + (size_t)w * u.list;
  const unsigned c = s.cnt[w];
  for (unsigned k = lane; k < c && idx0 + k < d.nb; k += 32) o.offs[idx0 + k] = s0 + list[k];
  if (lane == 0) {
    if (d.n == 0) {
      if (tile == 0 && w == 0) o.status[0] = 1;
    } else if (d.nb - 1 >= idx0 && d.nb - 1 < idx0 + c) {
      const unsigned long long p = s0 + list[d.nb - 1 - idx0];
      unsigned long long err = 0;
      const unsigned long long q = last_block_end(g, d, p, g.p + p + 4u, &err);
      if (q && q <= d.lim) o.status[0] = q + 1;
    }
  }
}

// A CTA runs one tile behind: it publishes a tile's count before it looks
// back for the tile before, so that a look-back's wait for the other CTAs'
// tiles overlaps a tile of work.
template <int NW>
__global__ void __launch_bounds__(NW * 32, NW > 4 ? 1024 / (NW * 32) : 1)
parse_guess_kernel(ParseGeom g, unsigned ntiles, ParseOut o, ParseGuess u) {
  extern __shared__ __align__(16) unsigned char psm[];
  __shared__ GuessTile<NW> sh[2];
  __shared__ unsigned s_claim, s_failed;
  const unsigned w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // block lengths by bit count byte of the two segments before the tile and
  // its own; then, twice, per segment the kept walks and the block list
  unsigned short *tab = reinterpret_cast<unsigned short *>(psm);
  unsigned short *lists_all = tab + (size_t)(NW + 2) * u.unit + 48;
  const ParseDims d(g, o);
  const BlockLen lens(g);
  // rounds (of four blocks) of 64 KB of the shortest blocks: more than
  // blockSize 64 can take, where ordinary data takes a few tens.  Decoding 4 M
  // zeros (us, every entry of 16 KB segments walked / no end but the last walk's
  // / now): plain codec, blockSize 64 1390 / 950 / 458, 128 1670 / 2380 / 493,
  // 256 2250 / 8530 / 860; topology, 64 544 / 306 / 189, 256 313 / 806 / 154.
  const unsigned rounds = 16384u / lens.base;
  unsigned cur = 0;
  bool pending = false;
  while (true) {
    if (threadIdx.x == 0) {
      s_claim = atomicAdd(u.words, 1u);
      s_failed = *reinterpret_cast<volatile unsigned *>(u.words + 1);
    }
    __syncthreads();
    const unsigned tile = s_claim;
    // after a failed guess the exact parse will run: only let the look-backs of others pass
    const bool failed = s_failed != 0u, more = tile < ntiles && !failed;
    if (failed && tile < ntiles && threadIdx.x == 0) publish_aggregate(u.desc, tile, 0ull, 0ull);
    GuessTile<NW> &s = sh[cur];
    unsigned short *lists = lists_all + (size_t)cur * NW * u.list;
    if (more) {
      const unsigned long long t0 = (unsigned long long)tile * NW * u.unit;
      const unsigned back = tile ? 2u * u.unit : 0u;
      const unsigned lead = stage_steps(g, t0 - back, back + NW * u.unit + 5u, lens, tab);
      __syncthreads();
      // step[p]: length of the block that starts at byte p of the tile
      const unsigned short *step = tab + lead + back + 4u;
      {
        const unsigned at = w * u.unit;                  // this warp's segment
        const unsigned long long s0 = t0 + at;
        unsigned entry = kNoEntry;
        if (s0 == 0) {
          entry = 0u;
        } else if (s0 < g.len) {
          // a walk from payload offset 0 is the true one
          unsigned short *keep = lists + (size_t)w * u.list;
          entry = warm_walks(step + at - u.unit, u.unit, s0 == u.unit ? 1u : g.M, rounds, keep);
          if (entry == kNoEntry && w == 0)
            entry = warm_walks(step - 2u * u.unit, 2u * u.unit, s0 == 2u * u.unit ? 1u : g.M, rounds, keep);
        }
        if (lane == 0) s.entry[w] = entry;
      }
      __syncthreads();
      if (w == 0) {
        unsigned c = 0, exit = kStuck, entry = lane < NW ? s.entry[lane] : kNoEntry;
        const unsigned at = lane * u.unit, end = at + u.unit;
        bool walk = entry != kNoEntry;
        while (true) {
          if (walk) {
            unsigned short *list = lists + (size_t)lane * u.list;
            unsigned p = at + entry, len = 1u;
            while (len && p < end) {         // length 0: past the last block, or a stream that is not valid
              len = step[p];
              list[c++] = (unsigned short)(p - at);
              p += len;
            }
            if (p >= end) exit = p - end;
          }
          // an entry the walks ahead left open is the exit of the segment before
          const unsigned before = __shfl_up_sync(0xffffffffu, exit, 1);
          walk = entry == kNoEntry && lane > 0 && lane < NW && before != kStuck;
          if (walk) entry = before;
          if (!__any_sync(0xffffffffu, walk)) break;
        }
        unsigned inc = c;
#pragma unroll
        for (int r = 1; r < NW; r <<= 1) {
          const unsigned v = __shfl_up_sync(0xffffffffu, inc, r);
          if (lane >= (unsigned)r) inc += v;
        }
        if (lane < NW) {
          s.entry[lane] = entry;
          s.exit[lane] = exit;
          s.cnt[lane] = c;
          s.off[lane] = inc - c;
        }
        if (lane == NW - 1) {
          s.tile = tile;
          s.total = inc;
          // the exit first: a reader of the descriptor, past a fence, sees it
          st_relaxed_u64(u.desc[tile].pad, exit);
          __threadfence();
          publish_aggregate(u.desc, tile, inc, 0ull);
        }
      }
    }
    __syncthreads();
    if (pending) guess_back<NW>(g, o, u, d, sh[cur ^ 1u], lists_all + (size_t)(cur ^ 1u) * NW * u.list);
    if (tile >= ntiles) break;
    pending = more;
    cur ^= 1u;
    __syncthreads();
  }
}

// blockSize 1: every block has the same length
__global__ void parse_ones_kernel(ParseGeom g, ParseOut o) {
  const unsigned long long n = o.n_dev ? *o.n_dev : o.n;
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  const unsigned len = 4u + (g.cpu ? 1u : 0u) + (g.tags ? 1u : 0u);
  if (i == 0) {
    const unsigned long long maxc =
        !o.ref_bound ? ~0ull : (o.n_dev ? (g.tags ? 8ull * n + 1024ull : 4ull * n + 4ull) : o.maxc);
    const unsigned long long lim = (maxc > 8 ? (maxc - 8 < g.len ? maxc - 8 : g.len) : 0);
    if (n * len > lim) o.status[1] = 3ull;
    else o.status[0] = n * len + 1;
  }
  for (unsigned long long k = i; k < n; k += stride) o.offs[k] = k * len;
}

static unsigned parse_M(int B, bool tags) { return block_bytes((unsigned)B, 32u, tags) + (B == 1 ? 1u : 0u); }

// Members of a group: up to 32, fewer (down to 8) where that lets the
// segment functions of a group fit 40 KB of shared memory (M <= 1280, every
// topology blockSize); larger blocks compose 32 members from L2.
constexpr size_t kStageBytes = 40960;

static int parse_lg_group(unsigned M, bool *staged) {
  for (int lg = 5; lg >= 3; lg--) {
    *staged = ((size_t)M * 4 << lg) <= kStageBytes;
    if (*staged) return lg;
  }
  return 5;
}

static unsigned parse_segments(unsigned long long len) {
  return (unsigned)(len ? (len + kSegBytes - 1) / kSegBytes : 1);
}

// Segments of a guess tile and their size (seven of the largest blocks): 8,
// fewer where the blocks are large, within 64 KB of block lengths (0: no
// guess, the exact parse alone: the plain codec's largest blocks).
static unsigned parse_guess_warps(unsigned M, unsigned *unit) {
  *unit = std::max(2048u, (7u * M + 15u) & ~15u);
  for (unsigned nw = 8; nw >= 2; nw >>= 1)
    if ((nw + 2) * *unit <= 32768u) return nw;
  return 0;
}

static size_t parse_guess_tiles(unsigned long long len, unsigned M) {
  unsigned unit;
  const unsigned nw = parse_guess_warps(M, &unit);
  return nw ? (size_t)((len + (unsigned long long)nw * unit - 1) / ((unsigned long long)nw * unit)) : 0;
}

static int parse_levels(unsigned nseg, int lgG, unsigned *cnt) {
  int L = 0;
  unsigned c = nseg;
  cnt[L++] = c;
  while (c > 1 && L < kMaxLevels) {
    c = (c + (1u << lgG) - 1) >> lgG;
    cnt[L++] = c;
  }
  return L;
}

size_t parse_scratch_bytes(unsigned long long buf_len, int B, bool tags) {
  if (B == 1) return 1024;
  const unsigned M = parse_M(B, tags);
  unsigned cnt[kMaxLevels];
  bool staged;
  const int lg = parse_lg_group(M, &staged);
  const int L = parse_levels(parse_segments(buf_len), lg, cnt);
  size_t s = a256((size_t)cnt[0] * M * 4) * (staged ? 1 : 2), done = 0;
  for (int l = 1; l < L; l++) {
    s += 2 * a256((size_t)cnt[l] * M * 8);
    done += cnt[l];
  }
  return s + a256(done * 4 + 4) + a256((parse_guess_tiles(buf_len, M) + 1) * sizeof(TileDesc)) + 1024;
}

int parse_stream(szp_b200_ctx *ctx, Arena &A, const unsigned char *d_payload, unsigned long long buf_len,
                 unsigned long long n, const unsigned long long *d_n, int B, bool tags, bool ref_bound,
                 unsigned long long *d_offs, unsigned long long *d_status, bool cpu) {
  cudaStream_t s = ctx->stream;
  ParseGeom g;
  g.cpu = cpu;
  g.p = d_payload;
  g.len = buf_len;
  g.B = B;
  g.tags = tags;
  g.full_tag = tags ? (2u * (unsigned)B + 7u) / 8u : 0u;
  g.M = parse_M(B, tags);
  ParseOut o;
  o.offs = d_offs;
  o.status = d_status;
  o.n = n;
  o.n_dev = d_n;
  o.maxc = tags ? 8ull * n + 1024ull : 4ull * n + 4ull;
  o.ref_bound = ref_bound;
  if (cuda_fail(cudaMemsetAsync(d_status, 0, 2 * sizeof(unsigned long long), s), "memset")) return -1;
  if (B == 1) {
    parse_ones_kernel<<<ctx->sm_count * 4, 256, 0, s>>>(g, o);
    ctx->launches += 1;
    return cuda_fail(cudaGetLastError(), "stream parser launch") ? -1 : 0;
  }
  if (buf_len >= (unsigned long long)kSegBytes << 30) { set_error("stream too long for the parser"); return -1; }
  const unsigned nseg = parse_segments(buf_len);
  ParseGuess u{};
  ParseTree t{};
  t.lgG = parse_lg_group(g.M, &t.staged);
  t.levels = parse_levels(nseg, t.lgG, t.cnt);
  if (t.levels > 1) {
    t.f0 = A.take<unsigned>((size_t)nseg * g.M);
    t.p0 = t.staged ? t.f0 : A.take<unsigned>((size_t)nseg * g.M);
    bool ok = t.f0 && t.p0;
    size_t done = 0;
    for (int l = 1; l < t.levels; l++) {
      t.f[l] = A.take<unsigned long long>((size_t)t.cnt[l] * g.M);
      t.p[l] = A.take<unsigned long long>((size_t)t.cnt[l] * g.M);
      ok = ok && t.f[l] && t.p[l];
      done += t.cnt[l];
    }
    unsigned *d = A.take<unsigned>(done);
    // the tiles' descriptors, then the guess's words
    const unsigned nw = parse_guess_warps(g.M, &u.unit);
    const size_t ntiles = parse_guess_tiles(buf_len, g.M);
    u.desc = A.take<TileDesc>(ntiles + 1);
    if (!ok || !d || !u.desc) { set_error("scratch arena too small for the stream parser"); return -1; }
    if (cuda_fail(cudaMemsetAsync(d, 0, done * 4, s), "memset")) return -1;
    for (int l = 1; l < t.levels; l++) { t.done[l] = d; d += t.cnt[l]; }
    u.words = reinterpret_cast<unsigned *>(u.desc + ntiles);
    if (cuda_fail(cudaMemsetAsync(u.desc, 0, (ntiles + 1) * sizeof(TileDesc), s), "memset")) return -1;
    if (nw) {
      u.list = std::max(g.M, u.unit / 5u + 2u);
      const size_t smem = 2 * ((size_t)(nw + 2) * u.unit + 48 + 2 * (size_t)nw * u.list);
      auto k = nw == 8 ? parse_guess_kernel<8> : nw == 4 ? parse_guess_kernel<4> : parse_guess_kernel<2>;
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      const unsigned per_sm = std::max(1u, (unsigned)(220u * 1024u / smem));
      k<<<(unsigned)std::min<size_t>(ntiles, (size_t)ctx->sm_count * per_sm), nw * 32, smem, s>>>(g, (unsigned)ntiles,
                                                                                                o, u);
      ctx->launches += 1;
    }
    const unsigned threads = std::min(1024u, (g.M + 31u) & ~31u);
    const size_t smem = std::max<size_t>(kSegStage, t.staged ? ((size_t)g.M * 4 << t.lgG) : 0);
    parse_seg_kernel<<<std::min(nseg, (unsigned)ctx->sm_count * 6u), threads, smem, s>>>(g, t, u, d_status);
    ctx->launches += 1;
  }
  parse_write_kernel<<<std::min(nseg, (unsigned)ctx->sm_count * 16u), kWriteThreads, 0, s>>>(g, t, o, u);
  ctx->launches += 1;
  return cuda_fail(cudaGetLastError(), "stream parser launch") ? -1 : 0;
}

}  // namespace tsz
