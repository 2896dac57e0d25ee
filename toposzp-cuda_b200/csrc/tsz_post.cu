// Post-processing of a decoded field with the exact serial-raster semantics of
// the reference drivers (example/test_cuda_topology.cu:117-326, :493-531 and
// example/test_cuda_topology_3d.cu:75-434, :600-631).
//
// Each reference pass visits points in raster order and updates them in
// place, so a point sees the FINAL values of earlier points and the
// PRE-PASS values of later points.  Only a pass's candidates change (extrema
// for the stencil and enforcement passes, lost saddles for RBF, saddles for
// the axis-pattern stencil), so the passes run over compact candidate lists
// and update F in place as well:
//   * a candidate's result goes to F[e] and, with the pass's generation, to
//     S[e] = (generation << 32) | float bits: one 64-bit word that a reader
//     takes whole (relaxed), so value and readiness never need ordering;
//   * a candidate is computed once every EARLIER candidate it reads has its
//     result for this pass (read from S); otherwise its warp looks again at
//     the missing words, a bounded number of times, and runs what became
//     ready in between, and then it is deferred to the next round;
//   * every LATER point a candidate reads lists that candidate among its own
//     earlier reads, so it cannot have been updated yet: F still holds its
//     pre-pass value, exactly as in the serial pass.
// Rounds repeat over the deferred items until none is left (their number is
// the longest chain of adjacent candidates in raster order).  When the
// stencil pass runs, enforcement is fused into it for every candidate with no
// candidate face neighbour, and the enforcement pass proper runs only over the
// rest (face_item_run, enforce_sparse_kernel).  The raw decoded value each
// point is clamped against is the item's own F value before its write when
// the field is the decoded field itself, else the original field's; the
// axis pass of the decoded field, which follows RBF, has them gathered first.
// Floating-point expressions use explicit round-to-nearest
// intrinsics so that no multiply-add is contracted (the reference host code is
// compiled without contraction).
#include <cfloat>

#include "tsz_lookback.cuh"
#include <algorithm>
#include <mutex>
#include <vector>

#include "tsz_ops.h"

namespace tsz {

enum { kPassStencil = 0, kPassEnforce = 1, kPassRbf = 2, kPassAxis = 3 };

// CTA-wide exclusive scan of one value per thread (kPostThreads threads)
__device__ __forceinline__ unsigned cta_excl_scan_post(unsigned v, unsigned *s_warp, unsigned *total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  unsigned wpre = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < 256 / 32; w++) {
    const unsigned sw = s_warp[w];
    if (w < warp) wpre += sw;
    tot += sw;
  }
  *total = tot;
  return wpre + inc - v;
}
constexpr int kPostThreads = 256;
constexpr int kPostPer = 8;
constexpr int kPostTile = kPostThreads * kPostPer;

__constant__ double c_w2[9];
__constant__ double c_w3[27];

struct PostArgs {
  float *F;                     // the field, updated in place
  // raw decoded value of a point: OL at its entry of the pass's list, else
  // ORIG at the point, else (both null: the field is the decoded field itself)
  // its own F value before its first write in the pass (F[e] changes only by
  // e's own item)
  const float *OL;
  const float *ORIG;
  float *RAW;                   // fused stencil on the decoded field itself: raw values of the items it leaves
  const unsigned *TL, *TH;      // bit planes of the types
  const int *sp;
  unsigned long long n_sp;
  Geom g;
  long long n;
  float eb;
  float eps;
  unsigned gen;                 // generation of the current pass
  unsigned long long *S;        // (generation << 32) | result bits, per point
  const unsigned *R;            // RBF candidates (lost saddles) bitmap
  const unsigned *X;            // interior-extremum bitmap (the stencil / enforcement candidates)
  const unsigned *XP;           // per bitmap word: list position of its first extremum (X entries before it)
  int *err;
  unsigned *restored;
  int spin_limit;               // grid-barrier polls before giving up (0: default)
  // stencil pass fused with enforcement (null: plain stencil pass): bitmap
  // over list positions of the items that still need the enforcement pass
  unsigned *NI;
  const unsigned *ONLY;         // a pass of one launch: bitmap of the list positions that it runs (null: all)
};

// No "memory" clobber: a result word is read whole and carries its own
// readiness, so these loads need no order with the other loads of an item, and
// the compiler may issue them together (a clobber would serialise every load
// after it behind the one before).  A retry re-reads after a barrier.
__device__ __forceinline__ unsigned long long ld_rlx(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void st_rlx(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ int ty(const PostArgs &a, long long q) {
  const long long w = q >> 5;
  const unsigned b = (unsigned)(q & 31);
  return (int)(((a.TL[w] >> b) & 1u) | (((a.TH[w] >> b) & 1u) << 1));
}

// coordinates of flat index e
struct C3 { long long x, y, z; };
__device__ __forceinline__ C3 coords(const Geom &g, long long e) {
  C3 c;
  long long r;
  if (g.nd == 2) { c.x = 0; c.y = fdivmod(e, g.d3, g.m_d3, r); c.z = r; }
  else { c.x = fdivmod(e, g.plane, g.m_plane, r); c.y = fdivmod(r, g.d3, g.m_d3, c.z); }
  return c;
}

// 4/6-neighbour classification on F (stable during a pass)
__device__ __forceinline__ int classify_F(const PostArgs &a, long long q) {
  const float *F = a.F;
  if (a.g.nd == 2)
    return classify4(F[q], F[q - a.g.d3], F[q + a.g.d3], F[q - 1], F[q + 1]);
  return classify6(F[q], F[q - a.g.plane], F[q + a.g.plane], F[q - a.g.d3], F[q + a.g.d3], F[q - 1],
                   F[q + 1]);
}

__device__ __forceinline__ bool bit_at(const unsigned *b, long long q) { return (b[q >> 5] >> (q & 31)) & 1u; }

// q is a candidate of pass PASS (q_interior: q lies in the interior)
template <int PASS>
__device__ __forceinline__ bool is_cand_known(const PostArgs &a, long long q, bool q_interior) {
  if (!q_interior) return false;
  if (PASS == kPassRbf) return bit_at(a.R, q);
  const int t = ty(a, q);
  if (PASS == kPassStencil || PASS == kPassEnforce) return t == 1 || t == 2;
  return t == 3;
}

__device__ __forceinline__ bool interior_off(const PostArgs &a, const C3 &c, int dx, int dy, int dz) {
  bool qi = c.y + dy >= 1 && c.y + dy <= a.g.d2 - 2 && c.z + dz >= 1 && c.z + dz <= a.g.d3 - 2;
  if (a.g.nd == 3) qi = qi && c.x + dx >= 1 && c.x + dx <= a.g.d1 - 2;
  return qi;
}

// neighbour of e at offset (dx, dy, dz) (dx = 0 in 2D) as the serial pass
// sees it; earlier candidates are resolved before e is computed
template <int PASS>
__device__ __forceinline__ float valo(const PostArgs &a, long long e, const C3 &c, int dx, int dy, int dz) {
  const long long q = e + (long long)dx * a.g.plane + (long long)dy * a.g.d3 + dz;
  if (q > e) return a.F[q];
  if (is_cand_known<PASS>(a, q, interior_off(a, c, dx, dy, dz)))
    return __uint_as_float((unsigned)ld_rlx(&a.S[q]));
  return a.F[q];
}

// The earlier candidates that an RBF / axis-pattern item may read and whose
// results for this pass it must wait for: the earlier points of the 3x3(x3)
// box and the points two steps back along each axis.  The candidate tests of
// all of them are issued first, then the result words of the candidates, so a
// check waits for two loads in a row, not one per point.
constexpr int kDepPolls = 1024;

template <int ND>
struct Deps {
  static constexpr int NB = ND == 3 ? 13 : 4;   // earlier box points
  unsigned q[NB + 3];
  float val[NB + 3];                             // their results
  unsigned cand, pend;                           // bit i: a candidate; its result is missing
};

template <int PASS, int ND>
__device__ __forceinline__ void deps_find(const PostArgs &a, long long e, const C3 &c, Deps<ND> &d) {
  int k = 0;
  d.cand = 0;
#pragma unroll
  for (int dx = (ND == 3 ? -1 : 0); dx <= 0; dx++)
#pragma unroll
    for (int dy = -1; dy <= 1; dy++)
#pragma unroll
      for (int dz = -1; dz <= 1; dz++) {
        if (dx == 0 && (dy > 0 || (dy == 0 && dz >= 0))) continue;
        const long long q = e + (long long)dx * a.g.plane + (long long)dy * a.g.d3 + dz;
        d.q[k] = (unsigned)q;
        d.cand |= (is_cand_known<PASS>(a, q, interior_off(a, c, dx, dy, dz)) ? 1u : 0u) << k;
        k++;
      }
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const int dx = j == 0 ? -2 : 0, dy = j == 1 ? -2 : 0, dz = j == 2 ? -2 : 0;
    const bool in = (ND == 3 || j > 0) && c.x + dx >= 0 && c.y + dy >= 0 && c.z + dz >= 0;
    const long long q = e + (long long)dx * a.g.plane + (long long)dy * a.g.d3 + dz;
    d.q[Deps<ND>::NB + j] = (unsigned)q;
    d.cand |= (in && is_cand_known<PASS>(a, q, interior_off(a, c, dx, dy, dz)) ? 1u : 0u) << (Deps<ND>::NB + j);
  }
  d.pend = d.cand;
}

// looks at the missing results once (all loads in flight together); true when
// none is missing any more
template <int ND>
__device__ __forceinline__ bool deps_ready(const PostArgs &a, Deps<ND> &d) {
  constexpr int N = Deps<ND>::NB + 3;
  unsigned long long w[N];
#pragma unroll
  for (int i = 0; i < N; i++) w[i] = ((d.pend >> i) & 1u) ? ld_rlx(&a.S[d.q[i]]) : 0ull;
#pragma unroll
  for (int i = 0; i < N; i++)
    if (((d.pend >> i) & 1u) && (unsigned)(w[i] >> 32) == a.gen) {
      d.val[i] = __uint_as_float((unsigned)w[i]);
      d.pend &= ~(1u << i);
    }
  return d.pend == 0u;
}

// ----------------------------------------------------------------------------
// per-point updates
// ----------------------------------------------------------------------------
__device__ __forceinline__ float clampf(float v, float lo, float hi) {
  if (v > hi) v = hi;
  if (v < lo) v = lo;
  return v;
}

// Face neighbours of a stencil / enforcement item as the serial pass sees
// them: xm, ym, zm (earlier points: results of earlier candidates, else F)
// and xp, yp, zp (later points: F).  In 2D the x pair is unused.
struct Face { float xm, xp, ym, yp, zm, zp; };

// 2D stencil (example/test_cuda_topology.cu:118-165)
__device__ __forceinline__ float stencil2(const PostArgs &a, const Face &f, float cur, int t, int s, float o) {
  const float hi = __fadd_rn(o, a.eb), lo = __fsub_rn(o, a.eb);
  float m = cur;
  const float nb[4] = {f.ym, f.yp, f.zm, f.zp};   // rows -1, +1, then columns -1, +1
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (t == 1 ? (nb[k] > m) : (nb[k] < m)) m = nb[k];
  float target;
  if (t == 1) target = __fmul_rn(m, __fadd_rn(1.0f, __fmul_rn((float)s, FLT_EPSILON)));
  else if (s == 0) target = __fmul_rn(m, __fsub_rn(1.0f, FLT_EPSILON));
  else target = __fmul_rn(m, __fsub_rn(1.0f, __fmul_rn(__fdiv_rn(1.0f, (float)s), FLT_EPSILON)));
  return clampf(target, lo, hi);
}

// 3D stencil (example/test_cuda_topology_3d.cu:77-128)
__device__ __forceinline__ float stencil3(const PostArgs &a, const Face &f, int t, int s, float o) {
  const float d = __fmul_rn(a.eb, 0.999f);
  const float hi = __fadd_rn(o, d), lo = __fsub_rn(o, d);
  float target;
  if (t == 1) {
    const float m = fmaxf(fmaxf(f.xm, f.xp), fmaxf(fmaxf(f.ym, f.yp), fmaxf(f.zm, f.zp)));
    target = __fmul_rn(m, __fadd_rn(1.0f, __fmul_rn((float)s, FLT_EPSILON)));
  } else {
    const float m = fminf(fminf(f.xm, f.xp), fminf(fminf(f.ym, f.yp), fminf(f.zm, f.zp)));
    target = (s == 0) ? __fmul_rn(m, __fsub_rn(1.0f, FLT_EPSILON))
                      : __fmul_rn(m, __fsub_rn(1.0f, __fmul_rn(__fdiv_rn(1.0f, (float)s), FLT_EPSILON)));
  }
  return clampf(target, lo, hi);
}

// enforcement (example/test_cuda_topology.cu:168-198, _3d.cu:131-167)
template <int ND>
__device__ __forceinline__ float enforce(const PostArgs &a, const Face &f, float cur, int t, float o) {
  const float d = __fmul_rn(a.eb, 0.999f);
  const float hi = __fadd_rn(o, d), lo = __fsub_rn(o, d);
  const float soft = __fmul_rn(0.25f, a.eps);
  float m;
  if (ND == 2) {
    // north, south, west, east
    m = (t == 1) ? fmaxf(fmaxf(f.ym, f.yp), fmaxf(f.zm, f.zp)) : fminf(fminf(f.ym, f.yp), fminf(f.zm, f.zp));
  } else {
    m = (t == 1) ? fmaxf(fmaxf(f.xm, f.xp), fmaxf(fmaxf(f.ym, f.yp), fmaxf(f.zm, f.zp)))
                 : fminf(fminf(f.xm, f.xp), fminf(fminf(f.ym, f.yp), fminf(f.zm, f.zp)));
  }
  if (t == 1) {
    float tg = __fadd_rn(m, soft);
    if (tg > hi) tg = hi;
    if (tg < lo) tg = lo;
    return (cur < tg) ? tg : cur;
  }
  float tg = __fsub_rn(m, soft);
  if (tg < lo) tg = lo;
  if (tg > hi) tg = hi;
  return (cur > tg) ? tg : cur;
}

// An item of the stencil or enforcement pass, held in registers across the
// local retries.  Its face neighbours as the serial pass sees them: the
// earlier ones (x-1 in 3D, y-1, z-1) are results of this pass where they are
// candidates (bits of X; the result word sits at the list position XP of the
// bitmap word plus the extrema before it in the word), F otherwise; the
// later ones are F.  Everything but the missing result words is loaded once;
// a retry reloads only those.
struct FaceItem {
  long long e;
  float cur, o;          // F at e before the item writes, and its raw value
  int t, s;              // type, sort position (stencil)
  Face f;
  unsigned wait;         // bit k: earlier candidate neighbour k not read yet
  unsigned pos[3];       // their list positions
  bool iso;              // no face neighbour is a candidate (fused stencil)
};

template <int PASS, int ND>
__device__ __forceinline__ void face_item_load(const PostArgs &a, const unsigned *__restrict__ list, unsigned idx,
                                               FaceItem &it) {
  const long long e = (long long)list[idx];
  const long long pl = a.g.plane, d3 = a.g.d3;
  it.e = e;
  it.t = (a.TL[e >> 5] >> (unsigned)(e & 31)) & 1u ? 1 : 2;   // an extremum: maximum 01, minimum 10
  it.s = (PASS == kPassStencil && idx < a.n_sp) ? a.sp[idx] : 0;
  it.cur = a.F[e];
  it.o = a.OL ? a.OL[idx] : (a.ORIG ? a.ORIG[e] : it.cur);
  // e is interior: every face neighbour lies in the field
  it.f.xm = ND == 3 ? a.F[e - pl] : 0.f;
  it.f.xp = ND == 3 ? a.F[e + pl] : 0.f;
  it.f.ym = a.F[e - d3];
  it.f.yp = a.F[e + d3];
  it.f.zm = a.F[e - 1];
  it.f.zp = a.F[e + 1];
  unsigned wait = 0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    it.pos[k] = 0;
    if (ND == 2 && k == 0) continue;
    const long long q = e - (k == 0 ? pl : (k == 1 ? d3 : 1ll));
    const long long wi = q >> 5;
    const unsigned bw = a.X[wi], b = (unsigned)(q & 31);
    wait |= ((bw >> b) & 1u) << k;
    it.pos[k] = a.XP[wi] + (unsigned)__popc(bw & ((1u << b) - 1u));
  }
  it.wait = wait;
  it.iso = false;
  if (PASS == kPassStencil && a.NI) {
    unsigned later = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      if (ND == 2 && k == 0) continue;
      const long long q = e + (k == 0 ? pl : (k == 1 ? d3 : 1ll));
      later |= (a.X[q >> 5] >> (unsigned)(q & 31)) & 1u;
    }
    it.iso = (wait | later) == 0u;
  }
}

// Reads the result words still missing; false while one is not final.
__device__ __forceinline__ bool face_item_ready(const PostArgs &a, FaceItem &it) {
  unsigned long long w[3];
#pragma unroll
  for (int k = 0; k < 3; k++) w[k] = ((it.wait >> k) & 1u) ? ld_rlx(&a.S[it.pos[k]]) : 0ull;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    if (((it.wait >> k) & 1u) && (unsigned)(w[k] >> 32) == a.gen) {
      const float v = __uint_as_float((unsigned)w[k]);
      if (k == 0) it.f.xm = v;
      else if (k == 1) it.f.ym = v;
      else it.f.zm = v;
      it.wait &= ~(1u << k);
    }
  }
  return it.wait == 0u;
}

// bits [b, b + 32) of a bitmap of nbits bits (zeros outside)
__device__ __forceinline__ unsigned get32(const unsigned *__restrict__ bm, long long b, long long nbits) {
  const long long w = b >> 5;  // arithmetic shift: floor for negative b
  const unsigned sh = (unsigned)(b & 31);
  const long long nw = (nbits + 31) >> 5;
  const unsigned lo = (w >= 0 && w < nw) ? bm[w] : 0u;
  const unsigned hi = (w + 1 >= 0 && w + 1 < nw) ? bm[w + 1] : 0u;
  return sh ? __funnelshift_r(lo, hi, sh) : lo;
}

// Locks of the RBF box around e (example/test_cuda_topology.cu:229-242,
// example/test_cuda_topology_3d.cu:325-341): box point q is locked when it is
// interior and an interior extremum (a bit of the extremum bitmap a.X) lies
// within Chebyshev distance 1 of it.  Read from the 5x5(x5) window of a.X
// around e, one 5-bit row segment per row (z - 2 .. z + 2).  A segment that
// runs past a row end reads points of the neighbouring row's boundary
// columns, and a row outside the field reads boundary rows or nothing; none
// of them holds an interior extremum, so the window needs no clipping.
// Bit (dx + 1) * 9 + (dy + 1) * 3 + (dz + 1) (dx = 0 in 2D: bit (dy + 1) * 3 + dz + 1).
template <int ND>
__device__ __forceinline__ unsigned box_locks(const PostArgs &a, long long e, const C3 &c) {
  constexpr int NX = ND == 3 ? 5 : 1;
  unsigned seg[NX][5];
#pragma unroll
  for (int i = 0; i < NX; i++)
#pragma unroll
    for (int j = 0; j < 5; j++) {
      const long long b = e + (ND == 3 ? (long long)(i - 2) * a.g.plane : 0ll) + (long long)(j - 2) * a.g.d3 - 2;
      seg[i][j] = get32(a.X, b, a.n) & 31u;
    }
  unsigned m = 0;
#pragma unroll
  for (int dx = (ND == 3 ? -1 : 0); dx <= (ND == 3 ? 1 : 0); dx++)
#pragma unroll
    for (int dy = -1; dy <= 1; dy++) {
      unsigned acc = 0;
#pragma unroll
      for (int ox = (ND == 3 ? -1 : 0); ox <= (ND == 3 ? 1 : 0); ox++)
#pragma unroll
        for (int oy = -1; oy <= 1; oy++) acc |= seg[(ND == 3 ? dx + ox + 2 : 0)][dy + oy + 2];
#pragma unroll
      for (int dz = -1; dz <= 1; dz++) {
        // window bits dz + 1 .. dz + 3 are the columns dz - 1 .. dz + 1
        if (((acc >> (dz + 1)) & 7u) && interior_off(a, c, dx, dy, dz))
          m |= 1u << ((ND == 3 ? (dx + 1) * 9 : 0) + (dy + 1) * 3 + (dz + 1));
      }
    }
  return m;
}

// What an RBF item reads besides the results it waits for, loaded before it
// waits: nothing of it changes before the item is done (a later candidate waits
// for the item, an earlier one's result comes from its word).
template <int ND>
struct RbfItem {
  static constexpr int N = ND == 3 ? 27 : 9, C = N / 2;   // box points, the centre
  float v[N];          // box value at (dx, dy, dz): v[(dx + 1) * 9 + (dy + 1) * 3 + (dz + 1)] (2D: dx = -1 gone)
  float far[6];        // two steps out: x-, y-, z- (as the serial pass sees them), x+, y+, z+
  unsigned chk;        // bit 2 k + s: the neighbour at side s (0 -, 1 +) of axis k is interior and regular
  unsigned locks;
  double den;
  float o;
};

template <int ND>
__device__ __forceinline__ double rbf_weight(unsigned locks, int i) {
  const double ww = ND == 3 ? c_w3[i] : c_w2[i];
  return ((locks >> i) & 1u) ? __dmul_rn(ww, 0.4) : ww;
}

template <int ND>
__device__ __forceinline__ void rbf_load(const PostArgs &a, long long e, const C3 &c, unsigned cand, float o,
                                         RbfItem<ND> &it) {
  constexpr int NB = Deps<ND>::NB;
  const long long pl = a.g.plane, d3 = a.g.d3;
#pragma unroll
  for (int i = 0; i < RbfItem<ND>::N; i++) {
    const int dx = ND == 3 ? i / 9 - 1 : 0, dy = (i / 3) % 3 - 1, dz = i % 3 - 1;
    // an earlier candidate's value is its result
    it.v[i] = i < NB && ((cand >> i) & 1u) ? 0.f : a.F[e + dx * pl + dy * d3 + dz];
  }
  // the far sides, wherever they exist; used where the serial pass reads them
  const long long step[3] = {pl, d3, 1};
  const long long at[3] = {c.x, c.y, c.z}, ext[3] = {a.g.d1, a.g.d2, a.g.d3};
  it.chk = 0;
#pragma unroll
  for (int k = ND == 3 ? 0 : 1; k < 3; k++) {
    it.far[k] = at[k] >= 2 && !((cand >> (NB + k)) & 1u) ? a.F[e - 2 * step[k]] : 0.f;
    it.far[3 + k] = at[k] + 2 < ext[k] ? a.F[e + 2 * step[k]] : 0.f;
    if (at[k] - 1 >= 1 && ty(a, e - step[k]) == 0) it.chk |= 1u << (2 * k);
    if (at[k] + 1 < ext[k] - 1 && ty(a, e + step[k]) == 0) it.chk |= 2u << (2 * k);
  }
  it.locks = box_locks<ND>(a, e, c);
  it.o = o;
  double den = 0.0;
#pragma unroll
  for (int i = 0; i < RbfItem<ND>::N; i++) den = __dadd_rn(den, rbf_weight<ND>(it.locks, i));
  it.den = den;
}

// the results it waited for, and the weighted mean of the box
template <int ND>
__device__ __forceinline__ float rbf_mean(const Deps<ND> &d, RbfItem<ND> &it) {
  constexpr int NB = Deps<ND>::NB;
#pragma unroll
  for (int i = 0; i < NB; i++)
    if ((d.cand >> i) & 1u) it.v[i] = d.val[i];
#pragma unroll
  for (int k = ND == 3 ? 0 : 1; k < 3; k++)
    if ((d.cand >> (NB + k)) & 1u) it.far[k] = d.val[NB + k];
  double num = 0.0;
#pragma unroll
  for (int i = 0; i < RbfItem<ND>::N; i++)
    num = __dadd_rn(num, __dmul_rn(rbf_weight<ND>(it.locks, i), (double)it.v[i]));
  return __double2float_rn(__ddiv_rn(num, it.den));
}

// A trial changes only the centre, so what a trial has to look at in a
// neighbour is worked out once: a neighbour is classified from one axis that
// has the centre in it and one (2D) or two (3D) that do not change.  The
// classification of all seven points in each of up to ten trials was most of
// an item's 3 K instructions, and items wait for one another in chains: RBF
// stage of 100x500x500 105 -> 75 us, of 1800x3600 68 -> 49.

// 2D, with the margin eps: a neighbour c is not regular exactly when both of its
// axes are above or below it.  far: its neighbour away from the centre; p, q:
// the pair across.
struct Side2 { bool above, below; };   // not regular when the centre is below / above c by more than eps

__device__ __forceinline__ Side2 side2(bool check, float c, float far, float p, float q, float eps) {
  const bool hh = c > __fadd_rn(p, eps) && c > __fadd_rn(q, eps);
  const bool hl = c < __fsub_rn(p, eps) && c < __fsub_rn(q, eps);
  const bool across = check && (hh || hl);
  return {across && c > __fadd_rn(far, eps), across && c < __fsub_rn(far, eps)};
}

// 3D: whether a neighbour c is regular with the centre below it, above it, or
// neither; p0, p1 and q0, q1: the pairs of its other two axes.
struct Side3 { bool below, above, level; };

__device__ __forceinline__ Side3 side3(bool check, float c, float far, float p0, float p1, float q0, float q1) {
  const bool h1 = c > p0 && c > p1, l1 = c < p0 && c < p1, h2 = c > q0 && c > q1, l2 = c < q0 && c < q1;
  const bool none = !((h1 || h2) && (l1 || l2));
  const bool high = !(h1 && h2) && !(l1 || l2);    // with its axis to the centre a high one
  const bool low = !(l1 && l2) && !(h1 || h2);
  return {!check || (c > far ? high : none), !check || (c < far ? low : none), !check || none};
}
__device__ __forceinline__ bool regular(const Side3 &s, float c, float tr) {
  return tr < c ? s.below : (tr > c ? s.above : s.level);
}

// 2D RBF saddle restoration (example/test_cuda_topology.cu:227-326)
__device__ __forceinline__ float rbf2(const PostArgs &a, const Deps<2> &d, RbfItem<2> &it, bool &ok) {
  ok = false;
  const float old = it.v[4];
  if (!(it.den > 0.0)) return old;
  float cand = rbf_mean<2>(d, it);
  const float m = __fmul_rn(a.eb, 0.999f);
  const float lo = __fsub_rn(it.o, m), hi = __fadd_rn(it.o, m);
  const float n = it.v[1], s = it.v[7], w = it.v[3], ea = it.v[5];
  {
    const float q = __fmul_rn(0.25f, a.eps);
    float clo = __fsub_rn(fminf(fmaxf(n, s), fmaxf(w, ea)), q);
    float chi = __fadd_rn(fmaxf(fminf(n, s), fminf(w, ea)), q);
    if (clo > chi) {
      const float mid = __fmul_rn(0.5f, __fadd_rn(clo, chi));
      clo = __fsub_rn(mid, q);
      chi = __fadd_rn(mid, q);
    }
    if (cand < clo) cand = clo;
    if (cand > chi) cand = chi;
  }
  if (cand < lo) cand = lo;
  if (cand > hi) cand = hi;
  const bool vu = (it.chk >> 2) & 1u, vd = (it.chk >> 3) & 1u, vl = (it.chk >> 4) & 1u, vr = (it.chk >> 5) & 1u;
  const float u2 = vu ? it.far[1] : 0.f, d2 = vd ? it.far[4] : 0.f, l2 = vl ? it.far[2] : 0.f,
              r2 = vr ? it.far[5] : 0.f;
  const float step = __fsub_rn(cand, old);
  const float eps = a.eps;
  // a neighbour's far point, and the pair across the axis to it
  const Side2 su = side2(vu, n, u2, it.v[0], it.v[2], eps), sd = side2(vd, s, d2, it.v[6], it.v[8], eps);
  const Side2 sl = side2(vl, w, l2, it.v[0], it.v[6], eps), sr = side2(vr, ea, r2, it.v[2], it.v[8], eps);
  const float np = __fadd_rn(n, eps), sp = __fadd_rn(s, eps), wp = __fadd_rn(w, eps), ep = __fadd_rn(ea, eps);
  const float nm = __fsub_rn(n, eps), sm = __fsub_rn(s, eps), wm = __fsub_rn(w, eps), em = __fsub_rn(ea, eps);
  float alpha = 1.0f;
  for (int k = 0; k < 10; k++) {
    float trial = __fadd_rn(old, __fmul_rn(alpha, step));
    if (trial < lo) trial = lo;
    if (trial > hi) trial = hi;
    const float tp = __fadd_rn(trial, eps), tm = __fsub_rn(trial, eps);
    const bool bad = (su.above && n > tp) || (su.below && n < tm) || (sd.above && s > tp) || (sd.below && s < tm) ||
                     (sl.above && w > tp) || (sl.below && w < tm) || (sr.above && ea > tp) || (sr.below && ea < tm);
    // a saddle: one axis above it, the other below
    const bool vh = trial > np && trial > sp, vlo = trial < nm && trial < sm;
    const bool hh = trial > wp && trial > ep, hlo = trial < wm && trial < em;
    if (!bad && ((vh && hlo) || (vlo && hh))) { ok = true; return trial; }
    alpha = __fmul_rn(alpha, 0.5f);
  }
  return old;
}

// 3D RBF (example/test_cuda_topology_3d.cu:317-434).  A trial changes only the
// centre value.
__device__ __forceinline__ float rbf3(const PostArgs &a, const Deps<3> &d, RbfItem<3> &it, bool &ok) {
  ok = false;
  const float old = it.v[13];
  if (!(it.den > 0.0)) return old;
  float cand = rbf_mean<3>(d, it);
  const float m = __fmul_rn(a.eb, 0.999f);
  const float lo = __fsub_rn(it.o, m), hi = __fadd_rn(it.o, m);
  if (cand < lo) cand = lo;
  if (cand > hi) cand = hi;
  const bool cxm = it.chk & 1u, cxp = (it.chk >> 1) & 1u, cym = (it.chk >> 2) & 1u, cyp = (it.chk >> 3) & 1u,
             czm = (it.chk >> 4) & 1u, czp = (it.chk >> 5) & 1u;
  const float fxm = cxm ? it.far[0] : 0.f, fym = cym ? it.far[1] : 0.f, fzm = czm ? it.far[2] : 0.f;
  const float fxp = cxp ? it.far[3] : 0.f, fyp = cyp ? it.far[4] : 0.f, fzp = czp ? it.far[5] : 0.f;
#define V3(dx, dy, dz) it.v[((dx) + 1) * 9 + ((dy) + 1) * 3 + ((dz) + 1)]
  const float xm = V3(-1, 0, 0), xp = V3(1, 0, 0), ym = V3(0, -1, 0), yp = V3(0, 1, 0), zm = V3(0, 0, -1),
              zp = V3(0, 0, 1);
  const Side3 sxm = side3(cxm, xm, fxm, V3(-1, -1, 0), V3(-1, 1, 0), V3(-1, 0, -1), V3(-1, 0, 1));
  const Side3 sxp = side3(cxp, xp, fxp, V3(1, -1, 0), V3(1, 1, 0), V3(1, 0, -1), V3(1, 0, 1));
  const Side3 sym = side3(cym, ym, fym, V3(-1, -1, 0), V3(1, -1, 0), V3(0, -1, -1), V3(0, -1, 1));
  const Side3 syp = side3(cyp, yp, fyp, V3(-1, 1, 0), V3(1, 1, 0), V3(0, 1, -1), V3(0, 1, 1));
  const Side3 szm = side3(czm, zm, fzm, V3(-1, 0, -1), V3(1, 0, -1), V3(0, -1, -1), V3(0, 1, -1));
  const Side3 szp = side3(czp, zp, fzp, V3(-1, 0, 1), V3(1, 0, 1), V3(0, -1, 1), V3(0, 1, 1));
  const float step = __fsub_rn(cand, old);
  float alpha = 1.0f;
  for (int k = 0; k < 10; k++) {
    float tr = __fadd_rn(old, __fmul_rn(alpha, step));
    if (tr < lo) tr = lo;
    if (tr > hi) tr = hi;
    // a saddle: an axis above it and one below
    const bool any_h = (tr > xm && tr > xp) || (tr > ym && tr > yp) || (tr > zm && tr > zp);
    const bool any_l = (tr < xm && tr < xp) || (tr < ym && tr < yp) || (tr < zm && tr < zp);
    if (any_h && any_l && regular(sxm, xm, tr) && regular(sxp, xp, tr) && regular(sym, ym, tr) &&
        regular(syp, yp, tr) && regular(szm, zm, tr) && regular(szp, zp, tr)) {
      ok = true;
      return tr;
    }
    alpha = __fmul_rn(alpha, 0.5f);
  }
#undef V3
  return old;
}

// values around e in 3D: index (dx+2, dy+2, dz+2) over a 5x5x5 window, filled lazily
struct Win3 {
  float v[5][5][5];
  unsigned char have[5][5][5];
  C3 c;  // coordinates of the center
};

template <int PASS>
__device__ __forceinline__ float w3getp(const PostArgs &a, long long e, Win3 &W, int dx, int dy, int dz,
                                        float center) {
  if (dx == 0 && dy == 0 && dz == 0) return center;
  unsigned char &h = W.have[dx + 2][dy + 2][dz + 2];
  if (!h) {
    W.v[dx + 2][dy + 2][dz + 2] = valo<PASS>(a, e, W.c, dx, dy, dz);
    h = 1;
  }
  return W.v[dx + 2][dy + 2][dz + 2];
}

template <int PASS>
__device__ __forceinline__ int cls6_at(const PostArgs &a, long long e, Win3 &W, int dx, int dy, int dz,
                                       float center) {
  return classify6(w3getp<PASS>(a, e, W, dx, dy, dz, center), w3getp<PASS>(a, e, W, dx - 1, dy, dz, center),
                   w3getp<PASS>(a, e, W, dx + 1, dy, dz, center), w3getp<PASS>(a, e, W, dx, dy - 1, dz, center),
                   w3getp<PASS>(a, e, W, dx, dy + 1, dz, center), w3getp<PASS>(a, e, W, dx, dy, dz - 1, center),
                   w3getp<PASS>(a, e, W, dx, dy, dz + 1, center));
}

// the center is a saddle and every regular neighbour stays regular
template <int PASS>
__device__ bool valid3(const PostArgs &a, long long e, const C3 &c, Win3 &W, float trial) {
  if (cls6_at<PASS>(a, e, W, 0, 0, 0, trial) != 3) return false;
  const long long pl = a.g.plane, d3 = a.g.d3;
  if (c.x - 1 >= 1 && ty(a, e - pl) == 0 && cls6_at<PASS>(a, e, W, -1, 0, 0, trial) != 0) return false;
  if (c.x + 1 < a.g.d1 - 1 && ty(a, e + pl) == 0 && cls6_at<PASS>(a, e, W, 1, 0, 0, trial) != 0) return false;
  if (c.y - 1 >= 1 && ty(a, e - d3) == 0 && cls6_at<PASS>(a, e, W, 0, -1, 0, trial) != 0) return false;
  if (c.y + 1 < a.g.d2 - 1 && ty(a, e + d3) == 0 && cls6_at<PASS>(a, e, W, 0, 1, 0, trial) != 0) return false;
  if (c.z - 1 >= 1 && ty(a, e - 1) == 0 && cls6_at<PASS>(a, e, W, 0, 0, -1, trial) != 0) return false;
  if (c.z + 1 < a.g.d3 - 1 && ty(a, e + 1) == 0 && cls6_at<PASS>(a, e, W, 0, 0, 1, trial) != 0) return false;
  return true;
}

// 3D axis-pattern saddle stencil (example/test_cuda_topology_3d.cu:187-314)
__device__ float axis3(const PostArgs &a, long long e, const C3 &c, float o, bool &ok) {
  ok = false;
  Win3 W;
  W.c = c;
  for (int i = 0; i < 125; i++) (&W.have[0][0][0])[i] = 0;
  const float old = a.F[e];
  if (cls6_at<kPassAxis>(a, e, W, 0, 0, 0, old) == 3) return old;
  const float d = __fmul_rn(a.eb, 0.999f);
  const float lo = __fsub_rn(o, d), hi = __fadd_rn(o, d);
  const float nb[6] = {w3getp<kPassAxis>(a, e, W, -1, 0, 0, old), w3getp<kPassAxis>(a, e, W, 1, 0, 0, old),
                       w3getp<kPassAxis>(a, e, W, 0, -1, 0, old), w3getp<kPassAxis>(a, e, W, 0, 1, 0, old),
                       w3getp<kPassAxis>(a, e, W, 0, 0, -1, old), w3getp<kPassAxis>(a, e, W, 0, 0, 1, old)};
  for (int pat = 1; pat <= 6; pat++) {
    float hthr = -1e30f, lthr = 1e30f;
    for (int ax = 0; ax < 3; ax++) {
      const float pmax = fmaxf(nb[2 * ax], nb[2 * ax + 1]);
      const float pmin = fminf(nb[2 * ax], nb[2 * ax + 1]);
      if ((pat >> ax) & 1) { if (pmax > hthr) hthr = pmax; }
      else { if (pmin < lthr) lthr = pmin; }
    }
    if (hthr >= lthr) continue;
    float target = __fmul_rn(0.5f, __fadd_rn(hthr, lthr));
    float nudge = __fmul_rn(__fsub_rn(lthr, hthr), 0.01f);
    if (nudge < FLT_EPSILON) nudge = FLT_EPSILON;
    if (target <= hthr) target = __fadd_rn(hthr, nudge);
    if (target >= lthr) target = __fsub_rn(lthr, nudge);
    if (target <= hthr || target >= lthr) continue;
    if (target > hi || target < lo) continue;
    if (valid3<kPassAxis>(a, e, c, W, target)) { ok = true; return target; }
  }
  return old;
}

// ----------------------------------------------------------------------------
// candidate lists
// ----------------------------------------------------------------------------

// Interior extrema in raster order (X), the interior-extremum and
// interior-saddle bitmaps (Eb, Sb) and, with Z given, the interior saddles in
// raster order, in one pass over the types' bit planes: persistent CTAs take
// tiles of kListTile points in order (one word of 32 points per thread),
// publish their counts and find their list offsets by decoupled look-back
// (extrema in the byte word, saddles in the count word), then write their
// entries through shared memory so each tile's slice of X and Z is stored
// contiguously (X staged from the front of one buffer, Z from its back: a
// point is in at most one list).  A CTA runs one tile behind: it publishes tile
// k's counts before it looks back for tile k-1, so the tiles that a look-back
// waits for are held by CTAs that have published them (tiles are claimed in
// order), and the wait has a tile of work behind it.  The last tile writes the
// totals to tot[0] = (extrema << 32) | saddles.  512^3 field: 241 us from a
// byte per type with both lists, 149 from the planes with X alone, 94
// with the look-back a tile behind and both counts in one scan.
constexpr int kListPer = 32;
constexpr int kListTile = kPostThreads * kListPer;

__global__ void __launch_bounds__(kPostThreads)
list_build_kernel(const unsigned *__restrict__ TL, const unsigned *__restrict__ TH, Geom g, long long n,
                  TileDesc *desc, unsigned *tile_ctr, int *err, unsigned *X, unsigned *Z, unsigned *Eb, unsigned *Sb,
                  unsigned long long *tot, unsigned *XP) {
  __shared__ unsigned s_w[kWarps];
  __shared__ unsigned short s_buf[2][kListTile];   // offsets in the tile
  __shared__ long long s_tile;
  __shared__ unsigned long long s_xb, s_zb;
  const long long ntiles = (n + kListTile - 1) / kListTile;
  long long prev = -1;
  unsigned p_te = 0, p_ts = 0, p_eo = 0;
  for (int cur = 0;; cur ^= 1) {
    if (threadIdx.x == 0) s_tile = (long long)atomicAdd(tile_ctr, 1u);
    __syncthreads();
    const long long tile = s_tile;
    const bool more = tile < ntiles;
    unsigned te = 0, ts = 0, eo = 0;
    if (more) {
      const long long i0 = tile * kListTile + (long long)threadIdx.x * kListPer;
      unsigned em = 0, sm = 0, im = 0;
      if (i0 < n) {
        const unsigned tl = TL[i0 >> 5], th = TH[i0 >> 5];
        long long r, x, y, z;
        if (g.nd == 2) { x = 0; y = fdivmod(i0, g.d3, g.m_d3, r); z = r; }
        else { x = fdivmod(i0, g.plane, g.m_plane, r); y = fdivmod(r, g.d3, g.m_d3, z); }
        if (z + kListPer - 1 < g.d3 && i0 + kListPer <= n) {
          // the 32 points share one row: interior columns 1 .. d3-2
          const bool row_in = y >= 1 && y <= g.d2 - 2 && (g.nd == 2 || (x >= 1 && x <= g.d1 - 2));
          if (row_in) {
            const long long lo = 1 - z, hi = g.d3 - 2 - z;   // interior offsets u in [lo, hi]
            const int ulo = lo > 0 ? (int)lo : 0, uhi = hi < kListPer - 1 ? (int)hi : kListPer - 1;
            if (ulo <= uhi) im = (uhi == 31 ? 0xffffffffu : ((2u << uhi) - 1u)) & ~((1u << ulo) - 1u);
          }
        } else if (g.d3 > kListPer && i0 + kListPer <= n) {
          // two rows: columns z .. d3-1 of one, then 0 .. of the next
          const unsigned k = (unsigned)(g.d3 - z);          // 1 .. 31
          const bool plane_in = g.nd == 2 || (x >= 1 && x <= g.d1 - 2);
          if (plane_in && y >= 1 && y <= g.d2 - 2) im = ((1u << k) - 1u) >> 1;
          if (plane_in && y + 1 <= g.d2 - 2) im |= ~((2u << k) - 1u);
        } else {
          for (int u = 0; u < kListPer && i0 + u < n; u++) {
            bool in = y >= 1 && y <= g.d2 - 2 && z >= 1 && z <= g.d3 - 2;
            if (g.nd == 3) in = in && x >= 1 && x <= g.d1 - 2;
            if (in) im |= 1u << u;
            z++;
            while (z >= g.d3) { z -= g.d3; y++; if (y >= g.d2) { y -= g.d2; x++; } }
          }
        }
        em = (tl ^ th) & im;
        sm = tl & th & im;
        Eb[i0 >> 5] = em;
        Sb[i0 >> 5] = sm;
      }
      // both counts in one scan: a tile has 8192 points
      unsigned tc;
      const unsigned co = cta_excl_scan_post((unsigned)__popc(em) | ((unsigned)__popc(sm) << 16), s_w, &tc);
      te = tc & 0xffffu;
      ts = tc >> 16;
      eo = co & 0xffffu;
      if (threadIdx.x == 0) publish_aggregate(desc, tile, te, ts);
      {
        unsigned short *buf = s_buf[cur];
        const unsigned at = threadIdx.x * kListPer;
        unsigned xe = eo, xs = kListTile - 1 - (co >> 16);
        unsigned mm = em;
        while (mm) { const int u = __ffs(mm) - 1; mm &= mm - 1; buf[xe++] = (unsigned short)(at + u); }
        mm = Z ? sm : 0u;
        while (mm) { const int u = __ffs(mm) - 1; mm &= mm - 1; buf[xs--] = (unsigned short)(at + u); }
      }
    }
    if (prev >= 0) {
      const Prefix pf = lookback_cta<kWarps>(desc, prev, p_te, p_ts, err);
      if (threadIdx.x == 0) {
        s_xb = pf.bytes;
        s_zb = pf.cnt;
        if (prev == ntiles - 1) *tot = ((pf.bytes + p_te) << 32) | (pf.cnt + p_ts);
      }
      __syncthreads();
      const unsigned long long xb = s_xb, zb = s_zb;
      const long long b0 = prev * kListTile;
      // list position of the first extremum of this thread's bitmap word
      const long long i0 = b0 + (long long)threadIdx.x * kListPer;
      if (i0 < n) XP[i0 >> 5] = (unsigned)(xb + p_eo);
      // a list position past n means corrupt tile offsets: recorded, not written
      if (xb + p_te > (unsigned long long)n || zb + p_ts > (unsigned long long)n) {
        if (threadIdx.x == 0) atomicExch(err, kErrMalformed);
      } else {
        const unsigned short *buf = s_buf[cur ^ 1];
        for (unsigned k = threadIdx.x; k < p_te; k += kPostThreads) X[xb + k] = (unsigned)b0 + buf[k];
        if (Z)
          for (unsigned k = threadIdx.x; k < p_ts; k += kPostThreads)
            Z[zb + k] = (unsigned)b0 + buf[kListTile - 1 - k];
      }
    }
    if (!more) break;
    prev = tile;
    p_te = te;
    p_ts = ts;
    p_eo = eo;
  }
}

// Lost saddles (RBF candidates): saddles of the original field that F no
// longer classifies as saddles (example/test_cuda_topology.cu:244-254).  A
// warp takes 32 words of the saddle bitmap, lists their points in shared
// memory in raster order and classifies them 32 at a time, so that its lanes
// read neighbouring points.
__global__ void __launch_bounds__(256)
fn_detect_kernel(PostArgs a, const unsigned *__restrict__ Sb, unsigned nwords, unsigned *__restrict__ R,
                 unsigned *__restrict__ Y, unsigned *y_count) {
  __shared__ unsigned short s_pt[8][1024];
  __shared__ unsigned s_lost[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned w0 = (blockIdx.x * 8u + warp) * 32u;
  if (w0 >= nwords) return;
  unsigned m = w0 + lane < nwords ? Sb[w0 + lane] : 0u;
  s_lost[warp][lane] = 0u;
  unsigned inc = __popc(m);
  const unsigned c = inc;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  const unsigned total = __shfl_sync(0xffffffffu, inc, 31);
  unsigned o = inc - c;
  while (m) {
    const int u = __ffs(m) - 1;
    m &= m - 1;
    s_pt[warp][o++] = (unsigned short)(32 * lane + u);
  }
  __syncwarp();
  const long long base = (long long)w0 * 32;
  for (unsigned k0 = 0; k0 < total; k0 += 32) {
    const unsigned k = k0 + lane;
    const long long q = base + (k < total ? s_pt[warp][k] : 0);
    const bool lost = k < total && classify_F(a, q) != 3;
    const unsigned lm = __ballot_sync(0xffffffffu, lost);
    if (!lm) continue;
    unsigned at = 0;
    if (lane == 0) at = atomicAdd(y_count, (unsigned)__popc(lm));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (lost) {
      Y[at + __popc(lm & ((1u << lane) - 1u))] = (unsigned)q;
      atomicOr(&s_lost[warp][(unsigned)(q - base) >> 5], 1u << (q & 31));
    }
  }
  __syncwarp();
  if (w0 + lane < nwords) R[w0 + lane] = s_lost[warp][lane];   // every word, with or without lost saddles
}

// raw values of a list's points
__global__ void gather_kernel(const unsigned *__restrict__ list, unsigned count, const float *__restrict__ src,
                              float *__restrict__ dst) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) dst[i] = src[list[i]];
}

// Outcome of one item of a pass.
enum { kItemDone = 0, kItemDeferred = 1, kItemNeedsEnforce = 2 };

__device__ __forceinline__ float stencil_nd(const PostArgs &a, const Face &f, float cur, int t, int s, float o,
                                            int nd) {
  return nd == 2 ? stencil2(a, f, cur, t, s, o) : stencil3(a, f, t, s, o);
}

// The stencil pass fused with enforcement (a.NI set), item idx at point e.
// The candidates split into the connected components of face adjacency, and
// each pass reads, besides unchanged points, only the candidates of the
// item's own component.  So a candidate with no candidate neighbour (three in
// four on smooth fields) runs its enforcement right after its stencil, on the
// same neighbour values, and stores only the final value (nothing reads its
// result words).  The items of larger components run the stencil as usual
// (result words, deferral) and report kItemNeedsEnforce; the enforcement pass
// runs over them alone.
template <int PASS, int ND>
__device__ __forceinline__ int face_item_run(const PostArgs &a, unsigned idx, FaceItem &it) {
  const long long e = it.e;
  float r;
  int st = kItemDone;
  if (PASS == kPassStencil) {
    r = stencil_nd(a, it.f, it.cur, it.t, it.s, it.o, ND);
    if (a.NI) {
      if (it.iso) {
        a.F[e] = enforce<ND>(a, it.f, r, it.t, it.o);
        return kItemDone;
      }
      if (a.RAW) a.RAW[idx] = it.o;   // F[e] holds the stencil result from here on
      st = kItemNeedsEnforce;
    }
  } else {
    r = enforce<ND>(a, it.f, it.cur, it.t, it.o);
  }
  // in place: every reader of e's pre-pass value has finished (they are the
  // earlier candidates e waited for); later readers take e's result from S
  // at e's list position (dense, one coalesced word per item)
  a.F[e] = r;
  st_rlx(&a.S[idx], ((unsigned long long)a.gen << 32) | __float_as_uint(r));
  return st;
}

// Items of the RBF or axis-pattern pass (list index idx), one per lane of a
// warp that calls it whole: an item's result goes to F and to S at its point.
// While an earlier candidate that an item reads is not final the item looks
// again, up to polls times, and is deferred after that (returns true).  The
// lanes look together and the ready ones compute in between: an item often
// waits for one in a neighbouring lane, which must not wait for it in turn at
// the end of a loop of its own (1.2 K lost saddles of a 100 x 500 x 500 field
// in chains: 315 us when it did, 109 without).
template <int PASS, int ND>
__device__ __forceinline__ bool pass_items(const PostArgs &a, const unsigned *__restrict__ list, unsigned idx,
                                           bool valid, int polls) {
  const long long e = valid ? (long long)list[idx] : 0;
  C3 c = {0, 0, 0};
  Deps<ND> d;
  d.pend = 0;
  if (valid) {
    c = coords(a.g, e);
    deps_find<PASS, ND>(a, e, c, d);
  }
  float o = 0.f;
  RbfItem<ND> it;
  if (valid) {
    o = a.OL ? a.OL[idx] : (a.ORIG ? a.ORIG[e] : a.F[e]);
    if (PASS == kPassRbf) rbf_load<ND>(a, e, c, d.cand, o, it);
  }
  bool pending = valid;
  for (int p = 0;; p++) {
    const bool ready = pending && deps_ready<ND>(a, d);
    if (ready) {
      bool ok = false;
      float r;
      if constexpr (PASS != kPassRbf) r = axis3(a, e, c, o, ok);
      else if constexpr (ND == 2) r = rbf2(a, d, it, ok);
      else r = rbf3(a, d, it, ok);
      if (ok) atomicAdd(a.restored, 1u);
      // in place: every reader of e's pre-pass value has finished (they are the
      // earlier candidates e waited for); later readers take e's result from S
      a.F[e] = r;
      st_rlx(&a.S[e], ((unsigned long long)a.gen << 32) | __float_as_uint(r));
      pending = false;
    }
    if (p >= polls || !__any_sync(0xffffffffu, pending)) break;
    if (!__any_sync(0xffffffffu, ready)) __nanosleep(p < 64 ? 32 : 256);
  }
  return pending;
}

// One item per lane of a warp that calls it whole; true while the item is
// still pending.  Its state is loaded once; then the warp looks at the missing
// results of all its items and runs the ready ones, again while that unblocks
// others (an item often waits for one in a neighbouring lane), and otherwise
// up to polls times.  In the fused stencil pass, the items left for the
// enforcement pass are marked in the a.NI bitmap here (one atomic per warp
// when the warp's items share a bitmap word, as in a round over the whole
// list).
constexpr int kShortPolls = 6;   // rounds whose items are not all in flight

template <int PASS, int ND>
__device__ __forceinline__ bool pass_item_local(const PostArgs &a, const unsigned *__restrict__ list, unsigned idx,
                                                bool valid, int polls) {
  if (PASS != kPassStencil && PASS != kPassEnforce) return pass_items<PASS, ND>(a, list, idx, valid, polls);
  bool pending = valid, need = false;
  FaceItem item;
  if (valid) face_item_load<PASS, ND>(a, list, idx, item);
  for (int p = 0;; p++) {
    const bool ready = pending && face_item_ready(a, item);
    if (ready) {
      need = face_item_run<PASS, ND>(a, idx, item) == kItemNeedsEnforce;
      pending = false;
    }
    if (!__any_sync(0xffffffffu, pending)) break;
    if (!__any_sync(0xffffffffu, ready)) {
      if (p >= polls) break;
      if (p >= kShortPolls) __nanosleep(p < 64 ? 32 : 256);
    }
  }
  if (PASS == kPassStencil && a.NI) {
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (m) {
      const int lane = threadIdx.x & 31;
      const int first = __ffs(m) - 1;
      const unsigned wi = idx >> 5;
      const unsigned w_first = __shfl_sync(0xffffffffu, wi, first);
      const unsigned bit = need ? 1u << (idx & 31) : 0u;
      if (__all_sync(0xffffffffu, !need || wi == w_first)) {
        const unsigned bits = __reduce_or_sync(0xffffffffu, bit);
        if (lane == first) atomicOr(&a.NI[w_first], bits);
      } else if (need) {
        atomicOr(&a.NI[wi], bit);
      }
    }
  }
  return pending;
}

// One round of a pass over a worklist of list indices (identity when W is
// null).  Items whose earlier candidates are not final yet go to Wn.
// eight CTAs per SM (32 registers): the round is latency-bound, more warps
// hide more of it
template <int PASS, int ND>
__global__ void __launch_bounds__(kPostThreads, 8)
pass_round_kernel(PostArgs a, const unsigned *__restrict__ list, const unsigned *__restrict__ W,
                  unsigned nw, unsigned *__restrict__ Wn, unsigned *wn_count) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned idx = 0;
  if (i < nw) idx = W ? W[i] : i;
  const bool defer = pass_item_local<PASS, ND>(a, list, idx, i < nw, kShortPolls);
  const unsigned m = __ballot_sync(0xffffffffu, defer);
  const int lane = threadIdx.x & 31;
  unsigned base = 0;
  if (lane == 0 && m) base = atomicAdd(wn_count, (unsigned)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (defer) Wn[base + __popc(m & ((1u << lane) - 1u))] = idx;
}


// Round 0 of the enforcement pass that follows the fused stencil pass: the
// items are the set bits of the bitmap NI over list positions.  Each CTA
// takes kSparseWords bitmap words (a window of the list in raster order),
// gathers their set positions in shared memory in order and runs them as a
// round does, so that neighbouring items still meet in one CTA and resolve
// by its local retries.  Deferred items go to Wn.
constexpr int kSparseWords = 24;
static_assert(kSparseWords * 32 % kPostThreads == 0 && kSparseWords <= 32, "window of whole thread strides");

template <int ND>
__global__ void __launch_bounds__(kPostThreads, 8)
enforce_sparse_kernel(PostArgs a, const unsigned *__restrict__ list, const unsigned *__restrict__ NI,
                      unsigned nwords, unsigned *__restrict__ Wn, unsigned *wn_count) {
  __shared__ unsigned s_idx[kSparseWords * 32];
  __shared__ unsigned s_word[kSparseWords], s_off[kSparseWords];
  __shared__ unsigned s_total;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned w0 = blockIdx.x * kSparseWords;
  if (warp == 0) {
    const unsigned wi = w0 + lane;
    const unsigned bits = (lane < kSparseWords && wi < nwords) ? NI[wi] : 0u;
    const unsigned c = __popc(bits);
    unsigned incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane < kSparseWords) {
      s_word[lane] = bits;
      s_off[lane] = incl - c;
    }
    if (lane == 31) s_total = incl;
  }
  __syncthreads();
  // every thread expands bit positions threadIdx.x + 256 j of the window, in
  // order: position p goes to the slot of its word plus the set bits before it
#pragma unroll
  for (int j = 0; j < kSparseWords * 32 / kPostThreads; j++) {
    const unsigned pbit = (unsigned)threadIdx.x + (unsigned)(j * kPostThreads);
    const unsigned wd = s_word[pbit >> 5], b = pbit & 31u;
    if ((wd >> b) & 1u) s_idx[s_off[pbit >> 5] + (unsigned)__popc(wd & ((1u << b) - 1u))] = w0 * 32u + pbit;
  }
  __syncthreads();
  const unsigned total = s_total;
  for (unsigned base = 0; base < total; base += kPostThreads) {
    const unsigned i = base + threadIdx.x;
    const bool valid = i < total;
    const unsigned idx = valid ? s_idx[i] : 0u;
    const bool defer = pass_item_local<kPassEnforce, ND>(a, list, idx, valid, kShortPolls);
    const unsigned m = __ballot_sync(0xffffffffu, defer);
    unsigned wb = 0;
    if (lane == 0 && m) wb = atomicAdd(wn_count, (unsigned)__popc(m));
    wb = __shfl_sync(0xffffffffu, wb, 0);
    if (defer) Wn[wb + __popc(m & ((1u << lane) - 1u))] = idx;
  }
}

// A round over a worklist whose length is on the device (*nw_dev), in a
// grid-stride loop over a grid of any size (no barrier inside).
template <int PASS, int ND>
__global__ void __launch_bounds__(kPostThreads, 2)
pass_round_dev_kernel(PostArgs a, const unsigned *__restrict__ list, const unsigned *__restrict__ W,
                      const unsigned *nw_dev, unsigned *__restrict__ Wn, unsigned *wn_count) {
  const unsigned nw = *nw_dev;
  const int lane = threadIdx.x & 31;
  const unsigned stride = gridDim.x * blockDim.x;
  // every item of the round in flight at once: an item may wait for the
  // earlier ones it reads, which are being computed beside it.  Otherwise one
  // look: the RBF stage of 1800x3600 is 75 us
  // so, 95 when a warp looks six times and goes on while a lane is ready.
  const int polls = nw <= stride ? kDepPolls : 0;
  for (unsigned base = blockIdx.x * blockDim.x; base < nw; base += stride) {
    const unsigned i = base + threadIdx.x;
    unsigned idx = 0;
    if (i < nw) idx = W ? W[i] : i;
    const bool defer = pass_item_local<PASS, ND>(a, list, idx, i < nw, polls);
    const unsigned m = __ballot_sync(0xffffffffu, defer);
    unsigned wb = 0;
    if (lane == 0 && m) wb = atomicAdd(wn_count, (unsigned)__popc(m));
    wb = __shfl_sync(0xffffffffu, wb, 0);
    if (defer) Wn[wb + __popc(m & ((1u << lane) - 1u))] = idx;
  }
}

// Grid-wide barrier of a cooperative launch (every CTA resident): one
// arrival counter and a generation word.  The last CTA to arrive resets the
// counter and advances the generation; the others wait for the generation to
// change.  The wait is bounded: after kBarSpinLimit polls the CTA records
// kErrWaitTimeout and leaves the barrier (the pass then reports an error).
constexpr int kBarSpinLimit = 1 << 22;

__device__ __forceinline__ unsigned ld_acq_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_rel_u32(unsigned *p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ bool grid_barrier(unsigned *bar, int *err, int spin_limit = 0) {
  const int limit = spin_limit > 0 ? spin_limit : kBarSpinLimit;
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    __threadfence();
    const unsigned g = ld_acq_u32(bar + 1);
    if (atomicAdd(bar, 1u) == gridDim.x - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      st_rel_u32(bar + 1, g + 1);
    } else {
      // exponential back-off keeps the pollers of all CTAs from crowding the
      // generation word's L2 line while the last arrivals are still counting
      int spins = 0;
      unsigned nap = 64;
      while (ld_acq_u32(bar + 1) == g) {
        if (++spins > limit) {
          ok = 0;
          atomicExch(err, kErrWaitTimeout);
          break;
        }
        __nanosleep(nap);
        if (nap < 1024) nap <<= 1;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// The rounds of a pass after round 1 (or all of them) in one cooperative
// launch: rounds are separated by grid barriers instead of host round trips.
// The worklist starts as W_start with *nstart_dev items (the deferred items of
// a round-0 launch) or, when W_start is null, as the list positions themselves,
// *total_dev of them when that is not null, else total.
// Worklists and counters written during the launch are read through L2
// (__ldcg), since other SMs wrote them.  Every CTA takes the same branch at
// every barrier: the counts it reads are final after the barrier.
// status: 0 done, 1 round limit, 2 no progress.
constexpr int kCoopRoundLimit = 100000;

// At least two CTAs per SM (128 registers): the long RBF items need the
// resident threads more than registers.
template <int PASS, int ND>
__global__ void __launch_bounds__(kPostThreads, 2)
pass_coop_kernel(PostArgs a, const unsigned *__restrict__ list, unsigned total,
                 const unsigned *total_dev, const unsigned *W_start, const unsigned *nstart_dev, unsigned *Wx,
                 unsigned *Wy, unsigned *cnts, unsigned *bar, unsigned long long *status) {
  const unsigned *W = W_start;   // null: list positions themselves
  unsigned nw = W_start ? __ldcg(nstart_dev) : (total_dev ? __ldcg(total_dev) : total);
  const bool after_round0 = W_start != nullptr;
  int b = 0;
  const unsigned stride = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (int round = 0; nw > 0; round++) {
    if (round >= kCoopRoundLimit) {
      if (blockIdx.x == 0 && threadIdx.x == 0) status[0] = 1;
      return;
    }
    unsigned *Wn = b ? Wy : Wx;
    // three counters in rotation: round r counts into cnts[r % 3].  The one
    // the next round uses was last read before the barrier that ended round
    // r - 1, which every CTA has passed once any CTA is in round r, so
    // clearing it now cannot hide a count from a slower CTA.
    unsigned *cnt = cnts + (round % 3);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicExch(cnts + ((round + 1) % 3), 0u);
    // in a worklist of many times the grid most items wait for ones that this
    // round does not reach: one look each (checkerboards, whose points wait for
    // one another in long chains: 1500x1700 574 ms with kShortPolls, 447 so;
    // 160x170x180 225, 163; 700x800, below the line, 42.9 with kShortPolls, 46.7
    // with one look)
    const int polls = nw <= stride ? kDepPolls : ((nw >> 3) <= stride ? kShortPolls : 0);
    for (unsigned base = blockIdx.x * blockDim.x; base < nw; base += stride) {
      const unsigned i = base + threadIdx.x;
      unsigned idx = 0;
      if (i < nw) idx = W ? __ldcg(W + i) : i;
      const bool defer = pass_item_local<PASS, ND>(a, list, idx, i < nw && (!a.ONLY || bit_at(a.ONLY, idx)), polls);
      const unsigned m = __ballot_sync(0xffffffffu, defer);
      unsigned wb = 0;
      if (lane == 0 && m) wb = atomicAdd(cnt, (unsigned)__popc(m));
      wb = __shfl_sync(0xffffffffu, wb, 0);
      if (defer) Wn[wb + __popc(m & ((1u << lane) - 1u))] = idx;
    }
    if (!grid_barrier(bar, a.err, a.spin_limit)) return;
    const unsigned next = __ldcg(cnt);
    if ((round > 0 || after_round0) && next >= nw) {
      if (blockIdx.x == 0 && threadIdx.x == 0) status[0] = 2;
      return;
    }
    W = Wn;
    nw = next;
    b ^= 1;
  }
}

// bit planes of the types, from an int or a byte per point (a warp per word)
template <class V>
__global__ void type_planes_kernel(const V *__restrict__ fn, long long n, unsigned *__restrict__ TL,
                                   unsigned *__restrict__ TH) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned t = i < n ? (unsigned)fn[i] : 0u;
  const unsigned lo = __ballot_sync(0xffffffffu, t & 1u), hi = __ballot_sync(0xffffffffu, t & 2u);
  if ((threadIdx.x & 31) == 0 && i < n) {
    TL[i >> 5] = lo;
    TH[i >> 5] = hi;
  }
}

static bool g_weights_ready[64];
static std::mutex g_weights_mu;

// once per device; contexts on several host threads may get here together
static cudaError_t upload_weights(int dev) {
  std::lock_guard<std::mutex> lk(g_weights_mu);
  if (dev >= 0 && dev < 64 && g_weights_ready[dev]) return cudaSuccess;
  // Gaussian weights in double with the reference formula
  // (example/test_cuda_topology.cu:259-265, example/test_cuda_topology_3d.cu:360-367)
  double s2 = 0.8 * 0.8;
  double w2[9], w3[27];
  for (int a = -1; a <= 1; a++)
    for (int b = -1; b <= 1; b++) w2[(a + 1) * 3 + (b + 1)] = exp(-((double)a * a + b * b) / (2.0 * s2));
  for (int a = -1; a <= 1; a++)
    for (int b = -1; b <= 1; b++)
      for (int c = -1; c <= 1; c++)
        w3[(a + 1) * 9 + (b + 1) * 3 + (c + 1)] = exp(-(double)(a * a + b * b + c * c) / (2.0 * s2));
  cudaError_t e = cudaMemcpyToSymbol(c_w2, w2, sizeof(w2));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_w3, w3, sizeof(w3));
  if (e == cudaSuccess && dev >= 0 && dev < 64) g_weights_ready[dev] = true;
  return e;
}

size_t post_scratch_bytes(unsigned long long n) {
  const unsigned long long ntiles = (n + kPostTile - 1) / kPostTile;
  const unsigned long long words = (n + 31) / 32;
  // type planes, descriptors, RBF + extrema + saddle bitmaps + extremum word
  // positions, lists X and Z, worklists (2), Y, raw values of X and Z
  return a256((ntiles + 1) * sizeof(TileDesc)) + 6 * a256(words * 4 + 4) + 7 * a256(n * 4) + 8192;
}


// generation counter of the result words (never reused while the buffer lives)
static unsigned next_gen(szp_b200_ctx *ctx) { return ++ctx->post_gen; }

// persistent result-word buffer of the workspace, zeroed when (re)allocated
unsigned long long *post_words(szp_b200_ctx *ctx, unsigned long long n) {
  if (ctx->post_S && ctx->post_S_cap >= n) return ctx->post_S;
  if (ctx->post_S) cudaFree(ctx->post_S);
  ctx->post_S = nullptr;
  ctx->post_S_cap = 0;
  if (cudaMalloc(&ctx->post_S, n * 8) != cudaSuccess) {
    cudaGetLastError();
    ctx->post_S = nullptr;
    set_error("device allocation of %llu result words failed", n);
    return nullptr;
  }
  if (cudaMemsetAsync(ctx->post_S, 0, n * 8, ctx->stream) != cudaSuccess) return nullptr;
  ctx->post_S_cap = n;
  ctx->post_gen = 0;
  return ctx->post_S;
}

// Grid of the cooperative tail of pass PASS on this workspace's device (all
// CTAs resident), or 0 when the workspace runs its tails as ordinary
// launches: no cooperative launch on the device, or a workspace whose stream
// shares the GPU with others (server workers), where a cooperative launch
// can only start once all of its CTAs fit beside the other streams' kernels.
template <int PASS, int ND>
static int coop_grid(szp_b200_ctx *ctx) {
  static int grid_for_dev[64];
  const int dev = ctx->device;
  if (ctx->coop_off || dev < 0 || dev >= 64) return 0;
  if (grid_for_dev[dev] == 0) {
    int coop = 0, nb = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, pass_coop_kernel<PASS, ND>, kPostThreads, 0) !=
            cudaSuccess ||
        nb <= 0) {
      cudaGetLastError();
      grid_for_dev[dev] = -1;
    } else {
      grid_for_dev[dev] = nb * ctx->sm_count;
    }
  }
  return grid_for_dev[dev] > 0 ? grid_for_dev[dev] : 0;
}

// CTAs of a round over a list of device-known length that are resident at once
template <int PASS, int ND>
static int dev_grid(szp_b200_ctx *ctx) {
  static int per_sm_for_dev[64];
  const int dev = ctx->device;
  if (dev < 0 || dev >= 64) return ctx->sm_count;
  if (per_sm_for_dev[dev] == 0) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, pass_round_dev_kernel<PASS, ND>, kPostThreads, 0) !=
        cudaSuccess)
      cudaGetLastError();
    per_sm_for_dev[dev] = nb > 0 ? nb : 1;
  }
  return per_sm_for_dev[dev] * ctx->sm_count;
}

// Rounds over deferred items as ordinary launches, kBurstRounds of them
// between host checks of the remaining count: W holds the items on entry
// (their count in the pass's n0), W and Wo alternate.  Every round completes at
// least the earliest pending item, so a burst that completes none reports an
// error.
constexpr int kBurstRounds = 4;
constexpr int kRoundLimit = 100000;

// The words of a pass: the length of its first worklist, three round counters,
// the barrier's counter and generation, the length of the second worklist.
// Each pass has its own, so that one memset clears them for all.
struct PassWords { unsigned n0, cnts[3], bar[2], n1, unused[9]; };
constexpr int kPassWord = 24;   // of the workspace's 64 words
static_assert(sizeof(PassWords) == 64 && kPassWord + 4 * 8 <= 64, "four passes' words");

template <int PASS>
static PassWords *pass_words(szp_b200_ctx *ctx) {
  static_assert(PASS >= 0 && PASS < 4, "pass numbers");
  return reinterpret_cast<PassWords *>(ctx->d_words + kPassWord) + PASS;
}

template <int PASS, int ND>
static int finish_rounds(szp_b200_ctx *ctx, PostArgs &a, const unsigned *list, unsigned *W, unsigned *Wo) {
  cudaStream_t s = ctx->stream;
  PassWords *pw = pass_words<PASS>(ctx);
  unsigned *c[3] = {&pw->n0, &pw->cnts[0], &pw->cnts[1]};
  unsigned *h_left = reinterpret_cast<unsigned *>(ctx->h_words + 15);
  int ci = 0;
  unsigned prev = 0xffffffffu;
  for (int r = 0; r < kRoundLimit; r += kBurstRounds) {
    for (int k = 0; k < kBurstRounds; k++) {
      unsigned *cn = c[(ci + 1) % 3];
      if (cuda_fail(cudaMemsetAsync(cn, 0, 4, s), "memset")) return -1;
      pass_round_dev_kernel<PASS, ND><<<ctx->sm_count * 4, kPostThreads, 0, s>>>(a, list, W, c[ci], Wo, cn);
      std::swap(W, Wo);
      ci = (ci + 1) % 3;
    }
    ctx->launches += kBurstRounds;
    if (cuda_fail(cudaGetLastError(), "pass round") ||
        cuda_fail(cudaMemcpyAsync(h_left, c[ci], 4, cudaMemcpyDeviceToHost, s), "D2H") ||
        cuda_fail(cudaStreamSynchronize(s), "pass round"))
      return -1;
    const unsigned left = *h_left;
    if (left == 0) return 0;
    if (left >= prev) { set_error("post-processing pass made no progress"); return -1; }
    prev = left;
  }
  set_error("post-processing pass did not converge");
  return -1;
}

// Runs one pass: round 0 as one launch over all of its items -- list
// positions 0 .. count-1, or 0 .. *count_dev-1 (count known only on the
// device), or the set bits of the bitmap ni_bits of ni_words words (the
// enforcement after the fused stencil) -- then the rounds over the deferred
// items: in one cooperative launch that reads its counts on the device (after
// one more ordinary round when round 0 ran over a list), or as bursts of
// ordinary launches (finish_rounds).  most: a bound of the items known on the
// host; when all of them fit the cooperative grid at once, one launch runs the
// whole pass (60x90, the stencil 22 -> 13 us, enforcement 19 -> 10, RBF 18 ->
// 14: such a field spends its time on launches).
template <int PASS, int ND>
static int run_pass(szp_b200_ctx *ctx, PostArgs &a, const unsigned *list, unsigned count,
                    unsigned most, const unsigned *count_dev, unsigned *W0, unsigned *W1,
                    const unsigned *ni_bits = nullptr, unsigned ni_words = 0) {
  if (ni_bits ? ni_words == 0 : (!count_dev && count == 0)) return 0;
  const int grid = coop_grid<PASS, ND>(ctx);
  cudaStream_t s = ctx->stream;
  PassWords *pw = pass_words<PASS>(ctx);
  unsigned *n0 = &pw->n0, *cnts = pw->cnts, *bar = pw->bar, *n1 = &pw->n1;
  unsigned long long *status = ctx->d_words + 9;
  const unsigned zero = 0;
  const unsigned *no_total = nullptr;
  if (grid && most <= (unsigned)grid * kPostThreads) {
    // every item in flight at once: one launch, no worklist to start from
    const unsigned *none = nullptr;
    a.ONLY = ni_bits;
    const unsigned **total = count_dev ? &count_dev : &no_total;
    void *args[] = {(void *)&a,    (void *)&list, (void *)&most, (void *)total,   (void *)&none,  (void *)&none,
                    (void *)&W0,   (void *)&W1,   (void *)&cnts, (void *)&bar,    (void *)&status};
    const unsigned need = (most + kPostThreads - 1) / kPostThreads;
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)pass_coop_kernel<PASS, ND>,
                                                      dim3(need ? need : 1), dim3(kPostThreads), args, 0, s);
    a.ONLY = nullptr;
    ctx->launches += 1;
    return cuda_fail(e, "cooperative pass launch") ? -1 : 0;
  }
  if (ni_bits)
    enforce_sparse_kernel<ND><<<(ni_words + kSparseWords - 1) / kSparseWords, kPostThreads, 0, s>>>(
        a, list, ni_bits, ni_words, W0, n0);
  else if constexpr (PASS == kPassRbf)
    // its items are counted on the device
    pass_round_dev_kernel<PASS, ND><<<dev_grid<PASS, ND>(ctx), kPostThreads, 0, s>>>(a, list, nullptr, count_dev, W0, n0);
  else
    pass_round_kernel<PASS, ND><<<(count + kPostThreads - 1) / kPostThreads, kPostThreads, 0, s>>>(
        a, list, nullptr, count, W0, n0);
  ctx->launches += 1;
  if (cuda_fail(cudaGetLastError(), "pass round")) return -1;
  if (!grid) return finish_rounds<PASS, ND>(ctx, a, list, W0, W1);
  const unsigned *W_start = W0, *nstart = n0;
  unsigned *Wx = W1, *Wy = W0;
  if (!count_dev) {
    // one more ordinary round (the round-0 remainder can still be large)
    pass_round_dev_kernel<PASS, ND><<<ctx->sm_count * 8, kPostThreads, 0, s>>>(a, list, W0, n0, W1, n1);
    ctx->launches += 1;
    if (cuda_fail(cudaGetLastError(), "pass round")) return -1;
    W_start = W1;
    nstart = n1;
    Wx = W0;
    Wy = W1;
  }
  void *args[] = {(void *)&a,       (void *)&list,   (void *)&zero, (void *)&no_total,
                  (void *)&W_start, (void *)&nstart, (void *)&Wx,  (void *)&Wy,   (void *)&cnts,
                  (void *)&bar,     (void *)&status};
  if (cuda_fail(cudaLaunchCooperativeKernel((const void *)pass_coop_kernel<PASS, ND>, dim3(grid), dim3(kPostThreads),
                                            args, 0, s),
                "cooperative pass launch"))
    return -1;
  ctx->launches += 1;
  return 0;
}

template <int ND>
static int run_all_passes(szp_b200_ctx *ctx, PostArgs &a, unsigned *X, unsigned nx, unsigned *Z, unsigned nz,
                          unsigned *Y, unsigned *W0, unsigned *W1, unsigned *R,
                          const unsigned *Eb, const unsigned *Sb, float *OX, const float *OZ,
                          int axis_stencil, bool raw_in_F) {
  cudaStream_t s = ctx->stream;
  const long long n = a.n;
  // raw_in_F: OX keeps the raw values of the items the fused stencil leaves
  // for enforcement
  a.OL = nullptr;
  a.RAW = nullptr;
  a.X = Eb;
  if (a.sp && a.n_sp > 0) {
    // stencil fused with enforcement; the items next to another candidate
    // are marked in a bitmap over list positions (in R, unused until the
    // lost-saddle detection) and only they run the enforcement pass
    const unsigned ni_words = (nx + 31) / 32;
    unsigned *NIb = R;
    if (cuda_fail(cudaMemsetAsync(NIb, 0, (size_t)ni_words * 4, s), "memset")) return -1;
    a.gen = next_gen(ctx);
    a.NI = NIb;
    a.RAW = raw_in_F ? OX : nullptr;
    if (run_pass<kPassStencil, ND>(ctx, a, X, nx, nx, nullptr, W0, W1)) return -1;
    a.NI = nullptr;
    a.RAW = nullptr;
    a.OL = raw_in_F ? OX : nullptr;   // raw values of the remaining items, stashed by the stencil
    tl_mark(ctx, "post_stencil");
    a.gen = next_gen(ctx);
    if (run_pass<kPassEnforce, ND>(ctx, a, X, 0, nx, nullptr, W0, W1, NIb, ni_words)) return -1;
  } else {
    a.gen = next_gen(ctx);
    if (run_pass<kPassEnforce, ND>(ctx, a, X, nx, nx, nullptr, W0, W1)) return -1;
  }
  tl_mark(ctx, "post_enforce");
  // the lost saddles (from F after enforcement); RBF reads the locks from the
  // extremum bitmap (box_locks)
  const long long words = (n + 31) / 32;
  unsigned *ycnt = reinterpret_cast<unsigned *>(ctx->d_words + 8);
  a.R = R;
  if (nz) fn_detect_kernel<<<(unsigned)((words + 255) / 256), 256, 0, s>>>(a, Sb, (unsigned)words, R, Y, ycnt);
  ctx->launches += nz ? 1 : 0;
  if (cuda_fail(cudaGetLastError(), "fn detect")) return -1;
  tl_mark(ctx, "post_fn_locks");
  // RBF runs over the lost saddles Y; their number stays on the device.
  // Saddles keep their raw values until RBF itself writes them.
  a.OL = nullptr;
  a.gen = next_gen(ctx);
  if (nz && run_pass<kPassRbf, ND>(ctx, a, Y, 0, nz, ycnt, W0, W1)) return -1;
  tl_mark(ctx, "post_rbf");
  if constexpr (ND == 3) {
    if (axis_stencil && nz) {
      a.OL = raw_in_F ? OZ : nullptr;   // gathered before the passes: RBF has changed some saddles
      a.gen = next_gen(ctx);
      if (run_pass<kPassAxis, ND>(ctx, a, Z, nz, nz, nullptr, W0, W1)) return -1;
      tl_mark(ctx, "post_axis");
    }
  }
  return 0;
}

// whether there are interior points to work on
bool post_has_work(const Geom &g) { return g.d2 >= 3 && g.d3 >= 3 && (g.nd != 3 || g.d1 >= 3); }

// Launches the list kernel: totals to word 2 (extrema << 32 | saddles), its
// status to word 5.  Words 2, 3 and 5 are zero on entry.
int post_lists_begin(szp_b200_ctx *ctx, const unsigned *d_TL, const unsigned *d_TH, TileDesc *desc, const Geom &g,
                     int axis_stencil, PostLists *l) {
  const long long n = g.d1 * g.d2 * g.d3;
  Arena &A = ctx->scratch;
  l->X = A.take<unsigned>(n); l->Z = A.take<unsigned>(n); l->Y = A.take<unsigned>(n);
  l->W0 = A.take<unsigned>(n); l->W1 = A.take<unsigned>(n);
  l->R = A.take<unsigned>((n + 31) / 32);
  l->Eb = A.take<unsigned>((n + 31) / 32 + 1);
  l->Sb = A.take<unsigned>((n + 31) / 32 + 1);
  l->XP = A.take<unsigned>((n + 31) / 32 + 1);
  l->OX = A.take<float>(n); l->OZ = A.take<float>(n);
  if (!l->X || !l->Z || !l->Y || !l->W0 || !l->W1 || !l->R || !l->Eb || !l->Sb || !l->XP || !l->OX || !l->OZ) {
    set_error("scratch arena too small for post-processing");
    return -1;
  }
  unsigned long long *w = ctx->d_words;
  const long long ltiles = (n + kListTile - 1) / kListTile;
  if (cuda_fail(cudaMemsetAsync(desc, 0, (ltiles + 1) * sizeof(TileDesc), ctx->stream), "memset")) return -1;
  const unsigned grid = (unsigned)std::min<long long>(ltiles, (long long)ctx->sm_count * 6);
  list_build_kernel<<<grid, kPostThreads, 0, ctx->stream>>>(
      d_TL, d_TH, g, n, desc, reinterpret_cast<unsigned *>(w + 3), reinterpret_cast<int *>(w + 5), l->X,
      axis_stencil && g.nd == 3 ? l->Z : nullptr, l->Eb, l->Sb, w + 2, l->XP);
  ctx->launches += 1;
  return cuda_fail(cudaGetLastError(), "lists") ? -1 : 0;
}

// Clears the words of the passes: [4] status, [5] restored, [7] status of the
// sort positions' decoder (kSortStatusWord), [8] lost saddles, [9] pass status,
// and the words of each pass.
int post_words_clear(szp_b200_ctx *ctx) {
  return cuda_fail(cudaMemsetAsync(ctx->d_words, 0, (kPassWord + 4 * 8) * 8, ctx->stream), "memset") ? -1 : 0;
}

// The passes over the lists of post_lists_begin, whose totals the caller has
// read; between the two, post_words_clear and then what decodes d_sp.
int postprocess_with(szp_b200_ctx *ctx, float *d_data, const float *d_orig, const unsigned *d_TL,
                     const unsigned *d_TH, unsigned long long *d_S, const PostLists &l, unsigned long long tot,
                     const int *d_sp, unsigned long long n_sp, const Geom &g, float eb, int axis_stencil,
                     int *restored_out) {
  const long long n = g.d1 * g.d2 * g.d3;
  int dev = 0;
  cudaGetDevice(&dev);
  if (cuda_fail(upload_weights(dev), "weights")) return -1;
  cudaStream_t s = ctx->stream;
  unsigned long long *w = ctx->d_words;
  // post-processing of the decoded field itself: each item reads its raw
  // value from F before it writes (no gathered raw lists), except the
  // axis-pattern pass, which runs after RBF has changed saddles
  const bool raw_in_F = d_orig == d_data;
  const bool axis_raw = axis_stencil && g.nd == 3;
  const unsigned nx = (unsigned)(tot >> 32), nz = (unsigned)(tot & 0xffffffffull);
  unsigned *Z = l.Z;
  float *OZ = l.OZ;
  if (axis_raw && raw_in_F && nz) {
    gather_kernel<<<(nz + 255) / 256, 256, 0, s>>>(Z, nz, d_data, OZ);
    ctx->launches += 1;
  }
  PostArgs a{};
  a.F = d_data;
  a.TL = d_TL;
  a.TH = d_TH;
  a.ORIG = raw_in_F ? nullptr : d_orig;
  a.sp = d_sp;
  a.n_sp = d_sp ? n_sp : 0;
  a.g = g;
  a.n = n;
  a.eb = eb;
  a.eps = fmaxf(1e-6f, 0.1f * eb);
  a.S = d_S;
  a.XP = l.XP;
  a.err = reinterpret_cast<int *>(w + 4);
  a.restored = reinterpret_cast<unsigned *>(w + 5);
  const int rc = (g.nd == 2)
                     ? run_all_passes<2>(ctx, a, l.X, nx, Z, nz, l.Y, l.W0, l.W1, l.R, l.Eb, l.Sb, l.OX, OZ,
                                         axis_stencil, raw_in_F)
                     : run_all_passes<3>(ctx, a, l.X, nx, Z, nz, l.Y, l.W0, l.W1, l.R, l.Eb, l.Sb, l.OX, OZ,
                                         axis_stencil, raw_in_F);
  if (rc) return -1;
  if (cuda_fail(cudaMemcpyAsync(ctx->h_words, w, 96, cudaMemcpyDeviceToHost, s), "D2H") ||
      cuda_fail(cudaStreamSynchronize(s), "postprocess"))
    return -1;
  if (ctx->h_words[kSortStatusWord] & 0xffffffffu) {
    set_error("decoder reported malformed sort-position stream");
    return -1;
  }
  const int err = (int)(ctx->h_words[4] & 0xffffffffu);
  if (err) { set_error("post-processing status %d", err); return -1; }
  if (ctx->h_words[9] == 1) { set_error("post-processing pass did not converge"); return -1; }
  if (ctx->h_words[9] == 2) { set_error("post-processing pass made no progress"); return -1; }
  if (restored_out) *restored_out = (int)(ctx->h_words[5] & 0xffffffffu);
  return 0;
}

// Bounded-wait check of the grid barrier: the last CTA of the launch leaves
// without arriving, so the others must give up after spin_limit polls and
// report kErrWaitTimeout (no CTA waits on anything that can hang).
__global__ void barrier_timeout_probe_kernel(unsigned *bar, int *err, int spin_limit) {
  if (blockIdx.x == gridDim.x - 1) return;
  grid_barrier(bar, err, spin_limit);
}

int selftest_grid_barrier(int spin_limit, int *status, float *ms) {
  unsigned *d = nullptr;
  if (cuda_fail(cudaMalloc(&d, 64), "cudaMalloc")) return -1;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int rc = -1;
  if (!cuda_fail(cudaMemset(d, 0, 64), "memset") && !cuda_fail(cudaEventCreate(&e0), "event") &&
      !cuda_fail(cudaEventCreate(&e1), "event")) {
    cudaEventRecord(e0, 0);
    barrier_timeout_probe_kernel<<<2, 64>>>(d, reinterpret_cast<int *>(d + 4), spin_limit);
    cudaEventRecord(e1, 0);
    int h = 0;
    if (!cuda_fail(cudaGetLastError(), "probe launch") &&
        !cuda_fail(cudaMemcpy(&h, d + 4, 4, cudaMemcpyDeviceToHost), "D2H")) {
      cudaEventElapsedTime(ms, e0, e1);
      *status = h;
      rc = 0;
    }
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFree(d);
  return rc;
}

bool post_planes(szp_b200_ctx *ctx, unsigned long long n, unsigned **TL, unsigned **TH) {
  *TL = ctx->scratch.take<unsigned>((n + 31) / 32 + 1);
  *TH = ctx->scratch.take<unsigned>((n + 31) / 32 + 1);
  return *TL && *TH;
}

int post_planes_from_bytes(szp_b200_ctx *ctx, const unsigned char *d_T, unsigned long long n, unsigned *TL,
                           unsigned *TH) {
  type_planes_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(d_T, (long long)n, TL, TH);
  ctx->launches += 1;
  return cuda_fail(cudaGetLastError(), "type planes") ? -1 : 0;
}

int postprocess(szp_b200_ctx *ctx, float *d_data, const float *d_orig, const int *d_types_i, const int *d_sp,
                unsigned long long n_sp, const Geom &g, float eb, int axis_stencil,
                int *restored_out) {
  const long long n = g.d1 * g.d2 * g.d3;
  if (!post_has_work(g)) { if (restored_out) *restored_out = 0; return 0; }
  if (n >= (1ll << 32)) { set_error("post-processing supports fields of fewer than 2^32 points"); return -1; }
  Arena &A = ctx->scratch;
  cudaStream_t s = ctx->stream;
  unsigned long long *S = post_words(ctx, (unsigned long long)n);
  unsigned *TL, *TH;
  const unsigned long long ntiles = (n + kPostTile - 1) / kPostTile;
  TileDesc *desc = A.take<TileDesc>(ntiles + 1);
  if (!S || !desc || !post_planes(ctx, n, &TL, &TH)) {
    set_error("scratch arena too small for post-processing");
    return -1;
  }
  type_planes_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_types_i, n, TL, TH);
  ctx->launches += 1;
  PostLists l;
  if (cuda_fail(cudaMemsetAsync(ctx->d_words, 0, 64, s), "memset") ||
      post_lists_begin(ctx, TL, TH, desc, g, axis_stencil, &l) ||
      cuda_fail(cudaMemcpyAsync(ctx->h_words, ctx->d_words, 64, cudaMemcpyDeviceToHost, s), "D2H") ||
      cuda_fail(cudaStreamSynchronize(s), "lists"))
    return -1;
  tl_mark(ctx, "post_lists");
  const int err = (int)(ctx->h_words[5] & 0xffffffffu);
  if (err) { set_error("post-processing status %d", err); return -1; }
  if (post_words_clear(ctx)) return -1;
  return postprocess_with(ctx, d_data, d_orig, TL, TH, S, l, ctx->h_words[2], d_sp, n_sp, g, eb, axis_stencil,
                          restored_out);
}

}  // namespace tsz
