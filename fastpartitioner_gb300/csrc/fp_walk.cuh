// LDG decisions taken again inside a speculative window: the scores, the exact
// pick from a position's stored candidates, and the walk of one CTA over a
// window's positions in order.  Shared by the refinement engine (fp_spec.cu)
// and the initial streams (fp_stream.cu).
#pragma once

#include "fp_spec_common.cuh"

namespace fp {
namespace spec {

constexpr int kBig = 1000000000;

// LDG scores (TV/partition.cpp:98-145 with TV's clamps, MGV/partition.cpp:28-65
// without).  They are first formed in float, from the penalty 1 - size / C off
// by less than 4e-7 * (1 + size / C); a score of count c is bounded within
// c * 1e-6 * (1 + size / C).  A part whose lower bound clears every other's
// upper bound is the argmax; near parts with one common count need no FP64
// either: with equal counts the score falls (weakly: division, subtraction and
// product round monotonically) as the size grows, and equal scores go to the
// smaller size, so the smallest size, then the first sighting, wins.  The
// exact double scores (722 cycles each here, against 22 for a redux.sync)
// decide what is left.
//
// Penalty of a part and the bound of its error per count, from rC = 1 / C
// rounded to float.
__device__ __forceinline__ float tol_of(float pen) { return 1e-6f * (1.0f + fabsf(1.0f - pen)); }
__device__ __forceinline__ float2 pen_of(int size, float rC) {
  const float pen = 1.0f - __fmul_rn((float)size, rC);
  return make_float2(pen, tol_of(pen));
}
// A drift below a / b with room for the roundings: floor(a / b) - 2 or less,
// capped; -1 if not positive.
__device__ __forceinline__ int slack_of(float a, float b) {
  const float x = __fdividef(a, b) * (1.0f - 2e-5f) - 2.0f;
  return !(x > -1.0f) ? -1 : x > 1.0e9f ? kBig : (int)x;
}

// Floats as integers of the same order, and back.
__device__ __forceinline__ int order_of(float f) {
  const int b = __float_as_int(f);
  return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float float_of(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// What one pass over scored parts keeps: the best lower bound (its upper bound,
// part and count) and the largest upper bound of the others, the largest
// penalty and count.
constexpr float kLow = -1e30f;
struct ScoreAcc {
  float blo = kLow, bhi = kLow, oh = kLow, up = kLow;
  unsigned be = 0;   // (count << 13) | part of the best
  int cm = 0;
  __device__ __forceinline__ void add(int p, int c, float2 w) {
    const float cf = (float)c, v = cf * w.x;
    const float lo = v - cf * w.y, hi = v + cf * w.y;
    up = fmaxf(up, w.x + w.y);
    cm = max(cm, c);
    if (lo > blo) {
      oh = fmaxf(oh, bhi);
      blo = lo;
      bhi = hi;
      be = ((unsigned)c << 13) | (unsigned)p;
    } else {
      oh = fmaxf(oh, hi);
    }
  }
  // meets the accumulators of the lanes whose ids differ in the low bits of
  // `lanes` - 1 (8 or 16 lanes to a position, or the whole warp: by redux.sync,
  // 22 cycles each, where the shuffles take some 80 per step)
  __device__ __forceinline__ void meet(int lanes) {
    if (lanes == 32) {
      const int kb = order_of(blo), mb = __reduce_max_sync(kAll, kb);
      const unsigned e = __reduce_min_sync(kAll, kb == mb ? be : ~0u);
      const int wl = __ffs(__ballot_sync(kAll, kb == mb && be == e)) - 1;
      oh = (int)(threadIdx.x & 31) == wl ? oh : fmaxf(oh, bhi);
      bhi = __shfl_sync(kAll, bhi, wl);
      blo = float_of(mb);
      be = e;
      oh = float_of(__reduce_max_sync(kAll, order_of(oh)));
      up = float_of(__reduce_max_sync(kAll, order_of(up)));
      cm = __reduce_max_sync(kAll, cm);
      return;
    }
#pragma unroll
    for (int off = 1; off < lanes; off <<= 1) {
      const float xl = __shfl_xor_sync(kAll, blo, off), xh = __shfl_xor_sync(kAll, bhi, off);
      const float xo = __shfl_xor_sync(kAll, oh, off), xu = __shfl_xor_sync(kAll, up, off);
      const unsigned xe = __shfl_xor_sync(kAll, be, off);
      const int xc = __shfl_xor_sync(kAll, cm, off);
      // equal bounds: the lower packed word on both sides, so that the lanes agree
      const bool take = xl > blo || (xl == blo && xe < be);
      oh = fmaxf(fmaxf(oh, xo), take ? bhi : xh);
      if (take) {
        blo = xl;
        bhi = xh;
        be = xe;
      }
      up = fmaxf(up, xu);
      cm = max(cm, xc);
    }
  }
  __device__ __forceinline__ bool one() const { return blo > 0.0f && oh < blo; }          // the argmax is clear
  __device__ __forceinline__ bool none() const { return !(fmaxf(bhi, oh) > 0.0f); }       // no part scores
  // drift of every part's size that leaves the clear argmax, or none, as it is
  __device__ __forceinline__ int slack_one(float Cf) const {
    const int cd = (int)(be >> 13);
    const float diff = blo - oh - 1e-6f * (fabsf(blo) + fabsf(oh));
    return min(slack_of(diff * Cf, (float)(cd + cm)), slack_of(blo * (1.0f - 1e-6f) * Cf, (float)cd));
  }
  __device__ __forceinline__ int slack_none(float Cf) const { return up <= kLow ? kBig : slack_of(-up * Cf, 1.0f); }
};

// Candidate entry of a part for the exact re-check: part (12 bits), count
// without the vertex itself (16 bits), 32-bit sighting key.  A vertex whose
// count or first net index does not fit (one with 65536 nets or more) stores
// no list: ncand = -1.
__device__ __forceinline__ unsigned long long cand_entry(int p, int c, unsigned f) {
  return ((unsigned long long)p << 52) | ((unsigned long long)c << 36) | f;
}

// A sighting key (32-bit, of a vertex one warp or CTA tallied) or a 64-bit key
// of absolute net indexes as (net index << 32 | slot).
__device__ __forceinline__ unsigned long long key64(unsigned f, int sb) { return wide_key(f, sb, 0); }
__device__ __forceinline__ unsigned long long key64(unsigned long long f, int) { return f; }
__device__ __forceinline__ unsigned key32(unsigned f, int, bool*) { return f; }
__device__ __forceinline__ unsigned key32(unsigned long long f, int sb, bool* wide) {
  *wide |= (f >> 32) > 0xffffull;
  return ((unsigned)(f >> 32) << sb) | (unsigned)f;
}
__device__ __forceinline__ unsigned min_key(unsigned f) { return __reduce_min_sync(kAll, f); }
__device__ __forceinline__ unsigned long long min_key(unsigned long long f) { return warp_min_u64(f); }

// Smallest size, then the smallest key among its holders (one warp, each lane
// one (size, key, part); part < 0: none); returns the part, -1 if no lane has one.
template <class F>
__device__ __forceinline__ int least_size_first(int size, F first, int part) {
  const int ms = __reduce_min_sync(kAll, part >= 0 ? size : 0x7fffffff);
  const F mf = min_key(part >= 0 && size == ms ? first : ~(F)0);
  const unsigned m = __ballot_sync(kAll, part >= 0 && size == ms && first == mf);
  return m ? __shfl_sync(kAll, part, __ffs(m) - 1) : -1;
}

// The window's positions as the walk stages them in shared memory: the words of
// up to kWalkLoad positions, per 32 of them (a group) what a drift of the sizes
// has to exceed to matter, and the first kWalkRow candidate entries of the
// group at hand (rows padded so that four rows read side by side meet no bank
// conflict).
constexpr int kWalkLoad = 1024, kWalkRow = 256, kWalkStride = kWalkRow + 8;
struct WalkSmem {
  unsigned long long ent[32 * kWalkStride];
  int4 meta[kWalkLoad];      // (own << 16) | decision, weight, acc, (ncand << 8) | flag
  int margin[kWalkLoad];     // drift the position tolerates (-1: always taken again)
  int gmin[kWalkLoad / 32];  // per group of 32: the smallest margin
  int nd[32], nslack[32];    // decisions taken again: (nets listing it << 13) | part (-1: no list), drift tolerated
  int drift;                 // largest change of one part's size so far by changed decisions (an upper bound)
  int group;                 // group to decide again (-1: none left), its positions, and those
  unsigned need, eval;       //   of them that have nets, in list
  int list[32];
};

// Least-loaded part of sz, lowest index on ties (one warp); *ms its size.
__device__ __forceinline__ int warp_least_loaded(const int* sz, int K, int* ms_out) {
  const int lane = threadIdx.x & 31;
  int ms = 0x7fffffff, mp = 0x7fffffff;
  for (int p = lane; p < K; p += 32) {
    const int x = sz[p];
    if (x < ms || mp == 0x7fffffff) { ms = x; mp = p; }
  }
  const int m = warp_min(ms);
  *ms_out = m;
  return warp_min(mp != 0x7fffffff && ms == m ? mp : 0x7fffffff);
}

// One warp decides a position again with the sizes sz, whatever its candidates:
// nc of them, cl all of its entries.  Returns the decision before TV's clamps,
// (nets listing it << 13) | part, and in *slack the drift of any part's size
// from these that leaves it as it is.
static __device__ __noinline__ int walk_pick_any(const DevInstance& I, float rC, float Cf, const int* sz, int nc,
                                          const unsigned long long* cl, int* slack) {
  const int lane = threadIdx.x & 31;
  const int K = I.K;
  const unsigned long long e0 = lane < nc ? lds(&cl[lane]) : 0;   // the first 32 stay in registers
  ScoreAcc A;
  for (int i = lane; i < nc; i += 32) {
    const unsigned long long e = i < 32 ? e0 : lds(&cl[i]);
    const int p = (int)(e >> 52), c = (int)((e >> 36) & 0xffffull);
    if (c > 0) A.add(p, c, pen_of(sz[p], rC));
  }
  A.meet(32);
  int nd = -1, sl = -1;
  if (A.one()) {
    nd = (int)A.be;
    sl = A.slack_one(Cf);
  } else if (A.none()) {
    // no part scores: the least-loaded one, and the nets listing it all the same
    int ms, cx = 0, s2 = 0x7fffffff;
    const int dn = warp_least_loaded(sz, K, &ms);
    for (int p = lane; p < K; p += 32)
      if (p != dn) s2 = min(s2, sz[p]);
    sl = min(A.slack_none(Cf), (warp_min(s2) - ms - 1) / 2);
    for (int i = lane; i < nc; i += 32) {
      const unsigned long long e = i < 32 ? e0 : lds(&cl[i]);
      if ((int)(e >> 52) == dn) cx = (int)((e >> 36) & 0xffffull);
    }
    nd = (warp_max(cx) << 13) | dn;
  } else {
    const float fb = fmaxf(A.blo, 0.0f);
    int np = -1, nsz = 0, cmin = 0x7fffffff, cmax = 0;
    unsigned nf = ~0u;
    for (int i = lane; i < nc; i += 32) {
      const unsigned long long e = i < 32 ? e0 : lds(&cl[i]);
      const int p = (int)(e >> 52), c = (int)((e >> 36) & 0xffffull), s = sz[p];
      const float2 w = pen_of(s, rC);
      if (c == 0 || (float)c * w.x + (float)c * w.y < fb) continue;
      cmin = min(cmin, c);
      cmax = max(cmax, c);
      if (np < 0 || s < nsz || (s == nsz && (unsigned)e < nf)) { np = p; nsz = s; nf = (unsigned)e; }
    }
    cmin = warp_min(cmin);
    cmax = warp_max(cmax);
    if (fb > 0.0f && cmin == cmax) {
      nd = (cmax << 13) | least_size_first<unsigned>(nsz, nf, np);
    } else {
      LdgKey best{-1.0, 0, -1, ~0ull};
      int bc = 0;
      for (int i = lane; i < nc; i += 32) {
        const unsigned long long e = i < 32 ? e0 : lds(&cl[i]);
        const int p = (int)(e >> 52), c = (int)((e >> 36) & 0xffffull), s = sz[p];
        const float2 w = pen_of(s, rC);
        if (c == 0 || (float)c * w.x + (float)c * w.y < fb) continue;
        const LdgKey k{ldg_score(c, s, I.C), s, p, e & 0xffffffffull};   // TV/partition.cpp:103-104
        if (ldg_better(k, best)) { best = k; bc = c; }
      }
      const int mine = best.part;
      best = warp_ldg_argmax(best);
      if (best.part >= 0) {
        nd = (__shfl_sync(kAll, bc, __ffs(__ballot_sync(kAll, mine == best.part)) - 1) << 13) | best.part;
      } else {
        int ms, cx = 0;
        const int dn = warp_least_loaded(sz, K, &ms);
        for (int i = lane; i < nc; i += 32) {
          const unsigned long long e = i < 32 ? e0 : lds(&cl[i]);
          if ((int)(e >> 52) == dn) cx = (int)((e >> 36) & 0xffffull);
        }
        nd = (warp_max(cx) << 13) | dn;
      }
    }
  }
  *slack = sl;
  return nd;
}

// TV's clamps on the decision *d of a vertex of part own (TV/partition.cpp:
// 135-143): returns the drift that leaves them as they are.
__device__ __forceinline__ int tv_clamp(const DevInstance& I, const int* sz, int own, int* d, int sl) {
  const int s0 = sz[*d];
  sl = min(sl, s0 > I.max_pw ? s0 - I.max_pw - 1 : I.max_pw - s0);
  if (s0 > I.max_pw) *d = own;
  const int s1 = sz[*d];
  sl = min(sl, s1 < I.min_pw ? I.min_pw - s1 - 1 : s1 - I.min_pw);
  if (s1 < I.min_pw) *d = own;
  return sl;
}

// A position's decision taken again with the sizes sz, TV's clamps included
// (-1: it has no candidate list), and the drift from them it tolerates.  One warp.
__device__ __forceinline__ int recheck(const DevInstance& I, float rC, float Cf, const int* sz, int nc,
                                       const unsigned long long* cl, bool tv, int own, int* slack) {
  *slack = -1;
  if (nc < 0) return -1;
  int d = walk_pick_any(I, rC, Cf, sz, nc, cl, slack) & 0x1fff;
  if (tv) *slack = tv_clamp(I, sz, own, &d, *slack);
  __syncwarp();
  return d;
}

// The marked positions of a group with nets decided again with the sizes sz by
// the whole CTA, 8, 16 or 32 lanes to a position: a lane keeps the best lower
// bound of its candidates' scores and the largest upper bound of the others,
// shuffles meet them.  One candidate clear of the rest wins and tolerates the
// drift that leaves it so; with none above zero the least-loaded part does.
// Near-ties of several counts and lists beyond the staged rows go to
// walk_pick_any, a warp each.
template <bool kStream>
__device__ __forceinline__ void walk_eval(const DevInstance& I, const SpecBuf& B, float Cf, bool tv, float rC,
                                          const int* sz, WalkSmem& S, int i0, int ol) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int n = __popc(S.eval);
  const int lg = n <= kSWarps ? 5 : n <= 2 * kSWarps ? 4 : 3;   // lanes to a position: 2^lg
  const int lanes = 1 << lg, sub = lane & (lanes - 1);
  if (wib * (32 >> lg) >= n) return;
  const int K = I.K;
  const int k = wib * (32 >> lg) + (lane >> lg);
  const bool todo = k < n;
  const int l = todo ? S.list[k] : 0;
  const int4 mt = todo ? S.meta[i0 + l] : make_int4(0, 0, 0, 0);
  const int nc = mt.w >> 8, of = mt.x >> 16;
  const bool staged = todo && nc >= 0 && nc <= kWalkRow;
  const unsigned long long* row = S.ent + (size_t)l * kWalkStride;
  ScoreAcc A;
  const int ncl = staged ? nc : 0;
  for (int x = sub; x < ncl; x += lanes) {
    const unsigned hi32 = (unsigned)(row[x] >> 32);
    const int p = (int)(hi32 >> 20), c = (int)((hi32 >> 4) & 0xffffu);
    if (c > 0) A.add(p, c, pen_of(sz[p], rC));
  }
  A.meet(lanes);
  const bool one = staged && A.one();
  const bool none = staged && A.none();
  int nd = nc < 0 ? -1 : 0, sl = -1;
  if (one) {
    nd = (int)A.be;
    sl = A.slack_one(Cf);
  }
  if (__any_sync(kAll, none)) {
    int ms, s2 = 0x7fffffff;
    const int am = warp_least_loaded(sz, K, &ms);
    for (int p = lane; p < K; p += 32)
      if (p != am) s2 = min(s2, sz[p]);
    s2 = warp_min(s2);
    int cd = 0;
    if (tv) {
      for (int x = sub; x < ncl; x += lanes) {
        const unsigned hi32 = (unsigned)(row[x] >> 32);
        if ((int)(hi32 >> 20) == am) cd = (int)((hi32 >> 4) & 0xffffu);
      }
      if (lanes == 32) cd = __reduce_max_sync(kAll, cd);
      else
        for (int off = 1; off < lanes; off <<= 1) cd = max(cd, __shfl_xor_sync(kAll, cd, off));
    }
    if (none) {
      nd = (cd << 13) | am;
      sl = min((s2 - ms - 1) / 2, A.slack_none(Cf));
    }
  }
  // near-ties of one count, one of them positive for sure: by size and first
  // sighting, as in ldg_decide
  bool tied = staged && !one && !none && A.blo > 0.0f;
  if (__any_sync(kAll, tied)) {
    int cmin = 0x7fffffff, cmax = 0;
    unsigned long long bk = ~0ull;
    int bp = 0;
    for (int x = sub; x < ncl; x += lanes) {
      const unsigned long long e = row[x];
      const unsigned hi32 = (unsigned)(e >> 32);
      const int p = (int)(hi32 >> 20), c = (int)((hi32 >> 4) & 0xffffu);
      const int s = sz[p];
      const float2 w = pen_of(s, rC);
      if (c == 0 || (float)c * w.x + (float)c * w.y < A.blo) continue;
      cmin = min(cmin, c);
      cmax = max(cmax, c);
      const unsigned long long key = ((unsigned long long)((unsigned)s ^ 0x80000000u) << 32) | (unsigned)e;
      if (key < bk) {
        bk = key;
        bp = p;
      }
    }
    if (lanes == 32) {
      cmin = __reduce_min_sync(kAll, cmin);
      cmax = __reduce_max_sync(kAll, cmax);
      const unsigned long long mk = warp_min_u64(bk);
      bp = __shfl_sync(kAll, bp, __ffs(__ballot_sync(kAll, bk == mk)) - 1);
    } else {
      for (int off = 1; off < lanes; off <<= 1) {
        cmin = min(cmin, __shfl_xor_sync(kAll, cmin, off));
        cmax = max(cmax, __shfl_xor_sync(kAll, cmax, off));
        const unsigned long long key = __shfl_xor_sync(kAll, bk, off);
        const int p = __shfl_xor_sync(kAll, bp, off);
        if (key < bk) {
          bk = key;
          bp = p;
        }
      }
    }
    tied = tied && cmin == cmax;
    if (tied) nd = (cmax << 13) | bp;
  }
  const bool slow = todo && nc >= 0 && !one && !none && !tied;
  for (unsigned sm = __ballot_sync(kAll, slow && sub == 0); sm; sm &= sm - 1) {
    const int src = __ffs(sm) - 1;
    int rs;
    const int r = walk_pick_any(I, rC, Cf, sz, __shfl_sync(kAll, nc, src),
                                B.cand + (size_t)(ol + i0 + __shfl_sync(kAll, l, src)) * K, &rs);
    if ((lane >> lg) == (src >> lg)) {
      nd = r;
      sl = rs;
    }
  }
  if (todo && nc >= 0 && tv) {
    int dn = nd & 0x1fff;
    if (kStream) {   // a part above max_pw ends the walk
      sl = min(sl, I.max_pw - sz[dn]);
      if (sz[dn] > I.max_pw) nd = -1;
    } else {
      sl = tv_clamp(I, sz, of, &dn, sl);
      nd = (nd & ~0x1fff) | dn;
    }
  }
  if (todo && sub == 0) {
    S.nd[l] = nd;
    S.nslack[l] = max(sl, 0);
  }
}

// Exclusive prefixes over the lanes of x and y: by popcounts when the lanes
// with one share it (unit weights), else by scans side by side.
__device__ __forceinline__ void lane_prefixes(unsigned x, unsigned y, unsigned* px, unsigned* py) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const unsigned mx = __ballot_sync(kAll, x != 0u), my = __ballot_sync(kAll, y != 0u);
  const unsigned x0 = __shfl_sync(kAll, x, (__ffs(mx) - 1) & 31), y0 = __shfl_sync(kAll, y, (__ffs(my) - 1) & 31);
  if (__all_sync(kAll, (x == 0u || x == x0) && (y == 0u || y == y0))) {
    *px = x0 * (unsigned)__popc(mx & below);
    *py = y0 * (unsigned)__popc(my & below);
    return;
  }
  unsigned ix = x, iy = y;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned t = __shfl_up_sync(kAll, ix, off), u = __shfl_up_sync(kAll, iy, off);
    if (lane >= off) {
      ix += t;
      iy += u;
    }
  }
  *px = ix - x;
  *py = iy - y;
}

// The walk (block 0, every thread).  The positions [zs, end_w) are visited in
// order with the exact sizes each would see: the window-start sizes plus the
// moves before it (the window's movers before zs are in mlist).  The
// validation has checked every decision against the window's movers as they
// are, so a position is decided again only if the decisions changed before it
// may have drifted the sizes beyond what it tolerates on top of those; the
// others keep their decision.  A changed decision goes to dfix with the
// predicted outcome: exact for TV (its accept test is a count of nets) and for
// vertices without nets, else the old decision's, or a move (MSV) / no move
// (MSRV) if that one stayed home.  The walk ends (ctl[0]) at a stale-marker
// risk or at a position without a candidate list; ctl[1] counts the changes.  The streams (kStream) place every vertex: it comes from part K,
// its decision needs no accept test, and TV's walk ends at a part above max_pw.
//
// It is bound by the latency of dependent instructions (about 5 cycles each in
// a lone warp), so it speculates once more, inside the CTA: groups of 32
// positions that no drift reaches are skipped whole; the positions to decide
// again of a group are decided side by side with the sizes at hand, each with
// the drift it tolerates from there; the first warp then takes them in order
// up to the first one that the moves before it may have changed, from which
// the rest of the group is decided again (on 16K vertices of unit weight, K =
// 8, about 9 positions stand per step).  A vertex without nets takes the
// least-loaded part, which its own kind moves with every step: those the
// first warp decides one by one.  Per window of 1M Zipf vertices under TV with
// sizes near the capacity (1215 positions, 67 changes): 446 us with every row
// staged and shuffles to meet the lanes, 293 us with the rows the drift reaches
// and redux.sync.
template <bool kStream>
__device__ void walk_window(const DevInstance& I, const SpecBuf& B, const int* sizes, float Cf, bool tv, bool msv,
                            int pos, int zs, int end_w, int nm, WalkSmem& S, int* sz, int* dl) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int K = I.K;
  const float rC = __fdiv_rn(1.0f, Cf);
  for (int p = threadIdx.x; p < K; p += blockDim.x) {
    sz[p] = sizes[p];
    dl[p] = 0;   // what the changed decisions changed
  }
  if (kStream && threadIdx.x == 0) {   // the streams' placements come from part K
    sz[K] = 0;
    dl[K] = 0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nm; i += blockDim.x) {
    const int4 m = lds(&B.mlist[i]);
    if (m.x >= zs - pos || m.y == 0) continue;
    atomicAdd(&sz[m.z & 0xffff], m.y);
    atomicAdd(&sz[m.z >> 16], -m.y);
  }
  if (threadIdx.x == 0) S.drift = 0;
  int hard = kNone, nchg = 0;   // warp 0
  bool stop = false;
  for (int zl = zs; zl < end_w && !stop; zl += kWalkLoad) {
    const int n = min(kWalkLoad, end_w - zl), ol = zl - pos;
    __syncthreads();   // the first warp has read the last positions' words
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int o = ol + i;
      const int nc = lds(&B.ncand[o]);
      S.meta[i] = make_int4(lds(&B.dec[o]), lds(&B.wt[o]), lds(&B.acc[o]), (nc << 8) | (int)lds(&B.flag[o]));
      S.margin[i] = lds(&B.rel[o]);
    }
    __syncthreads();
    const int ng = (n + 31) >> 5;
    for (int g = wib; g < ng; g += kSWarps) {
      const int i = g * 32 + lane;
      const bool in = i < n;
      int mg = 0x7fffffff;
      if (in) {
        const int fl = S.meta[i].w;
        const int sl = S.margin[i];
        mg = (fl & 32) || ((fl & 2) && zl + i != pos) || sl < -1 ? -1 : max(sl, 0);
        S.margin[i] = mg;
      }
      mg = warp_min(mg);
      if (lane == 0) S.gmin[g] = mg;
    }
    __syncthreads();
    for (int g = 0; g < ng && !stop; g++) {
      // groups that no drift reaches: the first warp applies their moves
      {
        int gn = g;
        for (const int dr = S.drift; gn < ng && dr <= S.gmin[gn]; gn++) {}
        if (wib == 0)
          for (; g < gn; g++) {
            const int i = g * 32 + lane;
            const int4 m = i < n ? S.meta[i] : make_int4(0, 0, 0, 0);
            if (m.w & 1) {
              atomicAdd(&sz[m.x & 0xffff], m.y);
              atomicAdd(&sz[m.x >> 16], -m.y);
            }
          }
        g = gn;
        if (g >= ng) break;
      }
      const int i0 = g * 32, nl = min(32, n - i0);
      // the candidates of the positions in mask: a warp per row, two rows' loads
      // in flight, only the entries there are
      const unsigned fits = __ballot_sync(kAll, lane < nl && (S.meta[i0 + lane].w >> 8) <= kWalkRow);
      auto stage = [&](unsigned mask) {
        for (int k = 0; k < wib && mask; k++) mask &= mask - 1;
        while (mask) {
          int rr[2], nc[2];
#pragma unroll
          for (int u = 0; u < 2; u++) {
            rr[u] = mask ? __ffs(mask) - 1 : 0;
            nc[u] = mask ? S.meta[i0 + rr[u]].w >> 8 : 0;
            for (int k = 0; k < kSWarps && mask; k++) mask &= mask - 1;
          }
          for (int x = lane; x < max(nc[0], nc[1]); x += 64) {
            unsigned long long e[2][2];
#pragma unroll
            for (int u = 0; u < 2; u++)
#pragma unroll
              for (int y = 0; y < 2; y++)
                e[u][y] = x + 32 * y < nc[u] ? lds(&B.cand[(size_t)(ol + i0 + rr[u]) * K + x + 32 * y]) : 0;
#pragma unroll
            for (int u = 0; u < 2; u++)
#pragma unroll
              for (int y = 0; y < 2; y++)
                if (x + 32 * y < nc[u]) S.ent[rr[u] * kWalkStride + x + 32 * y] = e[u][y];
          }
        }
      };
      // those that the drift so far reaches; more as it grows
      unsigned rows = fits & __ballot_sync(kAll, lane < nl && S.margin[i0 + lane] < 2 * S.drift + 4);
      stage(rows);
      __syncthreads();   // also: every thread has read S.drift
      // warp 0: the group at hand, its lanes' positions and their present outcome
      const bool in = lane < nl;
      const int4 m = in ? S.meta[i0 + lane] : make_int4(0, 0, 0, 0);
      const int own = m.x >> 16, w = m.y, mg = in ? S.margin[i0 + lane] : 0x7fffffff;
      const bool iso = (m.w & 8) != 0;
      int d = m.x & 0xffff, j = 0;
      bool mv = (m.w & 1) != 0, done = false;
      int drift = S.drift;
      auto exact_drift = [&]() {
        int D0 = 0;
        for (int p = lane; p < K; p += 32) D0 = max(D0, abs(dl[p]));
        return warp_max(D0);
      };
      if (wib == 0) drift = exact_drift();
      // the moves own -> to of the lanes of mm applied
      auto apply = [&](unsigned mm, int to) {
        if (!mm) return;
        if ((mm >> lane) & 1u) {
          atomicAdd(&sz[to], w);
          atomicAdd(&sz[own], -w);
        }
        __syncwarp();
      };
      while (true) {
        if (wib == 0) {
          unsigned need = 0;
          if (!done && hard == kNone) {
            need = __ballot_sync(kAll, in && lane >= j && drift > mg);
            if (!need) apply(__ballot_sync(kAll, mv && lane >= j), d);   // the rest keeps its outcome
          }
          const unsigned ev = __ballot_sync(kAll, ((need >> lane) & 1u) && !iso);
          if ((ev >> lane) & 1u) S.list[__popc(ev & ((1u << lane) - 1u))] = lane;
          if (lane == 0) {
            S.group = need ? g : -1;
            S.need = need;
            S.eval = ev;
          }
        }
        __syncthreads();
        if (S.group < 0) break;
        if (const unsigned miss = S.eval & fits & ~rows) {
          stage(miss);
          rows |= miss;
          __syncthreads();
        }
        walk_eval<kStream>(I, B, Cf, tv, rC, sz, S, i0, ol);
        __syncthreads();
        if (wib == 0) {
          // ---- take them in order
          const unsigned need = S.need;
          const bool again = (need >> lane) & 1u;
          const int nd = again && !iso ? S.nd[lane] : 0, nsl = again && !iso ? S.nslack[lane] : 0;
          const bool stale = (m.w & 2) && zl + i0 + lane != pos;
          const bool hardf = again && (stale || nd < 0);
          // the outcome of every position decided again, as if its decision stood
          bool mvn = mv;
          int dn = d;
          if (again && !iso && !hardf) {
            dn = nd & 0x1fff;
            if (dn != d)
              mvn = kStream || (dn != own && (tv ? m.z + (nd >> 13) >= 0 : d != own ? (m.w & 16) != 0 : msv));
          }
          const bool chg = dn != d;
          // drift from these sizes before each position, and what the changed
          // decisions before it add to the drift of the others
          unsigned Dn, cn;
          lane_prefixes(mvn && lane >= j ? (unsigned)w : 0u,
                        chg && lane >= j ? (mvn ? (unsigned)w : 0u) + (mv ? (unsigned)w : 0u) : 0u, &Dn, &cn);
          const long long lim = again ? (long long)nsl - Dn : (long long)mg - drift - cn;
          long long moren = 0, morec = 0;   // what the vertices without nets add to both
          while (true) {
            // the first position in doubt: decided again here and reached by the
            // moves since, or not decided again and reached now
            const unsigned db = __ballot_sync(
                kAll, in && lane >= j && ((again && (hardf || iso)) || (again ? moren : morec) > lim));
            const int f = db ? __ffs(db) - 1 : nl;
            // ---- positions [j, f) stand
            const bool keep = lane >= j && lane < f;
            const unsigned cm = __ballot_sync(kAll, keep && chg);
            if (cm) {
              if (keep && chg) {
                B.dfix[ol + i0 + lane] = dn | (mvn ? 1 << 16 : 0);
                B.flag[ol + i0 + lane] = (unsigned char)((m.w & 255) | 128);
                if (mvn) { atomicAdd(&dl[dn], w); atomicAdd(&dl[own], -w); }
                if (mv) { atomicAdd(&dl[d], -w); atomicAdd(&dl[own], w); }
              }
              nchg += __popc(cm);
            }
            if (keep && !chg && (m.w & 128)) B.flag[ol + i0 + lane] = (unsigned char)(m.w & 127);
            apply(__ballot_sync(kAll, keep && mvn), dn);
            j = f;
            if (f >= nl) break;
            const bool af = (need >> f) & 1u;
            if (__shfl_sync(kAll, hardf ? 1 : 0, f)) {
              hard = ((zl + i0 + f) << 3) | (__shfl_sync(kAll, stale ? 1 : 0, f) ? 1 : 2);
              break;
            }
            if (!af || !__shfl_sync(kAll, iso ? 1 : 0, f)) break;   // decided again from here
            // ---- vertices without nets, one by one (and their like after them)
            const unsigned im = need & __ballot_sync(kAll, iso);
            do {
              const int4 mt = S.meta[i0 + j];
              const int of = mt.x >> 16, df = mt.x & 0xffff, wf = mt.y;
              int ms;
              int q = warp_least_loaded(sz, K, &ms);
              if (kStream && tv && ms > I.max_pw) {
                hard = ((zl + i0 + j) << 3) | 2;
                break;
              }
              if (!kStream && tv && (ms > I.max_pw || ms < I.min_pw)) q = of;   // the clamps keep it home
              const bool m1 = (mt.w & 1) != 0;
              const bool m2 = q == df ? m1 : kStream || (q != of && (tv || (mt.w & 16)));
              if (q != df) {
                const int wo = m1 ? wf : 0, wn = m2 ? wf : 0;
                moren += wn - wo;   // (its old weight is in the others' Dn)
                morec += wn + wo;
                nchg++;
                if (lane == 0) {
                  B.dfix[ol + i0 + j] = q | (m2 ? 1 << 16 : 0);
                  B.flag[ol + i0 + j] = (unsigned char)((mt.w & 255) | 128);
                }
                if (lane < 3) atomicAdd(&dl[lane == 0 ? q : lane == 1 ? df : of], lane == 0 ? wn : lane == 1 ? -wo : wo - wn);
              } else if ((mt.w & 128) && lane == 0) {
                B.flag[ol + i0 + j] = (unsigned char)(mt.w & 127);
              }
              if (m2) {
                if (lane < 2) atomicAdd(&sz[lane == 0 ? q : of], lane == 0 ? wf : -wf);
                __syncwarp();
              }
              j++;
            } while (j < nl && ((im >> j) & 1u));
            if (j >= nl || hard != kNone) break;
          }
          // the positions taken keep what was decided
          if (lane < j) {
            mv = mvn;
            d = dn;
          }
          __syncwarp();
          drift = exact_drift();   // from here on
          done = j >= nl;
        }
      }
      if (threadIdx.x == 0) S.drift = drift;
      stop = __syncthreads_or(hard != kNone) != 0;
    }
  }
  if (threadIdx.x == 0) {
    B.ctl[0] = hard;
    B.ctl[1] = nchg;
    B.ctl[8] = kNone;   // the first mispredicted outcome (fix_position)
  }
}

}  // namespace spec
}  // namespace fp
