// Speculative grid-wide refinement for the LDG metrics: TV (TV/partition.cpp:
// 307-440), MSV (MGV/partition.cpp:222-477) and MSRV (MSRV/partition.cpp:240-517).
//
// The reference walks the vertices one by one; every decision reads the state
// left by all earlier moves.  Here one persistent cooperative kernel runs all
// passes as a sequence of rounds.  A round covers a window of the next vertices
// in visiting order:
//
//   A  evaluate   every warp of the grid decides its vertices against the
//                 current state, as if each were next.  A mover claims its nets
//                 (part-set-changing or count-only), and every vertex records
//                 how much part-size / volume drift its outcome tolerates.
//   B  validate   a vertex keeps its outcome iff nothing it read can have
//                 changed: no earlier mover of the window changed the part set
//                 of one of its nets, or the count of its own part there; the
//                 weight moved before it stays within its size slack (the LDG
//                 argmax, its tie-breaks and TV's clamps cannot flip); if it
//                 would leave its part, MSV's / MSRV's accept test comes out
//                 the same with the volumes and max-volume parts that the
//                 earlier movers leave (taken again from the decision's listed
//                 terms where they drifted beyond its slack or the max parts
//                 changed); for TV, no stale marker can apply.  The first
//                 invalid position cuts the
//                 window.  Decisions that the size drift changes do not: they are
//                 taken again -- a few in a long window all at once, otherwise by
//                 a walk of one CTA over the positions in order (walk_window) --
//                 their moves and claims are redone, and the window is validated
//                 again from the first of them.
//   C  commit     all movers before the cut are applied at once -- on any net
//                 they either are alone or only shift counts, which commute --
//                 and the next window starts at the cut.
//
// Every committed outcome therefore equals the reference's sequential outcome.
//
// A mover's slots (own part, destination) in each of its nets' lists are found
// once, by a flattened pass over the slots (locate_nets), and recorded per
// (vertex, net); the gain / loss terms and the commit then take O(1) per net.
// Vertices are classed by work (list slots over their nets, host-side): light
// ones are evaluated by one warp, medium ones by one CTA, and the heaviest (up
// to gmax per window) by teams of CTAs sized by their nets, which split the
// tally, the gain / loss sums and the move in two extra grid phases of the
// window.

#include "fp_walk.cuh"

#include <algorithm>

namespace fp {

namespace {

using namespace spec;

constexpr int kTV = 1, kMSV = 4, kMSRV = 5;
constexpr int kMaxWords = 4096 / 32;   // part masks of the largest K
constexpr int kListed = 64;            // flag bit: the offset has an entry in mlist

struct RoundCtx {
  const int* sizes;
  const float* penf;   // 1 - size / C in float (pen_of)
  const int* marker;
  const int* vol;
  const int* mark;
  int minpart, minsize, second, maxv, cc;
  float Cf;            // C rounded to float
};

// One warp decides a vertex from its tally.  cand / *ncand (if cand is not null)
// receive the re-check entries of the tallied parts (count > 0, no stale TV
// marker) and scan (if not null) TV's scanned-part bits; *slack_out the drift
// of every part's size under which the decision stands.
template <class F>
__device__ int ldg_decide(const DevInstance& I, const RoundCtx& R, const int* cnt, const F* first, int sb,
                          int metric, int v, int own, bool first_of_window, unsigned long long* cand,
                          int* ncand, uint32_t* scan, bool* special, int* slack_out) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int K = I.K;
  const bool tv = metric == kTV;
  int nc = 0;
  bool sp = false, wide = false;
  ScoreAcc A;
  auto usable = [&](int p, int c) { return c > 0 && !(tv && R.marker[p] == v); };
#pragma unroll 4
  for (int p0 = 0; p0 < K; p0 += 32) {
    const int p = p0 + lane;
    const int c = p < K ? cnt[p] : 0;
    const bool stale = tv && c > 0 && R.marker[p] == v;
    sp |= stale;
    const bool ok = c > 0 && !stale;
    const unsigned m = __ballot_sync(kAll, ok);
    if (ok) {
      const int cc = c - (p == own ? 1 : 0);
      if (cand) {
        wide |= c > 0xffff;
        cand[nc + __popc(m & below)] = cand_entry(p, cc, key32(first[p], sb, &wide));
      }
      if (cc > 0) A.add(p, cc, make_float2(R.penf[p], tol_of(R.penf[p])));
    }
    if (scan) {
      const unsigned ms = __ballot_sync(kAll, c > 0);
      if (lane == 0) scan[p0 >> 5] = ms;
    }
    nc += __popc(m);
  }
  wide = __any_sync(kAll, wide);
  if (cand && lane == 0) *ncand = wide ? -1 : nc;
  *special = __any_sync(kAll, sp) && !first_of_window;
  A.meet(32);
  int d0 = R.minpart, sl = -1;
  if (A.cm >= 1 << 19) {   // beyond the packed word (whole-grid vertices): exact scores
    A.blo = A.oh = 1.0f;
  }
  if (A.one()) {
    d0 = (int)(A.be & 0x1fffu);
    sl = A.slack_one(R.Cf);
  } else if (A.none()) {
    sl = min(A.slack_none(R.Cf), (R.second - R.minsize - 1) / 2);   // least-loaded part stays
  } else {
    // near parts: those whose upper bound reaches the largest lower bound
    const float fb = fmaxf(A.cm >= 1 << 19 ? 0.0f : A.blo, 0.0f);
    int np = -1, nsz = 0, cmin = 0x7fffffff, cmax = 0;
    F nf = ~(F)0;
    for (int p = lane; p < K; p += 32) {
      const int c = cnt[p], cc = c - (p == own ? 1 : 0);
      if (!usable(p, c) || cc <= 0) continue;
      const float cf = (float)cc, hi = cf * R.penf[p] + cf * tol_of(R.penf[p]);
      if (!(hi > 0.0f) || hi < fb) continue;
      cmin = min(cmin, cc);
      cmax = max(cmax, cc);
      const int sz = R.sizes[p];
      const F fp = first[p];
      if (np < 0 || sz < nsz || (sz == nsz && fp < nf)) {
        np = p;
        nsz = sz;
        nf = fp;
      }
    }
    cmin = warp_min(cmin);
    cmax = warp_max(cmax);
    if (fb > 0.0f && cmin == cmax) {
      d0 = least_size_first<F>(nsz, nf, np);
    } else {
      LdgKey best{-1.0, 0, -1, ~0ull};
      for (int p = lane; p < K; p += 32) {
        const int c = cnt[p], cc = c - (p == own ? 1 : 0);
        if (!usable(p, c) || cc <= 0) continue;
        const float cf = (float)cc, hi = cf * R.penf[p] + cf * tol_of(R.penf[p]);
        if (!(hi > 0.0f) || hi < fb) continue;   // cannot be a positive best
        const double pen = __dsub_rn(1.0, __ddiv_rn((double)R.sizes[p], I.C));   // TV/partition.cpp:103-104
        LdgKey k{__dmul_rn((double)cc, pen), R.sizes[p], p, key64(first[p], sb)};
        if (ldg_better(k, best)) best = k;
      }
      best = warp_ldg_argmax(best);
      if (best.part >= 0) d0 = best.part;
    }
  }
  int d = d0;
  if (tv) {
    const int s0 = R.sizes[d0];
    sl = min(sl, s0 > I.max_pw ? s0 - I.max_pw - 1 : I.max_pw - s0);
    if (s0 > I.max_pw) d = own;
    const int s1 = R.sizes[d];
    sl = min(sl, s1 < I.min_pw ? I.min_pw - s1 - 1 : s1 - I.min_pw);
    if (s1 < I.min_pw) d = own;
  }
  *slack_out = max(sl, -1);
  return d;
}

// The reference's gains / losses of the move own -> d on net e
// (MGV/partition.cpp:294-337, MSRV/partition.cpp:303-350) and the exact change
// of every part's volume that commit_rec will make (adelta), from the net's
// record r.
__device__ __forceinline__ void net_terms(const DevInstance& I, bool rv, int v, int own, int d, int e, uint32_t r,
                                          int* gains, int* losses, int* adelta) {
  const int n = lds(&I.ep_len[e]);
  const bool rem = rec_rem(r), add = rec_add(r);
  const int sv = __ldg(&I.src[e]);
  const int sp = sv == v ? own : lds(&I.part_vec[sv]);
  if (sv == v) {
    atomicAdd(&gains[own], n - 1);
    atomicAdd(&losses[d], n - 1);
  }
  if (rem) {
    if (sv != v) {
      atomicAdd(&gains[sp], 1);
      if (rv) atomicAdd(&gains[own], 1);
    } else {
      atomicAdd(&losses[d], -1);
    }
  }
  if (add) {
    if (sv != v) {
      atomicAdd(&losses[sp], 1);
      if (rv) atomicAdd(&losses[d], 1);
    } else {
      atomicAdd(&losses[d], 1);
    }
  }
  const int n1 = rem ? n - 1 : n;
  if (sv == v) {
    atomicAdd(&adelta[own], -(n - 1));
    atomicAdd(&adelta[d], n1 - 1);
  }
  if (rem) {
    if (sv != v) {
      atomicAdd(&adelta[sp], -1);
      if (rv) atomicAdd(&adelta[own], -1);
    }
  } else if (rv && sv == v) {
    atomicAdd(&adelta[own], 1);
  }
  if (!add) {
    if (rv && sv == v) atomicAdd(&adelta[d], -1);
  } else {
    atomicAdd(&adelta[sv == v ? d : sp], 1);
    if (rv && sv != v) atomicAdd(&adelta[d], 1);
  }
}

// Records of v's nets [n0, n1) for the move own -> d (one warp).  With volumes
// (MSV / MSRV) the gain / loss / volume terms are added to the arrays.  loc: the
// warp's 96 ints of scratch.  Returns this lane's counts of nets the move takes
// own off (low 16 bits) and appends d to (high 16), TV's leave gain and arrival
// loss (of a vertex one warp evaluates: fewer than 65536 nets).
__device__ int locate_range(const DevInstance& I, const SpecBuf& B, int metric, int v, int own, int d, uint32_t base,
                            int n0, int n1, int* loc, int* gains, int* losses, int* adelta) {
  const bool vol = metric != kTV, rv = metric == kMSRV;
  int ra = 0;
  locate_nets(I, B.rec, v, own, d, base, n0, n1, loc, [&](int e, uint32_t r) {
    ra += (rec_rem(r) ? 1 : 0) + (rec_add(r) ? 1 << 16 : 0);
    if (vol) net_terms(I, rv, v, own, d, e, r, gains, losses, adelta);
  });
  return ra;
}
// The same for warp wi of nw warps splitting all of v's nets (net_range).
__device__ __forceinline__ int locate_all(const DevInstance& I, const SpecBuf& B, int metric, int v, int own, int d,
                                          uint32_t base, int deg, int wi, int nw, int* loc, int* gains, int* losses,
                                          int* adelta) {
  int n0, n1;
  net_range(deg, wi, nw, &n0, &n1);
  return locate_range(I, B, metric, v, own, d, base, n0, n1, loc, gains, losses, adelta);
}

// Count claims, exactly: an open-addressed table from (net, part) to the first
// window position of a count-only mover that changes that part's count on that
// net.  Movers insert in evaluation and clear the slots they recorded at
// commit, so the table is empty between rounds.  A probe longer than kProbe
// marks the round (ctab_over), whose checks then fall back to the part mask.
constexpr int kProbe = 32;
__device__ __forceinline__ uint32_t ctab_hash(int e, int p) {
  uint32_t h = (uint32_t)e * 0x9E3779B1u ^ ((uint32_t)p * 0x85EBCA77u);
  return h ^ (h >> 15);
}
__device__ __forceinline__ unsigned long long ctab_keyof(int e, int p) {
  return ((unsigned long long)(unsigned)e << 12) | (unsigned)p;
}
__device__ uint32_t ctab_insert(const SpecBuf& B, int e, int p, int z, int par) {
  const unsigned long long key = ctab_keyof(e, p);
  uint32_t s = ctab_hash(e, p) & B.ctab_mask;
  for (int i = 0; i < kProbe; i++) {
    const unsigned long long prev = atomicCAS(&B.ctab_key[s], ~0ull, key);
    if (prev == ~0ull || prev == key) {
      atomicMin(&B.ctab_pos[s], z);
      atomicAdd(&B.ctab_cnt[s], 1);
      return s;
    }
    s = (s + 1) & B.ctab_mask;
  }
  atomicExch(&B.ctab_over[par], 1);
  return ~0u;
}
// First position of a count-only mover on (e, p) and the number of such movers
// in the round (*n); kNone if none, -1 if unknown.
__device__ int ctab_find(const SpecBuf& B, int e, int p, int* n) {
  const unsigned long long key = ctab_keyof(e, p);
  uint32_t s = ctab_hash(e, p) & B.ctab_mask;
  for (int i = 0; i < kProbe; i++) {
    const unsigned long long k = lds(&B.ctab_key[s]);
    if (k == key) {
      *n = lds(&B.ctab_cnt[s]);
      return lds(&B.ctab_pos[s]);
    }
    if (k == ~0ull) return kNone;
    s = (s + 1) & B.ctab_mask;
  }
  return -1;
}

// Claims of the mover at position z on its nets k0, k0 + kstep, ...: a change
// of the part set (or, with volumes, of the source's side) takes claim_m, a
// count-only change claim_c, the bits of the two parts and their table entries.
__device__ __forceinline__ void claim_nets(const DevInstance& I, const SpecBuf& B, bool vol, int z, int own, int d,
                                           uint32_t base, int deg, int k0, int kstep, int par) {
  const uint32_t bits = (1u << (own & 31)) | (1u << (d & 31));
  for (int k = k0; k < deg; k += kstep) {
    const int e = (int)__ldg(&I.vnets[base + k]);
    if (rec_setchange(lds(&B.rec[base + k]), vol)) {
      atomicMin(&B.claim_m[e], z);
    } else {
      atomicMin(&B.claim_c[e], z);
      atomicOr(&B.mask_c[e], bits);
      const uint32_t s1 = ctab_insert(B, e, own, z, par);
      const uint32_t s2 = ctab_insert(B, e, d, z, par);
      B.rec_slot[base + k] = make_uint2(s1, s2);
    }
  }
}

// Appends a mover of window offset o (weight wv, vn volume terms) to the
// round's list.  An offset is appended once per round (flag bit 6), so the list,
// with an entry per offset, is long enough.
__device__ __forceinline__ void list_mover(const DevInstance& I, const SpecBuf& B, int par, int o, int wv, int pk,
                                           int vn) {
  const int i = atomicAdd(&B.mcnt[par], 1);
  if (i >= B.wmax) {
    atomicSub(&B.mcnt[par], 1);
    dev_fail(I.status, kDevErrInvalid);
    return;
  }
  B.mlist[i] = make_int4(o, wv, pk, vn);
  B.midx[o] = i;
}
// The same for an offset decided again (fl: its flag before): a mover's entry is
// replaced, also that of one that an earlier change of the window made stay.
// Returns the flag bit of a listed offset.  (Not inlined: inside the kernel, whose
// registers are all taken, its statistic cost MSRV on 262144 Zipf vertices 6%.)
__device__ __noinline__ int relist_mover(const DevInstance& I, const SpecBuf& B, int par, int o, int fl, bool mover,
                                         int wv, int pk, int vn) {
  if (fl & kListed) {
    B.mlist[lds(&B.midx[o])] = make_int4(o, mover ? wv : 0, pk, mover ? vn : 0);
    if (mover && !(fl & 1)) atomicAdd(&B.stats[10], 1ull);
    return kListed;
  }
  if (!mover) return 0;
  list_mover(I, B, par, o, wv, pk, vn);
  return kListed;
}

__device__ __forceinline__ void ctab_clear(const SpecBuf& B, uint2 sl) {
  if (sl.x != ~0u) { B.ctab_key[sl.x] = ~0ull; B.ctab_pos[sl.x] = kNone; B.ctab_cnt[sl.x] = 0; }
  if (sl.y != ~0u) { B.ctab_key[sl.y] = ~0ull; B.ctab_pos[sl.y] = kNone; B.ctab_cnt[sl.y] = 0; }
}

// Clears the claims on net e (commit phase: movers' nets, replaced claims).
__device__ __forceinline__ void unclaim_net(const SpecBuf& B, int e) {
  B.claim_m[e] = kNone;
  B.claim_c[e] = kNone;
  B.mask_c[e] = 0;
}
// Clears the claims of a mover on its nets k0, k0 + kstep, ... and its entries of
// the count table.
__device__ __forceinline__ void unclaim_nets(const DevInstance& I, const SpecBuf& B, bool vol, uint32_t base, int deg,
                                             int k0, int kstep) {
  for (int k = k0; k < deg; k += kstep) {
    unclaim_net(B, (int)__ldg(&I.vnets[base + k]));
    if (!rec_setchange(lds(&B.rec[base + k]), vol)) ctab_clear(B, lds(&B.rec_slot[base + k]));
  }
}

// Takes deg entries of rlist for the claims of a move about to be replaced (one
// thread): the first, or one from which they do not fit.  (A full list is not
// counted on: the count stays far from overflow whatever the degrees.)
__device__ __noinline__ int replaced_entries(const SpecBuf& B, int par, int deg) {
  int* const n = &B.ctl[14 + par];
  return lds(n) > B.rmax ? B.rmax : atomicAdd(n, min(deg, B.rmax + 1));
}

// Lists the claims of a move about to be replaced, entries [at, at + deg) of
// rlist (nets k0, k0 + kstep, ...); false if they do not fit.  The claims stay
// until the commit: a superset keeps every later check conservative.
__device__ __forceinline__ bool list_replaced(const DevInstance& I, const SpecBuf& B, bool vol, uint32_t base, int deg,
                                              int k0, int kstep, int at) {
  const bool fits = deg <= B.rmax - at;
  for (int k = k0; k < min(deg, B.rmax - at); k += kstep) {
    const uint2 sl = !fits || rec_setchange(lds(&B.rec[base + k]), vol) ? make_uint2(~0u, ~0u)
                                                                        : lds(&B.rec_slot[base + k]);
    B.rlist[at + k] = make_int4(fits ? (int)__ldg(&I.vnets[base + k]) : -1, (int)sl.x, (int)sl.y, 0);
  }
  return fits;
}

// Did an earlier mover of the window change something the vertex at z read on
// its nets k0, k0 + kstep, ...?  0: nothing; 5: a part set; 6: the count of
// z's own part where it matters.  *after: z (a mover) changes the part set of a
// net whose counts an earlier mover changes, so the counts are committed first
// (a barrier more; the window used to end at z, 31 of 145 windows per pass on
// 10,000 mixed vertices under MSV and 176 of 1220 on 262144 Zipf vertices).
//
// Counts enter a decision only through "own has exactly one pin on the net",
// and only when the vertex would move (cand: decision != own; its move records
// hold own's slot).  Before the commit the count c it saw is still in place;
// earlier count-only moves can make it 1 only if c == 1 or if at least c - 1
// of the round's count-only movers touch (net, own).
__device__ __forceinline__ int conflicts(const DevInstance& I, const SpecBuf& B, bool vol, int z, int own,
                                         bool cand, bool mover, uint32_t base, int deg, int k0, int kstep, bool ov, bool* after) {
  const unsigned ob = 1u << (own & 31);
  int conf = 0;
  for (int k = k0; k < deg && !conf; k += kstep) {
    const int e = (int)__ldg(&I.vnets[base + k]);
    if (lds(&B.claim_m[e]) < z) {
      conf = 5;
    } else if (cand && lds(&B.claim_c[e]) < z) {
      bool hit;
      if (ov) {
        hit = (lds(&B.mask_c[e]) & ob) != 0;
      } else {
        int n = 0;
        const int fp = ctab_find(B, e, own, &n);
        if (fp < 0) {
          hit = true;
        } else if (fp >= z) {
          hit = false;
        } else {
          const int c = lds(&I.ep_cnt[(int)__ldg(&I.nptr[e]) + rec_jo(lds(&B.rec[base + k]))]);
          hit = c <= 1 || n >= c - 1;
        }
      }
      if (hit) conf = 6;
      else if (mover && rec_setchange(lds(&B.rec[base + k]), vol)) *after = true;
    }
  }
  return conf;
}

// Per-thread partial of the MSV / MSRV accept test (MGV/partition.cpp:339-362,
// MSRV/partition.cpp:352-376) over parts p0, p0 + pstep, ...
struct AcceptPart {
  bool failM, failN, mt;
  int fsl, msl, vd;
};

__device__ AcceptPart accept_partial(const RoundCtx& R, const int* gains, const int* losses, const int* adelta, int K,
                                     bool rv, int p0, int pstep) {
  AcceptPart a{false, false, false, -1, kBig, 0};
  for (int p = p0; p < K; p += pstep) {
    const int g = gains[p], l = losses[p];
    const int t = R.vol[p] + l - g;
    if (R.mark[p] == R.cc) {
      if (rv ? (g <= l) : (g < l)) a.failM = true;
      if (adelta[p] != 0) a.mt = true;
    } else {
      if (t >= R.maxv) { a.failN = true; a.fsl = max(a.fsl, t - R.maxv); }
      a.msl = min(a.msl, R.maxv - 1 - t);
    }
    a.vd = max(a.vd, abs(adelta[p]));
  }
  return a;
}

// The volume terms of window offset o (a decision that leaves its part): the
// parts with a loss or gain or an exact change, in part order; one warp.
// Returns their number, -1 if there are more than kVolTerms.
__device__ int store_terms(const SpecBuf& B, int o, int K, const int* gains, const int* losses, const int* adelta) {
  const int lane = threadIdx.x & 31;
  int n = 0;
  for (int p0 = 0; p0 < K; p0 += 32) {
    const int p = p0 + lane;
    const int df = p < K ? losses[p] - gains[p] : 0, ad = p < K ? adelta[p] : 0;
    const unsigned m = __ballot_sync(kAll, df != 0 || ad != 0);
    const int i = n + __popc(m & ((1u << lane) - 1u));
    if (((m >> lane) & 1u) && i < kVolTerms) {
      B.vterm[(size_t)o * kVolTerms + i] = make_int2(df, ad);
      B.vpart[(size_t)o * kVolTerms + i] = (unsigned short)p;
    }
    n += __popc(m);
  }
  if (n > kVolTerms) n = -1;
  if (lane == 0) B.vn[o] = n;
  return n;
}

// Max-volume parts while the window's movers are applied: state x holds after x
// of the movers that change the set (kVolEvents at most; the window ends at the
// next).  Outcomes rarely change with the volumes (none in a pass of the Zipf
// workloads, 2 on 10,000 mixed vertices), but a bound on the drift (the sum of the
// movers' largest changes) and every change of a max part used to end the
// window: 548 -> 145 windows per pass on 10,000 mixed vertices under MSV (K =
// 64), 25.9 -> 17.5 ms; MSRV on 262144 Zipf vertices (K = 256) 244 -> 112, 15.5
// -> 10.0 ms; MSV there 1546 -> 1220.
constexpr int kVolEvents = 15;   // (kVolEvents + 1) * ceil(K / 32) <= 8 * K for K >= 2
struct VolStates {
  int n;                       // such movers found
  int at[kVolEvents];          // their window offsets
  int maxv[kVolEvents + 1], nm[kVolEvents + 1], count[kVolEvents + 1];
  int over;                    // offset of the first mover without listed terms
  int end;                     // first offset whose max parts are not known
  int ne, next, m2, chg, add, off;   // scratch
};

// The accept test of window offset o (one warp) from its listed terms with the
// max parts `bits` (nm of them, volume maxv) and the other volumes vx(p),
// computed on the first call.  MGV/partition.cpp:339-362 and
// MSRV/partition.cpp:352-376 over the parts the move touches: an untouched max
// part fails MSRV's test; an untouched other part reaches maxv only under
// MSRV, whose changes differ from gain and loss by the source's own pin.
template <class Build, class Vx>
__device__ bool accept_terms(const SpecBuf& B, int o, int n, int K, bool rv, const uint32_t* bits, int nm, int maxv,
                             Build&& build, Vx&& vx) {
  const int lane = threadIdx.x & 31;
  bool fail = false, other = false;
  int neg = 0;
  for (int t = lane; t < n; t += 32) {
    const int p = (int)__ldcg(&B.vpart[(size_t)o * kVolTerms + t]);
    const int df = __ldcg(&B.vterm[(size_t)o * kVolTerms + t].x);
    if ((bits[p >> 5] >> (p & 31)) & 1u) {
      if (rv ? df >= 0 : df > 0) fail = true;
      else neg++;
    } else {
      other = true;
    }
  }
  if (__any_sync(kAll, fail)) return false;
  if (rv && warp_sum(neg) != nm) return false;
  if (!rv && !__any_sync(kAll, other)) return true;
  build();
  int high = 0;
  for (int t = lane; t < n; t += 32) {
    const int p = (int)__ldcg(&B.vpart[(size_t)o * kVolTerms + t]);
    const int df = __ldcg(&B.vterm[(size_t)o * kVolTerms + t].x);
    if ((bits[p >> 5] >> (p & 31)) & 1u) continue;
    if (vx(p) + df >= maxv) fail = true;
    high -= vx(p) >= maxv;
  }
  if (rv)
    for (int p = lane; p < K; p += 32) high += !((bits[p >> 5] >> (p & 31)) & 1u) && vx(p) >= maxv;
  return !__any_sync(kAll, fail) && (!rv || warp_sum(high) == 0);
}

// Outcome and volume slack: accepted -> stays accepted while no non-max part
// rises by more than msl; rejected on a max part -> local, stays rejected;
// rejected only on non-max parts -> stays rejected while the worst of them
// drops by at most fsl.
__device__ __forceinline__ void accept_final(bool failM, bool failN, int fsl, int msl, bool* good, int* vslack) {
  *good = !failM && !failN;
  *vslack = *good ? msl : (failM ? kBig : fsl);
}

__device__ __forceinline__ int block_reduce_max(int x, int* scr) {
  x = warp_max(x);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scr[threadIdx.x >> 5] = x;
  __syncthreads();
  int r = scr[0];
  for (int i = 1; i < (int)(blockDim.x >> 5); i++) r = max(r, scr[i]);
  __syncthreads();
  return r;
}
__device__ __forceinline__ int block_reduce_sum(int x, int* scr) {
  x = warp_sum(x);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scr[threadIdx.x >> 5] = x;
  __syncthreads();
  int s = 0;
  for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += scr[i];
  __syncthreads();
  return s;
}
__device__ __forceinline__ int block_reduce_min(int x, int* scr) {
  return -block_reduce_max(-x, scr);
}

// Evaluation of a medium vertex at position z by the whole CTA: the warps split
// the tally, warp 0 decides, the warps split the locate pass and the gain /
// loss terms.  All warps add to one set of K-sized arrays (native 32-bit
// shared-memory atomics): nothing is merged per warp.  Writes the same
// per-position record as a warp evaluation (flag bit 2 marks it).
__device__ void cta_eval_ldg(const DevInstance& I, const SpecBuf& B, const RoundCtx& R, int metric, int z, int pos,
                             int par, int sb, int* cnt_b, unsigned* first_b, int* gains_b, int* losses_b,
                             int* adelta_b, int* iscr, int* loc_b, bool logp) {
  __shared__ int sh[4];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int K = I.K;
  const int words = (K + 31) >> 5;
  const bool vol = metric != kTV, rv = metric == kMSRV;
  const int o = z - pos;
  const int v = __ldg(&B.porder[z]);
  const int own = lds(&I.part_vec[v]);
  const uint32_t base = __ldg(&I.vptr[v]);
  const int deg = (int)(__ldg(&I.vptr[v + 1]) - base);
  const long long t0 = clock64();
  for (int p = threadIdx.x; p < K; p += blockDim.x) {
    cnt_b[p] = 0;
    first_b[p] = ~0u;
    if (vol) { gains_b[p] = 0; losses_b[p] = 0; adelta_b[p] = 0; }
  }
  __syncthreads();
  int c1 = 0;
  int n0, n1;
  net_range(deg, wib, kSWarps, &n0, &n1);
  c1 = tally_range<true>(I, own, base, n0, n1, 0, sb, cnt_b, first_b);
  c1 = warp_sum(c1);
  if (lane == 0) iscr[wib] = c1;
  __syncthreads();
  int c1t = 0;
  for (int x = 0; x < kSWarps; x++) c1t += iscr[x];
  const long long t1 = clock64();
  if (wib == 0) {
    bool special;
    int slack;
    const int d = ldg_decide(I, R, cnt_b, first_b, sb, metric, v, own, z == pos, B.cand + (size_t)o * K,
                             &B.ncand[o], metric == kTV ? B.scan + (size_t)o * words : nullptr, &special, &slack);
    if (lane == 0) {
      sh[0] = d;
      sh[1] = special ? 1 : 0;
      sh[2] = slack;
    }
  }
  __syncthreads();
  const long long t2 = clock64();
  const int d = sh[0];
  const bool special = sh[1] != 0;
  const int slack = sh[2];
  bool mover = false, mt = false;
  int vs = kBig, vdd = 0, nt = 0;
  int rg = 0, rl = 0;   // decision record (with the log on)
  if (d != own) {
    // TV moves iff the leave gain covers the arrival loss; MSV / MSRV need the
    // accept test on the gain / loss sums.
    if (metric == kTV) {
      rg = c1t;
      rl = deg - cnt_b[d];
    }
    const bool need = metric == kTV ? c1t >= deg - cnt_b[d] : true;
    mover = metric == kTV && need;
    {   // records for every decision that moves: own's slot per net serves the validation
      locate_all(I, B, metric, v, own, d, base, deg, wib, kSWarps, loc_b + wib * 96, gains_b, losses_b, adelta_b);
      __syncthreads();
      if (vol) {
        const AcceptPart a = accept_partial(R, gains_b, losses_b, adelta_b, K, rv, threadIdx.x, blockDim.x);
        const bool fM = __syncthreads_or(a.failM);
        const bool fN = __syncthreads_or(a.failN);
        const bool amt = __syncthreads_or(a.mt);
        const int fsl = block_reduce_max(a.fsl, iscr);
        const int msl = block_reduce_min(a.msl, iscr);
        vdd = block_reduce_max(a.vd, iscr);
        if (wib == 0) nt = store_terms(B, o, K, gains_b, losses_b, adelta_b);
        bool good;
        accept_final(fM, fN, fsl, msl, &good, &vs);
        mover = good;
        mt = mover && amt;
        if (logp) {
          int g = 0, l = 0;
          for (int p = threadIdx.x; p < K; p += blockDim.x) { g += gains_b[p]; l += losses_b[p]; }
          rg = block_reduce_sum(g, iscr);
          rl = block_reduce_sum(l, iscr);
        }
      }
    }
  }
  if (mover) {
    claim_nets(I, B, vol, z, own, d, base, deg, threadIdx.x, blockDim.x, par);
    if (threadIdx.x == 0) {
      if (mt) atomicMin(&B.ctl[2 + par], z);
      list_mover(I, B, par, o, __ldg(&I.w[v]), (own << 16) | d, nt);
    }
  }
  if (threadIdx.x == 0) {
    if (logp) { B.rgain[o] = rg; B.rloss[o] = rl; }
    B.dec[o] = (own << 16) | d;
    B.flag[o] = (unsigned char)((mover ? 1 | kListed : 0) | (special ? 2 : 0) | 4 | (!vol || mover ? 16 : 0));
    B.slack[o] = slack;
    B.vslack[o] = vs;
    B.wt[o] = __ldg(&I.w[v]);
    B.acc[o] = c1t - deg;
    B.vd[o] = mover ? vdd : 0;
    // CTA evaluation statistics (cycles): tally and merge / decision / the rest
    const long long t3 = clock64();
    if (kTimingStats) {
      atomicAdd(&B.stats[29], (unsigned long long)(t1 - t0));
      atomicAdd(&B.stats[30], (unsigned long long)(t2 - t1));
      atomicAdd(&B.stats[31], (unsigned long long)(t3 - t2));
      atomicAdd(&B.stats[40], 1ull);
    }
  }
  __syncthreads();
}

// The position z (window offset o) whose decision the last walk changed: the
// move records, the accept test and the claims are redone for the new
// decision.  The replaced move's claims stay (list_replaced; where they do not
// fit, the window ends here instead, ctl[9]).  An outcome other than the walk
// predicted lowers ctl[8]: the decisions after it are validated again.
// One warp, the one owning position z.
__device__ void fix_position(const DevInstance& I, const SpecBuf& B, const RoundCtx& R, int metric, int z, int o,
                             int fl, int par, int* loc, int* gains, int* losses, int* adelta, bool logp) {
  const int lane = threadIdx.x & 31;
  const bool vol = metric != kTV, rv = metric == kMSRV;
  const int K = I.K;
  const int v = __ldg(&B.porder[z]);
  const uint32_t base = __ldg(&I.vptr[v]);
  const int deg = (int)(__ldg(&I.vptr[v + 1]) - base);
  const int own = lds(&B.dec[o]) >> 16;
  const int fx = lds(&B.dfix[o]);
  const int d = fx & 0xffff;
  const bool had = (fl & 1) != 0;
  if (had && deg) {
    const int at = __shfl_sync(kAll, lane == 0 ? replaced_entries(B, par, deg) : 0, 0);
    if (!list_replaced(I, B, vol, base, deg, lane, 32, at)) {
      if (lane == 0) {
        atomicMin(&B.ctl[9], (z << 3) | 2);
        B.flag[o] = (unsigned char)(fl & ~128);
      }
      return;
    }
    __syncwarp();
  }
  bool mover = false, mt = false, good = (fl & 16) != 0;
  int vs = kBig, vdd = 0, nt = 0;
  int rg = 0, rl = 0;
  if (deg == 0) {
    mover = d != own && (!vol || good);
    vs = lds(&B.vslack[o]);
    if (vol && lane == 0) B.vn[o] = 0;
  } else if (d != own) {
    if (vol) {
      for (int p = lane; p < K; p += 32) { gains[p] = 0; losses[p] = 0; adelta[p] = 0; }
      __syncwarp();
    }
    const int ra = locate_all(I, B, metric, v, own, d, base, deg, 0, 1, loc, gains, losses, adelta);
    __syncwarp();
    if (vol) {
      const AcceptPart a = accept_partial(R, gains, losses, adelta, K, rv, lane, 32);
      const bool fM = __any_sync(kAll, a.failM);
      const bool fN = __any_sync(kAll, a.failN);
      accept_final(fM, fN, warp_max(a.fsl), warp_min(a.msl), &good, &vs);
      mover = good;
      mt = mover && __any_sync(kAll, a.mt);
      vdd = warp_max(a.vd);
      nt = store_terms(B, o, K, gains, losses, adelta);
      if (logp) {
        for (int p = lane; p < K; p += 32) { rg += gains[p]; rl += losses[p]; }
        rg = warp_sum(rg);
        rl = warp_sum(rl);
      }
    } else {
      rg = warp_sum(ra & 0xffff);
      rl = warp_sum(ra >> 16);
      mover = rg >= rl;   // leave gain >= arrival loss (TV/partition.cpp:355-380)
    }
  }
  __syncwarp();
  if (mover) {
    claim_nets(I, B, vol, z, own, d, base, deg, lane, 32, par);
    if (lane == 0 && mt) atomicMin(&B.ctl[2 + par], z);
  }
  if (lane == 0) {
    if (logp) { B.rgain[o] = rg; B.rloss[o] = rl; }
    if (mover != (fx >> 16 != 0)) atomicMin(&B.ctl[8], z);
    const int listed = relist_mover(I, B, par, o, fl, mover, __ldg(&I.w[v]), (own << 16) | d, nt);
    B.dec[o] = (own << 16) | d;
    B.flag[o] = (unsigned char)((fl & (2 | 8)) | listed | (mover ? 1 : 0) | (good ? 16 : 0) | 32);
    B.vslack[o] = vs;
    B.vd[o] = mover ? vdd : 0;
  }
  __syncwarp();
}

// The same for a medium vertex or one of the whole grid, by one CTA (deg > 0).
__device__ void cta_fix(const DevInstance& I, const SpecBuf& B, const RoundCtx& R, int metric, int z, int o, int fl,
                        int par, int* loc_b, int* gains_b, int* losses_b, int* adelta_b, int* iscr, bool logp) {
  const int wib = threadIdx.x >> 5;
  const bool vol = metric != kTV, rv = metric == kMSRV;
  const int K = I.K;
  const int v = __ldg(&B.porder[z]);
  const uint32_t base = __ldg(&I.vptr[v]);
  const int deg = (int)(__ldg(&I.vptr[v + 1]) - base);
  const int own = lds(&B.dec[o]) >> 16;
  const int fx = lds(&B.dfix[o]);
  const int d = fx & 0xffff;
  const bool had = (fl & 1) != 0;
  if (had) {
    if (threadIdx.x == 0) iscr[0] = replaced_entries(B, par, deg);
    __syncthreads();
    if (!list_replaced(I, B, vol, base, deg, threadIdx.x, blockDim.x, iscr[0])) {
      if (threadIdx.x == 0) {
        atomicMin(&B.ctl[9], (z << 3) | 2);
        B.flag[o] = (unsigned char)(fl & ~128);
      }
      return;
    }
    __syncthreads();
  }
  if (vol)
    for (int p = threadIdx.x; p < K; p += blockDim.x) { gains_b[p] = 0; losses_b[p] = 0; adelta_b[p] = 0; }
  __syncthreads();
  bool mover = false, mt = false;
  int vs = kBig, vdd = 0, nt = 0, rg = 0, rl = 0;
  if (d != own) {
    const int ra = locate_all(I, B, metric, v, own, d, base, deg, wib, kSWarps, loc_b + wib * 96, gains_b, losses_b,
                              adelta_b);
    __syncthreads();
    if (vol) {
      const AcceptPart a = accept_partial(R, gains_b, losses_b, adelta_b, K, rv, threadIdx.x, blockDim.x);
      const bool fM = __syncthreads_or(a.failM);
      const bool fN = __syncthreads_or(a.failN);
      const bool amt = __syncthreads_or(a.mt);
      const int fsl = block_reduce_max(a.fsl, iscr);
      const int msl = block_reduce_min(a.msl, iscr);
      vdd = block_reduce_max(a.vd, iscr);
      if (wib == 0) nt = store_terms(B, o, K, gains_b, losses_b, adelta_b);
      accept_final(fM, fN, fsl, msl, &mover, &vs);
      mt = mover && amt;
      if (logp) {
        int g = 0, l = 0;
        for (int p = threadIdx.x; p < K; p += blockDim.x) { g += gains_b[p]; l += losses_b[p]; }
        rg = block_reduce_sum(g, iscr);
        rl = block_reduce_sum(l, iscr);
      }
    } else {
      rg = block_reduce_sum(ra & 0xffff, iscr);
      rl = block_reduce_sum(ra >> 16, iscr);
      mover = rg >= rl;
    }
  }
  if (mover) {
    claim_nets(I, B, vol, z, own, d, base, deg, threadIdx.x, blockDim.x, par);
    if (threadIdx.x == 0 && mt) atomicMin(&B.ctl[2 + par], z);
  }
  if (threadIdx.x == 0) {
    if (logp) { B.rgain[o] = rg; B.rloss[o] = rl; }
    if (mover != (fx >> 16 != 0)) atomicMin(&B.ctl[8], z);
    const int listed = relist_mover(I, B, par, o, fl, mover, __ldg(&I.w[v]), (own << 16) | d, nt);
    B.dec[o] = (own << 16) | d;
    B.flag[o] = (unsigned char)((fl & (2 | 4)) | listed | (mover ? 1 : 0) | (!vol || mover ? 16 : 0) | 32);
    B.vslack[o] = vs;
    B.vd[o] = mover ? vdd : 0;
  }
  __syncthreads();
}

// Changed decisions are taken at once, not walked, in a stretch longer than
// this with at most so many of them: a walk costs about 2 us per 10 positions
// it decides again, a validation of the whole window 12-25 us.
// Up to kJacobiFew are tried so at first in any stretch (7564 uniform vertices, K =
// 24, MSV: 9.7 -> 9.0 ms for three passes).
constexpr int kJacobiSpan = 1024, kJacobiFlips = 64, kJacobiFew = 4;

// MSRV: a window with more changed decisions than this ends behind its first
// change of the max-volume parts: walking them costs more than a new window, and
// most change nothing (three passes over 41936 mixed vertices of unit weight, K =
// 32: 10.6 ms with every change walked, 8.6 so, 8.9 with none).
constexpr int kWalkOverEvent = 4;

// Two CTAs per SM: without the hint the compiler trades registers for a third
// CTA and spills, which measured slower.
__global__ void __launch_bounds__(kSThreads, 2) spec_ldg_kernel(DevInstance I, SpecBuf B, int passes) {
  barrier_start();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long uscr[kSWarps];
  __shared__ int iscr[kSWarps];
  __shared__ int s_minpart, s_minsize, s_second, s_maxv, s_cc, s_count;
  // the window's whole-grid vertices: position, vertex, own part, first net
  // index, degree, decision, stale-marker risk, size slack
  __shared__ int s_gz[kMaxGridVerts], s_gv[kMaxGridVerts], s_go[kMaxGridVerts], s_gd[kMaxGridVerts];
  __shared__ uint32_t s_gb[kMaxGridVerts];
  __shared__ int s_gdec[kMaxGridVerts], s_gspec[kMaxGridVerts], s_gslk[kMaxGridVerts], s_gcnt[kMaxGridVerts];
  __shared__ int s_t0[kMaxGridVerts], s_t1[kMaxGridVerts];   // their teams of CTAs
  __shared__ int loc_b[kSWarps * 96];   // per-warp locate scratch
  __shared__ VolStates vs_s;
  __shared__ uint32_t cmask_s[kMaxWords];
  const int metric = I.metric;
  const bool vol = metric != kTV;
  const bool rv = metric == kMSRV;
  const int K = I.K;
  const int words = (K + 31) >> 5;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int gw = blockIdx.x * kSWarps + wib;
  const int nwarps = gridDim.x * kSWarps;
  const float Cf = (float)I.C;
  Carve cv{smem_raw};
  int* sizes_s = cv.take<int>(K);
  float* penf_s = cv.take<float>(K);
  int* marker_s = cv.take<int>(K);
  int* vol_s = cv.take<int>(K);
  int* mark_s = cv.take<int>(K);
  int* cnt_b = cv.take<int>((size_t)K * kSWarps);                    // per-warp arrays, warp x at x*K
  // sighting keys: the warps' 32-bit ones (warp x at x*K), or the 64-bit ones of
  // the window's whole-grid vertices (vertex j at j*K)
  unsigned long long* first64_b = cv.take<unsigned long long>((size_t)K * kSWarps);
  unsigned* first_b = reinterpret_cast<unsigned*>(first64_b);
  int* gains_b = cv.take<int>((size_t)K * kSWarps);
  int* losses_b = cv.take<int>((size_t)K * kSWarps);
  int* adelta_b = cv.take<int>((size_t)K * kSWarps);
  int* cnt = cnt_b + (size_t)wib * K;
  unsigned* first = first_b + (size_t)wib * K;
  const int sb = slot_bits(K);
  int* gains = gains_b + (size_t)wib * K;
  int* losses = losses_b + (size_t)wib * K;
  int* adelta = adelta_b + (size_t)wib * K;
  int* loc = loc_b + wib * 96;
  Vol V{I.send, rv ? I.recv : nullptr};
  // the walk's staged positions lie over the evaluation's arrays, its exact
  // sizes over the round's penalties (both rebuilt every round)
  WalkSmem& walk_s = *reinterpret_cast<WalkSmem*>(cnt_b);
  int* walk_dl = cnt_b + sizeof(WalkSmem) / sizeof(int);
  const float rC = __fdiv_rn(1.0f, Cf);
  int* walk_sz = reinterpret_cast<int*>(penf_s);

  int round = 0;
  int heavy_round = 0;
  int vr = 0;   // validations (parity selects the words of changed decisions)
  unsigned long long tA = gtimer();
  for (int it = 0; it < passes; it++) {
    const bool logp = I.recs != nullptr && it == passes - 1;   // decision records of the last pass
    int pos = 0;
    int W = min(nwarps, B.wmax);
    int hidx = 0, midx = 0;
    bool pass_start = true;
    bool prev_maxtouch = false;
    while (pos < B.npos) {
      const int par = round & 1;
      // ------------------------------------------------------------ round state
      for (int p = threadIdx.x; p < K; p += blockDim.x) {
        const int sz = lds(&I.part_sizes[p]);
        sizes_s[p] = sz;
        penf_s[p] = pen_of(sz, rC).x;
        if (metric == kTV) {
          // a part scanned in the last window takes its last scanner as marker
          // (block 0 stores it; the others read only parts not scanned there)
          const unsigned long long ml = lds(&B.mlast[p]);
          if (round > 0 && (int)(ml >> 32) == round) {
            const int mv = __ldg(&B.porder[(int)(ml & 0xffffffffu)]);
            marker_s[p] = mv;
            if (blockIdx.x == 0) I.marker[p] = mv;
          } else {
            marker_s[p] = lds(&I.marker[p]);
          }
        }
        if (vol) vol_s[p] = lds(&I.send[p]) + (rv ? lds(&I.recv[p]) : 0);
      }
      __syncthreads();
      block_min_part(sizes_s, K, uscr, &s_minpart, &s_minsize, &s_second);
      if (vol) {
        // Max-volume parts.  MSV rescans after every move (MGV/partition.cpp:
        // 453-472); MSRV rescans only when an old max part changed, against the
        // old maximum, appending to its list (MSRV/partition.cpp:486-513).
        int mx = -2147483647 - 1;
        for (int p = threadIdx.x; p < K; p += blockDim.x) mx = max(mx, vol_s[p]);
        mx = warp_max(mx);
        if (lane == 0) iscr[wib] = mx;
        __syncthreads();
        mx = iscr[0];
        for (int x = 1; x < kSWarps; x++) mx = max(mx, iscr[x]);
        __syncthreads();
        if (!rv || pass_start) {
          int local = 0;
          for (int p = threadIdx.x; p < K; p += blockDim.x) {
            const bool m = vol_s[p] == mx;
            mark_s[p] = m ? 1 : -1;
            local += m;
          }
          local = warp_sum(local);
          if (lane == 0) iscr[wib] = local;
          __syncthreads();
          if (threadIdx.x == 0) {
            int c = 0;
            for (int x = 0; x < kSWarps; x++) c += iscr[x];
            s_maxv = mx;
            s_cc = 1;
            s_count = c;
          }
          __syncthreads();
        } else if (prev_maxtouch) {
          bool changed = false;
          for (int p = threadIdx.x; p < K; p += blockDim.x)
            if (mark_s[p] == s_cc && vol_s[p] != s_maxv) changed = true;
          changed = __syncthreads_or(changed);
          if (changed && mx >= s_maxv) {
            const int ncc = mx > s_maxv ? s_cc + 1 : s_cc;
            int local = 0;
            for (int p = threadIdx.x; p < K; p += blockDim.x)
              if (vol_s[p] == mx) { mark_s[p] = ncc; local++; }
            local = warp_sum(local);
            if (lane == 0) iscr[wib] = local;
            __syncthreads();
            if (threadIdx.x == 0) {
              int c = 0;
              for (int x = 0; x < kSWarps; x++) c += iscr[x];
              s_count = (mx > s_maxv ? 0 : s_count) + c;
              s_maxv = mx;
              s_cc = ncc;
              if (s_count > K) dev_fail(I.status, kDevErrUnsupported);  // the reference overruns max_parts
            }
            __syncthreads();
          }
        }
      }
      __syncthreads();
      const RoundCtx R{sizes_s, penf_s, marker_s, vol_s, mark_s, s_minpart, s_minsize, s_second, s_maxv, s_cc, Cf};
      if (blockIdx.x == 0 && threadIdx.x == 0) B.stats[20] += gtimer() - tA;
      pass_start = false;
      prev_maxtouch = false;
      hidx = seek_pos(B.heavy_pos, B.nheavy, hidx, pos);
      midx = seek_pos(B.mid_pos, B.nmid, midx, pos);

      // ================================================================= round
      // A window holds up to gmax whole-grid vertices and ends before the next
      // one.
      int end_w = min(pos + W, B.npos);
      if (hidx + B.gmax < B.nheavy) end_w = min(end_w, (int)__ldg(&B.heavy_pos[hidx + B.gmax]));
      const int ns = min(B.gmax, seek_pos(B.heavy_pos, B.nheavy, hidx, end_w) - hidx);
      const int span = end_w - pos;
      // (a short window fills the first CTAs' warps: spread over all CTAs it kept
      // those of the medium vertices waiting, MSRV 51.6 -> 59 us per window)
      const int q = (span + nwarps - 1) / nwarps;
      const int cta_o0 = min((int)blockIdx.x * kSWarps * q, span);
      const int z0 = pos + min(gw * q, span);
      const int z1 = min(z0 + q, end_w);
      const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gthreads = gridDim.x * blockDim.x;
      const int hp = heavy_round & 1;   // whole-grid tallies, double-buffered by parity
      // slot j of this parity: K entries at hslot(j), 8 words of hmisc at hmslot(j)
      auto hslot = [&](int j) { return ((size_t)hp * kMaxGridVerts + j) * K; };
      auto hmslot = [&](int j) { return (hp * kMaxGridVerts + j) * 8; };
      const unsigned long long tR = gtimer();
      if ((int)threadIdx.x < ns) {
        const int z = __ldg(&B.heavy_pos[hidx + threadIdx.x]);
        const int v = __ldg(&B.porder[z]);
        const uint32_t b = __ldg(&I.vptr[v]);
        s_gz[threadIdx.x] = z;
        s_gv[threadIdx.x] = v;
        s_go[threadIdx.x] = lds(&I.part_vec[v]);
        s_gb[threadIdx.x] = b;
        s_gd[threadIdx.x] = (int)(__ldg(&I.vptr[v + 1]) - b);
      }
      __syncthreads();
      // ---- A1: tally slices of the whole-grid vertices by their teams of CTAs,
      // one set of arrays per CTA
      const int mend = seek_pos(B.mid_pos, B.nmid, midx, end_w);
      if (wib == 0 && ns)
        team_split(ns, s_gd, gridDim.x, (span + kSWarps * q - 1) / (kSWarps * q), mend - midx, s_t0, s_t1);
      __syncthreads();
      auto in_team = [&](int j) { return (int)blockIdx.x >= s_t0[j] && (int)blockIdx.x < s_t1[j]; };
      auto leads = [&](int j) { return (int)blockIdx.x == s_t0[j]; };
      // this CTA's share of vertex j's nets; its thread's first net and the step
      auto team_nets = [&](int j, int* c0, int* c1) {
        net_range(s_gd[j], (int)blockIdx.x - s_t0[j], s_t1[j] - s_t0[j], c0, c1);
      };
      auto team_tid = [&](int j) { return ((int)blockIdx.x - s_t0[j]) * (int)blockDim.x + (int)threadIdx.x; };
      auto team_threads = [&](int j) { return (s_t1[j] - s_t0[j]) * (int)blockDim.x; };
      for (int j = 0; j < ns; j++) {
        if (!in_team(j)) continue;
        const int own_s = s_go[j];
        const uint32_t base_s = s_gb[j];
        int* hcnt = B.hcnt + hslot(j);
        unsigned long long* hfirst = B.hfirst + hslot(j);
        int c0, c1;
        team_nets(j, &c0, &c1);
        // in pieces whose sighting keys fit 32 bits (all but always one)
        const int piece = key_nets(sb);
        for (int a0 = c0, a1 = c0; a0 < c1; a0 = a1) {
          a1 = a0 + min(piece, c1 - a0);
          for (int p = threadIdx.x; p < K; p += blockDim.x) { cnt_b[p] = 0; first_b[p] = ~0u; }
          __syncthreads();
          int own1 = 0, n0, n1;
          net_range(a1 - a0, wib, kSWarps, &n0, &n1);
          own1 = tally_range<true>(I, own_s, base_s, a0 + n0, a0 + n1, a0, sb, cnt_b, first_b);
          own1 = warp_sum(own1);
          if (lane == 0 && own1) atomicAdd(&B.hmisc[hmslot(j)], own1);
          __syncthreads();
          for (int p = threadIdx.x; p < K; p += blockDim.x) {
            if (cnt_b[p]) {
              atomicAdd(&hcnt[p], cnt_b[p]);
              atomicMin(&hfirst[p], wide_key(first_b[p], sb, a0));
            }
          }
          __syncthreads();   // the arrays serve the next piece and the evaluations below
        }
      }
      if (kTimingStats && ns && threadIdx.x == 0) atomicMax(&B.stats[38], gtimer() - tR);
      // ---- A: evaluate
      const long long cA = clock64();
      long long cV = 0;
      int nV = 0;
      for (int z = z0; z < z1; z++) {
        const int o = z - pos;
        const int v = __ldg(&B.porder[z]);
        const uint32_t base = __ldg(&I.vptr[v]);
        const int deg = (int)(__ldg(&I.vptr[v + 1]) - base);
        if (__ldg(&B.vclass[v]) != 0) continue;   // medium vertex: evaluated by the whole CTA below
        const long long cz = clock64();
        const int own = lds(&I.part_vec[v]);
        for (int p = lane; p < K; p += 32) { cnt[p] = 0; first[p] = ~0u; }
        __syncwarp();
        int c1 = 0;
        c1 = tally_range<true>(I, own, base, 0, deg, 0, sb, cnt, first);
        __syncwarp();
        c1 = warp_sum(c1);
        const long long cT = clock64();
        bool special;
        int slack;
        // candidates (part, count, first sighting) for an exact re-check of the
        // decision if the part sizes drift beyond its slack; TV's scanned parts
        const int d = ldg_decide(I, R, cnt, first, sb, metric, v, own, z == pos, B.cand + (size_t)o * K,
                                 &B.ncand[o], metric == kTV ? B.scan + (size_t)o * words : nullptr, &special, &slack);
        const long long cD = clock64();
        // The accept outcome of a vertex without nets does not depend on the
        // destination (all gains and losses are zero).
        const bool iso = deg == 0;
        bool mover = false, mt = false, good = metric == kTV;
        int vs = kBig, vdd = 0, nt = 0;
        if (metric == kTV) {
          if (d != own) {
            mover = c1 >= deg - cnt[d];
            // the records also serve the validation (own's slot per net)
            locate_all(I, B, metric, v, own, d, base, deg, 0, 1, loc, nullptr, nullptr, nullptr);
          }
        } else if (d != own || iso) {
          for (int p = lane; p < K; p += 32) { gains[p] = 0; losses[p] = 0; adelta[p] = 0; }
          __syncwarp();
          if (d != own) locate_all(I, B, metric, v, own, d, base, deg, 0, 1, loc, gains, losses, adelta);
          __syncwarp();
          AcceptPart a = accept_partial(R, gains, losses, adelta, K, rv, lane, 32);
          const bool fM = __any_sync(kAll, a.failM);
          const bool fN = __any_sync(kAll, a.failN);
          accept_final(fM, fN, warp_max(a.fsl), warp_min(a.msl), &good, &vs);
          mover = good && d != own;
          mt = mover && __any_sync(kAll, a.mt);
          vdd = warp_max(a.vd);
          if (d != own && deg) nt = store_terms(B, o, K, gains, losses, adelta);
          else if (lane == 0) B.vn[o] = 0;
        }
        __syncwarp();
        if (logp) {
          // decision record: TV's leave gain / arrival loss (TV/partition.cpp:355-378),
          // MSV / MSRV's gain and loss vectors summed (MGV/partition.cpp:294-337)
          int rg = 0, rl = 0;
          if (d != own) {
            if (metric == kTV) {
              rg = c1;
              rl = deg - cnt[d];
            } else {
              for (int p = lane; p < K; p += 32) { rg += gains[p]; rl += losses[p]; }
              rg = warp_sum(rg);
              rl = warp_sum(rl);
            }
          }
          if (lane == 0) { B.rgain[o] = rg; B.rloss[o] = rl; }
        }
        if (mover) {
          claim_nets(I, B, vol, z, own, d, base, deg, lane, 32, par);
          if (lane == 0) {
            if (mt) atomicMin(&B.ctl[2 + par], z);
            list_mover(I, B, par, o, __ldg(&I.w[v]), (own << 16) | d, nt);
          }
        }
        if (lane == 0) {
          B.dec[o] = (own << 16) | d;   // own read now: part_vec changes in the commit phase
          B.flag[o] = (unsigned char)((mover ? 1 | kListed : 0) | (special ? 2 : 0) | (iso ? 8 : 0) | (good ? 16 : 0));
          B.slack[o] = slack;
          B.vslack[o] = vs;
          B.wt[o] = __ldg(&I.w[v]);
          B.acc[o] = c1 - deg;
          B.vd[o] = mover ? vdd : 0;
        }
        if (kTimingStats && lane == 0) {
          atomicAdd(&B.stats[41], (unsigned long long)(cT - cz));
          atomicAdd(&B.stats[42], (unsigned long long)(cD - cT));
          atomicAdd(&B.stats[43], (unsigned long long)(clock64() - cD));
        }
        cV += clock64() - cz;
        nV++;
        __syncwarp();
      }
      if (kTimingStats && lane == 0 && nV) {
        // per-window statistics (cycles): slowest warp, and all light evaluations
        atomicMax(&B.stats[22], (unsigned long long)(clock64() - cA));
        atomicAdd(&B.stats[25], (unsigned long long)cV);
        atomicAdd(&B.stats[26], (unsigned long long)nV);
      }
      // medium vertices of the window: one CTA each, dealt out from the end of
      // the grid (a CTA with several among its own positions held the window up)
      __syncthreads();
      const long long cM = clock64();
      const int mi0 = midx + (int)(gridDim.x - 1 - blockIdx.x);
      for (int mi = mi0; mi < mend; mi += gridDim.x)
        cta_eval_ldg(I, B, R, metric, __ldg(&B.mid_pos[mi]), pos, par, sb, cnt_b, first_b, gains_b, losses_b,
                     adelta_b, iscr, loc_b, logp);
      __syncthreads();
      if (kTimingStats && threadIdx.x == 0) {
        const long long dm = clock64() - cM;
        if (dm > 2000) atomicMax(&B.stats[24], (unsigned long long)dm);
        atomicMax(&B.stats[36], gtimer() - tR);
      }
      if (ns) {
        if (!grid_barrier(B.bar, I.status)) return;
        const unsigned long long tG = gtimer();
        // ---- A2: decisions of the whole-grid vertices, taken in every CTA of their
        // teams from the global tallies (each is first of the window or not, like
        // any position), then their locate / gain-loss slices
        for (int j = 0; j < ns; j++) {
          if (!in_team(j)) continue;
          const size_t hs = hslot(j);
          const int zs = s_gz[j], vsup = s_gv[j], own_s = s_go[j];
          for (int p = threadIdx.x; p < K; p += blockDim.x) {
            cnt_b[p] = lds(&B.hcnt[hs + p]);
            first64_b[p] = lds(&B.hfirst[hs + p]);
            if (vol) { gains_b[p] = 0; losses_b[p] = 0; adelta_b[p] = 0; }
          }
          __syncthreads();
          if (wib == 0) {
            bool special;
            int slack;
            // the first CTA keeps the candidates for an exact re-check, TV's scanned parts
            const int os = zs - pos;
            const bool b0 = leads(j);
            const int d = ldg_decide(I, R, cnt_b, first64_b, sb, metric, vsup, own_s, zs == pos,
                                     b0 ? B.cand + (size_t)os * K : nullptr, b0 ? &B.ncand[os] : nullptr,
                                     b0 && metric == kTV ? B.scan + (size_t)os * words : nullptr, &special, &slack);
            if (lane == 0) {
              s_gdec[j] = d;
              s_gspec[j] = special ? 1 : 0;
              s_gslk[j] = slack;
              s_gcnt[j] = cnt_b[d];
            }
          }
          __syncthreads();
          const int d = s_gdec[j];
          if (d == own_s) continue;   // records for every decision that moves (the validation reads own's slots)
          int c0, c1, n0, n1;
          team_nets(j, &c0, &c1);
          net_range(c1 - c0, wib, kSWarps, &n0, &n1);
          locate_range(I, B, metric, vsup, own_s, d, s_gb[j], c0 + n0, c0 + n1, loc, gains_b, losses_b, adelta_b);
          __syncthreads();
          if (vol) {
            for (int p = threadIdx.x; p < K; p += blockDim.x) {
              if (gains_b[p]) atomicAdd(&B.hgain[hs + p], gains_b[p]);
              if (losses_b[p]) atomicAdd(&B.hloss[hs + p], losses_b[p]);
              if (adelta_b[p]) atomicAdd(&B.hadelta[hs + p], adelta_b[p]);
            }
            __syncthreads();   // the arrays serve the next vertex
          }
        }
        if (!grid_barrier(B.bar, I.status)) return;
        // ---- A3: accept tests (MSV / MSRV) in every CTA of the teams, claims, the records
        for (int j = 0; j < ns; j++) {
          if (!in_team(j)) continue;
          const size_t hs = hslot(j);
          const int zs = s_gz[j], vsup = s_gv[j], own_s = s_go[j], deg_s = s_gd[j], d = s_gdec[j];
          const uint32_t base_s = s_gb[j];
          const int os = zs - pos;
          const bool need = d != own_s &&
                            (metric == kTV ? lds(&B.hmisc[hmslot(j)]) >= deg_s - s_gcnt[j] : true);
          bool mover = metric == kTV && need, mt = false;
          int vs = kBig, vdd = 0, nt = 0;
          int rg = 0, rl = 0;   // decision record (with the log on)
          if (metric == kTV && d != own_s) {
            rg = lds(&B.hmisc[hmslot(j)]);
            rl = deg_s - s_gcnt[j];
          }
          if (vol && need) {
            for (int p = threadIdx.x; p < K; p += blockDim.x) {
              gains_b[p] = lds(&B.hgain[hs + p]);
              losses_b[p] = lds(&B.hloss[hs + p]);
              adelta_b[p] = lds(&B.hadelta[hs + p]);
            }
            __syncthreads();
            const AcceptPart a = accept_partial(R, gains_b, losses_b, adelta_b, K, rv, threadIdx.x, blockDim.x);
            const bool fM = __syncthreads_or(a.failM);
            const bool fN = __syncthreads_or(a.failN);
            const bool amt = __syncthreads_or(a.mt);
            const int fsl = block_reduce_max(a.fsl, iscr);
            const int msl = block_reduce_min(a.msl, iscr);
            vdd = block_reduce_max(a.vd, iscr);
            if (leads(j) && wib == 0) nt = store_terms(B, os, K, gains_b, losses_b, adelta_b);
            bool good;
            accept_final(fM, fN, fsl, msl, &good, &vs);
            mover = good;
            mt = mover && amt;
            if (logp) {
              int g = 0, l = 0;
              for (int p = threadIdx.x; p < K; p += blockDim.x) { g += gains_b[p]; l += losses_b[p]; }
              rg = block_reduce_sum(g, iscr);
              rl = block_reduce_sum(l, iscr);
            }
          }
          if (mover) claim_nets(I, B, vol, zs, own_s, d, base_s, deg_s, team_tid(j), team_threads(j), par);
          if (leads(j) && threadIdx.x == 0) {
            if (logp) { B.rgain[os] = rg; B.rloss[os] = rl; }
            B.dec[os] = (own_s << 16) | d;
            B.flag[os] = (unsigned char)((mover ? 1 | kListed : 0) | (s_gspec[j] ? 2 : 0) | 4 | (!vol || mover ? 16 : 0));
            B.slack[os] = s_gslk[j];
            B.vslack[os] = vs;
            B.wt[os] = __ldg(&I.w[vsup]);
            B.acc[os] = lds(&B.hmisc[hmslot(j)]) - deg_s;
            B.vd[os] = mover ? vdd : 0;
            if (mover && mt) atomicMin(&B.ctl[2 + par], zs);
            if (mover) list_mover(I, B, par, os, __ldg(&I.w[vsup]), (own_s << 16) | d, nt);
          }
          __syncthreads();
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) B.stats[33] += gtimer() - tG;
      }
      if (!grid_barrier(B.bar, I.status)) return;
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned long long tE = gtimer();
        B.stats[16] += tE - tA;
        tA = tE;
        B.stats[21] += B.stats[22];   // no CTA writes these again before the next phase A
        B.stats[22] = 0;
        B.stats[23] += B.stats[24];
        B.stats[24] = 0;
      }
      // ---- B: validate the positions [zfrom, zto): the lists (conflicts), the
      // volumes and, with sizes, the part sizes (the decision taken again where
      // they drifted beyond its slack).  The first position that an earlier
      // one invalidates lowers *cut_w, the first whose decision the exact sizes
      // change *flip_w (dfix holds its new decision, flag bit 7); with sizes, rel
      // receives the drift it tolerates beyond the window's movers as they are
      // (-2: its decision changes).
      int* const cut_w = &B.ctl[4 + par];
      // (the evaluation's arrays are free here)
      int* dsz_cta = gains_b;
      uint32_t* vbits = reinterpret_cast<uint32_t*>(losses_b);   // max parts, words per state
      int* dv_cta = adelta_b;                                    // volume changes before this CTA's positions,
      int* vol_x = adelta_b + K;                                 //   volumes at the last change of the max parts,
      int* dv_big = adelta_b + 2 * K;                            //   changes before a CTA's or the grid's vertex
      // the movers' terms (offset << 12 | part, change): behind the evaluation's
      // arrays where the walk's words reach beyond them, or in the half of the
      // sighting keys that only whole-grid vertices use; 1600 at least
      const int tail = (int)(sizeof(WalkSmem) / 8 + K / 2) - (int)((adelta_b + (size_t)K * kSWarps - cnt_b + 1) / 2) - 1;
      const bool behind = tail > K * (kSWarps / 2);
      int2* const stage = reinterpret_cast<int2*>(behind ? adelta_b + (((size_t)K * kSWarps + 3) & ~size_t(3))
                                                         : (int*)first_b + (((size_t)K * kSWarps + 1) & ~size_t(1)));
      const int stage_cap = behind ? tail - 2 : K * (kSWarps / 2);
      // the size changes (in dsz) and, with dv, the volume changes of the
      // window's movers before offset o (listed terms only: no position beyond the
      // first mover without them is taken); every thread of the CTA
      auto moved_before = [&](int o, int* dsz, int* dv) {
        for (int p = threadIdx.x; p < K; p += blockDim.x) {
          dsz[p] = 0;
          if (dv) dv[p] = 0;
        }
        __syncthreads();
        const int nm = lds(&B.mcnt[par]);
        for (int i = threadIdx.x; i < nm; i += blockDim.x) {
          const int4 m = lds(&B.mlist[i]);
          if (m.x >= o) continue;
          if (m.y != 0) {
            atomicAdd(&dsz[m.z & 0xffff], m.y);
            atomicAdd(&dsz[m.z >> 16], -m.y);
          }
          if (dv)
            for (int t = 0; t < m.w; t++) {
              const int ad = __ldcg(&B.vterm[(size_t)m.x * kVolTerms + t].y);
              if (ad) atomicAdd(&dv[(int)__ldcg(&B.vpart[(size_t)m.x * kVolTerms + t])], ad);
            }
        }
        __syncthreads();
      };
      // The max-volume parts between the window's movers (vs_s, vbits): applies
      // the movers in order up to each one that changes the set.  MSV scans anew
      // after every move (MGV/partition.cpp:453-472): only a move that touches a
      // max part changes it, as no other part reaches the maximum.  MSRV scans
      // when a listed part is off the old maximum (MSRV/partition.cpp:486-513),
      // after any move once that holds.  Every CTA does it for itself.
      auto vol_states = [&]() {
        const int nm = lds(&B.mcnt[par]);
        if (threadIdx.x == 0) {
          vs_s.n = 0;
          vs_s.over = kNone;
          vs_s.end = kNone;
          vs_s.maxv[0] = s_maxv;
          vs_s.count[0] = s_count;
        }
        for (int w = wib; w < words; w += kSWarps) {
          const int p = w * 32 + lane;
          const unsigned m = __ballot_sync(kAll, p < K && mark_s[p] == s_cc);
          if (lane == 0) vbits[w] = m;
        }
        for (int p = threadIdx.x; p < K; p += blockDim.x) vol_x[p] = vol_s[p];
        __syncthreads();
        int ovm = kNone, nmk = 0, off = 0;
        for (int i = threadIdx.x; i < nm; i += blockDim.x) {
          const int4 m = lds(&B.mlist[i]);
          if (m.w < 0) ovm = min(ovm, m.x);
        }
        if (ovm != kNone) atomicMin(&vs_s.over, ovm);
        for (int w = 0; w < words; w++) nmk += __popc(vbits[w]);
        if (threadIdx.x == 0) vs_s.nm[0] = nmk;
        if (rv)
          for (int p = threadIdx.x; p < K; p += blockDim.x)
            off |= mark_s[p] == s_cc && vol_s[p] != s_maxv;
        off = __syncthreads_or(off);
        if (lds(&B.ctl[2 + par]) == kNone && !off) return;   // no mover touches a max part
        // the movers' terms, unordered (half the window at a time where they do
        // not fit)
        int lim = min(vs_s.over, span);
        while (true) {
          if (threadIdx.x == 0) vs_s.ne = 0;
          __syncthreads();
          for (int i = threadIdx.x; i < nm; i += blockDim.x) {
            const int4 m = lds(&B.mlist[i]);
            if (m.x >= lim || m.w <= 0 || !(lds(&B.flag[m.x]) & 1)) continue;
            const int at = atomicAdd(&vs_s.ne, m.w);
            for (int t = 0; t < m.w && at + t < stage_cap; t++)
              stage[at + t] = make_int2((m.x << 12) | (int)__ldcg(&B.vpart[(size_t)m.x * kVolTerms + t]),
                                        __ldcg(&B.vterm[(size_t)m.x * kVolTerms + t].y));
          }
          __syncthreads();
          if (vs_s.ne <= stage_cap) break;
          lim = max(1, lim / 2);
          if (threadIdx.x == 0) vs_s.end = lim;
          __syncthreads();
        }
        const int ne = vs_s.ne;
        if (threadIdx.x == 0) {
          vs_s.next = kNone;
          vs_s.m2 = -2147483647 - 1;
          vs_s.chg = vs_s.add = vs_s.off = 0;
        }
        __syncthreads();
        int last = -1;
        for (int x = 0;; x++) {
          const uint32_t* bits = vbits + x * words;
          auto marked = [&](int p) { return ((bits[p >> 5] >> (p & 31)) & 1u) != 0; };
          int nx = kNone;
          for (int i = threadIdx.x; i < ne; i += blockDim.x) {
            const int2 t = stage[i];
            const int o = t.x >> 12;
            if (o > last && o < nx && (off || (t.y != 0 && marked(t.x & 0xfff)))) nx = o;
          }
          nx = warp_min(nx);
          if (lane == 0 && nx != kNone) atomicMin(&vs_s.next, nx);
          __syncthreads();
          nx = vs_s.next;
          if (nx == kNone) break;
          if (x == kVolEvents) {
            if (threadIdx.x == 0) vs_s.end = min(vs_s.end, nx);
            break;
          }
          for (int i = threadIdx.x; i < ne; i += blockDim.x) {
            const int2 t = stage[i];
            if ((t.x >> 12) > last && (t.x >> 12) <= nx && t.y) atomicAdd(&vol_x[t.x & 0xfff], t.y);
          }
          __syncthreads();
          last = nx;
          if (threadIdx.x == 0) {
            vs_s.next = kNone;
            vs_s.add = vs_s.off = vs_s.nm[x + 1] = 0;
          }
          const int mv0 = vs_s.maxv[x];
          int m2 = -2147483647 - 1;
          bool chg = !rv;
          for (int p = threadIdx.x; p < K; p += blockDim.x) {
            m2 = max(m2, vol_x[p]);
            if (marked(p) && vol_x[p] != mv0) chg = true;
          }
          m2 = warp_max(m2);
          chg = __any_sync(kAll, chg);
          if (lane == 0) {
            atomicMax(&vs_s.m2, m2);
            if (chg) vs_s.chg = 1;
          }
          __syncthreads();
          m2 = vs_s.m2;
          chg = vs_s.chg != 0;
          const bool fresh = !rv || (chg && m2 > mv0), more = rv && chg && m2 == mv0;
          const int mv1 = fresh ? m2 : mv0;
          for (int w = wib; w < words; w += kSWarps) {
            const int p = w * 32 + lane;
            const unsigned m = __ballot_sync(kAll, p < K && vol_x[p] == m2);
            const unsigned b = fresh ? m : more ? bits[w] | m : bits[w];
            const bool o2 = __any_sync(kAll, rv && p < K && ((b >> lane) & 1u) && vol_x[p] != mv1);
            if (lane == 0) {
              vbits[(x + 1) * words + w] = b;
              atomicAdd(&vs_s.nm[x + 1], __popc(b));
              atomicAdd(&vs_s.add, __popc(m));
              if (o2) vs_s.off = 1;
            }
          }
          __syncthreads();
          off = vs_s.off;
          if (threadIdx.x == 0) {
            vs_s.at[x] = nx;
            vs_s.maxv[x + 1] = mv1;
            vs_s.count[x + 1] = fresh ? vs_s.add : vs_s.count[x] + (more ? vs_s.add : 0);
            vs_s.n = x + 1;
            vs_s.m2 = -2147483647 - 1;
            vs_s.chg = 0;
          }
        }
        __syncthreads();
      };
      auto validate = [&](int zfrom, int zto, bool sizes, int* flip_w, int* nflip_w) {
        const bool ov = lds(&B.ctab_over[par]) != 0;
        bool after = false;
        if (vol) {
          vol_states();
          // the window ends behind a mover without listed terms, and at a change
          // of the max parts beyond those kept
          if (blockIdx.x == 0 && threadIdx.x == 0) {
            if (vs_s.over != kNone) atomicMin(cut_w, ((pos + vs_s.over + 1) << 3) | 3);
            if (vs_s.end != kNone) atomicMin(cut_w, ((pos + vs_s.end) << 3) | 4);
          }
        }
        auto vol_state = [&](int o) {   // of the max parts before offset o
          int x = 0;
          while (x < vs_s.n && vs_s.at[x] < o) x++;
          return x;
        };
        if (sizes || vol) {
          // the movers before this warp's first position
          moved_before(cta_o0, dsz_cta, vol ? dv_cta : nullptr);
          long long Vw = 0;
          long long Dw = 0;
          if (z0 < z1) {
            int D0 = 0, wi = 0, vi = 0;
            for (int p = lane; p < K; p += 32) D0 = max(D0, abs(dsz_cta[p]));
            for (int o = cta_o0 + lane; o < z0 - pos; o += 32) {
              if (lds(&B.flag[o]) & 1) wi += lds(&B.wt[o]);
              if (vol) vi += lds(&B.vd[o]);
            }
            Dw = (long long)warp_max(D0) + (unsigned)warp_sum(wi);
            if (vol) {
              int V0 = 0;
              for (int p = lane; p < K; p += 32) V0 = max(V0, abs(dv_cta[p]));
              Vw = (long long)warp_max(V0) + warp_sum(vi);
            }
          }
          for (int z = z0; z < min(z1, zto); z++) {
            const int o = z - pos;
            // the position's words in one round of independent loads
            const int wz = lds(&B.wt[o]), vz = lds(&B.vd[o]);
            const int fl = lds(&B.flag[o]);
            const int slk = lds(&B.slack[o]), vslk = lds(&B.vslack[o]);
            const int pk = lds(&B.dec[o]);
            const int v = __ldg(&B.porder[z]);
            if (z >= zfrom && !(fl & 4)) {      // the others: a CTA or the grid, below
              const uint32_t base = __ldg(&I.vptr[v]);
              const int deg = (int)(__ldg(&I.vptr[v + 1]) - base);
              const int own = pk >> 16;
              if (sizes && (Dw > max(slk, 0) || (fl & 32))) {
                // the exact sizes here: this CTA's movers before z on top of dsz_cta
                for (int p = lane; p < K; p += 32) cnt[p] = sizes_s[p] + dsz_cta[p];
                __syncwarp();
                for (int o2 = cta_o0 + lane; o2 < o; o2 += 32)
                  if (lds(&B.flag[o2]) & 1) {
                    const int w2 = lds(&B.wt[o2]), pk2 = lds(&B.dec[o2]);
                    atomicAdd(&cnt[pk2 & 0xffff], w2);
                    atomicAdd(&cnt[pk2 >> 16], -w2);
                  }
                __syncwarp();
                int ns1;
                const int d2 = recheck(I, rC, Cf, cnt, lds(&B.ncand[o]), B.cand + (size_t)o * K, metric == kTV, own, &ns1);
                const bool flip = d2 != (pk & 0xffff);
                if (lane == 0) {
                  if (flip) {
                    atomicMin(flip_w, (z << 3) | 2);
                    atomicAdd(nflip_w, 1);
                    B.dfix[o] = d2;
                    B.flag[o] = (unsigned char)(fl | 128);
                  } else if (fl & 128) {
                    B.flag[o] = (unsigned char)(fl & 127);
                  }
                  B.rel[o] = flip ? -2 : ns1;
                }
              } else if (sizes && lane == 0) {
                B.rel[o] = max(slk, 0) - (int)Dw;
                if (fl & 128) B.flag[o] = (unsigned char)(fl & 127);
              }
              // the volumes enter only the accept test of a vertex whose decision
              // leaves its part (MSRV/partition.cpp:308-400, MGV/partition.cpp:
              // 292-362): taken again where the max parts changed or the others
              // drifted beyond what it tolerates
              int why = ((fl & 2) && z != pos) ? 1 : 0;
              if (vol && !why && (pk & 0xffff) != own) {
                const int x = vol_state(o);
                if (x || Vw > max(vslk, 0)) {
                  const int nt = lds(&B.vn[o]);
                  int* vx = (int*)first;
                  const bool good = nt >= 0 && accept_terms(
                      B, o, nt, K, rv, vbits + x * words, vs_s.nm[x], vs_s.maxv[x],
                      [&]() {
                        for (int p = lane; p < K; p += 32) vx[p] = vol_s[p] + dv_cta[p];
                        __syncwarp();
                        for (int o2 = cta_o0; o2 < o; o2++)
                          if (lds(&B.flag[o2]) & 1) {
                            const int n2 = lds(&B.vn[o2]);
                            for (int t = lane; t < n2; t += 32) {
                              const int ad = __ldcg(&B.vterm[(size_t)o2 * kVolTerms + t].y);
                              if (ad) atomicAdd(&vx[(int)__ldcg(&B.vpart[(size_t)o2 * kVolTerms + t])], ad);
                            }
                          }
                        __syncwarp();
                      },
                      [&](int p) { return vx[p]; });
                  if (nt < 0 || good != ((fl & 1) != 0)) why = nt < 0 && x ? 4 : 3;
                  __syncwarp();
                }
              }
              if (!why) {
                const int c = conflicts(I, B, vol, z, own, (pk & 0xffff) != own, fl & 1, base, deg, lane, 32, ov, &after);
                const int c5 = __any_sync(kAll, c == 5), c6 = __any_sync(kAll, c == 6);
                why = c5 ? 5 : c6 ? 6 : 0;
              }
              if (why) {
                if (lane == 0) atomicMin(cut_w, (z << 3) | why);   // position, then cut reason
                break;
              }
            }
            if (fl & 1) Dw += wz;
            if (vol) Vw += vz;
          }
        } else {
          for (int z = max(z0, zfrom); z < min(z1, zto); z++) {   // TV, sizes known: the conflicts alone
            const int o = z - pos;
            const int fl = lds(&B.flag[o]), pk = lds(&B.dec[o]);
            if (fl & 4) continue;
            const int v = __ldg(&B.porder[z]);
            const uint32_t base = __ldg(&I.vptr[v]);
            const int deg = (int)(__ldg(&I.vptr[v + 1]) - base);
            const int own = pk >> 16;
            int why = ((fl & 2) && z != pos) ? 1 : 0;
            if (!why) {
              const int c = conflicts(I, B, vol, z, own, (pk & 0xffff) != own, fl & 1, base, deg, lane, 32, ov, &after);
              const int c5 = __any_sync(kAll, c == 5), c6 = __any_sync(kAll, c == 6);
              why = c5 ? 5 : c6 ? 6 : 0;
            }
            if (why) {
              if (lane == 0) atomicMin(cut_w, (z << 3) | why);
              break;
            }
          }
        }
        // medium vertices by their CTAs, whole-grid vertices: their nets by every
        // thread, the rest by one CTA
        auto check_big = [&](int z, int k0, int kstep, bool rest, bool grid) {
          const int o = z - pos;
          const int fl = lds(&B.flag[o]), pk = lds(&B.dec[o]);
          const int own = pk >> 16;
          const bool leaves = (pk & 0xffff) != own;
          const int v = __ldg(&B.porder[z]);
          const uint32_t base = __ldg(&I.vptr[v]);
          const int deg = (int)(__ldg(&I.vptr[v + 1]) - base);
          int why = 0;
          if (rest) {
            why = ((fl & 2) && z != pos) ? 1 : 0;
            if (sizes || vol) {
              __syncthreads();   // dsz_cta and cnt_b are read
              moved_before(o, cnt_b, vol ? dv_big : nullptr);
              if (vol && !why && leaves && wib == 0) {
                const int x = vol_state(o);
                int V0 = 0;
                for (int p = lane; p < K; p += 32) V0 = max(V0, abs(dv_big[p]));
                if (x || warp_max(V0) > max(lds(&B.vslack[o]), 0)) {
                  const int nt = lds(&B.vn[o]);
                  const bool good = nt >= 0 && accept_terms(
                      B, o, nt, K, rv, vbits + x * words, vs_s.nm[x], vs_s.maxv[x], []() {},
                      [&](int p) { return vol_s[p] + dv_big[p]; });
                  // (only the first thread reports it, below)
                  if (nt < 0 || good != ((fl & 1) != 0)) why = nt < 0 && x ? 4 : 3;
                }
              }
              if (sizes && wib == 0) {
                int D0 = 0;
                for (int p = lane; p < K; p += 32) D0 = max(D0, abs(cnt_b[p]));
                D0 = warp_max(D0);
                const int slk = max(lds(&B.slack[o]), 0);
                if (D0 > slk || (fl & 32)) {
                  for (int p = lane; p < K; p += 32) cnt_b[p] += sizes_s[p];
                  __syncwarp();
                  int ns1;
                  const bool flip = recheck(I, rC, Cf, cnt_b, lds(&B.ncand[o]), B.cand + (size_t)o * K, metric == kTV,
                                            own, &ns1) != (pk & 0xffff);
                  if (lane == 0) {
                    if (flip) {
                      atomicMin(flip_w, (z << 3) | 2);
                      atomicAdd(nflip_w, kJacobiFlips + 1);   // the walk's
                    } else if (fl & 128) {
                      B.flag[o] = (unsigned char)(fl & 127);
                    }
                    B.rel[o] = flip ? -2 : ns1;
                  }
                } else if (lane == 0) {
                  B.rel[o] = slk - D0;
                  if (fl & 128) B.flag[o] = (unsigned char)(fl & 127);
                }
              }
              __syncthreads();
            }
          }
          if (!why || grid) {
            const int c = conflicts(I, B, vol, z, own, leaves, fl & 1, base, deg, k0, kstep, ov, &after);
            if (c) atomicMin(cut_w, (z << 3) | c);
          }
          if (why && threadIdx.x == 0) atomicMin(cut_w, (z << 3) | why);
        };
        __syncthreads();
        for (int mi = mi0; mi < mend; mi += gridDim.x) {
          const int z = __ldg(&B.mid_pos[mi]);
          if (z >= zto) break;
          if (z >= zfrom) check_big(z, threadIdx.x, blockDim.x, true, false);
        }
        for (int j = 0; j < ns; j++) {
          const int z = s_gz[j];
          if (z >= zto) break;
          if (z >= zfrom && in_team(j)) check_big(z, team_tid(j), team_threads(j), leads(j), true);
        }
        if (after) B.ctl[12 + par] = 1;
      };
      // ---- B: validate; while decisions change, take the changes and validate
      // again from the first one.  Long stretches with few changes take them all
      // at once, each as the exact sizes before it then were (the validation
      // finds what that leaves wrong); otherwise one CTA walks them in order.
      // Measured on the 1M-vertex Zipf workload under TV (windows of 1,500
      // positions, five changes each): 315 us of walk per window, 75 us so.
      if (metric == kTV) {   // the parts scanned by this CTA's positions, for the markers below
        const int ctan = min(kSWarps * q, span - cta_o0);
        for (int x = threadIdx.x; x < words; x += blockDim.x) cmask_s[x] = 0;
        __syncthreads();
        for (int x = threadIdx.x; x < ctan * words; x += blockDim.x)
          if (const uint32_t m = lds(&B.scan[(size_t)cta_o0 * words + x])) atomicOr(&cmask_s[x % words], m);
        __syncthreads();
        for (int x = threadIdx.x; x < words; x += blockDim.x) B.cmask[(size_t)blockIdx.x * words + x] = cmask_s[x];
      }
      int cutw, hard = kNone, fcut = kNone;
      bool sizes = true;
      for (int zf = pos, nfix = 0;; nfix++) {
        int* const flip_w = &B.ctl[6 + (vr & 1)];
        int* const nflip_w = &B.ctl[10 + (vr & 1)];
        validate(zf, hard == kNone ? end_w : min(hard >> 3, end_w), sizes, flip_w, nflip_w);
        if (!grid_barrier(B.bar, I.status)) return;
        cutw = min(lds(cut_w), fcut);   // (no fix writes cut_w: CTAs ahead may be in theirs already)
        if (hard != kNone && (hard >> 3) < end_w) cutw = min(cutw, hard);
        const int flipw = lds(flip_w), nflip = lds(nflip_w);
        if (blockIdx.x == 0 && threadIdx.x == 0) {   // the next validation's words
          B.ctl[6 + ((vr & 1) ^ 1)] = kNone;
          B.ctl[10 + ((vr & 1) ^ 1)] = 0;
        }
        vr++;
        if (rv && sizes && nflip > kWalkOverEvent && vs_s.n > 0) {
          fcut = min(fcut, ((pos + vs_s.at[0] + 1) << 3) | 4);
          cutw = min(cutw, fcut);
        }
        if (!sizes || (flipw >> 3) >= (cutw >> 3)) break;
        zf = flipw >> 3;
        const int zc = min(end_w, cutw >> 3);
        if (nfix == B.maxfix) {
          cutw = flipw;
          break;
        }
        const bool at_once = (nfix == 0 && nflip <= kJacobiFew) || (zc - zf > kJacobiSpan && nflip <= kJacobiFlips);
        if (!at_once) {
          const unsigned long long tW = gtimer();
          if (blockIdx.x == 0)
            walk_window<false>(I, B, sizes_s, Cf, metric == kTV, metric == kMSV, pos, zf, zc, lds(&B.mcnt[par]), walk_s,
                               walk_sz, walk_dl);
          if (!grid_barrier(B.bar, I.status)) return;
          hard = lds(&B.ctl[0]);
          if (blockIdx.x == 0 && threadIdx.x == 0) {
            B.stats[44] += lds(&B.ctl[1]);
            B.stats[45] += gtimer() - tW;
          }
        } else {
          hard = kNone;
          if (blockIdx.x == 0 && threadIdx.x == 0) B.stats[44] += nflip;
        }
        // the changed positions redone by their warps
        for (int z = max(z0, zf); z < min(z1, hard == kNone ? zc : min(zc, hard >> 3)); z++) {
          const int fl = lds(&B.flag[z - pos]);
          if ((fl & 132) == 128)
            fix_position(I, B, R, metric, z, z - pos, fl, par, loc, gains, losses, adelta, logp);
        }
        __syncthreads();
        for (int mi = mi0; mi < mend; mi += gridDim.x) {
          const int z = __ldg(&B.mid_pos[mi]);
          if (z >= (hard == kNone ? zc : min(zc, hard >> 3))) break;
          const int fl = z >= zf ? lds(&B.flag[z - pos]) : 0;
          __syncthreads();   // every thread has read the flag
          if (fl & 128) cta_fix(I, B, R, metric, z, z - pos, fl, par, loc_b, gains_b, losses_b, adelta_b, iscr, logp);
        }
        for (int j = 0; j < ns; j++) {   // a whole-grid vertex by the first CTA of its team
          const int z = s_gz[j];
          if (!leads(j) || z < zf || z >= (hard == kNone ? zc : min(zc, hard >> 3))) continue;
          const int fl = lds(&B.flag[z - pos]);
          __syncthreads();
          if (fl & 128) cta_fix(I, B, R, metric, z, z - pos, fl, par, loc_b, gains_b, losses_b, adelta_b, iscr, logp);
        }
        if (!grid_barrier(B.bar, I.status)) return;
        // a walk whose outcomes came as predicted leaves exact sizes; else the
        // validation takes the decisions again
        fcut = min(fcut, lds(&B.ctl[9]));
        sizes = at_once || lds(&B.ctl[8]) != kNone;
        if (sizes) hard = kNone;
      }
      // ---- C: commit every mover before the cut.
      const int cut = cutw == kNone ? end_w : min(cutw >> 3, end_w);
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned long long tB = gtimer();
        B.stats[0]++;
        const int why = cutw == kNone ? 0 : (cutw & 7);
        B.stats[why <= 5 ? 3 + why : 21 + why]++;   // 6, 7: slots 27, 28
        B.stats[9] += cut - pos;
        // per-window maxima over CTAs (no CTA writes these again before the next phase A)
        B.stats[32] += B.stats[36];
        B.stats[34] += B.stats[38];
        B.stats[36] = 0;
        B.stats[38] = 0;
        B.stats[17] += tB - tA;
        tA = tB;
      }
      if (cut <= pos) {             // no progress: inconsistent claims; stop (all CTAs agree)
        if (threadIdx.x == 0) dev_fail(I.status, kDevErrInvalid);
        return;
      }
      if (logp) {
        // decision records of this warp's committed positions
        for (int z = z0 + lane; z < min(z1, cut); z += 32) {
          const int o = z - pos;
          const int fl = lds(&B.flag[o]);
          I.recs[__ldg(&B.porder[z])] =
              make_int4(lds(&B.dec[o]) & 0xffff, lds(&B.rgain[o]), lds(&B.rloss[o]), fl & 1);
        }
      }
      // the committed movers' nets [k0, step): all of them, or (counts_first) the
      // count-only ones and, behind a barrier, those whose part set changes
      const bool counts_first = lds(&B.ctl[12 + par]) != 0;
      for (int i = gtid, n = min(lds(&B.ctl[14 + par]), B.rmax); i < n; i += gthreads) {
        const int4 x = lds(&B.rlist[i]);
        if (x.x < 0) continue;
        unclaim_net(B, x.x);
        ctab_clear(B, make_uint2((unsigned)x.y, (unsigned)x.z));
      }
      for (int ph = counts_first ? 1 : 0;; ph++) {
        auto commit_nets = [&](int v, int own, int d, uint32_t base, int deg, int k0, int kstep) {
          for (int k = k0; k < deg; k += kstep) {
            const uint32_t rc = lds(&B.rec[base + k]);
            if (ph == 0 || rec_setchange(rc, vol) == (ph == 2))
              commit_rec(I, v, own, d, (int)__ldg(&I.vnets[base + k]), rc, vol ? &V : nullptr);
          }
        };
        auto commit_vertex = [&](int v, int own, int d) {
          atomicAdd(&B.stats[2], 1ull);
          I.part_vec[v] = d;
          const int wv = __ldg(&I.w[v]);
          atomicAdd(&I.part_sizes[own], -wv);
          atomicAdd(&I.part_sizes[d], wv);
          atomicAdd((unsigned long long*)&I.moves[it], 1ull);
        };
        for (int z = z0; z < z1; z++) {
          const int o = z - pos;
          const int fl = lds(&B.flag[o]);
          if ((fl & 5) != 1) continue;   // a mover that a warp evaluated
          const int v = __ldg(&B.porder[z]);
          const int pk = lds(&B.dec[o]);
          const int own = pk >> 16, d = pk & 0xffff;
          const uint32_t base = __ldg(&I.vptr[v]);
          const int deg = (int)(__ldg(&I.vptr[v + 1]) - base);
          if (z < cut) {
            commit_nets(v, own, d, base, deg, lane, 32);
            if (ph != 1 && lane == 0) commit_vertex(v, own, d);
          }
          if (ph != 1) unclaim_nets(I, B, vol, base, deg, lane, 32);
        }
        for (int mi = mi0; mi < mend; mi += gridDim.x) {
          const int z = __ldg(&B.mid_pos[mi]);
          const int o = z - pos;
          const int fl = lds(&B.flag[o]);
          if (!(fl & 1)) continue;
          const int v = __ldg(&B.porder[z]);
          const int pk = lds(&B.dec[o]);
          const int own = pk >> 16, d = pk & 0xffff;
          const uint32_t base = __ldg(&I.vptr[v]);
          const int deg = (int)(__ldg(&I.vptr[v + 1]) - base);
          if (z < cut) {
            commit_nets(v, own, d, base, deg, threadIdx.x, blockDim.x);
            if (ph != 1 && threadIdx.x == 0) commit_vertex(v, own, d);
          }
          if (ph != 1) unclaim_nets(I, B, vol, base, deg, threadIdx.x, blockDim.x);
        }
        for (int j = 0; j < ns; j++) {
          // a whole-grid vertex, by its team
          if (!in_team(j)) continue;
          const int tt = team_tid(j), tn = team_threads(j);
          const int zs = s_gz[j], vsup = s_gv[j], own_s = s_go[j], deg_s = s_gd[j];
          const uint32_t base_s = s_gb[j];
          const int os = zs - pos;
          if (lds(&B.flag[os]) & 1) {
            const int d = lds(&B.dec[os]) & 0xffff;
            if (zs < cut) {
              commit_nets(vsup, own_s, d, base_s, deg_s, tt, tn);
              if (ph != 1 && tt == 0) commit_vertex(vsup, own_s, d);
            }
            if (ph != 1) unclaim_nets(I, B, vol, base_s, deg_s, tt, tn);
          }
        }
        if (ph != 1) break;
        if (!grid_barrier(B.bar, I.status)) return;
      }
      if (B.niso && (metric != kMSRV || logp)) {
        // Vertices without nets, weight 0 (positions hold only the others):
        // each takes the least-loaded part at its place in the visiting order
        // (TV: unless the clamps keep it home) and changes nothing a later
        // decision reads, so they are decided here, after the cut, from the
        // exact sizes between the committed positions (MSRV never moves them;
        // there they are walked only for the decision records).
        int* dsz = gains_b;   // the committed movers' size changes before this CTA's first position
        __syncthreads();
        moved_before(cta_o0, dsz, nullptr);
        const int zb = min(z1, cut);
        if (z0 < zb) {
          int* sz = cnt;   // this warp's sizes, at its current position
          for (int p = lane; p < K; p += 32) sz[p] = sizes_s[p] + dsz[p];
          __syncwarp();
          for (int o2 = cta_o0 + lane; o2 < z0 - pos; o2 += 32) {
            if (!(lds(&B.flag[o2]) & 1)) continue;
            const int w = lds(&B.wt[o2]);
            const int pk = lds(&B.dec[o2]);
            atomicAdd(&sz[pk & 0xffff], w);
            atomicAdd(&sz[pk >> 16], -w);
          }
          __syncwarp();
          int amin = -1;
          long long nmoved = 0;
          auto group = [&](int k0, int k1) {
            if (k0 >= k1) return;
            if (amin < 0) {
              unsigned long long mk = ~0ull;
              for (int p = lane; p < K; p += 32) {
                const unsigned long long key = ((unsigned long long)((unsigned)sz[p] ^ 0x80000000u) << 32) | (unsigned)p;
                mk = key < mk ? key : mk;
              }
              for (int off = 16; off; off >>= 1) {
                const unsigned long long x = __shfl_xor_sync(kAll, mk, off);
                mk = x < mk ? x : mk;
              }
              amin = (int)(mk & 0xffffffffu);
            }
            const int sa = sz[amin];
            const bool home = metric == kTV && (sa > I.max_pw || sa < I.min_pw);
            for (int k = k0 + lane; k < k1; k += 32) {
              const int v = __ldg(&B.iso_list[k]);
              const int own = lds(&I.part_vec[v]);
              const int d = home ? own : amin;
              const bool mv = d != own && metric != kMSRV;
              if (mv) {
                I.part_vec[v] = d;
                nmoved++;
              }
              if (logp) I.recs[v] = make_int4(d, 0, 0, mv ? 1 : 0);
            }
          };
          if (pos == 0 && gw == 0) group(0, __ldg(&B.iso_before[0]));   // before the pass's first position
          for (int z = z0; z < zb; z++) {
            const int o = z - pos;
            const int w = lds(&B.wt[o]);
            if (w != 0 && (lds(&B.flag[o]) & 1)) {
              __syncwarp();
              if (lane == 0) {
                const int pk = lds(&B.dec[o]);
                sz[pk & 0xffff] += w;
                sz[pk >> 16] -= w;
              }
              __syncwarp();
              amin = -1;
            }
            group(__ldg(&B.iso_before[z]), __ldg(&B.iso_before[z + 1]));
          }
          nmoved = warp_sum64(nmoved);
          if (lane == 0 && nmoved) {
            atomicAdd((unsigned long long*)&I.moves[it], (unsigned long long)nmoved);
            atomicAdd(&B.stats[2], (unsigned long long)nmoved);
          }
        }
        __syncthreads();
      }
      if (ns) {
        // the other parity's tallies are cleared for the next window with
        // whole-grid vertices
        const size_t ob = (size_t)(hp ^ 1) * kMaxGridVerts * K;
        for (int p = gtid; p < kMaxGridVerts * K; p += gthreads) {
          B.hcnt[ob + p] = 0;
          B.hfirst[ob + p] = ~0ull;
          B.hgain[ob + p] = 0;
          B.hloss[ob + p] = 0;
          B.hadelta[ob + p] = 0;
        }
        if (gtid < 8 * kMaxGridVerts) B.hmisc[(hp ^ 1) * 8 * kMaxGridVerts + gtid] = 0;
        if (gtid == 0) B.stats[1] += ns;
        heavy_round++;
      }
      if (metric == kTV) {
        // marker = last scanner of each part among the committed positions: each
        // warp offers the last of its own positions per part that no later CTA
        // scanned, stamped with the window (round + 1), and the next round state
        // reads the maximum (with every warp offering every part it scanned the
        // commit of a window of 4400 positions of 1M Zipf vertices took 67 us
        // instead of 20: the atomics meet on K words)
        __syncthreads();
        for (int x = threadIdx.x; x < words; x += blockDim.x) cmask_s[x] = 0;
        __syncthreads();
        {
          const int per = kSWarps * q, whole = min((cut - pos) / per, (int)gridDim.x);   // CTAs whose positions all count
          for (int x = ((int)blockIdx.x + 1) * words + (int)threadIdx.x; x < whole * words; x += blockDim.x)
            if (const uint32_t m = lds(&B.cmask[x])) atomicOr(&cmask_s[x % words], m);
        }
        __syncthreads();
        const int zc = min(z1, cut);
        const unsigned long long stamp = (unsigned long long)(round + 1) << 32;
        for (int wd = lane; wd < words; wd += 32) {
          uint32_t seen = cmask_s[wd];
          for (int z = zc - 1; z >= z0 && seen != ~0u; z--) {
            uint32_t m = lds(&B.scan[(size_t)(z - pos) * words + wd]) & ~seen;
            seen |= m;
            while (m) {
              const int b = __ffs(m) - 1;
              m &= m - 1;
              atomicMax(&B.mlast[wd * 32 + b], stamp | (unsigned)z);
            }
          }
        }
      }
      if (gw == 0 && lane == 0) {
        B.ctl[2 + (par ^ 1)] = kNone;
        B.ctl[4 + (par ^ 1)] = kNone;
        B.ctl[12 + (par ^ 1)] = 0;
        B.ctl[14 + (par ^ 1)] = 0;
        B.ctl[9] = kNone;   // (read behind a fix's barrier, written by fixes alone)
        B.mcnt[par ^ 1] = 0;
        B.ctab_over[par ^ 1] = 0;
      }
      if (rv) {
        // MSRV's list of max parts after the committed movers; a last one without
        // listed terms is left to the next round's scan
        __syncthreads();
        int x = 0, c = 0;
        while (x < vs_s.n && pos + vs_s.at[x] < cut) {
          x++;
          c = max(c, vs_s.count[x]);
        }
        prev_maxtouch = vs_s.over != kNone && pos + vs_s.over < cut;
        const int cc0 = s_cc;
        __syncthreads();
        if (x) {
          for (int p = threadIdx.x; p < K; p += blockDim.x)
            mark_s[p] = (vbits[x * words + (p >> 5)] >> (p & 31)) & 1u ? cc0 : -1;
          if (threadIdx.x == 0) {
            s_maxv = vs_s.maxv[x];
            s_count = vs_s.count[x];
            if (c > K) dev_fail(I.status, kDevErrUnsupported);   // the reference overruns max_parts
          }
        }
        __syncthreads();
      }
      if (cut == end_w) {
        if (end_w == pos + W) W = min(2 * W, B.wmax);
      } else {
        // regrow from the last valid length, by at most a factor of four down:
        // every position past the cut is evaluated again, and walked (windows of
        // at least one position per warp instead: 16K-vertex Zipf with unit
        // weights under TV 47 -> 101 ms per pass, 256K degree weights MSV 243 ->
        // 260, MSRV 47.2 -> 46.4)
        W = min(B.wmax, max(B.wmin > 0 ? B.wmin : 128, max(W / 4, B.wgrow * (cut - pos))));
      }
      pos = cut;
      round++;
      if (!grid_barrier(B.bar, I.status)) return;
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned long long tC = gtimer();
        B.stats[18] += tC - tA;
        tA = tC;
      }
    }
  }
  if (metric == kTV && blockIdx.x == 0) {
    // markers of the last window (the loop's final barrier made them visible)
    for (int p = threadIdx.x; p < K; p += blockDim.x) {
      const unsigned long long ml = lds(&B.mlast[p]);
      if (round > 0 && (int)(ml >> 32) == round) I.marker[p] = __ldg(&B.porder[(int)(ml & 0xffffffffu)]);
    }
  }
}

}  // namespace

size_t spec_ldg_smem_bytes(int K) {
  auto a = [](size_t n) { return (n + 15) & ~size_t(15); };
  const size_t k4 = a(sizeof(int) * K);
  const size_t eval = 4 * a(sizeof(int) * (size_t)K * kSWarps) + a(sizeof(unsigned long long) * (size_t)K * kSWarps);
  return 5 * k4 + std::max(eval, sizeof(WalkSmem) + sizeof(int) * K);
}

cudaError_t launch_spec_ldg(const DevInstance& I, const SpecBuf& B, int passes, int num_sms, cudaStream_t st,
                            int* grid_out) {
  const size_t smem = spec_ldg_smem_bytes(I.K);
  const void* fn = (const void*)spec_ldg_kernel;
  cudaError_t err = allow_shared_memory(fn);
  if (err != cudaSuccess) return err;
  int per_sm = 0;
  err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kSThreads, smem);
  if (err != cudaSuccess) return err;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  int grid = per_sm * num_sms;
  if (grid * kSWarps > B.max_warps) grid = B.max_warps / kSWarps;
  if (grid_out) *grid_out = grid;
  DevInstance Ic = I;
  SpecBuf Bc = B;
  int p = passes;
  void* args[] = {&Ic, &Bc, &p};
  err = cudaLaunchCooperativeKernel(fn, grid, kSThreads, args, smem, st);
  if (err != cudaSuccess) return err;
  return cudaGetLastError();
}

}  // namespace fp
