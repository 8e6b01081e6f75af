// Speculative grid-wide refinement for CN (CN/partition.cpp:245-377): the walk
// goes over the nets in id order; a net with exactly two parts moves all pins
// of its smaller side to the other part, unless one of those pins is in a net
// that is not cut.
//
// A round covers a window of nets; every warp decides its nets against the
// current state.  Claims are stamped with the round number, so they never need
// to be cleared.  A net that will move pins ("acting") claims every net of
// those pins (its write set).  An acting net takes at most one part off a
// net (all its pins move old -> new), so behind n earlier acting nets a net of
// more than 2 + n parts still has more than two, and one of at least 2 + n is
// still cut.  A later net is therefore invalid only if an earlier acting net
// claimed its own list and it has at most 2 + n parts, or claimed a net of its
// smaller side that has fewer than 2 + n, or the uncut net that kept it from
// acting.  The first invalid net cuts the window.
//
// An acting net moves its pins one at a time in the reference, each move
// updating every net of the pin.  All of them move old -> new, so the k moves
// that land on one net have a result that depends on k only (cn_apply_net);
// the commit counts the moves per net, then one warp updates each touched net:
// the moves of the first acting net that claimed it, then those of the others,
// in order.  Large nets are shared by most pairs of acting nets; with write
// sets kept disjoint instead, a window of the 256K-net Zipf workload held 1.5
// of them.

#include "fp_spec_common.cuh"

namespace fp {

namespace {

using namespace spec;

// A window that moves few pins (27 on average on 262144 Zipf vertices), one of them
// on more than kCnChunk nets, spreads each one's nets over the warps: a hub's
// thousands of nets took one warp 60 us, C1 takes 10 so.  More pins keep the warps
// busy as they are, and pins of few nets need no search for shares (a commit on 86565
// mixed vertices 12.0 us with it, 10.7 without).
constexpr int kCnSpreadMoves = 256, kCnChunk = 128, kCnStep = 37;
constexpr int kShared = 1 << 30;   // cn_kcnt: several acting nets move pins of the net

// Round-stamped claim: the latest round wins, then the smallest position.
__device__ __forceinline__ unsigned long long ckey(int round, int pos) {
  return ((unsigned long long)(unsigned)round << 32) | (0xffffffffu - (unsigned)pos);
}
// Did a net position earlier than `pos` claim net x in this round?
__device__ __forceinline__ bool claim_before(const SpecBuf& B, int round, int x, int pos) {
  const unsigned long long c = lds(&B.claim64[x]);
  return (int)(c >> 32) == round && (int)(0xffffffffu - (unsigned)(c & 0xffffffffu)) < pos;
}

// Walk of the (pin, net) pairs of net e's pins [pb, pe) on part oldp, 32 pins
// at a time, the pairs flattened across the warp with 4 loads in flight per
// lane.
//   kMode 0: returns a net of those pins that is not cut (-1: none);
//   kMode 1: claims every such net for position e and records the pins to move
//            (window offset o, round parity par); returns -1;
//   kMode 2: returns 1 if an acting net before e claimed one of them that has
//            fewer than 2 + nb parts (nb acting nets before e), else -1.
// Modes 0 and 2 stop early when *stop (shared by the warps splitting a net's
// pins) is set.
// gstop: the same in global memory (the grid's warps splitting a net).
template <int kMode>
__device__ int cn_walk_range(const DevInstance& I, const SpecBuf& B, int e, int pb, int pe, int oldp, int round,
                             int o, int par, int nb, const volatile int* stop, const int* gstop = nullptr) {
  const int lane = threadIdx.x & 31;
  for (int b0 = pb; b0 < pe; b0 += 32) {
    if (kMode != 1 && stop && __shfl_sync(kAll, *stop, 0)) return -1;   // warp-uniform: lane 0's read
    if (kMode != 1 && gstop && __shfl_sync(kAll, lds(gstop), 0)) return -1;
    const int k = b0 + lane;
    int u = -1, d = 0;
    uint32_t ub = 0;
    if (k < pe) {
      u = (int)__ldg(&I.npins[k]);
      if (lds(&I.part_vec[u]) == oldp) {
        ub = __ldg(&I.vptr[u]);
        d = (int)(__ldg(&I.vptr[u + 1]) - ub);
      } else {
        u = -1;
      }
    }
    if (kMode == 0) {
      // a pin's cached witness: a net of the pin found uncut before; still
      // uncut, it ends the search without walking the pin's nets (hub pins
      // lie on millions of nets)
      const int w = u >= 0 ? lds(&B.cn_wit[u]) : -1;
      const int hit = (w >= 0 && lds(&I.ep_len[w]) == 1) ? w : -1;
      const unsigned m = __ballot_sync(kAll, hit >= 0);
      if (m) return __shfl_sync(kAll, hit, __ffs(m) - 1);
    }
    if (kMode == 1 && u >= 0) {
      B.cn_moved[atomicAdd(&B.cn_cnt[par], 1)] = make_int2(u, o);
      if (d > kCnChunk) B.cn_cnt[6 + par] = 1;
    }
    int incl = d;
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(kAll, incl, off);
      if (lane >= off) incl += t;
    }
    const int total = __shfl_sync(kAll, incl, 31);
    constexpr int kU = 4;
    for (int f0 = 0; f0 < total; f0 += 32 * kU) {
      int xs[kU];
#pragma unroll
      for (int q = 0; q < kU; q++) {
        const int f = f0 + q * 32 + lane;
        int lo = 0, hi = 31;
#pragma unroll
        for (int it = 0; it < 5; it++) {
          const int mid = (lo + hi) >> 1;
          const int val = __shfl_sync(kAll, incl, mid);
          if (f < val) hi = mid; else lo = mid + 1;
        }
        const uint32_t bl = __shfl_sync(kAll, ub, lo);
        const int dl = __shfl_sync(kAll, d, lo);
        const int il = __shfl_sync(kAll, incl, lo);
        xs[q] = f < total ? (int)__ldg(&I.vnets[bl + (uint32_t)(f - (il - dl))]) : -1;
      }
      if (kMode == 0) {
        int hit = -1, hq = 0;
#pragma unroll
        for (int q = 0; q < kU; q++)
          if (xs[q] >= 0 && hit < 0 && lds(&I.ep_len[xs[q]]) == 1) { hit = xs[q]; hq = q; }
        const unsigned m = __ballot_sync(kAll, hit >= 0);
        if (m) {
          const int src = __ffs(m) - 1;
          const int x = __shfl_sync(kAll, hit, src);
          // the pin of that pair keeps it as its witness
          const int f = f0 + __shfl_sync(kAll, hq, src) * 32 + src;
          int lo = 0, hi = 31;
#pragma unroll
          for (int it = 0; it < 5; it++) {
            const int mid = (lo + hi) >> 1;
            const int val = __shfl_sync(kAll, incl, mid);
            if (f < val) hi = mid; else lo = mid + 1;
          }
          const int uw = __shfl_sync(kAll, u, lo);
          if (lane == 0 && uw >= 0) B.cn_wit[uw] = x;
          return x;
        }
      } else if (kMode == 1) {
#pragma unroll
        for (int q = 0; q < kU; q++)
          if (xs[q] >= 0) atomicMax(&B.claim64[xs[q]], ckey(round, e));
      } else {
        bool c = false;
#pragma unroll
        for (int q = 0; q < kU; q++)
          if (xs[q] >= 0 && claim_before(B, round, xs[q], e) && lds(&I.ep_len[xs[q]]) < 2 + nb) c = true;
        if (__any_sync(kAll, c)) return 1;
      }
    }
  }
  return -1;
}

template <int kMode>
__device__ __forceinline__ int cn_walk(const DevInstance& I, const SpecBuf& B, int e, int oldp, int round, int o,
                                       int par, int nb = 0) {
  return cn_walk_range<kMode>(I, B, e, (int)__ldg(&I.nptr[e]), (int)__ldg(&I.nptr[e + 1]), oldp, round, o, par, nb,
                              nullptr);
}

// Acting nets of the round before net e (one warp; midx holds their ids).
__device__ __forceinline__ int cn_acting_before(const SpecBuf& B, int nact, int e) {
  int n = 0;
  for (int i = threadIdx.x & 31; i < nact; i += 32) n += lds(&B.midx[i]) < e;
  return warp_sum(n);
}
__device__ __forceinline__ void cn_list_acting(const SpecBuf& B, int par, int e) {
  B.midx[atomicAdd(&B.mcnt[par], 1)] = e;
}

// What the acting nets before e may have changed of what e's own list decides: e
// conflicts with nb of them if the result is at most 2 + nb (0: one claimed its
// witness; its parts: one claimed e itself; kNone: neither).  It does not depend
// on nb, so that its loads and those of the count are under way together.
__device__ __forceinline__ int cn_own_claims(const DevInstance& I, const SpecBuf& B, int round, int e, int unc) {
  const int n = lds(&I.ep_len[e]);
  const bool own = claim_before(B, round, e, e);
  if (unc >= 0 && claim_before(B, round, unc, e)) return 0;
  return own ? n : kNone;
}

// Warp gw's contiguous share (of nw warps) of net e's pins.
__device__ __forceinline__ void cn_grid_share(const DevInstance& I, int e, int gw, int nw, int* pb, int* pe) {
  const int b = (int)__ldg(&I.nptr[e]), n = (int)__ldg(&I.nptr[e + 1]) - b;
  const int g = (n + nw - 1) / nw;
  *pb = b + min(gw * g, n);
  *pe = b + min(gw * g + g, n);
}

// Two-part test of net e (CN/partition.cpp:262-270): old (smaller side) and
// new parts, false if the net does not span exactly two parts.
__device__ __forceinline__ bool cn_two(const DevInstance& I, int e, int* oldp, int* newp, int* oldc = nullptr) {
  if (lds(&I.ep_len[e]) != 2) return false;
  const int s = (int)__ldg(&I.nptr[e]);
  const int p1 = lds(&I.ep_part[s]), c1 = lds(&I.ep_cnt[s]);
  const int p2 = lds(&I.ep_part[s + 1]), c2 = lds(&I.ep_cnt[s + 1]);
  *oldp = c1 < c2 ? p1 : p2;
  *newp = c1 < c2 ? p2 : p1;
  if (oldc) *oldc = c1 < c2 ? c1 : c2;
  return true;
}

// Warp wib's contiguous share of net e's pins.
__device__ __forceinline__ void cn_pin_share(const DevInstance& I, int e, int* pb, int* pe) {
  const int b = (int)__ldg(&I.nptr[e]), n = (int)__ldg(&I.nptr[e + 1]) - b;
  const int g = (n + kSWarps - 1) / kSWarps, w = (int)(threadIdx.x >> 5);
  *pb = b + min(w * g, n);
  *pe = b + min(w * g + g, n);
}

// Evaluation of a net with many pins by the whole CTA: the warps split its
// pins (cn_eval's rules), then the claims of an acting net.
__device__ void cn_eval_cta(const DevInstance& I, const SpecBuf& B, int e, int o, int round, int par, bool logp) {
  __shared__ int sh_two, sh_old, sh_new, sh_unc, sh_cold;
  __shared__ volatile int sh_stop;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    sh_two = 0;
    sh_unc = -1;
    sh_stop = 0;
    if (lds(&I.ep_len[e]) == 2) {
      const int s = (int)__ldg(&I.nptr[e]);
      const int p1 = lds(&I.ep_part[s]), c1 = lds(&I.ep_cnt[s]);
      const int p2 = lds(&I.ep_part[s + 1]), c2 = lds(&I.ep_cnt[s + 1]);
      sh_two = 1;
      sh_old = c1 < c2 ? p1 : p2;
      sh_new = c1 < c2 ? p2 : p1;
      sh_cold = c1 < c2 ? c1 : c2;
    }
  }
  __syncthreads();
  int act = 0;
  const int oldp = sh_two ? sh_old : 0, newp = sh_two ? sh_new : 0;
  if (sh_two) {
    int pb, pe;
    cn_pin_share(I, e, &pb, &pe);
    const int hit = cn_walk_range<0>(I, B, e, pb, pe, oldp, 0, 0, 0, 0, &sh_stop);
    if (hit >= 0 && lane == 0) {
      atomicCAS(&sh_unc, -1, hit);   // any uncut net is a witness
      sh_stop = 1;
    }
    __syncthreads();
    act = sh_unc < 0;
    if (act) cn_walk_range<1>(I, B, e, pb, pe, oldp, round, o, par, 0, nullptr);
  }
  if (threadIdx.x == 0) {
    if (act) cn_list_acting(B, par, e);
    B.dec[o] = (oldp << 16) | newp;
    B.flag[o] = (unsigned char)act;
    B.slack[o] = sh_unc;   // the uncut net that blocks the move (-1: none)
    if (logp) B.rgain[o] = sh_two ? sh_cold : -1;
  }
  __syncthreads();
}

// Validation of a net with many pins by the whole CTA (the warp loop's rules);
// a conflict lowers the cut word.
__device__ void cn_validate_cta(const DevInstance& I, const SpecBuf& B, int e, int o, int round, int nact, int* cut) {
  __shared__ volatile int sh_conf;
  const int lane = threadIdx.x & 31;
  const int act = lds(&B.flag[o]);
  const int own = cn_own_claims(I, B, round, e, lds(&B.slack[o]));
  const int nb = cn_acting_before(B, nact, e);
  if (threadIdx.x == 0) sh_conf = own <= 2 + nb ? 1 : 0;
  __syncthreads();
  if (act && !sh_conf) {
    int pb, pe;
    cn_pin_share(I, e, &pb, &pe);
    if (cn_walk_range<2>(I, B, e, pb, pe, lds(&B.dec[o]) >> 16, round, 0, 0, nb, &sh_conf) > 0 && lane == 0) sh_conf = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0 && sh_conf) atomicMin(cut, (e << 3) | 5);
  __syncthreads();
}

// Evaluation of net e (one warp).  Returns 0 (no move), 1 (acting), and the
// old / new parts; *uncut = a net proving "no move" (-1 if e is not two-part).
__device__ int cn_eval(const DevInstance& I, const SpecBuf& B, int e, int* oldp_o, int* newp_o, int* uncut,
                       int* oldc_o) {
  *uncut = -1;
  *oldc_o = -1;
  if (lds(&I.ep_len[e]) != 2) return 0;
  const int s = (int)__ldg(&I.nptr[e]);
  const int p1 = lds(&I.ep_part[s]), c1 = lds(&I.ep_cnt[s]);
  const int p2 = lds(&I.ep_part[s + 1]), c2 = lds(&I.ep_cnt[s + 1]);
  const int oldp = c1 < c2 ? p1 : p2;
  const int newp = c1 < c2 ? p2 : p1;
  *oldp_o = oldp;
  *newp_o = newp;
  *oldc_o = c1 < c2 ? c1 : c2;
  // any pin on the smaller side with a net that is not cut?
  *uncut = cn_walk<0>(I, B, e, oldp, 0, 0, 0);
  return *uncut < 0 ? 1 : 0;
}

// A net's list where it lies, or staged in shared memory.
struct ListHere {
  const DevInstance& I;
  int s;
  __device__ int part(int j) const { return lds(&I.ep_part[s + j]); }
  __device__ int cnt(int j) const { return lds(&I.ep_cnt[s + j]); }
  __device__ void set_part(int j, int p) const { I.ep_part[s + j] = p; }
  __device__ void set_cnt(int j, int c) const { I.ep_cnt[s + j] = c; }
};
struct ListStaged {
  int2* l;
  __device__ int part(int j) const { return l[j].x; }
  __device__ int cnt(int j) const { return l[j].y; }
  __device__ void set_part(int j, int p) const { l[j].x = p; }
  __device__ void set_cnt(int j, int c) const { l[j].y = c; }
};

// k moves oldp -> newp of pins of a net with list L (n parts, room for cap), each
// the reference's REMOVAL then ADDING (CN/partition.cpp:311-370), applied at once
// by one warp: the lanes find the two slots, lane 0 replays the k steps.  Only
// the first step can append newp and only the last can remove oldp, so the
// k-fold result follows from the counts.  Returns the new length (every lane).
template <class List>
__device__ int cn_apply_moves(const DevInstance& I, const List& L, int n, int cap, int oldp, int newp, int k) {
  const int lane = threadIdx.x & 31;
  int jo = -1, jd = -1;
  for (int j0 = 0; j0 < n; j0 += 32) {
    const int j = j0 + lane;
    const int p = j < n ? L.part(j) : -1;
    const unsigned mo = __ballot_sync(kAll, p == oldp);
    const unsigned md = __ballot_sync(kAll, p == newp);
    if (mo && jo < 0) jo = j0 + __ffs(mo) - 1;
    if (md && jd < 0) jd = j0 + __ffs(md) - 1;
  }
  __syncwarp();
  if (lane == 0) {
    int co = jo >= 0 ? L.cnt(jo) : 0;
    int cd = jd >= 0 ? L.cnt(jd) : 0;
    if (jo < 0 || n > cap || co < k || k < 1) {
      dev_fail(I.status, kDevErrInvalid);
    } else {
      bool ok = true;
      // oldp's count reached zero: the last entry fills its slot
      auto remove_old = [&]() {
        const int last = n - 1;
        if (last != jo) {
          if (last == jd) {
            L.set_part(jo, newp);
            jd = jo;
          } else {
            L.set_part(jo, L.part(last));
            L.set_cnt(jo, L.cnt(last));
          }
        }
        L.set_part(last, -1);
        L.set_cnt(last, 0);
        n = last;
        jo = -1;
      };
      auto append_new = [&]() {
        if (n >= cap) { ok = false; return; }
        jd = n;
        cd = 1;
        L.set_part(jd, newp);
        n++;
      };
      if (jd >= 0) {
        co -= k;
        cd += k;
        if (co == 0) remove_old();
      } else {
        co -= 1;   // first move
        if (co == 0) {
          remove_old();
          append_new();   // k == 1
        } else {
          append_new();
          co -= k - 1;    // the other k - 1 moves
          cd += k - 1;
          if (co == 0) remove_old();
        }
      }
      if (!ok) {
        dev_fail(I.status, kDevErrInvalid);
      } else {
        if (jo >= 0) L.set_cnt(jo, co);
        L.set_cnt(jd, cd);
      }
    }
  }
  __syncwarp();
  return __shfl_sync(kAll, n, 0);
}

// The same on net x's list in global memory.
__device__ void cn_apply_net(const DevInstance& I, int x, int oldp, int newp, int k) {
  const int s = (int)__ldg(&I.nptr[x]);
  const int cap = (int)__ldg(&I.nptr[x + 1]) - s;
  const int n = cn_apply_moves(I, ListHere{I, s}, lds(&I.ep_len[x]), cap, oldp, newp, k);
  if ((threadIdx.x & 31) == 0) I.ep_len[x] = n;
  __syncwarp();
}

// The moves of several acting nets on net x in their order: k0 of the first one
// (pk0: old and new part), then those listed in cn_more (nmore entries), one warp.
// The list is staged in shared memory (list) and the acting nets gathered once
// (acts): a shared net of 262144 Zipf vertices (K = 256) has dozens, and each took
// a scan of cn_more and of the list in L2: 53 us of commit per window, 28 so.
// False if either does not fit.
constexpr int kCnStage = 256, kCnActs = 256;
__device__ bool cn_apply_shared(const DevInstance& I, const SpecBuf& B, int x, int pk0, int k0, int nmore, int2* list,
                                int2* acts) {
  const int lane = threadIdx.x & 31;
  int na = 0;
  for (int i0 = 0; i0 < nmore; i0 += 32) {
    const int2 m2 = i0 + lane < nmore ? lds(&B.cn_more[i0 + lane]) : make_int2(-1, 0);
    const unsigned m = __ballot_sync(kAll, m2.x == x);
    const int at = na + __popc(m & ((1u << lane) - 1u));
    if (m2.x == x && at < kCnActs) acts[at] = make_int2(m2.y, lds(&B.dec[m2.y]));
    na += __popc(m);
  }
  const int s = (int)__ldg(&I.nptr[x]);
  const int cap = (int)__ldg(&I.nptr[x + 1]) - s;
  const int n0 = lds(&I.ep_len[x]);
  const int room = min(min(cap, I.K), n0 + na + 1);   // each acting net adds a part at most
  if (na > kCnActs || n0 > cap || room > kCnStage) return false;
  for (int j = lane; j < room; j += 32) list[j] = j < n0 ? make_int2(lds(&I.ep_part[s + j]), lds(&I.ep_cnt[s + j])) : make_int2(-1, 0);
  __syncwarp();
  const ListStaged L{list};
  int n = cn_apply_moves(I, L, n0, room, pk0 >> 16, pk0 & 0xffff, k0);
  for (int last = -1;;) {
    int o = kNone, c = 0, pk = 0;
    for (int j = lane; j < na; j += 32) {
      const int2 t = acts[j];
      if (t.x <= last || t.x > o) continue;
      c = t.x == o ? c + 1 : 1;
      o = t.x;
      pk = t.y;
    }
    const int o1 = warp_min(o);
    if (o1 == kNone) break;
    pk = __shfl_sync(kAll, pk, __ffs(__ballot_sync(kAll, o == o1)) - 1);
    n = cn_apply_moves(I, L, n, room, pk >> 16, pk & 0xffff, warp_sum(o == o1 ? c : 0));
    last = o1;
  }
  for (int j = lane; j < max(n, n0); j += 32) {
    I.ep_part[s + j] = list[j].x;
    I.ep_cnt[s + j] = list[j].y;
  }
  if (lane == 0) I.ep_len[x] = n;
  __syncwarp();
  return true;
}

// Three CTAs per SM: without the hint the compiler spills to fit more.
__global__ void __launch_bounds__(kSThreads, 3) spec_cn_kernel(DevInstance I, SpecBuf B, int passes) {
  barrier_start();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int gw = blockIdx.x * kSWarps + wib;
  const int nwarps = gridDim.x * kSWarps;
  // the window's grid-evaluated nets: id, two-part, old and new part
  __shared__ int s_ge[kMaxGridVerts], s_gt[kMaxGridVerts], s_go[kMaxGridVerts], s_gn[kMaxGridVerts];
  unsigned long long tA = gtimer();
  int round = 1;   // claims of round 0 (the cleared array) never match
  int heavy_round = 0;
  __shared__ int s_gc[kMaxGridVerts];
  __shared__ int2 list_b[kSWarps * kCnStage];   // per-warp staged list and acting nets of a shared net
  __shared__ int2 acts_b[kSWarps * kCnActs];
  for (int it = 0; it < passes; it++) {
    // decision records of the last pass: (new part, pins moved, old part,
    // acting) of a two-part net, (-1, 0, -1, 0) of any other net
    const bool logp = I.recs != nullptr && it == passes - 1;
    int pos = 0;
    int W = min(nwarps * 4, B.wmax);
    int hidx = 0, midx = 0;
    while (pos < I.noe) {
      const int par = round & 1;
      // a window holds up to gmax nets evaluated by the grid and ends before the next
      hidx = seek_pos(B.heavy_pos, B.nheavy, hidx, pos);
      midx = seek_pos(B.mid_pos, B.nmid, midx, pos);
      int end_w = min(pos + W, I.noe);
      if (hidx + B.gmax < B.nheavy) end_w = min(end_w, (int)__ldg(&B.heavy_pos[hidx + B.gmax]));
      const int ns = min(B.gmax, seek_pos(B.heavy_pos, B.nheavy, hidx, end_w) - hidx);
      const int hp = heavy_round & 1;
      // slot j of this parity in hmisc: [0] uncut witness + 1 (0: none), [1] conflict
      auto hm = [&](int j) { return B.hmisc + (hp * kMaxGridVerts + j) * 8; };
      if ((int)threadIdx.x < ns) {
        const int e = __ldg(&B.heavy_pos[hidx + threadIdx.x]);
        int op = 0, np = 0, oc = -1;
        s_ge[threadIdx.x] = e;
        s_gt[threadIdx.x] = cn_two(I, e, &op, &np, &oc) ? 1 : 0;
        s_go[threadIdx.x] = op;
        s_gn[threadIdx.x] = np;
        s_gc[threadIdx.x] = oc;
      }
      __syncthreads();
      // ---- A0: the grid's warps split the pins of each grid net (uncut search)
      for (int j = 0; j < ns; j++) {
        if (!s_gt[j]) continue;
        int pb, pe;
        cn_grid_share(I, s_ge[j], gw, nwarps, &pb, &pe);
        const int hit = cn_walk_range<0>(I, B, s_ge[j], pb, pe, s_go[j], 0, 0, 0, 0, nullptr, hm(j));
        if (hit >= 0 && lane == 0) atomicCAS(hm(j), 0, hit + 1);
      }
      const int span = end_w - pos;
      const int q = (span + nwarps - 1) / nwarps;
      const int z0 = min(pos + gw * q, end_w);
      const int z1 = min(z0 + q, end_w);
      // ---- A: evaluate; acting nets claim the nets of the pins they move
      for (int e = z0; e < z1; e++) {
        const int o = e - pos;
        if ((int)(__ldg(&I.nptr[e + 1]) - __ldg(&I.nptr[e])) > B.cn_big) continue;   // the CTA evaluates it below
        int oldp = 0, newp = 0, unc = -1, oldc = -1;
        const int act = cn_eval(I, B, e, &oldp, &newp, &unc, &oldc);
        if (act) cn_walk<1>(I, B, e, oldp, round, o, par);
        if (lane == 0) {
          if (act) cn_list_acting(B, par, e);
          B.dec[o] = (oldp << 16) | newp;
          B.flag[o] = (unsigned char)act;
          B.slack[o] = unc;   // the uncut net that blocks the move (-1: none)
          if (logp) B.rgain[o] = oldc;
        }
        __syncwarp();
      }
      // nets with many pins of this CTA's positions: the whole CTA each
      const int cz0 = min(pos + blockIdx.x * kSWarps * q, end_w);
      const int cz1 = min(cz0 + kSWarps * q, end_w);
      for (int mi = seek_pos(B.mid_pos, B.nmid, midx, cz0); mi < B.nmid; mi++) {
        const int e = __ldg(&B.mid_pos[mi]);
        if (e >= cz1) break;
        cn_eval_cta(I, B, e, e - pos, round, par, logp);
      }
      if (!grid_barrier(B.bar, I.status)) return;
      if (ns) {
        // ---- A1: an acting grid net's claims and pins, split across the grid
        for (int j = 0; j < ns; j++) {
          const int e = s_ge[j], o = e - pos;
          const int unc = lds(hm(j)) - 1;
          const int act = s_gt[j] && unc < 0;
          if (act) {
            int pb, pe;
            cn_grid_share(I, e, gw, nwarps, &pb, &pe);
            cn_walk_range<1>(I, B, e, pb, pe, s_go[j], round, o, par, 0, nullptr);
          }
          if (blockIdx.x == 0 && threadIdx.x == 0) {
            if (act) cn_list_acting(B, par, e);
            B.dec[o] = s_gt[j] ? (s_go[j] << 16) | s_gn[j] : 0;
            B.flag[o] = (unsigned char)act;
            B.slack[o] = s_gt[j] ? unc : -1;
            if (logp) B.rgain[o] = s_gt[j] ? s_gc[j] : -1;
          }
        }
        if (!grid_barrier(B.bar, I.status)) return;
      }
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned long long tE = gtimer();
        B.stats[16] += tE - tA;
        tA = tE;
      }
      // ---- B: validate against earlier acting nets' claims
      const int nact = lds(&B.mcnt[par]);
      // (the acting nets before a warp's first net are counted once, beside its
      // words' loads; counted for each net, after them, a window of 86565 mixed
      // vertices, K = 128, took 8.7 us to validate instead of 8.0)
      for (int e = z0, before = -1; e < z1; e++) {
        const int o = e - pos;
        const int act = lds(&B.flag[o]);
        const int own = cn_own_claims(I, B, round, e, lds(&B.slack[o]));
        const int nb = before < 0 ? cn_acting_before(B, nact, e) : before;
        before = nb + act;
        if ((int)(__ldg(&I.nptr[e + 1]) - __ldg(&I.nptr[e])) > B.cn_big) continue;   // validated by the CTA below
        if (nb == 0) continue;
        bool conf = own <= 2 + nb;
        if (act && !conf) conf = cn_walk<2>(I, B, e, lds(&B.dec[o]) >> 16, round, 0, 0, nb) > 0;
        conf = __any_sync(kAll, conf);
        if (conf) {
          if (lane == 0) atomicMin(&B.ctl[par], (e << 3) | 5);
          break;
        }
      }
      __syncthreads();
      for (int mi = seek_pos(B.mid_pos, B.nmid, midx, cz0); mi < B.nmid; mi++) {
        const int e = __ldg(&B.mid_pos[mi]);
        if (e >= cz1) break;
        cn_validate_cta(I, B, e, e - pos, round, nact, &B.ctl[par]);
      }
      for (int j = 0; j < ns; j++) {
        // a grid net: its own list and witness by every warp (cheap), its
        // moving pins' nets split across the grid
        const int e = s_ge[j], o = e - pos;
        const int own = cn_own_claims(I, B, round, e, lds(&B.slack[o]));
        const int nb = cn_acting_before(B, nact, e);
        bool conf = own <= 2 + nb;
        if (!conf && lds(&B.flag[o])) {
          int pb, pe;
          cn_grid_share(I, e, gw, nwarps, &pb, &pe);
          conf = cn_walk_range<2>(I, B, e, pb, pe, s_go[j], round, 0, 0, nb, nullptr, hm(j) + 1) > 0;
          if (conf && lane == 0) atomicExch(hm(j) + 1, 1);
        }
        if (conf && lane == 0) atomicMin(&B.ctl[par], (e << 3) | 5);
      }
      if (!grid_barrier(B.bar, I.status)) return;
      const int cutw = lds(&B.ctl[par]);
      const int cut = cutw == kNone ? end_w : min(cutw >> 3, end_w);
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned long long tB = gtimer();
        B.stats[0]++;
        B.stats[cutw == kNone ? 3 : 8]++;
        B.stats[9] += cut - pos;
        B.stats[17] += tB - tA;
        tA = tB;
      }
      if (cut <= pos) {
        if (threadIdx.x == 0) dev_fail(I.status, kDevErrInvalid);
        return;
      }
      if (logp) {
        for (int e = z0 + lane; e < min(z1, cut); e += 32) {
          const int o = e - pos;
          const int oc = lds(&B.rgain[o]);
          const int act = lds(&B.flag[o]) & 1;
          const int pk = lds(&B.dec[o]);
          I.recs[e] = oc >= 0 ? make_int4(pk & 0xffff, act ? oc : 0, pk >> 16, act) : make_int4(-1, 0, -1, 0);
        }
      }
      // ---- C1: pins of acting nets before the cut: part, sizes, moves per net
      const int nmv = lds(&B.cn_cnt[par]);
      auto move_nets = [&](int2 mv, uint32_t j0, uint32_t j1) {
        const int pk = lds(&B.dec[mv.y]);
        for (uint32_t j = j0 + lane; j < j1; j += 32) {
          const int x = (int)__ldg(&I.vnets[j]);
          // the first acting net that claimed x counts its moves on it; those of
          // the others are listed (kShared marks the net)
          const int first = (int)(0xffffffffu - (unsigned)(lds(&B.claim64[x]) & 0xffffffffull));
          if (first == pos + mv.y) {
            if ((atomicAdd(&B.cn_kcnt[x], 1) & (kShared - 1)) == 0)
              B.cn_nets[atomicAdd(&B.cn_cnt[2 + par], 1)] = make_int2(x, pk);
          } else {
            atomicOr(&B.cn_kcnt[x], kShared);
            B.cn_more[atomicAdd(&B.cn_cnt[4 + par], 1)] = make_int2(x, mv.y);
          }
        }
      };
      auto move_pin = [&](int2 mv) {
        const int u = mv.x, pk = lds(&B.dec[mv.y]);
        const int oldp = pk >> 16, newp = pk & 0xffff;
        I.part_vec[u] = newp;
        const int wv = __ldg(&I.w[u]);
        atomicAdd(&I.part_sizes[oldp], -wv);
        atomicAdd(&I.part_sizes[newp], wv);
        atomicAdd((unsigned long long*)&I.moves[it], 1ull);
        atomicAdd(&B.stats[2], 1ull);
      };
      if (nmv > kCnSpreadMoves || !lds(&B.cn_cnt[6 + par])) {
        for (int i = gw; i < nmv; i += nwarps) {
          const int2 mv = lds(&B.cn_moved[i]);
          if (pos + mv.y >= cut) continue;
          move_nets(mv, __ldg(&I.vptr[mv.x]), __ldg(&I.vptr[mv.x + 1]));
          if (lane == 0) move_pin(mv);
        }
      } else {
        // few pins: kCnChunk nets of one per warp, chunk c of pin i to warp
        // i * kCnStep + c; the lanes look for this warp's chunks among 32 pins
        for (int i0 = 0; i0 < nmv; i0 += 32) {
          const int i = i0 + lane;
          int2 mv = make_int2(0, 0);
          uint32_t ub = 0, ue = 0;
          bool mine = false;
          if (i < nmv) {
            mv = lds(&B.cn_moved[i]);
            ub = __ldg(&I.vptr[mv.x]);
            ue = __ldg(&I.vptr[mv.x + 1]);
            mine = pos + mv.y < cut;
          }
          const int c0 = (gw + nwarps - i * kCnStep % nwarps) % nwarps;
          mine = mine && (c0 == 0 || c0 * (long long)kCnChunk < (long long)(ue - ub));
          for (unsigned m = __ballot_sync(kAll, mine); m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            const int2 mvs = make_int2(__shfl_sync(kAll, mv.x, src), __shfl_sync(kAll, mv.y, src));
            const uint32_t b = __shfl_sync(kAll, ub, src), e = __shfl_sync(kAll, ue, src);
            const int c1 = __shfl_sync(kAll, c0, src);
            for (long long c = c1; b + c * kCnChunk < e; c += nwarps)
              move_nets(mvs, (uint32_t)(b + c * kCnChunk), (uint32_t)min((long long)e, b + (c + 1) * kCnChunk));
            if (c1 == 0 && lane == 0) move_pin(mvs);
          }
        }
      }
      if (!grid_barrier(B.bar, I.status)) return;
      // ---- C2: every touched net once, with all of its moves
      const int nnet = lds(&B.cn_cnt[2 + par]);
      for (int i = gw; i < nnet; i += nwarps) {
        const int2 xe = lds(&B.cn_nets[i]);
        const int k = lds(&B.cn_kcnt[xe.x]);
        const int nmore = (k & kShared) ? lds(&B.cn_cnt[4 + par]) : 0;
        if (!(k & kShared) ||
            !cn_apply_shared(I, B, xe.x, xe.y, k & (kShared - 1), nmore, list_b + wib * kCnStage, acts_b + wib * kCnActs)) {
          cn_apply_net(I, xe.x, xe.y >> 16, xe.y & 0xffff, k & (kShared - 1));
          // the other acting nets' moves on it, in their order
          for (int last = -1; k & kShared;) {
            int o = kNone, c = 0;
            for (int i2 = lane; i2 < nmore; i2 += 32) {
              const int2 m2 = lds(&B.cn_more[i2]);
              if (m2.x != xe.x || m2.y <= last || m2.y > o) continue;
              c = m2.y == o ? c + 1 : 1;
              o = m2.y;
            }
            const int o1 = warp_min(o);
            if (o1 == kNone) break;
            const int pk2 = lds(&B.dec[o1]);
            cn_apply_net(I, xe.x, pk2 >> 16, pk2 & 0xffff, warp_sum(o == o1 ? c : 0));
            last = o1;
          }
        }
        if (lane == 0) B.cn_kcnt[xe.x] = 0;
      }
      if (gw == 0 && lane == 0) {
        B.ctl[par ^ 1] = kNone;
        B.cn_cnt[par ^ 1] = 0;
        B.cn_cnt[2 + (par ^ 1)] = 0;
        B.cn_cnt[4 + (par ^ 1)] = 0;
        B.cn_cnt[6 + (par ^ 1)] = 0;
        B.mcnt[par ^ 1] = 0;
      }
      if (ns) {
        // the other parity's grid-net words, for the next window with grid nets
        if (blockIdx.x == 0 && threadIdx.x < 8 * kMaxGridVerts) B.hmisc[(hp ^ 1) * 8 * kMaxGridVerts + threadIdx.x] = 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) B.stats[1] += ns;
        heavy_round++;
      }
      if (cut == end_w) {
        if (end_w == pos + W) W = min(2 * W, B.wmax);
      } else {
        W = max(1024, min(B.wmax, 2 * (cut - pos)));
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
}

}  // namespace

cudaError_t launch_spec_cn(const DevInstance& I, const SpecBuf& B, int passes, int num_sms, cudaStream_t st,
                           int* grid_out) {
  const void* fn = (const void*)spec_cn_kernel;
  int per_sm = 0;
  cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kSThreads, 0);
  if (err != cudaSuccess) return err;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  int grid = per_sm * num_sms;
  if (grid * kSWarps > B.max_warps) grid = B.max_warps / kSWarps;
  if (grid_out) *grid_out = grid;
  DevInstance Ic = I;
  SpecBuf Bc = B;
  int p = passes;
  void* args[] = {&Ic, &Bc, &p};
  err = cudaLaunchCooperativeKernel(fn, grid, kSThreads, args, 0, st);
  if (err != cudaSuccess) return err;
  return cudaGetLastError();
}

}  // namespace fp
