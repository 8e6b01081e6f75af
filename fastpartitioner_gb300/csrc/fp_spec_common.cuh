// Helpers shared by the speculative (grid-wide) refinement kernels.
#pragma once

#include "fp_device.cuh"

#include <cooperative_groups.h>

namespace fp {
namespace spec {

namespace cg = cooperative_groups;

constexpr int kSThreads = 256;
constexpr int kSWarps = kSThreads / 32;
constexpr int kNone = 0x7fffffff;
constexpr unsigned kAll = 0xffffffffu;

// Global nanosecond timer (per-phase time statistics).
__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Loads of state that other SMs write (L2, not the SM's L1).
template <class T>
__device__ __forceinline__ T lds(const T* p) { return __ldcg(p); }

// Grid-wide barrier of a co-resident (cooperatively launched) grid with a
// bounded wait.  bar[0] = arrivals, bar[2] = abort flag.  Every CTA adds to
// bar[0] once per barrier: CTA 0 adds 2^31 - (gridDim.x - 1), the others 1, so
// bit 31 flips exactly when the last CTA arrives and the low bits return to
// their value -- no reset, one atomic per CTA.  Returns false in every thread
// of the CTA if the wait gave up (another CTA stopped arriving) or another CTA
// aborted; the kernel then reports FP_ERR_DEVICE_TIMEOUT through `status` and
// returns.
//
// Failure-detection test hooks (fp_debug_barrier_fault; both zero unless a
// test sets them): bar[1] = n > 0 makes the grid's last CTA leave at its n-th
// barrier without arriving, as a CTA that stopped would; bar[3] > 0 replaces
// the poll limit, so that the other CTAs give up after that many polls.
// Per-warp / per-CTA timing statistics (atomics in the hot loops): collected
// only by builds with FP_TIMING_STATS defined.
#ifdef FP_TIMING_STATS
constexpr bool kTimingStats = true;
#else
constexpr bool kTimingStats = false;
#endif

constexpr unsigned kBarrierSpins = 1u << 21;   // polls of an L2 line with 32 ns naps: about a second or more

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barriers this CTA has entered in this launch (thread 0 only); a kernel
// calls barrier_start() before its first grid_barrier.
static __shared__ unsigned s_barriers;
__device__ __forceinline__ void barrier_start() {
  if (threadIdx.x == 0) s_barriers = 0;
}

__device__ __forceinline__ bool grid_barrier(unsigned* bar, int* status) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned n = ++s_barriers;
    const unsigned leave_at = __ldcg(&bar[1]);
    if (leave_at != 0u && n == leave_at && blockIdx.x == gridDim.x - 1) {
      ok = 0;   // test hook: this CTA stops arriving
    } else {
      const unsigned limit = __ldcg(&bar[3]) != 0u ? __ldcg(&bar[3]) : kBarrierSpins;
      const unsigned inc = blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u;
      __threadfence();
      const unsigned old = atomicAdd(&bar[0], inc);
      unsigned spins = 0;
      while (((old ^ ld_acquire(&bar[0])) & 0x80000000u) == 0u) {
        if ((++spins & 255u) == 0u && (ld_acquire(&bar[2]) != 0u || spins > limit)) {
          ok = 0;
          break;
        }
        __nanosleep(32);
      }
      if (!ok) {
        atomicExch(&bar[2], 1u);
        atomicCAS(status, 0, -4);   // FP_ERR_DEVICE_TIMEOUT
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// 32-bit warp reductions are one redux.sync (22 cycles measured, against about
// 180 for five dependent shuffles).
__device__ __forceinline__ int warp_sum(int x) { return __reduce_add_sync(kAll, x); }
__device__ __forceinline__ int warp_min(int x) { return __reduce_min_sync(kAll, x); }
__device__ __forceinline__ int warp_max(int x) { return __reduce_max_sync(kAll, x); }
// Minimum of a 64-bit key: the high words, then the low words of their holders.
__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long x) {
  const unsigned hi = __reduce_min_sync(kAll, (unsigned)(x >> 32));
  const unsigned lo = __reduce_min_sync(kAll, (unsigned)(x >> 32) == hi ? (unsigned)x : ~0u);
  return ((unsigned long long)hi << 32) | lo;
}
__device__ __forceinline__ long long warp_sum64(long long x) {
  for (int off = 16; off; off >>= 1) x += __shfl_xor_sync(kAll, x, off);
  return x;
}

__device__ __forceinline__ LdgKey warp_ldg_argmax(LdgKey k) {
  for (int off = 16; off; off >>= 1) {
    LdgKey o = shfl_key(k, off);
    if (ldg_better(o, k)) k = o;
  }
  return k;
}

struct Carve {
  unsigned char* p;
  template <class T>
  __device__ T* take(size_t n) {
    T* r = reinterpret_cast<T*>(p);
    p += (n * sizeof(T) + 15) & ~size_t(15);
    return r;
  }
};

// First index >= from of the ascending list `list` (n entries) whose value is
// >= x, or n; every lane of a warp.  One round trip to L2 if it is among the
// next 32 entries, three for up to 1024 (a binary search takes one per step: 2 us
// of every window; with it TM on 262144 Zipf vertices 46.7 -> 40.8 ms per pass,
// MSM on 1M 0.50 -> 0.43, TV there 11.0 -> 10.5 for two).
__device__ __forceinline__ int seek_pos(const int* list, int n, int from, int x) {
  const int lane = threadIdx.x & 31;
  unsigned m = __ballot_sync(kAll, from + lane < n && __ldg(&list[from + lane]) < x);
  from += __popc(m);
  if (m != kAll) return from;
  do {   // blocks of 32 whose last entry is before x
    const int i = from + 32 * lane + 31;
    m = __ballot_sync(kAll, i < n && __ldg(&list[i]) < x);
    from += 32 * __popc(m);
  } while (m == kAll);
  return from + __popc(__ballot_sync(kAll, from + lane < n && __ldg(&list[from + lane]) < x));
}

// Contiguous share [*b, *e) of a vertex's deg nets for warp wi of nw warps
// (balances vertices with few large nets across the warps of a group).
__device__ __forceinline__ void net_range(int deg, int wi, int nw, int* b, int* e) {
  const int g = (deg + nw - 1) / nw;
  *b = min(wi * g, deg);
  *e = min(*b + g, deg);
}

// Splits the grid's ncta CTAs among the window's ns whole-grid vertices (ns <=
// 32) by their nets deg, at least a quarter of an even share each: vertex j's
// team is the CTAs [t0[j], t1[j]) (one CTA of several teams when the grid is
// small).  The first `light` CTAs, which hold the light positions, and the last
// `mid`, which take the medium vertices, are left out where half the grid or more
// remains: theirs would be the window's longest shares (TM on 262144 Zipf vertices
// 41.5 -> 38.1 ms per pass, MSV's evaluation 38.1 -> 36.9 us).  One warp.
__device__ __forceinline__ void team_split(int ns, const int* deg, int ncta, int light, int mid, int* t0, int* t1) {
  const int lane = threadIdx.x & 31;
  const int c0 = 2 * (light + mid) <= ncta ? light : 0;
  const int n = 2 * (light + mid) <= ncta ? ncta - light - mid : ncta;
  const long long d = lane < ns ? deg[lane] : 0;
  const long long all = warp_sum64(d);
  const long long w = lane < ns ? 3 * d + all / ns + 1 : 0;
  long long incl = w;
  for (int off = 1; off < 32; off <<= 1) {
    const long long t = __shfl_up_sync(kAll, incl, off);
    if (lane >= off) incl += t;
  }
  const long long total = __shfl_sync(kAll, incl, 31);
  if (lane < ns) {
    const int a = min((int)((incl - w) * n / total), n - 1);
    t0[lane] = c0 + a;
    t1[lane] = c0 + max((int)(incl * n / total), a + 1);
  }
}

// Sighting keys: the reference breaks ties by the part seen first, in (net,
// slot) order.  A key is the net's index from the start of the tallied range
// above the slot, in 32 bits: shared-memory atomicMin has a native 32-bit form
// (about 50 cycles), the 64-bit one is a compare-and-swap loop (146 cycles
// uncontended).  The slot takes slot_bits(K) bits, so a range holds at most
// key_nets(sb) nets: more than a vertex evaluated by one warp or CTA has (65535
// nets, K <= 4096); a longer share of a whole-grid vertex is tallied in pieces,
// and the pieces meet in 64-bit keys of absolute net indexes (wide_key).
__device__ __forceinline__ int slot_bits(int K) { return 32 - __clz(K - 1); }
__device__ __forceinline__ int key_nets(int sb) { return sb <= 1 ? 0x7fffffff : (int)(1u << (32 - sb)); }
__device__ __forceinline__ unsigned long long wide_key(unsigned f, int sb, int n0) {
  return ((unsigned long long)((unsigned)n0 + (f >> sb)) << 32) | (f & ((1u << sb) - 1u));
}

// Visits the list slots of the nets [n0, n1) of a vertex (base: its offset in
// vnets), one warp, 32 nets at a time: begin(nb, e) for the batch from nb, where
// lane i's net nb + i is e (-1 past n1), then slot(lo, j, part, count) for every
// slot j of the net nb + lo (count: kCounts), then end(nb, e).
//
// The slots of a batch are flattened across the warp (inclusive scan of the
// list lengths), 4 per lane in flight.  A lane finds its slot's list by the
// number of lists that start at or before it: one redux.sync over the starts
// that fall in its 32 slots (a binary search over the scan takes five dependent
// shuffles).  Lists are short (about five slots), so a batch is mostly the chain
// net -> list -> slots: the next batch's nets and list heads are loaded before
// this one's slots.  Windows of 1M Zipf vertices under TV 106 -> 100 us of
// evaluation, of 262144 under MSRV 51.7 -> 49.7, MSV 42.3 -> 40.4; the message
// metrics' evaluation gains nothing by it and keeps its own pass.
template <bool kCounts, class Begin, class Slot, class End>
__device__ __forceinline__ void for_slots(const DevInstance& I, uint32_t base, int n0, int n1, Begin&& begin,
                                          Slot&& slot, End&& end) {
  const int lane = threadIdx.x & 31;
  auto net = [&](int k) { return k < n1 ? (int)__ldg(&I.vnets[base + k]) : -1; };
  int e = net(n0 + lane), e1 = net(n0 + 32 + lane);
  int s = 0, s_end = 0, n = 0;
  auto head = [&](int x) {
    s = x >= 0 ? (int)__ldg(&I.nptr[x]) : 0;
    s_end = x >= 0 ? (int)__ldg(&I.nptr[x + 1]) : 0;
    n = x >= 0 ? lds(&I.ep_len[x]) : 0;
  };
  head(e);
  for (int nb = n0; nb < n1; nb += 32) {
    const int ec = e, sc = s;
    int nc = n;
    if (nc < 0 || nc > s_end - s) {
      dev_fail(I.status, kDevErrInvalid);
      nc = 0;
    }
    e = e1;
    e1 = net(nb + 64 + lane);
    head(e);
    begin(nb, ec);
    int incl = nc;
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(kAll, incl, off);
      if (lane >= off) incl += t;
    }
    const int total = __shfl_sync(kAll, incl, 31), start = incl - nc;
    // lane x: the x-th list that has slots (its lane, first flat slot and address)
    const unsigned has = __ballot_sync(kAll, nc > 0);
    int xl = lane, xs = start, xa = sc - start;
    if (has & (has + 1)) {   // some list before others is empty
      int rank = lane, at = 0;
#pragma unroll
      for (int w = 16; w; w >>= 1) {
        const int c = __popc(has & (((1u << w) - 1u) << at));
        if (rank >= c) {
          rank -= c;
          at += w;
        }
      }
      xl = at;
      xs = __shfl_sync(kAll, xs, at);
      xa = __shfl_sync(kAll, xa, at);
    }
    int before = -1;   // lists that start before the 32 slots at hand, minus one
    constexpr int kU = 4;
    for (int f0 = 0; f0 < total; f0 += 32 * kU) {
      int lo[kU], jj[kU], aa[kU], pp[kU], cc[kU];
#pragma unroll
      for (int u = 0; u < kU; u++) {
        const int f = f0 + u * 32;
        const unsigned st = (unsigned)(start - f);
        const unsigned m = __reduce_or_sync(kAll, nc > 0 && st < 32u ? 1u << st : 0u);
        const int x = before + __popc(m & (0xffffffffu >> (31 - lane)));
        before += __popc(m);
        lo[u] = __shfl_sync(kAll, xl, x);
        jj[u] = f + lane - __shfl_sync(kAll, xs, x);
        const int a = __shfl_sync(kAll, xa, x);
        aa[u] = f + lane < total ? a + f + lane : -1;
      }
#pragma unroll
      for (int u = 0; u < kU; u++) {   // parts and counts together: one round trip
        pp[u] = aa[u] >= 0 ? lds(&I.ep_part[aa[u]]) : -1;
        cc[u] = kCounts && aa[u] >= 0 ? lds(&I.ep_cnt[aa[u]]) : 0;
      }
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (aa[u] >= 0) slot(lo[u], jj[u], pp[u], cc[u]);
    }
    end(nb, ec);
  }
}

// Adds to the part tally the nets [n0, n1) of a vertex: for every listed part,
// the number of nets listing it (cnt) and the sighting key of its first one
// (first; net indexes from k0).  Returns this lane's count of nets where `own`
// has exactly one pin.
template <bool kOwn>
__device__ __forceinline__ int tally_range(const DevInstance& I, int own, uint32_t base, int n0, int n1, int k0, int sb,
                                           int* cnt, unsigned* first) {
  const int K = I.K;
  int c1 = 0, nk = 0;
  for_slots<kOwn>(
      I, base, n0, n1, [&](int nb, int) { nk = nb - k0; },
      [&](int lo, int j, int p, int c) {
        if ((unsigned)p >= (unsigned)K) {
          dev_fail(I.status, kDevErrInvalid);
          return;
        }
        atomicAdd(&cnt[p], 1);
        atomicMin(&first[p], ((unsigned)(nk + lo) << sb) | (unsigned)j);
        if (kOwn && p == own && c == 1) c1++;
      },
      [](int, int) {});
  return c1;
}

// Record of one (vertex, net) pair of a vertex about to move own -> d, one
// 32-bit word at the pair's vnets index: the slot of `own` in the net's list,
// the slot of `d` (kNoSlot: not listed), own's count there is 1 (the move takes
// own off the list), v is the net's source.  The slots stay valid until the
// move is committed: a net whose part set changes has no other mover in the
// round, and count-only moves never move slots.
constexpr uint32_t kNoSlot = 0x1fffu;   // slots < K <= 4096
__device__ __forceinline__ uint32_t rec_pack(int jo, int jd, bool rem, bool src) {
  return (uint32_t)jo | ((uint32_t)(jd < 0 ? kNoSlot : (uint32_t)jd) << 13) | (rem ? 1u << 26 : 0u) |
         (src ? 1u << 27 : 0u);
}
__device__ __forceinline__ int rec_jo(uint32_t r) { return (int)(r & 0x1fffu); }
__device__ __forceinline__ int rec_jd(uint32_t r) {
  const uint32_t j = (r >> 13) & 0x1fffu;
  return j == kNoSlot ? -1 : (int)j;
}
__device__ __forceinline__ bool rec_rem(uint32_t r) { return (r >> 26) & 1u; }
__device__ __forceinline__ bool rec_add(uint32_t r) { return ((r >> 13) & 0x1fffu) == kNoSlot; }
__device__ __forceinline__ bool rec_src(uint32_t r) { return (r >> 27) & 1u; }
// The move changes the net's part set (or, with volumes, the net's send side).
__device__ __forceinline__ bool rec_setchange(uint32_t r, bool vol) {
  return rec_rem(r) || rec_add(r) || (vol && rec_src(r));
}

// Writes the records of the nets [n0, n1) of v for the move own -> d into
// rec[base + k] (one warp); each(e, r) gets every lane's net and record.
// loc: 96 ints of per-warp scratch.
template <class Each>
__device__ __forceinline__ void locate_nets(const DevInstance& I, uint32_t* rec, int v, int own, int d, uint32_t base,
                                            int n0, int n1, int* loc, Each&& each) {
  const int lane = threadIdx.x & 31;
  int* const sj = loc;
  int* const sd = loc + 32;
  int* const sc = loc + 64;
  for_slots<true>(
      I, base, n0, n1,
      [&](int, int) {
        sj[lane] = -1;
        sd[lane] = -1;
        sc[lane] = 0;
        __syncwarp();
      },
      [&](int lo, int j, int p, int c) {
        // own and d are listed at most once per net: one writer per entry
        if (p == own) {
          sj[lo] = j;
          sc[lo] = c == 1;
        }
        if (p == d) sd[lo] = j;
      },
      [&](int nb, int e) {
        __syncwarp();
        if (e >= 0) {
          const int jo = sj[lane];
          uint32_t r = 0;
          if (jo < 0) {
            dev_fail(I.status, kDevErrInvalid);   // v's own part must be listed on v's nets
          } else {
            r = rec_pack(jo, sd[lane], sc[lane] != 0, __ldg(&I.src[e]) == v);
            rec[base + nb + lane] = r;
          }
          each(e, r);
        }
        __syncwarp();
      });
}

// Volume arrays updated while a vertex moves (MSV: send only; MSRV: both).
struct Vol {
  int* send;
  int* recv;
};

// commit_net with the slots taken from the move's record (no list search).
__device__ __forceinline__ void commit_rec(const DevInstance& I, int v, int own, int d, int e, uint32_t r,
                                           const Vol* vol) {
  const int s = (int)__ldg(&I.nptr[e]);
  const int cap = (int)__ldg(&I.nptr[e + 1]) - s;
  int n = lds(&I.ep_len[e]);
  const int jo = rec_jo(r);
  int jd = rec_jd(r);
  if (jo >= n || jd >= n || n > cap || (jd < 0 && n == cap && !rec_rem(r))) {
    dev_fail(I.status, kDevErrInvalid);
    return;
  }
  const int sv = vol ? __ldg(&I.src[e]) : -1;
  const int sp = (vol && sv != v) ? lds(&I.part_vec[sv]) : d;
  if (vol && sv == v) atomicAdd(&vol->send[own], -(n - 1));
  const int co = atomicAdd(&I.ep_cnt[s + jo], -1) - 1;
  if (co == 0) {
    const int last = n - 1;
    I.ep_part[s + jo] = lds(&I.ep_part[s + last]);
    I.ep_cnt[s + jo] = lds(&I.ep_cnt[s + last]);
    I.ep_part[s + last] = -1;
    I.ep_cnt[s + last] = 0;
    if (jd == last) jd = jo;
    n = last;
    if (vol && sv != v) {
      atomicAdd(&vol->send[sp], -1);
      if (vol->recv) atomicAdd(&vol->recv[own], -1);
    }
  } else {
    if (vol && vol->recv && sv == v) atomicAdd(&vol->recv[own], 1);
  }
  if (vol && sv == v) atomicAdd(&vol->send[d], n - 1);
  if (jd >= 0) {
    atomicAdd(&I.ep_cnt[s + jd], 1);
    if (vol && vol->recv && sv == v) atomicAdd(&vol->recv[d], -1);
  } else {
    I.ep_part[s + n] = d;
    I.ep_cnt[s + n] = 1;
    n++;
    if (vol) {
      atomicAdd(&vol->send[sp], 1);
      if (vol->recv && sv != v) atomicAdd(&vol->recv[d], 1);
    }
  }
  if (co == 0 || jd < 0) I.ep_len[e] = n;
}

// One thread applies vertex v's move own -> d to net e: the reference's
// REMOVAL (decrement, swap-with-last when the count reaches zero) then ADDING
// (increment or append), TV/partition.cpp:388-436, with the send / received
// volume bookkeeping of MGV/partition.cpp:376-449 and MSRV/partition.cpp:387-483.
__device__ __forceinline__ void commit_net(const DevInstance& I, int v, int own, int d, int e, const Vol* vol) {
  const int s = (int)__ldg(&I.nptr[e]);
  const int cap = (int)__ldg(&I.nptr[e + 1]) - s;
  int n = lds(&I.ep_len[e]);
  int jo = -1, jd = -1;
  for (int j = 0; j < n && (jo < 0 || jd < 0); j++) {
    const int p = lds(&I.ep_part[s + j]);
    if (p == own) jo = j;
    if (p == d) jd = j;
  }
  if (jo < 0 || n > cap || (jd < 0 && n == cap && lds(&I.ep_cnt[s + jo]) > 1)) {
    dev_fail(I.status, kDevErrInvalid);
    return;
  }
  const int sv = vol ? __ldg(&I.src[e]) : -1;
  const int sp = (vol && sv != v) ? lds(&I.part_vec[sv]) : d;
  if (vol && sv == v) atomicAdd(&vol->send[own], -(n - 1));
  // Counts change atomically: movers committed in the same round may share a net
  // on which they only shift counts (their part sets are disjoint there).
  const int co = atomicAdd(&I.ep_cnt[s + jo], -1) - 1;
  if (co == 0) {
    const int last = n - 1;
    I.ep_part[s + jo] = lds(&I.ep_part[s + last]);
    I.ep_cnt[s + jo] = lds(&I.ep_cnt[s + last]);
    I.ep_part[s + last] = -1;
    I.ep_cnt[s + last] = 0;
    if (jd == last) jd = jo;
    n = last;
    if (vol && sv != v) {
      atomicAdd(&vol->send[sp], -1);
      if (vol->recv) atomicAdd(&vol->recv[own], -1);
    }
  } else {
    if (vol && vol->recv && sv == v) atomicAdd(&vol->recv[own], 1);
  }
  if (vol && sv == v) atomicAdd(&vol->send[d], n - 1);
  if (jd >= 0) {
    atomicAdd(&I.ep_cnt[s + jd], 1);
    if (vol && vol->recv && sv == v) atomicAdd(&vol->recv[d], -1);
  } else {
    I.ep_part[s + n] = d;
    I.ep_cnt[s + n] = 1;
    n++;
    if (vol) {
      atomicAdd(&vol->send[sp], 1);
      if (vol->recv && sv != v) atomicAdd(&vol->recv[d], 1);
    }
  }
  I.ep_len[e] = n;
}

// One warp applies v's move own -> d to the list of net e (REMOVAL then ADDING,
// as commit_net, without volumes); the lanes search the slots of own and d
// together.  The net must have no other mover at the same time.  Returns the
// list length after the move (every lane).
__device__ __forceinline__ int commit_net_warp(const DevInstance& I, int own, int d, int e) {
  const int lane = threadIdx.x & 31;
  const int s = (int)__ldg(&I.nptr[e]);
  const int cap = (int)__ldg(&I.nptr[e + 1]) - s;
  int n = lds(&I.ep_len[e]);
  int jo = -1, jd = -1;
  for (int j0 = 0; j0 < n; j0 += 32) {
    const int j = j0 + lane;
    const int p = j < n ? lds(&I.ep_part[s + j]) : -1;
    const unsigned mo = __ballot_sync(kAll, p == own);
    const unsigned md = __ballot_sync(kAll, p == d);
    if (mo && jo < 0) jo = j0 + __ffs(mo) - 1;
    if (md && jd < 0) jd = j0 + __ffs(md) - 1;
  }
  const int co = jo >= 0 ? lds(&I.ep_cnt[s + jo]) : 0;
  if (jo < 0 || n > cap || (jd < 0 && n == cap && co > 1)) {
    if (lane == 0) dev_fail(I.status, kDevErrInvalid);
    return n;
  }
  if (lane == 0) {
    if (co == 1) {
      const int last = n - 1;
      I.ep_part[s + jo] = lds(&I.ep_part[s + last]);
      I.ep_cnt[s + jo] = lds(&I.ep_cnt[s + last]);
      I.ep_part[s + last] = -1;
      I.ep_cnt[s + last] = 0;
      if (jd == last) jd = jo;
      n = last;
    } else {
      I.ep_cnt[s + jo] = co - 1;
    }
    if (jd >= 0) {
      I.ep_cnt[s + jd] = lds(&I.ep_cnt[s + jd]) + 1;
    } else {
      I.ep_part[s + n] = d;
      I.ep_cnt[s + n] = 1;
      n++;
    }
    I.ep_len[e] = n;
  }
  n = __shfl_sync(kAll, n, 0);
  __syncwarp();
  return n;
}

// Least-loaded part (lowest index on ties) and the second smallest size, for
// the LDG fallback (TV/partition.cpp:118-132) and its drift margin.
__device__ __forceinline__ void block_min_part(const int* sizes, int K, unsigned long long* scr, int* minpart,
                                               int* minsize, int* second) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  unsigned long long mk = ~0ull;
  for (int p = threadIdx.x; p < K; p += blockDim.x) {
    const unsigned long long key = ((unsigned long long)((unsigned)sizes[p] ^ 0x80000000u) << 32) | (unsigned)p;
    mk = key < mk ? key : mk;
  }
  mk = warp_min_u64(mk);
  __syncthreads();
  if (lane == 0) scr[wib] = mk;
  __syncthreads();
  mk = scr[0];
  for (int x = 1; x < (int)(blockDim.x >> 5); x++) mk = scr[x] < mk ? scr[x] : mk;
  const int mp = (int)(mk & 0xffffffffu);
  int s2 = 0x7fffffff;
  for (int p = threadIdx.x; p < K; p += blockDim.x)
    if (p != mp) s2 = min(s2, sizes[p]);
  s2 = warp_min(s2);
  __syncthreads();
  if (lane == 0) scr[wib] = (unsigned long long)(unsigned)s2;
  __syncthreads();
  int m2 = 0x7fffffff;
  for (int x = 0; x < (int)(blockDim.x >> 5); x++) m2 = min(m2, (int)(unsigned)scr[x]);
  __syncthreads();
  *minpart = mp;
  *minsize = sizes[mp];
  *second = m2;
}

}  // namespace spec
}  // namespace fp
