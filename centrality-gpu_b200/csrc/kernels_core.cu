// Per-source schedule on chain-contracted BCCs: one source per CTA at a time,
// FP64, every sweep over the core vertices (those off degree-2 chains) only.
//
// The reference sweeps every vertex of a BCC for every source, and merges the
// two ends' rows for a source on a chain (Codes/kernels_free.cu:154-473,
// Codes/kernels_active.cu:263-602, Codes/postprocesses.cu:205-470). Here a
// chain of k vertices is one arc of length k+1 between its ends:
//  * forward: level-synchronous over unit arcs as ever; a vertex found over a
//    chain arc is due k+1 levels later and waits in the bucket of that level
//    (one bucket per level still ahead, reused in a ring), where it counts only
//    if nothing reached it before. A bit per core vertex in shared memory says
//    whether it has its level yet: claims need no trip to L2, and only vertices
//    that have theirs are looked at for path counts.
//  * a source on a chain enters the core at both ends of its chain, due on
//    levels p+1 and k-p: no merge, no second BFS.
//  * chains, between the sweeps: each chain is walked once from the vertex where
//    the two ends' waves meet to either end, adding weights (sums of positive
//    terms throughout); that vertex shares its weight in proportion to the path
//    counts of the ends when they meet on it (Codes/postprocesses.cu:334-350).
//    The walk gives the chain vertices' dependencies and what each end receives.
//    A chain that carries shortest paths from one end to the other needs the
//    far end's q, so its vertices are left until after the backward sweep.
//  * backward: successor form as in kernels_plain.cu, where a chain arc is a
//    successor arc if the far end's shortest paths run through the chain, plus
//    what the chains give.
// Path counts carry a power of two per level as in kernels_plain.cu, with the
// same threshold. BC goes into the fixed-point counters (accum.cuh): the
// result does not depend on which CTA ran which source.
//
// What bounds it: round trips to L2 (700 cycles and more) and the instructions
// of the few warps that a level keeps busy, since a level is rarely wider than
// the CTA and each waits for the one before. So a frontier comes from shared
// memory, a short row brings its arcs with it, a record {key, path count then
// q} is one 16-byte load, and what can wait runs off the level loop with every
// lane busy: the chains, and the additions into the counters (a level only
// stores its dependencies). Long rows have one loop, not one per place that
// finds them: with 16 CTAs at different points of the kernel, instruction
// fetches were a quarter of the stalls. Against the whole-BCC kernel: an 80x80
// grid 31.2 -> 14.9 ms (14,867 sources), 2,870 sources of a 512x512 grid 356 ->
// 123 ms, 7,867 sources of R-MAT 14 with 20% chains 233 -> 91 ms. Without chains to
// contract it is the slower of the two (bcgpu.cu contracts()).
#include "accum.cuh"
#include "common.cuh"
#include "core.h"

#include <algorithm>
#include <climits>

namespace bcg {

namespace {

constexpr int kLight = 8;        // rows up to this many arcs: one thread, kCoreShort arcs in flight
constexpr int kWarpRow = 1024;   // rows up to this many: a warp; longer: the CTA
constexpr int kCtaQueue = 64;    // queue of the rows of a level the whole CTA takes one by one: the first ones

// A vertex's record in global memory, one 32-byte sector: its key, its path
// count (then q), its path count once more, its dependency.
struct __align__(32) Rec {
  int32_t key, pad;
  double v, sig, dep;
};

// A neighbour as its first load brings it: key, and path count or q.
struct Seen {
  int32_t key;
  double v;
};

template <int kBlock>
struct Shared {
  static constexpr int kQueue = kBlock < 128 ? 64 : kBlock < 256 ? 256 : 512;
  static constexpr int kRing = kBlock < 512 ? 8 * kBlock : 4096;
  static constexpr int kFront = 2 * kBlock;
  double red[2][kBlock / 32];
  int found[3];              // by level mod 3: vertices found for the next level
  int nwq[3], ncq[3];        // by level mod 3: queued long rows
  int emax[3];               // by level mod 3: largest exponent field beyond the rescaling threshold (0: none)
  int bucket[kCoreMaxChain + 3];  // entries of the buckets
  int nvia;
  int base;
  int64_t item;
  int wq[kQueue];            // long rows of a level: the first ones
  int cq[kCtaQueue];
  int front[2][kFront];      // by level parity: the first vertices of a level; all are in the slot's order
  int ring[kRing];           // the first entries of each bucket; the rest are in the slot
};

// The level loops have to stay in the instruction cache, with many CTAs in
// different parts of the kernel: what is rare, and what is long, is out of line.
__device__ __noinline__ double scaled_by(double v, int e) { return scale2(v, e); }
__device__ __forceinline__ double scaled(double v, int e) { return e ? scaled_by(v, e) : v; }

struct Slot {
  Rec *rec;
  double *in;                // [2 * chain + side] what the chain's own vertices give each end (side 1: right)
  int32_t *via;              // chains whose vertices wait for the backward sweep
  uint32_t *bits;            // shared memory: vertices that have their level
  int32_t *order, *ring;     // vertices by level; the buckets past their first entries
  int32_t *rows;             // long rows of a level past the first ones (queue_row)
  int32_t *lv, *lx;          // level offsets into order; level exponents
  int64_t bcap;
  int32_t scap;              // entries of a bucket in shared memory
  __device__ __forceinline__ Seen seen(int32_t u) const {
    const int4 x = __ldcg(reinterpret_cast<const int4 *>(rec + u));
    return Seen{x.x, __hiloint2double(x.w, x.z)};
  }
};

__device__ __forceinline__ Slot slot_of(const CoreArgs &a, unsigned char *smem, int ring_ints) {
  const auto &h = a.shape;
  unsigned char *p = a.ws + (int64_t)blockIdx.x * h.rest_bytes();
  Slot s;
  s.bcap = h.bcap;
  s.scap = ring_ints / h.ring;
  s.rec = reinterpret_cast<Rec *>(a.rec + (int64_t)blockIdx.x * h.rec_bytes());
  s.bits = reinterpret_cast<uint32_t *>(smem);
  s.in = reinterpret_cast<double *>(p);
  s.via = reinterpret_cast<int32_t *>(s.in + 2 * h.ccap);
  s.order = s.via + h.ccap;
  s.rows = s.order + h.cap;
  s.ring = s.rows + h.cap;
  s.lv = s.ring + (int64_t)h.ring * h.bcap;
  s.lx = s.lv + h.tcap + 3;
  return s;
}

// The BCC and source a CTA works on (uniform).
struct View {
  const CoreRow *rows;
  const int32_t *col, *k, *cid;  // from the BCC's first arc on
  const int32_t *reach;          // of the BCC's vertices
  int32_t ncore;
  int top;            // key of level 0
  int32_t own, pos, len;  // the source's chain (-1: a core source), its place on it, the chain's length
  int32_t endl, endr;
  bool scaled;        // some level of this source carries an exponent (backward)
  int64_t chain0;     // the BCC's first chain
};

// The head of a row: first arc, arcs, part, reach.
struct Head {
  int32_t e0, deg, part, reach;
};
__device__ __forceinline__ Head head_of(const View &g, int32_t v) {
  const int4 r = __ldg(reinterpret_cast<const int4 *>(g.rows + v));
  return Head{r.x, r.y, r.z, r.w};
}
// kCoreShort arcs of a row: far ends (-1: none), chain lengths and, backward,
// chain * 2 + side (-1: no chain).
struct Arcs {
  int32_t u[kCoreShort], k[kCoreShort], cid[kCoreShort];
};
// All arcs of a short row (of another, nothing of use): loaded with its head.
template <bool kBack>
__device__ __forceinline__ Arcs arcs_with(const View &g, int32_t v, const Head &h) {
  const int4 u = __ldg(reinterpret_cast<const int4 *>(g.rows[v].u));
  const int4 c = kBack ? __ldg(reinterpret_cast<const int4 *>(g.rows[v].cid)) : make_int4(-1, -1, -1, -1);
  Arcs r{{u.x, u.y, u.z, u.w}, {}, {c.x, c.y, c.z, c.w}};
#pragma unroll
  for (int j = 0; j < kCoreShort; ++j) r.k[j] = (h.part >> (8 * j)) & 0xff;
  return r;
}
// Arcs j0, j0 + step, ... of a longer row.
template <bool kBack>
__device__ __forceinline__ void arcs_from(const View &g, const Head &h, int j0, int step, Arcs &r) {
#pragma unroll
  for (int j = 0; j < kCoreShort; ++j) {
    const int e = j0 + j * step;
    const bool on = e < h.deg, ch = on && e >= h.part;
    r.u[j] = on ? ldg(g.col + h.e0 + e) : -1;
    r.k[j] = ch ? ldg(g.k + h.e0 + e) : 0;
    r.cid[j] = kBack && ch ? ldg(g.cid + h.e0 + e) : -1;
  }
}

// ================================================================ forward ===

// Level l of a forward sweep, the same for the whole CTA.
struct Level {
  int l, m, bk;  // l, l mod 3, l mod the ring
  int f1;        // end of the level's vertices in the order: those of the next level go there
  int x;         // exponent of the level before
};

// u gets level l+1: into its list.
template <class SH>
__device__ __forceinline__ void fwd_found(SH &sh, const Slot &w, const View &g, const Level &L, int32_t u) {
  w.rec[u].key = g.top - L.l - 1;
  const int at = atomicAdd(&sh.found[L.m], 1);
  w.order[L.f1 + at] = u;
  if (at < SH::kFront) sh.front[(L.l + 1) & 1][at] = u;
}
__device__ __forceinline__ bool claim(const Slot &w, int32_t u) {
  const uint32_t bit = 1u << (u & 31);
  return !(atomicOr(w.bits + (u >> 5), bit) & bit);
}
template <class SH>
__device__ __forceinline__ void bucket_add(SH &sh, const Slot &w, int b, int32_t u) {
  const int at = atomicAdd(&sh.bucket[b], 1);
  if (at < w.scap) sh.ring[b * w.scap + at] = u;
  else w.ring[(int64_t)b * w.bcap + at] = u;
}
template <class SH>
__device__ __forceinline__ int32_t bucket_get(const SH &sh, const Slot &w, int b, int at) {
  return at < w.scap ? sh.ring[b * w.scap + at] : w.ring[(int64_t)b * w.bcap + at];
}

// u is due on level l+1+k unless something reaches it before: into that bucket.
template <class SH>
__device__ __forceinline__ void fwd_later(SH &sh, const CoreArgs &a, const Slot &w, const Level &L, int32_t u, int k) {
  int b = L.bk + 1 + k;
  if (b >= a.shape.ring) b -= a.shape.ring;
  bucket_add(sh, w, b, u);
}

template <class SH>
__device__ __forceinline__ void fwd_done(SH &sh, const CoreArgs &a, const Slot &w, const View &g, int32_t x, const Level &L,
                                         double sum) {
  if (g.own >= 0) {  // the source's own chain brings one path to each of its ends
    if ((x == g.endl && L.l == g.pos + 1) || (x == g.endr && L.l == g.len - g.pos)) sum += scaled(1.0, -L.x);
  } else if (L.l == 0) {
    sum = 1.0;
  }
  w.rec[x].v = sum;
  w.rec[x].sig = sum;
  const int e = exp_bits(sum);
  if (e - 1023 > a.rescale_exp || e == 0x7ff) atomicMax(&sh.emax[L.m], e);
}

// Queues a long row of the level, by its length alone: the CTA and a warp sum a
// row in different orders, and the order of the queue is not the same twice. The
// slot's list holds a warp's rows from the front and the CTA's from the back (its
// end is the start of the ring); together they are no more than the level.
template <int kBlock>
__device__ __forceinline__ void queue_row(Shared<kBlock> &sh, const Slot &w, int m, int32_t v, int deg) {
  if (deg > kWarpRow) {
    const int at = atomicAdd(&sh.ncq[m], 1);
    if (at < kCtaQueue) sh.cq[at] = v;
    else w.ring[-1 - at] = v;
    return;
  }
  const int at = atomicAdd(&sh.nwq[m], 1);
  if (at < Shared<kBlock>::kQueue) sh.wq[at] = v;
  else w.rows[at] = v;
}

// The queued rows of a level, the very long ones by the whole CTA, the others by
// a warp each: row(v, head, first arc, step) sums arcs, done(v, head, sums)
// takes the result in one thread. Two sums, in an order that the row's length fixes.
template <int kBlock, class Row, class Done>
__device__ __forceinline__ void long_rows(Shared<kBlock> &sh, const Slot &w, const View &g, int nc, int nw, Row row,
                                          Done done) {
  constexpr int kWarps = kBlock / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rounds = nc + (nw + kWarps - 1) / kWarps;
  for (int r = 0; r < rounds; ++r) {
    const bool all = r < nc;
    const int at = all ? r : (r - nc) * kWarps + warp;
    const bool on = all || at < nw;
    const int32_t v = !on                                                 ? 0
                      : at < (all ? kCtaQueue : Shared<kBlock>::kQueue) ? (all ? sh.cq : sh.wq)[at]
                                                                        : (all ? w.ring[-1 - at] : w.rows[at]);
    const Head h = head_of(g, v);
    double x = 0.0, y = 0.0;
    if (on) row(h, all ? tid : lane, all ? kBlock : 32, x, y);
    x = warp_sum(x);
    y = warp_sum(y);
    if (all) {
      if (lane == 0) {
        sh.red[0][warp] = x;
        sh.red[1][warp] = y;
      }
      __syncthreads();
      x = y = 0.0;
      for (int i = 0; i < kWarps; ++i) {
        x += sh.red[0][i];
        y += sh.red[1][i];
      }
      __syncthreads();
    }
    if (on && (all ? tid : lane) == 0) done(v, h, x, y);
  }
}

// Arcs j0, j0 + step, ... of a vertex of the level (a short row's: r), kCoreShort at a time: the
// path counts of the far ends that have their levels; claims of the others. The
// loads and the claims of a group are in flight together.
template <class SH>
__device__ __forceinline__ double fwd_arcs(SH &sh, const CoreArgs &a, const Slot &w, const View &g, const Level &L,
                                           const Head &h, Arcs r, int j0, int step) {
  double sum = 0.0;
  for (; j0 < h.deg; j0 += kCoreShort * step) {
    if (h.deg > kCoreShort) arcs_from<false>(g, h, j0, step, r);
    Seen s[kCoreShort];
    uint32_t found = 0, later = 0;
#pragma unroll
    for (int j = 0; j < kCoreShort; ++j) {
      s[j] = Seen{INT_MIN, 0.0};
      if (r.u[j] < 0) continue;
      const uint32_t bit = 1u << (r.u[j] & 31);
      uint32_t *word = w.bits + (r.u[j] >> 5);
      if (*(volatile uint32_t *)word & bit) s[j] = w.seen(r.u[j]);
      else if (r.k[j]) later |= 1u << j;
      else if (!(atomicOr(word, bit) & bit)) found |= 1u << j;
    }
#pragma unroll
    for (int j = 0; j < kCoreShort; ++j)
      if (s[j].key == g.top - L.l + 1 + r.k[j]) sum += r.k[j] && L.x ? scaled(s[j].v, w.lx[L.l - 1 - r.k[j]] - L.x) : s[j].v;
    for (uint32_t any = found | later; any; any &= any - 1) {
      const int j = __ffs(any) - 1;
      const int32_t u = j == 0 ? r.u[0] : j == 1 ? r.u[1] : j == 2 ? r.u[2] : r.u[3];
      const int k = j == 0 ? r.k[0] : j == 1 ? r.k[1] : j == 2 ? r.k[2] : r.k[3];
      if (k) fwd_later(sh, a, w, L, u, k);
      else fwd_found(sh, w, g, L, u);
    }
  }
  return sum;
}

// BFS of the CTA from the view's source over the core. Returns the last level
// (-1 on an error), lv and lx filled up to it.
template <int kBlock>
__device__ int core_bfs(Shared<kBlock> &sh, const CoreArgs &a, const Slot &w, View &g, int32_t src) {
  const int tid = threadIdx.x;
  for (int i = tid; i < (g.ncore + 127) / 128; i += kBlock) reinterpret_cast<uint4 *>(w.bits)[i] = make_uint4(0, 0, 0, 0);
  for (int i = tid; i < a.shape.ring; i += kBlock) sh.bucket[i] = 0;
  if (tid < 3) { sh.found[tid] = 0; sh.nwq[tid] = 0; sh.ncq[tid] = 0; sh.emax[tid] = 0; }
  __syncthreads();
  if (tid == 0) {
    w.lv[0] = 0;
    if (g.own < 0) {
      w.bits[src >> 5] |= 1u << (src & 31);
      w.rec[src].key = g.top;
      w.order[0] = sh.front[0][0] = src;
    } else {
      bucket_add(sh, w, (g.pos + 1) % a.shape.ring, g.endl);
      bucket_add(sh, w, (g.len - g.pos) % a.shape.ring, g.endr);
    }
  }
  __syncthreads();
  int l = 0, bk = 0, m = 0, f0 = 0, f1 = g.own < 0 ? 1 : 0, x = 0;  // x: exponent of the level before
  while (true) {
    const int nxt = m == 2 ? 0 : m + 1, due = bk + 1 == a.shape.ring ? 0 : bk + 1;
    const Level L{l, m, bk, f1, x};
    const int total = f1 - f0;
    if (tid == 0) {  // counters of the level ahead: last read two barriers ago
      sh.found[nxt] = 0;
      sh.nwq[nxt] = 0;
      sh.ncq[nxt] = 0;
      sh.emax[nxt] = 0;
      sh.bucket[bk] = 0;  // drained; filled again from two levels on at the earliest
      w.lv[l + 1] = f1;
    }
    for (int c0 = 0; c0 < total; c0 += kBlock) {
      const int i = c0 + tid;
      if (i >= total) continue;
      const int32_t v = i < Shared<kBlock>::kFront ? sh.front[l & 1][i] : w.order[f0 + i];
      const Head h = head_of(g, v);
      const Arcs r = arcs_with<false>(g, v, h);
      if (h.deg <= kLight) fwd_done(sh, a, w, g, v, L, fwd_arcs(sh, a, w, g, L, h, r, 0, 1));
      else queue_row(sh, w, m, v, h.deg);
    }
    __syncthreads();
    const int nw = sh.nwq[m], nc = sh.ncq[m];
    if (nw | nc) {
      long_rows(sh, w, g, nc, nw,
                [&](const Head &h, int j0, int step, double &x, double &) { x = fwd_arcs(sh, a, w, g, L, h, Arcs{}, j0, step); },
                [&](int32_t v, const Head &, double x, double) { fwd_done(sh, a, w, g, v, L, x); });
      __syncthreads();
    }
    const int nd = sh.bucket[due];
    if (nd) {  // vertices due on the next level that nothing has reached
      for (int i = tid; i < nd; i += kBlock) {
        const int32_t u = bucket_get(sh, w, due, i);
        if (claim(w, u)) fwd_found(sh, w, g, L, u);
      }
      __syncthreads();
    }
    const int big = sh.emax[m], found = sh.found[m];
    int xl = x;
    if (big) {  // uniform: the level's counts are divided by a power of two
      if (big == 0x7ff) {
        set_err(a.err, kDevOverflow);
      } else {
        const int s = big - 1023;
        xl += s;
        bool lost = false;
        for (int i = tid; i < total; i += kBlock) {
          const int32_t v = w.order[f0 + i];
          const double y = scaled(w.rec[v].sig, -s);
          lost |= exp_bits(y) == 0;
          w.rec[v].v = y;
          w.rec[v].sig = y;
        }
        if (lost) set_err(a.err, kDevOverflow);
        g.scaled = true;
      }
    }
    if (tid == 0) w.lx[l] = xl;
    x = xl;
    if ((found == 0 && f1 >= g.ncore) || l + 2 > a.shape.tcap) {
      __syncthreads();
      if (f1 >= g.ncore) return l;
      if (tid == 0) set_err(a.err, kDevDisconnected);  // a connected BCC takes at most tcap levels
      return -1;
    }
    if (big) __syncthreads();  // rescaled counts and lx before the next level reads them
    f0 = f1;
    f1 += found;
    ++l;
    m = nxt;
    bk = due;
  }
}

// ================================================================ chains ===

struct End {
  int d, x;  // level, exponent of the level
  double s;  // path count
};

// Dependencies of the m vertices st .. st+m-1 (local ids) between ends A (next
// to st) and B, into the counters: from the vertex where the ends' waves meet
// outwards, each vertex has what the vertices behind it gave. ca, cb: what
// comes in at the outermost vertex fed from A, from B (through the chain, or 0);
// on return what A, B receive.
__device__ __forceinline__ void walk(const View &g, int32_t st, int m, const End &A, const End &B, double wsrc,
                                     unsigned long long *acc, int *err, double &ca, double &cb) {
  const int d = B.d + m - A.d - 1;  // vertex j is fed from A if 2j < d, from B if 2j > d
  const bool tie = d >= 0 && (d & 1) == 0 && (d >> 1) < m;
  const int from_a = tie ? d >> 1 : d < 0 ? 0 : min(m, (d >> 1) + 1);  // vertices 0 .. from_a - 1 are fed from A
  if (tie) {
    const double wt = (double)ldg(g.reach + st + from_a) + 1.0;
    ca = wt / (1.0 + scaled(B.s / A.s, B.x - A.x));
    cb = wt / (1.0 + scaled(A.s / B.s, A.x - B.x));
  }
  for (int j = from_a - 1; j >= 0; --j) {
    if (ca != 0.0) acc_add(acc + (int64_t)kAccDigits * (st + j), ca * wsrc, err);
    ca += (double)ldg(g.reach + st + j) + 1.0;
  }
  for (int j = from_a + (tie ? 1 : 0); j < m; ++j) {
    if (cb != 0.0) acc_add(acc + (int64_t)kAccDigits * (st + j), cb * wsrc, err);
    cb += (double)ldg(g.reach + st + j) + 1.0;
  }
}

__device__ __forceinline__ End end_of(const Slot &w, const View &g, int32_t v) {
  const int d = g.top - __ldcg(&w.rec[v].key);
  return End{d, g.scaled ? w.lx[d] : 0, w.rec[v].sig};
}

// After the forward sweep: every chain's vertices, and what its ends receive
// from them; the vertices of a chain that carries paths from end to end, which
// wait for the far end's q, are only summed.
template <int kBlock>
__device__ void chains(Shared<kBlock> &sh, const CoreArgs &a, const Slot &w, const View &g, int64_t c0, int64_t c1,
                       double wsrc, unsigned long long *acc) {
  for (int64_t c = c0 + threadIdx.x; c < c1; c += kBlock) {
    const int4 ct = __ldg(a.ctab + c);
    const End A = end_of(w, g, ct.x), B = end_of(w, g, ct.y);
    double ca = 0.0, cb = 0.0;
    const int gap = B.d - A.d;
    if (c == g.own) {  // two stretches, each between an end and the source
      const End source{0, 0, 1.0};
      double none = 0.0;
      if (A.d <= g.pos) walk(g, ct.z, g.pos, A, source, wsrc, acc, a.err, ca, none);
      none = 0.0;
      if (B.d <= ct.w - 1 - g.pos) walk(g, ct.z + g.pos + 1, ct.w - 1 - g.pos, source, B, wsrc, acc, a.err, none, cb);
    } else if (gap > ct.w || gap < -ct.w) {
      double sum = 0.0;
      for (int j = 0; j < ct.w; ++j) sum += (double)ldg(g.reach + ct.z + j) + 1.0;
      ca = gap > 0 ? sum : 0.0;
      cb = gap > 0 ? 0.0 : sum;
    } else {
      walk(g, ct.z, ct.w, A, B, wsrc, acc, a.err, ca, cb);
    }
    // on its own chain an end fed from the source waits for its q as well
    if (c == g.own ? A.d > g.pos || B.d > ct.w - 1 - g.pos : gap > ct.w || gap < -ct.w)
      w.via[atomicAdd(&sh.nvia, 1)] = (int32_t)(c - c0);
    w.in[2 * (c - c0)] = ca;
    w.in[2 * (c - c0) + 1] = cb;
  }
}

// After the backward sweep: the vertices of the chains that waited.
template <int kBlock>
__device__ void chains_left(Shared<kBlock> &sh, const CoreArgs &a, const Slot &w, const View &g, int64_t c0, double wsrc,
                            unsigned long long *acc) {
  const int n = sh.nvia;
  for (int i = threadIdx.x; i < n; i += kBlock) {
    const int64_t c = c0 + w.via[i];
    const int4 ct = __ldg(a.ctab + c);
    const End A = end_of(w, g, ct.x), B = end_of(w, g, ct.y);
    const double qa = __ldcg(&w.rec[ct.x].v), qb = __ldcg(&w.rec[ct.y].v);
    double ca = 0.0, cb = 0.0, none = 0.0;
    if (c == g.own) {
      const End source{0, 0, 1.0};
      cb = scaled(qa, -A.x);  // one path from the source through the stretch
      if (A.d > g.pos) walk(g, ct.z, g.pos, A, source, wsrc, acc, a.err, none, cb);
      ca = scaled(qb, -B.x);
      none = 0.0;
      if (B.d > ct.w - 1 - g.pos) walk(g, ct.z + g.pos + 1, ct.w - 1 - g.pos, source, B, wsrc, acc, a.err, ca, none);
    } else {
      if (B.d > A.d) ca = scaled(A.s * qb, A.x - B.x);
      else cb = scaled(B.s * qa, B.x - A.x);
      walk(g, ct.z, ct.w, A, B, wsrc, acc, a.err, ca, cb);
    }
  }
}

// =============================================================== backward ===

// The successor term of an arc over a chain of k vertices of a vertex on level l.
__device__ __forceinline__ double bwd_term(const Slot &w, const View &g, const Seen &r, int k, int l) {
  if (r.key != g.top - l - 1 - k) return 0.0;
  const double v = r.v;
  return g.scaled ? scaled(v, w.lx[l] - w.lx[l + 1 + k]) : v;
}
__device__ __forceinline__ const double *chain_in(const Slot &w, const View &g, int cid) {
  return w.in + 2 * ((cid >> 1) - g.chain0) + (cid & 1);
}

__device__ __forceinline__ void bwd_done(const CoreArgs &a, const Slot &w, int reach, int32_t v, double s, double q,
                                         double in) {
  const double delta = s * q + in;
  const double qv = ((double)reach + 1.0 + delta) / s;
  w.rec[v].v = qv;
  w.rec[v].dep = delta;
  if (exp_bits(qv) == 0x7ff || exp_bits(delta) == 0x7ff || exp_bits(s) == 0) set_err(a.err, kDevOverflow);
}

// Arcs j0, j0 + step, ... of a vertex on level l (a short row's: r).
__device__ __forceinline__ void bwd_arcs(const Slot &w, const View &g, const Head &h, Arcs r, int j0, int step, int l,
                                         double &q, double &in) {
  for (; j0 < h.deg; j0 += kCoreShort * step) {
    if (h.deg > kCoreShort) arcs_from<true>(g, h, j0, step, r);
    Seen s[kCoreShort];
    double ci[kCoreShort];
#pragma unroll
    for (int j = 0; j < kCoreShort; ++j) {
      s[j] = r.u[j] >= 0 ? w.seen(r.u[j]) : Seen{INT_MIN, 0.0};
      ci[j] = r.cid[j] >= 0 ? *chain_in(w, g, r.cid[j]) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kCoreShort; ++j) {
      q += bwd_term(w, g, s[j], r.k[j], l);
      in += ci[j];
    }
  }
}

template <int kBlock>
__device__ void core_sweep(Shared<kBlock> &sh, const CoreArgs &a, const Slot &w, const View &g, int last) {
  const int tid = threadIdx.x;
  if (tid < 3) { sh.nwq[tid] = 0; sh.ncq[tid] = 0; }
  __syncthreads();
  int f1 = w.lv[last + 1], f0 = w.lv[last];
  for (int l = last, m = 0; l >= 1; --l, m = m == 2 ? 0 : m + 1) {
    const int nxt = m == 2 ? 0 : m + 1, e0 = w.lv[l - 1];
    if (tid == 0) { sh.nwq[nxt] = 0; sh.ncq[nxt] = 0; }
    for (int i = f0 + tid; i < f1; i += kBlock) {
      const int32_t v = w.order[i];
      const Head h = head_of(g, v);
      const Arcs r = arcs_with<true>(g, v, h);
      const double s = w.rec[v].sig;
      if (h.deg > kLight) {
        queue_row(sh, w, m, v, h.deg);
        continue;
      }
      double q = 0.0, in = 0.0;
      bwd_arcs(w, g, h, r, 0, 1, l, q, in);
      bwd_done(a, w, h.reach, v, s, q, in);
    }
    __syncthreads();
    const int nw = sh.nwq[m], nc = sh.ncq[m];
    if (nw | nc) {
      long_rows(sh, w, g, nc, nw,
                [&](const Head &h, int j0, int step, double &x, double &y) { bwd_arcs(w, g, h, Arcs{}, j0, step, l, x, y); },
                [&](int32_t v, const Head &h, double x, double y) { bwd_done(a, w, h.reach, v, w.rec[v].sig, x, y); });
      __syncthreads();
    }
    f1 = f0;
    f0 = e0;
  }
}

// ================================================================= kernel ===

template <int kBlock>
__global__ void __launch_bounds__(kBlock, 1024 / kBlock) core_kernel(CoreArgs a) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ Shared<kBlock> sh;
  const Slot w = slot_of(a, s_raw, Shared<kBlock>::kRing);
  if (threadIdx.x == 0) sh.base = a.epochs[blockIdx.x];
  __syncthreads();
  while (true) {
    if (threadIdx.x == 0) {
      // stop early (uniformly for the CTA) once any CTA has flagged an error
      const int64_t k = a.lo + (int64_t)atomicAdd(a.next, 1ull);
      sh.item = (*(volatile int *)a.err != kDevOk || k >= a.hi) ? -1 : k;
    }
    __syncthreads();
    if (sh.item < 0) break;
    const CoreSource it = a.src[sh.item];
    const int64_t vo = a.vtx_off[it.bcc];
    const int64_t e0 = a.row[vo];
    View g;
    g.rows = a.rows + a.row_off[it.bcc];
    g.col = a.xcol + e0;
    g.k = a.xk + e0;
    g.cid = a.xcid + e0;
    g.reach = a.reach + vo;
    g.ncore = a.n_plain[it.bcc];
    g.scaled = false;
    g.chain0 = a.chain_off[it.bcc];
    g.own = -1;
    g.pos = g.len = 0;
    g.endl = g.endr = -1;
    if (it.src >= g.ncore) {
      g.own = a.vchain[vo + it.src];
      const int4 ct = a.ctab[g.own];
      g.endl = ct.x;
      g.endr = ct.y;
      g.pos = it.src - ct.z;
      g.len = ct.w;
    }
    // keys stay below 2^30: past that every record of the slot starts over
    const int span = a.shape.tcap + 2;
    int base = sh.base;
    if (base >= (1 << 30) - 2 * span) {
      for (int64_t k = threadIdx.x; k < a.shape.cap; k += kBlock) w.rec[k].key = 0;
      base = 1;
      __syncthreads();
    }
    g.top = base + span;
    const int last = g.ncore <= a.shape.cap ? core_bfs(sh, a, w, g, it.src) : -1;
    if (last >= 0) {
      const double wsrc = (double)a.reach[vo + it.src] + 1.0;
      unsigned long long *acc = a.acc + (int64_t)kAccDigits * vo;
      const int64_t nch = a.chain_off[it.bcc + 1] - g.chain0;
      if (threadIdx.x == 0) sh.nvia = 0;
      __syncthreads();
      chains(sh, a, w, g, g.chain0, g.chain0 + nch, wsrc, acc);
      core_sweep(sh, a, w, g, last);  // starts and ends with a barrier
      chains_left(sh, a, w, g, g.chain0, wsrc, acc);
      const int32_t skip = g.own < 0 ? it.src : -1;  // a source has no dependency on itself
      for (int32_t v = threadIdx.x; v < g.ncore; v += kBlock) {
        const double delta = w.rec[v].dep;
        if (v != skip && delta != 0.0) acc_add(acc + (int64_t)kAccDigits * v, delta * wsrc, a.err);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (g.ncore > a.shape.cap) set_err(a.err, kDevWorkspace);
      sh.base = base + span + 1;
    }
  }
  if (threadIdx.x == 0) a.epochs[blockIdx.x] = sh.base;
}

// ============================================================ contraction ===

// Chain table entries and the chains of the chain vertices: a thread per chain.
__global__ void chain_table_kernel(const int64_t *vtx_off, const int64_t *chain_off, const int32_t *chain_start,
                                   const int32_t *chain_len, const int32_t *chain_l, const int32_t *chain_r,
                                   const int8_t *on, int32_t n_bcc, int4 *ctab, int32_t *vchain) {
  const int64_t nch = chain_off[n_bcc];
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < nch; c += (int64_t)gridDim.x * blockDim.x) {
    int32_t lo = 0, hi = n_bcc - 1;  // the BCC: the last whose range starts at or before c
    while (lo < hi) {
      const int32_t mid = (lo + hi + 1) / 2;
      if (chain_off[mid] <= c) lo = mid;
      else hi = mid - 1;
    }
    ctab[c] = make_int4(chain_l[c], chain_r[c], chain_start[c], chain_len[c]);
    if (!on[lo]) continue;
    const int64_t vo = vtx_off[lo];
    for (int32_t j = 0; j < chain_len[c]; ++j) vchain[vo + chain_start[c] + j] = (int32_t)c;
  }
}

// Rows of the core vertices, a warp per row (a hub's row is thousands of arcs
// long): arcs between core vertices first, chain arcs after them, each in the
// order of the packed row.
__global__ void __launch_bounds__(256) contract_kernel(const int64_t *row, const int32_t *col, const int64_t *vtx_off,
                                                       const int32_t *n_plain, const int32_t *reach, const int8_t *on,
                                                       int32_t n_bcc, int64_t n_packed, const int4 *ctab,
                                                       const int32_t *vchain, const int64_t *row_off, CoreRow *rows,
                                                       int32_t *xcol, int32_t *xk, int32_t *xcid) {
  const int lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1;
  for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n_packed;
       v += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    int32_t lo = 0, hi = n_bcc - 1;
    while (lo < hi) {
      const int32_t mid = (lo + hi + 1) / 2;
      if (vtx_off[mid] <= v) lo = mid;
      else hi = mid - 1;
    }
    const int64_t vo = vtx_off[lo];
    const int32_t npl = n_plain[lo];
    if (!on[lo] || v - vo >= npl) continue;
    const int64_t e0 = row[v], e1 = row[v + 1], base = row[vo];
    int32_t unit = 0;
    for (int64_t e = e0 + lane; e - lane < e1; e += 32) unit += __popc(__ballot_sync(0xffffffffu, e < e1 && col[e] < npl));
    int64_t u = e0, c = e0 + unit;
    for (int64_t e = e0 + lane; e - lane < e1; e += 32) {
      const bool in = e < e1;
      const int32_t y = in ? col[e] : 0;
      const uint32_t mu = __ballot_sync(0xffffffffu, in && y < npl), mc = __ballot_sync(0xffffffffu, in && y >= npl);
      if (in && y < npl) {
        const int64_t o = u + __popc(mu & below);
        xcol[o] = y;
        xk[o] = 0;
        xcid[o] = 0;
      } else if (in) {
        const int64_t o = c + __popc(mc & below);
        const int32_t ch = vchain[vo + y];
        const int4 ct = ctab[ch];
        const bool right = !(ct.x == (int32_t)(v - vo) && y == ct.z);
        xcol[o] = right ? ct.x : ct.y;
        xk[o] = ct.w;
        xcid[o] = ch * 2 + (right ? 1 : 0);
      }
      u += __popc(mu);
      c += __popc(mc);
    }
    __syncwarp();
    if (lane == 0) {
      CoreRow r{(int32_t)(e0 - base), (int32_t)(e1 - e0), unit, reach[v], {-1, -1, -1, -1}, {-1, -1, -1, -1}, {0, 0, 0, 0}};
      if (r.deg <= kCoreShort) {
        r.part = 0;
        for (int j = 0; j < r.deg; ++j) {  // written above by this warp
          r.u[j] = xcol[e0 + j];
          r.part |= xk[e0 + j] << (8 * j);
          if (xk[e0 + j]) r.cid[j] = xcid[e0 + j];
        }
      }
      rows[row_off[lo] + v - vo] = r;
    }
  }
}

}  // namespace

cudaError_t core_contract(const int64_t *row, const int32_t *col, const int64_t *vtx_off, const int32_t *n_plain,
                          const int32_t *reach, const int64_t *chain_off, const int32_t *chain_start,
                          const int32_t *chain_len, const int32_t *chain_l, const int32_t *chain_r, const int8_t *on,
                          int32_t n_bcc, int64_t n_packed, const int64_t *row_off, CoreRow *rows, int32_t *xcol,
                          int32_t *xk, int32_t *xcid, int4 *ctab, int32_t *vchain, cudaStream_t stream) {
  const int blocks = (int)std::min<int64_t>((n_packed + 7) / 8, 148 * 8);
  chain_table_kernel<<<blocks, 256, 0, stream>>>(vtx_off, chain_off, chain_start, chain_len, chain_l, chain_r, on, n_bcc,
                                                 ctab, vchain);
  contract_kernel<<<blocks, 256, 0, stream>>>(row, col, vtx_off, n_plain, reach, on, n_bcc, n_packed, ctab, vchain,
                                              row_off, rows, xcol, xk, xcid);
  return cudaGetLastError();
}

namespace {
const void *core_fn(int block) {
  switch (block) {
    case 64: return (const void *)core_kernel<64>;
    case 128: return (const void *)core_kernel<128>;
    case 256: return (const void *)core_kernel<256>;
    case 512: return (const void *)core_kernel<512>;
    default: return nullptr;
  }
}
cudaError_t allow_smem(int block) {
  const size_t fixed = block == 64    ? sizeof(Shared<64>)
                       : block == 128 ? sizeof(Shared<128>)
                       : block == 256 ? sizeof(Shared<256>)
                                      : sizeof(Shared<512>);
  return cudaFuncSetAttribute(core_fn(block), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemPerCta - (int)fixed);
}
}  // namespace

int core_ctas_per_sm(int block, const CoreArgs::CoreShape &shape) {
  const void *fn = core_fn(block);
  int n = 0;
  if (!fn) return 0;
  if (allow_smem(block) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, block, (size_t)shape.smem_bytes()) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

cudaError_t launch_core(const CoreArgs &a, int block, int grid, cudaStream_t stream) {
  const void *fn = core_fn(block);
  if (!fn) return cudaErrorInvalidValue;
  const size_t smem = (size_t)a.shape.smem_bytes();
  const cudaError_t e = allow_smem(block);
  if (e != cudaSuccess) return e;
  CoreArgs args = a;
  void *params[] = {&args};
  return cudaLaunchKernel(fn, dim3(grid), dim3(block), params, smem, stream);
}

}  // namespace bcg
