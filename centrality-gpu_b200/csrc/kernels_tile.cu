// Small-BCC schedule: one CTA per range of sources of one BCC, every array a
// source touches in shared memory.
//
// The reference runs every BCC through the same per-source kernel, one
// source per CTA (Codes/kernels_free.cu:154-473, launch shape
// Codes/begin_gpupgm.cu:52-65), with its rows in global memory, whatever the
// BCC's size; on a batch of thousands of small graphs the CTAs then wait on
// global-memory latency at every arc. Here a BCC that fits shared memory is
// run from shared memory only:
//  * the slice (row offsets, 16-bit neighbour ids in pairs; tile.h TileSlice) is
//    brought in by one cp.async.bulk (a plain bulk copy from this GPU's global
//    memory into this CTA's shared memory, completion on an mbarrier whose wait
//    is bounded) and serves every source of the item;
//  * levels, path counts (then q in place) and the visit order of each source
//    live in shared memory: one set per warp in the warp class (a warp per
//    source, eight in flight), one per source group in the CTA class (the
//    whole CTA on one source, or eight, four or two groups of a 1024-thread CTA
//    on their own sources from the one slice, wherever their arrays fit);
//  * forward: level-synchronous, each frontier vertex pulls sigma from its
//    predecessors and claims its successors in one scan of its row. Warp class:
//    a row of up to kLaneDeg arcs by one lane, a longer one by the warp. CTA
//    class: by one thread, by kSub lanes or by a warp (kLightPairs,
//    kMediumPairs); on a level that holds 1 / kWide of the BCC, successors are
//    stamped with plain stores and collected by a pass over the stamps, since
//    claiming them one by one was two thirds of a source's time;
//  * backward: successor form, q(w) = (reach(w)+1+delta(w))/sigma(w) and
//    delta(v) = sigma(v) * sum q (Codes/kernels_free.cu:391,409), q
//    overwriting sigma in place;
//  * chain (degree-2) vertices are ordinary vertices and sources here: on a
//    BCC this small their BFS costs about what the endpoint merge of the
//    per-source schedule does;
//  * BC: contributions delta * (reach(s)+1) (Codes/kernels_free.cu:425) go to
//    shared-memory fixed-point counters (warp class: integer atomics, any
//    order) or to an FP64 partial row per source group (CTA class: a group's
//    sources, fixed by the item, run one after another, each vertex written
//    by one thread, so the order is fixed), then once per item into the
//    global fixed-point counters.
// Path counts are FP64 without per-level scaling: the plan routes a BCC here
// only when no path count can pass 2^1000 ((2 ecc + 1) levels of at most
// maxdeg predecessors each); one that does, or a non-finite value, flags
// kDevOverflow.
#include "accum.cuh"
#include "common.cuh"
#include "tile.h"

#include <algorithm>
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace bcg {

namespace {

constexpr int kThreads = kTileWarps * 32;
constexpr int kLaneDeg = 8;  // warp class: rows up to this many arcs: one lane; longer rows: the warp
// CTA class, rows in pairs of arcs: up to kLightPairs by one thread as its vertex
// comes up; up to kMediumPairs queued for kSub lanes; longer ones queued for a
// warp; a row beyond the queues' room by the thread that found it, with the same
// sum. BA graphs: six
// vertices in seven have up to four arcs, and the hubs hold a third of the arcs.
constexpr int kLightPairs = 4;
constexpr int kMediumPairs = 16;
constexpr int kSub = 4;
constexpr int kLongQueue = 1024;
// A level of at least 1 / kWide of the BCC's vertices does not claim its
// successors one by one: it stamps them (the same value whoever stores it) and
// then collects the stamped ones with a pass over all stamps. BA batches of 30
// graphs of 4,500-5,000 and 120 of 1,000-1,500 vertices, and the 2,000-vertex
// graph: 75.4, 23.4 and 0.23 ms with rows of up to 8 arcs by a thread and the
// others by a warp, every successor claimed; 67.1, 16.3 and 0.35 with the row
// classes above; 43.9, 10.9, 0.195 / 42.0, 10.4, 0.186 / 41.1, 10.2, 0.182 / 40.5,
// 10.1, 0.183 stamping from 1/8 / 1/16 / 1/32 / 1/64 of the BCC on.
constexpr int kWide = 32;

struct Ctl {
  unsigned long long bar;  // mbarrier of the slice copy
  int item, next, bcc, pad;
  int tails[kTileWarps];
};

__host__ __device__ constexpr int64_t align16(int64_t x) { return (x + 15) / 16 * 16; }

// ---- shared-memory layouts (host and device agree through these)
struct WarpLayout {  // ctl | counters [nmax][kAccDigits] | per warp: d [nmax], S [nmax], sq [nmax] | slice
  __host__ __device__ static int64_t cnt() { return align16(sizeof(Ctl)); }
  __host__ __device__ static int64_t per_warp(int64_t nmax) { return align16(8 * nmax) + 2 * align16(4 * nmax); }
  __host__ __device__ static int64_t warps(int64_t nmax) { return cnt() + align16(nmax * kAccDigits * 8); }
  __host__ __device__ static int64_t slice(int64_t nmax) { return warps(nmax) + kTileWarps * per_warp(nmax); }
};
// CTA class: kBlock threads in kBlock / kGroup groups, each group on its own
// sources with its own arrays and barrier, all groups on the one staged slice.
// ctl | per group: sq [nmax] | d uint16 [nmax] | S uint16 [nmax] | lv uint16
//     [kLevels] | queues of medium and long rows uint16 [kQueue] each | Counts |
// slice (one group: levels and queues of the class limits; several: the smaller
// limits of the grouped classes, tile.h).
struct Counts {  // by level mod 3
  int found[3], medium[3], large[3], pad[3];
};
template <int kBlock, int kGroup>
struct CtaLayout {
  static constexpr int kG = kBlock / kGroup;
  static constexpr int kLevels = kG == 1 ? kTileMaxLevels : kTileGroupMaxLevels;
  static constexpr int kQueue = kG == 1 ? kLongQueue : kGroup < 128 ? kGroup : kGroupLongQueue;
  __host__ __device__ static int64_t d(int64_t nmax) { return align16(8 * nmax); }
  __host__ __device__ static int64_t S(int64_t nmax) { return d(nmax) + align16(2 * nmax); }
  __host__ __device__ static int64_t lv(int64_t nmax) { return S(nmax) + align16(2 * nmax); }
  __host__ __device__ static int64_t q(int64_t nmax) { return lv(nmax) + align16(2 * kLevels); }
  __host__ __device__ static int64_t ctr(int64_t nmax) { return q(nmax) + align16(2 * 2 * kQueue); }
  __host__ __device__ static int64_t group_bytes(int64_t nmax) { return ctr(nmax) + align16(sizeof(Counts)); }
  __host__ __device__ static int64_t group(int g, int64_t nmax) { return align16(sizeof(Ctl)) + g * group_bytes(nmax); }
  __host__ __device__ static int64_t slice(int64_t nmax) { return group(kG, nmax); }
  // the group's barrier: the CTA's own when the group is the CTA, else named barrier g+1
  __device__ __forceinline__ static void sync(int g) {
    if constexpr (kG == 1) {
      __syncthreads();
    } else if constexpr (kGroup == 32) {
      __syncwarp();
    } else {
      asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(kGroup) : "memory");
    }
  }
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// mbarrier and bulk-copy primitives (PTX ISA: mbarrier, cp.async.bulk).
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// Global -> this CTA's shared memory; bytes a multiple of 16, both ends 16-byte aligned.
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads of dst before the copy's writes
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// Waits for phase `parity` of the barrier, at most limit_ns; false on timeout.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity, unsigned long long limit_ns) {
  const unsigned long long t0 = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (global_ns() - t0 > limit_ns) return false;
  }
  return true;
}

// One BCC as the kernels read it: local row offsets (uint16 or int32) and
// neighbours (shared memory), reach (global).
struct View {
  const int32_t *R32;
  const uint16_t *R16;  // set for a narrow slice
  const uint16_t *C;
  const int32_t *rch;
  __device__ __forceinline__ int pair(int32_t w) const { return R16 ? (int)R16[w] : R32[w]; }  // w's first pair
  __device__ __forceinline__ int row(int32_t w) const { return 2 * pair(w); }                  // w's first arc
  __device__ __forceinline__ uint32_t two(int p) const { return reinterpret_cast<const uint32_t *>(C)[p]; }
};

// Pulls the next item for the CTA (thread 0) and stages its BCC's slice if
// the CTA does not hold it already. Returns false when the CTA is done (no
// item left, an error flagged, or the slice did not arrive in time).
__device__ bool next_item(const TileArgs &a, Ctl &ctl, unsigned char *slice, unsigned &phase, TileItem &it,
                          int64_t &vo, int32_t &nb) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    const int64_t k = (int64_t)atomicAdd(a.next_item, 1ull);
    ctl.item = (*(volatile int *)a.err != kDevOk || a.item_begin + k >= a.item_end) ? -1 : (int)k;
    ctl.next = 0;
  }
  __syncthreads();  // also: every thread is done with the previous item's slice and rows
  if (ctl.item < 0) return false;
  it = a.items[a.item_begin + ctl.item];
  vo = a.vtx_off[it.bcc];
  nb = (int32_t)(a.vtx_off[it.bcc + 1] - vo);
  const int64_t soff = a.slice_off[it.bcc] & ~int64_t(15);
  if (a.src) {  // places in the source list, clipped to the launch's range
    it.s0 = max(it.s0, a.src_lo);
    it.s1 = min(it.s1, a.src_hi);
  }
  if (nb > a.nmax || a.slice_off[it.bcc] < 0 || it.s0 < 0 || (!a.src && it.s1 > nb)) {  // uniform over the CTA
    if (tid == 0) set_err(a.err, kDevBadItem);
    return false;
  }
  if (ctl.bcc != it.bcc) {  // uniform: ctl.bcc was last written before a barrier
    if (tid == 0) {
      const unsigned bytes = (unsigned)a.slice_bytes[it.bcc];
      mbar_expect_tx(&ctl.bar, bytes);
      bulk_copy(slice, a.slices + soff, bytes, &ctl.bar);
    }
    if (!mbar_wait(&ctl.bar, phase, a.wait_ns)) {
      // the copy did not complete in time: record it, wait (again bounded)
      // for the copy in flight to land in this CTA's shared memory, stop
      set_err(a.err, kDevTimeout);
      mbar_wait(&ctl.bar, phase, a.wait_ns);
      return false;
    }
    phase ^= 1u;
  }
  return true;
}

// Local id of source k of an item.
__device__ __forceinline__ int32_t source_of(const TileArgs &a, int32_t k) { return a.src ? __ldg(a.src + k) : k; }

__device__ __forceinline__ View view_of(const TileArgs &a, const unsigned char *slice, int32_t nb, int64_t vo,
                                        int32_t bcc) {
  const bool narrow = (a.slice_off[bcc] & 1) != 0;
  return View{reinterpret_cast<const int32_t *>(slice), narrow ? reinterpret_cast<const uint16_t *>(slice) : nullptr,
              reinterpret_cast<const uint16_t *>(slice + TileSlice::col_at(nb, narrow)), a.reach + vo};
}

// Appends x to the visit order S: one atomic per group of lanes appending at
// once (the lanes that reach this call together), not one per lane.
template <typename ST>
__device__ __forceinline__ void append(ST *S, int *tail, int32_t x) {
  cg::coalesced_group g = cg::coalesced_threads();
  int pos = 0;
  if (g.thread_rank() == 0) pos = atomicAdd(tail, (int)g.size());
  S[g.shfl(pos, 0) + (int)g.thread_rank()] = (ST)x;
}

// Claims unvisited vertex x (level -1) for level lev; true for the one claim
// that wins.
__device__ __forceinline__ bool claim(int32_t *d, int32_t x, int lev) { return atomicCAS(d + x, -1, lev) == -1; }

// Forward scan of one row by one thread (four arcs' loads in flight, sums in
// arc order): pulls sigma from level dprev, claims unvisited vertices for
// dnext (appended to S at *tail).
template <typename DT, typename ST>
__device__ __forceinline__ double pull_row(const View &g, int e0, int e1, DT *d, const double *sq, ST *S, int *tail,
                                           int dprev, int dnext) {
  double acc = 0.0;
  for (int e = e0; e < e1; e += 4) {
    int32_t x[4], dx[4];
    double sv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = e + j < e1 ? (int32_t)g.C[e + j] : -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) dx[j] = x[j] >= 0 ? (int)d[x[j]] : INT_MAX;
#pragma unroll
    for (int j = 0; j < 4; ++j) sv[j] = dx[j] == dprev ? sq[x[j]] : 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (dx[j] == dprev) acc += sv[j];
      else if (dx[j] == -1 && claim(d, x[j], dnext)) append(S, tail, x[j]);
    }
  }
  return acc;
}

// The same for a long row, by a whole warp (lanes over arcs, fixed-order sum).
template <typename DT, typename ST>
__device__ __forceinline__ double pull_row_warp(const View &g, int e0, int e1, DT *d, const double *sq, ST *S, int *tail,
                                                int dprev, int dnext, int lane) {
  double acc = 0.0;
  for (int e = e0 + lane; e < e1; e += 32) {
    const int32_t x = g.C[e];
    const int dx = d[x];
    if (dx == dprev) acc += sq[x];
    else if (dx == -1 && claim(d, x, dnext)) append(S, tail, x);
  }
  return warp_sum(acc);
}

// Sum of q over the successors (level dsucc) of one row, by one thread.
template <typename DT>
__device__ __forceinline__ double push_row(const View &g, int e0, int e1, const DT *d, const double *sq, int dsucc) {
  double acc = 0.0;
  for (int e = e0; e < e1; e += 4) {
    int32_t x[4];
    bool hit[4];
    double qv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = e + j < e1 ? (int32_t)g.C[e + j] : -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) hit[j] = x[j] >= 0 && (int)d[x[j]] == dsucc;
#pragma unroll
    for (int j = 0; j < 4; ++j) qv[j] = hit[j] ? sq[x[j]] : 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (hit[j]) acc += qv[j];
  }
  return acc;
}

template <typename DT>
__device__ __forceinline__ double push_row_warp(const View &g, int e0, int e1, const DT *d, const double *sq, int dsucc,
                                                int lane) {
  double acc = 0.0;
  for (int e = e0 + lane; e < e1; e += 32) {
    const int32_t x = g.C[e];
    if ((int)d[x] == dsucc) acc += sq[x];
  }
  return warp_sum(acc);
}

// delta and q of w from the successors' sum, r = reach(w) + 1; returns delta (q
// overwrites sigma).
__device__ __forceinline__ double finish(double r, int32_t w, double sum, double *sq, int *err) {
  const double sw = sq[w];
  const double delta = sw * sum;
  const double qw = (r + delta) / sw;
  // counts past 2^1000 too: their q would lose bits below FP64's normal range
  if (exp_bits(qw) == 0x7ff || exp_bits(delta) == 0x7ff || (unsigned)(exp_bits(sw) - 1) >= 1023 + 1000)
    set_err(err, kDevOverflow);
  sq[w] = qw;
  return delta;
}

// ======================================================= warp per source ===

// BFS of one warp from s (rows in this warp's shared memory, level offsets lv
// in global memory). Returns the number of levels.
__device__ int warp_bfs(const View &g, int32_t nb, int32_t s, int32_t *d, double *sq, int32_t *S, int32_t *lv,
                        int *tail, int lane) {
  for (int v = lane; v < nb; v += 32) d[v] = -1;
  __syncwarp();
  if (lane == 0) {
    d[s] = 0;
    S[0] = s;
    sq[s] = 1.0;
    lv[0] = 0;
    lv[1] = 1;
    *tail = 1;
  }
  __syncwarp();
  int lev = 0, f0 = 0, f1 = 1;
  while (true) {
    const int dprev = lev == 0 ? INT_MIN : lev - 1, dnext = lev + 1;
    for (int c0 = f0; c0 < f1; c0 += 32) {
      const int i = c0 + lane;
      int32_t w = -1, e0 = 0, e1 = 0;
      if (i < f1) {
        w = S[i];
        e0 = g.row(w);
        e1 = g.row(w + 1);
      }
      const bool big = e1 - e0 > kLaneDeg;
      if (w >= 0 && !big) {
        const double acc = pull_row(g, e0, e1, d, sq, S, tail, dprev, dnext);
        if (lev > 0) sq[w] = acc;
      }
      uint32_t bigs = __ballot_sync(0xffffffffu, w >= 0 && big);
      while (bigs) {
        const int j = __ffs(bigs) - 1;
        bigs &= bigs - 1;
        const int32_t wj = __shfl_sync(0xffffffffu, w, j);
        const int a0 = __shfl_sync(0xffffffffu, e0, j), a1 = __shfl_sync(0xffffffffu, e1, j);
        const double acc = pull_row_warp(g, a0, a1, d, sq, S, tail, dprev, dnext, lane);
        if (lane == 0 && lev > 0) sq[wj] = acc;
      }
    }
    __syncwarp();
    const int t = *(volatile int *)tail;
    if (t == f1) break;
    if (lane == 0) lv[lev + 2] = t;
    f0 = f1;
    f1 = t;
    ++lev;
    __syncwarp();
  }
  return lev + 1;
}

__device__ void warp_sweep(const View &g, int nlev, const int32_t *d, double *sq, const int32_t *S, const int32_t *lv,
                           double wsrc, unsigned long long *cnt, int lane, int *err) {
  for (int lev = nlev - 1; lev >= 1; --lev) {
    const int dsucc = lev + 1, a0 = lv[lev], a1 = lv[lev + 1];
    for (int c0 = a0; c0 < a1; c0 += 32) {
      const int i = c0 + lane;
      int32_t w = -1, e0 = 0, e1 = 0;
      if (i < a1) {
        w = S[i];
        e0 = g.row(w);
        e1 = g.row(w + 1);
      }
      const bool big = e1 - e0 > kLaneDeg;
      double sum = 0.0;
      if (w >= 0 && !big) sum = push_row(g, e0, e1, d, sq, dsucc);
      uint32_t bigs = __ballot_sync(0xffffffffu, w >= 0 && big);
      while (bigs) {
        const int j = __ffs(bigs) - 1;
        bigs &= bigs - 1;
        const int b0 = __shfl_sync(0xffffffffu, e0, j), b1 = __shfl_sync(0xffffffffu, e1, j);
        const double part = push_row_warp(g, b0, b1, d, sq, dsucc, lane);
        if (lane == j) sum = part;
      }
      if (w >= 0) {
        const double delta = finish((double)__ldg(g.rch + w) + 1.0, w, sum, sq, err);  // this level's q: read by the level above only
        if (delta != 0.0) acc_add(cnt + (int64_t)kAccDigits * w, delta * wsrc, err);
      }
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kThreads, 1) tile_warp_kernel(TileArgs a) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  Ctl &ctl = *reinterpret_cast<Ctl *>(s_raw);
  unsigned long long *cnt = reinterpret_cast<unsigned long long *>(s_raw + WarpLayout::cnt());
  unsigned char *slice = s_raw + WarpLayout::slice(a.nmax);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char *mine = s_raw + WarpLayout::warps(a.nmax) + (int64_t)warp * WarpLayout::per_warp(a.nmax);
  double *sq = reinterpret_cast<double *>(mine);
  int32_t *d = reinterpret_cast<int32_t *>(mine + align16(8 * (int64_t)a.nmax));
  int32_t *S = d + align16(4 * (int64_t)a.nmax) / 4;
  int32_t *lv = a.ws_lv + ((int64_t)blockIdx.x * kTileWarps + warp) * a.cap;
  if (tid == 0) {
    mbar_init(&ctl.bar, 1);
    ctl.bcc = -1;
  }
  __syncthreads();
  unsigned phase = 0;
  TileItem it;
  int64_t vo;
  int32_t nb;
  while (next_item(a, ctl, slice, phase, it, vo, nb)) {
    for (int64_t k = tid; k < (int64_t)kAccDigits * nb; k += kThreads) cnt[k] = 0ull;
    __syncthreads();
    if (tid == 0) ctl.bcc = it.bcc;  // read again only after the next barrier
    const View g = view_of(a, slice, nb, vo, it.bcc);
    while (true) {  // the warps take the item's sources one at a time
      int k = 0;
      if (lane == 0) k = atomicAdd(&ctl.next, 1);
      k = __shfl_sync(0xffffffffu, k, 0);
      if (it.s0 + k >= it.s1) break;
      const int32_t s = source_of(a, it.s0 + k);
      const int nlev = warp_bfs(g, nb, s, d, sq, S, lv, &ctl.tails[warp], lane);
      warp_sweep(g, nlev, d, sq, S, lv, (double)__ldg(g.rch + s) + 1.0, cnt, lane, a.err);
    }
    __syncthreads();
    unsigned long long *acc = a.acc + (int64_t)kAccDigits * vo;  // integer adds: any order
    for (int64_t k = tid; k < (int64_t)kAccDigits * nb; k += kThreads) {
      const unsigned long long c = cnt[k];
      if (c) atomicAdd(acc + k, c);
    }
  }
}

// ======================================================== CTA per source ===

// What one group of threads works on. Levels are stamped base + level, so that
// the next source finds every stamp stale (below its base) and clears nothing.
struct Group {
  double *sq;       // path counts, then q
  uint16_t *d, *S;  // stamps; vertices by level
  uint16_t *lv;     // level offsets into S
  uint16_t *medium, *large;
  Counts *n;
  int base;
};

// Claims unvisited vertex x (stamp below base) with stamp `next`: a CAS on the
// word of two stamps, again while only the other one changed.
__device__ __forceinline__ bool claim(const Group &G, int32_t x, int next) {
  unsigned *word = reinterpret_cast<unsigned *>(G.d) + (x >> 1);
  const int sh = (x & 1) * 16;
  unsigned old = *reinterpret_cast<volatile unsigned *>(word);
  while ((int)(old >> sh & 0xffffu) < G.base) {
    const unsigned was = atomicCAS(word, old, (old & ~(0xffffu << sh)) | (unsigned)next << sh);
    if (was == old) return true;
    old = was;
  }
  return false;
}

// Pairs p0, p0 + step, ... < p1 of a row, two at a time, forward: the path
// counts of the neighbours on the level before (stamp prev); the others that
// have none yet are stamped for the next level -- on a wide level just that, else
// claimed, and appended to S from f1 on.
__device__ __forceinline__ double fwd_pairs(const View &g, const Group &G, int p0, int p1, int step, int prev, bool wide,
                                            int f1, int *found) {
  double sum = 0.0;
  for (; p0 < p1; p0 += 2 * step) {
    const uint32_t a = g.two(p0), b = p0 + step < p1 ? g.two(p0 + step) : a;
    const int32_t x[4] = {(int32_t)(a & 0xffffu), (int32_t)(a >> 16), (int32_t)(b & 0xffffu), (int32_t)(b >> 16)};
    int dx[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) dx[j] = G.d[x[j]];
    if (p0 + step >= p1) dx[2] = dx[3] = 0xffff;  // no second pair: neither found nor to be claimed
    double v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = dx[j] == prev ? G.sq[x[j]] : 0.0;
    if (wide) {  // uniform over the group
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (dx[j] < G.base) *(volatile uint16_t *)(G.d + x[j]) = (uint16_t)(prev + 2);
    } else {
      uint32_t won = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (dx[j] < G.base && claim(G, x[j], prev + 2)) won |= 1u << j;
      if (won) {
        int at = f1 + atomicAdd(found, __popc(won));
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (won >> j & 1u) G.S[at++] = (uint16_t)x[j];
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) sum += v[j];
  }
  return sum;
}

// Appends the vertices with stamp `stamp` to S from f1 on, eight stamps to a
// load, in a group of kGroup threads.
template <int kGroup>
__device__ __forceinline__ void collect(const Group &G, int nb, int stamp, int f1, int *found, int tid) {
  const int lane = tid & 31;
  for (int c = 0; c < nb; c += 8 * kGroup) {  // uniform over the group
    const int v0 = c + 8 * tid;
    uint4 q = make_uint4(0, 0, 0, 0);  // stamps are never 0
    if (v0 < nb) q = *reinterpret_cast<const uint4 *>(G.d + v0);
    const unsigned w[4] = {q.x, q.y, q.z, q.w};
    uint32_t hit = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if ((int)(w[j] & 0xffffu) == stamp) hit |= 1u << (2 * j);
      if ((int)(w[j] >> 16) == stamp) hit |= 2u << (2 * j);
    }
    if (nb - v0 < 8) hit &= v0 < nb ? (1u << (nb - v0)) - 1 : 0;  // places beyond the BCC hold anything
    const int mine = __popc(hit);
    int upto = mine;  // of the lanes up to this one
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += y;
    }
    int at = 0;
    if (lane == 31 && upto) at = atomicAdd(found, upto);
    at = f1 + __shfl_sync(0xffffffffu, at, 31) + upto - mine;
    for (; hit; hit &= hit - 1) G.S[at++] = (uint16_t)(v0 + __ffs(hit) - 1);
  }
}

// The same backward: the sum of q over the neighbours on the level after.
__device__ __forceinline__ double bwd_pairs(const View &g, const Group &G, int p0, int p1, int step, int next) {
  double sum = 0.0;
  for (; p0 < p1; p0 += 2 * step) {
    const uint32_t a = g.two(p0), b = p0 + step < p1 ? g.two(p0 + step) : a;
    const int32_t x[4] = {(int32_t)(a & 0xffffu), (int32_t)(a >> 16), (int32_t)(b & 0xffffu), (int32_t)(b >> 16)};
    int dx[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) dx[j] = G.d[x[j]];
    if (p0 + step >= p1) dx[2] = dx[3] = 0;
    double v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = dx[j] == next ? G.sq[x[j]] : 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) sum += v[j];
  }
  return sum;
}

// A row that found its queue full, by one thread: what `width` lanes give and
// their butterfly sums up to, so that the sum does not depend on the order in
// which a level's rows were queued.
template <class Row>
__device__ __forceinline__ double row_alone(int p0, int p1, Row row) {
  const int width = p1 - p0 <= kMediumPairs ? kSub : 32;
  double half[6];  // sums of 1, 2, 4, ... lanes waiting for their other half
  double sum = 0.0;
  for (int i = 0; i < width; ++i) {
    // warp_sum adds lanes 16 apart first, queued_rows' sums neighbours first
    sum = row(p0 + (width == 32 ? (int)(__brev(i) >> 27) : i), p1, width);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      if (!(i >> k & 1)) {
        half[k] = sum;
        break;
      }
      sum = half[k] + sum;
    }
  }
  return sum;
}

// Queues a row of `pairs` for several lanes; false if it has to be done here.
template <class L>
__device__ __forceinline__ bool queue_row(const Group &G, int m, int32_t w, int pairs) {
  if (pairs <= kLightPairs) return false;
  int *n = pairs <= kMediumPairs ? &G.n->medium[m] : &G.n->large[m];
  const int at = atomicAdd(n, 1);
  if (at >= L::kQueue) return false;
  (pairs <= kMediumPairs ? G.medium : G.large)[at] = (uint16_t)w;
  return true;
}

// The queued rows of a level: kSub lanes each, then a warp each. row(first pair,
// end, step) gives a lane's sum, done(w, sum) takes the total in one lane.
template <class L, int kGroup, class Row, class Done>
__device__ __forceinline__ void queued_rows(const View &g, const Group &G, int nm, int nl, int tid, Row row, Done done) {
  const int sub = tid % kSub, lane = tid & 31;
  for (int c = 0; c < nm; c += kGroup / kSub) {
    const int k = c + tid / kSub;
    const int32_t w = k < nm ? G.medium[k] : 0;
    double sum = k < nm ? row(g.pair(w) + sub, g.pair(w + 1), kSub) : 0.0;
#pragma unroll
    for (int o = 1; o < kSub; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (k < nm && sub == 0) done(w, sum);
  }
  for (int k = tid >> 5; k < nl; k += kGroup / 32) {
    const int32_t w = G.large[k];
    const double sum = warp_sum(row(g.pair(w) + lane, g.pair(w + 1), 32));
    if (lane == 0) done(w, sum);
  }
}

// BFS of one group (the whole CTA, or a fixed share of its threads) from s: one
// group barrier per level, one more where rows were queued, and on a wide level.
// Counts of level l are at
// l % 3; those of level l+1 are cleared at the start of level l, two barriers
// after their last reader. Returns the number of levels, -1 on an error.
template <int kBlock, int kGroup>
__device__ int cta_bfs(const View &g, const Group &G, int nb, int32_t s, int *err, int grp, int tid) {
  using L = CtaLayout<kBlock, kGroup>;
  if (tid < 3) {
    G.n->found[tid] = 0;
    G.n->medium[tid] = 0;
    G.n->large[tid] = 0;
  }
  if (tid == 0) {
    G.d[s] = (uint16_t)G.base;
    G.S[0] = (uint16_t)s;
    G.lv[0] = 0;
    G.lv[1] = 1;
  }
  L::sync(grp);
  int lev = 0, m = 0, f0 = 0, f1 = 1;
  while (true) {
    const int nxt = m == 2 ? 0 : m + 1;
    if (tid == 0) {
      G.n->found[nxt] = 0;
      G.n->medium[nxt] = 0;
      G.n->large[nxt] = 0;
    }
    const int prev = G.base + lev - 1;  // no stamp of this source on the source's own level
    int *found = &G.n->found[m];
    const bool wide = (f1 - f0) * kWide >= nb;
    for (int i = f0 + tid; i < f1; i += kGroup) {
      const int32_t w = G.S[i];
      const int p0 = g.pair(w), p1 = g.pair(w + 1);
      if (queue_row<L>(G, m, w, p1 - p0)) continue;
      auto row = [&](int q0, int q1, int step) { return fwd_pairs(g, G, q0, q1, step, prev, wide, f1, found); };
      const double sum = p1 - p0 <= kLightPairs ? row(p0, p1, 1) : row_alone(p0, p1, row);
      G.sq[w] = lev ? sum : 1.0;
    }
    L::sync(grp);
    const int nm = min(*(volatile int *)&G.n->medium[m], L::kQueue), nl = min(*(volatile int *)&G.n->large[m], L::kQueue);
    if (nm | nl) {
      queued_rows<L, kGroup>(
          g, G, nm, nl, tid, [&](int p0, int p1, int step) { return fwd_pairs(g, G, p0, p1, step, prev, wide, f1, found); },
          [&](int32_t w, double sum) { G.sq[w] = lev ? sum : 1.0; });
      L::sync(grp);
    }
    if (wide) {
      collect<kGroup>(G, nb, prev + 2, f1, found, tid);
      L::sync(grp);
    }
    const int t = f1 + *(volatile int *)found;
    if (t == f1) break;
    if (lev + 2 >= L::kLevels) {  // uniform; routing keeps BCCs below this depth
      if (tid == 0) set_err(err, kDevWorkspace);
      return -1;
    }
    if (tid == 0) G.lv[lev + 2] = (uint16_t)t;
    f0 = f1;
    f1 = t;
    ++lev;
    m = nxt;
  }
  return lev + 1;
}

// One source's contribution c to vertex w: to the group's FP64 row P (one
// writer per vertex and source; an addition at L2, so that no load is waited
// for), or straight into the BCC's fixed-point counters when there is no row.
__device__ __forceinline__ void contribute(double *P, unsigned long long *acc, int32_t w, double c, int *err) {
  if (P) atomicAdd(P + w, c);
  else if (c != 0.0) acc_add(acc + (int64_t)kAccDigits * w, c, err);
}

// Dependency sweep of one group, barriers as in cta_bfs; each vertex's
// contribution is made by one thread.
template <int kBlock, int kGroup>
__device__ void cta_sweep(const View &g, const Group &G, int nlev, double wsrc, double *P, unsigned long long *acc, int *err,
                          int grp, int tid) {
  using L = CtaLayout<kBlock, kGroup>;
  L::sync(grp);  // the last level's counts have been read
  if (tid < 3) {
    G.n->medium[tid] = 0;
    G.n->large[tid] = 0;
  }
  L::sync(grp);
  for (int lev = nlev - 1, m = 0; lev >= 1; --lev, m = m == 2 ? 0 : m + 1) {
    const int nxt = m == 2 ? 0 : m + 1, next = G.base + lev + 1, a1 = G.lv[lev + 1];
    if (tid == 0) {
      G.n->medium[nxt] = 0;
      G.n->large[nxt] = 0;
    }
    for (int i = G.lv[lev] + tid; i < a1; i += kGroup) {
      const int32_t w = G.S[i];
      const int p0 = g.pair(w), p1 = g.pair(w + 1);
      if (queue_row<L>(G, m, w, p1 - p0)) continue;
      const double r = (double)__ldg(g.rch + w) + 1.0;
      auto row = [&](int q0, int q1, int step) { return bwd_pairs(g, G, q0, q1, step, next); };
      const double sum = p1 - p0 <= kLightPairs ? row(p0, p1, 1) : row_alone(p0, p1, row);
      contribute(P, acc, w, finish(r, w, sum, G.sq, err) * wsrc, err);
    }
    L::sync(grp);
    const int nm = min(*(volatile int *)&G.n->medium[m], L::kQueue), nl = min(*(volatile int *)&G.n->large[m], L::kQueue);
    if (nm | nl) {
      queued_rows<L, kGroup>(
          g, G, nm, nl, tid, [&](int p0, int p1, int step) { return bwd_pairs(g, G, p0, p1, step, next); },
          [&](int32_t w, double sum) {
            contribute(P, acc, w, finish((double)__ldg(g.rch + w) + 1.0, w, sum, G.sq, err) * wsrc, err);
          });
      L::sync(grp);
    }
  }
}

// 1024 / kBlock CTAs per SM at most (the shared-memory buckets), so 64
// registers per thread whatever the block size. Group grp of the CTA takes
// the item's sources s0 + grp, s0 + grp + G, ... one after another (a fixed
// assignment: its FP64 row P is summed in a fixed order), then flushes P into
// the integer counters (any order).
template <int kBlock, int kGroup>
__global__ void __launch_bounds__(kBlock, 1024 / kBlock) tile_cta_kernel(TileArgs a) {
  using L = CtaLayout<kBlock, kGroup>;
  extern __shared__ __align__(16) unsigned char s_raw[];
  const int64_t nmax = a.nmax;
  Ctl &ctl = *reinterpret_cast<Ctl *>(s_raw);
  const int grp = threadIdx.x / kGroup, gtid = threadIdx.x % kGroup;
  unsigned char *mine = s_raw + L::group(grp, nmax);
  // the group's FP64 row (global, L2-resident), if the launch has them
  double *P = a.ws_P ? a.ws_P + ((int64_t)blockIdx.x * L::kG + grp) * a.cap_P : nullptr;
  Group G;
  G.sq = reinterpret_cast<double *>(mine);
  G.d = reinterpret_cast<uint16_t *>(mine + L::d(nmax));
  G.S = reinterpret_cast<uint16_t *>(mine + L::S(nmax));
  G.lv = reinterpret_cast<uint16_t *>(mine + L::lv(nmax));
  G.medium = reinterpret_cast<uint16_t *>(mine + L::q(nmax));
  G.large = G.medium + L::kQueue;
  G.n = reinterpret_cast<Counts *>(mine + L::ctr(nmax));
  G.base = 1 << 16;  // the first source clears the stamps
  unsigned char *slice = s_raw + L::slice(nmax);
  const int tid = threadIdx.x;
  if (tid == 0) {
    mbar_init(&ctl.bar, 1);
    ctl.bcc = -1;
  }
  __syncthreads();
  unsigned phase = 0;
  TileItem it;
  int64_t vo;
  int32_t nb;
  while (next_item(a, ctl, slice, phase, it, vo, nb)) {
    if (P)
      for (int v = gtid; v < nb; v += kGroup) __stcg(P + v, 0.0);
    __syncthreads();
    if (tid == 0) ctl.bcc = it.bcc;  // read again only after the next barrier
    const View g = view_of(a, slice, nb, vo, it.bcc);
    unsigned long long *acc = a.acc + (int64_t)kAccDigits * vo;
    for (int32_t k = it.s0 + grp; k < it.s1; k += L::kG) {  // the group's sources in order: P's sums are fixed
      const int32_t s = source_of(a, k);
      if (G.base + L::kLevels + 2 > 0xffff) {  // stamps start over
        for (int v = gtid; v < (int)((nmax + 1) / 2); v += kGroup) reinterpret_cast<unsigned *>(G.d)[v] = 0;
        G.base = 2;
        L::sync(grp);
      }
      const int nlev = cta_bfs<kBlock, kGroup>(g, G, nb, s, a.err, grp, gtid);
      if (nlev < 0) break;
      cta_sweep<kBlock, kGroup>(g, G, nlev, (double)__ldg(g.rch + s) + 1.0, P, acc, a.err, grp, gtid);
      G.base += nlev + 1;
    }
    __syncthreads();
    if (!P) continue;  // uniform over the grid
    for (int v = gtid; v < nb; v += kGroup) {
      const double c = __ldcg(P + v);
      if (c != 0.0) acc_add(acc + (int64_t)kAccDigits * v, c, a.err);
    }
  }
}

}  // namespace

int block_of(int cls) {
  return cls == kTileCta512 || cls == kTileCta512x8 ? 512 : cls >= kTileCta1024 && cls <= kTileCta1024x8 ? 1024 : kThreads;
}

size_t tile_smem_bytes(int cls, int64_t nmax, int64_t slice_max) {
  const int64_t head = cls == kTileWarp       ? WarpLayout::slice(nmax)
                       : cls == kTileCta      ? CtaLayout<256, 256>::slice(nmax)
                       : cls == kTileCta512   ? CtaLayout<512, 512>::slice(nmax)
                       : cls == kTileCta1024  ? CtaLayout<1024, 1024>::slice(nmax)
                       : cls == kTileCta1024x2 ? CtaLayout<1024, 512>::slice(nmax)
                       : cls == kTileCta1024x4 ? CtaLayout<1024, 256>::slice(nmax)
                       : cls == kTileCta1024x8 ? CtaLayout<1024, 128>::slice(nmax)
                       : cls == kTileCta512x8  ? CtaLayout<512, 64>::slice(nmax)
                                               : CtaLayout<256, 32>::slice(nmax);
  return (size_t)(head + align16(slice_max));
}

int tile_groups(int cls) { return cls == kTileCta1024x2 ? 2 : cls == kTileCta1024x4 ? 4 : cls >= kTileCta1024x8 ? 8 : 1; }

// At most kItemSources: the CTA runs them (a warp each, or one after another)
// from one staged slice; larger BCCs are split so that many CTAs share them, and
// a class with few sources in all gets smaller items, so that it still has
// several per resident CTA -- but an item feeds every warp of the warp class and
// every group of a grouped CTA.
int32_t tile_item_sources(int cls, int64_t grid, int64_t sources) {
  constexpr int64_t kItemSources = 128, kItemsPerCta = 4;
  const int64_t least = cls == kTileWarp ? kTileWarps : tile_groups(cls);
  return (int32_t)std::max<int64_t>(least, std::min<int64_t>(kItemSources, sources / (grid * kItemsPerCta)));
}

int tile_class(int64_t n, int64_t slice_bytes, size_t lim) {
  auto fits = [&](int cls) { return tile_smem_bytes(cls, n, slice_bytes) <= lim; };
  if (n > kTileMaxVertices) return -1;
  if (n <= kTileGroups32 && fits(kTileCta256x8)) return kTileCta256x8;
  if (n <= kTileGroups64 && fits(kTileCta512x8)) return kTileCta512x8;
  if (n <= kTileWarpMaxVertices) return -1;  // the warp class takes more shared memory still
  const int64_t per = kTileSmPerSm / ((int64_t)tile_smem_bytes(kTileCta, n, slice_bytes) + kTileReserved);
  if (per <= 7 && fits(kTileCta1024x8)) return kTileCta1024x8;
  if (per >= 4) return kTileCta;
  if (fits(kTileCta1024x4)) return kTileCta1024x4;
  if (per == 3) return kTileCta;
  if (per == 2) return kTileCta512;
  if (fits(kTileCta1024x2)) return kTileCta1024x2;
  return fits(kTileCta1024) ? kTileCta1024 : -1;
}

size_t tile_smem_limit(int device) {
  int v = 0;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) return 0;
  return (size_t)v;
}

namespace {
const void *tile_fn(int cls) {
  return cls == kTileWarp       ? reinterpret_cast<const void *>(tile_warp_kernel)
         : cls == kTileCta      ? reinterpret_cast<const void *>(tile_cta_kernel<256, 256>)
         : cls == kTileCta512   ? reinterpret_cast<const void *>(tile_cta_kernel<512, 512>)
         : cls == kTileCta1024  ? reinterpret_cast<const void *>(tile_cta_kernel<1024, 1024>)
         : cls == kTileCta1024x2 ? reinterpret_cast<const void *>(tile_cta_kernel<1024, 512>)
         : cls == kTileCta1024x4 ? reinterpret_cast<const void *>(tile_cta_kernel<1024, 256>)
         : cls == kTileCta1024x8 ? reinterpret_cast<const void *>(tile_cta_kernel<1024, 128>)
         : cls == kTileCta512x8  ? reinterpret_cast<const void *>(tile_cta_kernel<512, 64>)
                                 : reinterpret_cast<const void *>(tile_cta_kernel<256, 32>);
}
cudaError_t allow_smem(int cls) {
  return cudaFuncSetAttribute(tile_fn(cls), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemPerCta);
}
}  // namespace

int tile_ctas_per_sm(int cls, size_t smem) {
  int n = 0;
  if (allow_smem(cls) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_fn(cls), block_of(cls), smem) != cudaSuccess) return 0;
  return n;
}

cudaError_t launch_tile(int cls, const TileArgs &a, int grid, size_t smem, cudaStream_t stream) {
  const cudaError_t e = allow_smem(cls);
  if (e != cudaSuccess) return e;
  switch (cls) {
    case kTileWarp: tile_warp_kernel<<<grid, kThreads, smem, stream>>>(a); break;
    case kTileCta: tile_cta_kernel<256, 256><<<grid, 256, smem, stream>>>(a); break;
    case kTileCta512: tile_cta_kernel<512, 512><<<grid, 512, smem, stream>>>(a); break;
    case kTileCta1024: tile_cta_kernel<1024, 1024><<<grid, 1024, smem, stream>>>(a); break;
    case kTileCta1024x2: tile_cta_kernel<1024, 512><<<grid, 1024, smem, stream>>>(a); break;
    case kTileCta1024x4: tile_cta_kernel<1024, 256><<<grid, 1024, smem, stream>>>(a); break;
    case kTileCta1024x8: tile_cta_kernel<1024, 128><<<grid, 1024, smem, stream>>>(a); break;
    case kTileCta512x8: tile_cta_kernel<512, 64><<<grid, 512, smem, stream>>>(a); break;
    case kTileCta256x8: tile_cta_kernel<256, 32><<<grid, 256, smem, stream>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace bcg
