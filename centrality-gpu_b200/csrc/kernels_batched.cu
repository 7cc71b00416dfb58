// BATCHED schedule: many sources per pass as a bitmask multi-source BFS over
// each BCC with its degree-2 chains contracted.
//
// Contracted graph. Within a BCC the core vertices (local ids < n_plain) keep
// their arcs to each other ("unit arcs"); a chain c of k degree-2 vertices
// between the core endpoints L and R becomes one arc L-R of length k+1 in
// both endpoint rows ("chain arcs", listed after the unit arcs of a row).
// Chain vertices never enter the level-synchronous phases: their levels, path
// counts and dependencies follow in closed form from the two endpoint columns
// (the reference's ear postprocessing, Codes/postprocesses.cu:205-351, done
// here for every source of the pass at once).
//
// Slots. One pass ("batch") covers up to B = 32*W sources of one BCC (on small
// cores the kernel runs several passes as one, see merge_passes):
//   core source     level 0 at the vertex;
//   chain source    the vertex at position p (0-based from L) of a chain of
//                   k vertices: seeded at L on level p+1 and at R on level
//                   k-p, one path each (its two directions along the chain).
// State of the core vertices, vertex-major and slot-minor ([v][B]) so a warp
// reads the 32 slots of a word as one coalesced row segment:
//   d[v][b]     level (int32)            sigma[v][b] path count (FP64, scaled)
//   q[v][b]     (reach(v)+1+delta)/sigma (FP64, or FP32 in the compensated mode)
//   lm[t][v][w] bitmask of the slots that reach v at level t: the frontier of
//               the forward phase and the successor test of the backward phase
// Forward: level-synchronous pull. A core vertex still unseen by some slot
// scans its row once per 128 slots: a unit arc to u hits the slots in
// lm[t][u], a chain arc of length k+1 hits those in lm[t-k][u]; the hits'
// path counts are summed (the reference's per-source atomicCAS/atomicAdd BFS,
// Codes/kernels_free.cu:286-362).
// Backward: successor form (Codes/kernels_free.cu:377-421), delta(v) =
// sigma(v) * sum of q over successors, where a chain arc of length k+1 is a
// successor arc when the chain carries the far end's shortest paths (the far
// end sits on level lev+k+1), plus what v receives from the chain vertices
// themselves: a closed form in prefix sums of reach+1 along the chain and the
// two ends' path counts, evaluated for every (vertex, slot) in one parallel
// phase between the forward and the backward sweeps.
// Chain vertices: one warp per chain evaluates every chain vertex's dependency
// from the endpoint columns, two neighbouring slots a lane.
// Path counts carry a per-(slot, level) power-of-two base X so deep graphs do
// not overflow FP64: a level is rescaled when its largest count passes
// 2^rescale_exp (900 by default).
// BC: FP64 partials per vertex and 128 slots, summed in fixed order: the same bits
// on every run of the same unit ranges (the reference uses FP32 atomics,
// Codes/kernels_free.cu:423-426). Passes that run as one are summed as one.
// The whole GPU works on one batch at a time: a cooperative persistent kernel
// with a grid barrier whose waits are bounded (error flag, no hang).
#include "accum.cuh"
#include "batched.h"
#include "common.cuh"
#include "internal.h"

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>
#include <new>
#include <numeric>
#include <type_traits>
#include <utility>
#include <vector>

namespace bcg {

namespace {

constexpr int kThreads = 256;
constexpr int kWarpsPerCta = kThreads / 32;
// Core rows longer than kHeavyDeg arcs are scanned in chunks by whole CTAs
// (RMAT-20 at 512 sources per pass: 143.7 / 153.7 / 160.4 / 160.4 / 162.3 /
// 156.1 GTEPS for 128 / 256 / 512 / 1024 / 2048 / 4096) ...
#ifndef BCGPU_BATCHED_HEAVY_DEG
#define BCGPU_BATCHED_HEAVY_DEG 1024
#endif
constexpr int kHeavyDeg = BCGPU_BATCHED_HEAVY_DEG;
// ... or than this, on cores small enough that one row is a level's critical path
// (R-MAT 14, 16 passes of 512 one by one / by 8: 61.9 / 39.2 ms for 32, 54.9 /
// 32.1 for 128, 55.8 / 31.3 for 512).
constexpr int kHeavyDegSmall = 512;
constexpr int kSmallCore = 16384;  // cores below this many vertices use kHeavyDegSmall
// Where rows of up to twice that length are as many as the warps in flight, a warp
// each keeps them all busy, and a chunked row's partial sum in memory and its
// combine are saved; where they are few, a level waits for them. Two passes of 512
// at 20% and 60% of the source order, rows up to 1024 / 2048 arcs on a warp, by rows
// of 1025 to 2048 arcs: 4,845 (R-MAT 20) 167 and 143 / 159 and 135 ms, 5,985 (R-MAT
// 21, 12 edges a vertex) 275 and 222 / 264 and 213, 4,843 (R-MAT 20 of 24) 216 and
// 169 / 216 and 171; 989 (R-MAT 20 of 8) 94 and 80 / 107 and 92, 460 and 362
// (skewed random, 34 and 37 million arcs) 87 and 180 / 106 and 219; R-MAT 17 and 18
// (two passes in the middle) 22.3 and 46.4 / 23.1 and 51.1, R-MAT 19 even.
constexpr int kHeavyDegMany = 2 * kHeavyDeg;
constexpr int64_t kManyRows = 4096;  // rows of kHeavyDeg to kHeavyDegMany arcs that make them many
#ifndef BCGPU_BATCHED_CHUNK
#define BCGPU_BATCHED_CHUNK 2048
#endif
constexpr int kChunkArcs = BCGPU_BATCHED_CHUNK;  // arcs per heavy chunk
constexpr int kHalf = 4;           // words per pass over a vertex row
// Resident CTAs per SM the kernel is compiled for (registers per thread =
// 65536 / (kThreads * kMinCtas)); profiling builds may override it. Two passes of
// 512 sources take, for 5 / 4 CTAs per SM: R-MAT 20 139.4 / 139.6 ms, R-MAT 17
// 23.8 / 22.3 and in FP64 24.6 / 22.7; all passes of R-MAT 14 140.7 / 139.5. (With one
// hit in flight R-MAT 20 took 164.9 / 155.0 / 158.1 ms for 4 / 5 / 6.)
#ifndef BCGPU_BATCHED_MIN_CTAS
#define BCGPU_BATCHED_MIN_CTAS 4
#endif
constexpr int kMinCtas = BCGPU_BATCHED_MIN_CTAS;
// Light-row tasks per warp and level at least (smaller vertex blocks when
// the core is small), so the slowest tasks at a level's end are short: on
// RMAT-20 (512 sources per pass) 8 / 16 / 32 gave 147.2 / 150.4 / 151.8 GTEPS.
#ifndef BCGPU_BATCHED_TASKS
#define BCGPU_BATCHED_TASKS 32
#endif
constexpr int kTasksPerWarp = BCGPU_BATCHED_TASKS;

// One source of a pass. chain < 0: the core vertex src (level 0). Otherwise
// src is the chain vertex at position pos of chain `chain` (global index).
struct Slot {
  int32_t src, chain, pos, pad;
};

// Where a chain source enters the core: slot of pass `pass` reaches core vertex
// v on `level` with one path along its chain.
struct Seed {
  int32_t v, level, slot, pass;
};

struct Batch {
  int32_t bcc, nslots, words, nseeds;
  int32_t max_seed;  // deepest seed level (0: none)
  int32_t kmax;      // longest chain of the BCC: the longest arc is kmax+1
  int32_t heavy_deg; // rows longer than this are chunked over whole CTAs
  int32_t narm;      // entries of the pass's arming list
  int64_t slot_off, seed_off;
  int64_t arm_off;   // arming list: (vertex, level) of the core sources and seeded vertices
};

// Control block in global memory (one per plan).
struct Ctrl {
  unsigned int bar_count;
  unsigned int bar_gen;
  int more[2];    // forward, by level parity: some slot found a new vertex on the level
  int rescale[2]; // forward, by level parity: some slot needs a rescale on the level
  int range_err;  // FP32 q left FP32's exponent range in this batch
  int pad;
  unsigned long long found;  // forward: (core vertex, slot) pairs reached so far
};

constexpr int32_t kNoSlot = -2;

struct Args {
  // contracted rows of the core vertices; BCC b's rows start at hvo[b]
  const int64_t *hvo;
  const int64_t *hrow;    // [n_core_rows + n_bcc] global arc offsets
  const int64_t *hsplit;  // first chain arc of each row
  const int32_t *hcol;    // neighbour (local core id)
  const int32_t *hk;      // chain arcs: vertices on the chain (the arc is one longer)
  const int32_t *hcid;    // chain arcs: chain index * 2 + (the row's vertex is the chain's right end)
  const int32_t *reach;
  const int64_t *vtx_off;
  const int32_t *n_plain;
  // chains (global index)
  const int64_t *chain_off;
  const int32_t *chain_start, *chain_len, *chain_l, *chain_r;
  const int64_t *cpre_off;  // chain -> its k+1 prefix sums of reach+1 (from the left end) in cpre; -1: all reach 0
  const double *cpre;
  // heavy rows (contracted degree > kHeavyDeg), chunked
  const int64_t *heavy_off;  // per BCC range in heavy[]
  const int32_t *heavy;      // local ids
  const int64_t *hchunk_off; // per BCC range in the chunk table
  const int32_t *hchunk_v;   // chunk -> heavy index (within its BCC's heavy list)
  const int64_t *hchunk_e0;  // chunk arc range [e0, e1) (global arc offsets)
  const int64_t *hchunk_e1;
  const int32_t *hfirst;     // heavy index -> first chunk (BCC-relative), hfirst[h+1] ends it
  double *hacc;              // [chunks][W][32] partial successor / path-count sums
  uint32_t *hmask;           // [chunks][W] partial masks
  const Batch *batches;
  const Slot *slots;
  const Seed *seeds;
  const int2 *arms;
  int64_t b0, b1;
  // workspace (core rows)
  int32_t *d;
  double *sig;
  void *q;
  uint32_t *lm;     // [tcap+2][n_cap][W]
  uint32_t *seen;   // [n_cap][W]
  int32_t *lmin;    // [n_cap] first level on which some slot reached the vertex
  int32_t *armed;   // [n_cap] first level on which some slot can reach the vertex (a neighbour was reached)
  // [4*(tcap+3)+2] work counters: light rows forward (t), backward (tcap+3+lev); heavy chunks (2*(tcap+3)+t,
  // 3*(tcap+3)+lev); chain in-flow (4*(tcap+3)); chain vertices (4*(tcap+3)+1)
  int *wq;
  double *bcpart;   // [n_cap][W] BC partials of the core vertices (a light row's 128 slots in their first word)
  double *cdep;     // [n_cap][W][32] dependency a core vertex receives from its chains' vertices
  double *wsrc;     // [B] reach(source)+1 of each slot of the pass
  int32_t *schain;  // [B] chain of each slot's source (-1: a core vertex; kNoSlot: no slot)
  int32_t *X;       // [B][tcap+2]
  int32_t *rexp;    // [B] per-level max exponent (rescale)
  int64_t n_cap;    // core rows allocated (>= largest core)
  int32_t W;        // words per row (row stride): those of `merge` passes
  int32_t width;    // slots of a pass
  int32_t merge;    // passes run as one, at most
  int32_t tcap;     // levels allocated
  int32_t rescale_exp;
  unsigned long long wait_ns;  // limit of one grid-barrier wait
  int32_t pad;
  double *bc;
  Ctrl *ctrl;
  int *err;
  int *redo;        // per batch: 1 = FP32 range exceeded, contributions not added
};

__device__ __forceinline__ bool failed(const Args &a) { return *(volatile int *)a.err != kDevOk; }

// The same answer for every thread of the CTA (thread 0 decides).
__device__ __forceinline__ bool cta_failed(const Args &a) {
  __shared__ int s_fail;
  __syncthreads();
  if (threadIdx.x == 0) s_fail = failed(a) ? 1 : 0;
  __syncthreads();
  return s_fail != 0;
}

// Grid-wide barrier for a cooperative launch. Waits are bounded: after
// a.wait_ns of device time the CTA records kDevTimeout and continues; once
// any error is flagged every barrier returns at once so the kernel drains
// quickly.
__device__ void grid_sync(const Args &a) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned int *gen = &a.ctrl->bar_gen;
    const unsigned int g = *gen;
    __threadfence();
    const unsigned int arrived = atomicAdd(&a.ctrl->bar_count, 1u);
    if (arrived == gridDim.x - 1) {
      a.ctrl->bar_count = 0;
      __threadfence();
      atomicAdd(&a.ctrl->bar_gen, 1u);
    } else {
      wait_while_equal(gen, g, a.wait_ns, a.err, [&] { return failed(a); });
    }
    __threadfence();
  }
  __syncthreads();
}

// Phase timers for profiling builds only (-DBCGPU_PHASE_TIMERS): CTA 0's
// thread 0 accumulates %globaltimer deltas between grid barriers.
#ifdef BCGPU_PHASE_TIMERS
__device__ unsigned long long g_phase_ns[32];
__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
#define PHASE_INIT() unsigned long long ph_t = (blockIdx.x == 0 && threadIdx.x == 0) ? gtimer() : 0ull
#define PHASE_MARK(id)                                             \
  do {                                                             \
    if (blockIdx.x == 0 && threadIdx.x == 0) {                     \
      const unsigned long long ph_n = gtimer();                    \
      g_phase_ns[id] += ph_n - ph_t;                               \
      ph_t = ph_n;                                                 \
    }                                                              \
  } while (0)
#define PHASE_COUNT(id) do { if (blockIdx.x == 0 && threadIdx.x == 0) g_phase_ns[id] += 1; } while (0)
#else
#define PHASE_INIT() do {} while (0)
#define PHASE_MARK(id) do {} while (0)
#define PHASE_COUNT(id) do {} while (0)
#endif

__device__ __forceinline__ int64_t gwarp() { return ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; }
__device__ __forceinline__ int64_t nwarps() { return ((int64_t)gridDim.x * blockDim.x) >> 5; }

// ---- compensated FP32 accumulation of terms >= 0: the exact error of each sum
// (Dekker's fast two-sum, the larger of the two first) goes into c
struct Comp32 {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float t = s + x;
    c += fminf(s, x) - (t - fmaxf(s, x));
    s = t;
  }
  __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

// ============================================================ chain math ===
// A stretch of a chain between two ends A and B holding m chain vertices,
// seen from A: its vertex i (0 <= i < m) lies i+1 arcs from A and m-i from B.
// pre(x) is the sum of reach+1 over its first x vertices counted from A.
// Prefix sum x of a chain: P[x], or x itself on a chain whose vertices have
// nothing hanging off them (P null: no table, no load).
__device__ __forceinline__ double chain_pre(const double *P, int x) { return P ? __ldg(P + x) : (double)x; }

struct Stretch {
  const double *P;  // the chain's prefix sums from its left end (k+1 entries), or null (all reach 0)
  int lo, hi;       // chain positions [lo, hi) of the stretch
  bool rev;         // A is the right-hand end (position hi)
  __device__ __forceinline__ int m() const { return hi - lo; }
  __device__ __forceinline__ double pre(int x) const {
    return rev ? chain_pre(P, hi) - chain_pre(P, hi - x) : chain_pre(P, lo + x) - chain_pre(P, lo);
  }
  __device__ __forceinline__ double wt(int i) const { return pre(i + 1) - pre(i); }
  __device__ __forceinline__ Stretch flip() const { return Stretch{P, lo, hi, !rev}; }
};

// An end of a stretch for one slot, as loaded: its level d, path count
// sigma = s * 2^x and q = qs * 2^-x (qs only read when the stretch carries
// the end's shortest paths). The slot's own source is {0, 0, 1, 0}.
struct End {
  int d, x;
  double s, qs;
};
__device__ __forceinline__ End source_end() { return End{0, 0, 1.0, 0.0}; }

// The share of A's paths, sA / (sA + sB), while no level was rescaled: one division
// where 1 / (1 + sB / sA) takes two. Halves, so that the sum of two counts that
// FP64 holds is one as well.
__device__ __forceinline__ double path_share(double sA, double sB) { return 0.5 * sA / (0.5 * sA + 0.5 * sB); }

// Dependency of stretch vertex i on the slot's source when i takes its
// shortest paths from A (2i < D): the chain vertices beyond i on the A-fed
// side each add reach+1; the last A-fed vertex either ties (shares its paths
// with B: adds its reach+1 times sigma_A / (sigma_A + sigma_B)) or, when it is
// the vertex next to B and B's shortest paths run through the stretch, passes
// on sigma_A * q(B) (kTail). i = -1 gives what A itself receives.
template <bool kTail>
__device__ __forceinline__ double fed_dep(const Stretch &s, int i, const End &A, const End &B, int D) {
  const int m = s.m();
  const int P = min(m - 1, D / 2);  // last vertex fed from A
  if ((D & 1) == 0 && D / 2 <= m - 1) return s.pre(P) - s.pre(i + 1) + s.wt(P) / (1.0 + scale2(B.s / A.s, B.x - A.x));
  double v = s.pre(P + 1) - s.pre(i + 1);
  if (kTail && P == m - 1 && B.d == A.d + m + 1) v += scale2(A.s * B.qs, A.x - B.x);
  return v;
}

// Dependency of stretch vertex i (0 <= i < m) on the slot's source (out of
// line: only the rare slots whose source sits on the chain take this path).
__device__ __noinline__ double stretch_dep(const Stretch &s, int i, const End &A, const End &B) {
  const int m = s.m();
  const int D = B.d + m - A.d - 1;  // vertex i is fed from A iff 2i <= D, from B iff 2i >= D
  if (2 * i < D) return fed_dep<true>(s, i, A, B, D);
  if (2 * i > D) return fed_dep<true>(s.flip(), m - 1 - i, B, A, A.d + m - B.d - 1);
  return 0.0;  // fed from both ends: no successor on the chain
}

// What end A receives from the stretch's vertices (its neighbour on the
// stretch is its successor iff that neighbour is fed from A: D >= 0), less
// the term through B (sigma_A * q(B) when B's paths run through the
// stretch), which the backward sweep adds as a successor arc.
__device__ __forceinline__ double end_dep(const Stretch &s, const End &A, const End &B) {
  const int D = B.d + s.m() - A.d - 1;
  if (s.m() == 0 || D < 0) return 0.0;
  return fed_dep<false>(s, -1, A, B, D);
}

// ============================================================== forward ====
// A task is one vertex row for a quarter: kHalf 32-slot words, 128 slots. Lane j
// loads arc j's neighbour and its mask words (one aligned 16-byte load); the arcs
// that hit go to the warp's shared memory in arc order and are walked there, each
// with one load of its values: lane l has slots 4l ... 4l+3 of the quarter, whose
// values are one sector (FP64) or half of one. Adds follow arc order, so sums are
// deterministic.
constexpr int kLaneSlots = 4;  // slots of a lane: consecutive ones
static_assert(kLaneSlots * 32 == kHalf * 32, "a warp's lanes cover a quarter");

// Per-slot accumulator of a row pass: FP64, or compensated FP32.
template <bool kComp>
struct Acc {
  double s = 0.0;
  __device__ __forceinline__ void add(double x) { s += x; }
  __device__ __forceinline__ double value() const { return s; }
};
template <>
struct Acc<true> {
  Comp32 c;
  __device__ __forceinline__ void add(double x) { c.add((float)x); }
  __device__ __forceinline__ double value() const { return c.value(); }
};

// Per-warp shared memory: partial sums (by slot of the quarter) and hit masks of
// the heavy-row chunks, combined across the CTA's warps in fixed order; the hits
// of a strip of 32 arcs: masks, neighbours, levels.
struct WarpScratch {
  double acc[kHalf * 32];
  uint32_t any[kHalf];
  uint32_t hit[32][kHalf];
  uint32_t hit_u[32];
  int32_t hit_lvl[32];
};

// A lane's place in a quarter: its word and the first of its slots' bits there.
__device__ __forceinline__ int lane_word(int lane) { return lane >> 3; }
__device__ __forceinline__ int lane_bit(int lane) { return (lane & 7) * kLaneSlots; }

// A lane's four values, past L1 (other SMs wrote them): one load.
__device__ __forceinline__ void ld_slots(const double *p, double (&x)[kLaneSlots]) {
  asm volatile("ld.global.cg.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3]) : "l"(p));
}
__device__ __forceinline__ void ld_slots(const float *p, float (&x)[kLaneSlots]) {
  const float4 v = __ldcg(reinterpret_cast<const float4 *>(p));
  x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void st_slots(double *p, const double (&x)[kLaneSlots]) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x[0]), "d"(x[1]), "d"(x[2]), "d"(x[3]) : "memory");
}
__device__ __forceinline__ void st_slots(float *p, const float (&x)[kLaneSlots]) {
  *reinterpret_cast<float4 *>(p) = make_float4(x[0], x[1], x[2], x[3]);
}

// The word whose bits the lanes of an eight hold, in all of them.
__device__ __forceinline__ uint32_t word_of(uint32_t bits, int lane) {
  uint32_t m = bits << lane_bit(lane);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) m |= __shfl_xor_sync(0xffffffffu, m, o);
  return m;
}

__device__ __forceinline__ uint4 ld4(const uint32_t *p) { return __ldcg(reinterpret_cast<const uint4 *>(p)); }

// Loads the kHalf-word mask row at p (first nw words, nw a multiple of 4).
__device__ __forceinline__ void load_row(const uint32_t *p, int nw, uint32_t (&m)[kHalf]) {
#pragma unroll
  for (int g = 0; g < kHalf / 4; ++g) {
    const uint4 x = 4 * g < nw ? ld4(p + 4 * g) : make_uint4(0, 0, 0, 0);
    m[4 * g] = x.x; m[4 * g + 1] = x.y; m[4 * g + 2] = x.z; m[4 * g + 3] = x.w;
  }
}

// Walks the arcs of a strip of 32 (lane j: neighbour u, level lvl, hit masks f)
// that hit in some word, in arc order, and adds their values (vrow: this lane's
// first slot); got: the lane's slots that were hit.
template <typename T, bool kComp, int kLev>
__device__ __forceinline__ void walk_hits(const Args &a, WarpScratch &S, const T *vrow, uint32_t u, int lvl,
                                          const uint32_t (&f)[kHalf], uint32_t &got, Acc<kComp> (&acc)[kLaneSlots],
                                          int lane, int w0 = 0, int t = 0, bool scaled = false) {
  const bool mine = (f[0] | f[1] | f[2] | f[3]) != 0u;
  const uint32_t hits = __ballot_sync(0xffffffffu, mine);
  if (!hits) return;
  if (mine) {
    const int at = __popc(hits & ((1u << lane) - 1u));
    *reinterpret_cast<uint4 *>(S.hit[at]) = make_uint4(f[0], f[1], f[2], f[3]);
    S.hit_u[at] = u;
    if (kLev) S.hit_lvl[at] = lvl;
  }
  __syncwarp();
  // level exponent bases of the lane's slots: slot k's at xb + k * (tcap + 2)
  const int32_t *xb = kLev ? a.X + (int64_t)(w0 * 32 + kLaneSlots * lane) * (a.tcap + 2) : nullptr;
  const uint32_t *mine_at = &S.hit[0][lane_word(lane)];
  const int sh = lane_bit(lane), n = __popc(hits);
  const int64_t stride = (int64_t)a.W * 32;
  int i = 0;
  if (kLev == 0 && sizeof(T) == 4) {  // two hits' loads in flight: FP64 values would spill
    for (; i + 2 <= n; i += 2) {
      const uint32_t m0 = mine_at[i * kHalf] >> sh & 15u, m1 = mine_at[i * kHalf + kHalf] >> sh & 15u;
      got |= m0 | m1;
      T x[kLaneSlots] = {(T)0, (T)0, (T)0, (T)0}, y[kLaneSlots] = {(T)0, (T)0, (T)0, (T)0};
      if (m0) ld_slots(vrow + (int64_t)S.hit_u[i] * stride, x);
      if (m1) ld_slots(vrow + (int64_t)S.hit_u[i + 1] * stride, y);
#pragma unroll
      for (int k = 0; k < kLaneSlots; ++k) {
        acc[k].add((double)(m0 >> k & 1u ? x[k] : (T)0));
        acc[k].add((double)(m1 >> k & 1u ? y[k] : (T)0));
      }
    }
  }
  for (; i < n; ++i) {
    const uint32_t m = mine_at[i * kHalf] >> sh & 15u;
    const T *vu = vrow + (int64_t)S.hit_u[i] * stride;
    got |= m;
    T x[kLaneSlots] = {(T)0, (T)0, (T)0, (T)0};
    if (m) ld_slots(vu, x);
    if (kLev && scaled) {
      const int lj = S.hit_lvl[i];
#pragma unroll
      for (int k = 0; k < kLaneSlots; ++k)
        if (m >> k & 1u) {
          const int xl = __ldcg(xb + k * (a.tcap + 2) + lj), xt = __ldcg(xb + k * (a.tcap + 2) + t);
          x[k] = (T)scale2((double)x[k], kLev == 1 ? xl - xt : xt - xl);
        }
    }
#pragma unroll
    for (int k = 0; k < kLaneSlots; ++k) acc[k].add((double)(m >> k & 1u ? x[k] : (T)0));
  }
  __syncwarp();  // the next strip writes the same places
}

// One pull / successor pass over arcs [e0, e1) for words [w0, w0+nw):
//   filt[k]  the slots of word w0+k that are looked for (uniform)
//   masks    level masks: of level t (unit arcs, kLev == 0), or the
//            level-0 base of lm for chain arcs, whose arc e reads level
//            t - hk[e] (kLev == 1, forward: sigma rebased from that level's
//            X to level t's) or level t + hk[e] (kLev == 2, backward: q
//            rebased to level t's X; levels above tend are empty)
//   vals     per-slot values gathered on a hit (sigma, or q)
// Adds into acc, and the lane's hit slots into got.
template <typename T, bool kComp, int kLev>
__device__ __forceinline__ void row_pass(const Args &a, WarpScratch &S, const uint32_t *masks, const T *vals, int64_t e0,
                                         int64_t e1, int w0, int nw, const uint32_t (&filt)[kHalf], uint32_t &got,
                                         Acc<kComp> (&acc)[kLaneSlots], int lane, int t, bool scaled = false, int tend = 0) {
  const int W = a.W;
  for (int64_t base = e0; base < e1; base += 32) {
    const int64_t e = base + lane;
    bool valid = e < e1;
    const int32_t u = valid ? ldg(a.hcol + e) : 0;
    int lvl = t;
    if (kLev == 1) {
      lvl = valid ? t - ldg(a.hk + e) : -1;
      valid = valid && lvl >= 0;
    } else if (kLev == 2) {
      lvl = valid ? t + ldg(a.hk + e) : INT_MAX;
      valid = valid && lvl <= tend;
    }
    uint32_t f[kHalf];
    const uint32_t *mrow = kLev ? masks + ((int64_t)(valid ? lvl : 0) * a.n_cap + u) * W + w0 : masks + (int64_t)u * W + w0;
    load_row(mrow, valid ? nw : 0, f);
#pragma unroll
    for (int k = 0; k < kHalf; ++k) f[k] &= filt[k];
    walk_hits<T, kComp, kLev>(a, S, vals + (int64_t)w0 * 32 + kLaneSlots * lane, u, lvl, f, got, acc, lane, w0, t, scaled);
  }
}

// Path counts that a lane's slots (the first: b, of kN) of the forward step got:
// their levels and counts (the heaviest count of a level that needs rescaling is
// noted). Slots outside `got` keep theirs.
template <int kN>
__device__ __forceinline__ void put_counts(const Args &a, int32_t v, int b, int t, uint32_t got, const double (&acc)[kN]) {
  const int64_t idx = (int64_t)v * a.W * 32 + b;
  bool whole = false;
  if constexpr (kN == kLaneSlots) {
    whole = got == 15u;
    if (whole) {
      *reinterpret_cast<int4 *>(a.d + idx) = make_int4(t + 1, t + 1, t + 1, t + 1);
      st_slots(a.sig + idx, acc);
    }
  }
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    if (!(got >> k & 1u)) continue;
    if (!whole) {
      a.d[idx + k] = t + 1;
      a.sig[idx + k] = acc[k];
    }
    if (exp_bits(acc[k]) - 1023 >= a.rescale_exp && acc[k] > pow2(a.rescale_exp)) {  // acc > 2^rescale_exp, acc normal
      atomicMax(a.rexp + b + k, exp_bits(acc[k]) - 1023);
      a.ctrl->rescale[t & 1] = 1;
    }
  }
}

// Stores the result of one (vertex, word) of a heavy row; lane 0 returns
// the number of slots that reached the vertex.
__device__ __forceinline__ int finish_pull(const Args &a, int32_t v, int w, int t, uint32_t newm, int lane,
                                           double acc) {
  if (!newm) return 0;
  put_counts<1>(a, v, w * 32 + lane, t, newm >> lane & 1u, {acc});
  if (lane == 0) {
    a.lm[((int64_t)(t + 1) * a.n_cap + v) * a.W + w] = newm;
    a.seen[(int64_t)v * a.W + w] |= newm;
    atomicMin(a.lmin + v, t + 1);
  }
  return lane == 0 ? __popc(newm) : 0;
}

// Arms the neighbours of a vertex first reached on level lvl: a neighbour
// across an arc of length k+1 can be reached from it on level lvl+k+1.
__device__ __forceinline__ void arm_arcs(const Args &a, int64_t e0, int64_t e1, int lvl, int64_t tid, int64_t nthr) {
  for (int64_t e = e0 + tid; e < e1; e += nthr) atomicMin(a.armed + ldg(a.hcol + e), lvl + 1 + ldg(a.hk + e));
}

// ============================================================== backward ===

__device__ __forceinline__ int level_index(const Args &a, int d) { return min(max(d, 0), a.tcap + 1); }
__device__ __forceinline__ int level_base(const Args &a, int b, int d) {
  return __ldcg(a.X + (int64_t)b * (a.tcap + 2) + level_index(a, d));
}

// What a slot of an end receives from a chain of k vertices with prefix sums P (out
// of line: chains with something hanging off, rescaled levels, and the slots whose
// source sits on the chain, at pos >= 0).
__device__ __noinline__ double chain_in_any(const double *P, int k, bool right, int pos, const End &A, const End &B) {
  if (pos < 0) return end_dep(Stretch{P, 0, k, right}, A, B);
  return end_dep(right ? Stretch{P, pos + 1, k, true} : Stretch{P, 0, pos, false}, A, source_end());  // ends at the source
}

// What core vertex v receives from the vertices of its chains, for 32 * kInSlots
// slots, this lane's from b on (the part that needs only forward results): cdep.
// Chain-arc data are loaded lane-parallel, 32 arcs at a time, and handed around; an
// arc's levels and path counts at its far end are loaded together (a tie needs the
// path counts on about half the slots, so a warp nearly always needs them). Bound
// by the instructions of the closed form, and by registers. Two passes of 512 on
// R-MAT 20: 23.9 ms with one slot a lane and two divisions a tie; 17.8 with two
// slots; with two or four arcs in flight 20.6 and 23.3, with four slots 31.8 (spills).
constexpr int kInSlots = 2;
__device__ __forceinline__ void chain_in(const Args &a, const Slot *slots, int32_t v, int b, int64_t c0, int64_t c1,
                                         int lane, bool scaled) {
  const int64_t stride = (int64_t)a.W * 32;
  const int64_t iv = (int64_t)v * stride + b;
  const int2 dv = __ldcg(reinterpret_cast<const int2 *>(a.d + iv)), cv = __ldcg(reinterpret_cast<const int2 *>(a.schain + b));
  const double2 sv = __ldcg(reinterpret_cast<const double2 *>(a.sig + iv));
  const int32_t dA[kInSlots] = {dv.x, dv.y}, ch[kInSlots] = {cv.x, cv.y};
  const double sA[kInSlots] = {sv.x, sv.y};
  double sum[kInSlots] = {0.0, 0.0};
  for (int64_t base = c0; base < c1; base += 32) {
    const int64_t e = base + lane;
    int32_t u = 0, cid = 0, k = 0;
    int64_t poff = 0;
    if (e < c1) {
      u = ldg(a.hcol + e);
      cid = ldg(a.hcid + e);
      k = ldg(a.hk + e);
      poff = ldg(a.cpre_off + (cid >> 1));
    }
    const int cnt = (int)min((int64_t)32, c1 - base);
    for (int j = 0; j < cnt; ++j) {
      const int64_t iu = (int64_t)__shfl_sync(0xffffffffu, u, j) * stride + b;
      const int2 dB = __ldcg(reinterpret_cast<const int2 *>(a.d + iu));
      const double2 sB = __ldcg(reinterpret_cast<const double2 *>(a.sig + iu));
      const int cj = __shfl_sync(0xffffffffu, cid, j), kj = __shfl_sync(0xffffffffu, k, j);
      const int64_t pj = __shfl_sync(0xffffffffu, poff, j);
#pragma unroll
      for (int r = 0; r < kInSlots; ++r) {
        const bool same = ch[r] == (cj >> 1);  // the source sits on this chain
        const int db = r ? dB.y : dB.x;
        const double sb = r ? sB.y : sB.x;
        if (!same && pj < 0 && !scaled) {
          // nothing hangs off the chain: prefix sums are positions; the
          // vertices up to P = D/2 are fed from A, the one at D/2 ties when D is even
          const int D = db + kj - dA[r] - 1, P = D >> 1;
          if (D < 0) continue;
          if (!(D & 1) && P < kj) sum[r] += (double)P + path_share(sA[r], sb);
          else sum[r] += (double)(min(kj - 1, P) + 1);
        } else if (ch[r] != kNoSlot) {
          const End A{dA[r], scaled ? level_base(a, b + r, dA[r]) : 0, sA[r], 0.0};
          const End B{db, scaled ? level_base(a, b + r, db) : 0, sb, 0.0};
          sum[r] += chain_in_any(pj < 0 ? nullptr : a.cpre + pj, kj, cj & 1, same ? slots[b + r].pos : -1, A, B);
        }
      }
    }
  }
  *reinterpret_cast<double2 *>(a.cdep + iv) = make_double2(sum[0], sum[1]);
}

// delta and q of a lane's slots (the first: b, of kN) of a vertex at level lev, and
// the BC partial of the warp's slots (in word w0's place); every load is issued
// before the first use.
template <typename QT, int kN>
__device__ __forceinline__ void finish_dep(const Args &a, int32_t reach, int32_t v, int w0, int b, int lev, uint32_t act,
                                           int lane, const double (&sum)[kN], bool chains, bool scaled) {
  constexpr bool kF32 = sizeof(QT) == 4;
  const int64_t idx = (int64_t)v * a.W * 32 + b;
  double sv[kN], in[kN], ws[kN];
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    sv[k] = 1.0;
    in[k] = ws[k] = 0.0;
  }
  if (act) {
    if constexpr (kN == kLaneSlots) {
      ld_slots(a.sig + idx, sv);
      ld_slots(a.wsrc + b, ws);
      if (chains) ld_slots(a.cdep + idx, in);
    } else {
      sv[0] = __ldcg(a.sig + idx);
      ws[0] = __ldcg(a.wsrc + b);
      if (chains) in[0] = __ldcg(a.cdep + idx);
    }
  }
  double contrib = 0.0;
  QT qs[kN];
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    if (!(act >> k & 1u)) continue;
    const int64_t xb = (int64_t)(b + k) * (a.tcap + 2) + lev;
    const int xd = scaled ? a.X[xb] - a.X[xb + 1] : 0;
    const double delta = scale2(sv[k] * sum[k], xd) + in[k];
    const double qv = ((double)reach + 1.0 + delta) / sv[k];
    if (kF32) {
      const double aq = fabs(qv);
      if (!(aq >= (double)FLT_MIN * 0x1p24 && aq <= (double)FLT_MAX * 0x1p-24)) atomicExch(&a.ctrl->range_err, 1);
    }
    qs[k] = (QT)qv;
    contrib += delta * ws[k];
  }
  QT *q = reinterpret_cast<QT *>(a.q) + idx;
  bool whole = false;
  if constexpr (kN == kLaneSlots) {
    whole = act == 15u;
    if (whole) st_slots(q, qs);
  }
  if (!whole) {
#pragma unroll
    for (int k = 0; k < kN; ++k)
      if (act >> k & 1u) q[k] = qs[k];
  }
  contrib = warp_sum(contrib);  // fixed-order reduction of the slots
  if (lane == 0) atomicAdd(a.bcpart + (int64_t)v * a.W + w0, contrib);  // one writer a level: no wait for the old value
}

// Vertex blocks of a phase: each warp's first block is its own index, later
// ones come from the phase's work counter (no atomics at all when the level
// has no more blocks than the grid has warps).
__device__ __forceinline__ int64_t next_block(int *counter, int lane) {
  int b = 0;
  if (lane == 0) b = atomicAdd(counter, 1);
  return nwarps() + __shfl_sync(0xffffffffu, b, 0);
}

// A block's rows, one per lane, in 32 bits each: a row's place after the block's
// first, and its arcs (low half) and unit arcs (high half) when it is a light
// one. Blocks are consecutive vertices: neighbouring rows share cached mask
// rows, and with blocks handed out in order a level ends on the cheap late
// vertices of the BFS order (177.3 GTEPS on RMAT-20, against 172.0 with every
// block strided over the core).
struct RowLane {
  uint32_t at = 0, len = 0;
  static __device__ __forceinline__ RowLane load(const int64_t *HR, const int64_t *HS, int64_t v, int64_t rb,
                                                 int32_t heavy_deg) {
    const int64_t e0 = HR[v], e1 = HR[v + 1], sp = HS[v];
    return RowLane{(uint32_t)(e0 - rb), e1 - e0 <= heavy_deg ? (uint32_t)(e1 - e0) | (uint32_t)(sp - e0) << 16 : 0u};
  }
  __device__ __forceinline__ bool light() const { return len != 0; }
  // the first neighbours (unit arcs) of lane j's row, one a lane
  __device__ __forceinline__ uint32_t strip(const Args &a, int64_t rb, int j, int lane) const {
    const uint32_t at_j = __shfl_sync(0xffffffffu, at, j), len_j = __shfl_sync(0xffffffffu, len, j);
    return lane < (int)(len_j >> 16) ? (uint32_t)ldg(a.hcol + rb + at_j + lane) : 0u;
  }
};
static_assert(kHeavyDegMany < 1 << 16, "a light row's length takes 16 bits");

// Heavy-row chunk tasks of a phase: each CTA's first task is its own index;
// later ones in a fixed stride (BCGPU_BATCHED_HEAVY_DYN 0) or from the
// phase's work counter (1: a CTA that drew short chunks takes more; 153.0
// against 151.3-151.4 GTEPS on RMAT-20 at 512 sources per pass).
#ifndef BCGPU_BATCHED_HEAVY_DYN
#define BCGPU_BATCHED_HEAVY_DYN 1
#endif
__device__ __forceinline__ int64_t next_chunk_task(int64_t task, int *counter) {
#if BCGPU_BATCHED_HEAVY_DYN
  __shared__ int s_next;
  __syncthreads();  // every thread has read the previous s_next
  if (threadIdx.x == 0) s_next = atomicAdd(counter, 1);
  __syncthreads();
  return (int64_t)gridDim.x + s_next;
#else
  (void)counter;
  return task + gridDim.x;
#endif
}

}  // namespace

// --------------------------------------------------------------- kernel ----

template <typename QT>
__global__ void __launch_bounds__(kThreads, kMinCtas) batched_kernel(Args a) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  WarpScratch *scratch = reinterpret_cast<WarpScratch *>(s_raw);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  WarpScratch &S = scratch[wib];
  const int W = a.W;
  constexpr bool kComp = sizeof(QT) == 4;
  PHASE_INIT();

  int npass = 1;
  for (int64_t bi = a.b0; bi < a.b1; bi += npass) {
    if (cta_failed(a)) return;
    // the next passes of the same BCC as one: their slots, seeds and arming
    // lists follow each other, and all but a BCC's last pass are full
    Batch bt = a.batches[bi];
    for (npass = 1; npass < a.merge && bi + npass < a.b1; ++npass) {
      const Batch &nx = a.batches[bi + npass];
      if (nx.bcc != bt.bcc) break;
      bt.nslots += nx.nslots;
      bt.nseeds += nx.nseeds;
      bt.narm += nx.narm;
      bt.max_seed = max(bt.max_seed, nx.max_seed);
    }
    bt.words = (bt.nslots + 31) / 32;
    const Slot *slots = a.slots + bt.slot_off;
    const Seed *seeds = a.seeds + bt.seed_off;
    const int words = bt.words;
    const int groups = (words + 3) / 4;
    const int wpad = groups * 4;  // rows are processed in whole 4-word groups
    const int64_t vo = a.vtx_off[bt.bcc];
    const int32_t n = a.n_plain[bt.bcc];  // core vertices
    const int64_t *HR = a.hrow + a.hvo[bt.bcc];
    const int64_t *HS = a.hsplit + a.hvo[bt.bcc];
    const int32_t *rch = a.reach + vo;
    const int32_t *hv = a.heavy + a.heavy_off[bt.bcc];
    const int32_t nheavy = (int32_t)(a.heavy_off[bt.bcc + 1] - a.heavy_off[bt.bcc]);
    const int64_t hc0 = a.hchunk_off[bt.bcc];
    const int64_t nchunks = a.hchunk_off[bt.bcc + 1] - hc0;
    const int32_t *hcv = a.hchunk_v + hc0;
    const int64_t *hce0 = a.hchunk_e0 + hc0, *hce1 = a.hchunk_e1 + hc0;
    const int32_t *hfst = a.hfirst + a.heavy_off[bt.bcc] + bt.bcc;  // nheavy+1 entries per BCC
    const int64_t gthreads = (int64_t)gridDim.x * blockDim.x;
    const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    // Warp tasks of the light rows: (vertex block, kHalf-word quarter of the
    // row), so a row's quarters run on different warps. Blocks hold bs <= 32
    // vertices (lane l < bs takes vertex blk + l*nblk): whole 32-vertex blocks
    // on large cores, smaller ones on small cores so that every warp of the
    // grid gets work on a level.
    const int halves = wpad / kHalf;
    const int64_t bs_want = ((int64_t)n * halves + nwarps() * kTasksPerWarp - 1) / (nwarps() * kTasksPerWarp);
    const int bs = bs_want >= 32 ? 32 : bs_want < 1 ? 1 : (int)bs_want;
    const int64_t nblk = ((int64_t)n + bs - 1) / bs;
    const int64_t ntask = nblk * halves;

    // ---- init: seen = slots beyond the batch, partials, level-0/1 masks, X, rexp, work counters
    for (int64_t i = gtid; i < (int64_t)n * W; i += gthreads) {
      const int w = (int)(i % W);
      const int live = min(32, max(0, bt.nslots - 32 * w));
      a.seen[i] = live == 32 ? 0u : ~((1u << live) - 1u);
      a.bcpart[i] = 0.0;
      a.lm[i] = 0;                         // level 0
      a.lm[(int64_t)a.n_cap * W + i] = 0;  // level 1
      if (w == 0) { a.lmin[i / W] = INT_MAX; a.armed[i / W] = INT_MAX; }
    }
    for (int64_t i = gtid; i < (int64_t)W * 32; i += gthreads) {
      a.rexp[i] = INT_MIN;
      a.X[i * (a.tcap + 2)] = 0;
      a.wsrc[i] = i < bt.nslots ? (double)rch[slots[i].src] + 1.0 : 0.0;
      a.schain[i] = i < bt.nslots ? slots[i].chain : kNoSlot;
    }
    for (int64_t i = gtid; i < 4 * ((int64_t)a.tcap + 3) + 2; i += gthreads) a.wq[i] = 0;
    if (gtid == 0) {
      a.ctrl->more[0] = a.ctrl->more[1] = 0;
      a.ctrl->rescale[0] = a.ctrl->rescale[1] = 0;
      a.ctrl->range_err = 0;
      a.ctrl->found = 0;
    }
    grid_sync(a);
    for (int64_t b = gtid; b < bt.nslots; b += gthreads) {  // core sources at level 0
      const Slot s = slots[b];
      if (s.chain >= 0) continue;
      const int64_t idx = ((int64_t)s.src * W + (b >> 5)) * 32 + (b & 31);
      a.d[idx] = 0;
      a.sig[idx] = 1.0;
      atomicOr(a.lm + (int64_t)s.src * W + (b >> 5), 1u << (b & 31));
      atomicOr(a.seen + (int64_t)s.src * W + (b >> 5), 1u << (b & 31));
      atomicMin(a.lmin + s.src, 0);
      atomicAdd(&a.ctrl->found, 1ull);
    }
    for (int64_t i = gwarp(); i < bt.narm; i += nwarps()) {  // neighbours of sources and seeded vertices
      const int2 m = a.arms[bt.arm_off + i];
      arm_arcs(a, HR[m.x], HR[m.x + 1], m.y, lane, 32);
    }
    grid_sync(a);
    PHASE_MARK(0);

    // ---- forward: levels t -> t+1
    int t = 0, tlast = 0;
    // Some level so far was rescaled: else every X is 0, and none is read. A slot's
    // levels are next to each other in X, so that a warp's read of it takes 32
    // sectors, where the path counts take 8, and waits for the slot's level first:
    // chain in-flow on R-MAT 20, two passes of 512, 28 -> 22.9 ms without it.
    bool scaled = false;
    const unsigned long long all_found = (unsigned long long)n * (unsigned long long)bt.nslots;
    while (true) {
      unsigned int nf = 0;  // pairs this lane found on this level (fewer than 2^32: a lane's slots of a warp's rows)
      // Once a warp and phase: every warp writes the same words, and a store for
      // each row reached made that one address what the level waited for.
      auto report = [&](unsigned long long found) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) found += __shfl_xor_sync(0xffffffffu, found, o);
        if (lane != 0 || !found) return;
        atomicAdd(&a.ctrl->found, found);
        a.ctrl->more[t & 1] = 1;
      };
      if (t + 1 > a.tcap) { set_err(a.err, kDevWorkspace); break; }
      const uint32_t *lmt = a.lm + (int64_t)t * a.n_cap * W;
      // the next level's flags and masks start clear (nothing reads them on this level)
      if (gtid == 0) {
        a.ctrl->more[(t + 1) & 1] = 0;
        a.ctrl->rescale[(t + 1) & 1] = 0;
      }
      for (int64_t i = gtid; i < (int64_t)n * W; i += gthreads) a.lm[(int64_t)(t + 2) * a.n_cap * W + i] = 0;
      // heavy rows: chunks of their arcs, one CTA per (chunk, half); partials
      // are combined across the CTA's warps, then across chunks after the barrier
      for (int64_t task = blockIdx.x; task < nchunks * halves;
           task = next_chunk_task(task, a.wq + 2 * (a.tcap + 3) + t)) {
        const int64_t c = task / halves;
        const int w0 = (int)(task % halves) * kHalf;
        const int nw = min(kHalf, wpad - w0);
        const int32_t v = hv[hcv[c]];
        uint32_t unseen[kHalf], got = 0;
        load_row(a.seen + (int64_t)v * W + w0, nw, unseen);
        uint32_t u_any = 0;
#pragma unroll
        for (int k = 0; k < kHalf; ++k) { unseen[k] = k < nw ? ~unseen[k] : 0u; u_any |= unseen[k]; }
        Acc<false> acc[kLaneSlots];
        if (u_any && __ldcg(a.armed + v) <= t + 1) {  // uniform over the CTA
          const int64_t e0 = hce0[c], e1 = hce1[c], sp = HS[v];
          const int64_t per = (e1 - e0 + kWarpsPerCta - 1) / kWarpsPerCta;
          const int64_t s0 = e0 + wib * per, s1 = min(e1, s0 + per);
          if (s0 < min(s1, sp)) row_pass<double, false, 0>(a, S, lmt, a.sig, s0, min(s1, sp), w0, nw, unseen, got, acc, lane, t, scaled);
          if (max(s0, sp) < s1) row_pass<double, false, 1>(a, S, a.lm, a.sig, max(s0, sp), s1, w0, nw, unseen, got, acc, lane, t, scaled);
        }
#pragma unroll
        for (int k = 0; k < kLaneSlots; ++k) S.acc[kLaneSlots * lane + k] = acc[k].value();
        got = word_of(got, lane);
        if (lane_bit(lane) == 0) S.any[lane_word(lane)] = got;  // this warp's hit masks, for the combine
        __syncthreads();
        for (int k = wib; k < nw; k += kWarpsPerCta) {  // fixed warp order
          double tot = 0.0;
          uint32_t mm = 0;
          for (int x = 0; x < kWarpsPerCta; ++x) { tot += scratch[x].acc[k * 32 + lane]; mm |= scratch[x].any[k]; }
          a.hacc[((hc0 + c) * W + w0 + k) * 32 + lane] = tot;
          if (lane == 0) a.hmask[(hc0 + c) * W + w0 + k] = mm;
        }
        __syncthreads();
      }
      // light rows: (vertex block, quarter) tasks. Lane l holds vertex l's row and
      // unseen slots; the next active row's first neighbours are loaded while
      // this one's counts are gathered. Bound by the latency of a row's chain of
      // loads (neighbours, their masks, counts), 32 warps an SM in flight, and by
      // instructions issued. Two passes of 512 on R-MAT 20, forward / backward rows:
      // 51.1 / 69.2 ms with a word's slot a lane, that is four loads, five shuffles
      // and four masks a hit; 41.4 / 58.9 ms with four slots a lane.
      for (int64_t tk = gwarp(); tk < ntask; tk = next_block(a.wq + t, lane)) {
        const int64_t v0 = tk / halves * bs;
        const int w0 = (int)(tk % halves) * kHalf;
        const int64_t vl = v0 + lane;
        RowLane row{};
        uint4 un = make_uint4(0, 0, 0, 0);
        int32_t lmin = 0;
        const int64_t rb = HR[v0];
        if (lane < bs && vl < n) {
          const uint4 seen = ld4(a.seen + vl * W + w0);
          const int32_t armed = __ldcg(a.armed + vl);
          lmin = __ldcg(a.lmin + vl);
          row = RowLane::load(HR, HS, vl, rb, bt.heavy_deg);
          if (armed <= t + 1 && row.light()) un = make_uint4(~seen.x, ~seen.y, ~seen.z, ~seen.w);
        }
        uint32_t todo = __ballot_sync(0xffffffffu, (un.x | un.y | un.z | un.w) != 0u);
        uint32_t ahead = todo ? row.strip(a, rb, __ffs(todo) - 1, lane) : 0u;
        while (todo) {
          const int j = __ffs(todo) - 1;
          todo &= todo - 1;
          const uint32_t u = ahead;
          if (todo) ahead = row.strip(a, rb, __ffs(todo) - 1, lane);
          const int32_t v = (int32_t)v0 + j;
          const int64_t e0 = rb + __shfl_sync(0xffffffffu, row.at, j);
          const uint32_t len = __shfl_sync(0xffffffffu, row.len, j);
          const int units = (int)(len >> 16), arcs = (int)(len & 0xffff);
          const uint32_t unseen[kHalf] = {__shfl_sync(0xffffffffu, un.x, j), __shfl_sync(0xffffffffu, un.y, j),
                                          __shfl_sync(0xffffffffu, un.z, j), __shfl_sync(0xffffffffu, un.w, j)};
          uint32_t f[kHalf], got = 0;
          load_row(lmt + (int64_t)u * W + w0, lane < units ? kHalf : 0, f);
#pragma unroll
          for (int k = 0; k < kHalf; ++k) f[k] &= unseen[k];
          Acc<false> acc[kLaneSlots];
          walk_hits<double, false, 0>(a, S, a.sig + (int64_t)w0 * 32 + kLaneSlots * lane, u, 0, f, got, acc, lane);
          if (units > 32)
            row_pass<double, false, 0>(a, S, lmt, a.sig, e0 + 32, e0 + units, w0, kHalf, unseen, got, acc, lane, t);
          if (units < arcs)
            row_pass<double, false, 1>(a, S, a.lm, a.sig, e0 + units, e0 + arcs, w0, kHalf, unseen, got, acc, lane, t, scaled);
          if (!__ballot_sync(0xffffffffu, got != 0u)) continue;
          nf += __popc(got);
          const double sum[kLaneSlots] = {acc[0].value(), acc[1].value(), acc[2].value(), acc[3].value()};
          put_counts<kLaneSlots>(a, v, w0 * 32 + kLaneSlots * lane, t, got, sum);
          got = word_of(got, lane);
          if (lane_bit(lane) == 0) {  // a lane for each word
            const int k = lane_word(lane);
            a.lm[((int64_t)(t + 1) * a.n_cap + v) * W + w0 + k] = got;
            a.seen[(int64_t)v * W + w0 + k] = ~(k == 0 ? unseen[0] : k == 1 ? unseen[1] : k == 2 ? unseen[2] : unseen[3]) | got;
          }
          int first = 0;
          const bool fresh = __shfl_sync(0xffffffffu, lmin, j) == INT_MAX;  // not reached on an earlier level
          if (lane == 0 && fresh) first = atomicMin(a.lmin + v, t + 1) == INT_MAX;
          if (fresh && __shfl_sync(0xffffffffu, first, 0)) arm_arcs(a, e0, e0 + arcs, t + 1, lane, 32);
        }
      }
      report(nf);
      nf = 0;
      grid_sync(a);
      PHASE_MARK(1);
      PHASE_COUNT(16);
      if (nheavy) {
        for (int64_t task = gwarp(); task < (int64_t)nheavy * wpad; task += nwarps()) {
          const int32_t h = (int32_t)(task / wpad);
          const int w = (int)(task % wpad);
          const int32_t v = hv[h];
          if (!~__ldcg(a.seen + (int64_t)v * W + w)) continue;
          double acc = 0.0;
          uint32_t m = 0;
          for (int32_t c = hfst[h]; c < hfst[h + 1]; ++c) {
            acc += __ldcg(a.hacc + ((hc0 + c) * W + w) * 32 + lane);
            m |= __ldcg(a.hmask + (hc0 + c) * W + w);
          }
          nf += finish_pull(a, v, w, t, m, lane, acc);  // heavy rows arm in the next phase
        }
        report(nf);
        grid_sync(a);
        PHASE_MARK(2);
      }
      if (bt.nseeds) {  // chain sources entering the core at level t+1 (one path each)
        for (int64_t i = gtid; i < bt.nseeds; i += gthreads) {
          const Seed s = seeds[i];
          if (s.level != t + 1) continue;
          const int b = s.slot + (int)(s.pass - bi) * a.width, w = b >> 5;
          const uint32_t bit = 1u << (b & 31);
          const int64_t idx = ((int64_t)s.v * W + w) * 32 + (b & 31);
          const double one = scale2(1.0, -a.X[(int64_t)b * (a.tcap + 2) + t]);
          const uint32_t old = atomicOr(a.seen + (int64_t)s.v * W + w, bit);
          if (!(old & bit)) {
            a.d[idx] = t + 1;
            a.sig[idx] = one;
            atomicOr(a.lm + ((int64_t)(t + 1) * a.n_cap + s.v) * W + w, bit);
            atomicMin(a.lmin + s.v, t + 1);
            a.ctrl->more[t & 1] = 1;
            atomicAdd(&a.ctrl->found, 1ull);
          } else if (a.d[idx] == t + 1) {
            a.sig[idx] += one;  // reached on this level from the core as well
          }
        }
        grid_sync(a);
      }
      const int more = *(volatile int *)&a.ctrl->more[t & 1];
      const int resc = *(volatile int *)&a.ctrl->rescale[t & 1];
      const unsigned long long found = *(volatile unsigned long long *)&a.ctrl->found;
      // heavy rows first reached on level t+1 arm their neighbours, one CTA per chunk
      for (int64_t c = blockIdx.x; c < nchunks; c += gridDim.x)
        if (__ldcg(a.lmin + hv[hcv[c]]) == t + 1) arm_arcs(a, hce0[c], hce1[c], t + 1, threadIdx.x, blockDim.x);
      // base exponent of level t+1; rescale it when some slot's counts passed 2^rescale_exp
      for (int64_t b = gtid; b < (int64_t)W * 32; b += gthreads) {
        const int re = __ldcg(a.rexp + b);
        a.X[b * (a.tcap + 2) + t + 1] = a.X[b * (a.tcap + 2) + t] + (re > a.rescale_exp ? re : 0);
      }
      if (resc) {
        for (int64_t task = gwarp(); task < (int64_t)n * words; task += nwarps()) {
          const int32_t v = (int32_t)(task / words);
          const int w = (int)(task % words);
          const uint32_t m = __ldcg(a.lm + ((int64_t)(t + 1) * a.n_cap + v) * W + w);
          const int re = __ldcg(a.rexp + w * 32 + lane);
          if (((m >> lane) & 1u) && re > a.rescale_exp) {
            const int64_t idx = ((int64_t)v * W + w) * 32 + lane;
            a.sig[idx] = scale2(a.sig[idx], -re);
          }
        }
      }
      grid_sync(a);  // level t+1's base and counts are final; everyone has read the flags
      if (resc) {
        for (int64_t b = gtid; b < (int64_t)W * 32; b += gthreads) a.rexp[b] = INT_MIN;
        grid_sync(a);
      }
      if (more) tlast = t + 1;
      scaled = scaled || resc;
      if (cta_failed(a)) break;
      // done when every slot has reached every core vertex (later seeds then
      // reach seen vertices only); else level t+2 needs a non-empty level
      // within the longest arc, or a seed
      if (found >= all_found) break;
      if (t + 1 - tlast > bt.kmax && t + 2 > bt.max_seed) break;
      ++t;
      PHASE_MARK(3);
    }
    PHASE_MARK(3);
    if (cta_failed(a)) return;
    // every slot must have reached every core vertex of the BCC
    for (int64_t i = gtid; i < (int64_t)n * words; i += gthreads) {
      const int32_t v = (int32_t)(i / words);
      const int w = (int)(i % words);
      if (~__ldcg(a.seen + (int64_t)v * W + w) != 0u) set_err(a.err, kDevDisconnected);
    }
    // what the core vertices receive from their chains' vertices
    if (bt.kmax) {
      const int parts = (words + kInSlots - 1) / kInSlots;
      for (int64_t task = gwarp(); task < (int64_t)n * parts; task = next_block(a.wq + 4 * (a.tcap + 3), lane)) {
        const int32_t v = (int32_t)(task / parts);
        const int64_t c0 = HS[v], c1 = HR[v + 1];
        if (c0 < c1) chain_in(a, slots, v, ((int)(task % parts) * 32 + lane) * kInSlots, c0, c1, lane, scaled);
      }
      grid_sync(a);
    }
    PHASE_MARK(4);

    // ---- backward: lev = tlast .. 1 (level tlast+1 is empty and not cleared:
    // the deepest level has no unit-arc successors)
    for (int lev = tlast; lev >= 1; --lev) {
      const uint32_t *lm_here = a.lm + (int64_t)lev * a.n_cap * W;
      const uint32_t *lm_next = a.lm + (int64_t)(lev + 1) * a.n_cap * W;
      const QT *q = reinterpret_cast<const QT *>(a.q);
      // heavy rows: chunked successor sums, combined below
      for (int64_t task = blockIdx.x; task < nchunks * halves;
           task = next_chunk_task(task, a.wq + 3 * (a.tcap + 3) + lev)) {
        const int64_t c = task / halves;
        const int w0 = (int)(task % halves) * kHalf;
        const int nw = min(kHalf, wpad - w0);
        const int32_t v = hv[hcv[c]];
        uint32_t act[kHalf], got = 0;
        load_row(lm_here + (int64_t)v * W + w0, nw, act);
        uint32_t a_any = 0;
#pragma unroll
        for (int k = 0; k < kHalf; ++k) {
          act[k] = k < nw ? act[k] : 0u;
          a_any |= act[k];
        }
        Acc<kComp> acc[kLaneSlots];
        if (a_any) {  // uniform over the CTA
          const int64_t e0 = hce0[c], e1 = hce1[c], sp = HS[v];
          const int64_t per = (e1 - e0 + kWarpsPerCta - 1) / kWarpsPerCta;
          const int64_t s0 = e0 + wib * per, s1 = min(e1, s0 + per);
          if (lev < tlast && s0 < min(s1, sp))
            row_pass<QT, kComp, 0>(a, S, lm_next, q, s0, min(s1, sp), w0, nw, act, got, acc, lane, lev + 1, scaled);
          if (max(s0, sp) < s1) row_pass<QT, kComp, 2>(a, S, a.lm, q, max(s0, sp), s1, w0, nw, act, got, acc, lane, lev + 1, scaled, tlast);
        }
#pragma unroll
        for (int k = 0; k < kLaneSlots; ++k) S.acc[kLaneSlots * lane + k] = acc[k].value();
        __syncthreads();
        for (int k = wib; k < nw; k += kWarpsPerCta) {  // fixed warp order
          double tot = 0.0;
          for (int x = 0; x < kWarpsPerCta; ++x) tot += scratch[x].acc[k * 32 + lane];
          a.hacc[((hc0 + c) * W + w0 + k) * 32 + lane] = tot;
        }
        __syncthreads();
      }
      const int wqi = a.tcap + 3 + lev;
      for (int64_t tk = gwarp(); tk < ntask; tk = next_block(a.wq + wqi, lane)) {
        const int64_t v0 = tk / halves * bs;
        const int w0 = (int)(tk % halves) * kHalf;
        const int64_t vl = v0 + lane;
        RowLane row{};
        uint4 on = make_uint4(0, 0, 0, 0);  // the vertex's slots on this level
        int32_t reach = 0;
        const int64_t rb = HR[v0];
        if (lane < bs && vl < n) {
          on = ld4(lm_here + vl * W + w0);
          row = RowLane::load(HR, HS, vl, rb, bt.heavy_deg);
          reach = rch[vl];
          if (!row.light()) on = make_uint4(0, 0, 0, 0);
        }
        uint32_t todo = __ballot_sync(0xffffffffu, (on.x | on.y | on.z | on.w) != 0u);
        uint32_t ahead = todo ? row.strip(a, rb, __ffs(todo) - 1, lane) : 0u;
        while (todo) {
          const int j = __ffs(todo) - 1;
          todo &= todo - 1;
          const uint32_t u = ahead;
          if (todo) ahead = row.strip(a, rb, __ffs(todo) - 1, lane);
          const int32_t v = (int32_t)v0 + j;
          const int64_t e0 = rb + __shfl_sync(0xffffffffu, row.at, j);
          const uint32_t len = __shfl_sync(0xffffffffu, row.len, j);
          const int units = (int)(len >> 16), arcs = (int)(len & 0xffff);
          const uint32_t act[kHalf] = {__shfl_sync(0xffffffffu, on.x, j), __shfl_sync(0xffffffffu, on.y, j),
                                       __shfl_sync(0xffffffffu, on.z, j), __shfl_sync(0xffffffffu, on.w, j)};
          Acc<kComp> acc[kLaneSlots];
          uint32_t got = 0;
          if (lev < tlast) {
            uint32_t f[kHalf];
            load_row(lm_next + (int64_t)u * W + w0, lane < units ? kHalf : 0, f);
#pragma unroll
            for (int k = 0; k < kHalf; ++k) f[k] &= act[k];
            walk_hits<QT, kComp, 0>(a, S, q + (int64_t)w0 * 32 + kLaneSlots * lane, u, 0, f, got, acc, lane);
            if (units > 32)
              row_pass<QT, kComp, 0>(a, S, lm_next, q, e0 + 32, e0 + units, w0, kHalf, act, got, acc, lane, lev + 1);
          }
          if (units < arcs)
            row_pass<QT, kComp, 2>(a, S, a.lm, q, e0 + units, e0 + arcs, w0, kHalf, act, got, acc, lane, lev + 1, scaled, tlast);
          const double sum[kLaneSlots] = {acc[0].value(), acc[1].value(), acc[2].value(), acc[3].value()};
          const int k = lane_word(lane);
          const uint32_t own = (k == 0 ? act[0] : k == 1 ? act[1] : k == 2 ? act[2] : act[3]) >> lane_bit(lane) & 15u;
          finish_dep<QT, kLaneSlots>(a, __shfl_sync(0xffffffffu, reach, j), v, w0, w0 * 32 + kLaneSlots * lane, lev, own, lane,
                                     sum, units < arcs, scaled);
        }
      }
      if (nheavy) {
        grid_sync(a);
        PHASE_MARK(5);
        for (int64_t task = gwarp(); task < (int64_t)nheavy * wpad; task += nwarps()) {
          const int32_t h = (int32_t)(task / wpad);
          const int w = (int)(task % wpad);
          const int32_t v = hv[h];
          const uint32_t act = __ldcg(lm_here + (int64_t)v * W + w);
          if (!act) continue;
          double sum = 0.0;
          for (int32_t c = hfst[h]; c < hfst[h + 1]; ++c) sum += __ldcg(a.hacc + ((hc0 + c) * W + w) * 32 + lane);
          finish_dep<QT, 1>(a, rch[v], v, w, w * 32 + lane, lev, act >> lane & 1u, lane, {sum}, HS[v] < HR[v + 1], scaled);
        }
      }
      grid_sync(a);
      PHASE_MARK(6);
      PHASE_COUNT(17);
    }

    // ---- chain vertices: one warp per chain, every slot, two neighbouring ones a
    // lane; each lane sums its slots' contributions (registers for chains of up to
    // kRegVerts vertices), then one warp reduction per chain vertex goes straight
    // into BC (one writer per vertex: fixed order). Bound by the instructions of
    // the closed form: two passes of 512 on R-MAT 20 took 28.3 ms with a slot a lane
    // and two divisions for each side of a tie, 16.5 so.
    if (bt.kmax) {
      constexpr int kRegVerts = 8;
      const int bad = *(volatile int *)&a.ctrl->range_err;
      const int64_t ch0 = a.chain_off[bt.bcc];
      const int64_t nch = a.chain_off[bt.bcc + 1] - ch0;
      const QT *qq = reinterpret_cast<const QT *>(a.q);
      for (int64_t task = gwarp(); task < nch; task = next_block(a.wq + 4 * (a.tcap + 3) + 1, lane)) {
        const int64_t c = ch0 + task;
        const int32_t L = a.chain_l[c], R = a.chain_r[c], cs = a.chain_start[c], k = a.chain_len[c];
        const int64_t poff = a.cpre_off[c];
        const double *P = poff < 0 ? nullptr : a.cpre + poff;
        double part[kRegVerts];
#pragma unroll
        for (int j = 0; j < kRegVerts; ++j) part[j] = 0.0;
        for (int b = 2 * lane; b < wpad * 32; b += 64) {
          const int64_t iL = (int64_t)L * W * 32 + b, iR = (int64_t)R * W * 32 + b;
          // the ends' levels, then only the path counts / q the closed forms use
          const int2 dL2 = __ldcg(reinterpret_cast<const int2 *>(a.d + iL)), dR2 = __ldcg(reinterpret_cast<const int2 *>(a.d + iR));
          const int2 on2 = __ldcg(reinterpret_cast<const int2 *>(a.schain + b));
          const double2 ws2 = __ldcg(reinterpret_cast<const double2 *>(a.wsrc + b));
          const int32_t dL[2] = {dL2.x, dL2.y}, dR[2] = {dR2.x, dR2.y}, on[2] = {on2.x, on2.y};
          const double ws[2] = {ws2.x, ws2.y};
          bool tie[2], sig = false, via = false;
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int D = dR[r] + k - dL[r] - 1;
            tie[r] = D >= 0 && !(D & 1) && D < 2 * k;
            const bool far = D > 2 * k - 1 || D < -1;  // |level difference| = k + 1: one end's paths come over the chain
            sig |= tie[r] || far;
            via |= far;
          }
          double2 sL2 = make_double2(1.0, 1.0), sR2 = sL2;
          QT qL[2] = {}, qR[2] = {};
          if (sig) {
            sL2 = __ldcg(reinterpret_cast<const double2 *>(a.sig + iL));
            sR2 = __ldcg(reinterpret_cast<const double2 *>(a.sig + iR));
          }
          if (via) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              qL[r] = __ldcg(qq + iL + r);
              qR[r] = __ldcg(qq + iR + r);
            }
          }
          const double sL[2] = {sL2.x, sL2.y}, sR[2] = {sR2.x, sR2.y};
          bool own = false;  // a slot's source sits on the chain
          int lo[2], hi[2];
          double fL[2], fR[2];  // L-side and R-side constants
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            own |= on[r] == c;
            lo[r] = 0;
            hi[r] = k;  // nothing from this slot
            fL[r] = fR[r] = 0.0;
            if (on[r] == kNoSlot || on[r] == c) continue;
            // in prefix sums from L: vertex j is fed from L iff 2j <= D; a tie
            // vertex t = D/2 shares its reach+1 between the sides in proportion to
            // sigma_L, sigma_R; else the L-fed vertices end at D/2, and the far
            // end's q enters when the chain carries its shortest paths.
            const int D = dR[r] + k - dL[r] - 1;
            lo[r] = D < 0 ? 0 : min(k, (D >> 1) + (tie[r] ? 0 : 1));  // vertices [0, lo) are fed from L
            hi[r] = tie[r] ? lo[r] + 1 : lo[r];                       // [hi, k) from R
            const int x = scaled ? level_base(a, b + r, dL[r]) - level_base(a, b + r, dR[r]) : 0;
            const double p0 = chain_pre(P, lo[r]), p1 = chain_pre(P, hi[r]);
            fL[r] = p0;
            fR[r] = -p1;
            if (tie[r]) {
              fL[r] += scaled ? (p1 - p0) / (1.0 + scale2(sR[r] / sL[r], -x)) : (p1 - p0) * path_share(sL[r], sR[r]);
              fR[r] += scaled ? (p1 - p0) / (1.0 + scale2(sL[r] / sR[r], x)) : (p1 - p0) * path_share(sR[r], sL[r]);
            } else if (D >= 2 * k) {
              fL[r] += scale2(sL[r] * (double)qR[r], x);
            } else if (D <= -2) {
              fR[r] += scale2(sR[r] * (double)qL[r], -x);
            }
          }
          auto dep = [&](int r, int j) {
            const double y = j < lo[r] ? fL[r] - chain_pre(P, j + 1) : chain_pre(P, j) + fR[r];
            return j >= lo[r] && j < hi[r] ? 0.0 : y * ws[r];
          };
          auto add = [&](int j, double x) {
            const double tot = warp_sum(x);
            if (lane == 0 && !bad) a.bc[vo + cs + j] += tot;
          };
          if (k <= kRegVerts) {
#pragma unroll
            for (int j = 0; j < kRegVerts; ++j)
              if (j < k) part[j] += dep(0, j) + dep(1, j);
          } else {
            for (int j = 0; j < k; ++j) add(j, dep(0, j) + dep(1, j));
          }
          if (__any_sync(0xffffffffu, own)) {  // rare: [L, source] and [source, R]
            for (int r = 0; r < 2; ++r) {
              const bool mine = (r ? on2.y : on2.x) == c;
              const double wr = r ? ws2.y : ws2.x;
              int pos = 0;
              End eL{0, 0, 1.0, 0.0}, eR{0, 0, 1.0, 0.0};
              if (mine) {
                pos = slots[b + r].pos;
                eL.d = r ? dL2.y : dL2.x;
                eR.d = r ? dR2.y : dR2.x;
                eL.s = __ldcg(a.sig + iL + r);
                eR.s = __ldcg(a.sig + iR + r);
                if (eL.d == pos + 1) eL.qs = (double)__ldcg(qq + iL + r);  // fed from the source
                if (eR.d == k - pos) eR.qs = (double)__ldcg(qq + iR + r);
                eL.x = scaled ? level_base(a, b + r, eL.d) : 0;
                eR.x = scaled ? level_base(a, b + r, eR.d) : 0;
              }
              for (int j = 0; j < k; ++j) {
                double x = 0.0;
                if (mine && j < pos) x = stretch_dep(Stretch{P, 0, pos, false}, j, eL, source_end()) * wr;
                if (mine && j > pos) x = stretch_dep(Stretch{P, pos + 1, k, false}, j - pos - 1, source_end(), eR) * wr;
                add(j, x);
              }
            }
          }
        }
        if (k <= kRegVerts) {
#pragma unroll
          for (int j = 0; j < kRegVerts; ++j) {
            if (j >= k) continue;
            const double tot = warp_sum(part[j]);
            if (lane == 0 && !bad) a.bc[vo + cs + j] += tot;
          }
        }
      }
    }
    grid_sync(a);
    PHASE_MARK(8);

    // ---- fold the batch into BC (fixed word order), unless FP32 range failed
    const int bad = *(volatile int *)&a.ctrl->range_err;
    if (bad) {
      if (gtid < npass) a.redo[bi + gtid] = 1;
    } else {
      for (int64_t v = gtid; v < n; v += gthreads) {  // core vertices (chain vertices were added above)
        double s = 0.0;
        for (int w = 0; w < words; ++w) s += a.bcpart[v * W + w];
        a.bc[vo + v] += s;
      }
    }
    grid_sync(a);
    PHASE_MARK(7);
  }
}

// ================================================================= host ====

// An allocator whose value-initialising construct leaves trivially
// constructible elements uninitialised: table vectors that are resized and
// then fully overwritten by parallel loops skip a sequential zero fill (and
// their pages are first touched by the parallel writers).
template <class T>
struct NoInit : std::allocator<T> {
  template <class U>
  struct rebind {
    using other = NoInit<U>;
  };
  NoInit() = default;
  template <class U>
  NoInit(const NoInit<U> &) {}
  template <class U>
  void construct(U *p) noexcept {
    ::new ((void *)p) U;
  }
  template <class U, class... A>
  void construct(U *p, A &&...a) {
    ::new ((void *)p) U(std::forward<A>(a)...);
  }
};
template <class T>
using HostBuf = std::vector<T, NoInit<T>>;

struct BatchedPlan {
  int width = 0;       // B
  int W = 0;           // words
  int merge = 1;       // passes run as one, at most
  int tcap = 0;
  int64_t n_cap = 0;
  bool f32 = true;
  int grid = 0;
  size_t smem = 0;
  int64_t bytes = 0;
  int64_t h2d = 0;  // bytes uploaded by batched_create
  int64_t d2h = 0;  // bytes batched_create read back (the row checks' flag)
  cudaMemPool_t pool = nullptr;  // allocs come from this pool on `stream` (null: cudaMalloc)
  cudaStream_t stream = nullptr;
  std::vector<void *> allocs;
  Args args{};
  std::vector<int64_t> u_src, u_teps, u_bfs, u_aux, u_visits;
  std::vector<Batch> h_batches;
  HostBuf<Slot> h_slots;
  HostBuf<Seed> h_seeds;
  std::vector<int2> h_arms;
  std::vector<int64_t> h_vtx_off;
  int64_t n_batches = 0;
};

namespace {

// Eccentricity of local vertex 0 in the BCC: every level of every source is
// at most 2 * ecc.
int bcc_ecc(const int64_t *row, const int32_t *col, int64_t vo, int32_t nb, std::vector<int32_t> &dist,
            std::vector<int32_t> &queue) {
  dist.assign((size_t)nb, -1);
  queue.resize((size_t)nb);
  int head = 0, tail = 0;
  queue[tail++] = 0;
  dist[0] = 0;
  int ecc = 0;
  while (head < tail) {
    const int32_t x = queue[head++];
    ecc = std::max(ecc, dist[x]);
    for (int64_t e = row[vo + x]; e < row[vo + x + 1]; ++e) {
      const int32_t y = col[e];
      if (dist[y] < 0) { dist[y] = dist[x] + 1; queue[tail++] = y; }
    }
  }
  return ecc;
}

}  // namespace

int batched_width(int requested) {
  const int width = requested > 0 ? requested : 512;
  return std::max(32, std::min(1024, (width + 31) / 32 * 32));
}

namespace {

// Passes of `width` slots run as one on a core of n vertices: a level of a pass
// costs its slowest row whatever else there is to do, so a small core gets more
// slots per level, up to 80 million (vertex, slot) pairs (2.2 GB of workspace);
// beyond that the grid is full either way. R-MAT 14 (9,107 core vertices, 16
// passes of 512): 54.9 ms one by one, 40.0 / 33.8 / 31.3 by 2 / 4 / 8; R-MAT 16
// (32,842, 8 passes of 256, FP64) 83.0, 64.0 / 55.7 / 50.2; R-MAT 18 (121,000, 4
// of 512) 115.5, 110.6 / 111.0 by 2 / 4.
constexpr int64_t kMergePairs = 80 * 1000 * 1000;
int merge_passes(int64_t n, int width) { return (int)std::max<int64_t>(1, kMergePairs / (n * width)); }

}  // namespace

// Source order of BCC b: bounded BFS balls of nearby vertices (chain vertices
// included), so a pass's sources see every vertex within a narrow band of
// levels: few active levels per vertex, dense 32-slot hits. A ball grows only
// through vertices not yet taken, so each vertex's arcs are scanned once and
// late balls cost no rescans of finished regions. The greedy stops at the
// first ball boundary at or after `need` vertices: the order of a larger
// `need` extends it (a lazy plan that fills only some passes needs a prefix).
void batched_source_order(const bc_bccs *B, int32_t b, int width, int64_t need, std::vector<int32_t> &order) {
  const int64_t vo = B->vtx_off[b];
  const int32_t nb = (int32_t)(B->vtx_off[b + 1] - vo);
  order.clear();
  need = std::min<int64_t>(need, nb);
  if (need <= 0) return;
  order.reserve((size_t)need + (size_t)width);
  // taken: one bit per vertex (small enough to stay in the host's caches).
  // A ball's queue may list a vertex more than once (every taken vertex
  // queues its untaken neighbours); it is taken at its first listing and
  // skipped at the later ones, so the order is that of a queue holding each
  // vertex once. A vertex queued by an earlier ball but not taken may join
  // a later one.
  std::vector<uint64_t> taken(((size_t)nb + 63) / 64, 0);
  auto is_taken = [&](int32_t y) { return (taken[(size_t)y >> 6] >> (y & 63)) & 1u; };
  std::vector<int32_t> q;
  const int64_t arc_budget = 16 * (int64_t)width;  // bounds the host work per ball
  for (int32_t seed = 0; seed < nb && (int64_t)order.size() < need; ++seed) {
    if (is_taken(seed)) continue;
    q.clear();
    q.push_back(seed);
    int64_t got = 0, scanned = 0;
    for (size_t h = 0; h < q.size() && got < width; ++h) {
      // software pipeline over the queue: row offsets 16 entries ahead, the
      // row's arcs 8 ahead (rows are short: ~9 arcs on RMAT)
      if (h + 16 < q.size()) __builtin_prefetch(&B->row[vo + q[h + 16]]);
      if (h + 8 < q.size()) __builtin_prefetch(&B->col[B->row[vo + q[h + 8]]]);
      const int32_t x = q[h];
      if (is_taken(x)) continue;
      taken[(size_t)x >> 6] |= 1ull << (x & 63);
      order.push_back(x);
      ++got;
      if (scanned >= arc_budget) continue;  // keep draining the queue, stop growing it
      const int64_t e0 = B->row[vo + x], e1 = std::min(B->row[vo + x + 1], e0 + arc_budget - scanned);
      scanned += e1 - e0;
      for (int64_t e = e0; e < e1; ++e) {
        const int32_t y = B->col[e];
        if (!is_taken(y)) q.push_back(y);
      }
    }
  }
}

namespace {

// The contracted rows of the core vertices of the BCCs in multi-source
// passes, built on the device from the packed CSR already there (the host
// computes only the row offsets hrow and, per packed chain vertex, its chain
// and position): one warp per row writes the row's unit arcs, then its chain
// arcs, each in the order of the vertex's CSR row -- so the rows are those a
// sequential fill gives. Entries of rbcc < 0 are a BCC's end offsets. A
// non-core neighbour outside every chain sets bit 1 of *bad, a core vertex
// next to the inside of a chain bit 2. Bound by the rows' traffic (16 bytes an
// arc): a lane an arc keeps a hub's row -- 9,700 arcs on the R-MAT 16 graph --
// from being one thread's serial chain (a thread a row: 3.7 ms there; the fill with
// the uploads around it 4.65 -> 0.96 ms).
__global__ void contract_rows_kernel(const int64_t *row, const int32_t *col, const int64_t *vtx_off,
                                     const int32_t *n_plain, const int32_t *rbcc, const int64_t *hvo,
                                     const int64_t *hrow, int64_t nrows, const int32_t *gcof, const int32_t *gcpos,
                                     const int32_t *chain_len, const int32_t *chain_l, const int32_t *chain_r,
                                     int64_t *hsplit, int32_t *hcol, int32_t *hk, int32_t *hcid, int *bad) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; i < nrows; i += warps) {
    const int32_t b = rbcc[i];
    if (b < 0) {
      if (lane == 0) hsplit[i] = hrow[i];
      continue;
    }
    const int64_t vo = vtx_off[b];
    const int32_t npl = n_plain[b], x = (int32_t)(i - hvo[b]);
    const int64_t e0 = row[vo + x], e1 = row[vo + x + 1];
    int64_t o = hrow[i];
    for (int64_t e = e0; e < e1; e += 32) {
      const int32_t y = e + lane < e1 ? col[e + lane] : npl;
      const unsigned unit = __ballot_sync(0xffffffffu, y < npl);
      if (y < npl) {
        const int64_t at = o + __popc(unit & below);
        hcol[at] = y;
        hk[at] = 0;
        hcid[at] = -1;
      }
      o += __popc(unit);
    }
    if (lane == 0) hsplit[i] = o;
    for (int64_t e = e0; e < e1; e += 32) {
      const int32_t y = e + lane < e1 ? col[e + lane] : 0;
      int32_t c = -1, k = 0;
      int right = 0;
      if (e + lane < e1 && y >= npl) {
        c = gcof[vo + y];
        if (c < 0) {
          atomicOr(bad, 1);
        } else {
          const int32_t pos = gcpos[vo + y];
          k = chain_len[c];
          if (x == chain_l[c] && pos == 0) right = 0;
          else if (x == chain_r[c] && pos == k - 1) right = 1;
          else {
            atomicOr(bad, 2);
            c = -1;
          }
        }
      }
      const unsigned arm = __ballot_sync(0xffffffffu, c >= 0);
      if (c >= 0) {
        const int64_t at = o + __popc(arm & below);
        hcol[at] = right ? chain_l[c] : chain_r[c];
        hk[at] = k;
        hcid[at] = c * 2 + right;
      }
      o += __popc(arm);
    }
  }
}

// Fills P (allocated by batched_create, which releases it on any failure).
int batched_build(const bc_bccs *B, const BatchedConfig &cfg, const int64_t *row, const int32_t *col,
                  const int32_t *reach, const int64_t *vtx_off, const int32_t *chain_start, const int32_t *chain_len,
                  const int32_t *chain_l, const int32_t *chain_r, double *bc, int *err, cudaStream_t stream,
                  BatchedPlan *P, std::string *msg) {
  auto bail = [&](int code, const std::string &m) {
    if (msg) *msg = m;
    return code;
  };
  P->f32 = cfg.delta_fp32c;
  const int width = batched_width(cfg.width);
  P->width = width;
  P->W = (width / 32 + 3) / 4 * 4;  // row stride: whole 4-word groups (16-byte mask loads)
  const int W = P->W;

  // ---- contracted rows, chain prefix sums, heavy chunks, passes
  std::vector<int64_t> hvo, hrow, cpre_off;
  std::vector<int32_t> rbcc;          // per hrow entry: its BCC, -1 for a BCC's end offset
  HostBuf<int32_t> gcof, gcpos;       // per packed vertex of a BCC in passes: chain (global, -1: core), position
  int64_t narcs = 0;                  // contracted arcs so far
  std::vector<double> cpre;
  HostBuf<Slot> slots;  // every entry written by the pass fill
  HostBuf<Seed> seeds;
  std::vector<int2> arms;
  std::vector<int64_t> heavy_off{0}, hchunk_off{0}, hchunk_e0, hchunk_e1;
  std::vector<int32_t> heavy, hchunk_v, hfirst;
  std::vector<int32_t> dist, queue;
  std::vector<int32_t> cof, cpos;  // chain vertex -> chain (global), position
  int64_t ncap = 1;
  int tcap = 2;
  cpre_off.resize((size_t)B->n_chains);
  gcof.resize((size_t)std::max<int64_t>(B->n_packed, 1));
  gcpos.resize(gcof.size());
  for (int32_t b = 0; b < B->n_bcc; ++b) {
    const int64_t vo = B->vtx_off[b];
    const int32_t nb = (int32_t)(B->vtx_off[b + 1] - vo);
    const int32_t npl = B->n_plain[b];
    const int64_t ce0 = B->chain_off[b], ce1 = B->chain_off[b + 1];
    if (cfg.bccs_on && !(*cfg.bccs_on)[b]) {  // scheduled elsewhere: empty per-BCC table entries
      hvo.push_back((int64_t)hrow.size());
      hfirst.push_back((int32_t)((int64_t)hchunk_v.size() - hchunk_off.back()));
      heavy_off.push_back((int64_t)heavy.size());
      hchunk_off.push_back((int64_t)hchunk_v.size());
      continue;
    }
    ncap = std::max<int64_t>(ncap, npl);
    const int64_t arcs = B->row[vo + nb] - B->row[vo];
    // chain membership, and the shape the closed forms rely on: each chain
    // vertex has exactly its two chain neighbours, the ends are distinct core
    // vertices. Checked in parallel; the error reported is the one a pass in
    // chain order meets first (per chain: equal ends, then a vertex an
    // earlier chain holds, then the neighbours).
    const int64_t nchb = ce1 - ce0;
    std::vector<int32_t> first((size_t)nb, INT32_MAX);  // smallest chain (BCC-relative) holding each vertex
    std::vector<int32_t> csize((size_t)nchb + 1, 0);     // prefix-sum entries of each chain (0: nothing hangs off it)
    std::vector<uint8_t> cerr((size_t)nchb, 0);          // 1 equal ends, 3 bad neighbours (2 = overlap, below)
    int kmax = 0;
#pragma omp parallel for schedule(static) reduction(max : kmax)
    for (int64_t i = 0; i < nchb; ++i) {
      const int64_t c = ce0 + i;
      const int32_t st = B->chain_start[c], k = B->chain_len[c], L = B->chain_l[c], R = B->chain_r[c];
      kmax = std::max(kmax, k);
      if (L == R) { cerr[(size_t)i] = 1; continue; }
      bool flat = true;
      for (int32_t j = 0; j < k; ++j) {
        int32_t *f = &first[(size_t)(st + j)];
        int32_t cur = __atomic_load_n(f, __ATOMIC_RELAXED);
        while ((int32_t)i < cur && !__atomic_compare_exchange_n(f, &cur, (int32_t)i, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED)) {
        }
        const int32_t x = st + j, prev = j == 0 ? L : x - 1, next = j == k - 1 ? R : x + 1;
        const int64_t e0 = B->row[vo + x], e1 = B->row[vo + x + 1];
        if (e1 - e0 != 2 || !((B->col[e0] == prev && B->col[e0 + 1] == next) || (B->col[e0] == next && B->col[e0 + 1] == prev)))
          cerr[(size_t)i] = 3;
        flat = flat && B->reach[vo + x] == 0;
      }
      csize[(size_t)i + 1] = flat ? 0 : k + 1;
    }
    int64_t bad_chain = nchb;  // the first chain with an error
#pragma omp parallel for schedule(static) reduction(min : bad_chain)
    for (int64_t i = 0; i < nchb; ++i) {
      if (cerr[(size_t)i] != 1) {
        const int32_t st = B->chain_start[ce0 + i], k = B->chain_len[ce0 + i];
        for (int32_t j = 0; j < k; ++j)
          if (first[(size_t)(st + j)] < (int32_t)i) cerr[(size_t)i] = 2;  // an earlier chain holds the vertex
      }
      if (cerr[(size_t)i]) bad_chain = std::min(bad_chain, i);
    }
    if (bad_chain < nchb) {
      const int e = cerr[(size_t)bad_chain];
      return bail(BCGPU_EINVAL, e == 1 ? "a chain whose two ends are the same vertex"
                                 : e == 2 ? "chains overlap"
                                          : "a chain vertex whose neighbours are not its chain neighbours");
    }
    for (int64_t i = 0; i < nchb; ++i) csize[(size_t)i + 1] += csize[(size_t)i];
    const int64_t cpre0 = (int64_t)cpre.size();
    cpre.resize((size_t)(cpre0 + csize[(size_t)nchb]));
    cof.assign((size_t)nb, -1);
    cpos.assign((size_t)nb, -1);
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < nchb; ++i) {
      const int64_t c = ce0 + i;
      const int32_t st = B->chain_start[c], k = B->chain_len[c];
      for (int32_t j = 0; j < k; ++j) {
        cof[(size_t)(st + j)] = (int32_t)c;
        cpos[(size_t)(st + j)] = j;
      }
      const bool flat = csize[(size_t)i + 1] == csize[(size_t)i];
      cpre_off[c] = flat ? -1 : cpre0 + csize[(size_t)i];
      if (!flat) {
        double *P = cpre.data() + cpre0 + csize[(size_t)i], acc = 0.0;
        P[0] = 0.0;
        for (int32_t j = 0; j < k; ++j) {
          acc += (double)B->reach[vo + st + j] + 1.0;
          P[j + 1] = acc;
        }
      }
    }
    HOST_MARK("b: chains");
    // contracted rows: unit arcs first, then chain arcs
    hvo.push_back((int64_t)hrow.size());
    int heavy_deg = kHeavyDegSmall;
    if (npl >= kSmallCore) {
      int64_t longer = 0;
#pragma omp parallel for schedule(static) reduction(+ : longer)
      for (int32_t x = 0; x < npl; ++x) {
        const int64_t deg = B->row[vo + x + 1] - B->row[vo + x];
        longer += deg > kHeavyDeg && deg <= kHeavyDegMany;
      }
      heavy_deg = longer < kManyRows ? kHeavyDeg : kHeavyDegMany;
    }
    // Every arc of a core vertex becomes one contracted arc (a unit arc, or
    // the chain arc of the chain vertex it leads to), so the contracted rows
    // have the original degrees: offsets first, then the rows in parallel.
    std::copy(cof.begin(), cof.end(), gcof.begin() + vo);  // the device fill reads them per packed vertex
    std::copy(cpos.begin(), cpos.end(), gcpos.begin() + vo);
    const size_t rb = hrow.size();
    hrow.resize(rb + (size_t)npl + 1);
    hrow[rb] = narcs;
    for (int32_t x = 0; x < npl; ++x) hrow[rb + x + 1] = hrow[rb + x] + (B->row[vo + x + 1] - B->row[vo + x]);
    narcs = hrow[rb + npl];
    rbcc.resize(rb + (size_t)npl, b);
    hrow.pop_back();  // the BCC's end offset is pushed below, after its heavy rows
    int32_t hidx = 0;
    for (int32_t x = 0; x < npl; ++x) {
      const int64_t r0 = hrow[rb + x], r1 = x + 1 < npl ? hrow[rb + x + 1] : narcs;
      if (r1 - r0 <= heavy_deg) continue;
      heavy.push_back(x);
      hfirst.push_back((int32_t)((int64_t)hchunk_v.size() - hchunk_off.back()));
      for (int64_t e = r0; e < r1; e += kChunkArcs) {
        hchunk_v.push_back(hidx);
        hchunk_e0.push_back(e);
        hchunk_e1.push_back(std::min<int64_t>(r1, e + kChunkArcs));
      }
      ++hidx;
    }
    hrow.push_back(narcs);
    rbcc.push_back(-1);
    hfirst.push_back((int32_t)((int64_t)hchunk_v.size() - hchunk_off.back()));
    heavy_off.push_back((int64_t)heavy.size());
    hchunk_off.push_back((int64_t)hchunk_v.size());
    const int32_t ecc = cfg.ecc0 && (*cfg.ecc0)[b] >= 0 ? (*cfg.ecc0)[b] : bcc_ecc(B->row, B->col, vo, nb, dist, queue);
    tcap = std::max(tcap, 2 * ecc + kmax + 3);

    const int64_t bat0g = (int64_t)P->h_batches.size(), nbat = ((int64_t)nb + width - 1) / width;
    const int64_t jf0 = std::min(nbat, std::max<int64_t>(0, cfg.fill_begin - bat0g));
    const int64_t jf1 = std::max(jf0, std::min(nbat, cfg.fill_end - bat0g));
    const size_t need = (size_t)std::min<int64_t>(nb, jf1 * (int64_t)width);
    std::vector<int32_t> own_order;
    const std::vector<int32_t> *order_p = cfg.order_of ? &cfg.order_of(b) : nullptr;
    if (!order_p) {
      batched_source_order(B, b, width, (int64_t)need, own_order);
      order_p = &own_order;
    }
    const std::vector<int32_t> &order = *order_p;
    if (order.size() < need) return bail(BCGPU_EINVAL, "source order shorter than the passes need");
    HOST_MARK("b: order");
    // Passes of `width` consecutive sources of the order. Slots and seeds are
    // sized up front (a chain source has two seeds), then every pass fills
    // its own ranges in parallel; the arming lists (variable length after
    // deduplication) are built per pass and concatenated in pass order.
    const size_t bat0 = P->h_batches.size(), slot0 = slots.size(), seed0 = seeds.size();
    std::vector<int64_t> seed_at((size_t)nbat + 1, 0);
#pragma omp parallel for schedule(static)
    for (int64_t j = jf0; j < jf1; ++j) {
      const size_t i0 = (size_t)j * width, i1 = std::min(order.size(), i0 + (size_t)width);
      int64_t cnt = 0;
      for (size_t i = i0; i < i1; ++i) cnt += order[i] >= npl ? 2 : 0;
      seed_at[j + 1] = cnt;
    }
    for (int64_t j = 0; j < nbat; ++j) seed_at[j + 1] += seed_at[j];
    P->h_batches.resize(bat0 + (size_t)nbat);
    slots.resize(slot0 + (size_t)nb);
    seeds.resize(seed0 + (size_t)seed_at[nbat]);
    std::vector<std::vector<int2>> arm_of((size_t)nbat);
#pragma omp parallel for schedule(dynamic, 16)
    for (int64_t j = 0; j < nbat; ++j) {
      const size_t i0 = (size_t)j * width, i1 = std::min((size_t)nb, i0 + (size_t)width);
      const bool fill = j >= jf0 && j < jf1;
      Batch bt{};
      bt.bcc = b;
      bt.nslots = (int32_t)(i1 - i0);
      bt.words = (bt.nslots + 31) / 32;
      bt.kmax = kmax;
      bt.heavy_deg = heavy_deg;
      bt.slot_off = (int64_t)(slot0 + i0);
      bt.seed_off = (int64_t)seed0 + seed_at[j];
      int64_t sd = bt.seed_off;
      std::vector<int2> &arm = arm_of[j];
      if (fill) arm.reserve((size_t)bt.nslots * 2);
      for (size_t i = i0; fill && i < i1; ++i) {
        const int32_t s = order[i];
        const int32_t slot = (int32_t)(i - i0);
        if (s < npl) {
          slots[slot0 + i] = Slot{s, -1, 0, 0};
          arm.push_back(make_int2(s, 0));
          continue;
        }
        const int64_t c = cof[s];
        const int32_t p = cpos[s], k = B->chain_len[c];
        slots[slot0 + i] = Slot{s, (int32_t)c, p, 0};
        seeds[sd++] = Seed{B->chain_l[c], p + 1, slot, (int32_t)(bat0 + j)};
        seeds[sd++] = Seed{B->chain_r[c], k - p, slot, (int32_t)(bat0 + j)};
        bt.max_seed = std::max(bt.max_seed, std::max(p + 1, k - p));
      }
      bt.nseeds = (int32_t)(sd - bt.seed_off);
      // arming list: each core source (level 0) and seeded vertex (its lowest seed level), once
      for (int64_t i = bt.seed_off; i < sd; ++i) arm.push_back(make_int2(seeds[i].v, seeds[i].level));
      std::sort(arm.begin(), arm.end(), [](const int2 &x, const int2 &y) { return x.x != y.x ? x.x < y.x : x.y < y.y; });
      size_t u = 0;
      for (size_t i = 0; i < arm.size(); ++i)
        if (i == 0 || arm[i].x != arm[i - 1].x) arm[u++] = arm[i];
      arm.resize(u);
      bt.narm = (int32_t)u;
      P->h_batches[bat0 + j] = bt;
    }
    for (int64_t j = 0; j < nbat; ++j) {
      Batch &bt = P->h_batches[bat0 + j];
      bt.arm_off = (int64_t)arms.size();
      arms.insert(arms.end(), arm_of[j].begin(), arm_of[j].end());
      std::vector<int2>().swap(arm_of[j]);
      P->u_src.push_back(bt.nslots);
      P->u_teps.push_back((int64_t)bt.nslots * arcs);
      P->u_bfs.push_back(bt.nslots);
      P->u_aux.push_back(0);
      P->u_visits.push_back((int64_t)bt.nslots * nb);
    }
  }
  HOST_MARK("b: passes");
  P->tcap = tcap;
  P->n_cap = ncap;
  P->n_batches = (int64_t)P->h_batches.size();
  auto prefix = [](std::vector<int64_t> &v) {
    std::vector<int64_t> p(v.size() + 1, 0);
    for (size_t i = 0; i < v.size(); ++i) p[i + 1] = p[i] + v[i];
    v.swap(p);
  };
  prefix(P->u_src); prefix(P->u_teps); prefix(P->u_bfs); prefix(P->u_aux); prefix(P->u_visits);

  // ---- device workspace
  const int64_t n = P->n_cap;
  const int64_t qb = P->f32 ? 4 : 8;
  const int64_t nch = (int64_t)hchunk_v.size();
  auto need_of = [&](int64_t w) {
    return n * w * 32 * (4 + 8 + 8 + qb) + (int64_t)(tcap + 2) * n * w * 4 + n * w * 4 + n * 12 + n * w * 8 +
           w * 32 * (tcap + 2) * 4 + nch * w * 32 * 8;
  };
  const int64_t need = need_of(W);
  auto workspace_of = [&](int64_t w) {  // every byte of it, as allocated below
    return n * (w * 32 * (4 + 8 + qb + 8) + (int64_t)(tcap + 2) * w * 4 + w * 4 + 8 + w * 8) + (4 * ((int64_t)tcap + 3) + 2) * 4 +
           w * 32 * (8 + 4 + ((int64_t)tcap + 2) * 4 + 4) + (int64_t)sizeof(Ctrl) +
           std::max<int64_t>(P->n_batches, 1) * 4 + std::max<int64_t>(nch, 1) * w * (32 * 8 + 4);
  };
  if (need > cfg.limit_bytes)
    return bail(BCGPU_ENOMEM, "batched workspace " + std::to_string(need >> 20) + " MiB exceeds the limit " +
                                  std::to_string(cfg.limit_bytes >> 20) + " MiB (lower the batch width)");
  P->pool = cfg.pool;
  P->stream = stream;
  auto alloc = [&](void **p, int64_t bytes) -> bool {
    const size_t sz = (size_t)std::max<int64_t>(bytes, 16);
    cudaError_t e = P->pool ? cudaMallocFromPoolAsync(p, sz, P->pool, stream) : cudaMalloc(p, sz);
    if (e == cudaErrorMemoryAllocation && P->pool) {  // trim the pool's unused reserve once and retry
      cudaGetLastError();
      if (cudaStreamSynchronize(stream) == cudaSuccess && cudaMemPoolTrimTo(P->pool, 0) == cudaSuccess)
        e = cudaMallocFromPoolAsync(p, sz, P->pool, stream);
    }
    if (e != cudaSuccess) return false;
    P->allocs.push_back(*p);
    P->bytes += bytes;
    return true;
  };
  Args &a = P->args;
  void *p = nullptr;
  bool ok = true;
  // tables
  auto upload = [&](const void **dst, const void *src, int64_t bytes) -> bool {
    if (!alloc(&p, bytes)) return false;
    *dst = p;
    if (bytes == 0) return true;
    if (cudaMemcpyAsync(p, src, (size_t)bytes, cudaMemcpyHostToDevice, stream) != cudaSuccess) return false;
    P->h2d += bytes;
    return true;
  };
  ok = ok && upload((const void **)&a.hvo, hvo.data(), (int64_t)hvo.size() * 8);
  ok = ok && upload((const void **)&a.hrow, hrow.data(), (int64_t)hrow.size() * 8);
  ok = ok && upload((const void **)&a.n_plain, B->n_plain, (int64_t)B->n_bcc * 4);
  // the contracted rows themselves: filled on the device from the packed CSR
  const int32_t *d_rbcc = nullptr, *d_gcof = nullptr, *d_gcpos = nullptr;
  int *d_bad = nullptr;
  ok = ok && upload((const void **)&d_rbcc, rbcc.data(), (int64_t)rbcc.size() * 4);
  ok = ok && upload((const void **)&d_gcof, gcof.data(), (int64_t)gcof.size() * 4);
  ok = ok && upload((const void **)&d_gcpos, gcpos.data(), (int64_t)gcpos.size() * 4);
  ok = ok && alloc(&p, (int64_t)hrow.size() * 8); a.hsplit = (const int64_t *)p;
  ok = ok && alloc(&p, narcs * 4); a.hcol = (const int32_t *)p;
  ok = ok && alloc(&p, narcs * 4); a.hk = (const int32_t *)p;
  ok = ok && alloc(&p, narcs * 4); a.hcid = (const int32_t *)p;
  ok = ok && alloc(&p, 4); d_bad = (int *)p;
  if (ok && !hrow.empty()) {
    ok = cudaMemsetAsync(d_bad, 0, sizeof(int), stream) == cudaSuccess;
    const int64_t nr = (int64_t)hrow.size();
    const int blocks = (int)std::min<int64_t>((nr + 7) / 8, 148 * 16);  // a warp a row
    if (ok) {
      contract_rows_kernel<<<blocks, 256, 0, stream>>>(row, col, vtx_off, a.n_plain, d_rbcc, a.hvo, a.hrow, nr, d_gcof,
                                                       d_gcpos, chain_len, chain_l, chain_r, (int64_t *)a.hsplit,
                                                       (int32_t *)a.hcol, (int32_t *)a.hk, (int32_t *)a.hcid, d_bad);
      ok = cudaGetLastError() == cudaSuccess;
    }
  }
  ok = ok && upload((const void **)&a.chain_off, B->chain_off, (int64_t)(B->n_bcc + 1) * 8);
  ok = ok && upload((const void **)&a.cpre_off, cpre_off.data(), (int64_t)cpre_off.size() * 8);
  ok = ok && upload((const void **)&a.cpre, cpre.data(), (int64_t)cpre.size() * 8);
  ok = ok && upload((const void **)&a.heavy_off, heavy_off.data(), (int64_t)heavy_off.size() * 8);
  ok = ok && upload((const void **)&a.heavy, heavy.data(), (int64_t)heavy.size() * 4);
  ok = ok && upload((const void **)&a.hchunk_off, hchunk_off.data(), (int64_t)hchunk_off.size() * 8);
  ok = ok && upload((const void **)&a.hchunk_v, hchunk_v.data(), nch * 4);
  ok = ok && upload((const void **)&a.hchunk_e0, hchunk_e0.data(), nch * 8);
  ok = ok && upload((const void **)&a.hchunk_e1, hchunk_e1.data(), nch * 8);
  ok = ok && upload((const void **)&a.hfirst, hfirst.data(), (int64_t)hfirst.size() * 4);
  ok = ok && upload((const void **)&a.batches, P->h_batches.data(), (int64_t)P->h_batches.size() * (int64_t)sizeof(Batch));
  {  // slots: only those of the filled passes are copied (the rest are never read)
    int64_t s0 = (int64_t)slots.size(), s1 = 0;
    for (int64_t j = std::max<int64_t>(0, cfg.fill_begin); j < std::min(P->n_batches, cfg.fill_end); ++j) {
      s0 = std::min(s0, P->h_batches[(size_t)j].slot_off);
      s1 = std::max(s1, P->h_batches[(size_t)j].slot_off + P->h_batches[(size_t)j].nslots);
    }
    ok = ok && alloc(&p, (int64_t)slots.size() * (int64_t)sizeof(Slot));
    a.slots = (const Slot *)p;
    if (ok && s1 > s0) {
      const size_t bytes = (size_t)(s1 - s0) * sizeof(Slot);
      ok = cudaMemcpyAsync((Slot *)p + s0, slots.data() + s0, bytes, cudaMemcpyHostToDevice, stream) == cudaSuccess;
      P->h2d += (int64_t)bytes;
    }
  }
  ok = ok && upload((const void **)&a.seeds, seeds.data(), (int64_t)seeds.size() * (int64_t)sizeof(Seed));
  ok = ok && upload((const void **)&a.arms, arms.data(), (int64_t)arms.size() * (int64_t)sizeof(int2));
  // Passes run as one: as many as the rule allows, the plan will run and, with the
  // tables above, fit what the rest of the plan leaves; a pass has to end on a
  // whole group of words.
  const int64_t filled = std::min(P->n_batches, cfg.fill_end) - std::max<int64_t>(0, cfg.fill_begin);
  P->merge = W * 32 == width ? (int)std::max<int64_t>(1, std::min<int64_t>(merge_passes(n, width), filled)) : 1;
  while (P->merge > 1 && P->bytes + workspace_of((int64_t)P->merge * W) > cfg.merge_bytes) --P->merge;
  const int64_t WA = (int64_t)P->merge * W;  // words a row is allocated
  ok &= ok && alloc(&p, n * WA * 32 * 4); a.d = (int32_t *)p;
  ok &= ok && alloc(&p, n * WA * 32 * 8); a.sig = (double *)p;
  ok &= ok && alloc(&p, n * WA * 32 * qb); a.q = p;
  ok &= ok && alloc(&p, (int64_t)(tcap + 2) * n * WA * 4); a.lm = (uint32_t *)p;
  ok &= ok && alloc(&p, n * WA * 4); a.seen = (uint32_t *)p;
  ok &= ok && alloc(&p, n * 4); a.lmin = (int32_t *)p;
  ok &= ok && alloc(&p, n * 4); a.armed = (int32_t *)p;
  ok &= ok && alloc(&p, (4 * ((int64_t)tcap + 3) + 2) * 4); a.wq = (int *)p;
  ok &= ok && alloc(&p, n * WA * 8); a.bcpart = (double *)p;
  ok &= ok && alloc(&p, n * WA * 32 * 8); a.cdep = (double *)p;
  ok &= ok && alloc(&p, WA * 32 * 8); a.wsrc = (double *)p;
  ok &= ok && alloc(&p, WA * 32 * 4); a.schain = (int32_t *)p;
  ok &= ok && alloc(&p, WA * 32 * (tcap + 2) * 4); a.X = (int32_t *)p;
  ok &= ok && alloc(&p, WA * 32 * 4); a.rexp = (int32_t *)p;
  ok &= ok && alloc(&p, sizeof(Ctrl)); a.ctrl = (Ctrl *)p;
  ok &= ok && alloc(&p, (int64_t)std::max<int64_t>(P->n_batches, 1) * 4); a.redo = (int *)p;
  ok = ok && alloc(&p, std::max<int64_t>(nch, 1) * WA * 32 * 8); a.hacc = (double *)p;
  ok = ok && alloc(&p, std::max<int64_t>(nch, 1) * WA * 4); a.hmask = (uint32_t *)p;
  HOST_MARK("b: ws alloc");
  if (!ok) return bail(BCGPU_ENOMEM, "cudaMalloc or upload of the batched workspace failed");
  cudaError_t e = cudaMemsetAsync(a.ctrl, 0, sizeof(Ctrl), stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(a.redo, 0, (size_t)std::max<int64_t>(P->n_batches, 1) * 4, stream);
  int h_bad = 0;
  if (e == cudaSuccess && !hrow.empty()) {
    e = cudaMemcpyAsync(&h_bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, stream);
    P->d2h += (int64_t)sizeof(int);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);  // the host vectors go out of scope
  HOST_MARK("b: uploads+sync");
  P->h_slots = std::move(slots);
  if (cfg.keep_host_tables) {
    P->h_seeds = std::move(seeds);
    P->h_arms = std::move(arms);
  }
  P->h_vtx_off.assign(B->vtx_off, B->vtx_off + B->n_bcc + 1);
  if (e != cudaSuccess) return bail(BCGPU_ECUDA, std::string("batched upload: ") + cudaGetErrorString(e));
  if (h_bad & 1) return bail(BCGPU_EINVAL, "a non-core vertex outside every chain");
  if (h_bad & 2) return bail(BCGPU_EINVAL, "a core vertex adjacent to the inside of a chain");
  a.reach = reach; a.vtx_off = vtx_off;
  a.chain_start = chain_start; a.chain_len = chain_len; a.chain_l = chain_l; a.chain_r = chain_r;
  a.n_cap = P->n_cap; a.W = W; a.width = width; a.merge = 1; a.tcap = tcap; a.bc = bc; a.err = err;
  a.rescale_exp = cfg.rescale_exp > 0 ? cfg.rescale_exp : 900;
  a.wait_ns = cfg.wait_ns;

  // cooperative grid: every CTA resident
  int dev = 0, sms = 0, per_sm = 0, coop = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  if (!coop) return bail(BCGPU_ECUDA, "device lacks cooperative launch");
  const size_t smem = sizeof(WarpScratch) * kWarpsPerCta;
  if (cudaFuncSetAttribute(batched_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaFuncSetAttribute(batched_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return bail(BCGPU_ECUDA, "cannot reserve shared memory for the batched kernel");
  if (P->f32) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_kernel<float>, kThreads, smem);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_kernel<double>, kThreads, smem);
  P->smem = smem;
  if (per_sm < 1) return bail(BCGPU_ECUDA, "batched kernel does not fit an SM");
  P->grid = sms * per_sm;
  return BCGPU_OK;
}

}  // namespace

int batched_create(const bc_bccs *B, const BatchedConfig &cfg, const int64_t *row, const int32_t *col,
                   const int32_t *reach, const int64_t *vtx_off, const int32_t *chain_start, const int32_t *chain_len,
                   const int32_t *chain_l, const int32_t *chain_r, double *bc, int *err, cudaStream_t stream,
                   BatchedPlan **out, std::string *msg) {
  BatchedPlan *P = nullptr;
  int rc;
  try {  // a host allocation that throws releases the partial plan like any other failure
    P = new BatchedPlan;
    rc = batched_build(B, cfg, row, col, reach, vtx_off, chain_start, chain_len, chain_l, chain_r, bc, err, stream, P,
                       msg);
  } catch (const std::bad_alloc &) {
    if (msg) *msg = "host allocation failed while building the passes";
    rc = BCGPU_ENOMEM;
  }
  if (rc != BCGPU_OK) {
    batched_destroy(P);
    return rc;
  }
  *out = P;
  return BCGPU_OK;
}

void batched_destroy(BatchedPlan *p) {
  if (!p) return;
  for (void *a : p->allocs) {
    if (p->pool) cudaFreeAsync(a, p->stream);
    else cudaFree(a);
  }
  delete p;
}

int64_t batched_device_bytes(const BatchedPlan *p) { return p ? p->bytes : 0; }

uint64_t batched_pass_digest(const BatchedPlan *p, int64_t pass) {
  if (!p || pass < 0 || pass >= (int64_t)p->h_batches.size()) return 0;
  const Batch &b = p->h_batches[(size_t)pass];
  if ((int64_t)p->h_seeds.size() < b.seed_off + b.nseeds || (int64_t)p->h_arms.size() < b.arm_off + b.narm) return 0;
  uint64_t h = 1469598103934665603ull;  // FNV-1a
  auto mix = [&h](const void *q, size_t n) {
    const unsigned char *c = (const unsigned char *)q;
    for (size_t i = 0; i < n; ++i) h = (h ^ c[i]) * 1099511628211ull;
  };
  const int32_t head[8] = {b.bcc, b.nslots, b.words, b.nseeds, b.max_seed, b.kmax, b.heavy_deg, b.narm};
  mix(head, sizeof head);
  mix(p->h_slots.data() + b.slot_off, sizeof(Slot) * (size_t)b.nslots);
  mix(p->h_seeds.data() + b.seed_off, sizeof(Seed) * (size_t)b.nseeds);
  mix(p->h_arms.data() + b.arm_off, sizeof(int2) * (size_t)b.narm);
  return h;
}
int64_t batched_h2d_bytes(const BatchedPlan *p) { return p ? p->h2d : 0; }
int64_t batched_d2h_bytes(const BatchedPlan *p) { return p ? p->d2h : 0; }
int64_t batched_status_bytes(const BatchedPlan *p) {
  return p ? (int64_t)sizeof(int) * std::max<int64_t>(p->n_batches, 1) : 0;
}
int batched_width(const BatchedPlan *p) { return p ? p->width : 0; }

void batched_unit_sources(const BatchedPlan *p, int64_t begin, int64_t end, std::vector<int64_t> &out) {
  for (int64_t bi = begin; bi < end; ++bi) {
    const Batch &bt = p->h_batches[bi];
    const int64_t vo = p->h_vtx_off[bt.bcc];
    for (int32_t i = 0; i < bt.nslots; ++i) out.push_back(vo + p->h_slots[bt.slot_off + i].src);
  }
}

int batched_pass_shape(const BatchedPlan *p, int64_t pass, int32_t *bcc, int32_t *nslots) {
  if (!p || pass < 0 || pass >= p->n_batches) return BCGPU_EINVAL;
  *bcc = p->h_batches[pass].bcc;
  *nslots = p->h_batches[pass].nslots;
  return BCGPU_OK;
}

int batched_pass_rows(const BatchedPlan *p, int64_t pass, const int32_t *chain_start, int32_t n_core,
                      cudaStream_t stream, std::vector<int32_t> &src, std::vector<int32_t> &d, std::vector<double> &sigma,
                      std::string *msg) {
  if (pass < 0 || pass >= p->n_batches) {
    *msg = "not a multi-source pass";
    return BCGPU_EINVAL;
  }
  const Batch &bt = p->h_batches[pass];
  const int B = bt.nslots, WB = p->W * 32, L = p->tcap + 2;
  std::vector<int32_t> hd((size_t)n_core * WB), hx((size_t)WB * L);
  std::vector<double> hs((size_t)n_core * WB);
  cudaError_t e = cudaMemcpyAsync(hd.data(), p->args.d, hd.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(hs.data(), p->args.sig, hs.size() * sizeof(double), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(hx.data(), p->args.X, hx.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) {
    *msg = std::string("pass row read-back: ") + cudaGetErrorString(e);
    return BCGPU_ECUDA;
  }
  src.resize((size_t)B);
  d.resize((size_t)B * n_core);
  sigma.resize((size_t)B * n_core);
  for (int b = 0; b < B; ++b) {
    const Slot &sl = p->h_slots[bt.slot_off + b];
    src[b] = sl.chain < 0 ? sl.src : chain_start[sl.chain] + sl.pos;
    for (int32_t v = 0; v < n_core; ++v) {
      const size_t i = (size_t)v * WB + b;
      const int lv = hd[i];
      d[(size_t)b * n_core + v] = lv;
      // stored count s at level lv stands for s * 2^X(slot, lv)
      sigma[(size_t)b * n_core + v] = std::ldexp(hs[i], hx[(size_t)b * L + std::min(std::max(lv, 0), L - 1)]);
    }
  }
  return BCGPU_OK;
}

void batched_unit_work(const BatchedPlan *p, std::vector<int64_t> &sources, std::vector<int64_t> &teps,
                       std::vector<int64_t> &bfs, std::vector<int64_t> &aux, std::vector<int64_t> &visits) {
  sources = p->u_src; teps = p->u_teps; bfs = p->u_bfs; aux = p->u_aux; visits = p->u_visits;
}

#ifdef BCGPU_PHASE_TIMERS
}  // namespace bcg
extern "C" int bc_debug_phase_times(unsigned long long *out, int reset) {
  if (cudaMemcpyFromSymbol(out, bcg::g_phase_ns, sizeof(unsigned long long) * 32) != cudaSuccess) return 2;
  if (reset) {
    unsigned long long z[32] = {0};
    cudaMemcpyToSymbol(bcg::g_phase_ns, z, sizeof(z));
  }
  return 0;
}
namespace bcg {
#endif

int batched_failed_batches(BatchedPlan *p, cudaStream_t stream, int64_t *count) {
  std::vector<int> h((size_t)std::max<int64_t>(p->n_batches, 1), 0);
  cudaError_t e = cudaMemcpyAsync(h.data(), p->args.redo, h.size() * sizeof(int), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return BCGPU_ECUDA;
  int64_t c = 0;
  for (int x : h) c += x != 0;
  *count = c;
  return BCGPU_OK;
}

int batched_run(BatchedPlan *p, int64_t begin, int64_t end, cudaStream_t stream, int *launches, std::string *msg) {
  if (end <= begin) return BCGPU_OK;
  Args a = p->args;
  a.b0 = begin;
  a.b1 = end;
  a.merge = (int)std::min<int64_t>(p->merge, end - begin);
  a.W = a.merge * p->W;  // a lone pass keeps the row stride batched_pass_rows reads
  void *params[] = {&a};
  cudaError_t e = cudaMemsetAsync(&p->args.ctrl->bar_count, 0, 2 * sizeof(unsigned int), stream);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (e == cudaSuccess) e = cudaStreamIsCapturing(stream, &cap);
  const void *fn = p->f32 ? (const void *)batched_kernel<float> : (const void *)batched_kernel<double>;
  if (e == cudaSuccess && cap == cudaStreamCaptureStatusActive) {
    // recorded into a CUDA graph: a kernel node carrying the cooperative attribute
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p->grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = p->smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelExC(&cfg, fn, params);
  } else if (e == cudaSuccess) {
    e = cudaLaunchCooperativeKernel(fn, p->grid, kThreads, params, p->smem, stream);
  }
  if (e != cudaSuccess) {
    if (msg) *msg = std::string("cooperative launch: ") + cudaGetErrorString(e);
    return BCGPU_ECUDA;
  }
  if (launches) *launches += 1;
  return BCGPU_OK;
}

}  // namespace bcg
