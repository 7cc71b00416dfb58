// bc_begin_free_noalloc: the free-source BC call for callers that cannot
// allocate device memory (no cudaMalloc, cudaFree or allocating library call
// on this path). Everything the kernels need beyond the caller's own device
// buffers lives in one file-scope __device__ array of fixed size, which every
// GPU that loads this library holds until the process exits.
//
// A BCC that fits shared memory runs on the small-BCC kernels, every SM busy
// whatever the array holds; its slice is built on the device. Nothing is known
// of its depth and path counts beforehand, so a run that ends on the limits of
// those kernels (levels, counts past 2^1000) is run again on the per-source
// kernel, with as many rows as fit the array. 1,500 sources of a BCC of 4,001
// vertices took 17.4 ms on the per-source kernel's 16 CTAs; now 0.33 ms.
#include "bcgpu.h"
#include "common.cuh"
#include "internal.h"
#include "plain.h"
#include "tile.h"

#include <algorithm>
#include <cstdio>
#include <mutex>
#include <string>

namespace bcg {
namespace {

// Limits of one call: a BCC of at most kMaxVertices vertices and at most
// kMaxVertices sources; on the per-source kernel, kSlots CTAs of the largest
// (more of smaller ones), one source each at a time.
constexpr int64_t kMaxVertices = 16384;
constexpr int64_t kSlots = 16;
constexpr int64_t kRowCap = kMaxVertices + 2;  // per-slot row capacity the kernel checks

constexpr int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }
// rows of kSlots slots of the largest BCCs, or whatever else fits there
constexpr int64_t kOffRow = align256(kSlots * kWsIntRows * kRowCap * 4) + align256(kSlots * kWsDblRows * kRowCap * 8);
constexpr int64_t kBytesRow = align256((kMaxVertices + 1) * 8);
constexpr int64_t kOffItems = kOffRow + kBytesRow;
constexpr int64_t kBytesItems = align256(kMaxVertices * (int64_t)sizeof(PlainItem));
constexpr int64_t kOffAcc = kOffItems + kBytesItems;  // fixed-point BC counters, kAccDigits per vertex
constexpr int64_t kBytesAcc = align256(kMaxVertices * kAccDigits * 8);
constexpr int64_t kOffCtl = kOffAcc + kBytesAcc;  // vtx_off[2], counter, epochs[2*kSlots], err
constexpr int64_t kBytesCtl = align256(16 + 8 + 8 * kSlots + 4);
constexpr int64_t kScratchBytes = kOffCtl + kBytesCtl;  // 20,909,056 bytes (about 20 MiB)
static_assert(kScratchBytes == 20909056, "the size the header documents");
static_assert(kMaxVertices <= kAccMaxAdds, "one call's sources must fit the fixed-point counters' headroom");

static __device__ __align__(256) unsigned char g_scratch[kScratchBytes];

// The small-BCC kernels' part, in place of the rows: slice and items.
constexpr int64_t kOffSlice = 0;
constexpr int64_t kBytesSlice = 256 * 1024;  // more than a CTA's shared memory
constexpr int64_t kOffTileItems = kOffSlice + kBytesSlice;
constexpr int64_t kBytesTileItems = kMaxVertices * (int64_t)sizeof(TileItem);
constexpr int64_t kOffTileMeta = kOffTileItems + kBytesTileItems;  // slice_off, slice_bytes
static_assert(kOffTileMeta + 256 <= kOffRow, "the small-BCC kernels' part fits the rows' place");

struct Layout {
  int32_t *ws_i;
  double *ws_f;
  int64_t ws_n;   // rows' capacity
  int slots;
  int64_t *row;
  PlainItem *items;
  unsigned long long *acc;
  int64_t *vtx_off;
  unsigned long long *counter;
  int32_t *epochs;
  int *err;
};

// For BCCs of n vertices: as many slots as the array holds, at least kSlots.
Layout layout(unsigned char *base, int64_t n) {
  Layout L;
  L.ws_n = n + 2;
  const int64_t slot = L.ws_n * (kWsDblRows * 8 + kWsIntRows * 4) + 2 * 4;  // rows and two epochs
  L.slots = (int)std::min<int64_t>(kOffRow / slot, 148 * 4);
  L.row = reinterpret_cast<int64_t *>(base + kOffRow);
  L.items = reinterpret_cast<PlainItem *>(base + kOffItems);
  L.acc = reinterpret_cast<unsigned long long *>(base + kOffAcc);
  L.vtx_off = reinterpret_cast<int64_t *>(base + kOffCtl);
  L.counter = reinterpret_cast<unsigned long long *>(base + kOffCtl + 16);
  L.err = reinterpret_cast<int *>(base + kOffCtl + 24 + 8 * kSlots);
  L.ws_f = reinterpret_cast<double *>(base);
  if (L.slots > kSlots) {
    L.ws_i = reinterpret_cast<int32_t *>(L.ws_f + L.slots * kWsDblRows * L.ws_n);
    L.epochs = L.ws_i + L.slots * kWsIntRows * L.ws_n;
  } else {  // the largest BCCs' epochs have a place of their own
    L.slots = (int)kSlots;
    L.ws_i = reinterpret_cast<int32_t *>(L.ws_f + kSlots * kWsDblRows * L.ws_n);
    L.epochs = reinterpret_cast<int32_t *>(base + kOffCtl + 24);
  }
  return L;
}

// Builds the work items of one call: row offsets widened to int64, one item
// per source. Malformed input (offsets, neighbour ids, sources) sets the error
// flag, and the BC kernel then takes no work. With rows of a new layout
// (first != 0) it also sets the level-stamp epochs to 1; the rows were cleared
// just before. Calls of the same layout keep the epochs and stamps the previous
// one left (every stamp is below its row's epoch, and the kernel wraps a row
// back to zero before an epoch could overflow). The fixed-point counters are
// found cleared by the previous call's fold.
__global__ void setup_kernel(Layout L, const int32_t *R, const int32_t *C, int32_t n, int32_t m, const int32_t *src,
                             int32_t nsrc, int first) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = tid; i <= n; i += stride) {
    const int32_t r = R[i];
    if (r < 0 || r > m || (i == 0 && r != 0) || (i == n && r != m) || (i < n && R[i + 1] < r))
      set_err(L.err, kDevBadItem);
    L.row[i] = r;
  }
  for (int64_t e = tid; e < m; e += stride)
    if (C[e] < 0 || C[e] >= n) set_err(L.err, kDevBadItem);
  for (int64_t i = tid; i < nsrc; i += stride) {
    int32_t s = src[i];
    if (s < 0 || s >= n) {
      set_err(L.err, kDevBadItem);
      s = 0;
    }
    L.items[i] = PlainItem{0, s, 0, 0, 1};
  }
  if (first)
    for (int64_t i = tid; i < 2 * L.slots; i += stride) L.epochs[i] = 1;
  if (tid == 0) {
    L.vtx_off[0] = 0;
    L.vtx_off[1] = n;
    *L.counter = 0;
  }
}

// First pair of row i, which starts at arc r, in a slice laid out without a
// prefix sum: rows get the pairs they need, some one more.
__host__ __device__ __forceinline__ int64_t slice_pair(int64_t r, int64_t i) { return (r + i + 1) / 2; }

// The same for the small-BCC kernels: the BCC's slice, and items of per sources
// each. The same checks; the kernels take no work after an error.
__global__ void slice_kernel(unsigned char *base, Layout L, const int32_t *R, const int32_t *C, int32_t n, int32_t m,
                             const int32_t *src, int32_t nsrc, int32_t per) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const bool narrow = TileSlice::narrow(slice_pair(m, n));
  unsigned char *slice = base + kOffSlice;
  uint16_t *col = reinterpret_cast<uint16_t *>(slice + TileSlice::col_at(n, narrow));
  for (int64_t i = tid / 32; i <= n; i += stride / 32) {  // a warp per row
    const int lane = (int)(tid & 31);
    const int32_t r = R[i], r1 = i < n ? R[i + 1] : m;
    if (r < 0 || r > m || (i == 0 && r != 0) || (i == n && r != m) || r1 < r || r1 > m) {
      if (lane == 0) set_err(L.err, kDevBadItem);
      continue;
    }
    const int64_t p = slice_pair(r, i);
    if (lane == 0) {
      if (narrow) reinterpret_cast<uint16_t *>(slice)[i] = (uint16_t)p;
      else reinterpret_cast<int32_t *>(slice)[i] = (int32_t)p;
    }
    if (i == n) continue;
    const int64_t places = 2 * (slice_pair(r1, i + 1) - p);
    for (int64_t j = lane; j < places; j += 32) {
      int32_t c = (int32_t)i;  // a spare place
      if (j < r1 - r) {
        c = C[r + j];
        if (c < 0 || c >= n) {
          set_err(L.err, kDevBadItem);
          c = 0;
        }
      }
      col[2 * p + j] = (uint16_t)c;
    }
  }
  for (int64_t i = tid; i < nsrc; i += stride)
    if (src[i] < 0 || src[i] >= n) set_err(L.err, kDevBadItem);
  TileItem *items = reinterpret_cast<TileItem *>(base + kOffTileItems);
  for (int64_t i = tid; i * per < nsrc; i += stride)
    items[i] = TileItem{0, (int32_t)(i * per), (int32_t)min((int64_t)nsrc, (i + 1) * per), 0};
  if (tid == 0) {
    L.vtx_off[0] = 0;
    L.vtx_off[1] = n;
    *L.counter = 0;
    *reinterpret_cast<int64_t *>(base + kOffTileMeta) = narrow ? 1 : 0;
    *reinterpret_cast<int32_t *>(base + kOffTileMeta + 8) = (int32_t)TileSlice::bytes(n, slice_pair(m, n));
  }
}

// One run of the call: clears the error flag and bc, checks and lays out the
// input, runs the sources, folds the counters into bc. cls >= 0: the small-BCC
// kernels.
cudaError_t enqueue(unsigned char *base, const Layout &L, int cls, size_t smem, int grid, bool rows_first,
                    bool acc_first, const int32_t *R, const int32_t *C, int32_t n, int32_t m, const int32_t *src,
                    int32_t nsrc, const int32_t *reach, double *bc, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(L.err, 0, sizeof(int), stream);
  if (e == cudaSuccess && cls < 0 && rows_first)  // row records: unvisited
    e = cudaMemsetAsync(L.ws_f, 0, sizeof(double) * (size_t)(L.slots * kWsDblRows * L.ws_n), stream);
  if (e == cudaSuccess && acc_first) e = cudaMemsetAsync(L.acc, 0, (size_t)kBytesAcc, stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(bc, 0, sizeof(double) * (size_t)n, stream);
  if (e != cudaSuccess) return e;
  if (cls < 0) {
    setup_kernel<<<64, 256, 0, stream>>>(L, R, C, n, m, src, nsrc, rows_first ? 1 : 0);
    e = cudaGetLastError();
    if (e != cudaSuccess || nsrc == 0) return e;
    PlainArgs a{};
    a.row = L.row;
    a.col = C;
    a.reach = reach;
    a.vtx_off = L.vtx_off;
    a.items = L.items;
    a.item_begin = 0;
    a.item_end = nsrc;
    a.next_item = L.counter;
    a.acc = L.acc;
    a.ws_i = L.ws_i;
    a.ws_f = L.ws_f;
    a.ws_n = L.ws_n;
    a.epochs = L.epochs;
    a.rows_slot = -1;  // no row export on this path (launch_rows is never called with these arguments)
    a.rescale_exp = 900;
    a.err = L.err;
    e = launch_plain(a, 256, (int)std::min<int64_t>(L.slots, nsrc), stream);
  } else {
    const int32_t per = tile_item_sources(cls, grid, nsrc);
    slice_kernel<<<64, 256, 0, stream>>>(base, L, R, C, n, m, src, nsrc, per);
    e = cudaGetLastError();
    if (e != cudaSuccess || nsrc == 0) return e;
    TileArgs a{};
    a.vtx_off = L.vtx_off;
    a.reach = reach;
    a.slices = base + kOffSlice;
    a.slice_off = reinterpret_cast<const int64_t *>(base + kOffTileMeta);
    a.slice_bytes = reinterpret_cast<const int32_t *>(base + kOffTileMeta + 8);
    a.items = reinterpret_cast<const TileItem *>(base + kOffTileItems);
    a.item_begin = 0;
    a.item_end = (nsrc + per - 1) / per;
    a.src = src;
    a.src_lo = 0;
    a.src_hi = nsrc;
    a.next_item = L.counter;
    a.acc = L.acc;
    a.nmax = n;
    a.slice_max = (int32_t)TileSlice::bytes(n, slice_pair(m, n));
    a.wait_ns = kDefaultWaitNs;
    a.err = L.err;
    e = launch_tile(cls, a, (int)std::min<int64_t>(grid, a.item_end), smem, stream);
  }
  if (e == cudaSuccess) e = launch_fold(L.acc, bc, 0, n, stream);  // counters -> bc, counters cleared
  return e;
}

// Device address of g_scratch per device, looked up once with that device
// current; g_rows: vertices whose row layout the array's rows and epochs are in,
// as a finished per-source call leaves them (0: none), g_acc: the counters are
// clear. Both are down while a call runs, so a failed call leaves them down.
std::mutex g_mu;
unsigned char *g_addr[64] = {nullptr};
int32_t g_rows[64] = {0};
bool g_acc[64] = {false};

}  // namespace
}  // namespace bcg

extern "C" int bc_begin_free_noalloc(bc_ctx *ctx, const int32_t *R, const int32_t *C, int32_t n, int32_t m,
                                     const int32_t *req_nodes, int32_t n_req, const int32_t *reach, double *bc,
                                     double *time_s) {
  using namespace bcg;
  if (!ctx || !R || !C || !reach || !bc || (n_req > 0 && !req_nodes)) return BCGPU_EINVAL;
  if (n < 3 || m < 0 || n_req < 0) return BCGPU_EINVAL;
  if (n > kMaxVertices || n_req > kMaxVertices) {
    char msg[160];
    std::snprintf(msg, sizeof msg,
                  "bc_begin_free_noalloc: %d vertices / %d sources exceed the fixed scratch limit of %lld each", n,
                  n_req, (long long)kMaxVertices);
    ctx_set_error(ctx, msg);
    return BCGPU_EOVERFLOW;
  }
  int dev = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;  // the context's own events: nothing is created here
  ctx_device_stream(ctx, &dev, &stream, &e0, &e1);
  if (dev < 0 || dev >= 64 || cudaSetDevice(dev) != cudaSuccess) return BCGPU_ECUDA;
  unsigned char *base = nullptr;
  int32_t rows = 0;
  bool acc = false;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_addr[dev]) {
      void *p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_scratch);  // first call on this device
      if (e != cudaSuccess) {
        ctx_set_error(ctx, cudaGetErrorString(e));
        return BCGPU_ECUDA;
      }
      g_addr[dev] = static_cast<unsigned char *>(p);
    }
    base = g_addr[dev];
    rows = g_rows[dev];
    acc = g_acc[dev];
    g_rows[dev] = 0;
    g_acc[dev] = false;
  }
  const Layout L = layout(base, n);
  // the small-BCC kernels where the BCC fits
  const int64_t slice = TileSlice::bytes(n, slice_pair(m, n));
  int cls = m <= INT32_MAX / 4 ? tile_class(n, slice, tile_smem_limit(dev)) : -1;
  size_t smem = 0;
  int grid = 0, sms = 0;
  if (cls >= 0) {
    smem = tile_smem_bytes(cls, n, slice);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
      grid = sms * tile_ctas_per_sm(cls, smem);
    if (grid < 1) cls = -1;
  }
  const bool timing = time_s != nullptr;
  if (timing) cudaEventRecord(e0, stream);
  cudaError_t e = cudaSuccess;
  int h_err = 0;
  for (;;) {
    e = enqueue(base, L, cls, smem, grid, rows != n, !acc, R, C, n, m, req_nodes, n_req, reach, bc, stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h_err, L.err, sizeof(int), cudaMemcpyDeviceToHost, stream);
    if (timing) cudaEventRecord(e1, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (cls >= 0) rows = 0;
    if (e != cudaSuccess || cls < 0 || (h_err != kDevWorkspace && h_err != kDevOverflow)) break;
    cls = -1;  // deeper, or with more paths, than the small-BCC kernels hold
    acc = false;
  }
  if (timing) {
    float ms = 0.f;
    if (e == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess) *time_s += ms * 1e-3;
  }
  if (e != cudaSuccess) {
    ctx_set_error(ctx, cudaGetErrorString(e));
    return BCGPU_ECUDA;
  }
  if (h_err != kDevOk) {
    const std::string msg = std::string("bc_begin_free_noalloc: ") +
                            (h_err == kDevBadItem ? "malformed CSR or source list (offsets, neighbour or source ids)"
                                                  : dev_err_text(h_err));
    ctx_set_error(ctx, msg.c_str());
    return dev_err_status(h_err);
  }
  std::lock_guard<std::mutex> lock(g_mu);
  g_rows[dev] = cls < 0 ? n : 0;
  g_acc[dev] = true;
  return BCGPU_OK;
}
