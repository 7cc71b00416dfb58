// Host-visible interface of the per-source schedule on chain-contracted BCCs
// (kernels_core.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace bcg {

// One source of the list: a core vertex (local id < n_plain) or a chain vertex.
struct CoreSource {
  int32_t bcc, src;
};

// A core vertex's row: its first arc (from the BCC's first), its arcs, and its
// reach. A short row's arcs are in it, so that one load brings them: far end (-1: none),
// chain * 2 + side (-1: no chain), vertices on the chain. part: a short row's
// chain lengths, a byte each; else the arcs to core vertices, which come first.
constexpr int kCoreShort = 4;
struct __align__(64) CoreRow {
  int32_t e0, deg, part, reach;
  int32_t u[kCoreShort], cid[kCoreShort], pad[4];
};

struct CoreArgs {
  const int64_t *row;       // [n_packed+1] global arc offsets
  const int64_t *vtx_off;   // [n_bcc+1]
  const int32_t *n_plain;   // [n_bcc]
  const int32_t *reach;     // [n_packed]
  const int64_t *chain_off; // [n_bcc+1]
  // contracted rows, at the arc positions of the packed CSR (core_contract)
  const CoreRow *rows;      // core vertices, BCC b's from row_off[b] on
  const int64_t *row_off;   // [n_bcc]
  const int32_t *xcol;      // [n_arcs] far core vertex: the neighbour, or the chain's other end
  const int32_t *xk;        // [n_arcs] vertices on the chain (0: an arc between core vertices)
  const int32_t *xcid;      // [n_arcs] chain * 2 + (the row is the chain's right end)
  const int4 *ctab;         // [n_chains] left end, right end, first vertex (local ids), vertices
  const int32_t *vchain;    // [n_packed] chain of a chain vertex
  const CoreSource *src;
  int64_t lo, hi;                 // places of the list to run
  unsigned long long *next;       // zeroed before each launch
  unsigned long long *acc;        // [n_packed][kAccDigits] fixed-point BC counters (plain.h)
  unsigned char *rec;             // records, CoreShape::rec_bytes per CTA; start zeroed (key 0: unvisited)
  unsigned char *ws;              // the rest of a slot, CoreShape::rest_bytes per CTA
  struct CoreShape {
    int64_t cap;                  // core vertices a slot holds
    int64_t bcap;                 // vertices a bucket holds (chain arcs + 2)
    int64_t ccap;                 // chains a slot holds
    int32_t tcap;                 // levels a slot holds
    int32_t ring;                 // buckets of delayed vertices (longest chain + 3)
    __host__ __device__ int64_t rec_bytes() const { return 32 * cap; }
    __host__ __device__ int64_t smem_bytes() const { return (cap + 127) / 128 * 16; }  // a bit per core vertex
    __host__ __device__ int64_t rest_bytes() const {
      const int64_t b = 20 * ccap + 4 * (2 * cap + ring * bcap) + 8 * ((int64_t)tcap + 3);
      return (b + 255) / 256 * 256;
    }
  } shape;
  int32_t *epochs;                // [slots] key base of the slot's records
  int32_t rescale_exp;
  int *err;
};

constexpr int kCoreMaxChain = 61;  // longest chain: the bucket counters are in shared memory

// Fills rows, xcol, xk, xcid, ctab and vchain of the BCCs with on[b] != 0 from
// the packed CSR and the chain table (both on the device). The chains have to
// be paths of their BCC with two different ends (bcgpu.cu checks).
cudaError_t core_contract(const int64_t *row, const int32_t *col, const int64_t *vtx_off, const int32_t *n_plain,
                          const int32_t *reach, const int64_t *chain_off, const int32_t *chain_start,
                          const int32_t *chain_len, const int32_t *chain_l, const int32_t *chain_r, const int8_t *on,
                          int32_t n_bcc, int64_t n_packed, const int64_t *row_off, CoreRow *rows, int32_t *xcol,
                          int32_t *xk, int32_t *xcid, int4 *ctab, int32_t *vchain, cudaStream_t stream);
// CTAs of `block` threads resident per SM (0: none fits).
int core_ctas_per_sm(int block, const CoreArgs::CoreShape &shape);
// block: 64 ... 512 threads (1024 / block CTAs fit an SM).
cudaError_t launch_core(const CoreArgs &a, int block, int grid, cudaStream_t stream);

}  // namespace bcg
