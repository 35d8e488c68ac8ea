// Stable counting sort of particles by cell (countingsort, pic2d.f90:1303-1329).
//
// The reference histograms the cell keys, turns the histogram into
// allocations by an exclusive scan, and scatters each particle to the next
// free slot of its cell in array order, which makes the sort stable. On the
// GPU the same permutation comes from:
//   1. a histogram of the dense cell keys (warp-aggregated atomics) and an
//      exclusive scan -> per-cell counts and offsets (ptlalloc);
//   2. a least-significant-digit radix sort of (key, index) pairs, up to 9 bits
//      per pass; every pass is a stable multisplit (per-block digit histograms,
//      a device-wide scan in digit-major order, and a scatter that ranks equal
//      digits by warp match + per-warp counters in array order), so the final
//      index order is exactly the stable order by cell;
//   3. a gather of every particle array through that permutation.
#pragma once
#include "device_common.cuh"
#include "kernels_push.cuh"

namespace pbd {

// --------------------------------------------------------------- scan
constexpr int SCAN_BT = 256, SCAN_IPT = 16, SCAN_TILE = SCAN_BT * SCAN_IPT;

// In-place exclusive scan of buf[0, SCAN_TILE) by a block of SCAN_BT threads
// (the values stored, a barrier passed); ws holds SCAN_BT/32 + 1 ints. Returns
// the chunk's total to every thread.
__device__ __forceinline__ int32_t block_scan_excl(int32_t* buf, int32_t* ws) {
  const int t = threadIdx.x;
  int32_t local = 0;
#pragma unroll
  for (int k = 0; k < SCAN_IPT; ++k) {
    const int32_t x = buf[t * SCAN_IPT + k];
    buf[t * SCAN_IPT + k] = local;
    local += x;
  }
  // block-wide exclusive scan of the per-thread totals
  int32_t inc = local;
  const unsigned lane = lane_id();
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t y = __shfl_up_sync(FULL, inc, d);
    if (lane >= (unsigned)d) inc += y;
  }
  if (lane == 31) ws[t >> 5] = inc;
  __syncthreads();
  if (t < 32) {
    int32_t w = t < SCAN_BT / 32 ? ws[t] : 0;
    int32_t wi = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int32_t y = __shfl_up_sync(FULL, wi, d);
      if (lane >= (unsigned)d) wi += y;
    }
    if (t < SCAN_BT / 32) ws[t] = wi - w;
    if (t == SCAN_BT / 32 - 1) ws[SCAN_BT / 32] = wi;
  }
  __syncthreads();
  const int32_t excl = ws[t >> 5] + inc - local;
#pragma unroll
  for (int k = 0; k < SCAN_IPT; ++k) buf[t * SCAN_IPT + k] += excl;
  __syncthreads();
  return ws[SCAN_BT / 32];
}

// Exclusive scan of each SCAN_TILE chunk of in[] into out[] (in may equal
// out); chunk totals to sums[].
static __global__ void __launch_bounds__(SCAN_BT) k_scan_local(const int32_t* in, int32_t* out, int64_t n,
                                                              int32_t* sums) {
  __shared__ int32_t buf[SCAN_TILE];
  __shared__ int32_t ws[SCAN_BT / 32 + 1];
  const int t = threadIdx.x;
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
#pragma unroll
  for (int k = 0; k < SCAN_IPT; ++k) {
    const int64_t i = base + k * SCAN_BT + t;
    buf[k * SCAN_BT + t] = i < n ? in[i] : 0;
  }
  __syncthreads();
  const int32_t total = block_scan_excl(buf, ws);
  if (t == 0) sums[blockIdx.x] = total;
#pragma unroll
  for (int k = 0; k < SCAN_IPT; ++k) {
    const int64_t i = base + k * SCAN_BT + t;
    if (i < n) out[i] = buf[k * SCAN_BT + t];
  }
}

static __global__ void k_scan_add(int32_t* data, int64_t n, const int32_t* sums) {
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
  const int32_t add = sums[blockIdx.x];
  for (int k = threadIdx.x; k < SCAN_TILE; k += blockDim.x) {
    const int64_t i = base + k;
    if (i < n) data[i] += add;
  }
}

// ------------------------------------------------------------ histogram
// keys[i] = dense cell of particle i (ix*my + iy); counts[key] += 1.
static __global__ void k_cell_keys(const uint32_t* cell, int64_t n, int my, int32_t* keys, int32_t* counts) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool ok = i < n;
  int key = -1;
  if (ok) {
    const uint32_t w = cell[i];
    key = cw_ix(w) * my + cw_iy(w);
    if (keys) keys[i] = key;
  }
  const unsigned peers = __match_any_sync(FULL, key);
  if (ok && (lane_id() == (unsigned)(__ffs(peers) - 1))) atomicAdd(&counts[key], __popc(peers));
}

// Sort of an array in which every cell's particles form one contiguous run
// (concatenated cell-sorted pieces with disjoint cells, e.g. a slab's own
// particles followed by its ghost bands): k_cell_runs counts the run starts
// of each cell and records the position of one, k_runs_ok flags a cell with
// more than one run, and k_run_scatter moves each particle to
// offset(cell) + (its index - the run start), the stable sort's position.
static __global__ void k_cell_runs(const uint32_t* cell, int64_t n, int my, int32_t* nruns, int32_t* runstart) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t w = cell[i];
    const int key = cw_ix(w) * my + cw_iy(w);
    int prev = -1;
    if (i > 0) {
      const uint32_t v = cell[i - 1];
      prev = cw_ix(v) * my + cw_iy(v);
    }
    if (key != prev) {
      atomicAdd(&nruns[key], 1);
      runstart[key] = (int32_t)i;
    }
  }
}

static __global__ void k_runs_ok(const int32_t* nruns, int64_t ncells, int* flag) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += (int64_t)gridDim.x * blockDim.x)
    if (nruns[c] > 1) atomicOr(flag, 1);
}

template <class T>
__global__ void k_run_scatter(int64_t n, int my, const int32_t* off, const int32_t* runstart, const uint32_t* ci,
                              Comps<T> in, const int32_t* pidi, uint32_t* co, Comps<T> out, int32_t* pido) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t w = ci[i];
    const int key = cw_ix(w) * my + cw_iy(w);
    const int64_t d = (int64_t)off[key] + (i - runstart[key]);
    co[d] = w;
    put_part(out, d, get_part(in, i));
    if (pido) pido[d] = pidi[i];
  }
}

// Histogram of caller-provided keys, flagging keys outside [0, ncells).
static __global__ void k_key_hist(const int32_t* keys, int64_t n, int32_t ncells, int32_t* counts, int* status) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool ok = i < n;
  int key = -1;
  if (ok) {
    key = keys[i];
    if (key < 0 || key >= ncells) {
      atomicOr(status, 8);
      key = -2;
    }
  }
  const unsigned peers = __match_any_sync(FULL, key);
  if (ok && key >= 0 && (lane_id() == (unsigned)(__ffs(peers) - 1))) atomicAdd(&counts[key], __popc(peers));
}

// ----------------------------------------------------------- radix sort
constexpr int RB = 256, RIPT = 16, RTILE = RB * RIPT, RWARPS = RB / 32;
constexpr int RBITS = 9, RBINS = 1 << RBITS;  // digits of at most 9 bits: 18-bit keys in two passes

// Per-block histogram of one digit, written digit-major: hist[d * nblocks + b].
static __global__ void __launch_bounds__(RB) k_radix_up(const int32_t* keys, int64_t n, int shift, int bits,
                                                        int32_t* hist, int nblocks) {
  __shared__ int32_t h[RBINS];
  const int t = threadIdx.x, bins = 1 << bits;
  for (int d = t; d < bins; d += RB) h[d] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * RTILE;
#pragma unroll 4
  for (int k = 0; k < RIPT; ++k) {
    const int64_t i = base + k * RB + t;
    const int d = i < n ? ((keys[i] >> shift) & (bins - 1)) : RBINS;
    const unsigned peers = __match_any_sync(FULL, d);
    if (d < RBINS && lane_id() == (unsigned)(__ffs(peers) - 1)) atomicAdd(&h[d], __popc(peers));
  }
  __syncthreads();
  for (int d = t; d < bins; d += RB) hist[(int64_t)d * nblocks + blockIdx.x] = h[d];
}

// Second half of an exclusive scan of n values whose chunks of SCAN_TILE are scanned (k_scan_local;
// totals in sums): every block adds the totals before its chunk.
static __global__ void __launch_bounds__(SCAN_BT) k_scan_prefix(int32_t* data, int64_t n, const int32_t* sums) {
  __shared__ int32_t ws[SCAN_BT / 32];
  int32_t add = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += SCAN_BT) add += sums[k];
  add = __reduce_add_sync(FULL, add);
  if (lane_id() == 0) ws[threadIdx.x >> 5] = add;
  __syncthreads();
  add = 0;
#pragma unroll
  for (int k = 0; k < SCAN_BT / 32; ++k) add += ws[k];
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
#pragma unroll 4
  for (int k = threadIdx.x; k < SCAN_TILE; k += SCAN_BT)
    if (base + k < n) data[base + k] += add;
}

// Stable scatter of one digit. Warp w owns the contiguous index range
// [base + w*32*RIPT, base + (w+1)*32*RIPT), item k of lane l at offset k*32 + l,
// so (warp, item, lane) order is array order. The block's pairs are put in digit
// order in shared memory first and stored from there, so that a warp's stores fall into a
// few runs instead of 32 places, and 9-bit digits take two passes where 8 took three: 5 M keys of
// 131 thousand cells, three passes of 65 us stored straight, two of 47 us so (bound by the
// ranking: 16 warp matches in a row).
// kout null: the last pass, only the values are wanted.
static __global__ void __launch_bounds__(RB) k_radix_down(const int32_t* kin, const int32_t* vin, int64_t n, int shift,
                                                          int bits, const int32_t* hist_off, int nblocks,
                                                          int32_t* kout, int32_t* vout) {
  __shared__ uint16_t cnt[RWARPS][RBINS];
  __shared__ int32_t start[RBINS], gofs[RBINS];
  __shared__ int32_t skey[RTILE], sval[RTILE];
  __shared__ int32_t ws[RWARPS];
  const int t = threadIdx.x, w = t >> 5, bins = 1 << bits;
  const unsigned lane = lane_id(), lt = lanemask_lt();
  for (int e = t; e < RWARPS * RBINS / 2; e += RB) reinterpret_cast<uint32_t*>(&cnt[0][0])[e] = 0u;
  __syncthreads();
  const int64_t block0 = (int64_t)blockIdx.x * RTILE, base = block0 + (int64_t)w * 32 * RIPT;
  int32_t key[RIPT], val[RIPT];
  int pos[RIPT];
#pragma unroll
  for (int k = 0; k < RIPT; ++k) {
    const int64_t i = base + k * 32 + lane;
    key[k] = i < n ? kin[i] : 0;
    val[k] = i < n ? (vin ? vin[i] : (int32_t)i) : 0;
  }
#pragma unroll
  for (int k = 0; k < RIPT; ++k) {
    const bool ok = base + k * 32 + lane < n;
    const int d = ok ? ((key[k] >> shift) & (bins - 1)) : RBINS;
    const unsigned peers = __match_any_sync(FULL, d);
    const int before = ok ? cnt[w][d] : 0;
    __syncwarp();
    if (ok && (peers & lt) == 0) cnt[w][d] = (uint16_t)(before + __popc(peers));
    __syncwarp();
    pos[k] = before + __popc(peers & lt);
  }
  __syncthreads();
  // bins 2t and 2t + 1: each warp's first place in the bin, and the bin's in the block
  int tot[2] = {0, 0};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int d = 2 * t + h;
    if (d < bins)
#pragma unroll
      for (int ww = 0; ww < RWARPS; ++ww) {
        const int c = cnt[ww][d];
        cnt[ww][d] = (uint16_t)tot[h];
        tot[h] += c;
      }
  }
  int inc = tot[0] + tot[1];
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int y = __shfl_up_sync(FULL, inc, s);
    if ((int)lane >= s) inc += y;
  }
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  int first = inc - tot[0] - tot[1];
#pragma unroll
  for (int k = 0; k < RWARPS; ++k) first += k < w ? ws[k] : 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int d = 2 * t + h;
    if (d < bins) {
      start[d] = first;
      gofs[d] = hist_off[(int64_t)d * nblocks + blockIdx.x] - first;
    }
    first += tot[0];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < RIPT; ++k)
    if (base + k * 32 + lane < n) {
      const int d = (key[k] >> shift) & (bins - 1);
      const int p = start[d] + cnt[w][d] + pos[k];
      skey[p] = key[k];
      sval[p] = val[k];
    }
  __syncthreads();
  const int m = (int)min((int64_t)RTILE, n - block0);
  for (int i = t; i < m; i += RB) {
    const int32_t kk = skey[i];
    const int32_t p = gofs[(kk >> shift) & (bins - 1)] + i;
    if (kout) kout[p] = kk;
    vout[p] = sval[i];
  }
}

// ----------------------------------------------------------------- gather
template <class T>
__global__ void k_gather(const int32_t* perm, int64_t n, const uint32_t* ci,
                              Comps<T> in, const int32_t* pidi, uint32_t* co, Comps<T> out, int32_t* pido) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
    const int32_t s = perm[j];
    co[j] = ci[s];
    put_part(out, j, get_part(in, s));
    if (pido) pido[j] = pidi[s];
  }
}

// Tile ranges from cell offsets: tile t starts at cell (t / tpc)*my + (t % tpc)*ty.
static __global__ void k_tile_off(const int32_t* off, int ntiles, int tpc, int ty, int my, int32_t n,
                           int32_t* tile_off) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t > ntiles) return;
  if (t == ntiles) {
    tile_off[t] = n;
    return;
  }
  const int ix = t / tpc;
  tile_off[t] = off[(int64_t)ix * my + (int64_t)(t - ix * tpc) * ty];
}

// Equal-count partition of positions (particles not sorted by cell).
static __global__ void k_tile_off_uniform(int ntiles, int64_t n, int32_t* tile_off) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t <= ntiles) tile_off[t] = (int32_t)(n * t / ntiles);
}

}  // namespace pbd

namespace pbd {

// ------------------------------------------------------- fused counting sort
// When the particles were sorted by cell before the push, a particle of tile T
// (a run of cells of one column) lands in T's window: the cells adjacent to T.
// The push counts the new cells per (tile, window bin); with those counts the
// stable counting sort needs no radix passes:
//   count(cell) = sum over the tiles whose window holds the cell,
//   slot(particle) = offset(cell) + [particles of earlier tiles in the cell]
//                  + [earlier particles of its own tile in the cell],
// where "earlier" is array order, i.e. tile order then position in the tile.

struct FusedSortParams {
  int mx, my, ybc, ty, tpc, ntiles, nb;
  const int32_t* tilecnt;  // [ntiles][nb] from the push
  int32_t* counts;         // [mx*my + 1] per-cell counts (last entry 0)
  int32_t* off;            // exclusive scan of counts
  int32_t* base;           // [ntiles][nb] first slot of each (tile, bin)
  int32_t* sums;           // batched: the chunks' totals, then their exclusive scan
};

// The (tile, bin) entries of a cell: the tiles whose windows hold it are those of
// columns cx - 1, cx, cx + 1 (wrapped) and of the tile rows of rows cy - 1, cy, cy + 1
// (wrapped, or none beyond a wall). Entry (i, j), i and j in tile order, is at col[i] +
// row[j] of the [ntiles][nb] tables; a tile row that repeats an earlier one has row < 0. No
// arrays indexed at run time and two divisions a cell: with the tiles searched for one by one, as
// edge cells used to be, every warp of a 64-row column waited for its two edge cells
// (counts 10.6 us and offsets 12.2 us on 64x64 cells).
struct CellEntries {
  int64_t col[3];
  int row[3];
};
__device__ __forceinline__ CellEntries cell_entries(const FusedSortParams& a, int cx, int cy) {
  CellEntries e;
  // columns in increasing order; bin column 1 for the cell's own, 0 for the column
  // after the cell's (the cell is before it), 2 for the column before it
  const int xm = cx == 0 ? a.mx - 1 : cx - 1, xp = cx == a.mx - 1 ? 0 : cx + 1;
  const int64_t tn = (int64_t)a.tpc * a.nb;
  const int w = a.ty + 2;
  const int64_t em = xm * tn + 2 * w, e0 = cx * tn + w, ep = xp * tn;
  const bool first = cx == 0, last = cx == a.mx - 1;  // order: 0 1 mx-1, or 0 mx-2 mx-1
  e.col[0] = first ? e0 : (last ? ep : em);
  e.col[1] = first ? ep : (last ? em : e0);
  e.col[2] = first ? em : (last ? e0 : ep);
  const int t0 = cy / a.ty, r0 = cy - t0 * a.ty;
  const bool top = cy == a.my - 1;
  // tile row and window row (cy - y0 + 1, wrapped) of the neighbour rows' tiles
  int tm = r0 > 0 ? t0 : t0 - 1, bm = cy - tm * a.ty + 1;
  int tp = (r0 < a.ty - 1 && !top) ? t0 : t0 + 1, bp = cy - tp * a.ty + 1;
  if (cy == 0) {
    tm = a.ybc == 0 ? a.tpc - 1 : t0;
    bm = cy - tm * a.ty + 1 + (a.ybc == 0 ? a.my : 0);
  }
  if (top) {
    tp = a.ybc == 0 ? 0 : t0;
    bp = cy - tp * a.ty + 1 - (a.ybc == 0 ? a.my : 0);
  }
  const int vm = tm * a.nb + bm, v0 = t0 * a.nb + r0 + 1, vp = tp * a.nb + bp;
  // in increasing order of the tile row: wrapped rows come last (row 0's) or first (row my - 1's)
  const bool mlast = tm > t0, pfirst = tp < t0;
  const int um = tm == t0 ? -1 : vm, up = (tp == t0 || (tp == tm && um >= 0)) ? -1 : vp;
  e.row[0] = pfirst ? up : (mlast ? v0 : um);
  e.row[1] = pfirst ? um : (mlast ? up : v0);
  e.row[2] = pfirst ? v0 : (mlast ? um : up);
  return e;
}

// (tilecnt by plain loads, not __ldg: k_fused_tables starts while the push still writes it, so that it is not
// read-only for the kernel's lifetime, and a non-coherent load may be moved above the wait for the push.)
__device__ __forceinline__ int32_t fused_count(const FusedSortParams& a, int c) {
  const int cx = c / a.my, cy = c - cx * a.my;
  const CellEntries e = cell_entries(a, cx, cy);
  int32_t v[9], s = 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) v[k] = e.row[k % 3] >= 0 ? a.tilecnt[e.col[k / 3] + e.row[k % 3]] : 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) s += v[k];
  return s;
}

// First slots of the (tile, bin) entries of cell c, whose particles start at `o`: a running sum in tile order.
__device__ __forceinline__ void fused_slots(const FusedSortParams& a, int c, int32_t o) {
  const int cx = c / a.my, cy = c - cx * a.my;
  const CellEntries e = cell_entries(a, cx, cy);
  int32_t v[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) v[k] = e.row[k % 3] >= 0 ? a.tilecnt[e.col[k / 3] + e.row[k % 3]] : 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    if (e.row[k % 3] >= 0) a.base[e.col[k / 3] + e.row[k % 3]] = o;
    o += v[k];
  }
}

// The fused sort's tables. Chunks of CS_TILE cells: the cell counts and their exclusive scan
// within the chunk (chunk_counts), then, with the particles before the chunk known, the cells'
// offsets, each (tile, bin)'s first slot (the offset plus the cell's particles in
// earlier tiles) and each tile's position range (chunk_tables).
//
// Up to CS_MAXCHUNKS chunks one launch does both (k_fused_tables): every block leaves its chunk's
// total with a mark in `words` and adds up those before its own, which are a few KB in L2.
// A block that has waited long enough counts the missing chunk's cells itself, so no
// order of the blocks is assumed.
// Latency-bound: two launches took 4.5 + 6.4 us and the gap between them on 128x128 cells, one
// 8.9 us; the step 57.0 -> 55.1 us there, 36.8 -> 33.4 us on 64x64 cells, 74.3 -> 71.3 us on
// 193x131. Beyond, k_counts_scan and k_fused_offsets
// with the totals scanned between them: there a block's sum over all the totals before it would grow with the
// square of the chunks. Chunks of 1024 cells so that 131 thousand cells still fill 128 blocks.
constexpr int CS_BT = 256, CS_IPT = 4, CS_TILE = CS_BT * CS_IPT;
constexpr int CS_MAXCHUNKS = 8192;
constexpr int CS_POLLS = 1 << 16;

struct ChunkSmem {
  int32_t buf[CS_TILE];  // the chunk's counts, then their scan
  int32_t ws[CS_BT / 32];
};

// Counts and their scan within the chunk (in sm.buf); the chunk's total, in the last thread.
__device__ __forceinline__ int32_t chunk_counts(const FusedSortParams& a, int64_t chunk, ChunkSmem& sm) {
  int32_t(&buf)[CS_TILE] = sm.buf;
  const int t = threadIdx.x;
  const int64_t ncells = (int64_t)a.mx * a.my, base = chunk * CS_TILE;
#pragma unroll
  for (int k = 0; k < CS_IPT; ++k) {
    const int64_t c = base + k * CS_BT + t;
    const int32_t v = c < ncells ? fused_count(a, (int)c) : 0;
    buf[k * CS_BT + t] = v;
    if (c <= ncells) a.counts[c] = v;
  }
  __syncthreads();
  int32_t v[CS_IPT], s = 0;
#pragma unroll
  for (int k = 0; k < CS_IPT; ++k) {
    v[k] = s;
    s += buf[t * CS_IPT + k];
  }
  int32_t inc = s;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t y = __shfl_up_sync(FULL, inc, d);
    if ((int)lane_id() >= d) inc += y;
  }
  if (lane_id() == 31) sm.ws[t >> 5] = inc;
  __syncthreads();
  int32_t before = 0;
#pragma unroll
  for (int k = 0; k < CS_BT / 32; ++k) before += k < (t >> 5) ? sm.ws[k] : 0;
  const int32_t excl = before + inc - s;
#pragma unroll
  for (int k = 0; k < CS_IPT; ++k) buf[t * CS_IPT + k] = excl + v[k];
  __syncthreads();
  return before + inc;
}

// The tables of cell c, whose particles start at `o` (c = ncells: the end).
__device__ __forceinline__ void chunk_tables(const FusedSortParams& a, int64_t c, int32_t o, int32_t* tile_off) {
  a.off[c] = o;
  if (c == (int64_t)a.mx * a.my) {
    tile_off[a.ntiles] = o;
    return;
  }
  const int cx = (int)c / a.my, cy = (int)c - cx * a.my;
  if (cy % a.ty == 0) tile_off[cx * a.tpc + cy / a.ty] = o;
  fused_slots(a, (int)c, o);
}

// words: [0] blocks done, then a word per chunk (its total, marked in bit 32);
// all zero before, and after.
static __global__ void __launch_bounds__(CS_BT) k_fused_tables(FusedSortParams a, unsigned long long* words,
                                                               int32_t* tile_off) {
  __shared__ ChunkSmem sm;
  __shared__ int32_t part[CS_BT / 32];
  __shared__ int done;
  cudaGridDependencySynchronize();
  const int t = threadIdx.x, chunk = blockIdx.x;
  volatile unsigned long long* totals = words + 1;
  const int32_t total = chunk_counts(a, chunk, sm);
  if (t == CS_BT - 1) totals[chunk] = (1ull << 32) | (unsigned)total;
  const int64_t ncells = (int64_t)a.mx * a.my, base = (int64_t)chunk * CS_TILE;
  int32_t before = 0;
  for (int k = t; k < chunk; k += CS_BT) {
    unsigned long long v = totals[k];
    for (int polls = 0; !(v >> 32) && polls < CS_POLLS; ++polls) v = totals[k];
    if (v >> 32) {
      before += (int32_t)v;
    } else {
      const int64_t c0 = (int64_t)k * CS_TILE, c1 = min(c0 + CS_TILE, ncells);
      for (int64_t c = c0; c < c1; ++c) before += fused_count(a, (int)c);
    }
  }
  before = __reduce_add_sync(FULL, before);
  if (lane_id() == 0) part[t >> 5] = before;
  __syncthreads();
  before = 0;
#pragma unroll
  for (int k = 0; k < CS_BT / 32; ++k) before += part[k];
#pragma unroll
  for (int k = 0; k < CS_IPT; ++k) {
    const int64_t c = base + k * CS_BT + t;
    if (c <= ncells) chunk_tables(a, c, before + sm.buf[k * CS_BT + t], tile_off);
  }
  // (not earlier: the ranking's waiting blocks would take the field solve's places, 68 -> 78 us a step of sparse beams)
  cudaTriggerProgrammaticLaunchCompletion();
  // Every block has left its total and read the others' once all are counted: the last one clears them. The
  // barrier above puts this block's store and reads before thread 0's first fence, and the fences put
  // them before its count and every other block's before the clearing: a total that
  // landed after the zero of its word would be taken for one of the next launch.
  if (t == 0) {
    __threadfence();
    done = (int)atomicAdd(&words[0], 1ull);
    __threadfence();
  }
  __syncthreads();
  if (done != (int)gridDim.x - 1) return;
  for (int k = t; k < (int)gridDim.x + 1; k += CS_BT) words[k] = 0ull;
}

static __global__ void __launch_bounds__(CS_BT) k_counts_scan(FusedSortParams a, int32_t* sums) {
  __shared__ ChunkSmem sm;
  const int64_t ncells = (int64_t)a.mx * a.my, base = (int64_t)blockIdx.x * CS_TILE;
  const int32_t total = chunk_counts(a, blockIdx.x, sm);
#pragma unroll
  for (int k = 0; k < CS_IPT; ++k) {
    const int64_t c = base + k * CS_BT + threadIdx.x;
    if (c <= ncells) a.off[c] = sm.buf[k * CS_BT + threadIdx.x];
  }
  if (threadIdx.x == CS_BT - 1) sums[blockIdx.x] = total;
}

// `sums`: prefix sums of the chunks' totals.
static __global__ void __launch_bounds__(CS_BT) k_fused_offsets(FusedSortParams a, const int32_t* sums,
                                                                int32_t* tile_off) {
  const int64_t ncells = (int64_t)a.mx * a.my, base = (int64_t)blockIdx.x * CS_TILE;
  const int32_t prefix = sums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < CS_IPT; ++k) {
    const int64_t c = base + k * CS_BT + threadIdx.x;
    if (c <= ncells) chunk_tables(a, c, a.off[c] + prefix, tile_off);
  }
}

// Batched domains: the tables in three launches (grid row blockIdx.y = domain), the chunks'
// totals scanned between (k_scan_batched).
static __global__ void __launch_bounds__(CS_BT) k_fused_counts_batched(const FusedSortParams* d) {
  __shared__ FusedSortParams a;
  __shared__ ChunkSmem sm;
  if (threadIdx.x == 0) a = d[blockIdx.y];
  __syncthreads();
  const int64_t ncells = (int64_t)a.mx * a.my;
  for (int64_t chunk = blockIdx.x; chunk * CS_TILE <= ncells; chunk += gridDim.x) {
    const int32_t total = chunk_counts(a, chunk, sm);
    if (threadIdx.x == CS_BT - 1) a.sums[chunk] = total;
#pragma unroll
    for (int k = 0; k < CS_IPT; ++k) {
      const int64_t c = chunk * CS_TILE + k * CS_BT + threadIdx.x;
      if (c <= ncells) a.off[c] = sm.buf[k * CS_BT + threadIdx.x];
    }
    __syncthreads();
  }
}

static __global__ void k_fused_base_batched(const FusedSortParams* d) {
  __shared__ FusedSortParams a;
  if (threadIdx.x == 0) a = d[blockIdx.y];
  __syncthreads();
  const int ncells = a.mx * a.my;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c <= ncells; c += gridDim.x * blockDim.x) {
    const int32_t o = a.off[c] + a.sums[c / CS_TILE];
    a.off[c] = o;
    if (c < ncells) fused_slots(a, c, o);
  }
}

template <class T>
struct ScatterParams {
  int mx, my, ybc, ty, tpc, nb;
  const int32_t* tile_off;  // position ranges of the tiles (those the push used)
  const int32_t* base;      // [ntiles][nb]
  const uint32_t* ci;       // the pushed particles' cell words
  int32_t* perm;            // sorted slot -> element of ci
};

constexpr int SC_MAXNB = 3 * (64 + 2) + 1;  // window bins of the largest tile, plus a sentinel

// ------------------------------------------------- permutation-only sort
// The stable ranking of a tile's particles by new cell (warp match_any +
// per-warp counters, array order), from the cell words only: the
// particle at array element p of the tile gets its sorted slot d, and
// perm[d] = p. The particle data stay where they are; the next push reads
// them through perm (PushParams::src), and a gather (k_gather) applies perm
// when the arrays themselves must be in cell order.
// Chunks of 256 threads x 8 particles: 26.2 M particles 70 us; 256 x 16 75, 256 x 12 76, 512 x 8 75,
// 512 x 4 92, 128 x 16 79 (blocks of 512 would save 1 us of 9 at 1 M).
#ifndef PBPIC_PERM_IPT
#define PBPIC_PERM_IPT 8  // particles per thread in one chunk of the ranking
#endif
constexpr int SP_IPT = PBPIC_PERM_IPT, SP_BT = 256, SP_WARPS = SP_BT / 32, SP_CHUNK = SP_BT * SP_IPT;

// Per-warp bin counts and the block's running ranks of one tile.
struct ScatterSmem {
  int32_t cnt[SP_WARPS][SC_MAXNB];
  int32_t run[SC_MAXNB], sbase[SC_MAXNB];
};

template <class T>
__device__ __forceinline__ void perm_tile(const ScatterParams<T>& a, const int t, ScatterSmem& sm) {
  int32_t(&cnt)[SP_WARPS][SC_MAXNB] = sm.cnt;
  int32_t* perm = a.perm;
  const int ixt = t / a.tpc, y0 = (t - ixt * a.tpc) * a.ty, y1 = min(y0 + a.ty, a.my);
  const int pbeg = a.tile_off[t], pend = a.tile_off[t + 1];
  const int w = threadIdx.x >> 5;
  const unsigned lane = lane_id(), lt = lanemask_lt();
  // the window wraps only for the first and last columns and, with periodic y, the first and last tile rows
  const bool edge = ixt == 0 || ixt == a.mx - 1 || (a.ybc == 0 && (y0 == 0 || y1 == a.my));
  const int nrow = y1 - y0 + 1;  // window rows 0..nrow
  for (int b = threadIdx.x; b < a.nb; b += blockDim.x) {
    sm.run[b] = 0;
    sm.sbase[b] = a.base[(int64_t)t * a.nb + b];
  }
  for (int c0 = pbeg; c0 < pend; c0 += SP_CHUNK) {
    for (int e = threadIdx.x; e < SP_WARPS * SC_MAXNB; e += blockDim.x) (&cnt[0][0])[e] = 0;
    __syncthreads();
    int bin[SP_IPT], pos[SP_IPT];
    uint32_t vc[SP_IPT];
    if (c0 + SP_CHUNK <= pend && !edge) {
      // a whole chunk of a tile whose window does not wrap: each bin straight from the cell steps
#pragma unroll
      for (int k = 0; k < SP_IPT; ++k) vc[k] = a.ci[c0 + w * (32 * SP_IPT) + k * 32 + (int)lane];
#pragma unroll
      for (int k = 0; k < SP_IPT; ++k) {
        const int bx = (int)cw_ix(vc[k]) - ixt + 1, by = (int)cw_iy(vc[k]) - y0 + 1;
        bin[k] = ((unsigned)bx <= 2u && (unsigned)by <= (unsigned)nrow) ? bx * (a.ty + 2) + by : a.nb;
      }
    } else {
#pragma unroll
      for (int k = 0; k < SP_IPT; ++k) {  // every load of the chunk before the ranking
        const int p = c0 + w * (32 * SP_IPT) + k * 32 + (int)lane;
        vc[k] = p < pend ? a.ci[p] : 0u;
      }
#pragma unroll
      for (int k = 0; k < SP_IPT; ++k) {
        const int p = c0 + w * (32 * SP_IPT) + k * 32 + (int)lane;
        int b = a.nb;  // sentinel: beyond the tile
        if (p < pend) {
          b = window_bin(cw_ix(vc[k]), cw_iy(vc[k]), ixt, y0, y1, a.ty, a.mx, a.my, a.ybc);
          if (b < 0) b = a.nb;  // cannot happen: the push kept every particle in its window
        }
        bin[k] = b;
      }
    }
#pragma unroll
    for (int k = 0; k < SP_IPT; ++k) {
      const int b = bin[k];
      const unsigned peers = __match_any_sync(FULL, b);
      const int before = cnt[w][b];
      __syncwarp();
      if ((peers & lt) == 0) cnt[w][b] = before + __popc(peers);
      __syncwarp();
      pos[k] = before + __popc(peers & lt);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < a.nb; b += blockDim.x) {
      int32_t r = sm.run[b];
#pragma unroll
      for (int ww = 0; ww < SP_WARPS; ++ww) {
        const int32_t c = cnt[ww][b];
        cnt[ww][b] = r;
        r += c;
      }
      sm.run[b] = r;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SP_IPT; ++k) {
      if (bin[k] < a.nb) {
        const int p = c0 + w * (32 * SP_IPT) + k * 32 + (int)lane;
        perm[(int64_t)sm.sbase[bin[k]] + cnt[w][bin[k]] + pos[k]] = p;
      }
    }
    __syncthreads();
  }
}

template <class T>
__global__ void __launch_bounds__(SP_BT) k_fused_perm(ScatterParams<T> a) {
  __shared__ ScatterSmem sm;
  cudaGridDependencySynchronize();
  perm_tile(a, blockIdx.x, sm);
}

// The identity permutation: arrays already in cell order, read through perm.
static __global__ void k_iota(int32_t* perm, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    perm[i] = (int32_t)i;
}

// Batched permutation-only sort: persistent blocks over the (domain, tile) table.
template <class T>
__global__ void __launch_bounds__(SP_BT)
    k_fused_perm_batched(const ScatterParams<T>* descs, const int2* tiles, int ntiles, int* counter) {
  __shared__ ScatterSmem sm;
  __shared__ ScatterParams<T> a;
  __shared__ int next;
  while (true) {
    if (threadIdx.x == 0) next = atomicAdd(counter, 1);
    __syncthreads();
    const int t = next;
    if (t >= ntiles) break;
    const int2 it = tiles[t];
    if (threadIdx.x == 0) a = descs[it.x];
    __syncthreads();
    perm_tile(a, it.y, sm);
    __syncthreads();
  }
}

}  // namespace pbd

namespace pbd {

// Tile ranges of batched domains (grid row blockIdx.y = domain).
struct TileOffDesc {
  const int32_t* off;  // the domain's cell offsets (global positions)
  int ntiles, tpc, ty, my;
  int32_t end;         // global position after the domain's last particle
  int32_t* tile_off;
};

static __global__ void k_tile_off_batched(const TileOffDesc* d) {
  const TileOffDesc a = d[blockIdx.y];
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t <= a.ntiles; t += gridDim.x * blockDim.x) {
    if (t == a.ntiles) {
      a.tile_off[t] = a.end;
    } else {
      const int ix = t / a.tpc;
      a.tile_off[t] = a.off[(int64_t)ix * a.my + (int64_t)(t - ix * a.tpc) * a.ty];
    }
  }
}

}  // namespace pbd
