// subcycle.cu -- the sub-cycle around the short-range kick, on the device:
// Particles::map1 (the half-stream) and Particles::resortParticles (the
// stable counting sort by grid cell that precedes every kick), from
// src/cpu/Particles.cxx:732-758 and :402-488.
#include "subcycle.cuh"

#include <algorithm>

#include "rcb_device.cuh"
#include "chain.cuh"
#include "device_info.cuh"

namespace hsr {

namespace {

// x += pt * v with separate rounding of the product and the sum, as the
// reference's x[i] + prefactor * tau * vx[i] with pt = prefactor * tau.
__global__ void k_stream(float *x, float *y, float *z, const float *vx, const float *vy,
                         const float *vz, int64_t n, float pt) {
  chain_enter();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    x[i] = __fadd_rn(x[i], __fmul_rn(pt, vx[i]));
    y[i] = __fadd_rn(y[i], __fmul_rn(pt, vy[i]));
    z[i] = __fadd_rn(z[i], __fmul_rn(pt, vz[i]));
  }
}

// Cell of a particle (Particles::array_index with lo = 0, hi = ng):
// (floor(x) * ng1 + floor(y)) * ng2 + floor(z); false when outside the box.
__device__ __forceinline__ bool cell_of(float x, float y, float z, int32_t ng0, int32_t ng1,
                                        int32_t ng2, uint32_t *k) {
  const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
  // the reference casts floorf to int; compare in float first so huge or
  // non-finite values land out of the box instead of overflowing the cast
  const bool in = fx >= 0.f && fx < float(ng0) && fy >= 0.f && fy < float(ng1) && fz >= 0.f &&
                  fz < float(ng2);
  if (in) *k = (uint32_t(int(fx)) * uint32_t(ng1) + uint32_t(int(fy))) * uint32_t(ng2) + uint32_t(int(fz));
  return in;
}

// Radix keys: the cell, or Ng when outside the box.
__global__ void k_cell_keys(const float *x, const float *y, const float *z, int64_t n, int32_t ng0,
                            int32_t ng1, int32_t ng2, uint32_t *key, uint32_t *val,
                            unsigned long long *inbox) {
  chain_enter();
  const uint32_t Ng = uint32_t(ng0) * uint32_t(ng1) * uint32_t(ng2);
  unsigned long long c = 0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    uint32_t k;
    const bool in = cell_of(x[i], y[i], z[i], ng0, ng1, ng2, &k);
    if (!in) k = Ng;
    key[i] = k;
    val[i] = uint32_t(i);
    c += in;
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(inbox, c);
}

// ---- stable LSD radix sort of (key, value), 8-bit digits -------------------
constexpr int kRadixThreads = 256;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixPer = 16;
constexpr int kRadixTile = kRadixThreads * kRadixPer;  // elements per block

// hist[d * nblocks + b]: elements of block b with digit d.
__global__ void __launch_bounds__(kRadixThreads)
    k_radix_hist(const uint32_t *key, int64_t n, int shift, int64_t nblocks, int64_t *hist) {
  __shared__ int h[256];
  for (int d = threadIdx.x; d < 256; d += blockDim.x) h[d] = 0;
  __syncthreads();
  const int64_t b = blockIdx.x;
  const int64_t base = b * kRadixTile;
  for (int k = threadIdx.x; k < kRadixTile; k += blockDim.x) {
    const int64_t i = base + k;
    if (i < n) atomicAdd(&h[(key[i] >> shift) & 0xff], 1);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += blockDim.x) hist[int64_t(d) * nblocks + b] = h[d];
}

// Stable scatter: warp w of block b takes the block's elements
// [w * 512, (w + 1) * 512) in order, 32 at a time; ranks among equal digits
// follow the element order (lane order inside a step, warp order across).
__global__ void __launch_bounds__(kRadixThreads)
    k_radix_scatter(const uint32_t *key, const uint32_t *val, int64_t n, int shift,
                    int64_t nblocks, const int64_t *offs, uint32_t *okey, uint32_t *oval) {
  __shared__ int wh[kRadixWarps][256];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int d = lane; d < 256; d += 32) wh[w][d] = 0;
  __syncwarp();
  const int64_t b = blockIdx.x;
  const int64_t base = b * kRadixTile + int64_t(w) * (kRadixTile / kRadixWarps);
  constexpr int kSteps = kRadixTile / kRadixWarps / 32;
  // phase 1: per-warp digit counts
  for (int s = 0; s < kSteps; ++s) {
    const int64_t i = base + s * 32 + lane;
    if (i < n) atomicAdd(&wh[w][(key[i] >> shift) & 0xff], 1);
  }
  __syncthreads();
  // exclusive prefix over warps per digit, plus the block's global offset
  for (int d = threadIdx.x; d < 256; d += blockDim.x) {
    int64_t run = offs[int64_t(d) * nblocks + b];
    for (int q = 0; q < kRadixWarps; ++q) {
      const int c = wh[q][d];
      wh[q][d] = int(run - offs[int64_t(d) * nblocks + b]);
      run += c;
    }
  }
  __syncthreads();
  // phase 2: ranks in order
  for (int s = 0; s < kSteps; ++s) {
    const int64_t i = base + s * 32 + lane;
    const bool ok = i < n;
    const uint32_t k = ok ? key[i] : 0u;
    const int d = ok ? int((k >> shift) & 0xff) : 256 + lane;  // distinct dummy digits
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    const int leader = __ffs(peers) - 1;
    int start = 0;
    if (ok) start = wh[w][d];
    __syncwarp();
    if (ok && lane == leader) wh[w][d] = start + __popc(peers);
    __syncwarp();
    if (ok) {
      const int64_t dst = offs[int64_t(d) * nblocks + b] + start + rank;
      okey[dst] = k;
      oval[dst] = val[i];
    }
  }
}

// ---- counting sort by cell --------------------------------------------------
// A particle's place is its cell's offset plus its rank among the cell's
// particles: six launches, where three radix passes with their scans take 15
// and leave most SMs without a block below a few hundred thousand particles.  A cell's particles arrive in
// any order, so each counts the ones of its cell with a smaller index, which
// makes the sort stable.  Particles outside the box get a pseudo-cell for
// every 32 indices behind the grid's cells, which keeps their order with the
// same rule and no long cell.
constexpr uint32_t kOutRun = 32;       // indices per pseudo-cell
// Longest cell whose ranks are counted: a set with a longer one has paid for both
// sorts.  A whole sub-cycle call less its kick, 2.6 M particles: 1.88 ms counted
// with a cell of 900, 2.04 by both with one of 1100 (1.95 by radix alone); but
// with half of them in cells of 1000 or 1100 2.19 counted and 1.92 by radix, and
// with five cells of 20,000 3.01 and 1.96.  70 thousand, a cell of 1100: 0.39
// counted, 0.45 by radix, 0.50 by both.
constexpr int kMaxOcc = 1024;
constexpr int kCellThreads = 256;
constexpr int kCellPer = 16;
constexpr int kCellTile = kCellThreads * kCellPer;  // cells per block of the scan
constexpr int64_t kMaxTiles = 4096;

// Words of counter: in-box particles, longest cell.
struct CellCount {
  unsigned long long inbox;
  unsigned int longest;
  unsigned int pad;
};

// The half-stream (DRIFT), each particle's cell and its arrival in the cell.
template <bool DRIFT>
__global__ void __launch_bounds__(kCellThreads)
    k_cell_count(KickArrays A, int64_t n, float pt, int32_t ng0, int32_t ng1, int32_t ng2,
                 uint32_t *key, uint32_t *slot, uint32_t *cnt, CellCount *out) {
  chain_enter();
  const uint32_t Ng = uint32_t(ng0) * uint32_t(ng1) * uint32_t(ng2);
  unsigned c = 0, most = 0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    float x = A.f[0][i], y = A.f[1][i], z = A.f[2][i];
    if (DRIFT) {
      A.f[0][i] = x = __fadd_rn(x, __fmul_rn(pt, A.f[3][i]));
      A.f[1][i] = y = __fadd_rn(y, __fmul_rn(pt, A.f[4][i]));
      A.f[2][i] = z = __fadd_rn(z, __fmul_rn(pt, A.f[5][i]));
    }
    uint32_t k;
    const bool in = cell_of(x, y, z, ng0, ng1, ng2, &k);
    if (!in) k = Ng + uint32_t(i) / kOutRun;
    const uint32_t at = atomicAdd(&cnt[k], 1u);
    key[i] = k;
    slot[i] = at;
    c += in;
    most = max(most, at + 1);
  }
  c = __reduce_add_sync(0xffffffffu, c);
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0) {
    if (c) atomicAdd(&out->inbox, (unsigned long long)c);
    if (most > kOutRun) atomicMax(&out->longest, most);
  }
}

__device__ __forceinline__ uint32_t block_sum_u32(uint32_t v, uint32_t *sh) {
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = 0;
  for (int w = 0; w < kCellThreads / 32; ++w) t += sh[w];
  __syncthreads();
  return t;
}

__global__ void __launch_bounds__(kCellThreads)
    k_cell_tiles(const uint32_t *__restrict__ cnt, int64_t ncell, uint32_t *tile) {
  chain_enter();
  __shared__ uint32_t sh[kCellThreads / 32];
  const int64_t base = int64_t(blockIdx.x) * kCellTile;
  uint32_t v = 0;
#pragma unroll
  for (int k = 0; k < kCellPer; ++k) {
    const int64_t i = base + k * kCellThreads + threadIdx.x;
    v += i < ncell ? cnt[i] : 0u;
  }
  v = block_sum_u32(v, sh);
  if (threadIdx.x == 0) tile[blockIdx.x] = v;
}

// Each block adds up the tiles before its own (at most kMaxTiles) instead of
// waiting for a scan of them.
__global__ void __launch_bounds__(kCellThreads)
    k_cell_offsets(const uint32_t *__restrict__ cnt, int64_t ncell,
                   const uint32_t *__restrict__ tile, uint32_t *offs) {
  chain_enter();
  __shared__ uint32_t sh[kCellThreads / 32];
  uint32_t before = 0;
  for (unsigned t = threadIdx.x; t < blockIdx.x; t += kCellThreads) before += tile[t];
  before = block_sum_u32(before, sh);
  const int64_t i0 = int64_t(blockIdx.x) * kCellTile + int64_t(threadIdx.x) * kCellPer;
  uint32_t v[kCellPer], t = 0;
#pragma unroll
  for (int k = 0; k < kCellPer; ++k) {
    v[k] = i0 + k < ncell ? cnt[i0 + k] : 0u;
    t += v[k];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  uint32_t run = before + x - t;
  for (int w = 0; w < warp; ++w) run += sh[w];
#pragma unroll
  for (int k = 0; k < kCellPer; ++k) {
    if (i0 + k < ncell) offs[i0 + k] = run;
    run += v[k];
  }
}

__global__ void k_cell_place(const uint32_t *__restrict__ key, const uint32_t *__restrict__ slot,
                             const uint32_t *__restrict__ offs, int64_t n, const CellCount *c,
                             uint32_t *order) {
  chain_enter();
  if (c->longest > kMaxOcc) return;  // the radix sort follows
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    order[offs[key[i]] + slot[i]] = uint32_t(i);
}

__device__ __forceinline__ void move_particle(const KickArrays &A, const KickArrays &S, int64_t i,
                                              int64_t to) {
  const float x = A.f[0][i], y = A.f[1][i], z = A.f[2][i], vx = A.f[3][i], vy = A.f[4][i],
              vz = A.f[5][i], phi = A.f[7][i];
  const int64_t id = A.id[i];
  const uint16_t mask = A.mask[i];
  S.f[0][to] = x;
  S.f[1][to] = y;
  S.f[2][to] = z;
  S.f[3][to] = vx;
  S.f[4][to] = vy;
  S.f[5][to] = vz;
  S.f[7][to] = phi;
  S.id[to] = id;
  S.mask[to] = mask;
}

// Thread p takes the p-th particle by cell, finds its rank in the cell and
// moves its arrays to their place in the staging copy.
__global__ void k_cell_move(const uint32_t *__restrict__ order, const uint32_t *__restrict__ key,
                            const uint32_t *__restrict__ offs, const uint32_t *__restrict__ cnt,
                            int64_t n, const CellCount *c, KickArrays A, KickArrays S) {
  chain_enter();
  if (c->longest > kMaxOcc) return;
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n;
       p += int64_t(gridDim.x) * blockDim.x) {
    const uint32_t i = order[p], k = key[i];
    const uint32_t lo = offs[k], m = cnt[k];
    uint32_t rank = 0;
    if (m > 1)
      for (uint32_t q = 0; q < m; ++q) rank += order[lo + q] < i;
    move_particle(A, S, i, int64_t(lo) + rank);
  }
}

// The radix sort's permutation applied to the arrays.
__global__ void k_perm_move(const uint32_t *__restrict__ perm, int64_t n, KickArrays A, KickArrays S) {
  chain_enter();
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n;
       p += int64_t(gridDim.x) * blockDim.x)
    move_particle(A, S, perm[p], p);
}

// The staging copy back into the arrays, the masses set to one.
__global__ void k_move_back(KickArrays S, KickArrays A, int64_t n, const CellCount *c) {
  chain_enter();
  if (c && c->longest > kMaxOcc) return;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    move_particle(S, A, i, i);
    A.f[6][i] = 1.0f;
  }
}

inline unsigned grid_of(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  return unsigned(std::max<int64_t>(1, std::min<int64_t>(b, int64_t(sm_count()) * 32)));
}

}  // namespace

cudaError_t launch_stream(float *x, float *y, float *z, const float *vx, const float *vy,
                          const float *vz, int64_t n, float pt, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  launch_chained(k_stream, grid_of(n), 256, 0, s, x, y, z, vx, vy, vz, n, pt);
  return cudaGetLastError();
}

namespace {

// Scratch of a resort: staging copies, then either sort's tables in the same
// space.
struct ResortLayout {
  size_t f[8], id, mask, count, tables, bytes;
  ResortLayout(int64_t n, const int32_t ng[3]) {
    auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
    const size_t m = size_t(std::max<int64_t>(n, 1));
    size_t o = 0;
    for (int i = 0; i < 8; ++i) {
      f[i] = o;
      if (i != 6) o = up(o + m * 4);  // masses are set, not moved
    }
    id = o;
    o = up(o + m * 8);
    mask = o;
    o = up(o + m * 2);
    count = o;
    o = up(o + sizeof(CellCount));
    tables = o;
    // radix sort: keys and values twice, histograms, offsets, scan scratch
    const int64_t h = 256 * std::max<int64_t>((n + kRadixTile - 1) / kRadixTile, 1);
    size_t r = 4 * up(m * 4) + 2 * up(size_t(h) * 8) + up(size_t(scan_tmp_size(h)) * 8);
    // counting sort: keys, slots, order, counts and offsets of the cells, tiles
    if (counted(n, ng))
      r = std::max(r, 3 * up(m * 4) + 2 * up(size_t(cells(n, ng)) * 4) + up(size_t(kMaxTiles) * 4));
    bytes = o + r;
  }
  static int64_t grid_cells(const int32_t ng[3]) { return int64_t(ng[0]) * ng[1] * ng[2]; }
  static int64_t cells(int64_t n, const int32_t ng[3]) {
    return grid_cells(ng) + (n + kOutRun - 1) / kOutRun;
  }
  // The counting sort goes through every cell twice and a radix pass through
  // every particle three times, so a grid of many more cells than particles
  // takes the radix sort (a sub-cycle call less its kick: 0.37 ms counted and
  // 0.45 by radix for 70 thousand particles in 80^3 cells, 0.53 and 0.62 for 300
  // thousand in 128^3, seven cells a particle each; at 27 a particle 0.56 and
  // 0.62: the line is on the safe side); so does one of more than 16 M cells,
  // whose tiles are too many to be added up by each block.
  static bool counted(int64_t n, const int32_t ng[3]) {
    return grid_cells(ng) <= 8 * n && cells(n, ng) <= kMaxTiles * kCellTile;
  }
  KickArrays staged(char *p) const {
    KickArrays k;
    for (int i = 0; i < 8; ++i) k.f[i] = reinterpret_cast<float *>(p + f[i]);
    k.f[6] = nullptr;
    k.id = reinterpret_cast<int64_t *>(p + id);
    k.mask = reinterpret_cast<uint16_t *>(p + mask);
    return k;
  }
};

struct Carve {
  char *p;
  template <typename T>
  T *take(int64_t count) {
    T *q = reinterpret_cast<T *>(p);
    p += (size_t(count) * sizeof(T) + 255) & ~size_t(255);
    return q;
  }
};

}  // namespace

size_t resort_scratch_bytes(int64_t n, const int32_t ng[3]) { return ResortLayout(n, ng).bytes; }

cudaError_t drift_and_resort(int64_t n, const int32_t ng[3], const KickArrays &A, const float *pt,
                             void *scratch, int64_t *n_inbox, cudaStream_t s) {
  *n_inbox = 0;
  if (n <= 0) return cudaSuccess;
  const ResortLayout L(n, ng);
  char *base = static_cast<char *>(scratch);
  const KickArrays S = L.staged(base);
  CellCount *count = reinterpret_cast<CellCount *>(base + L.count);
  CellCount got{};
  cudaError_t e = cudaMemsetAsync(count, 0, sizeof(CellCount), s);
  if (e != cudaSuccess) return e;
  const unsigned grid = grid_of(n);
  if (ResortLayout::counted(n, ng)) {
    const int64_t ncell = ResortLayout::cells(n, ng);
    const unsigned tiles = unsigned((ncell + kCellTile - 1) / kCellTile);
    Carve c{base + L.tables};
    uint32_t *key = c.take<uint32_t>(n), *slot = c.take<uint32_t>(n), *order = c.take<uint32_t>(n);
    uint32_t *cnt = c.take<uint32_t>(ncell), *offs = c.take<uint32_t>(ncell);
    uint32_t *tile = c.take<uint32_t>(kMaxTiles);
    e = cudaMemsetAsync(cnt, 0, size_t(ncell) * 4, s);
    if (e != cudaSuccess) return e;
    if (pt)
      launch_chained(k_cell_count<true>, grid, kCellThreads, 0, s, A, n, *pt, ng[0], ng[1], ng[2],
                     key, slot, cnt, count);
    else
      launch_chained(k_cell_count<false>, grid, kCellThreads, 0, s, A, n, 0.f, ng[0], ng[1], ng[2],
                     key, slot, cnt, count);
    launch_chained(k_cell_tiles, tiles, kCellThreads, 0, s, cnt, ncell, tile);
    launch_chained(k_cell_offsets, tiles, kCellThreads, 0, s, cnt, ncell, tile, offs);
    launch_chained(k_cell_place, grid, 256, 0, s, key, slot, offs, n, count, order);
    launch_chained(k_cell_move, grid, 256, 0, s, order, key, offs, cnt, n, count, A, S);
    launch_chained(k_move_back, grid, 256, 0, s, S, A, n, count);
    e = cudaMemcpyAsync(&got, count, sizeof(got), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    *n_inbox = int64_t(got.inbox);
    if (got.longest <= kMaxOcc) return cudaGetLastError();
    // a cell of more particles: ranks by counting would take too long
    e = cudaMemsetAsync(count, 0, sizeof(CellCount), s);
    if (e != cudaSuccess) return e;
  } else if (pt) {
    e = launch_stream(A.f[0], A.f[1], A.f[2], A.f[3], A.f[4], A.f[5], n, *pt, s);
    if (e != cudaSuccess) return e;
  }
  const int64_t nblocks = (n + kRadixTile - 1) / kRadixTile;
  const int64_t h = 256 * nblocks;
  Carve c{base + L.tables};
  uint32_t *key = c.take<uint32_t>(n), *val = c.take<uint32_t>(n), *key2 = c.take<uint32_t>(n),
           *val2 = c.take<uint32_t>(n);
  int64_t *hist = c.take<int64_t>(h), *offs = c.take<int64_t>(h);
  int64_t *tmp = c.take<int64_t>(scan_tmp_size(h));
  launch_chained(k_cell_keys, grid, 256, 0, s, A.f[0], A.f[1], A.f[2], n, ng[0], ng[1], ng[2], key,
                 val, &count->inbox);
  const uint64_t Ng = uint64_t(ResortLayout::grid_cells(ng));
  int bits = 1;
  while ((uint64_t(1) << bits) <= Ng) ++bits;
  for (int shift = 0; shift < bits; shift += 8) {
    k_radix_hist<<<unsigned(nblocks), kRadixThreads, 0, s>>>(key, n, shift, nblocks, hist);
    e = exclusive_scan_i64(hist, offs, h, nullptr, tmp, s);
    if (e != cudaSuccess) return e;
    k_radix_scatter<<<unsigned(nblocks), kRadixThreads, 0, s>>>(key, val, n, shift, nblocks, offs,
                                                                key2, val2);
    std::swap(key, key2);
    std::swap(val, val2);
  }
  launch_chained(k_perm_move, grid, 256, 0, s, val, n, A, S);
  launch_chained(k_move_back, grid, 256, 0, s, S, A, n, nullptr);
  e = cudaMemcpyAsync(&got, count, sizeof(got), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  *n_inbox = int64_t(got.inbox);
  return cudaGetLastError();
}

}  // namespace hsr
