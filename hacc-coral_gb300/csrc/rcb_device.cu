// rcb_device.cu -- RCB tree, interaction lists and batched work items built on
// the GPU (see rcb_device.cuh for the method).
#include "rcb_device.cuh"
#include "chain.cuh"
#include "device_info.cuh"

#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

namespace hsr {

namespace {

// ---- exactly rounded float helpers: never fused, as the reference rounds ----
__device__ __forceinline__ float fmul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub_(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float smin_(float a, float b) { return (b < a) ? b : a; }
// ((a*a) + (b*b)) + (c*c)
__device__ __forceinline__ float norm2_(float a, float b, float c) {
  return fadd_(fadd_(fmul_(a, a), fmul_(b, b)), fmul_(c, c));
}

__host__ __device__ __forceinline__ int64_t max64(int64_t a, int64_t b) { return a > b ? a : b; }
__host__ __device__ __forceinline__ int64_t min64(int64_t a, int64_t b) { return a < b ? a : b; }

// Exponent of the lowest set bit of a float (INT_MAX for zero, INT_MIN for
// inf/NaN).  A sum of terms that are all multiples of 2^e is exact in double,
// in any order, while the sum of magnitudes stays below 2^(53 + e).
__device__ __forceinline__ int lsb_exp(float t) {
  const uint32_t b = __float_as_uint(t) & 0x7fffffffu;
  if (b == 0) return INT_MAX;
  int e = int(b >> 23);
  if (e == 255) return INT_MIN;
  uint32_t m = b & 0x7fffffu;
  if (e == 0) e = 1;
  else m |= 0x800000u;
  return e - 150 + (__ffs(int(m)) - 1);
}

constexpr int kChunkThreads = 256;  // threads per statistics / partition chunk
constexpr int kChainSteps = 32;     // chain steps before a subtree block jumps pointers
constexpr int kPlainSteps = 4;      // single chain steps before the chunk partition jumps runs

enum { C_NFALLBACK = 2, C_NLEAF = 3, C_NSEG = 4, C_NENT = 5,
       C_PAIRS = 6, C_PADDED = 7, C_NITEMS = 8, C_BIG = 9, C_TDONE1 = 10, C_TDONE2 = 11,
       C_NTIGHT = 12, C_SEGOVF = 13, C_ERR = 15, C_BUCKET = 16, C_FILL = 48,
       C_SUBFB = 80, C_CHAINS = 81, C_TICKET = 82, C_SEQ = 83, C_COUNT = 84 };

// Segments a leaf's walk can leave in its own region of the one-pass walk (8
// bytes each); a leaf with more is walked a second time, its segments placed.
// At most kLocalSegs, and fewer where the regions of every leaf that there can be
// would take more than kWalkBytes (above 262,144 leaves): at a leaf size of 1 or
// 2 the regions would be the largest buffer of all (2 KB a leaf, held as long as
// the tree).
constexpr int kLocalSegs = 256;
constexpr int64_t kWalkBytes = int64_t(512) << 20;
inline int local_segs(int64_t leaves) {
  return int(std::min<int64_t>(kLocalSegs, kWalkBytes / (leaves * int64_t(sizeof(int2)))));
}

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---------------------------------------------------------------------------
// Scan
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;
constexpr int64_t kScanBlock = kScanThreads * kScanPer;

__global__ void __launch_bounds__(kScanThreads)
    k_scan_block(const int64_t *in, int64_t *out, int64_t n, int64_t *bsum, int64_t *total) {
  chain_enter();
  __shared__ int64_t wsum[32];
  const int64_t base = int64_t(blockIdx.x) * kScanBlock + int64_t(threadIdx.x) * kScanPer;
  int64_t v[kScanPer];
  int64_t t = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    v[k] = base + k < n ? in[base + k] : 0;
    t += v[k];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t x = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int64_t w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  const int64_t excl = x - t + (warp > 0 ? wsum[warp - 1] : 0);
  int64_t run = excl;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == kScanThreads - 1) {
    bsum[blockIdx.x] = run;
    if (total) *total = run;  // single-block scans only (the caller passes it then)
  }
}

__global__ void k_scan_add(int64_t *out, int64_t n, const int64_t *boff) {
  chain_enter();
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) out[i] += boff[i / kScanBlock];
}


}  // namespace

int64_t scan_tmp_size(int64_t n) {
  const int64_t nb = (n + kScanBlock - 1) / kScanBlock;
  return nb <= 1 ? 2 : nb + 1 + scan_tmp_size(nb);
}

cudaError_t exclusive_scan_i64(const int64_t *in, int64_t *out, int64_t n, int64_t *total,
                               int64_t *tmp, cudaStream_t s) {
  if (n <= 0) {
    if (total) return cudaMemsetAsync(total, 0, sizeof(int64_t), s);
    return cudaSuccess;
  }
  const int64_t nb = (n + kScanBlock - 1) / kScanBlock;
  launch_chained(k_scan_block, unsigned(nb), kScanThreads, 0, s, in, out, n, tmp,
                 nb == 1 ? total : nullptr);
  if (nb == 1) return cudaGetLastError();
  // scan the block sums in place, then add them
  cudaError_t e = exclusive_scan_i64(tmp, tmp, nb, total, tmp + nb + 1, s);
  if (e != cudaSuccess) return e;
  launch_chained(k_scan_add, unsigned((n + 255) / 256), 256, 0, s, out, n, tmp);
  return cudaGetLastError();
}

namespace {

// ---------------------------------------------------------------------------
// Level kernels
// ---------------------------------------------------------------------------

// Exclusive scan over one block of kScanThreads threads, kScanPer values each
// (v in, out out); returns the block total to every thread.
__device__ __forceinline__ int64_t block_exclusive_scan(const int64_t (&v)[kScanPer],
                                                        int64_t (&out)[kScanPer]) {
  __shared__ int64_t wsum[32];
  int64_t t = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) t += v[k];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t x = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int64_t w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  int64_t run = x - t + (warp > 0 ? wsum[warp - 1] : 0);
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    out[k] = run;
    run += v[k];
  }
  return wsum[31];
}

// Exclusive scans of a and b in place, in one block, for n up to a few blocks'
// worth; the totals into *ta and *tb.  (Two three-kernel scans otherwise.)
constexpr int64_t kScanPairMax = 4 * kScanBlock;
__global__ void __launch_bounds__(kScanThreads)
    k_scan_pair(const int64_t *a, const int64_t *b, int64_t *oa, int64_t *ob, int64_t n,
                int64_t *ta, int64_t *tb) {
  chain_enter();
  int64_t ca = 0, cb = 0;
  for (int64_t base = 0; base < n; base += kScanBlock) {
    const int64_t i0 = base + int64_t(threadIdx.x) * kScanPer;
    int64_t v[kScanPer], o[kScanPer];
    for (int which = 0; which < 2; ++which) {
      const int64_t *in = which ? b : a;
      int64_t *out = which ? ob : oa;
      int64_t &carry = which ? cb : ca;
#pragma unroll
      for (int k = 0; k < kScanPer; ++k) v[k] = i0 + k < n ? in[i0 + k] : 0;
      const int64_t total = block_exclusive_scan(v, o);
#pragma unroll
      for (int k = 0; k < kScanPer; ++k)
        if (i0 + k < n) out[i0 + k] = carry + o[k];
      carry += total;
      __syncthreads();  // the scan's shared sums are reused
    }
  }
  if (threadIdx.x == 0) {
    *ta = ca;
    *tb = cb;
  }
}

__device__ __forceinline__ float key_of(const float4 &p, int d) {
  return d == 0 ? p.x : (d == 1 ? p.y : p.z);
}

// Block-wide exclusive scan of one int per thread.
__device__ __forceinline__ int block_excl_scan(int v, int *sh_warp, int *total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < (int)(blockDim.x >> 5) ? sh_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    sh_warp[lane] = w;
  }
  __syncthreads();
  const int excl = x - v + (warp > 0 ? sh_warp[warp - 1] : 0);
  *total = sh_warp[(blockDim.x >> 5) - 1];
  __syncthreads();
  return excl;
}

// ---------------------------------------------------------------------------
// The levels of large nodes.
//
// A level is five launches: statistics (k_level_stats), left counts
// (k_level_count), left elements (k_part_left), right elements
// (k_part_right) and the long swap chains (k_part_chains), a block per chunk of
// a few thousand elements.  What follows a node's last chunk -- its split decision, the
// scan of its chunks' left counts -- and what follows the level's last chunk --
// the children, their chunks -- is done by the block that finishes last, and
// the level's extent lives in device memory (LevelCtl), so the host launches
// the levels that the particle count calls for and waits once for all of them.
// (Seventeen launches and a synchronisation a level took 100 us a level at
// 32^3 particles and 160 at 128^3.)
// A child small enough for a subtree block becomes a root of k_subtree at
// once, whatever its level, and takes no chunk of the levels below: in a
// clustered set the last halos take several levels more than the rest.
// A level whose centre-of-mass bounds leave a node undecided raises `abort`:
// the launches after it do nothing, and the host runs the certification
// kernels for it and goes on from there.
// ---------------------------------------------------------------------------
struct LevelSpan {
  int32_t level;  // which level this slot describes
  int32_t run;    // 0: no level here (no node is left for the level loop)
  int32_t nb, ne;  // its nodes, subtree roots among them
  int32_t nchunk;  // chunks of the others
  int32_t live;    // the others
  int32_t maxcnt;  // the largest of them
  int32_t pad;
};
constexpr int kCtlLevels = 64;
struct LevelCtl {
  LevelSpan lev[2];    // by level parity
  int32_t abort;       // level + 1 of a level with undecided nodes, or 0
  int32_t nroots;      // subtree roots so far
  int32_t done;        // no node is left for the level loop
  int32_t node_end;    // nodes of all levels
  // the set's range, as bits of floats: largest |w x|, |w y|, |w z|, |w|; smallest and
  // largest w by its bits, sign and all; smallest over the elements of the largest
  // of |w x|, |w y| and |w z|, and smallest |w|, zeros aside.  (Maxima only, of
  // the minima's complements: the block starts as zeros.)
  unsigned range[8];
  unsigned ticket;     // chunks of the level counted
  int32_t next_level;  // the level made last
  int32_t begin[kCtlLevels];  // first node of a level, by level modulo kCtlLevels
};
// A chunk is PT elements a thread of its block: the fewest of 4, 8 and 16 that
// leave at most kLevelBlocks chunks an SM, one wave of blocks.  More elements a
// thread are more dependent loads (a level of 68 thousand elements: 62 us with
// 16, 44 with 4); more blocks than a wave, and the per-block work (reductions,
// tickets) counts twice (the levels of a 1.15 M set: 0.66 ms with 16 or 4, 0.60
// with 8; of 2.6 M: 1.10 ms with 16, 1.31 with 4, 1.13 with 24).
constexpr int64_t kLevelBlocks = 4;
template <int PT>
__host__ __device__ constexpr int32_t chunk_size() { return PT * kChunkThreads; }
template <int PT>
__device__ __forceinline__ int32_t chunks_of(int32_t count) {
  return (count + chunk_size<PT>() - 1) / chunk_size<PT>();
}

// Whether level `level` is to be worked on, and its extent.  (Blocks of its
// statistics may start after another has raised abort for the same level.)
__device__ __forceinline__ bool level_runs(const LevelCtl *ctl, int32_t level, LevelSpan &S,
                                           bool stats = false) {
  S = ctl->lev[level & 1];
  const int32_t a = *reinterpret_cast<const volatile int32_t *>(&ctl->abort);
  return S.run && S.level == level && (a == 0 || (stats && a == level + 1));
}

struct ChunkRange {
  int32_t node, begin, len, local;  // local: first element's position inside the node
};

template <int PT>
__device__ __forceinline__ ChunkRange chunk_range(const DNode *nodes, const int32_t *chunk_node,
                                                  const int32_t *chunk_base, int32_t nb,
                                                  int32_t chunk) {
  ChunkRange r;
  r.node = chunk_node[chunk];
  const DNode &N = nodes[r.node];
  r.local = (chunk - chunk_base[r.node - nb]) * chunk_size<PT>();
  r.begin = N.offset + r.local;
  r.len = min(chunk_size<PT>(), N.count - r.local);
  return r;
}

// Child s (0 left, 1 right) of split node N, as four 16-byte stores.
__device__ __forceinline__ void write_child(DNode &dst, const DNode &N, int s) {
  DNode C;
  C.count = s == 0 ? N.nleft : N.count - N.nleft;
  C.offset = s == 0 ? N.offset : N.offset + N.nleft;
  C.cl = C.cr = 0;
  for (int d = 0; d < 3; ++d) {
    C.xmin[d] = N.xmin[d];
    C.xmax[d] = N.xmax[d];
    C.xc[d] = 0.f;
  }
  C.tdr = 0.f;
  C.split_dim = -1;
  C.nleft = 0;
  static_assert(sizeof(DNode) == 64, "DNode is four 16-byte words");
  const int4 *src = reinterpret_cast<const int4 *>(&C);
  int4 *out = reinterpret_cast<int4 *>(&dst);
#pragma unroll
  for (int w = 0; w < 4; ++w) out[w] = src[w];
}

// Order-preserving map of a float to an unsigned integer.
__device__ __forceinline__ uint32_t f2o(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// ---------------------------------------------------------------------------
// Exact sums of float terms on the FP32 and integer pipes.
//
// With every |t| below 2^(k-2), the sum v = t + 1.5 2^k stays in one binade, so
// its bits count t rounded to multiples of 2^(k-23), h = v - 1.5 2^k is exact,
// and r = t - h (exact, |r| <= 2^(k-24)) goes the same way onto multiples of
// 2^(k-45): t = iv 2^(k-23) + iv2 2^(k-45) with |iv| <= 2^21, |iv2| <= 2^21, and
// what is left (terms with bits below 2^(k-45)) marks the node's sums as
// truncated, by at most half a unit a term.  Sums of the two integers are exact
// in any order.  Eleven single-rate operations a term; shifting each term into
// 128-bit fixed point took more than twice as many, and FP64, and every
// conversion to or from a 64-bit type, runs at a small fraction of that rate on
// this part.  One scale for the three coordinates' terms and one for the masses,
// from the largest of the whole set.
//
// In a set of wide range (one particle a million times heavier than the rest,
// or that much farther away) two integers hold too few bits of the small terms,
// and nearly every centre of mass would be left to the sequential sums.  There a
// third integer, on multiples of 2^(k-67), takes what the second leaves.
// ---------------------------------------------------------------------------
struct SumScale {
  int k;        // the scale's exponent
  float m1, m2;  // 1.5 2^k and 1.5 2^(k-22)
  __device__ __forceinline__ explicit SumScale(unsigned mx) {
    const int e = int(mx >> 23) - 127;  // mx < 2^(e+1); subnormal or zero: -127
    k = max(e + 3, -80);
    m1 = binade(k);
    m2 = binade(k - 22);
  }
  __device__ static __forceinline__ float binade(int e) {  // 1.5 2^e
    return __uint_as_float((unsigned(e + 127) << 23) | 0x400000u);
  }
  __device__ __forceinline__ float m3() const { return binade(k - 44); }
  // terms too large for the scale's arithmetic, infinities and NaN
  __device__ static __forceinline__ bool bad(unsigned mx) { return mx >= (247u << 23); }
};

// Reduced statistics of a set of elements (a node, a warp's share).
struct alignas(16) NodeAcc {
  // sums (x, y, z, m) of iv and iv2; wide: of iv and of iv2 2^22 + iv3
  long long h[4], l[4];
  // the terms' least significant bit: ors of iv2's bits; wide: of low_mark's
  unsigned o[4];
  unsigned lo[3], hi[3];    // bounding box (f2o)
  unsigned wmin;            // smallest mass (f2o)
  unsigned trunc;           // some term had bits below the last integer's
};
constexpr int kAccWords16 = int(sizeof(NodeAcc) / 16);
static_assert(sizeof(NodeAcc) == 112, "NodeAcc is seven 16-byte words");

__device__ __forceinline__ void acc_zero(NodeAcc &a) {
  for (int q = 0; q < 4; ++q) {
    a.h[q] = a.l[q] = 0;
    a.o[q] = 0u;
  }
  for (int d = 0; d < 3; ++d) {
    a.lo[d] = 0xffffffffu;
    a.hi[d] = 0u;
  }
  a.wmin = 0xffffffffu;
  a.trunc = 0u;
}

// The lowest set bit (0 to 43, by the low 22 bits of iv2 and iv3) of a wide
// term as one of 31 marks, and the lowest position that a mark can stand for.
__device__ __forceinline__ unsigned low_mark(unsigned iv2, unsigned iv3) {
  const unsigned lo = iv3 & 0x3fffffu, hi = iv2 & 0x3fffffu;
  if (!(lo | hi)) return 0u;
  const int at = lo ? __ffs(int(lo)) - 1 : 21 + __ffs(int(hi));
  return 1u << (at * 5 / 7);
}
__device__ __forceinline__ int low_of_mark(int mark) { return (7 * mark + 4) / 5; }

// Whether a set's range calls for the third integer: its largest mass 2^12 times
// its smallest; its largest term 2^20 times the largest of the element that has the
// smallest one (2^10 times is what a box of millions has beside its origin); or the
// largest term of one axis 2^5 times that of another (a sheet, a column); zeros
// aside.  Two integers lose whole sets a little above (a kick of 2.6 M particles in
// 137 cells, one of them 10^5 times as heavy or at 10^7 cells: 24 and 27 ms, with
// three 3.0 and 2.9; the tree of a sheet of 2 M, 2^-8 as thick as wide: 3.5 and 0.93
// ms), and below the third only costs (the kick without the heavy one: 2.90 and
// 3.01 ms; masses spread over a factor of 10^4: 3.44 and 3.04; sheets of 70 thousand
// and 2 M, 2^-5: trees of 0.245 and 1.09 ms, with three 0.255 and 0.94).
constexpr int kWideTerm = 20, kWideMass = 12, kWideAxis = 5;
__device__ __forceinline__ unsigned largest_term(const LevelCtl *ctl) {
  return max(max(ctl->range[0], ctl->range[1]), ctl->range[2]);
}
__device__ __forceinline__ bool wide_range(const LevelCtl *ctl) {
  // (bits of positive floats: 2^23 a power of two; nothing but zeros: ~0)
  const unsigned mx = largest_term(ctl), m = ctl->range[3], lt = ~ctl->range[6], lm = ~ctl->range[7];
  bool wide = (mx > lt && mx - lt >= unsigned(kWideTerm) << 23) ||
              (m > lm && m - lm >= unsigned(kWideMass) << 23);
#pragma unroll
  for (int d = 0; d < 3; ++d)
    wide |= ctl->range[d] != 0u && mx - ctl->range[d] >= unsigned(kWideAxis) << 23;
  return wide;
}

// The scales of a set's terms, and its mass where all are the same (the
// simulation's own kicks set them all to 1): the mass sums then follow from the
// counts and cost nothing.
struct SumScales {
  SumScale c, m;
  bool uniform, bad, wide;
  unsigned wbits;
  __device__ __forceinline__ SumScales(const LevelCtl *ctl, bool wide_sums)
      : c(largest_term(ctl)), m(ctl->range[3]), wide(wide_sums) {
    wbits = ctl->range[5];
    bad = SumScale::bad(largest_term(ctl)) || SumScale::bad(ctl->range[3]);
    // (the bits with the sign: as many +w as -w are no set of one mass; and one
    // that the integers do not hold goes the way that says so)
    int h;
    long long l;
    unsigned o;
    uniform = wbits == ~ctl->range[4] && mass_digits(h, l, o);
  }
  // The integers of the one mass, as NodeAcc sums them; whether they hold it.
  __device__ __forceinline__ bool mass_digits(int &h, long long &l, unsigned &o) const {
    const float w = __uint_as_float(wbits);
    const float v = __fadd_rn(w, m.m1);
    const float r = __fsub_rn(w, __fsub_rn(v, m.m1));
    const float v2 = __fadd_rn(r, m.m2);
    const float r2 = __fsub_rn(r, __fsub_rn(v2, m.m2));
    const unsigned iv2 = __float_as_uint(v2) - __float_as_uint(m.m2);
    h = int(__float_as_uint(v) - __float_as_uint(m.m1));
    l = int(iv2);
    o = iv2;
    if (!wide) return r2 == 0.f;
    const float m3 = m.m3(), v3 = __fadd_rn(r2, m3);
    const unsigned iv3 = __float_as_uint(v3) - __float_as_uint(m3);
    l = (l << 22) + int(iv3);
    o = low_mark(iv2, iv3);
    return __fsub_rn(v3, m3) == r2;
  }
  // The mass words of a node of `count` elements.
  __device__ __forceinline__ void masses(NodeAcc &a, int32_t count) const {
    if (!uniform) return;
    int h;
    long long l;
    mass_digits(h, l, a.o[3]);
    a.h[3] = (long long)h * count;
    if (!wide) {
      a.l[3] = l * count;
    } else {  // |l| <= 2^43: what passes 2^44 goes to h
      const __int128 p = __int128(l) * count;
      a.h[3] += (long long)(p >> 44);
      a.l[3] = (long long)p & ((1ll << 44) - 1);
    }
    a.wmin = f2o(__uint_as_float(wbits));
  }
};

// Values reduced over a warp (W = 32) or over each eight lanes (W = 8): lane l
// ends with value l & 7 (reduce8) or l & 3 (reduce4).  Each of the first steps
// exchanges half of the values that are left, so eight reductions take 9
// shuffles, not 40.
template <typename T, typename Op>
__device__ __forceinline__ T reduce_half(T a, T b, int m, Op op) {
  const bool up = threadIdx.x & m;  // keeps a on lanes without bit m, b on the others
  const T mine = up ? b : a, theirs = up ? a : b;
  return op(mine, __shfl_xor_sync(0xffffffffu, theirs, m));
}
template <int W, typename T, typename Op>
__device__ __forceinline__ T reduce4(T v0, T v1, T v2, T v3, Op op) {
  T c = reduce_half(reduce_half(v0, v1, 1, op), reduce_half(v2, v3, 1, op), 2, op);
#pragma unroll
  for (int o = 4; o < W; o <<= 1) c = op(c, __shfl_xor_sync(0xffffffffu, c, o));
  return c;
}
template <int W, typename T, typename Op>
__device__ __forceinline__ T reduce8(T v0, T v1, T v2, T v3, T v4, T v5, T v6, T v7, Op op) {
  const T b0 = reduce_half(reduce_half(v0, v1, 1, op), reduce_half(v2, v3, 1, op), 2, op);
  const T b1 = reduce_half(reduce_half(v4, v5, 1, op), reduce_half(v6, v7, 1, op), 2, op);
  T c = reduce_half(b0, b1, 4, op);
#pragma unroll
  for (int o = 8; o < W; o <<= 1) c = op(c, __shfl_xor_sync(0xffffffffu, c, o));
  return c;
}

// One lane's share.
template <bool WIDE>
struct LaneAcc {
  unsigned h[4], l[4], o[4];  // sums of the bits of v and v2 (modulo 2^32), ors of v2's
  unsigned t[WIDE ? 4 : 1], ot[WIDE ? 4 : 1];  // the same of the third integer
  float lo[3], hi[3], wmin, left;
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      h[q] = l[q] = o[q] = 0u;
      if (WIDE) t[q] = ot[q] = 0u;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lo[d] = INFINITY;
      hi[d] = -INFINITY;
    }
    wmin = INFINITY;
    left = 0.f;
  }
  __device__ __forceinline__ void term(int q, float x, const SumScale &s) {
    const float v = __fadd_rn(x, s.m1);
    const float r = __fsub_rn(x, __fsub_rn(v, s.m1));
    const float v2 = __fadd_rn(r, s.m2);
    if (WIDE) {
      const float r2 = __fsub_rn(r, __fsub_rn(v2, s.m2));
      const float m3 = s.m3(), v3 = __fadd_rn(r2, m3);
      left = fmaxf(left, fabsf(__fsub_rn(__fsub_rn(v3, m3), r2)));
      t[q] += __float_as_uint(v3);
      ot[q] |= __float_as_uint(v3);
    } else {
      left = fmaxf(left, fabsf(__fsub_rn(__fsub_rn(v2, s.m2), r)));
    }
    h[q] += __float_as_uint(v);
    l[q] += __float_as_uint(v2);
    o[q] |= __float_as_uint(v2);
  }
  __device__ __forceinline__ void add(const float4 &p, const SumScales &S) {
    term(0, fmul_(p.w, p.x), S.c);
    term(1, fmul_(p.w, p.y), S.c);
    term(2, fmul_(p.w, p.z), S.c);
    if (!S.uniform) {
      term(3, p.w, S.m);
      wmin = fminf(wmin, p.w);
    }
    lo[0] = fminf(lo[0], p.x); hi[0] = fmaxf(hi[0], p.x);
    lo[1] = fminf(lo[1], p.y); hi[1] = fmaxf(hi[1], p.y);
    lo[2] = fminf(lo[2], p.z); hi[2] = fmaxf(hi[2], p.z);
  }
  // The sums of a warp (W = 32; of each eight lanes, W = 8) into *out, word by
  // word from different lanes; cnt: this lane's elements (at most 512), few: the
  // warp's are at most 1023 (an int holds the sums of one integer).
  template <int W>
  __device__ __forceinline__ void reduce(NodeAcc *out, bool write, int cnt, bool few,
                                         const SumScales &S) const {
    int hv[4], lv[4];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      hv[q] = int(h[q] - unsigned(cnt) * __float_as_uint(S.c.m1));
      lv[q] = int(l[q] - unsigned(cnt) * __float_as_uint(S.c.m2));
    }
    hv[3] = S.uniform ? 0 : int(h[3] - unsigned(cnt) * __float_as_uint(S.m.m1));
    lv[3] = S.uniform ? 0 : int(l[3] - unsigned(cnt) * __float_as_uint(S.m.m2));
    using LL = long long;
    LL sum;
    unsigned ov[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) ov[q] = o[q];
    if (WIDE) {
      LL w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const bool on = q < 3 || !S.uniform;
        const SumScale &sc = q < 3 ? S.c : S.m;
        w[q] = on ? LL(lv[q]) * (1 << 22) + int(t[q] - unsigned(cnt) * __float_as_uint(sc.m3())) : 0;
        ov[q] = low_mark(o[q], ot[q]);
      }
      sum = reduce8<W>(LL(hv[0]), LL(hv[1]), LL(hv[2]), LL(hv[3]), w[0], w[1], w[2], w[3],
                       [](LL a, LL b) { return a + b; });
    } else if (few) {
      sum = reduce8<W>(hv[0], hv[1], hv[2], hv[3], lv[0], lv[1], lv[2], lv[3],
                       [](int a, int b) { return a + b; });
    } else {
      sum = reduce8<W>(LL(hv[0]), LL(hv[1]), LL(hv[2]), LL(hv[3]), LL(lv[0]), LL(lv[1]), LL(lv[2]),
                       LL(lv[3]), [](LL a, LL b) { return a + b; });
    }
    const unsigned bits = reduce4<W>(ov[0], ov[1], ov[2], ov[3], [](unsigned a, unsigned b) { return a | b; });
    // minima; the upper bounds complemented, and 0 where a term was truncated
    const unsigned mn = reduce8<W>(f2o(lo[0]), f2o(lo[1]), f2o(lo[2]), ~f2o(hi[0]), ~f2o(hi[1]),
                                   ~f2o(hi[2]), f2o(wmin), left != 0.f ? 0u : 1u,
                                   [](unsigned a, unsigned b) { return min(a, b); });
    const int f = threadIdx.x & (W - 1);
    if (write && f < 8) {
      (f < 4 ? out->h[f] : out->l[f - 4]) = sum;
      if (f < 4) out->o[f] = bits;
      if (f < 3) out->lo[f] = mn;
      else if (f < 6) out->hi[f - 3] = ~mn;
      else if (f == 6) out->wmin = mn;
      else out->trunc = 1u - mn;
    }
  }
};

// Word f of n records merged, a lane a word: sums 0-7 (into *sum), then o, lo,
// hi, wmin and trunc (into *bits).
constexpr int kAccWords = 20;
__device__ __forceinline__ bool acc_or(int f) { return f < 12 || f == 19; }
__device__ __forceinline__ bool acc_max(int f) { return f >= 15 && f < 18; }
__device__ __forceinline__ void merge_word(const NodeAcc *part, int n, int f, long long *sum,
                                           unsigned *bits) {
  long long s = 0;
  unsigned u = acc_or(f) || acc_max(f) ? 0u : 0xffffffffu;
  for (int v = 0; v < n; ++v) {
    if (f < 8) {
      s += reinterpret_cast<const long long *>(part + v)[f];
    } else {
      const unsigned w = reinterpret_cast<const unsigned *>(part + v)[f + 8];
      u = acc_or(f) ? (u | w) : (acc_max(f) ? max(u, w) : min(u, w));
    }
  }
  *sum = s;
  *bits = u;
}

__device__ __forceinline__ double pow2(int e) {  // normal range
  return __longlong_as_double((long long)(e + 1023) << 52);
}
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float(unsigned(e + 127) << 23); }

// Correctly rounded double of h 2^22 + l (units of 2^(k-45)); wide: of h 2^44 + l
// (units of 2^(k-67)).
__device__ double units_to_double(long long h, long long l, bool wide = false) {
  if (!wide && h < (1ll << 40) && h > -(1ll << 40)) return __ll2double_rn((h << 22) + l);
  const __int128 v = (__int128(h) << (wide ? 44 : 22)) + l;
  const bool neg = v < 0;
  const unsigned __int128 u = neg ? (unsigned __int128)(-v) : (unsigned __int128)v;
  const unsigned long long hi = (unsigned long long)(u >> 64), lo = (unsigned long long)u;
  const int bits = hi ? 128 - __clzll((long long)hi) : 64 - __clzll((long long)lo);
  const int sh = bits > 63 ? bits - 63 : 0;
  // the top 63 bits with the rest folded into a sticky bit, rounded once
  unsigned long long m = (unsigned long long)(u >> sh);
  if (sh > 0 && (u & ((((unsigned __int128)1) << sh) - 1)) != 0) m |= 1ull;
  const double r = __dmul_rn(__ull2double_rn(m), pow2(sh));
  return neg ? -r : r;
}

// Float that the reference's (float)(sx / sm) gives, if the bounds decide it.
// sx, sm: the sums computed here; bx, bm: bounds on |reference sum - sum here|.
__device__ bool certify(double sx, double bx, double sm, double bm, float *out) {
  const double xl = sx - bx, xh = sx + bx, ml = sm - bm, mh = sm + bm;
  if (!(ml > 0.0) || !isfinite(xl) || !isfinite(xh) || !isfinite(mh)) return false;
  const double q0 = __ddiv_rd(xl, mh), q1 = __ddiv_rd(xl, ml), q2 = __ddiv_ru(xh, mh),
               q3 = __ddiv_ru(xh, ml);
  double lo = fmin(fmin(q0, q1), fmin(q2, q3));
  double hi = fmax(fmax(q0, q1), fmax(q2, q3));
  // the reference rounds its quotient to double once more
  lo -= fabs(lo) * 0x1p-51;
  hi += fabs(hi) * 0x1p-51;
  const float fl = __double2float_rn(lo), fh = __double2float_rn(hi);
  if (fl != fh) return false;
  *out = fl;
  return true;
}

// The sums of a node's terms and what bounds their distance from the
// reference's sequential ones, in units of 2^(k-45) (wide: 2^(k-67)).
struct NodeSums {
  double x[4];   // the exact sums, rounded to double
  float abs[4];  // at least sum |terms|
  float err[4];  // at least |reference sum - x|
  bool exact[4];  // the reference's sum is exactly x
};

__device__ __forceinline__ NodeSums node_sums(const NodeAcc &A, int32_t count, bool wide) {
  NodeSums S;
  // The reference's sequential sum lies within (n - 1) u sum|terms| of the
  // exact sum, to first order; (n + 64) u (1 + 2^-20) covers the rest.  The sums
  // here are exact except for truncated terms (half a unit each) and their
  // rounding to double.
  const float n = __int2float_ru(count);
  const float g = __fmul_ru(__fmul_ru(__fadd_ru(n, 64.f), 0x1p-53f), 1.f + 0x1p-20f);
  const float slack = A.trunc ? n : 0.f;
  const bool wpos = o2f(A.wmin) >= 0.f;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    S.x[q] = units_to_double(A.h[q], A.l[q], wide);
    const float xa = __double2float_ru(fabs(S.x[q]));
    // sum of |terms|: the sum itself where none is negative, else n times the
    // scale's largest term (2^(k-2))
    const bool pos = wpos && (q == 3 || o2f(A.lo[q]) >= 0.f);
    S.abs[q] = pos ? __fadd_ru(xa, slack) : __fmul_ru(n, wide ? 0x1p65f : 0x1p43f);
    // Exact: every term a multiple of 2^emin (none truncated) and the
    // magnitudes summing below 2^(53 + emin) -- then the reference's
    // sequential sum and this one are the same exact value, a double.
    const unsigned b = wide ? A.o[q] : A.o[q] & 0x3fffffu;
    const int at = b ? __ffs(int(b)) - 1 : 31;
    // no iv2 (and iv3): whole multiples of 2^22 (2^44) units
    const int emin = wide ? low_of_mark(at) : min(at, 22);
    S.exact[q] = !A.trunc && S.abs[q] < pow2f(53 + emin);
    S.err[q] = S.exact[q] ? 0.f : __fadd_ru(__fmaf_ru(g, S.abs[q], slack), __fmul_ru(xa, 0x1p-52f));
  }
  return S;
}

// A node's exact sum h 2^22 + l as an unevaluated sum of two floats, within err
// of it (2^-45 of it where its two parts do not cancel); |h| and |l| below 2^46.
__device__ __forceinline__ void two_sum_f(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
__device__ __forceinline__ void sum_pair(long long h, long long l, float &hi, float &lo, float &err) {
  const float ha = __int2float_rn(int(h >> 24)) * 0x1p46f, hb = __int2float_rn(int(h & 0xffffff)) * 0x1p22f;
  const float la = __int2float_rn(int(l >> 24)) * 0x1p24f, lb = __int2float_rn(int(l & 0xffffff));
  float a, ea, b, eb, s, es;
  two_sum_f(ha, hb, a, ea);
  two_sum_f(la, lb, b, eb);
  two_sum_f(a, b, s, es);
  two_sum_f(s, __fadd_rn(es, __fadd_rn(ea, eb)), hi, lo);
  err = __fmul_ru(__fadd_ru(fabsf(a), fabsf(b)), 0x1p-46f);
}

// The centre of mass on the FP32 pipe alone: the sums as float pairs, the
// quotient as q0 + q1 with its residual from fused multiply-adds (within 2^-43
// of x / m), decided where q0 + q1 -/+ the error bound round to one float.  (FP64
// leaves a chain of 5000 cycles to every level of a subtree.)  What it leaves
// open goes to the FP64 sums.
__device__ __forceinline__ bool quotients_f32(const NodeAcc &A, int32_t count, int kx, int km,
                                              float *xc) {
  const float n = __int2float_ru(count);
  const float g = __fmul_ru(__fmul_ru(__fadd_ru(n, 64.f), 0x1p-53f), 1.f + 0x1p-20f);
  const float slack = A.trunc ? n : 0.f;
  const bool wpos = o2f(A.wmin) >= 0.f;
  float hi[4], lo[4], err[4];
  bool exact[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const long long lim = 1ll << 46;
    if (A.h[q] >= lim || A.h[q] <= -lim || A.l[q] >= lim || A.l[q] <= -lim) return false;
    float pair_err;
    sum_pair(A.h[q], A.l[q], hi[q], lo[q], pair_err);
    // as in node_sums, whose comments give the reasons
    const float xa = __fadd_ru(__fmul_ru(fabsf(hi[q]), 1.f + 0x1p-20f), pair_err);
    const bool pos = wpos && (q == 3 || o2f(A.lo[q]) >= 0.f);
    const float sabs = pos ? __fadd_ru(xa, slack) : __fmul_ru(n, 0x1p43f);
    const unsigned b = A.o[q] & 0x3fffffu;
    const int emin = b ? __ffs(int(b)) - 1 : 22;
    exact[q] = !A.trunc && sabs < pow2f(53 + emin);
    err[q] = __fadd_ru(pair_err, exact[q] ? 0.f : __fmaf_ru(g, sabs, slack));
  }
  const float ml = __fsub_rd(__fmul_rd(hi[3], 1.f - 0x1p-20f), err[3]);
  const int ks = kx - km;
  if (!(ml > 0.f) || ks < -60 || ks > 60) return false;
  const float ri = __frcp_ru(ml), r = __frcp_rn(hi[3]), scale = pow2f(ks);
  bool ok = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float q0 = __fmul_rn(hi[d], r);
    // x - q0 m: the products' high parts cancel exactly in the fused operation
    float rem = __fmaf_rn(-q0, hi[3], hi[d]);
    rem = __fadd_rn(rem, __fmaf_rn(-q0, lo[3], lo[d]));
    const float q1 = __fmul_rn(rem, r);
    float f, e;
    two_sum_f(q0, q1, f, e);
    const float qa = __fmul_ru(fabsf(hi[d]), __fmul_ru(ri, 1.f + 0x1p-20f));
    const float w = __fmaf_ru(qa, 0x1p-42f, __fmul_ru(__fmaf_ru(qa, err[3], err[d]), ri));
    const float fl = __fadd_rn(f, __fsub_rd(e, w)), fh = __fadd_rn(f, __fadd_ru(e, w));
    const float v = __fmul_rn(fl, scale);
    // (a scaled result near the subnormals would round again)
    if (fl == fh && (fl == 0.f || fabsf(v) > 0x1p-100f)) xc[d] = v;
    // exact sums whose quotient is a tie between two floats (an even count)
    else if (exact[d] && exact[3])
      xc[d] = __double2float_rn(__dmul_rn(
          __ddiv_rn(units_to_double(A.h[d], A.l[d]), units_to_double(A.h[3], A.l[3])), pow2(ks)));
    else ok = false;
  }
  return ok;
}

// The floats that the reference's (float)(x / m) gives, where the bounds decide
// them: false where one is left open.  One reciprocal a node and three FP64
// multiply-adds a coordinate: a Newton step takes the float reciprocal to 46
// bits, the quotient is corrected by its residual (within 2^-52 of x / m), and
// the error bounds are taken in float, rounded up.
__device__ __forceinline__ bool quotients(const NodeSums &S, int kx, int km, float *xc) {
  const float ml = __fsub_rd(__double2float_rd(S.x[3]), S.err[3]);
  if (!(ml > 0.f)) return false;
  const float ri = __frcp_ru(ml);
  const double m = S.x[3];
  double r = double(__frcp_rn(__double2float_rn(m)));
  r = __fma_rn(r, __fma_rn(-m, r, 1.0), r);
  const double scale = pow2(kx - km);
  bool ok = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double x = S.x[d];
    double q = __dmul_rn(x, r);
    q = __fma_rn(__fma_rn(-q, m, x), r, q);
    // |reference quotient - q| <= (err_x + |q| err_m) / (m - err_m), plus both
    // quotients' own rounding
    const float qa = __fmul_ru(__double2float_ru(fabs(x)), ri);
    const float e = __fmul_ru(__fmaf_ru(qa, S.err[3], S.err[d]), ri);
    const double w = double(__fmaf_ru(qa, 0x1p-50f, e));
    const float lo = __double2float_rn(__dmul_rn(__dsub_rn(q, w), scale)),
                hi = __double2float_rn(__dmul_rn(__dadd_rn(q, w), scale));
    if (lo == hi) xc[d] = lo;
    else if (S.exact[d] && S.exact[3])
      xc[d] = __double2float_rn(__dmul_rn(__ddiv_rn(x, m), scale));
    else ok = false;
  }
  return ok;
}

// The node's box, split axis and (where the bounds decide it) centre of mass
// from its reduced statistics; false when the centre of mass is left undecided.
__device__ bool decide_node(DNode &N, const NodeAcc &A, const SumScales &S, int32_t force_fallback,
                            int32_t nd) {
  for (int d = 0; d < 3; ++d) {
    N.xmin[d] = o2f(A.lo[d]);
    N.xmax[d] = o2f(A.hi[d]);
  }
  // leaf by size, or the split axis: the longest box edge, ties to the later
  // axis (RCBForceTree.cxx:837-852); it needs the box only, not the centre
  N.nleft = 0;
  if (N.count <= nd) {
    N.split_dim = -1;
  } else {
    const float l0 = fsub_(N.xmax[0], N.xmin[0]), l1 = fsub_(N.xmax[1], N.xmin[1]),
                l2 = fsub_(N.xmax[2], N.xmin[2]);
    N.split_dim = (l0 > l1 && l0 > l2) ? 0 : (l1 > l2 ? 1 : 2);
  }
  if (force_fallback != 0 || S.bad) return false;
  return (!S.wide && quotients_f32(A, N.count, S.c.k, S.m.k, N.xc)) ||
         quotients(node_sums(A, N.count, S.wide), S.c.k, S.m.k, N.xc);
}

// A tighter bound for sums that node_sums leaves open: an addition rounds only
// where the term, or the running sum since an earlier such term, has bits below
// the last place U of the running sum; so with `low` such terms (bits below U,
// U = the last place of twice sum |terms|) the sequential sum is within
// 2 (low + 32) U of the exact one.
__device__ __forceinline__ int last_place(float abs_units) {  // exponent of U, in units
  return int(__float_as_uint(abs_units) >> 23) - 127 + 1 - 52;
}
__device__ __forceinline__ void tighten(NodeSums &S, const int *low, const NodeAcc &A, int32_t count) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (S.exact[q]) continue;
    const float e = __fadd_ru(
        __fmul_ru(2.f * (float(low[q]) + 33.f), pow2f(max(-126, last_place(S.abs[q])))),
        __fadd_ru(A.trunc ? __int2float_ru(count) : 0.f,
                  __fmul_ru(__double2float_ru(fabs(S.x[q])), 0x1p-52f)));
    S.err[q] = fminf(S.err[q], e);
  }
}

// The elements into the first buffer, their input indices, and the largest
// terms for the sums' scale.
__global__ void __launch_bounds__(256)
    k_elements(const float4 *__restrict__ in, int64_t n, float4 *__restrict__ pos,
               int32_t *__restrict__ oid, LevelCtl *ctl) {
  chain_enter();
  unsigned mt[3] = {0, 0, 0}, mm = 0, mn = 0xffffffffu, mx = 0, nt = 0xffffffffu, nm = 0xffffffffu;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const float4 p = in[i];
    pos[i] = p;
    oid[i] = int32_t(i);
    const unsigned t[3] = {__float_as_uint(fmul_(p.w, p.x)) & 0x7fffffffu,
                           __float_as_uint(fmul_(p.w, p.y)) & 0x7fffffffu,
                           __float_as_uint(fmul_(p.w, p.z)) & 0x7fffffffu};
    const unsigned w = __float_as_uint(p.w) & 0x7fffffffu;
#pragma unroll
    for (int d = 0; d < 3; ++d) mt[d] = max(mt[d], t[d]);
    mm = max(mm, w);
    nt = min(nt, max(max(t[0], t[1]), t[2]) - 1u);  // (zero as the largest: it is left aside)
    nm = min(nm, w - 1u);
    mn = min(mn, __float_as_uint(p.w));
    mx = max(mx, __float_as_uint(p.w));
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) mt[d] = __reduce_max_sync(0xffffffffu, mt[d]);
  mm = __reduce_max_sync(0xffffffffu, mm);
  mn = __reduce_min_sync(0xffffffffu, mn);
  mx = __reduce_max_sync(0xffffffffu, mx);
  nt = __reduce_min_sync(0xffffffffu, nt);
  nm = __reduce_min_sync(0xffffffffu, nm);
  const unsigned v[8] = {mt[0], mt[1], mt[2], mm, ~mn, mx, ~nt, ~nm};  // as LevelCtl::range
  __shared__ unsigned sh[8];
  if (threadIdx.x < 8) sh[threadIdx.x] = 0u;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) atomicMax(&sh[i], v[i]);
  }
  __syncthreads();
  if (threadIdx.x < 8) atomicMax(&ctl->range[threadIdx.x], sh[threadIdx.x]);
}

// The root, its chunks and the first level.  The launches that follow were made
// for a set of either range (`wide`): where it is the other one, there is no level
// and nothing is done, and the host launches all of it again for this one.
constexpr int kErrRange = 6;  // C_ERR: the other range
template <int PT>
__global__ void __launch_bounds__(256)
    k_root(DNode *nodes, int64_t n, TreeConfig cfg, LevelCtl *ctl, int32_t *chunk_node,
           int32_t *chunk_base, NodeAcc *acc, unsigned *ticket, int2 *roots, int32_t sub_max,
           bool wide, int32_t *err) {
  chain_enter();
  const bool other = wide_range(ctl) != wide;
  const int32_t nc = chunks_of<PT>(int32_t(n));
  const bool sub = n <= sub_max;
  if (!sub)
    for (int32_t c = threadIdx.x; c < nc; c += blockDim.x) chunk_node[c] = 0;
  if (threadIdx.x != 0) return;
  DNode &R = nodes[0];
  R.count = int32_t(n);
  R.offset = 0;
  R.cl = R.cr = 0;
  for (int d = 0; d < 3; ++d) {
    R.xmin[d] = cfg.min[d];
    R.xmax[d] = cfg.max[d];
    R.xc[d] = 0.f;
  }
  R.tdr = 0.f;
  R.split_dim = -1;
  R.nleft = 0;
  if (!sub) {
    chunk_base[0] = 0;
    acc_zero(acc[0]);
    ticket[0] = 0u;
  }
  ctl->lev[0] = LevelSpan{0, sub || other ? 0 : 1, 0, 1, nc, 1, int32_t(n), 0};
  ctl->lev[1] = LevelSpan{-1, 0, 0, 0, 0, 0, 0, 0};
  ctl->begin[0] = 0;
  if (sub) roots[0] = make_int2(0, 0);
  ctl->nroots = sub ? 1 : 0;
  ctl->done = sub && !other;
  ctl->node_end = 1;
  if (other) *err = kErrRange;
}

// A chunk's `len` elements into its warps' records.
template <int PT, bool WIDE>
__device__ __forceinline__ void chunk_sums(const float4 *__restrict__ pos, int32_t len,
                                           const SumScales &S, NodeAcc *part) {
  constexpr int kU = 4;
  LaneAcc<WIDE> a;
  a.zero();
  int cnt = 0;
  for (int j0 = 0; j0 < PT && j0 * kChunkThreads < len; j0 += kU) {
    float4 p[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int e = (j0 + u) * kChunkThreads + threadIdx.x;
      if (e < len) p[u] = pos[e];
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int e = (j0 + u) * kChunkThreads + threadIdx.x;
      if (e < len) {
        a.add(p[u], S);
        ++cnt;
      }
    }
  }
  a.template reduce<32>(&part[threadIdx.x >> 5], true, cnt, true, S);  // a warp has at most 512 elements
}

// Statistics of every node of the level, and its split decision by the block
// that adds a node's last chunk.
template <int PT, bool WIDE = false>
__global__ void __launch_bounds__(kChunkThreads, kLevelBlocks)
    k_level_stats(const float4 *__restrict__ pos, DNode *nodes, LevelCtl *ctl, int32_t level,
                  const int32_t *__restrict__ chunk_node, const int32_t *__restrict__ chunk_base,
                  NodeAcc *acc, unsigned *ticket, int32_t *fallback, int64_t *counters,
                  int32_t force_fallback, int32_t nd) {
  chain_enter();
  LevelSpan L;
  if (!level_runs(ctl, level, L, true) || int32_t(blockIdx.x) >= L.nchunk) return;
  constexpr int kW = kChunkThreads / 32;
  __shared__ NodeAcc part[kW];
  const ChunkRange R = chunk_range<PT>(nodes, chunk_node, chunk_base, L.nb, int32_t(blockIdx.x));
  const SumScales S(ctl, WIDE);
  chunk_sums<PT, WIDE>(pos + R.begin, R.len, S, part);
  __syncthreads();
  if (threadIdx.x >= 32) return;
  // a thread per word: the warps' records into the node's, one atomic each
  NodeAcc &T = acc[R.node - L.nb];
  const int f = threadIdx.x;
  long long sum = 0;
  unsigned bits = 0;
  if (f < kAccWords) merge_word(part, kW, f, &sum, &bits);
  if (WIDE) {
    // what passes 2^44 of the lower integers' sums goes to the upper ones', so
    // that the chunks of any node fit 64 bits
    const long long up = f >= 4 && f < 8 ? (sum + (1ll << 43)) >> 44 : 0;
    sum -= up * (1ll << 44);
    const long long add = __shfl_down_sync(0xffffffffu, up, 4);
    if (f < 4) sum += add;
  }
  if (f < kAccWords) {
    unsigned *word = reinterpret_cast<unsigned *>(&T) + 8 + f;
    if (f < 8) atomicAdd(reinterpret_cast<unsigned long long *>(&T) + f, (unsigned long long)sum);
    else if (acc_or(f)) atomicOr(word, bits);
    else if (acc_max(f)) atomicMax(word, bits);
    else atomicMin(word, bits);
  }
  __threadfence();
  __syncwarp();
  if (threadIdx.x != 0) return;
  DNode N = nodes[R.node];
  if (atomicAdd(&ticket[R.node - L.nb], 1u) + 1u != unsigned(chunks_of<PT>(N.count))) return;
  __threadfence();
  ticket[R.node - L.nb] = 0u;  // k_level_count counts the chunks again
  NodeAcc A;
  const int4 *src = reinterpret_cast<const int4 *>(&T);
  int4 *dst = reinterpret_cast<int4 *>(&A);
#pragma unroll
  for (int q = 0; q < kAccWords16; ++q) dst[q] = __ldcg(src + q);
  S.masses(A, N.count);
  if (!decide_node(N, A, S, force_fallback, nd)) {
    fallback[atomicAdd((unsigned long long *)&counters[C_NFALLBACK], 1ull)] = R.node;
    atomicExch(&ctl->abort, level + 1);
  }
  nodes[R.node] = N;
}

template <int PT>
constexpr auto k_level_stats_wide = k_level_stats<PT, true>;

// Left counts of the level's chunks and each warp's left elements before its
// share of the chunk (the shares of k_part_left); only the split coordinate is
// loaded, every lane's loads in flight at once.  The block that counts a node's
// last chunk scans the node's chunks; the one that counts the level's last
// chunk makes the children and the next level.
template <int PT>
__global__ void __launch_bounds__(kChunkThreads)
    k_level_count(const float4 *__restrict__ pos, DNode *nodes, LevelCtl *ctl, int32_t level,
                  const int32_t *__restrict__ chunk_node, const int32_t *__restrict__ chunk_base,
                  int32_t *next_chunk_node, int32_t *next_chunk_base, int32_t *left_cnt,
                  int32_t *left_base, int32_t *wpre, NodeAcc *acc, unsigned *ticket, int2 *roots,
                  int64_t *counters, int32_t sub_max) {
  chain_enter();
  LevelSpan L;
  if (!level_runs(ctl, level, L) || int32_t(blockIdx.x) >= L.nchunk) return;
  constexpr int kWarps = kChunkThreads / 32, kSub = 32 * PT;
  __shared__ int wt[kWarps];
  __shared__ int sh_warp[32];
  __shared__ int last;
  const int32_t chunk = int32_t(blockIdx.x);
  const ChunkRange R = chunk_range<PT>(nodes, chunk_node, chunk_base, L.nb, chunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t count = nodes[R.node].count, d = nodes[R.node].split_dim;
  if (d >= 0) {
    const float split = nodes[R.node].xc[d];
    const float *key = reinterpret_cast<const float *>(pos + R.begin) + d;
    float kv[PT];
#pragma unroll
    for (int u = 0; u < PT; ++u) {
      const int e = warp * kSub + 32 * u + lane;
      kv[u] = e < R.len ? key[4 * e] : INFINITY;
    }
    int c = 0;
#pragma unroll
    for (int u = 0; u < PT; ++u) c += warp * kSub + 32 * u + lane < R.len && kv[u] < split;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) wt[warp] = c;
    __syncthreads();
    if (threadIdx.x < kWarps) {
      int pre = 0, tot = 0;
      for (int w = 0; w < kWarps; ++w) {
        pre += w < int(threadIdx.x) ? wt[w] : 0;
        tot += wt[w];
      }
      wpre[chunk * kWarps + threadIdx.x] = pre;
      if (threadIdx.x == 0) left_cnt[chunk] = tot;
    }
  }
  // the node's last chunk: exclusive scan of its chunks' left counts
  __threadfence();
  __syncthreads();
  const int32_t nc = chunks_of<PT>(count);
  if (threadIdx.x == 0) last = atomicAdd(&ticket[R.node - L.nb], 1u) + 1u == unsigned(nc);
  __syncthreads();
  if (last && d >= 0) {
    __threadfence();
    const int32_t cb = chunk_base[R.node - L.nb];
    int run = 0;
    for (int32_t c0 = 0; c0 < nc; c0 += kChunkThreads) {
      const int32_t c = c0 + int32_t(threadIdx.x);
      const int v = c < nc ? __ldcg(left_cnt + cb + c) : 0;
      int total;
      const int ex = block_excl_scan(v, sh_warp, &total);
      if (c < nc) left_base[cb + c] = run + ex;
      run += total;
    }
    if (threadIdx.x == 0) nodes[R.node].nleft = run;
  }
  // the level's last chunk: children, two per node split into two non-empty
  // parts, and the next level's chunks
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&ctl->ticket, 1u) + 1u == unsigned(L.nchunk);
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int32_t nl = L.ne - L.nb, nroots = ctl->nroots;
  int splits = 0, chunks = 0, subs = 0, largest = 0;
  for (int32_t i0 = 0; i0 < nl; i0 += kChunkThreads) {
    const int32_t i = i0 + int32_t(threadIdx.x);
    DNode N;
    bool split = false;
    if (i < nl) {
      const int4 *src = reinterpret_cast<const int4 *>(nodes + L.nb + i);
      int4 *dst = reinterpret_cast<int4 *>(&N);
#pragma unroll
      for (int q = 0; q < 4; ++q) dst[q] = __ldcg(src + q);
      split = N.split_dim >= 0 && N.nleft > 0 && N.nleft < N.count;
    }
    const int32_t n0 = split ? N.nleft : 0, n1 = split ? N.count - N.nleft : 0;
    const bool s0 = split && n0 <= sub_max, s1 = split && n1 <= sub_max;  // subtree roots
    const int32_t c0 = s0 ? 0 : chunks_of<PT>(n0), c1 = s1 ? 0 : chunks_of<PT>(n1);
    int ts, tc, tr;
    const int rank = splits + block_excl_scan(split ? 1 : 0, sh_warp, &ts);
    const int32_t cb = chunks + block_excl_scan(c0 + c1, sh_warp, &tc);
    const int32_t rb = nroots + subs + block_excl_scan(int(s0) + int(s1), sh_warp, &tr);
    if (split) {
      const int32_t cl = L.ne + 2 * rank;
      write_child(nodes[cl], N, 0);
      write_child(nodes[cl + 1], N, 1);
      nodes[L.nb + i].cl = cl;
      nodes[L.nb + i].cr = cl + 1;
      next_chunk_base[2 * rank] = cb;
      next_chunk_base[2 * rank + 1] = cb + c0;
      for (int32_t c = 0; c < c0; ++c) next_chunk_node[cb + c] = cl;
      for (int32_t c = 0; c < c1; ++c) next_chunk_node[cb + c0 + c] = cl + 1;
      if (s0) roots[rb] = make_int2(cl, (level + 1) & 1);
      if (s1) roots[rb + int(s0)] = make_int2(cl + 1, (level + 1) & 1);
      if (!s0) largest = max(largest, n0);
      if (!s1) largest = max(largest, n1);
    }
    if (i < nl) ticket[i] = 0u;
    splits += ts;
    chunks += tc;
    subs += tr;
  }
  largest = __reduce_max_sync(0xffffffffu, largest);
  if (lane == 0) wt[warp] = largest;
  __syncthreads();
  for (int32_t i = threadIdx.x; i < 2 * splits; i += kChunkThreads) {
    acc_zero(acc[i]);
    ticket[i] = 0u;
  }
  if (threadIdx.x != 0) return;
  for (int w = 0; w < kWarps; ++w) largest = max(largest, wt[w]);
  const int32_t ne = L.ne + 2 * splits;
  ctl->lev[(level + 1) & 1] =
      LevelSpan{level + 1, chunks > 0 ? 1 : 0, L.ne, ne, chunks, 2 * splits - subs, largest, 0};
  ctl->begin[(level + 1) % kCtlLevels] = L.ne;
  ctl->next_level = level + 1;
  ctl->ticket = 0u;
  ctl->nroots = nroots + subs;
  ctl->done = chunks == 0;
  ctl->node_end = ne;
  counters[C_CHAINS] = 0;  // the level's queue of long swap chains
}

// Left particles go to their rank; idx[rank] records where each came from.
// Warp w takes the chunk's elements [w * kSub, (w + 1) * kSub) 32 at a time
// (coalesced), kB steps' loads in flight; ranks follow array order through
// the warps' left counts before them (k_level_count) and a ballot prefix
// within each step.
template <int PT>
__global__ void __launch_bounds__(kChunkThreads)
    k_part_left(const float4 *__restrict__ pos, const int32_t *__restrict__ oid, const DNode *nodes,
                const LevelCtl *ctl, int32_t level, const int32_t *__restrict__ chunk_node,
                const int32_t *__restrict__ chunk_base, const int32_t *left_base,
                const int32_t *wpre, float4 *tpos, int32_t *toid, int32_t *idx, int32_t *ridx) {
  chain_enter();
  LevelSpan L;
  if (!level_runs(ctl, level, L) || int32_t(blockIdx.x) >= L.nchunk) return;
  constexpr int kWarps = kChunkThreads / 32;
  constexpr int kSub = 32 * PT;  // a warp's share of the chunk
  constexpr int kB = 4;
  const int32_t chunk = int32_t(blockIdx.x);
  const ChunkRange R = chunk_range<PT>(nodes, chunk_node, chunk_base, L.nb, chunk);
  const DNode &N = nodes[R.node];
  if (N.split_dim < 0) {
    // a leaf keeps its elements: copied once into the next level's buffer
    for (int k = threadIdx.x; k < R.len; k += kChunkThreads) {
      tpos[R.begin + k] = pos[R.begin + k];
      toid[R.begin + k] = oid[R.begin + k];
    }
    return;
  }
  const int d = N.split_dim;
  const float split = N.xc[d];
  const int32_t off = N.offset, nleft = N.nleft;
  const int lane = threadIdx.x & 31, warp = int(threadIdx.x >> 5);
  const unsigned below = (1u << lane) - 1u;
  const int sub_end = min(kSub, R.len - warp * kSub);  // elements of this warp's share
  int r = left_base[chunk] + wpre[chunk * kWarps + warp];
  for (int j0 = 0; j0 < sub_end; j0 += 32 * kB) {
    float4 p[kB];
    int32_t o[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int e = warp * kSub + j0 + 32 * u + lane;
      if (j0 + 32 * u < sub_end && e < R.len) {
        p[u] = pos[R.begin + e];
        o[u] = oid[R.begin + e];
      } else {
        p[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        o[u] = 0;
      }
    }
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      if (j0 + 32 * u >= sub_end) break;  // the same for the whole warp
      const int e = warp * kSub + j0 + 32 * u + lane;
      const bool in = e < R.len;
      const bool l = in && key_of(p[u], d) < split;
      const unsigned bal = __ballot_sync(0xffffffffu, l);
      const int q = r + __popc(bal & below);  // left elements before this one
      if (l) {
        tpos[off + q] = p[u];
        toid[off + q] = o[u];
        idx[off + q] = R.local + e;
      } else if (in) {
        ridx[off + (R.local + e - q)] = R.local + e;
        if (R.local + e >= nleft) {
          // a right element at or after nleft: no swap touches it, it stays
          tpos[R.begin + e] = p[u];
          toid[R.begin + e] = o[u];
        }
      }
      r += __popc(bal);
    }
  }
}

// A swap chain still running after the partition's single steps: its
// position in the node, the node and the element's position in the level's
// array.
struct ChainItem {
  int32_t q, node;
  int64_t src;
};
static_assert(sizeof(ChainItem) == sizeof(int4), "a chain item fills one int4 of the queue");

// One or more steps of the chain q -> idx[q] -> ... (q < nleft): the q-th
// left element has c = idx[q] - q right elements before it, and so has every
// left element up to the c-th right element (at ridx[c]), whose ranks run to
// b = ridx[c] - c.  Within that run each step adds c, so the chain leaves
// [q, min(b, nleft)) at the first of q + c, q + 2c, ... at or past it.
// Returns a position > q; *bad on an inconsistent partition.
__device__ __forceinline__ int32_t chain_jump(int32_t q, int32_t nleft, int32_t nright,
                                              const int32_t *idx, const int32_t *ridx, bool *bad) {
  const int32_t c = idx[q] - q;
  if (c <= 0) {  // cannot happen for a valid partition (a chain never meets a fixed point)
    *bad = true;
    return nleft;
  }
  int32_t lim = nleft;
  if (c < nright) {
    const int32_t b = ridx[c] - c;
    if (b <= q) {  // cannot happen for a valid partition
      *bad = true;
      return nleft;
    }
    lim = min(lim, b);
  }
  const int32_t k = lim > q + c ? (lim - q + c - 1) / c : 1;
  return q + k * c;
}

// The other particles: those at or after position nleft stay (k_part_left
// writes them); one at p < nleft moves along p -> idx[p] -> ... until it
// lands at or after nleft (the reference's swap sequence,
// RCBForceTree.cxx:647-669), taken a run of equal steps at a time
// (chain_jump).  Positions increase strictly along a chain, so it ends within
// count jumps.
template <int PT>
__global__ void __launch_bounds__(kChunkThreads)
    k_part_right(const float4 *__restrict__ pos, const int32_t *__restrict__ oid, const DNode *nodes,
                 const LevelCtl *ctl, int32_t level, const int32_t *__restrict__ chunk_node,
                 const int32_t *__restrict__ chunk_base, const int32_t *__restrict__ idx,
                 float4 *tpos, int32_t *toid, int32_t *err,
                 int64_t *counters, ChainItem *chains, int64_t chain_cap) {
  chain_enter();
  LevelSpan L;
  if (!level_runs(ctl, level, L) || int32_t(blockIdx.x) >= L.nchunk) return;
  constexpr int NT = kChunkThreads;
  const int tid = threadIdx.x;
  const ChunkRange R = chunk_range<PT>(nodes, chunk_node, chunk_base, L.nb, int32_t(blockIdx.x));
  const DNode &N = nodes[R.node];
  if (N.split_dim < 0) return;
  const int d = N.split_dim;
  const float split = N.xc[d];
  const int32_t is = N.nleft;
  const int32_t *nidx = idx + N.offset;
  if (R.local >= is) return;  // every element here stays (k_part_left)
  // The thread's PT elements take their first kPlainSteps steps in lockstep,
  // so up to PT independent loads are in flight per step (most
  // chains end within a few).  The chains still running go to the level's
  // chain queue (k_part_chains follows them a chain per thread): long chains
  // gather in a few regions of a level, thousands in one chunk.
  constexpr int kPerT = PT;
  const float *key = reinterpret_cast<const float *>(pos + R.begin) + d;
  int32_t q[kPerT];
  unsigned right = 0;
#pragma unroll
  for (int j = 0; j < kPerT; ++j) {
    const int k = tid + j * NT;
    q[j] = R.local + k;
    if (k < R.len && q[j] < is && !(key[4 * k] < split)) right |= 1u << j;
  }
  unsigned active = right;
  bool bad = false;
  for (int32_t step = 0; active && step < kPlainSteps; ++step) {
    int32_t nq[kPerT];
#pragma unroll
    for (int j = 0; j < kPerT; ++j) nq[j] = (active >> j & 1u) ? nidx[q[j]] : q[j];
#pragma unroll
    for (int j = 0; j < kPerT; ++j) {
      if (!(active >> j & 1u)) continue;
      if (nq[j] <= q[j] || nq[j] >= N.count) {  // cannot happen for a valid partition
        bad = true;
        active &= ~(1u << j);
        right &= ~(1u << j);
        continue;
      }
      q[j] = nq[j];
      if (nq[j] >= is) active &= ~(1u << j);
    }
  }
  // one queue reservation per warp
  const int lane = threadIdx.x & 31;
  const int na = __popc(active);
  int incl = na;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  unsigned long long base = 0;
  if (lane == 31 && incl > 0)
    base = atomicAdd((unsigned long long *)&counters[C_CHAINS], (unsigned long long)incl);
  base = __shfl_sync(0xffffffffu, base, 31);
  int64_t slot = int64_t(base) + incl - na;
  // the landed elements, four loads in flight at a time
  const unsigned landed = right & ~active;
#pragma unroll
  for (int j0 = 0; j0 < kPerT; j0 += 4) {
    float4 p[4];
    int32_t o[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (landed >> (j0 + u) & 1u) {
        p[u] = pos[R.begin + tid + (j0 + u) * NT];
        o[u] = oid[R.begin + tid + (j0 + u) * NT];
      }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (landed >> (j0 + u) & 1u) {
        tpos[N.offset + q[j0 + u]] = p[u];
        toid[N.offset + q[j0 + u]] = o[u];
      }
  }
#pragma unroll
  for (int j = 0; j < kPerT; ++j) {
    if (!(active >> j & 1u)) continue;
    if (slot < chain_cap) chains[slot] = ChainItem{q[j], R.node, R.begin + tid + j * NT};
    else bad = true;  // cannot happen: a chain per element at most
    ++slot;
  }
  if (bad) atomicExch(err, 2);
}

// The level's long swap chains, a thread each, a run of equal steps at a
// time (chain_jump); each lands its element.
__global__ void __launch_bounds__(256)
    k_part_chains(const float4 *__restrict__ pos, const int32_t *__restrict__ oid,
                  const DNode *nodes, const LevelCtl *ctl, int32_t level,
                  const ChainItem *__restrict__ chains, int64_t chain_cap, const int64_t *counters, const int32_t *__restrict__ idx,
                  const int32_t *__restrict__ ridx, float4 *tpos, int32_t *toid, int32_t *err) {
  chain_enter();
  LevelSpan L;
  if (!level_runs(ctl, level, L)) return;
  const int64_t nq = min64(counters[C_CHAINS], chain_cap);
  for (int64_t c = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; c < nq;
       c += int64_t(gridDim.x) * blockDim.x) {
    const ChainItem it = chains[c];
    const DNode &N = nodes[it.node];
    const int32_t is = N.nleft, nright = N.count - N.nleft;
    const int32_t *nidx = idx + N.offset, *nridx = ridx + N.offset;
    int32_t qq = it.q;
    bool b = false;
    for (int32_t k = 0; qq < is && k <= N.count && !b; ++k)
      qq = chain_jump(qq, is, nright, nidx, nridx, &b);
    if (b || qq < is || qq >= N.count) {  // cannot happen for a valid partition
      atomicExch(err, 2);
      continue;
    }
    tpos[N.offset + qq] = pos[it.src];
    toid[N.offset + qq] = oid[it.src];
  }
}


// ---------------------------------------------------------------------------
// Tight certification of the centre of mass for the nodes the loose bound
// could not decide (the list that k_level_stats leaves, at most kTightNodes of
// them per level).  The reference's sequential sum s_k = fl(s_{k-1} + t_k)
// differs from the exact sum by sum_k d_k, where the rounding error d_k is
// zero when s_{k-1} and t_k are both multiples of ulp(s_k) (then the exact
// sum is representable), and |d_k| <= ulp(s_k) / 2 otherwise.  ulp(s_k) is
// bounded from the exact prefix sums P_k: |s_k - P_k| is below the loose
// bound, so the binade of s_k lies within that of [P_k - E, P_k + E].  The
// resulting bound B counts only the terms that can round, which for
// coordinates of O(100) is a few thousand times ulp, not n ulp: the quotient
// is then decided on both sides of the bound far more often.  The exact sum
// itself is taken in double-double (error far below B).  Nodes the tight
// bound cannot decide either stay on the list for the sequential sum.
// ---------------------------------------------------------------------------
constexpr int kTightChunk = 2048;   // elements per chunk (8 per thread)
constexpr int kTightThreads = 256;
constexpr int kTightNodes = 64;     // fallback nodes per level taken by this pass
// blocks of the tight-certification passes: two per SM (grid-stride over chunks)
inline unsigned tight_blocks() { return unsigned(2 * sm_count()); }

struct TightChunk {  // per chunk of a listed node
  double hi[4], lo[4];  // double-double sum of the chunk's terms (x, y, z, m)
  double a[4];          // sum of |terms|
  double pre[4];        // approximate prefix sum of the terms before the chunk
};
struct TightNode {
  double hi[4], lo[4], a[4];
  double b[4];          // rounding-error bound of the sequential sum
};

__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e) {
  s = __dadd_rn(a, b);
  const double bb = __dsub_rn(s, a);
  e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
}
__device__ __forceinline__ void dd_add(double &hi, double &lo, double bhi, double blo) {
  double s, e;
  two_sum(hi, bhi, s, e);
  e = __dadd_rn(e, __dadd_rn(lo, blo));
  hi = __dadd_rn(s, e);
  lo = __dsub_rn(e, __dsub_rn(hi, s));
}

// Chunks of the listed nodes in one index space: node f owns chunks
// [cbase[f], cbase[f + 1]).  Computed per block into shared memory.
__device__ int tight_layout(const DNode *nodes, const int32_t *fallback, const int64_t *counters,
                            int32_t *cbase, int32_t skip) {
  const int nt = skip ? 0 : int(min64(counters[C_NFALLBACK], kTightNodes));
  if (threadIdx.x == 0) {
    int32_t run = 0;
    for (int f = 0; f < nt; ++f) {
      cbase[f] = run;
      run += (nodes[fallback[f]].count + kTightChunk - 1) / kTightChunk;
    }
    cbase[nt] = run;
  }
  __syncthreads();
  return nt;
}

__device__ __forceinline__ void terms_of(const float4 &p, double t[4], int lsb[4]) {
  const float fx = fmul_(p.w, p.x), fy = fmul_(p.w, p.y), fz = fmul_(p.w, p.z);
  t[0] = double(fx);
  t[1] = double(fy);
  t[2] = double(fz);
  t[3] = double(p.w);
  lsb[0] = lsb_exp(fx);
  lsb[1] = lsb_exp(fy);
  lsb[2] = lsb_exp(fz);
  lsb[3] = lsb_exp(p.w);
}

// Pass 1: double-double chunk sums; the last block to finish forms each
// node's chunk prefixes and totals.
__global__ void __launch_bounds__(kTightThreads)
    k_cm_tight_sums(const float4 *__restrict__ pos, const DNode *nodes, const int32_t *fallback,
                    int64_t *counters, TightChunk *chunks, TightNode *tn, int32_t skip) {
  __shared__ int32_t cbase[kTightNodes + 1];
  __shared__ double red[kTightThreads / 32][12];
  __shared__ int last;
  const int nt = tight_layout(nodes, fallback, counters, cbase, skip);
  const int total = cbase[nt];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int g = blockIdx.x; g < total; g += gridDim.x) {
    int f = 0;
    while (f + 1 < nt && cbase[f + 1] <= g) ++f;
    const DNode &N = nodes[fallback[f]];
    const int64_t b0 = int64_t(N.offset) + int64_t(g - cbase[f]) * kTightChunk;
    const int64_t e0 = min64(int64_t(N.offset) + N.count, b0 + kTightChunk);
    double hi[4] = {0, 0, 0, 0}, lo[4] = {0, 0, 0, 0}, a[4] = {0, 0, 0, 0};
    for (int64_t i = b0 + threadIdx.x; i < e0; i += kTightThreads) {
      double t[4];
      int lsb[4];
      terms_of(pos[i], t, lsb);
      for (int q = 0; q < 4; ++q) {
        dd_add(hi[q], lo[q], t[q], 0.0);
        a[q] = __dadd_ru(a[q], fabs(t[q]));
      }
    }
    for (int o = 16; o > 0; o >>= 1)
      for (int q = 0; q < 4; ++q) {
        const double oh = __shfl_xor_sync(0xffffffffu, hi[q], o);
        const double ol = __shfl_xor_sync(0xffffffffu, lo[q], o);
        dd_add(hi[q], lo[q], oh, ol);
        a[q] = __dadd_ru(a[q], __shfl_xor_sync(0xffffffffu, a[q], o));
      }
    if (lane == 0)
      for (int q = 0; q < 4; ++q) {
        red[warp][q] = hi[q];
        red[warp][4 + q] = lo[q];
        red[warp][8 + q] = a[q];
      }
    __syncthreads();
    if (threadIdx.x == 0) {
      TightChunk c{};
      for (int q = 0; q < 4; ++q) {
        c.hi[q] = red[0][q];
        c.lo[q] = red[0][4 + q];
        c.a[q] = red[0][8 + q];
      }
      for (int w = 1; w < kTightThreads / 32; ++w)
        for (int q = 0; q < 4; ++q) {
          dd_add(c.hi[q], c.lo[q], red[w][q], red[w][4 + q]);
          c.a[q] = __dadd_ru(c.a[q], red[w][8 + q]);
        }
      chunks[g] = c;
    }
    __syncthreads();
  }
  // the last block to finish forms the prefixes and totals
  __threadfence();
  if (threadIdx.x == 0)
    last = atomicAdd((unsigned long long *)&counters[C_TDONE1], 1ull) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // a node at a time, 64 threads a sum: each adds up a run of chunks, one a sum
  // the 64 runs, and then each goes through its run again for the prefixes (a
  // thread a node took 2.4 of the 2.6 ms of a node of 2.4 M elements)
  constexpr int kRuns = kTightThreads / 4;
  __shared__ double rh[4][kRuns], rl[4][kRuns], ra[4][kRuns];
  const int q = threadIdx.x / kRuns, run = threadIdx.x % kRuns;
  for (int f = 0; f < nt; ++f) {
    const int32_t c0 = cbase[f], nc = cbase[f + 1] - c0;
    const int32_t per = (nc + kRuns - 1) / kRuns;
    const int32_t g0 = c0 + min(nc, run * per), g1 = c0 + min(nc, (run + 1) * per);
    double hi = 0, lo = 0, a = 0;
    for (int32_t g = g0; g < g1; ++g) {
      dd_add(hi, lo, chunks[g].hi[q], chunks[g].lo[q]);
      a = __dadd_ru(a, chunks[g].a[q]);
    }
    rh[q][run] = hi;
    rl[q][run] = lo;
    ra[q][run] = a;
    __syncthreads();
    if (run == 0) {
      hi = lo = a = 0;
      for (int r = 0; r < kRuns && r * per < nc; ++r) {
        const double h = rh[q][r], l = rl[q][r];
        rh[q][r] = hi;  // before the run
        rl[q][r] = lo;
        dd_add(hi, lo, h, l);
        a = __dadd_ru(a, ra[q][r]);
      }
      tn[f].hi[q] = hi;
      tn[f].lo[q] = lo;
      tn[f].a[q] = a;
      tn[f].b[q] = 0.0;
    }
    __syncthreads();
    hi = rh[q][run];
    lo = rl[q][run];
    for (int32_t g = g0; g < g1; ++g) {
      chunks[g].pre[q] = hi + lo;
      dd_add(hi, lo, chunks[g].hi[q], chunks[g].lo[q]);
    }
    __syncthreads();  // the next node's runs take these ones' place
  }
  if (threadIdx.x == 0) counters[C_TDONE1] = 0;
}

// Binade exponent range of the values in [v - e, v + e].
__device__ __forceinline__ void binades(double v, double e, int &emin, int &emax) {
  const double lo = v - e, hi = v + e;
  const double amax = fmax(fabs(lo), fabs(hi));
  emax = amax > 0.0 ? ilogb(amax) : -1074;
  if (lo <= 0.0 && hi >= 0.0) emin = -1074;
  else emin = ilogb(fmin(fabs(lo), fabs(hi)));
}

// Pass 2: the rounding-error bound per listed node; the last block certifies
// and writes the centres of mass (certified nodes leave the list as -1).
__global__ void __launch_bounds__(kTightThreads)
    k_cm_tight_bound(const float4 *__restrict__ pos, DNode *nodes, int32_t *fallback,
                     int64_t *counters, const TightChunk *chunks, TightNode *tn, int32_t skip) {
  __shared__ int32_t cbase[kTightNodes + 1];
  __shared__ float4 el[kTightChunk];
  __shared__ double wsum[kTightThreads / 32][4];
  __shared__ double bred[kTightThreads / 32][4];
  __shared__ int last;
  const int nt = tight_layout(nodes, fallback, counters, cbase, skip);
  const int total = cbase[nt];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kPerT = kTightChunk / kTightThreads;
  for (int g = blockIdx.x; g < total; g += gridDim.x) {
    int f = 0;
    while (f + 1 < nt && cbase[f + 1] <= g) ++f;
    const DNode &N = nodes[fallback[f]];
    const int64_t b0 = int64_t(N.offset) + int64_t(g - cbase[f]) * kTightChunk;
    const int len = int(min64(int64_t(N.offset) + N.count - b0, kTightChunk));
    for (int i = threadIdx.x; i < len; i += kTightThreads) el[i] = pos[b0 + i];
    __syncthreads();
    // this thread's elements [8 tid, 8 tid + 8): local sums, then a block scan
    double loc[4] = {0, 0, 0, 0};
    for (int k = 0; k < kPerT; ++k) {
      const int i = threadIdx.x * kPerT + k;
      if (i < len) {
        double t[4];
        int lsb[4];
        terms_of(el[i], t, lsb);
        for (int q = 0; q < 4; ++q) loc[q] += t[q];
      }
    }
    double inc[4];
    for (int q = 0; q < 4; ++q) {
      inc[q] = loc[q];
      for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, inc[q], o);
        if (lane >= o) inc[q] += v;
      }
      if (lane == 31) wsum[warp][q] = inc[q];
    }
    __syncthreads();
    const TightChunk &C = chunks[g];
    const TightNode &T = tn[f];
    double P[4], E[4], bsum[4] = {0, 0, 0, 0};
    for (int q = 0; q < 4; ++q) {
      double wpre = 0;
      for (int w = 0; w < warp; ++w) wpre += wsum[w][q];
      P[q] = C.pre[q] + wpre + (inc[q] - loc[q]);
      // |s_k - P_k| (sequential error) and the error of this approximate
      // prefix are each below (n + 64) u sum|t|
      E[q] = 4.0 * (double(N.count) + 64.0) * 0x1p-53 * T.a[q];
    }
    for (int k = 0; k < kPerT; ++k) {
      const int i = threadIdx.x * kPerT + k;
      if (i >= len) break;
      double t[4];
      int lsb[4];
      terms_of(el[i], t, lsb);
      const bool first = b0 + i == N.offset;
      for (int q = 0; q < 4; ++q) {
        const double prev = P[q];
        P[q] += t[q];
        if (first || t[q] == 0.0) continue;  // 0 + t and s + 0 are exact
        int pmin, pmax, cmin, cmax;
        binades(prev, E[q], pmin, pmax);
        binades(P[q], E[q], cmin, cmax);
        const int ulp_e = max(cmax, -1022) - 52;  // largest possible ulp(s_k)
        const bool exact = pmin >= cmax && lsb[q] != INT_MIN && lsb[q] >= ulp_e;
        if (!exact) bsum[q] = __dadd_ru(bsum[q], ldexp(1.0, ulp_e - 1));
      }
    }
    for (int q = 0; q < 4; ++q) {
      for (int o = 16; o > 0; o >>= 1) bsum[q] = __dadd_ru(bsum[q], __shfl_xor_sync(0xffffffffu, bsum[q], o));
      if (lane == 0) bred[warp][q] = bsum[q];
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int q = 0; q < 4; ++q) {
        double b = 0;
        for (int w = 0; w < kTightThreads / 32; ++w) b = __dadd_ru(b, bred[w][q]);
        if (b > 0) atomicAdd(&tn[f].b[q], b);
      }
    __syncthreads();
  }
  __threadfence();
  if (threadIdx.x == 0)
    last = atomicAdd((unsigned long long *)&counters[C_TDONE2], 1ull) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int f = threadIdx.x; f < nt; f += blockDim.x) {
    const TightNode &T = tn[f];
    DNode &N = nodes[fallback[f]];
    double sx[4], bx[4];
    for (int q = 0; q < 4; ++q) {
      sx[q] = T.hi[q] + T.lo[q];
      // B (atomics rounded to nearest: slack), the double-double error and
      // the rounding of hi + lo
      bx[q] = T.b[q] * (1.0 + 0x1p-30) + (double(N.count) + 64.0) * 0x1p-98 * T.a[q] +
              fabs(sx[q]) * 0x1p-52;
    }
    float v[3];
    bool ok = true;
    for (int d = 0; d < 3 && ok; ++d) ok = certify(sx[d], bx[d], sx[3], bx[3], &v[d]);
    if (ok) {
      for (int d = 0; d < 3; ++d) N.xc[d] = v[d];
      fallback[f] = -1;
      atomicAdd((unsigned long long *)&counters[C_NTIGHT], 1ull);
    }
  }
  if (threadIdx.x == 0) counters[C_TDONE2] = 0;
}

// The reference's centre of mass for the listed nodes, summed sequentially
// in array order in double (BGQCM.c:186-211).
__global__ void k_cm_fallback(const float4 *__restrict__ pos, DNode *nodes, const int32_t *fallback,
                              const int64_t *counters) {
  const int64_t nf = counters[C_NFALLBACK];
  for (int64_t f = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; f < nf;
       f += int64_t(gridDim.x) * blockDim.x) {
    if (fallback[f] < 0) continue;  // certified by the tight pass
    DNode &N = nodes[fallback[f]];
    double x = 0, y = 0, z = 0, m = 0;
    for (int32_t i = 0; i < N.count; ++i) {
      const float4 p = pos[N.offset + i];
      x = __dadd_rn(x, double(fmul_(p.w, p.x)));
      y = __dadd_rn(y, double(fmul_(p.w, p.y)));
      z = __dadd_rn(z, double(fmul_(p.w, p.z)));
      m = __dadd_rn(m, double(p.w));
    }
    N.xc[0] = __double2float_rn(__ddiv_rn(x, m));
    N.xc[1] = __double2float_rn(__ddiv_rn(y, m));
    N.xc[2] = __double2float_rn(__ddiv_rn(z, m));
  }
}

// The level's centres are all decided: the launches after go on.
__global__ void k_decided(LevelCtl *ctl, int64_t *counters) {
  counters[C_SEQ] += counters[C_NFALLBACK] - counters[C_NTIGHT];
  counters[C_NFALLBACK] = counters[C_NTIGHT] = 0;
  ctl->abort = 0;
}

// ---------------------------------------------------------------------------
// Whole subtrees in one block.  One block per node of at most kSubMax elements
// that the level loop leaves builds that node's entire subtree with its
// positions in shared memory, read once: level by level, each node's
// statistics (box, exact centre-of-mass sums and their certification, the
// reference's sequential sum where the bounds leave it open), the split
// decision, the partition at the centre of mass (left elements to their ranks,
// right elements along the swap chains, pointer jumping for long chains -- the
// reference's swap sequence, RCBForceTree.cxx:623-672) and the children.  What
// a partition moves is each element's 16-bit index, not its 20 bytes; the
// elements are written once, in tree order, at the end.  Every step of a level
// is a few dependent shared-memory accesses: with the elements in L2, and moved
// at every level, a level cost 20-60 us of latency whatever its size (a block of
// 4780 elements took 231 us, 256 blocks of 10 thousand 455 us).
// The level's nodes are shared out to teams of warps: a whole block for one
// node, down to a warp per node on deep levels, kSubBatch nodes at a time.  The
// subtree's nodes go to a scratch region (2 x count records per root, at twice
// the root's element offset) in per-root breadth-first order; k_subtree_place
// later numbers all of them by level and offset.
// ---------------------------------------------------------------------------
constexpr int kSubMax = 8192;        // largest subtree root (elements)
constexpr int kSubThreads = 1024;    // one block per SM
constexpr int kSubWarps = kSubThreads / 32;
constexpr int kSubBatch = 256;       // nodes of a level taken at a time
constexpr int kSubLevel = 512;       // level whose nodes stay in shared memory
constexpr int kSubDepth = 48;        // deepest level below a root; deeper: the level loop
constexpr int kSubBytes = 16 + 3 * 2;  // shared memory an element

// Barrier over the warps of a team: named barrier 1 + team for teams of
// several warps (at most 8 teams), __syncwarp for one warp.
__device__ __forceinline__ void team_sync(int team, int nw) {
  if (nw == 1) {
    __syncwarp();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(nw * 32) : "memory");
  }
}

// Node of the batch in progress.
struct SubNode {
  int32_t lo, count;  // its elements: [lo, lo + count) of the subtree
  int32_t dim;        // split axis, -1: a leaf by size
  int32_t nleft;
  float xc[3];
};

template <bool WIDE>
__global__ void __launch_bounds__(kSubThreads, 1)
    k_subtree(const DNode *__restrict__ nodes, const LevelCtl *ctl, const int2 *__restrict__ roots,
              float4 *pos_a, int32_t *oid_a, const float4 *pos_b, const int32_t *oid_b, DNode *sub,
              int32_t *sub_first, int32_t *hist, int32_t cap, int32_t force_fallback, int32_t nd,
              int64_t *counters) {
  chain_enter();
  extern __shared__ float4 P[];  // positions by input slot; then the 16-bit tables
  uint16_t *cur = reinterpret_cast<uint16_t *>(P + cap);  // input slot by position
  uint16_t *nxt = cur + cap;
  uint16_t *const chain = nxt + cap;  // swap chains: source position of the q-th left element
  __shared__ NodeAcc st[kSubBatch];
  __shared__ NodeAcc wst[kSubWarps];
  __shared__ SubNode H[kSubBatch];
  __shared__ uint16_t lv_lo[2][kSubLevel], lv_count[2][kSubLevel];  // nodes of this level, the next
  __shared__ int wtot[kSubWarps];
  __shared__ int tflag[8];              // per team of several warps: a chain too long / jumping changed
  __shared__ int first[kSubDepth + 2];  // first local node of each depth
  __shared__ int sh_warp[32];
  __shared__ int open_[kSubBatch];      // nodes whose centre is undecided
  __shared__ int nopen, largest;
  if (!ctl->done || ctl->abort) return;
  const int32_t r = int32_t(blockIdx.x);
  if (r >= ctl->nroots) {  // the host launched for the most there can be
    for (int dd = int(threadIdx.x); dd < kSubDepth; dd += kSubThreads)
      hist[int64_t(dd) * gridDim.x + r] = 0;
    return;
  }
  const SumScales S(ctl, WIDE);
  const int2 root = roots[r];
  const int rcnt = nodes[root.x].count;
  const int32_t roff = nodes[root.x].offset;
  DNode *loc = sub + 2 * int64_t(roff);  // this root's 2 x count records
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (rcnt > cap) {  // the launch's shared memory does not hold it
    if (threadIdx.x == 0) atomicExch(reinterpret_cast<int32_t *>(counters + C_ERR), 3);
    return;
  }
  const bool par = root.y != 0;  // the buffer that holds its elements
  const int32_t *src_id = (par ? oid_b : oid_a) + roff;
  constexpr int kPerT = kSubMax / kSubThreads;
  {
    const float4 *src = (par ? pos_b : pos_a) + roff;
#pragma unroll
    for (int u = 0; u < kPerT; ++u) {
      const int i = u * kSubThreads + int(threadIdx.x);
      if (i < rcnt) {
        P[i] = src[i];
        cur[i] = uint16_t(i);
      }
    }
  }
  if (threadIdx.x == 0) {
    lv_lo[0][0] = 0;
    lv_count[0][0] = uint16_t(rcnt);
    first[0] = 0;
    first[1] = 1;
    nopen = 0;
    largest = 0;
  }
  __syncthreads();
  const float *const Pf = reinterpret_cast<const float *>(P);
  int f0 = 0, f1 = 1, depth = 0;
  while (f1 > f0) {
    int base = f1;  // the next level's nodes made so far end here
    const int lv = depth & 1;
    for (int b0 = f0; b0 < f1; b0 += kSubBatch) {
      const int F = min(kSubBatch, f1 - b0);
      int count = 0;
      if (int(threadIdx.x) < F) {
        const int i = b0 - f0 + int(threadIdx.x);
        int lo;
        if (f1 - f0 <= kSubLevel) {
          lo = lv_lo[lv][i];
          count = lv_count[lv][i];
        } else {
          lo = loc[f0 + i].offset - roff;
          count = loc[f0 + i].count;
        }
        H[threadIdx.x] = SubNode{lo, count, -1, 0, {0.f, 0.f, 0.f}};
      }
      if (warp * 32 < F) {
        const int m = __reduce_max_sync(0xffffffffu, count);
        if (lane == 0) atomicMax(&largest, m);
      }
      __syncthreads();
      // teams: the whole block for one node, halving per doubling of the batch
      // to a warp per node from 9 nodes on (at most 8 teams of several warps,
      // named barriers 1-8), and eight lanes per node where there are more than
      // warps and none is large
      const bool oct = F > kSubWarps && largest <= 512;
      int nw = 1;
      if (F <= 8) {
        int p2 = 1;
        while (p2 < F) p2 <<= 1;
        nw = kSubWarps / p2;
      }
      const int team = warp / nw, w0 = team * nw, wi = warp - w0;
      const int sl = oct ? lane & 7 : lane;               // lane of the node's in this warp
      const int lanes = oct ? 8 : 32;                     // of the node in this warp
      const int tl = wi * 32 + sl, TN = oct ? 8 : nw * 32;  // of the node in the block
      const int fstep = oct ? kSubWarps * 4 : kSubWarps / nw;
      const int fbase = oct ? warp * 4 : team, fsub = oct ? lane >> 3 : 0;
      // ---- statistics ----
      for (int fb = fbase; fb < F; fb += fstep) {
        const int f = fb + fsub;
        const int c = f < F ? H[f].count : 0, lo = f < F ? H[f].lo : 0;
        // few enough warps that a lane has about 8 elements: what a warp's
        // reduction costs is some 4 elements a lane
        const int uw = nw == 1 ? 1 : min(nw, max(1, c / 256));
        LaneAcc<WIDE> a;
        a.zero();
        int cnt = 0;
        if (oct) {
          for (int e = sl; e < c; e += 8, ++cnt) a.add(P[cur[lo + e]], S);
          __syncwarp();
          a.template reduce<8>(&st[min(f, kSubBatch - 1)], f < F, cnt, true, S);
        } else if (wi < uw) {
          for (int e = tl; e < c; e += uw * 32, ++cnt) a.add(P[cur[lo + e]], S);
          __syncwarp();
          a.template reduce<32>(uw == 1 ? &st[f] : &wst[warp], true, cnt,
                                32 * ((c + uw * 32 - 1) / (uw * 32)) <= 1023, S);
        }
        if (nw > 1) {
          team_sync(team, nw);
          if (uw > 1 && wi == 0 && lane < kAccWords) {
            long long sum;
            unsigned bits;
            merge_word(wst + w0, uw, lane, &sum, &bits);
            if (lane < 8) reinterpret_cast<long long *>(&st[f])[lane] = sum;
            else reinterpret_cast<unsigned *>(&st[f])[lane + 8] = bits;
          }
          team_sync(team, nw);
        }
      }
      __syncthreads();
      // ---- decisions, a thread per node ----
      if (int(threadIdx.x) < F && H[threadIdx.x].count > 0) {  // an empty root stays as it is
        const int f = threadIdx.x;
        DNode N;
        N.count = H[f].count;
        S.masses(st[f], N.count);
        if (!decide_node(N, st[f], S, force_fallback, nd)) open_[atomicAdd(&nopen, 1)] = f;
        H[f].dim = N.split_dim;
        for (int d = 0; d < 3; ++d) H[f].xc[d] = N.xc[d];
      }
      if (threadIdx.x == 0) largest = 0;
      __syncthreads();
      const int no = nopen;
      if (no > 0) {
        // undecided: a warp each counts the terms that can round (tighten),
        // and where that is not enough lane 0 sums as the reference does
        // (double, in array order, BGQCM.c:181-212)
        for (int k = warp; k < no; k += kSubWarps) {
          const int f = open_[k];
          const int c = H[f].count, lo = H[f].lo;
          float xc[3];
          bool ok = false;
          if (force_fallback == 0 && !S.bad) {
            NodeSums Q = node_sums(st[f], c, S.wide);
            int low[4] = {0, 0, 0, 0};
            const int low_e = S.wide ? 67 : 45, ux = S.c.k - low_e, um = S.m.k - low_e;
            for (int e = lane; e < c; e += 32) {
              const float4 p = P[cur[lo + e]];
              low[0] += lsb_exp(fmul_(p.w, p.x)) < last_place(Q.abs[0]) + ux;
              low[1] += lsb_exp(fmul_(p.w, p.y)) < last_place(Q.abs[1]) + ux;
              low[2] += lsb_exp(fmul_(p.w, p.z)) < last_place(Q.abs[2]) + ux;
              low[3] += lsb_exp(p.w) < last_place(Q.abs[3]) + um;
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 4; ++q) low[q] = __reduce_add_sync(0xffffffffu, low[q]);
            tighten(Q, low, st[f], c);
            ok = quotients(Q, S.c.k, S.m.k, xc);
          }
          if (lane == 0) {
            if (!ok) {
              double x = 0, y = 0, z = 0, m = 0;
              for (int i = 0; i < c; ++i) {
                const float4 p = P[cur[lo + i]];
                x = __dadd_rn(x, double(fmul_(p.w, p.x)));
                y = __dadd_rn(y, double(fmul_(p.w, p.y)));
                z = __dadd_rn(z, double(fmul_(p.w, p.z)));
                m = __dadd_rn(m, double(p.w));
              }
              xc[0] = __double2float_rn(__ddiv_rn(x, m));
              xc[1] = __double2float_rn(__ddiv_rn(y, m));
              xc[2] = __double2float_rn(__ddiv_rn(z, m));
              atomicAdd((unsigned long long *)&counters[C_SUBFB], 1ull);
            }
            for (int d = 0; d < 3; ++d) H[f].xc[d] = xc[d];
          }
        }
        __syncthreads();
        if (threadIdx.x == 0) nopen = 0;
      }
      // ---- partition at the centre of mass ----
      for (int fb = fbase; fb < F; fb += fstep) {
        const int f = fb + fsub;
        const bool have = f < F;
        const int c = have ? H[f].count : 0, lo = have ? H[f].lo : 0, dim = have ? H[f].dim : -1;
        const uint16_t *const in = cur + lo;
        uint16_t *const out = nxt + lo, *const ch = chain + lo;
        // a leaf: its order into the other table as well
        if (dim < 0)
          for (int e = tl; e < c; e += TN) out[e] = in[e];
        if (!oct && dim < 0) continue;  // the whole team
        const int d = max(dim, 0);
        const float split = have ? H[f].xc[d] : 0.f;
        const int cp = dim < 0 ? 0 : c;  // elements to partition
        const int share = oct ? cp : (((cp + nw - 1) / nw) + 31) & ~31;
        const int beg = oct ? 0 : min(cp, wi * share), end = min(cp, beg + share);
        // the same number of steps for the lanes of a warp
        const int steps = __reduce_max_sync(0xffffffffu, (end - beg + lanes - 1) / lanes);
        const int shift = oct ? lane & 24 : 0;
        const unsigned mask = oct ? 0xffu : 0xffffffffu, below = (1u << sl) - 1u;
        int rank = 0, nleft = 0;
        for (int k = 0; k < steps; ++k) {
          const int e = beg + k * lanes + sl;
          const unsigned bal = __ballot_sync(0xffffffffu, e < end && Pf[4 * in[e] + d] < split);
          nleft += __popc(bal >> shift & mask);
        }
        if (nw > 1) {
          const int mine = nleft;
          if (lane == 0) wtot[warp] = mine;
          if (tl == 0) tflag[team] = 0;
          team_sync(team, nw);
          // the team's totals, a lane a warp: inclusive scan
          int v = lane < nw ? wtot[w0 + lane] : 0;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
          }
          nleft = __shfl_sync(0xffffffffu, v, 31);
          rank = __shfl_sync(0xffffffffu, v, wi) - mine;
        }
        for (int k = 0; k < steps; ++k) {
          const int e = beg + k * lanes + sl;
          const bool on = e < end;
          const int s = on ? in[e] : 0;
          const bool l = on && Pf[4 * s + d] < split;
          const unsigned bal = __ballot_sync(0xffffffffu, l) >> shift & mask;
          if (l) {
            const int q = rank + __popc(bal & below);
            out[q] = uint16_t(s);
            ch[q] = uint16_t(e);
          } else if (on && e >= nleft) {
            out[e] = uint16_t(s);  // a right element at or after nleft: no swap touches it
          }
          rank += __popc(bal);
        }
        team_sync(team, nw);
        bool any_long = false, bad = false;
        for (int e = tl; e < nleft; e += TN) {
          const int s = in[e];
          if (Pf[4 * s + d] < split) continue;
          int q = e, hops = 0;
          while (q < nleft && hops < kChainSteps) {
            const int nq = ch[q];
            if (nq <= q || nq >= c) {  // cannot happen for a valid partition
              bad = true;
              break;
            }
            q = nq;
            ++hops;
          }
          if (q < nleft) any_long = !bad;
          else out[q] = uint16_t(s);
        }
        if (bad) atomicExch(reinterpret_cast<int32_t *>(counters + C_ERR), 2);
        __syncwarp();
        bool jump = __any_sync(0xffffffffu, any_long);
        if (nw > 1) {
          if (jump && lane == 0) tflag[team] = 1;
          team_sync(team, nw);
          jump = tflag[team] != 0;
        }
        if (jump) {
          // pointer jumping: afterwards ch[q] is the end of the chain through q
          // (each entry moves along its own chain, so every read sees a point of
          // that chain): log2(count) + 1 rounds
          for (int round = 0; round < 40; ++round) {
            team_sync(team, nw);
            if (nw > 1 && tl == 0) tflag[team] = 0;
            team_sync(team, nw);
            bool changed = false;
            for (int q = tl; q < nleft; q += TN) {
              const int j = ch[q];
              if (j != q && j < nleft) {  // j == q: a left element no swap moves
                ch[q] = ch[j];
                changed = true;
              }
            }
            __syncwarp();
            changed = __any_sync(0xffffffffu, changed);
            if (nw > 1) {
              if (changed && lane == 0) tflag[team] = 1;
              team_sync(team, nw);
              changed = tflag[team] != 0;
            }
            if (!changed) break;
          }
          team_sync(team, nw);
          for (int e = tl; e < nleft; e += TN) {
            const int s = in[e];
            if (Pf[4 * s + d] < split) continue;
            const int q = ch[e];
            if (q < nleft || q >= c) {  // cannot happen for a valid partition
              atomicExch(reinterpret_cast<int32_t *>(counters + C_ERR), 2);
              continue;
            }
            out[q] = uint16_t(s);
          }
        }
        if (have && dim >= 0 && tl == 0) H[f].nleft = nleft;
        team_sync(team, nw);
      }
      __syncthreads();
      // ---- records and children: two per node split into two non-empty parts ----
      const int f = int(threadIdx.x);
      int flag = 0;
      if (f < F && H[f].dim >= 0) flag = H[f].nleft > 0 && H[f].nleft < H[f].count;
      int tot = 0;
      const int rk = block_excl_scan(flag, sh_warp, &tot);
      if (f < F) {
        DNode N;
        N.count = H[f].count;
        N.offset = roff + H[f].lo;
        const int cl = base + 2 * rk;
        N.cl = flag ? cl : 0;
        N.cr = flag ? cl + 1 : 0;
        for (int d = 0; d < 3; ++d) {
          N.xmin[d] = H[f].count > 0 ? o2f(st[f].lo[d]) : 0.f;
          N.xmax[d] = H[f].count > 0 ? o2f(st[f].hi[d]) : 0.f;
          N.xc[d] = H[f].xc[d];
        }
        N.tdr = 0.f;
        N.split_dim = H[f].dim;
        N.nleft = H[f].nleft;
        if (H[f].count == 0) {  // an empty set's root keeps the caller's box
          N = nodes[root.x];
          N.cl = N.cr = 0;
        }
        const int4 *src = reinterpret_cast<const int4 *>(&N);
        int4 *out = reinterpret_cast<int4 *>(&loc[b0 + f]);
#pragma unroll
        for (int w = 0; w < 4; ++w) out[w] = src[w];
        if (flag) {
          // the children's extents: for the next level's headers
          const int n0 = H[f].nleft, n1 = H[f].count - n0, i = cl - f1;
          *reinterpret_cast<int2 *>(&loc[cl]) = make_int2(n0, N.offset);
          *reinterpret_cast<int2 *>(&loc[cl + 1]) = make_int2(n1, N.offset + n0);
          if (i + 1 < kSubLevel) {
            lv_lo[lv ^ 1][i] = uint16_t(H[f].lo);
            lv_count[lv ^ 1][i] = uint16_t(n0);
            lv_lo[lv ^ 1][i + 1] = uint16_t(H[f].lo + n0);
            lv_count[lv ^ 1][i + 1] = uint16_t(n1);
          }
        }
      }
      base += 2 * tot;
      __syncthreads();
    }
    f0 = f1;
    f1 = base;
    ++depth;
    if (threadIdx.x == 0) first[depth + 1] = f1;
    if (f1 > f0 && depth >= kSubDepth) {  // deeper than the bookkeeping holds
      if (threadIdx.x == 0) atomicExch(reinterpret_cast<int32_t *>(counters + C_ERR), 4);
      return;
    }
    uint16_t *const t = cur;
    cur = nxt;
    nxt = t;
    __syncthreads();
  }
  // per depth: first local node and count (depth 0 is the root)
  for (int dd = int(threadIdx.x); dd <= kSubDepth + 1; dd += kSubThreads)
    sub_first[int64_t(r) * (kSubDepth + 2) + dd] = dd <= depth + 1 ? first[min(dd, depth + 1)] : f1;
  for (int dd = 1 + int(threadIdx.x); dd <= kSubDepth; dd += kSubThreads)
    hist[int64_t(dd - 1) * gridDim.x + r] = dd <= depth ? first[dd + 1] - first[dd] : 0;
  // the elements in tree order, into the first buffer (which may be the one
  // read: the ids are gathered before any is written)
  int32_t ids[kPerT];
#pragma unroll
  for (int u = 0; u < kPerT; ++u) {
    const int i = u * kSubThreads + int(threadIdx.x);
    ids[u] = i < rcnt ? src_id[cur[i]] : 0;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kPerT; ++u) {
    const int i = u * kSubThreads + int(threadIdx.x);
    if (i < rcnt) {
      pos_a[roff + i] = P[cur[i]];
      oid_a[roff + i] = ids[u];
    }
  }
}

// Whether every subtree root's records are there: a block of k_subtree that
// gives up (C_ERR) leaves its row of sub_first and its column of hist as an
// earlier build, of another shape, left them, and the host looks only after the
// kernels below have run.
__device__ __forceinline__ bool subtrees_made(const LevelCtl *ctl, const int64_t *counters) {
  return ctl->done && !ctl->abort && counters[C_ERR] == 0;
}

// Per depth below the subtree roots (a block each): every root's first node
// among that depth's (exclusive scan over the roots) and the depth's total.
__global__ void __launch_bounds__(kScanThreads)
    k_subtree_scan(const LevelCtl *ctl, const int64_t *counters, int32_t *hist, int32_t max_roots,
                   int64_t *tot) {
  chain_enter();
  __shared__ int sh_warp[32];
  int32_t *row = hist + int64_t(blockIdx.x) * max_roots;
  const int32_t nr = subtrees_made(ctl, counters) ? ctl->nroots : 0;
  int run = 0;
  for (int32_t r0 = 0; r0 < nr; r0 += kScanThreads) {
    const int32_t r = r0 + int32_t(threadIdx.x);
    int total;
    const int ex = block_excl_scan(r < nr ? row[r] : 0, sh_warp, &total);
    if (r < nr) row[r] = run + ex;
    run += total;
  }
  if (threadIdx.x == 0) tot[blockIdx.x] = run;
}

// Copies every subtree node to its place after the level loop's nodes: by
// depth below its root, then by root, then in the block's breadth-first order,
// so a node always comes after its parent.  pos holds the scans of
// k_subtree_scan.
// Does nothing when the node array is too small (the host grows it and
// launches this again).
__global__ void __launch_bounds__(256)
    k_subtree_place(DNode *nodes, const LevelCtl *ctl, const int64_t *counters,
                    const int2 *__restrict__ roots, const DNode *sub, const int32_t *sub_first,
                    const int32_t *pos, int32_t max_roots, const int64_t *tot, int64_t node_cap) {
  chain_enter();
  __shared__ int fs[kSubDepth + 2];
  __shared__ int64_t base[kSubDepth + 1];
  const int32_t r = int32_t(blockIdx.x);
  if (!subtrees_made(ctl, counters) || r >= ctl->nroots) return;
  const int32_t root = roots[r].x;
  for (int dd = threadIdx.x; dd <= kSubDepth + 1; dd += blockDim.x)
    fs[dd] = sub_first[int64_t(r) * (kSubDepth + 2) + dd];
  if (threadIdx.x == 0) {
    int64_t at = ctl->node_end;
    for (int dd = 0; dd < kSubDepth; ++dd) {
      base[dd] = at;
      at += tot[dd];
    }
    base[kSubDepth] = at;
  }
  __syncthreads();
  if (base[kSubDepth] > node_cap) return;
  const int32_t roff = nodes[root].offset;
  const DNode *loc = sub + 2 * int64_t(roff);
  const int total = fs[kSubDepth + 1];
  auto depth_of = [&](int j) {
    int dd = 1;
    while (dd <= kSubDepth && fs[dd + 1] <= j) ++dd;
    return dd;
  };
  auto global = [&](int j, int dd) {
    return int32_t(base[dd - 1] + pos[int64_t(dd - 1) * max_roots + r] + (j - fs[dd]));
  };
  for (int j = 1 + int(threadIdx.x); j < total; j += blockDim.x) {
    const int dd = depth_of(j);
    DNode N = loc[j];
    if (N.cl) {
      N.cl = global(N.cl, dd + 1);
      N.cr = global(N.cr, dd + 1);
    }
    nodes[global(j, dd)] = N;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    DNode N = loc[0];
    if (N.cl) {
      N.cl = global(N.cl, 1);
      N.cr = global(N.cr, 1);
    }
    nodes[root] = N;
  }
}

// ---------------------------------------------------------------------------
// Pseudo-particles (RCBForceTree.cxx:519-569, 788-800, 856-889)
// ---------------------------------------------------------------------------
// The 12-point design (RCBForceTree.cxx:227-272): the icosahedron's vertices
// (0, +-b, +-a) and their cyclic permutations, a = 0.525731112119134,
// b = 0.85065080835204, in the reference's order.  Fixed: every tree reads
// it, whatever its point count (a monopole's one point sits at xc, offset 0).
#define HSR_IA 0.525731112119134f
#define HSR_IB 0.85065080835204f
__constant__ float c_design[12][3] = {
    {0, HSR_IB, HSR_IA},   {0, HSR_IB, -HSR_IA},  {HSR_IA, 0, HSR_IB},   {-HSR_IA, 0, HSR_IB},
    {HSR_IB, HSR_IA, 0},   {-HSR_IB, HSR_IA, 0},  {0, -HSR_IB, -HSR_IA}, {0, -HSR_IB, HSR_IA},
    {-HSR_IA, 0, -HSR_IB}, {HSR_IA, 0, -HSR_IB},  {-HSR_IB, -HSR_IA, 0}, {HSR_IB, -HSR_IA, 0}};
#undef HSR_IA
#undef HSR_IB

__device__ __forceinline__ float pptdr_(const DNode &t) {
  return smin_(fsub_(t.xmax[0], t.xc[0]),
               smin_(fsub_(t.xmax[1], t.xc[1]),
                     smin_(fsub_(t.xmax[2], t.xc[2]),
                           smin_(fsub_(t.xc[0], t.xmin[0]),
                                 smin_(fsub_(t.xc[1], t.xmin[1]), fsub_(t.xc[2], t.xmin[2]))))));
}

// Design point j of a node: its centre of mass plus tdr times the unit point
// (offset 0 for the monopole's one point).
template <int K>
__device__ __forceinline__ void pppt_(int j, float tdr, const float *xc, float &x, float &y,
                                      float &z) {
  const float ex = K == 12 ? c_design[j][0] : 0.f, ey = K == 12 ? c_design[j][1] : 0.f,
              ez = K == 12 ? c_design[j][2] : 0.f;
  x = fadd_(fmul_(tdr, ex), xc[0]);
  y = fadd_(fmul_(tdr, ey), xc[1]);
  z = fadd_(fmul_(tdr, ez), xc[2]);
}

// One pseudo-particle's mass over its node's sources, added in source order.
template <int K>
struct PointMass {
  float xj, yj, zj, rj2, rj, m;
  __device__ __forceinline__ void start(int j, float tdr, const float *xc) {
    float x, y, z;
    pppt_<K>(j, tdr, xc, x, y, z);
    xj = fsub_(x, xc[0]);
    yj = fsub_(y, xc[1]);
    zj = fsub_(z, xc[2]);
    rj2 = norm2_(xj, yj, zj);
    rj = __fsqrt_rn(rj2);
    m = 0.f;
  }
  __device__ __forceinline__ void add(float sx, float sy, float sz, float sm, float tdr,
                                      const float *xc) {
    const float xi = fsub_(sx, xc[0]), yi = fsub_(sy, xc[1]), zi = fsub_(sz, xc[2]);
    const float ri = __fsqrt_rn(norm2_(xi, yi, zi));
    float odr1 = 0.f, odr2 = 0.f;
    if (rj2 != 0.f) {
      const float aij = __fdiv_rn(fadd_(fadd_(fmul_(xi, xj), fmul_(yi, yj)), fmul_(zi, zj)),
                                  fmul_(ri, rj));
      const float rt = __fdiv_rn(ri, tdr);
      odr1 = fmul_(fmul_(3.0f / K, rt), aij);
      const float a = fmul_(fmul_(5.0f / K, rt), rt);
      const float b = fsub_(fmul_(fmul_(3.0f, aij), aij), 1.0f);
      // the reference multiplies a * 0.5 * b in double and rounds once: a
      // product of two floats is exact there, and so is half of b here (b is
      // 0 or far above the subnormals)
      odr2 = fmul_(a, fmul_(0.5f, b));
    }
    m = fadd_(m, fmul_(sm, fadd_(fadd_(1.0f / K, odr1), odr2)));
  }
};

// The leaf test of calcInternodeForces (RCBForceTree.cxx:1150-1197): leaves
// with a face of their box inside the force box on every axis.
__device__ __forceinline__ bool leaf_in_force_box(const DNode &T, const TreeConfig &cfg) {
  bool inside = T.count > 0;
  for (int i = 0; i < 3; ++i)
    inside &= (T.xmax[i] < cfg.max_force[i] && T.xmax[i] > cfg.min_force[i]) ||
              (T.xmin[i] < cfg.max_force[i] && T.xmin[i] > cfg.min_force[i]);
  return inside;
}

// Links upward: up[t] = (parent, 0) of every node; the arrival counter's bit 8
// marks a left child (its sibling is t + 1: children are made in pairs).
constexpr int kLeftChild = 0x100;
__global__ void k_links(const DNode *nodes, int32_t nnodes, int2 *up) {
  chain_enter();
  const int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nnodes) return;
  const int32_t cl = nodes[t].cl;
  if (t == 0) up[0] = make_int2(-1, 0);
  if (cl > 0) {
    up[cl] = make_int2(t, kLeftChild);
    up[cl + 1] = make_int2(t, 0);
  }
}

// Every node's pseudo-particles (masses into ppm, points into the position
// table), tdr and the number of processed leaves below it, from the leaves up
// in one launch: a warp per leaf does its leaf, and whichever warp arrives
// second at a node goes on with it.  Lane j < K holds point j and adds the
// node's sources in the reference's order (all of a leaf's particles, or each
// child's particles or points, left child first), so the points of a node run
// in parallel and no level waits for a launch of its own.  A monopole leaf's
// mass is the sequential float sum of its particles' masses, loaded 32 at a
// time and added in order from shuffles (monopole_climb).  (With one lane a node and a launch a
// level, 12-point masses took 3.6 of the 9.8 ms of a clustered 48^3 forward and
// adjoint, and a 32^3 kick's monopoles 52 us.)
// A monopole's climb loads the parent's record and links, and the sibling's
// count, while its own results become visible, and has its own mass in a
// register, so a step waits for the fence, the arrival and the sibling's mass
// only (a kick of 4780 particles: 365 to 348 us, of 67,836: 523 to 510).
__device__ __forceinline__ void monopole_climb(DNode *nodes, int32_t nnodes, int2 *up,
                                               const float4 *__restrict__ pos, float *ppm,
                                               float4 *table, int64_t n, const TreeConfig &cfg,
                                               int32_t *processed, int32_t t, int lane) {
  const unsigned full = 0xffffffffu;
  DNode T = nodes[t];
  int2 U = up[t];
  int32_t below = leaf_in_force_box(T, cfg) ? 1 : 0;
  float m = 0.f;
  // a leaf's mass in its particles' order; a leaf left by a failed split keeps
  // zero (its children are empty)
  if (T.count <= cfg.nd && T.count > 1) {
    const float *w = reinterpret_cast<const float *>(pos + T.offset) + 3;
    for (int32_t i0 = 0; i0 < T.count; i0 += 32) {
      const float v = i0 + lane < T.count ? w[4 * (i0 + lane)] : 0.f;
      const int nv = min(32, T.count - i0);
      for (int i = 0; i < nv; ++i) m = fadd_(m, __shfl_sync(full, v, i));
    }
  }
  for (int climbed = 0; climbed <= nnodes; ++climbed) {
    const int32_t parent = U.x;
    const bool left = U.y & kLeftChild;
    const int32_t sib = left ? t + 1 : t - 1;
    DNode TP{};
    int2 UP = make_int2(-1, 0);
    int32_t scount = 0, soff = 0;
    if (t != 0) {
      TP = nodes[parent];
      UP = up[parent];
      scount = nodes[sib].count;
      soff = nodes[sib].offset;
    }
    if (lane == 0) {
      const float tdr = fmul_(cfg.ppc, pptdr_(T));
      float x, y, z;
      pppt_<1>(0, tdr, T.xc, x, y, z);
      ppm[t] = m;
      table[n + t] = make_float4(x, y, z, m);
      nodes[t].tdr = tdr;
      processed[t] = below;
    }
    if (t == 0) return;
    __threadfence();
    __syncwarp();
    int arrived = 0;
    if (lane == 0) arrived = atomicAdd(&up[parent].y, 1) & 0xff;
    if (__shfl_sync(full, arrived, 0) == 0) return;  // the sibling's warp goes on
    __threadfence();
    // the children's masses, left first; a child of one particle is that
    // particle, one of none adds nothing
    const float mine = T.count == 1 ? pos[T.offset].w : m;
    const float other = scount > 1 ? __ldcg(ppm + sib) : (scount == 1 ? pos[soff].w : 0.f);
    below += __ldcg(processed + sib);
    const float l = left ? mine : other, r = left ? other : mine;
    const int32_t lc = left ? T.count : scount, rc = left ? scount : T.count;
    m = 0.f;
    if (lc > 0) m = fadd_(m, l);
    if (rc > 0) m = fadd_(m, r);
    t = parent;
    T = TP;
    U = UP;
  }
}

template <int K>
__global__ void __launch_bounds__(128)
    k_pseudo_up(DNode *nodes, int32_t nnodes, int2 *up, const float4 *__restrict__ pos, float *ppm,
                float4 *table, int64_t n, TreeConfig cfg, int32_t *processed) {
  chain_enter();
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int32_t t = int32_t((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
  if (t >= nnodes) return;  // whole warps
  if (nodes[t].cl != 0) return;
  if (K == 1) {
    monopole_climb(nodes, nnodes, up, pos, ppm, table, n, cfg, processed, t, lane);
    return;
  }
  for (int climbed = 0; climbed <= nnodes; ++climbed) {
    const DNode T = nodes[t];
    const float tdr = fmul_(cfg.ppc, pptdr_(T));
    const int j = lane < K ? lane : 0;
    PointMass<K> P;
    P.start(j, tdr, T.xc);
    int32_t below = 0;  // processed leaves
    if (T.cl == 0) {
      below = leaf_in_force_box(T, cfg) ? 1 : 0;
      // masses from its particles when it has more than K; a leaf left by a
      // failed split keeps zero masses (its children are empty)
      if (T.count <= cfg.nd && T.count > K) {
        const float4 *p = pos + T.offset;
#pragma unroll 4
        for (int32_t i = 0; i < T.count; ++i) {
          const float4 q = p[i];
          P.add(q.x, q.y, q.z, q.w, tdr, T.xc);
        }
      }
    } else {
      for (int s = 0; s < 2; ++s) {
        const int32_t c = T.cl + s;
        const DNode &C = nodes[c];
        const int32_t cc = C.count;
        below += __ldcg(processed + c);
        if (cc <= K) {
          const float4 *p = pos + C.offset;
          for (int32_t i = 0; i < cc; ++i) {
            const float4 q = p[i];
            P.add(q.x, q.y, q.z, q.w, tdr, T.xc);
          }
        } else {
          const float ctdr = __ldcg(&C.tdr);
          const float cxc[3] = {C.xc[0], C.xc[1], C.xc[2]};
#pragma unroll
          for (int i = 0; i < K; ++i) {
            float x, y, z;
            pppt_<K>(i, ctdr, cxc, x, y, z);
            P.add(x, y, z, __ldcg(ppm + int64_t(c) * K + i), tdr, T.xc);
          }
        }
      }
    }
    if (lane < K) {
      float x, y, z;
      pppt_<K>(j, tdr, T.xc, x, y, z);
      ppm[int64_t(t) * K + j] = P.m;
      table[n + int64_t(t) * K + j] = make_float4(x, y, z, P.m);
    }
    if (lane == 0) {
      nodes[t].tdr = tdr;
      processed[t] = below;
    }
    if (t == 0) return;
    const int32_t parent = up[t].x;
    __threadfence();
    __syncwarp();
    int arrived = 0;
    if (lane == 0) arrived = atomicAdd(&up[parent].y, 1) & 0xff;
    if (__shfl_sync(full, arrived, 0) == 0) return;  // the sibling's warp goes on
    __threadfence();
    t = parent;
  }
}

// ---------------------------------------------------------------------------
// Processed leaves, in the reference's DFS order, which visits the right child
// first: a leaf's rank is the number of processed leaves right of its path,
// counted on the way up.
// ---------------------------------------------------------------------------
__global__ void k_leaf_rank(const DNode *nodes, int32_t nnodes, const int2 *up,
                            const int32_t *processed, int32_t *leaf_ids, int64_t *counters) {
  chain_enter();
  const int32_t t0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (t0 >= nnodes) return;
  if (t0 == 0) counters[C_NLEAF] = processed[0];
  if (nodes[t0].cl != 0 || processed[t0] == 0) return;
  int32_t rank = 0, t = t0;
  for (int climbed = 0; t > 0 && climbed <= nnodes; ++climbed) {
    const int2 u = up[t];
    if (u.y & kLeftChild) rank += processed[t + 1];
    t = u.x;
  }
  leaf_ids[rank] = t0;
}

// ---------------------------------------------------------------------------
// Interaction lists (calcInternodeForce, RCBForceTree.cxx:923-1144), a warp
// per processed leaf.
//
// The reference's walk is a depth-first search whose emissions must keep their
// order.  One lane taking one node at a time is a chain of dependent node
// loads (116-260 of them a leaf at leaf sizes 128-32), so the warp takes the
// top 32 stack entries at once: every lane decides its node, and the results
// go back in stack order -- an interaction in place as a finished entry, two
// children in place of their parent -- while the finished entries ahead of
// the first expanded one, whose place in the list is then known, leave the
// stack for the list.  11-18 steps a leaf instead of 116-260.
// ---------------------------------------------------------------------------
constexpr int kWalkWarps = 4;
constexpr int kWalkCap = 640;      // stack entries a leaf; the window narrows as it
constexpr int kWalkReserve = 256;  // fills, to one node at a time over the last 256

// The leaves are the first counters[C_NLEAF] of leaf_ids (max_leaves bounds
// them: the host need not wait for their number).
// MODE 1, leaves with more than `room` segments only: writes the segments at
// seg_base / list_base; 2: counts (segments and
// entries per leaf) and writes the first `room` segments (start, count) of
// each leaf into its own region, flagging leaves with more in
// counters[C_SEGOVF].
template <int MODE>
__global__ void __launch_bounds__(32 * kWalkWarps)
    k_walk(const DNode *__restrict__ nodes, int32_t nnodes, const int32_t *leaf_ids,
           int64_t max_leaves, TreeConfig cfg, int64_t n, int64_t *seg_cnt, int64_t *list_len,
           const int64_t *seg_base, const int64_t *list_base, SegDesc *segs, int2 *local, int room,
           int32_t *err, int64_t *counters) {
  chain_enter();
  static_assert(MODE == 1 || MODE == 2, "walk mode");
  // entries: a node still to decide (x = node, y = 0, or -1 for a child of an
  // ancestor of the leaf, which no distance test drops), or a finished segment
  // (x = start, y = count > 0)
  __shared__ int2 stack_[kWalkWarps][kWalkCap];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
  const int64_t li = int64_t(blockIdx.x) * kWalkWarps + w;
  if (li >= max_leaves) return;  // whole warps
  if (li >= counters[C_NLEAF]) {
    if (MODE == 2 && lane == 0) seg_cnt[li] = list_len[li] = 0;
    return;
  }
  if (MODE == 1 && seg_cnt[li] <= room) return;  // its region holds them
  int2 *const st = stack_[w];
  const int32_t tl = leaf_ids[li];
  const DNode T = nodes[tl];
  const float fsr = cfg.fsrrmax;
  const float fsr2 = fmul_(fsr, fsr);
  const float tan_oa = cfg.tan_oa;
  const int k = cfg.tdpts;
  int64_t nseg = 0, len = 0;
  int2 *const region = local + li * room;
  const int64_t sb = MODE == 1 ? seg_base[li] : 0, lb = MODE == 1 ? list_base[li] : 0;
  // the lanes' segments (start, count), in lane order, where `on`
  auto emit = [&](bool on, int32_t start, int32_t count) {
    const unsigned m = __ballot_sync(full, on);
    const int64_t q = nseg + __popc(m & below);
    int incl = on ? count : 0;  // the segments of one step are disjoint: at most n entries
    if (MODE == 1) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += v;
      }
      if (on) segs[sb + q] = SegDesc{start, count, lb + len + incl - count};
      len += __shfl_sync(full, incl, 31);
    } else {
      if (on && q < room) region[q] = make_int2(start, count);
      len += __reduce_add_sync(full, incl);
    }
    nseg += __popc(m);
  };
  if (lane == 0) st[0] = make_int2(0, -1);
  __syncwarp();
  int sp = 1;
  int64_t visited = 0;
  while (sp > 0) {
    const int width = min(min(32, sp), max(1, kWalkCap - kWalkReserve - sp));
    int nout = 0;
    int2 o0 = make_int2(0, 0), o1 = o0;  // this lane's results, in list order
    bool expand = false, fresh = false, bad = false;
    if (lane < width) {
      const int2 e = st[sp - 1 - lane];
      if (e.y > 0) {
        nout = 1;
        o0 = e;
      } else {
        const int32_t t = e.x;
        fresh = true;
        bad = t < 0 || t >= nnodes;
        DNode Q{};
        if (!bad) {
          Q = nodes[t];
          bad = Q.cl >= nnodes || Q.cr >= nnodes;
        }
        bool go = !bad && Q.count > 0;
        const bool anc =
            t != tl && Q.offset <= T.offset && T.offset + T.count <= Q.offset + Q.count;
        if (go && !anc && e.y == 0) {
          // per-axis gap between the target leaf's box and the node's
          for (int i = 0; i < 3; ++i) {
            float dist = 0.f;
            if (T.xmax[i] < Q.xmin[i]) dist = fsub_(Q.xmin[i], T.xmax[i]);
            else if (T.xmin[i] > Q.xmax[i]) dist = fsub_(T.xmin[i], Q.xmax[i]);
            if (dist > fsr) go = false;
          }
        }
        if (go) {
          bool big = true;
          float dist2 = 0.f;
          if (!anc) {
            const float dx = fsub_(Q.xc[0], T.xc[0]), dy = fsub_(Q.xc[1], T.xc[1]),
                        dz = fsub_(Q.xc[2], T.xc[2]);
            dist2 = norm2_(dx, dy, dz);
            const float sx = fsub_(Q.xmax[0], Q.xmin[0]), sy = fsub_(Q.xmax[1], Q.xmin[1]),
                        sz = fsub_(Q.xmax[2], Q.xmin[2]);
            const float l2 = smin_(fmul_(sx, sx), smin_(fmul_(sy, sy), fmul_(sz, sz)));
            const float dtt2 = fmul_(fmul_(dist2, tan_oa), tan_oa);
            big = l2 > dtt2;
            for (int i = 0; i < 2 && !big; ++i)
              for (int j = 0; j < 2 && !big; ++j) {
                const float x1 = fsub_((i == 0 ? Q.xmin : Q.xmax)[0], T.xc[0]);
                const float y1 = fsub_((j == 0 ? Q.xmin : Q.xmax)[1], T.xc[1]);
                const float z1 = fsub_(Q.xmin[2], T.xc[2]);
                const float x2 = fsub_((i == 0 ? Q.xmax : Q.xmin)[0], T.xc[0]);
                const float y2 = fsub_((j == 0 ? Q.xmax : Q.xmin)[1], T.xc[1]);
                const float z2 = fsub_(Q.xmax[2], T.xc[2]);
                big = norm2_(fsub_(x1, x2), fsub_(y1, y2), fsub_(z1, z2)) > dtt2;
              }
          }
          if (anc || (big && (Q.cl != 0 || Q.cr != 0))) {
            // the right child first; the leaf itself comes last of all
            const int fl = anc ? -1 : 0;
            if (Q.cr > 0 && !(anc && Q.cr == tl)) {
              o0 = make_int2(Q.cr, fl);
              nout = 1;
            }
            if (Q.cl > 0 && !(anc && Q.cl == tl)) {
              (nout ? o1 : o0) = make_int2(Q.cl, fl);
              ++nout;
            }
            expand = nout > 0;
          } else if (big || !(dist2 > fsr2)) {  // (a node without mass: NaN)
            nout = 1;
            o0 = big || Q.count <= k ? make_int2(Q.offset, Q.count)
                                     : make_int2(int32_t(n + int64_t(t) * k), k);
          }
        }
      }
    }
    if (__any_sync(full, bad)) {
      if (bad) atomicExch(err, 3);
      break;
    }
    visited += __popc(__ballot_sync(full, fresh));
    if (visited > int64_t(nnodes) + 1) {  // a tree walk visits each node at most once
      if (lane == 0) atomicExch(err, 3);
      break;
    }
    const unsigned ex = __ballot_sync(full, expand);
    const int lead = ex ? __ffs(int(ex)) - 1 : width;
    if (lead > 0) emit(lane < lead && nout > 0, o0.x, o0.y);
    if (lane < lead) nout = 0;
    const unsigned c1 = __ballot_sync(full, nout >= 1), c2 = __ballot_sync(full, nout == 2);
    const int total = __popc(c1) + __popc(c2);
    const int base = sp - width;
    if (base + total > kWalkCap) {
      if (lane == 0) atomicExch(err, 1);
      break;
    }
    const int at = base + total - 1 - (__popc(c1 & below) + __popc(c2 & below));
    __syncwarp();  // every lane has read its entry
    if (nout >= 1) st[at] = o0;
    if (nout == 2) st[at - 1] = o1;
    sp = base + total;
    __syncwarp();
  }
  emit(lane == 0, T.offset, T.count);
  if (MODE == 2 && lane == 0) {
    seg_cnt[li] = nseg;
    list_len[li] = len;
    if (nseg > room) atomicExch((unsigned long long *)&counters[C_SEGOVF], 1ull);
  }
}

// Room in the buffers that the list kernels write, for launches made before the
// host has seen the counts: they do nothing where a count is above it (or the
// walk has failed or needs its second pass), and the host launches them again
// once it has made room.  idx < 0: the host knows that there is room.
struct ListRoom {
  int64_t idx, segs, items;
};
__device__ __forceinline__ bool lists_fit(const int64_t *counters, const ListRoom &R) {
  return R.idx < 0 || (counters[C_NENT] <= R.idx && counters[C_NSEG] <= R.segs &&
                       counters[C_SEGOVF] == 0 && counters[C_ERR] == 0);
}

// Expands each leaf's segments into the index array at the leaf's list_base,
// keeping only the entries within sqrt(cull2) of the leaf's box (cull2 <= 0:
// every entry): the others are farther than the cutoff from every particle of
// the leaf, so the reference's mask gives them exactly 0.  Warp per leaf: the
// leaf's box as centre and half-width (widened by 4 ulps of the coordinates,
// as in the batched kernel), then its segments 32 at a time as one run of
// entries -- the segment of a lane's entry from the segment starts inside the
// 32-entry window, so short segments leave no lane idle -- kU windows' loads
// in flight, the kept entries compacted by ballot.  The segments come from the
// walk's regions and are also packed leaf after leaf into segs, with their place
// in the full lists; a leaf with more segments than its region holds has them
// there already, from the second walk.
__global__ void __launch_bounds__(256)
    k_expand_pruned(const int2 *__restrict__ local, int local_room, SegDesc *__restrict__ segs,
                    const int64_t *__restrict__ seg_base, const int64_t *__restrict__ seg_cnt,
                    const int64_t *__restrict__ list_base, const DNode *__restrict__ nodes,
                    const int32_t *__restrict__ leaf_ids, const int64_t *__restrict__ counters,
                    ListRoom room, const float4 *__restrict__ table, float cull2,
                    int32_t *__restrict__ idx, int64_t *__restrict__ kept) {
  chain_enter();
  if (!lists_fit(counters, room)) return;
  const int64_t nleaves = counters[C_NLEAF];
  constexpr int kU = 4;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t li = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; li < nleaves;
       li += warps) {
    const DNode &T = nodes[leaf_ids[li]];
    const float lox = T.xmin[0], loy = T.xmin[1], loz = T.xmin[2];
    const float hix = T.xmax[0], hiy = T.xmax[1], hiz = T.xmax[2];
    const float hx = fmaf(fmaxf(fabsf(lox), fabsf(hix)), 4.8e-7f, 0.5f * (hix - lox));
    const float hy = fmaf(fmaxf(fabsf(loy), fabsf(hiy)), 4.8e-7f, 0.5f * (hiy - loy));
    const float hz = fmaf(fmaxf(fabsf(loz), fabsf(hiz)), 4.8e-7f, 0.5f * (hiz - loz));
    const float cx = 0.5f * (lox + hix), cy = 0.5f * (loy + hiy), cz = 0.5f * (loz + hiz);
    const int64_t lbase = list_base[li], sbase = seg_base[li];
    int32_t *out = idx + lbase;
    int64_t nk = 0, done = 0;  // entries kept, entries before this batch of segments
    const int nsegs = int(seg_cnt[li]);
    const bool in_region = nsegs <= local_room;
    const int2 *const region = local + li * local_room;
    for (int q0 = 0; q0 < nsegs; q0 += 32) {
      const bool on = q0 + lane < nsegs;
      int start = 0, count = 0;
      if (on) {
        if (in_region) {
          const int2 S = region[q0 + lane];
          start = S.x;
          count = S.y;
        } else {
          const SegDesc S = segs[sbase + q0 + lane];
          start = S.start;
          count = S.count;
        }
      }
      int incl = count;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += v;
      }
      const int pre = incl - count;
      const int total = __shfl_sync(full, incl, 31);
      if (in_region && on) segs[sbase + q0 + lane] = SegDesc{start, count, lbase + done + pre};
      const int shift = start - pre;  // table index of entry e of this segment: shift + e
      for (int b0 = 0; b0 < total; b0 += 32 * kU) {
        float4 J[kU];
        int32_t at[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int b = b0 + 32 * u;
          // segments starting before the window, and where others start in it
          const int before = __popc(__ballot_sync(full, on && pre < b));
          const unsigned bit = on && pre >= b && pre < b + 32 ? 1u << (pre - b) : 0u;
          const unsigned starts = __reduce_or_sync(full, bit);
          const int s = before - 1 + __popc(starts & (below | (1u << lane)));
          at[u] = __shfl_sync(full, shift, max(0, min(31, s))) + b + lane;
          if (b + lane < total) J[u] = table[at[u]];
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          bool keep = b0 + 32 * u + lane < total;
          if (keep && cull2 > 0.f) {
            const float dx = fmaxf(fabsf(J[u].x - cx) - hx, 0.f);
            const float dy = fmaxf(fabsf(J[u].y - cy) - hy, 0.f);
            const float dz = fmaxf(fabsf(J[u].z - cz) - hz, 0.f);
            keep = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < cull2;
          }
          const unsigned m = __ballot_sync(full, keep);
          if (keep) out[nk + __popc(m & below)] = at[u];
          nk += __popc(m);
        }
      }
      done += total;
    }
    if (lane == 0) kept[li] = nk;
  }
}


// ---------------------------------------------------------------------------
// Groups of <= 32 spatially close particles per processed leaf (Morton order
// inside the leaf's box) and the batched kernel's work items.
// ---------------------------------------------------------------------------
constexpr int kGroupSort = 1024;
constexpr int kGroupHalf = 16;  // particles of a group with a box of their own (adjoint)
constexpr int kGW = 256;     // leaves up to this size are grouped by one warp
constexpr int kGWarps = 4;   // warps (leaves) per block of k_groups_warp
constexpr int kGroupThreads = 256;
constexpr int kGroupBlocks = 8;  // blocks of k_groups an SM holds (2048 threads)

// Where a segment of c > kGroupHalf particles is split: between groups, and a
// group between its first 16 particles and the rest.
__device__ __forceinline__ int group_split(int c, int G) {
  return c > G ? G * (((c + G - 1) / G + 1) / 2) : kGroupHalf;
}

// Splits a leaf into groups of G particles (the last one shorter) by recursive
// median splits along the longest axis, left parts a multiple of G, and each
// group once more at `half` (G where the halves do not matter: that level is a
// third of the time): the particles are close, so the pair kernels' box tests
// keep few list entries.  Every level sorts all segments of the leaf at once by
// (segment, coordinate along the segment's longest axis).
__device__ void group_large_leaf(const DNode &T, const float4 *__restrict__ pos, int32_t *gidx,
                                 int G, int half) {
  __shared__ uint64_t key[kGroupSort];
  __shared__ int32_t val[kGroupSort];
  __shared__ int32_t seg_a[kGroupSort / 16 + 1], seg_c[kGroupSort / 16 + 1];
  __shared__ uint32_t seg_lo[3][kGroupSort / 16 + 1], seg_hi[3][kGroupSort / 16 + 1];
  __shared__ int nseg_s, more_s;
  const int32_t c = T.count;
  if (c > kGroupSort) {
    for (int32_t i = threadIdx.x; i < c; i += blockDim.x) gidx[T.offset + i] = T.offset + i;
    return;
  }
  int m = 1;
  while (m < c) m <<= 1;
  // padding slots sort last but pass through the upper half on the way
  for (int i = threadIdx.x; i < m; i += blockDim.x) val[i] = i < c ? T.offset + i : -1;
  if (threadIdx.x == 0) {
    seg_a[0] = 0;
    seg_c[0] = c;
    nseg_s = 1;
  }
  __syncthreads();
  for (int level = 0; level < 16; ++level) {
    const int nseg = nseg_s;
    // boxes of the segments that still need a split
    for (int q = threadIdx.x; q < nseg; q += blockDim.x)
      for (int d = 0; d < 3; ++d) {
        seg_lo[d][q] = 0xffffffffu;
        seg_hi[d][q] = 0u;
      }
    __syncthreads();
    for (int i = threadIdx.x; i < c; i += blockDim.x) {
      int q = 0;
      while (q + 1 < nseg && seg_a[q + 1] <= i) ++q;
      if (seg_c[q] <= half) continue;
      const float4 p = pos[val[i]];
      const uint32_t o[3] = {f2o(p.x), f2o(p.y), f2o(p.z)};
      for (int d = 0; d < 3; ++d) {
        atomicMin(&seg_lo[d][q], o[d]);
        atomicMax(&seg_hi[d][q], o[d]);
      }
    }
    __syncthreads();
    // sort key: segment, then the coordinate on the segment's longest axis
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
      uint64_t kv = ~0ull;
      if (i < c) {
        int q = 0;
        while (q + 1 < nseg && seg_a[q + 1] <= i) ++q;
        uint32_t ko = 0;
        if (seg_c[q] > half) {
          float ext[3];
          for (int d = 0; d < 3; ++d) ext[d] = o2f(seg_hi[d][q]) - o2f(seg_lo[d][q]);
          const int ax = (ext[0] >= ext[1] && ext[0] >= ext[2]) ? 0 : (ext[1] >= ext[2] ? 1 : 2);
          const float4 p = pos[val[i]];
          ko = f2o(ax == 0 ? p.x : (ax == 1 ? p.y : p.z));
        } else {
          ko = uint32_t(i);  // settled segments keep their order
        }
        kv = (uint64_t(q) << 32) | ko;
      }
      key[i] = kv;
    }
    __syncthreads();
    for (int size = 2; size <= m; size <<= 1)
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
          const int j = i ^ stride;
          if (j > i) {
            const bool up = (i & size) == 0;
            const uint64_t ka = key[i], kb = key[j];
            if ((ka > kb) == up) {
              key[i] = kb;
              key[j] = ka;
              const int32_t t = val[i];
              val[i] = val[j];
              val[j] = t;
            }
          }
        }
        __syncthreads();
      }
    // split every segment above `half`
    if (threadIdx.x == 0) {
      int n2 = 0;
      int32_t na[kGroupSort / 16 + 1], nc[kGroupSort / 16 + 1];
      int more = 0;
      for (int q = 0; q < nseg; ++q) {
        const int32_t a0 = seg_a[q], c0 = seg_c[q];
        if (c0 <= half) {
          na[n2] = a0;
          nc[n2++] = c0;
          continue;
        }
        const int32_t left = group_split(c0, G);
        na[n2] = a0;
        nc[n2++] = left;
        na[n2] = a0 + left;
        nc[n2++] = c0 - left;
        more |= left > half || c0 - left > half;
      }
      for (int q = 0; q < n2; ++q) {
        seg_a[q] = na[q];
        seg_c[q] = nc[q];
      }
      nseg_s = n2;
      more_s = more;
    }
    __syncthreads();
    if (!more_s) break;
  }
  for (int i = threadIdx.x; i < c; i += blockDim.x) gidx[T.offset + i] = val[i];
}

// The leaves that k_groups_warp found too large, a block each at a time: as many
// blocks as the SMs hold share them out.  (A block a leaf of the whole set, most
// of them returning at once, takes 31 us of a 128^3 kick; a block per 256 leaves,
// one after the other, 11 ms of a 32^3 kick with leaves of 512.)
__global__ void __launch_bounds__(kGroupThreads)
    k_groups(const DNode *nodes, const int32_t *big, const int64_t *nbig,
             const float4 *__restrict__ pos, int32_t *gidx, int G, int half) {
  const int64_t n = *nbig;
  for (int64_t b = blockIdx.x; b < n; b += gridDim.x) {
    group_large_leaf(nodes[big[b]], pos, gidx, G, half);
    __syncthreads();  // the next leaf reuses the shared arrays
  }
}

// Warp-per-leaf grouping for leaves of at most kGW particles (the usual
// case; larger leaves are left to k_groups, in big).  Same median splits as k_groups: per
// level, every segment above `half` particles is sorted along its longest
// axis by ranking (each element counts the keys below its own, ties by
// position) and split at group_split().
__global__ void __launch_bounds__(32 * kGWarps)
    k_groups_warp(const DNode *nodes, const int32_t *leaf_ids, const int64_t *nleaves,
                  const float4 *__restrict__ pos, int32_t *gidx, int G, int half, int32_t *big,
                  int64_t *nbig) {
  __shared__ float key[kGWarps][kGW];
  __shared__ int32_t val[kGWarps][2][kGW];
  __shared__ uint8_t segid[kGWarps][kGW];
  __shared__ int16_t seg_a[kGWarps][kGW / 16 + 1], seg_c[kGWarps][kGW / 16 + 1];
  __shared__ int8_t seg_ax[kGWarps][kGW / 16 + 1];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t li = int64_t(blockIdx.x) * kGWarps + w;
  if (li >= *nleaves) return;
  const DNode &T = nodes[leaf_ids[li]];
  const int c = T.count;
  if (c > kGW && lane == 0)
    big[atomicAdd(reinterpret_cast<unsigned long long *>(nbig), 1ull)] = leaf_ids[li];
  if (c <= 0 || c > kGW) return;
  if (c <= half) {
    for (int i = lane; i < c; i += 32) gidx[T.offset + i] = T.offset + i;
    return;
  }
  for (int i = lane; i < c; i += 32) {
    val[w][0][i] = T.offset + i;
    segid[w][i] = 0;
  }
  int nseg = 1;
  if (lane == 0) {
    seg_a[w][0] = 0;
    seg_c[w][0] = int16_t(c);
  }
  __syncwarp();
  int cur = 0;
  for (int level = 0; level < 16; ++level) {
    // longest axis of every segment to split
    bool any = false;
    for (int q = 0; q < nseg; ++q) {
      const int a0 = seg_a[w][q], c0 = seg_c[w][q];
      if (c0 <= half) continue;
      any = true;
      float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
      for (int i = a0 + lane; i < a0 + c0; i += 32) {
        const float4 p = pos[val[w][cur][i]];
        lo[0] = fminf(lo[0], p.x); hi[0] = fmaxf(hi[0], p.x);
        lo[1] = fminf(lo[1], p.y); hi[1] = fmaxf(hi[1], p.y);
        lo[2] = fminf(lo[2], p.z); hi[2] = fmaxf(hi[2], p.z);
      }
      for (int d = 0; d < 3; ++d) {
        lo[d] = warp_min(lo[d]);
        hi[d] = warp_max(hi[d]);
      }
      const float e0 = hi[0] - lo[0], e1 = hi[1] - lo[1], e2 = hi[2] - lo[2];
      if (lane == 0) seg_ax[w][q] = int8_t((e0 >= e1 && e0 >= e2) ? 0 : (e1 >= e2 ? 1 : 2));
    }
    if (!any) break;
    __syncwarp();
    for (int i = lane; i < c; i += 32) {
      const int q = segid[w][i];
      float k = 0.f;
      if (seg_c[w][q] > half) {
        const float4 p = pos[val[w][cur][i]];
        const int ax = seg_ax[w][q];
        k = ax == 0 ? p.x : (ax == 1 ? p.y : p.z);
        // NaN last: ranks that leave no slot out
        k = k == k ? k : INFINITY;
      }
      key[w][i] = k;
    }
    __syncwarp();
    for (int i = lane; i < c; i += 32) {
      const int q = segid[w][i];
      const int a0 = seg_a[w][q], c0 = seg_c[w][q];
      int np = i;
      if (c0 > half) {
        const float ki = key[w][i];
        int r = 0;
        for (int j = a0; j < a0 + c0; ++j) {
          const float kj = key[w][j];
          r += (kj < ki) || (kj == ki && j < i);
        }
        np = a0 + r;
      }
      val[w][cur ^ 1][np] = val[w][cur][i];
    }
    __syncwarp();
    cur ^= 1;
    // split every segment above `half`
    if (lane == 0) {
      int16_t na[kGW / 16 + 1], nc[kGW / 16 + 1];
      int n2 = 0;
      for (int q = 0; q < nseg; ++q) {
        const int a0 = seg_a[w][q], c0 = seg_c[w][q];
        if (c0 <= half) {
          na[n2] = int16_t(a0);
          nc[n2++] = int16_t(c0);
          continue;
        }
        const int left = group_split(c0, G);
        na[n2] = int16_t(a0);
        nc[n2++] = int16_t(left);
        na[n2] = int16_t(a0 + left);
        nc[n2++] = int16_t(c0 - left);
      }
      for (int q = 0; q < n2; ++q) {
        seg_a[w][q] = na[q];
        seg_c[w][q] = nc[q];
      }
      seg_ax[w][kGW / 16] = int8_t(n2);  // count, read back below
    }
    __syncwarp();
    nseg = seg_ax[w][kGW / 16];
    for (int q = 0; q < nseg; ++q)
      for (int i = seg_a[w][q] + lane; i < seg_a[w][q] + seg_c[w][q]; i += 32) segid[w][i] = uint8_t(q);
    __syncwarp();
  }
  for (int i = lane; i < c; i += 32) gidx[T.offset + i] = val[w][cur][i];
}

__device__ __forceinline__ int len_bucket(int64_t len) {
  // 32 buckets, longest lists first
  const int b = 63 - __clzll((unsigned long long)max64(len, 1));
  return 31 - min(31, b);
}

// Work items per length bucket, block sums first; the last block turns them
// into the buckets' first positions.  DESC: also the leaf descriptors and the
// list statistics.
template <bool DESC>
__global__ void __launch_bounds__(128)
    k_leaf_items(const DNode *nodes, const int32_t *leaf_ids, const int64_t *list_len,
                 const int64_t *kept_len, const int64_t *list_base, LeafDesc *ld, int64_t jsplit,
                 int G, int64_t *counters, ListRoom room) {
  chain_enter();
  if (!lists_fit(counters, room)) return;
  const int64_t nleaves = counters[C_NLEAF];
  __shared__ unsigned long long hist[32];
  __shared__ bool last;
  if (threadIdx.x < 32) hist[threadIdx.x] = 0;
  __syncthreads();
  const int64_t li = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  long long pairs = 0, padded = 0;
  if (li < nleaves) {
    LeafDesc d{};
    if (DESC) {
      const DNode &T = nodes[leaf_ids[li]];
      d.offset = T.offset;
      d.count = T.count;
      d.list_len = int32_t(list_len[li]);
      d.kept_len = int32_t(kept_len[li]);
      d.list_begin = list_base[li];
      ld[li] = d;
      pairs = (long long)T.count * list_len[li];
      padded = (long long)((T.count + 31) / 32) * 32 * d.kept_len;
    } else {
      d = ld[li];
    }
    const int64_t nch = max64(1, (d.kept_len + jsplit - 1) / jsplit);
    atomicAdd(&hist[len_bucket(min64(d.kept_len, jsplit))],
              (unsigned long long)(int64_t((d.count + G - 1) / G) * nch));
  }
  if (DESC) {
    for (int o = 16; o > 0; o >>= 1) {
      pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
      padded += __shfl_xor_sync(0xffffffffu, padded, o);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd((unsigned long long *)&counters[C_PAIRS], (unsigned long long)pairs);
      atomicAdd((unsigned long long *)&counters[C_PADDED], (unsigned long long)padded);
    }
  }
  __syncthreads();
  if (threadIdx.x < 32 && hist[threadIdx.x])
    atomicAdd((unsigned long long *)&counters[C_BUCKET + threadIdx.x], hist[threadIdx.x]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0)
    last = atomicAdd((unsigned long long *)&counters[C_TICKET], 1ull) == gridDim.x - 1;
  __syncthreads();
  if (!last || threadIdx.x >= 32) return;
  __threadfence();
  const int64_t mine = __ldcg(counters + C_BUCKET + threadIdx.x);
  int64_t run = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t v = __shfl_up_sync(0xffffffffu, run, o);
    if (int(threadIdx.x) >= o) run += v;
  }
  counters[C_FILL + threadIdx.x] = run - mine;
  if (threadIdx.x == 31) counters[C_NITEMS] = run;
}

__global__ void __launch_bounds__(128)
    k_item_fill(const LeafDesc *ld, int64_t jsplit, int G, int64_t *counters, PairItem *items,
                ListRoom room) {
  chain_enter();
  if (!lists_fit(counters, room) || (room.idx >= 0 && counters[C_NITEMS] > room.items)) return;
  const int64_t nleaves = counters[C_NLEAF];
  // positions inside the block's share of each bucket, then one global
  // reservation a bucket
  __shared__ unsigned long long cnt[32], base[32];
  if (threadIdx.x < 32) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int64_t li = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  LeafDesc L{};
  int64_t nch = 0, items_n = 0;
  unsigned long long at = 0;
  int b = 0;
  if (li < nleaves) {
    L = ld[li];
    nch = max64(1, (L.kept_len + jsplit - 1) / jsplit);
    items_n = int64_t((L.count + G - 1) / G) * nch;
    b = len_bucket(min64(L.kept_len, jsplit));
    at = atomicAdd(&cnt[b], (unsigned long long)items_n);
  }
  __syncthreads();
  if (threadIdx.x < 32 && cnt[threadIdx.x])
    base[threadIdx.x] =
        atomicAdd((unsigned long long *)&counters[C_FILL + threadIdx.x], cnt[threadIdx.x]);
  __syncthreads();
  if (items_n == 0) return;
  PairItem *out = items + base[b] + at;
  const int32_t ng = (L.count + G - 1) / G;
  for (int32_t g = 0; g < ng; ++g)
    for (int64_t c = 0; c < nch; ++c) {
      PairItem it{};
      it.j_begin = L.list_begin + c * jsplit;
      it.j_len = int32_t(min64(jsplit, L.kept_len - c * jsplit));
      it.g_begin = L.offset + G * g;
      it.g_count = min(G, L.count - G * g);
      it.flags = nch > 1 ? 1 : 0;
      *out++ = it;
    }
}

// Three arrays into tree order, perm read once: out[d stride + i] = in_d[perm[i]].
__global__ void k_gather3_f32(const float *__restrict__ a, const float *__restrict__ b,
                              const float *__restrict__ c, const int32_t *__restrict__ perm,
                              float *out, int64_t stride, int64_t n) {
  chain_enter();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int32_t j = perm[i];
    const float va = a[j], vb = b[j], vc = c[j];
    out[i] = va;
    out[stride + i] = vb;
    out[2 * stride + i] = vc;
  }
}

// Everything a kick permutes, perm read once: velocities to the kick's
// buffer, phi, ids and masks to the staging arrays.  TABLE also splits the
// tree-ordered table into positions and masses, for results that go back to
// the host while the pairs run; device arrays get those from k_finish.
template <bool TABLE>
__global__ void k_outputs(KickArrays in, const float4 *__restrict__ table,
                          const int32_t *__restrict__ perm, float *__restrict__ vel, KickArrays out,
                          int64_t n) {
  chain_enter();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int32_t j = perm[i];
    const float v0 = in.f[3][j], v1 = in.f[4][j], v2 = in.f[5][j], h = in.f[7][j];
    const int64_t d = in.id[j];
    const uint16_t k = in.mask[j];
    vel[i] = v0;
    vel[n + i] = v1;
    vel[2 * n + i] = v2;
    out.f[7][i] = h;
    out.id[i] = d;
    out.mask[i] = k;
    if (TABLE) {
      const float4 p = table[i];
      out.f[0][i] = p.x;
      out.f[1][i] = p.y;
      out.f[2][i] = p.z;
      out.f[6][i] = p.w;
    }
  }
}

// A kick's results into the caller's device arrays, all ten in one launch
// (thirteen copies are 3 us each at a few thousand particles, a tenth of the
// call).
__global__ void k_finish(const float4 *__restrict__ table, const float *__restrict__ vel,
                         KickArrays st, KickArrays out, int64_t n) {
  chain_enter();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const float4 p = table[i];
    const float v0 = vel[i], v1 = vel[n + i], v2 = vel[2 * n + i], h = st.f[7][i];
    const int64_t d = st.id[i];
    const uint16_t k = st.mask[i];
    out.f[0][i] = p.x;
    out.f[1][i] = p.y;
    out.f[2][i] = p.z;
    out.f[3][i] = v0;
    out.f[4][i] = v1;
    out.f[5][i] = v2;
    out.f[6][i] = p.w;
    out.f[7][i] = h;
    out.id[i] = d;
    out.mask[i] = k;
  }
}

__global__ void k_pack4(const float *x, const float *y, const float *z, const float *m, float4 *out,
                        int64_t n) {
  chain_enter();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    out[i] = make_float4(x[i], y[i], z[i], m[i]);
}

// Three tree-ordered arrays back to the caller's order, perm read once:
// out_d[perm[i]] = in[d stride + i], or += for ADD.  The outputs may be the
// same array (each thread's three accesses stay in order).
template <bool ADD>
__global__ void k_scatter3_f32(const float *__restrict__ in, int64_t stride,
                               const int32_t *__restrict__ perm, float *o0, float *o1, float *o2,
                               int64_t n) {
  chain_enter();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int32_t j = perm[i];
    const float a = in[i], b = in[stride + i], c = in[2 * stride + i];
    if (ADD) {
      o0[j] += a;
      o1[j] += b;
      o2[j] += c;
    } else {
      o0[j] = a;
      o1[j] = b;
      o2[j] = c;
    }
  }
}

// Monopole pseudo-particle gradients passed to the particles: a warp per
// leaf sums xbar / m of the nodes on its root-to-leaf path (root first, the
// same float additions as a level-by-level top-down pass) and adds m_k times
// the sum to each of its particles.  The path follows the child holding the
// leaf's offset (left when below offset + nleft).
__global__ void k_adj_paths(const DNode *__restrict__ nodes, int32_t nnodes,
                            const float4 *__restrict__ table, int64_t n, float *xbx, float *xby,
                            float *xbz, int32_t *err) {
  const int32_t leaf = int32_t((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (leaf >= nnodes) return;  // whole warps
  const DNode &L = nodes[leaf];
  if (L.cl != 0 || L.cr != 0 || L.count <= 0) return;
  const int32_t lo = L.offset;
  float a0 = 0.f, a1 = 0.f, a2 = 0.f;
  int32_t t = 0;
  for (int depth = 0;; ++depth) {
    const float m = table[n + t].w;
    const float inv = m != 0.f ? 1.f / m : 0.f;
    a0 = a0 + xbx[n + t] * inv;
    a1 = a1 + xby[n + t] * inv;
    a2 = a2 + xbz[n + t] * inv;
    if (t == leaf) break;
    const DNode &T = nodes[t];
    const int32_t c = lo < T.offset + T.nleft ? T.cl : T.cr;
    if (c <= 0 || c >= nnodes || depth > 256) {  // cannot happen in a valid tree
      if (lane == 0) atomicExch(err, 5);
      return;
    }
    t = c;
  }
  if (a0 == 0.f && a1 == 0.f && a2 == 0.f) return;
  for (int32_t i = lane; i < L.count; i += 32) {
    const int32_t k = L.offset + i;
    const float m = table[k].w;
    xbx[k] += m * a0;
    xby[k] += m * a1;
    xbz[k] += m * a2;
  }
}

// ---------------------------------------------------------------------------
// Adjoint of the 12-point pseudo-particles (RCBForceTree.cxx:519-568,
// :786-799, :855-889).  A node's point a sits at p_a = xc + tdr e_a and has
// the mass ppm_a = sum_s m_s f_a(y_s - xc, tdr) over its sources s (its
// particles, or each child's particles or points), in exact arithmetic
//   f_a(d, tdr) = 1/K + (3/K) (d.e_a)/tdr + (5/(2K)) (3 (d.e_a)^2 - |d|^2)/tdr^2
// (1/K alone for tdr = 0); tdr = ppc x (the least distance from xc to a face
// of the node's box) and xc the node's centre of mass.  Given the cotangents
// of every point's position (xbar) and mass (mbar), the nodes are taken top
// down: each passes its points' cotangents to its sources (a child's points
// before that child is taken), to its xc and to its tdr; the tdr cotangent
// then goes to the particle on the face pptdr took, and every xc cotangent to
// the node's particles (m_i / M).
// ---------------------------------------------------------------------------
constexpr int kQuad = 12;

// A warp per node of level [lb, le).
__global__ void k_quad_adj_level(const DNode *__restrict__ nodes, int32_t lb, int32_t le,
                                 const float4 *__restrict__ table, int64_t n, int32_t nd,
                                 float *xbx, float *xby, float *xbz, float *mb, float *xcbar,
                                 float *tdrbar) {
  __shared__ float sx[8][kQuad][4];  // per warp: the node's points' cotangents (x, y, z, m)
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int32_t t = lb + int32_t((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
  if (t >= le) return;  // whole warps
  const DNode &T = nodes[t];
  const int32_t c = T.count;
  const bool leaf = T.cl == 0 && T.cr == 0;
  // no points used (a node of at most 12 particles is listed by its
  // particles), or a leaf left by a failed split (massless points, no sources)
  if (c <= kQuad || (leaf && c > nd)) return;
  const int64_t pb = n + int64_t(kQuad) * t;
  if (lane < kQuad) {
    sx[w][lane][0] = xbx[pb + lane];
    sx[w][lane][1] = xby[pb + lane];
    sx[w][lane][2] = xbz[pb + lane];
    sx[w][lane][3] = mb[pb + lane];
  }
  __syncwarp();
  const float xc0 = T.xc[0], xc1 = T.xc[1], xc2 = T.xc[2], tdr = T.tdr;
  const float K = float(kQuad);
  float gx = 0.f, gy = 0.f, gz = 0.f, gt = 0.f;  // xc and tdr cotangents
  // p_a = xc + tdr e_a
  if (lane < kQuad) {
    const float ax = sx[w][lane][0], ay = sx[w][lane][1], az = sx[w][lane][2];
    gx += ax;
    gy += ay;
    gz += az;
    gt += ax * c_design[lane][0] + ay * c_design[lane][1] + az * c_design[lane][2];
  }
  // one source at table index j: its cotangents, and its share of xc's and tdr's
  auto source = [&](int64_t j, bool point) {
    const float4 y = table[j];
    const float dx = y.x - xc0, dy = y.y - xc1, dz = y.z - xc2;
    float fx = 0.f, fy = 0.f, fz = 0.f, ft = 0.f, fm = 0.f;
    if (tdr == 0.f) {
      for (int a = 0; a < kQuad; ++a) fm += sx[w][a][3];
      fm *= 1.f / K;
    } else {
      const float it = 1.f / tdr, it2 = it * it;
      const float d2 = dx * dx + dy * dy + dz * dz;
      for (int a = 0; a < kQuad; ++a) {
        const float ex = c_design[a][0], ey = c_design[a][1], ez = c_design[a][2];
        const float M = sx[w][a][3];
        const float q = dx * ex + dy * ey + dz * ez;
        const float p2 = 3.f * q * q - d2;
        fm += M * (1.f / K + (3.f / K) * q * it + (2.5f / K) * p2 * it2);
        // d f / d d = (3/K) e / tdr + (5/(2K)) (6 q e - 2 d) / tdr^2
        const float ce = M * ((3.f / K) * it + (15.f / K) * q * it2);
        const float cd = -M * (5.f / K) * it2;
        fx += ce * ex + cd * dx;
        fy += ce * ey + cd * dy;
        fz += ce * ez + cd * dz;
        // d f / d tdr = -(3/K) q / tdr^2 - (5/K) (3 q^2 - |d|^2) / tdr^3
        ft -= M * ((3.f / K) * q * it2 + (5.f / K) * p2 * it2 * it);
      }
    }
    const float m = y.w;
    xbx[j] += m * fx;
    xby[j] += m * fy;
    xbz[j] += m * fz;
    gx -= m * fx;
    gy -= m * fy;
    gz -= m * fz;
    gt += m * ft;
    if (point) mb[j] += fm;
  };
  if (leaf) {
    for (int32_t s = lane; s < c; s += 32) source(T.offset + s, false);
  } else {
    for (int side = 0; side < 2; ++side) {
      const int32_t ch = side == 0 ? T.cl : T.cr;
      if (ch <= 0) continue;
      const DNode &C = nodes[ch];
      if (C.count <= 0) continue;
      if (C.count <= kQuad) {
        for (int32_t s = lane; s < C.count; s += 32) source(C.offset + s, false);
      } else if (lane < kQuad) {
        source(n + int64_t(kQuad) * ch + lane, true);
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    gx += __shfl_xor_sync(0xffffffffu, gx, o);
    gy += __shfl_xor_sync(0xffffffffu, gy, o);
    gz += __shfl_xor_sync(0xffffffffu, gz, o);
    gt += __shfl_xor_sync(0xffffffffu, gt, o);
  }
  if (lane == 0) {
    xcbar[3 * int64_t(t) + 0] = gx;
    xcbar[3 * int64_t(t) + 1] = gy;
    xcbar[3 * int64_t(t) + 2] = gz;
    tdrbar[t] = gt;
  }
}

// A block per node: tdr = ppc (x_max,d - xc_d) or ppc (xc_d - x_min,d), the
// face pptdr takes (its float expression, ties to the earlier face); the
// cotangent goes to the first particle of the node on that face and to xc.
__global__ void k_quad_adj_tdr(const DNode *__restrict__ nodes, int32_t nnodes,
                               const float4 *__restrict__ table, float ppc, float *xbx, float *xby,
                               float *xbz, float *xcbar, const float *tdrbar) {
  __shared__ int32_t best;
  const int32_t t = blockIdx.x;
  if (t >= nnodes) return;
  const float tb = tdrbar[t];
  const DNode &T = nodes[t];
  if (tb == 0.f || T.count <= 0) return;
  float cand[6];
  for (int d = 0; d < 3; ++d) {
    cand[d] = fsub_(T.xmax[d], T.xc[d]);
    cand[3 + d] = fsub_(T.xc[d], T.xmin[d]);
  }
  const float v = smin_(cand[0], smin_(cand[1], smin_(cand[2], smin_(cand[3],
                                                                   smin_(cand[4], cand[5])))));
  int face = 5;
  for (int j = 5; j >= 0; --j)
    if (cand[j] == v) face = j;
  const int d = face % 3;
  const float target = face < 3 ? T.xmax[d] : T.xmin[d];
  if (threadIdx.x == 0) best = INT32_MAX;
  __syncthreads();
  for (int32_t i = threadIdx.x; i < T.count; i += blockDim.x) {
    const float4 p = table[T.offset + i];
    const float x = d == 0 ? p.x : (d == 1 ? p.y : p.z);
    if (x == target) atomicMin(&best, i);
  }
  __syncthreads();
  if (threadIdx.x != 0 || best == INT32_MAX) return;
  const float g = ppc * tb;
  const int64_t k = T.offset + best;
  float *xb = d == 0 ? xbx : (d == 1 ? xby : xbz);
  atomicAdd(xb + k, face < 3 ? g : -g);
  xcbar[3 * int64_t(t) + d] += face < 3 ? -g : g;
}

// A warp per leaf: xbar_k += m_k sum over the nodes P on the leaf's
// root-to-leaf path of xcbar_P / M_P, M_P the node's mass (the sum of its
// points' masses, which is the sum of its particles' masses).
__global__ void k_quad_adj_paths(const DNode *__restrict__ nodes, int32_t nnodes,
                                 const float4 *__restrict__ table, int64_t n, float *xbx,
                                 float *xby, float *xbz, const float *xcbar, int32_t *err) {
  const int32_t leaf = int32_t((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (leaf >= nnodes) return;  // whole warps
  const DNode &L = nodes[leaf];
  if (L.cl != 0 || L.cr != 0 || L.count <= 0) return;
  const int32_t lo = L.offset;
  float a0 = 0.f, a1 = 0.f, a2 = 0.f;
  int32_t t = 0;
  for (int depth = 0;; ++depth) {
    const float b0 = xcbar[3 * int64_t(t)], b1 = xcbar[3 * int64_t(t) + 1],
                b2 = xcbar[3 * int64_t(t) + 2];
    if (b0 != 0.f || b1 != 0.f || b2 != 0.f) {
      // the node's mass: lane a < 12 reads point a, summed over the warp
      float m = lane < kQuad ? table[n + int64_t(kQuad) * t + lane].w : 0.f;
      for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
      if (m != 0.f) {
        a0 += b0 / m;
        a1 += b1 / m;
        a2 += b2 / m;
      }
    }
    if (t == leaf) break;
    const DNode &T = nodes[t];
    const int32_t c = lo < T.offset + T.nleft ? T.cl : T.cr;
    if (c <= 0 || c >= nnodes || depth > 256) {  // cannot happen in a valid tree
      if (lane == 0) atomicExch(err, 5);
      return;
    }
    t = c;
  }
  if (a0 == 0.f && a1 == 0.f && a2 == 0.f) return;
  for (int32_t i = lane; i < L.count; i += 32) {
    const int32_t k = L.offset + i;
    const float m = table[k].w;
    xbx[k] += m * a0;
    xby[k] += m * a1;
    xbz[k] += m * a2;
  }
}

inline unsigned grid_for(int64_t n, int threads, int64_t cap = 0) {
  if (cap <= 0) cap = int64_t(sm_count()) * 32;
  int64_t b = (n + threads - 1) / threads;
  return unsigned(std::max<int64_t>(1, std::min(b, cap)));
}

}  // namespace

// ---------------------------------------------------------------------------
// Host orchestration
// ---------------------------------------------------------------------------

DeviceTree::~DeviceTree() {
  void *ptrs[] = {epos_, tpos_, oid_, toid_, idx_, nodes_, ppm_, chunk_node_, chunk_base_, big_leaves_,
                  left_cnt_, left_base_, acc_, ticket_, scan_tmp_, node_tmp_, fallback_, counters_, leaf_ids_,
                  up_, processed_, roots_, leafdesc_, segs_, idx_list_, items_, gidx_,
                  tight_chunks_, tight_nodes_, segs_local_, ridx_, sub_nodes_, sub_first_,
                  sub_hist_, wpre_, chains_};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  if (h_counters_) cudaFreeHost(h_counters_);
  if (aux_) {
    cudaStreamSynchronize(aux_);
    cudaStreamDestroy(aux_);
  }
  if (ev_fork_) cudaEventDestroy(ev_fork_);
  if (ev_groups_) cudaEventDestroy(ev_groups_);
}

template <typename T>
cudaError_t DeviceTree::grow(T *&p, size_t &cap, size_t count, cudaStream_t s, bool keep) {
  if (count <= cap && p) return cudaSuccess;
  size_t want = std::max<size_t>(count + count / 4, 256);
  T *q = nullptr;
  cudaError_t e = cudaMalloc(&q, want * sizeof(T));
  if (e != cudaSuccess) return e;
  if (keep && p && cap) {
    e = cudaMemcpyAsync(q, p, cap * sizeof(T), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
  }
  if (p) cudaFree(p);
  p = q;
  cap = want;
  return cudaSuccess;
}

#define DT_CHECK(x)                         \
  do {                                      \
    cudaError_t e_ = (x);                   \
    if (e_ != cudaSuccess) return e_;       \
  } while (0)

cudaError_t DeviceTree::build(const TreeConfig &cfg, int64_t n, const float4 *pos_in, int64_t jsplit,
                              cudaStream_t s) {
  info_ = DeviceTreeInfo{};
  err_ = nullptr;
  padded_pairs_ = 0;
  if (aux_) {  // a previous build that stopped early may have left its groups running
    DT_CHECK(cudaStreamSynchronize(aux_));
    groups_ready_ = 0;
  }
  const auto t0 = std::chrono::steady_clock::now();
  const int k = cfg.tdpts;
  const size_t nn = size_t(std::max<int64_t>(n, 1));
  DT_CHECK(grow(tight_chunks_, cap_tc_,
                (size_t(n) / kTightChunk + kTightNodes + 1) * (sizeof(TightChunk) / sizeof(double)), s));
  DT_CHECK(grow(tight_nodes_, cap_tn_, size_t(kTightNodes) * (sizeof(TightNode) / sizeof(double)), s));
  // (room for the pseudo-particles of an even tree behind the particles: the
  // table is epos_ with them appended)
  DT_CHECK(grow(epos_, cap_e_, nn + size_t(cfg.tdpts) * (4 * nn / std::max(1, cfg.nd) + 64), s));
  DT_CHECK(grow(tpos_, cap_t_, nn, s));
  DT_CHECK(grow(oid_, cap_o_, nn, s));
  DT_CHECK(grow(toid_, cap_to_, nn, s));
  DT_CHECK(grow(idx_, cap_i_, nn, s));
  DT_CHECK(grow(ridx_, cap_ri_, nn, s));
  // counters, subtree totals and level extents in one block (and a pinned
  // copy), zeroed and read back together
  constexpr size_t kTotOff = C_COUNT * sizeof(int64_t), kCtlOff = kTotOff + kSubDepth * sizeof(int64_t);
  constexpr size_t kStateBytes = kCtlOff + sizeof(LevelCtl);
  static_assert(kCtlOff % alignof(LevelCtl) == 0, "alignment");
  if (!counters_) {
    DT_CHECK(cudaHostAlloc(&h_counters_, kStateBytes, cudaHostAllocDefault));
    for (auto *k : {k_subtree<false>, k_subtree<true>})
      DT_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSubMax * kSubBytes));
    DT_CHECK(cudaMalloc(&counters_, kStateBytes));
    // the kernels' error flag lives in a counter slot: read back with the counters
    walk_err_ = reinterpret_cast<int32_t *>(counters_ + C_ERR);
  }
  auto at = [](int64_t *p, size_t off) { return reinterpret_cast<char *>(p) + off; };
  auto *ctl = reinterpret_cast<LevelCtl *>(at(counters_, kCtlOff));
  auto *hc = reinterpret_cast<LevelCtl *>(at(h_counters_, kCtlOff));
  auto *sub_tot = reinterpret_cast<int64_t *>(at(counters_, kTotOff));
  const auto *h_sub = reinterpret_cast<const int64_t *>(at(h_counters_, kTotOff));
  DT_CHECK(cudaMemsetAsync(counters_, 0, kStateBytes, s));
  const size_t want_nodes = size_t(std::max<int64_t>(64, 4 * n / std::max(1, cfg.nd) + 64));
  DT_CHECK(grow(nodes_, cap_nodes_, want_nodes, s));
  if (n > 0) {
    launch_chained(k_elements, grid_for(n, 256, int64_t(sm_count()) * 8), 256, 0, s, pos_in, n,
                   epos_, oid_, ctl);
    ++info_.launches;
  }

  // ---- levels ----
  // Nodes of at most sub_max elements are built whole, a block each; with the
  // tight-certification hook, or after a subtree deeper than a block's
  // bookkeeping, every level runs here.
  const bool subtrees = n == 0 || (!sub_off_ && cfg.force_cm_fallback != 2);
  const int32_t sub_max = subtrees ? kSubMax : -1;
  const int64_t wave = kLevelBlocks * sm_count();
  const int pt = n <= wave * chunk_size<4>() ? 4 : (n <= wave * chunk_size<8>() ? 8 : 16);
  const int64_t chunk = int64_t(pt) * kChunkThreads;
#define LEVEL_LAUNCH(kern, grid, ...)                                             \
  do {                                                                            \
    if (pt == 4) launch_chained(kern<4>, grid, kChunkThreads, 0, s, __VA_ARGS__); \
    else if (pt == 8) launch_chained(kern<8>, grid, kChunkThreads, 0, s, __VA_ARGS__); \
    else launch_chained(kern<16>, grid, kChunkThreads, 0, s, __VA_ARGS__);        \
    ++info_.launches;                                                             \
  } while (0)
  std::vector<int32_t> level_begin{0};
  int64_t live = 1, level_max = n, nroots = 0;  // the next level's nodes and the roots so far
  int32_t level = 0, level_ne = 1;
  bool counted = true;  // false: the level's statistics are there, its centres just decided
  for (bool started = false;;) {
    // as many levels as halve the largest node down to a subtree; few when the
    // level is already wide (a deep, uneven tree)
    int batch = 0;
    if (!(subtrees && level_max <= sub_max)) {
      batch = 1;
      const int64_t goal = subtrees ? sub_max : std::max<int64_t>(cfg.nd, 1);
      while ((level_max >> batch) > goal && batch < 16 && (live << batch) < 2048) ++batch;
    }
    // nodes after i more levels that take chunks there: more than sub_max
    // elements each
    auto wide = [&](int i) {
      return std::min<int64_t>(live << i, subtrees ? n / sub_max + 1 : std::max<int64_t>(n, 1));
    };
    const int64_t after = live << batch;  // nodes that the last level can make
    const size_t max_chunks = size_t(n / chunk + wide(batch) + 1);
    const size_t nodes_most =
        std::min<size_t>(size_t(2 * n + 1), size_t(level_ne) + size_t(live << (batch + 1)));
    const int64_t max_roots = nroots + after;
    DT_CHECK(grow(nodes_, cap_nodes_, nodes_most, s, true));
    DT_CHECK(grow(roots_, cap_ro_, size_t(max_roots), s, true));
    // (the chunk maps and accumulators of the level in progress move along)
    DT_CHECK(grow_chunks(std::max(max_chunks, size_t(after)), size_t(after) + 1, s));
    int32_t *cn[2] = {chunk_node_, chunk_node_ + cap_cn_ / 2};
    int32_t *cb[2] = {chunk_base_, chunk_base_ + cap_cb_ / 2};
    DT_CHECK(grow(left_cnt_, cap_lc_, max_chunks, s));
    DT_CHECK(grow(left_base_, cap_lb_, max_chunks, s));
    DT_CHECK(grow(wpre_, cap_wp_, max_chunks * (kChunkThreads / 32), s));
    DT_CHECK(grow(fallback_, cap_fb_, size_t(after) + 1, s));
    if (batch > 0) DT_CHECK(grow(chains_, cap_ch_, size_t(std::max<int64_t>(n, 1)), s));
    auto *acc = reinterpret_cast<NodeAcc *>(acc_);
    if (!started) {
      LEVEL_LAUNCH(k_root, 1, nodes_, n, cfg, ctl, cn[0], cb[0], acc, ticket_, roots_, sub_max,
                   wide_, walk_err_);
      started = true;
    }
    float4 *pb[2] = {epos_, tpos_};
    int32_t *ob[2] = {oid_, toid_};
    for (int i = 0; i < batch; ++i) {
      const int32_t l = level + i;
      const int from = l & 1, to = from ^ 1;
      const unsigned grid = unsigned(n / chunk + wide(i) + 1);
      if (counted && wide_)
        LEVEL_LAUNCH(k_level_stats_wide, grid, pb[from], nodes_, ctl, l, cn[from], cb[from], acc, ticket_,
                     fallback_, counters_, cfg.force_cm_fallback, cfg.nd);
      else if (counted)
        LEVEL_LAUNCH(k_level_stats, grid, pb[from], nodes_, ctl, l, cn[from], cb[from], acc, ticket_,
                     fallback_, counters_, cfg.force_cm_fallback, cfg.nd);
      counted = true;
      LEVEL_LAUNCH(k_level_count, grid, pb[from], nodes_, ctl, l, cn[from], cb[from], cn[to], cb[to],
                   left_cnt_, left_base_, wpre_, acc, ticket_, roots_, counters_, sub_max);
      LEVEL_LAUNCH(k_part_left, grid, pb[from], ob[from], nodes_, ctl, l, cn[from], cb[from],
                   left_base_, wpre_, pb[to], ob[to], idx_, ridx_);
      LEVEL_LAUNCH(k_part_right, grid, pb[from], ob[from], nodes_, ctl, l, cn[from], cb[from], idx_,
                   pb[to], ob[to], walk_err_, counters_, reinterpret_cast<ChainItem *>(chains_),
                   int64_t(cap_ch_));
      launch_chained(k_part_chains, unsigned(4 * sm_count()), 256, 0, s, pb[from], ob[from], nodes_,
                     ctl, l, reinterpret_cast<const ChainItem *>(chains_), int64_t(cap_ch_),
                     counters_, idx_, ridx_, pb[to], ob[to], walk_err_);
      ++info_.launches;
    }
    if (subtrees) {
      DT_CHECK(grow(sub_nodes_, cap_sub_, size_t(2 * std::max<int64_t>(n, 1)), s));
      DT_CHECK(grow(sub_first_, cap_sf_, size_t(max_roots) * (kSubDepth + 2), s));
      DT_CHECK(grow(sub_hist_, cap_sh_, size_t(max_roots) * kSubDepth, s));
      const int32_t cap = int32_t((std::min<int64_t>(n, sub_max) + 7) & ~int64_t(7));
      launch_chained(wide_ ? k_subtree<true> : k_subtree<false>, unsigned(max_roots), kSubThreads,
                     size_t(cap) * kSubBytes, s, nodes_, ctl, roots_, epos_, oid_, tpos_, toid_, sub_nodes_, sub_first_,
                     sub_hist_, cap, cfg.force_cm_fallback, cfg.nd, counters_);
      launch_chained(k_subtree_scan, kSubDepth, kScanThreads, 0, s, ctl, counters_, sub_hist_,
                     int32_t(max_roots), sub_tot);
      launch_chained(k_subtree_place, unsigned(max_roots), 256, 0, s, nodes_, ctl,
                     counters_, roots_, sub_nodes_, sub_first_, sub_hist_, int32_t(max_roots),
                     sub_tot, int64_t(cap_nodes_));
      info_.launches += 3;
    }
    DT_CHECK(cudaGetLastError());
    DT_CHECK(cudaMemcpyAsync(h_counters_, counters_, kStateBytes, cudaMemcpyDeviceToHost, s));
    DT_CHECK(cudaStreamSynchronize(s));
    const int32_t err = *reinterpret_cast<const int32_t *>(h_counters_ + C_ERR);
    if (err == 4) {
      // a subtree deeper than kSubDepth levels: build again level by level
      sub_off_ = true;
      const cudaError_t e = build(cfg, n, pos_in, jsplit, s);
      sub_off_ = false;
      return e;
    }
    if (err == kErrRange) {  // (in the first pass only)
      wide_ = !wide_;
      started = false;
      DT_CHECK(cudaMemsetAsync(walk_err_, 0, sizeof(int32_t), s));
      continue;
    }
    if (err) {
      err_ = err == 3 ? "subtree: a node outgrew the block's shared memory"
                      : "partition chain check failed";
      return cudaErrorUnknown;
    }
    // the levels made so far, and the extent of the one that is next
    while (int32_t(level_begin.size()) <= hc->next_level)
      level_begin.push_back(hc->begin[level_begin.size() % kCtlLevels]);
    level = hc->next_level;
    const LevelSpan &X = hc->lev[level & 1];
    live = X.live;
    nroots = hc->nroots;
    level_ne = hc->node_end;
    level_max = X.maxcnt;
    if (hc->abort) {
      // undecided centres of mass in this level: certify them, or sum as the
      // reference does, then go on from its left counts
      k_cm_tight_sums<<<tight_blocks(), kTightThreads, 0, s>>>(
          pb[level & 1], nodes_, fallback_, counters_, reinterpret_cast<TightChunk *>(tight_chunks_),
          reinterpret_cast<TightNode *>(tight_nodes_), cfg.force_cm_fallback == 1);
      k_cm_tight_bound<<<tight_blocks(), kTightThreads, 0, s>>>(
          pb[level & 1], nodes_, fallback_, counters_,
          reinterpret_cast<const TightChunk *>(tight_chunks_),
          reinterpret_cast<TightNode *>(tight_nodes_), cfg.force_cm_fallback == 1);
      k_cm_fallback<<<unsigned(std::min<int64_t>((live + 127) / 128, 1024)), 128, 0, s>>>(
          pb[level & 1], nodes_, fallback_, counters_);
      k_decided<<<1, 1, 0, s>>>(ctl, counters_);
      info_.launches += 4;
      DT_CHECK(cudaGetLastError());
      counted = false;
      continue;
    }
    if (hc->done) {
      if (!subtrees) break;
      int64_t total = level_ne;
      for (int d = 0; d < kSubDepth; ++d) total += h_sub[d];
      if (total > INT32_MAX) return cudaErrorInvalidValue;
      if (size_t(total) > cap_nodes_) {
        DT_CHECK(grow(nodes_, cap_nodes_, size_t(total), s, true));
        launch_chained(k_subtree_place, unsigned(max_roots), 256, 0, s, nodes_, ctl,
                       counters_, roots_, sub_nodes_, sub_first_, sub_hist_, int32_t(max_roots),
                       sub_tot, int64_t(cap_nodes_));
        ++info_.launches;
        DT_CHECK(cudaGetLastError());
      }
      // the ranges that hold every node after its parent: levels, then subtree
      // depths
      int64_t end = level_ne;
      level_begin.push_back(int32_t(end));
      for (int d = 0; d < kSubDepth && h_sub[d] > 0; ++d) {
        end += h_sub[d];
        level_begin.push_back(int32_t(end));
      }
      level_ne = int32_t(total);
      break;
    }
  }
#undef LEVEL_LAUNCH
  info_.cm_fallbacks = h_counters_[C_SUBFB] + h_counters_[C_SEQ];
  const int32_t ne = level_ne;
  levels_ = level_begin;
  const int32_t nnodes = ne;
  info_.nodes = nnodes;
  const auto t1 = std::chrono::steady_clock::now();
  build_ms_ = std::chrono::duration<double, std::milli>(t1 - t0).count();
  info_.levels = int64_t(level_begin.size()) - 1;

  // ---- pseudo-particles and processed leaves, from the leaves up ----
  const int64_t ntab = n + int64_t(nnodes) * k;
  // a binary tree's leaves: the processed ones are at most as many
  const int64_t max_leaves = (int64_t(nnodes) + 1) / 2;
  DT_CHECK(grow(ppm_, cap_ppm_, size_t(nnodes) * k + 1, s));
  DT_CHECK(grow(epos_, cap_e_, size_t(std::max<int64_t>(ntab, 1)), s, true));
  float4 *table = epos_;
  DT_CHECK(grow(up_, cap_up_, size_t(nnodes), s));
  DT_CHECK(grow(processed_, cap_pr_, size_t(nnodes), s));
  DT_CHECK(grow(leaf_ids_, cap_leaf_, size_t(max_leaves), s));
  DT_CHECK(grow(big_leaves_, cap_big_, size_t(max_leaves), s));
  const unsigned gN = unsigned((nnodes + 127) / 128), gP = unsigned((int64_t(nnodes) * 32 + 127) / 128);
  launch_chained(k_links, gN, 128, 0, s, nodes_, nnodes, up_);
  if (k == 12)
    launch_chained(k_pseudo_up<12>, gP, 128, 0, s, nodes_, nnodes, up_, epos_, ppm_, table, n, cfg,
                   processed_);
  else
    launch_chained(k_pseudo_up<1>, gP, 128, 0, s, nodes_, nnodes, up_, epos_, ppm_, table, n, cfg,
                   processed_);
  launch_chained(k_leaf_rank, gN, 128, 0, s, nodes_, nnodes, up_, processed_, leaf_ids_, counters_);
  info_.launches += 3;
  DT_CHECK(cudaGetLastError());
  // the groups need only the leaves: on the second stream, beside the walk
  // (forked here, launched after the walk)
  group_ = cfg.group == 16 ? 16 : 32;
  DT_CHECK(grow(gidx_, cap_gidx_, size_t(std::max<int64_t>(n, 1)), s));
  if (!aux_) {
    DT_CHECK(cudaStreamCreateWithFlags(&aux_, cudaStreamNonBlocking));
    DT_CHECK(cudaEventCreateWithFlags(&ev_fork_, cudaEventDisableTiming));
    DT_CHECK(cudaEventCreateWithFlags(&ev_groups_, cudaEventDisableTiming));
  }
  DT_CHECK(cudaEventRecord(ev_fork_, s));
  DT_CHECK(cudaStreamWaitEvent(aux_, ev_fork_, 0));

  // ---- lists: count, scan, write ----
  const size_t nlw = size_t(max_leaves);
  DT_CHECK(grow(node_tmp_, cap_nt_, 5 * nlw + 4, s));
  int64_t *seg_cnt = node_tmp_, *list_len = node_tmp_ + nlw, *seg_base = node_tmp_ + 2 * nlw,
          *list_base = node_tmp_ + 3 * nlw;
  DT_CHECK(grow(scan_tmp_, cap_scan_, size_t(scan_tmp_size(int64_t(nlw))), s));
  // one pass writing each leaf's segments into its own region; the scans
  // then place them (a leaf with more segments than that is walked a second
  // time)
  const int room_segs = local_segs(max_leaves);
  DT_CHECK(grow(segs_local_, cap_segl_, std::max<size_t>(nlw * size_t(room_segs), 1), s));
  launch_chained(k_walk<2>, unsigned((max_leaves + kWalkWarps - 1) / kWalkWarps), 32 * kWalkWarps,
                 0, s, nodes_, nnodes, leaf_ids_, max_leaves, cfg, n, seg_cnt, list_len, nullptr,
                 nullptr, nullptr, segs_local_, room_segs, walk_err_, counters_);
  ++info_.launches;
  // the groups after the walk's blocks, which then have their SMs first
  DT_CHECK(launch_groups(max_leaves, group_, cfg.halves ? kGroupHalf : group_, aux_));
  DT_CHECK(cudaEventRecord(ev_groups_, aux_));
  groups_ready_ = group_;
  if (max_leaves <= kScanPairMax) {
    launch_chained(k_scan_pair, 1, kScanThreads, 0, s, seg_cnt, list_len, seg_base, list_base,
                   max_leaves, counters_ + C_NSEG, counters_ + C_NENT);
    ++info_.launches;
  } else {
    DT_CHECK(scan_counted(seg_cnt, seg_base, max_leaves, counters_ + C_NSEG, scan_tmp_, s));
    DT_CHECK(scan_counted(list_len, list_base, max_leaves, counters_ + C_NENT, scan_tmp_, s));
  }
  DT_CHECK(cudaGetLastError());
  DT_CHECK(grow(leafdesc_, cap_ld_, nlw, s));
  int64_t *kept = node_tmp_ + 4 * nlw;
  constexpr ListRoom kRoom{-1, -1, -1};
  // the index lists and the work items' counts
  auto expand = [&](int64_t leaves, const ListRoom &room) {
    const unsigned blocks = unsigned(std::min<int64_t>((leaves + 7) / 8, int64_t(sm_count()) * 64));
    launch_chained(k_expand_pruned, blocks, 256, 0, s, segs_local_, room_segs, segs_, seg_base,
                   seg_cnt, list_base, nodes_, leaf_ids_, counters_, room, table, cfg.prune2,
                   idx_list_, kept);
    launch_chained(k_leaf_items<true>, unsigned((leaves + 127) / 128), 128, 0, s, nodes_, leaf_ids_,
                   list_len, kept, list_base, leafdesc_, jsplit, group_, counters_, room);
    info_.launches += 2;
  };
  // With the buffers of an earlier build the lists and the items are launched
  // before the host has seen their sizes; one look then tells whether all of it
  // fitted.  (A look after the walk and another after the item counts cost a
  // kick of 5 to 70 thousand particles 25 us.)
  const ListRoom room{int64_t(cap_idx_), int64_t(cap_seg_), int64_t(cap_items_)};
  const bool ahead = room.idx > 0 && room.segs > 0 && room.items > 0;
  if (ahead) {
    expand(max_leaves, room);
    DT_CHECK(cudaStreamWaitEvent(s, ev_groups_, 0));
    groups_ready_ = 0;
    launch_chained(k_item_fill, unsigned((max_leaves + 127) / 128), 128, 0, s, leafdesc_, jsplit,
                   group_, counters_, items_, room);
    ++info_.launches;
    DT_CHECK(cudaGetLastError());
  }
  DT_CHECK(cudaMemcpyAsync(h_counters_, counters_, C_COUNT * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  DT_CHECK(cudaStreamSynchronize(s));
  const int32_t h_err = *reinterpret_cast<const int32_t *>(h_counters_ + C_ERR);
  if (h_err) {
    err_ = h_err == 1 ? "interaction-list walk exceeded its stack"
                      : "interaction-list walk visited more nodes than the tree has";
    return cudaErrorUnknown;
  }
  const int64_t nleaves = h_counters_[C_NLEAF];
  info_.processed_leaves = nleaves;
  const int64_t nseg = h_counters_[C_NSEG];
  const int64_t nent = h_counters_[C_NENT];
  info_.segments = nseg;
  info_.list_entries = nent;
  const bool local = !h_counters_[C_SEGOVF];
  if (!ahead || !local || nent > room.idx || nseg > room.segs) {
    DT_CHECK(grow(segs_, cap_seg_, size_t(std::max<int64_t>(nseg, 1)), s));
    DT_CHECK(grow(idx_list_, cap_idx_, size_t(std::max<int64_t>(nent, 1)), s));
    if (nleaves > 0) {
      if (!local) {
        const unsigned gW = unsigned((nleaves + kWalkWarps - 1) / kWalkWarps);
        launch_chained(k_walk<1>, gW, 32 * kWalkWarps, 0, s, nodes_, nnodes, leaf_ids_, nleaves, cfg,
                       n, seg_cnt, nullptr, seg_base, list_base, segs_, nullptr, room_segs, walk_err_,
                       counters_);
        ++info_.launches;
      }
      expand(nleaves, kRoom);
    }
    DT_CHECK(cudaGetLastError());
    DT_CHECK(fill_items(jsplit, s));
  } else {
    DT_CHECK(place_items(jsplit, h_counters_[C_NITEMS] <= room.items, s));
  }
  lists_ms_ = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t1).count();
  return cudaSuccess;
}

// Room for `chunks` chunks a level (two maps, by level parity) and `nodes`
// nodes' accumulators and tickets, what is there kept.
cudaError_t DeviceTree::grow_chunks(size_t chunks, size_t nodes, cudaStream_t s) {
  if (2 * chunks > cap_cn_) {
    const size_t half = chunks + chunks / 4 + 128, old = cap_cn_ / 2;
    for (int32_t **p : {&chunk_node_, &chunk_base_}) {
      int32_t *q = nullptr;
      DT_CHECK(cudaMalloc(&q, 2 * half * sizeof(int32_t)));
      if (*p) {
        for (int m = 0; m < 2; ++m)
          DT_CHECK(cudaMemcpyAsync(q + m * half, *p + m * old, old * sizeof(int32_t),
                                   cudaMemcpyDeviceToDevice, s));
        DT_CHECK(cudaStreamSynchronize(s));
        cudaFree(*p);
      }
      *p = q;
    }
    cap_cn_ = cap_cb_ = 2 * half;
  }
  size_t bytes = cap_ac_ * sizeof(NodeAcc);
  DT_CHECK(grow(acc_, bytes, nodes * sizeof(NodeAcc), s, true));
  size_t tickets = cap_ac_;
  DT_CHECK(grow(ticket_, tickets, nodes, s, true));
  cap_ac_ = std::min(bytes / sizeof(NodeAcc), tickets);
  return cudaSuccess;
}

cudaError_t DeviceTree::scan_counted(const int64_t *in, int64_t *out, int64_t n, int64_t *total,
                                     int64_t *tmp, cudaStream_t s) {
  // one block-scan launch per level of the recursion plus one add per level above the last
  for (int64_t m = n; m > 0;) {
    ++info_.launches;
    const int64_t nb = (m + kScanBlock - 1) / kScanBlock;
    if (nb == 1) break;
    ++info_.launches;
    m = nb;
  }
  return exclusive_scan_i64(in, out, n, total, tmp, s);
}

cudaError_t DeviceTree::regroup(int group, int64_t jsplit, cudaStream_t s) {
  if (group != 16 && group != 32) return cudaErrorInvalidValue;
  group_ = group;
  const int64_t nleaves = info_.processed_leaves;
  DT_CHECK(cudaMemsetAsync(counters_ + C_BUCKET, 0, 32 * sizeof(int64_t), s));
  DT_CHECK(cudaMemsetAsync(counters_ + C_TICKET, 0, sizeof(int64_t), s));
  DT_CHECK(cudaMemsetAsync(counters_ + C_BIG, 0, sizeof(int64_t), s));
  if (nleaves > 0) {
    DT_CHECK(launch_groups(nleaves, group, group, s));
    launch_chained(k_leaf_items<false>, unsigned((nleaves + 127) / 128), 128, 0, s, nullptr, nullptr,
                   nullptr, nullptr, nullptr, leafdesc_, jsplit, group, counters_,
                   ListRoom{-1, -1, -1});
    ++info_.launches;
  }
  return fill_items(jsplit, s);
}

cudaError_t DeviceTree::launch_groups(int64_t max_leaves, int G, int half, cudaStream_t s) {
  k_groups_warp<<<unsigned((max_leaves + kGWarps - 1) / kGWarps), 32 * kGWarps, 0, s>>>(
      nodes_, leaf_ids_, counters_ + C_NLEAF, epos_, gidx_, G, half, big_leaves_, counters_ + C_BIG);
  k_groups<<<unsigned(std::min<int64_t>(max_leaves, int64_t(sm_count()) * kGroupBlocks)),
             kGroupThreads, 0, s>>>(nodes_, big_leaves_, counters_ + C_BIG, epos_, gidx_, G, half);
  info_.launches += 2;
  return cudaGetLastError();
}

// The items of the leaves whose buckets k_leaf_items placed; joins the groups.
cudaError_t DeviceTree::fill_items(int64_t jsplit, cudaStream_t s) {
  if (groups_ready_) DT_CHECK(cudaStreamWaitEvent(s, ev_groups_, 0));  // launched by build()
  groups_ready_ = 0;
  DT_CHECK(cudaMemcpyAsync(h_counters_, counters_, C_COUNT * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  DT_CHECK(cudaStreamSynchronize(s));
  return place_items(jsplit, false, s);
}

// The items' totals from the counters read back, and the items themselves
// unless they are placed already.
cudaError_t DeviceTree::place_items(int64_t jsplit, bool placed, cudaStream_t s) {
  const int64_t nleaves = info_.processed_leaves;
  const int64_t nitems = nleaves > 0 ? h_counters_[C_NITEMS] : 0;
  info_.items = nitems;
  info_.pairs = h_counters_[C_PAIRS];
  padded_pairs_ = h_counters_[C_PADDED];
  DT_CHECK(grow(items_, cap_items_, size_t(std::max<int64_t>(nitems, 1)), s));
  if (nitems > 0 && !placed) {
    launch_chained(k_item_fill, unsigned((nleaves + 127) / 128), 128, 0, s, leafdesc_, jsplit,
                   group_, counters_, items_, ListRoom{-1, -1, -1});
    ++info_.launches;
  }
  return cudaGetLastError();
}

cudaError_t launch_gather3_f32(const float *a, const float *b, const float *c, const int32_t *perm,
                               float *out, int64_t stride, int64_t n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  launch_chained(k_gather3_f32, grid_for(n, 256), 256, 0, s, a, b, c, perm, out, stride, n);
  return cudaGetLastError();
}
cudaError_t launch_outputs(const KickArrays &in, const float4 *table, bool split_table,
                           const int32_t *perm, float *vel, const KickArrays &out, int64_t n,
                           cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (split_table)
    launch_chained(k_outputs<true>, grid_for(n, 256), 256, 0, s, in, table, perm, vel, out, n);
  else
    launch_chained(k_outputs<false>, grid_for(n, 256), 256, 0, s, in, table, perm, vel, out, n);
  return cudaGetLastError();
}
cudaError_t launch_finish(const float4 *table, const float *vel, const KickArrays &staged,
                          const KickArrays &out, int64_t n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  launch_chained(k_finish, grid_for(n, 256), 256, 0, s, table, vel, staged, out, n);
  return cudaGetLastError();
}
cudaError_t launch_scatter3_f32(const float *in, int64_t stride, const int32_t *perm,
                                float *const out[3], bool add, int64_t n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (add)
    launch_chained(k_scatter3_f32<true>, grid_for(n, 256), 256, 0, s, in, stride, perm, out[0],
                   out[1], out[2], n);
  else
    launch_chained(k_scatter3_f32<false>, grid_for(n, 256), 256, 0, s, in, stride, perm, out[0],
                   out[1], out[2], n);
  return cudaGetLastError();
}

cudaError_t launch_pseudo_adjoint(const DNode *nodes, const std::vector<int32_t> &levels,
                                  const float4 *table, int64_t n, float *xbx, float *xby,
                                  float *xbz, int32_t *err, cudaStream_t s) {
  if (levels.size() < 2) return cudaSuccess;
  const int32_t nnodes = levels.back();
  if (nnodes <= 0) return cudaSuccess;
  k_adj_paths<<<unsigned((int64_t(nnodes) * 32 + 255) / 256), 256, 0, s>>>(nodes, nnodes, table, n,
                                                                           xbx, xby, xbz, err);
  return cudaGetLastError();
}

cudaError_t launch_pseudo_adjoint_quad(const DNode *nodes, const std::vector<int32_t> &levels,
                                       const float4 *table, int64_t n, int32_t nd, float ppc,
                                       float *xbx, float *xby, float *xbz, float *mb, float *xcbar,
                                       float *tdrbar, int32_t *err, cudaStream_t s) {
  if (levels.size() < 2) return cudaSuccess;
  const int32_t nnodes = levels.back();
  if (nnodes <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(xcbar, 0, size_t(nnodes) * 3 * sizeof(float), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(tdrbar, 0, size_t(nnodes) * sizeof(float), s);
  if (e != cudaSuccess) return e;
  for (size_t l = 0; l + 1 < levels.size(); ++l) {
    const int32_t lb = levels[l], le = levels[l + 1];
    if (le > lb)
      k_quad_adj_level<<<unsigned((int64_t(le - lb) * 32 + 255) / 256), 256, 0, s>>>(
          nodes, lb, le, table, n, nd, xbx, xby, xbz, mb, xcbar, tdrbar);
  }
  k_quad_adj_tdr<<<unsigned(nnodes), 256, 0, s>>>(nodes, nnodes, table, ppc, xbx, xby, xbz, xcbar,
                                                  tdrbar);
  k_quad_adj_paths<<<unsigned((int64_t(nnodes) * 32 + 255) / 256), 256, 0, s>>>(
      nodes, nnodes, table, n, xbx, xby, xbz, xcbar, err);
  return cudaGetLastError();
}

cudaError_t launch_pack4(const float *x, const float *y, const float *z, const float *m,
                         float4 *out, int64_t n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  launch_chained(k_pack4, grid_for(n, 256), 256, 0, s, x, y, z, m, out, n);
  return cudaGetLastError();
}
}  // namespace hsr
