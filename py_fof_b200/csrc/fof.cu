// Friends-of-friends linking on the device.
//
// Replaces process_single_region + the fof_fortran driver
// (fof_fortran.f90:109-362, :496-949) and atomic_dsu.c.  All input regions of
// a call are processed together:
//   1. fof_bbox_kernel    per-region unwrap about the first particle + bbox
//   2. host               reference cell geometry per region (same formulas,
//                         same libm pow) -> region table
//   3. fof_key_kernel     global cell key per particle, cell histogram and the
//                         particle's slot in its cell
//   4. fof_scatter_kernel FP32 coordinates (real(x_rel,4)) in cell order.  The
//                         order inside a cell is arbitrary; where the
//                         reference's CRS order (cell, then ascending index)
//                         decides something, the numbering of the candidates
//                         and their first member, step 8 restores it.  (Option
//                         cell_order: the CRS order itself.)
//   5. fof_cells_kernel   dense cells and their warp chunks
//   6. link kernels       pair tests over the reference's neighbour cells
//                         (fof_link_dense_kernel for cells with more than
//                         DENSE_T particles and their pairs with sparse
//                         cells, fof_link_kernel for sparse-cell pairs),
//                         lock-free atomicCAS union (lower index wins)
//   7. fof_root_kernel    full compression + warp-aggregated group sizes
//   8. ordered compaction of the roots of large groups, then by index inside
//                         a cell -> candidate ids (region order, then root CRS
//                         position: the reference halo numbering)
//   9. outputs, FP64 centre-of-mass / angular momentum per candidate
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

#include "context.cuh"
#include "fof.cuh"
#include "fof_internal.cuh"
#include "primitives.cuh"
#include "unbind.cuh"

namespace pyfof {

namespace {

// particles per block of the bbox, key and scatter kernels: 16 per thread, 4
// where few blocks would leave most SMs idle
constexpr int TILE = 4096, TILE_SMALL = 1024;
constexpr int64_t kTileSmallUpTo = 1 << 19;
constexpr int LU = 4;       // particles whose loads a thread has in flight there
constexpr int BLK = 256;

__device__ __forceinline__ int region_of_key(const uint64_t *cell_off, int nreg, uint64_t key) {
  int lo = 0, hi = nreg;  // first r with cell_off[r] > key, minus one
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (cell_off[mid] <= key) lo = mid + 1; else hi = mid;
  }
  return lo - 1;
}

__device__ __forceinline__ void warp_minmax(double &mn, double &mx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
}

// Coordinates of particles i0, i0 + BLK, ..: all loads issued before any is
// used (left in the loop, the branches of unwrap keep them apart, and the
// kernels ran at a third of the memory rate).  Past `end`: `fill`.
__device__ __forceinline__ void load_tile(const Coords &xp, int64_t i0, int64_t end, const double (&fill)[3],
                                          double (&x)[LU][3]) {
#pragma unroll
  for (int u = 0; u < LU; ++u) {
    const int64_t i = i0 + u * BLK;
#pragma unroll
    for (int d = 0; d < 3; ++d) x[u][d] = i < end ? xp.get(i, d) : fill[d];
  }
}

__global__ void __launch_bounds__(BLK) fof_bbox_kernel(Coords xp, const RegionDev *__restrict__ R,
                                                       const Tile *__restrict__ T, double L,
                                                       double half,
                                                       unsigned long long *__restrict__ bbox,
                                                       int32_t *flags) {
  const Tile t = T[blockIdx.x];
  const RegionDev &r = R[t.region];
  if (!r.active) return;
  double anc[3], mn[3], mx[3];
  for (int d = 0; d < 3; ++d) {
    anc[d] = xp.get(r.start, d);
    mn[d] = INFINITY;
    mx[d] = -INFINITY;
  }
  bool bad = false;
  for (int64_t i0 = t.begin + threadIdx.x; i0 < t.end; i0 += LU * BLK) {
    double x[LU][3];
    load_tile(xp, i0, t.end, anc, x);
#pragma unroll
    for (int u = 0; u < LU; ++u)  // (past the end: the anchor, a particle of the region)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        bad |= !isfinite(x[u][d]);
        const double v = unwrap(x[u][d], anc[d], half, L);
        mn[d] = fmin(mn[d], v);
        mx[d] = fmax(mx[d], v);
      }
  }
  if (bad) atomicExch(&flags[FLAG_ERR], kNonFinite);
  __shared__ double smn[3][BLK / 32], smx[3][BLK / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = 0; d < 3; ++d) {
    warp_minmax(mn[d], mx[d]);
    if (lane == 0) { smn[d][warp] = mn[d]; smx[d][warp] = mx[d]; }
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    const int d = threadIdx.x;
    double a = INFINITY, b = -INFINITY;
    for (int w = 0; w < BLK / 32; ++w) { a = fmin(a, smn[d][w]); b = fmax(b, smx[d][w]); }
    if (a <= b) {
      atomicMin(&bbox[6 * (int64_t)t.region + d], dbl_to_ord(a));
      atomicMax(&bbox[6 * (int64_t)t.region + 3 + d], dbl_to_ord(b));
    }
  }
}

// Zero-based cell of a coordinate, floor((x - origin) / size) clamped to the
// grid (fof_fortran.f90:598).  The product with the reciprocal is within a
// few ulps of the quotient, so its floor is the quotient's unless it lies
// that close to a cell boundary; only then is the division done.
__device__ __forceinline__ int32_t cell_coord(double x, double origin, double size, double inv, int32_t n) {
  const double y = __dadd_rn(x, -origin);
  const double q = y * inv;
  double f = floor(q);
  const double tol = 1e-15 * fabs(q) + 1e-300;
  if (!(q - f > tol && f + 1.0 - q > tol)) f = floor(__ddiv_rn(y, size));
  if (!(f >= 0.0)) f = 0.0;
  const double top = (double)(n - 1);
  if (f > top) f = top;
  return __double2int_rz(f);
}

// all != 0: particles of inactive regions get the sentinel key and a slot too
// (the sorts of option cell_order take all particles).  flags[FLAG_SPREAD]:
// warps, one sample of 32 consecutive particles each, whose keys span more
// than `far`.
__global__ void __launch_bounds__(BLK) fof_key_kernel(Coords xp, const RegionDev *__restrict__ R,
                                                      const Tile *__restrict__ T, double L,
                                                      double half, uint32_t sentinel, int all,
                                                      uint32_t far, uint32_t *__restrict__ keys,
                                                      uint32_t *__restrict__ counts,
                                                      uint32_t *__restrict__ rank, int32_t *flags) {
  const Tile t = T[blockIdx.x];
  const RegionDev &r = R[t.region];
  if (!r.active) {
    if (all)
      for (int64_t i = t.begin + threadIdx.x; i < t.end; i += BLK) {
        keys[i] = sentinel;
        rank[i] = atomicAdd(&counts[sentinel], 1u);
      }
    return;
  }
  double anc[3];
  for (int d = 0; d < 3; ++d) anc[d] = xp.get(r.start, d);
  for (int64_t i0 = t.begin + threadIdx.x; i0 < t.end; i0 += LU * BLK) {
    double x[LU][3];
    load_tile(xp, i0, t.end, anc, x);
    uint32_t key[LU];
#pragma unroll
    for (int u = 0; u < LU; ++u) {
      uint32_t c[3];
#pragma unroll
      for (int d = 0; d < 3; ++d)
        c[d] = (uint32_t)cell_coord(unwrap(x[u][d], anc[d], half, L), r.origin[d], r.size[d], r.inv_size[d],
                                    r.N[d]);
      key[u] = (uint32_t)r.cell_off + c[0] + (uint32_t)r.N[0] * (c[1] + (uint32_t)r.N[1] * c[2]);
    }
    if (i0 < t.begin + BLK) {  // the tile's first round (past the end: the anchor's key)
      const unsigned act = __activemask();
      const uint32_t lo = __reduce_min_sync(act, key[0]), hi = __reduce_max_sync(act, key[0]);
      if (hi - lo > far && (threadIdx.x & 31) == 0) atomicAdd(&flags[FLAG_SPREAD], 1);
    }
#pragma unroll
    for (int u = 0; u < LU; ++u) {
      const int64_t i = i0 + u * BLK;
      if (i < t.end) {
        keys[i] = key[u];
        rank[i] = atomicAdd(&counts[key[u]], 1u);  // a slot in the cell, in no particular order
      }
    }
  }
}

// FP32 coordinates to cell start + slot.  Reads the coordinates again, in
// input order (24 B a particle, coalesced), and writes 16 B at the sorted
// position (its cell there, skey, comes from fof_cells_kernel, in order).
// (A gather by sorted index reads three sectors per particle
// instead, after a sort of the indices.)
__global__ void __launch_bounds__(BLK) fof_scatter_kernel(Coords xp, const RegionDev *__restrict__ R,
                                                          const Tile *__restrict__ T, double L, double half,
                                                          const uint32_t *__restrict__ keys,
                                                          const uint32_t *__restrict__ rank,
                                                          const uint32_t *__restrict__ cstart,
                                                          float4 *__restrict__ pos, uint32_t *__restrict__ prid) {
  const Tile t = T[blockIdx.x];
  const RegionDev &r = R[t.region];
  if (!r.active) return;
  double anc[3];
  for (int d = 0; d < 3; ++d) anc[d] = xp.get(r.start, d);
  for (int64_t i0 = t.begin + threadIdx.x; i0 < t.end; i0 += LU * BLK) {
    double x[LU][3];
    uint32_t k[LU], p[LU];
#pragma unroll
    for (int u = 0; u < LU; ++u) {
      const int64_t i = i0 + u * BLK;
      k[u] = i < t.end ? keys[i] : 0u;
      p[u] = i < t.end ? rank[i] : 0u;
    }
    load_tile(xp, i0, t.end, anc, x);
#pragma unroll
    for (int u = 0; u < LU; ++u) p[u] += cstart[k[u]];
#pragma unroll
    for (int u = 0; u < LU; ++u) {
      const int64_t i = i0 + u * BLK;
      if (i >= t.end) break;
      float v[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) v[d] = __double2float_rn(unwrap(x[u][d], anc[d], half, L));
      pos[p[u]] = make_float4(v[0], v[1], v[2], __int_as_float((int)i));
      if (prid) prid[p[u]] = (uint32_t)t.region;
    }
  }
}

// The same in two steps for one region whose consecutive particles lie far
// apart (use_partition).  The direct scatter then writes single 16-byte pieces
// all over an output larger than L2, each a sector read and written in HBM:
// 1.26 ms (with the cells) for a shuffled box of 15.8 M particles; five passes
// over windows of the output that fit L2 took 0.94 ms.  Here a tile first deals its particles
// to kBuckets ranges of cells, whose places in the output are known (cell
// starts): a run of the output per tile and bucket, reserved by one atomic;
// then the particles move on to their slots, a bucket's megabyte at a time.
constexpr int kBuckets = 256;

__device__ __forceinline__ uint32_t bucket_of(uint32_t key, uint32_t ncell) {
  return (uint32_t)(((uint64_t)key * kBuckets) / ncell);
}

// cursor[b] = first position of bucket b (its first cell: the lowest key
// with bucket_of(key) = b)
__global__ void fof_bucket_start_kernel(const uint32_t *__restrict__ cstart, uint32_t ncell,
                                        uint32_t *__restrict__ cursor) {
  const uint32_t b = threadIdx.x;
  if (b < (uint32_t)kBuckets) cursor[b] = cstart[((uint64_t)b * ncell + kBuckets - 1) / kBuckets];
}

constexpr int PTILE = 4096;

__global__ void __launch_bounds__(BLK) fof_partition_kernel(Coords xp, int64_t n, double L, double half,
                                                            const uint32_t *__restrict__ keys,
                                                            const uint32_t *__restrict__ rank, uint32_t ncell,
                                                            uint32_t *__restrict__ cursor, float4 *__restrict__ tpos,
                                                            uint2 *__restrict__ tkey) {
  __shared__ uint32_t cnt[kBuckets], base[kBuckets];
  static_assert(kBuckets == BLK, "a bucket per thread");
  cnt[threadIdx.x] = 0;
  __syncthreads();
  const int64_t b0 = (int64_t)blockIdx.x * PTILE, end = min(n, b0 + PTILE);
  uint32_t key[PTILE / BLK], at[PTILE / BLK];
#pragma unroll
  for (int j = 0; j < PTILE / BLK; ++j) {
    const int64_t i = b0 + j * BLK + threadIdx.x;
    key[j] = i < end ? keys[i] : 0u;
  }
#pragma unroll
  for (int j = 0; j < PTILE / BLK; ++j)
    if (b0 + j * BLK + threadIdx.x < end) at[j] = atomicAdd(&cnt[bucket_of(key[j], ncell)], 1u);
  __syncthreads();
  const uint32_t c = cnt[threadIdx.x];
  base[threadIdx.x] = c ? atomicAdd(&cursor[threadIdx.x], c) : 0u;
  __syncthreads();
  double anc[3];
  for (int d = 0; d < 3; ++d) anc[d] = xp.get(0, d);
#pragma unroll
  for (int j0 = 0; j0 < PTILE / BLK; j0 += LU) {
    const int64_t i0 = b0 + j0 * BLK + threadIdx.x;
    double x[LU][3];
    load_tile(xp, i0, end, anc, x);
    uint32_t s[LU];
#pragma unroll
    for (int u = 0; u < LU; ++u) s[u] = i0 + u * BLK < end ? rank[i0 + u * BLK] : 0u;
#pragma unroll
    for (int u = 0; u < LU; ++u) {
      if (i0 + u * BLK >= end) break;
      float v[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) v[d] = __double2float_rn(unwrap(x[u][d], anc[d], half, L));
      const uint32_t q = base[bucket_of(key[j0 + u], ncell)] + at[j0 + u];
      tpos[q] = make_float4(v[0], v[1], v[2], __int_as_float((int)(i0 + u * BLK)));
      tkey[q] = make_uint2(key[j0 + u], s[u]);
    }
  }
}

__global__ void __launch_bounds__(BLK) fof_place_kernel(const float4 *__restrict__ tpos,
                                                        const uint2 *__restrict__ tkey, int64_t n,
                                                        const uint32_t *__restrict__ cstart,
                                                        float4 *__restrict__ pos) {
  const int64_t i0 = (int64_t)blockIdx.x * (LU * BLK) + threadIdx.x;
  uint2 k[LU];
  float4 v[LU];
#pragma unroll
  for (int u = 0; u < LU; ++u)
    if (i0 + u * BLK < n) {
      k[u] = tkey[i0 + u * BLK];
      v[u] = tpos[i0 + u * BLK];
    }
#pragma unroll
  for (int u = 0; u < LU; ++u)
    if (i0 + u * BLK < n) pos[cstart[k[u].x] + k[u].y] = v[u];
}

// Whether the two-step scatter pays: one region, most sampled warps hold
// particles far apart, and the output (16 B a particle) is above 64 MB, half
// of L2.
static bool use_partition(int nreg, int64_t n_active, int64_t ntiles, int32_t spread) {
  return nreg == 1 && 16.0 * (double)n_active > 64e6 && (int64_t)spread * 2 >= ntiles * (BLK / 32);
}

// ---- the CRS order itself (option cell_order) ------------------------------
// The key kernel's counters give every particle a distinct slot in its
// cell; scattering to cell start + slot groups the particles by cell, and
// sorting each cell's original indices restores the stable order of the
// reference's counting sort (ascending original index within a cell).

__global__ void fof_cell_scatter_kernel(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ rank,
                                        const uint32_t *__restrict__ cstart, int64_t n,
                                        uint32_t *__restrict__ skey, uint32_t *__restrict__ sidx) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t k = keys[i];
    const uint32_t p = cstart[k] + rank[i];
    skey[p] = k;
    sidx[p] = (uint32_t)i;
  }
}

constexpr int CELL_SORT_SMALL = 32;   // cells up to this size: one thread, insertion sort
constexpr int CELL_SORT_MAX = 8192;   // cells up to this size: one block, bitonic sort

__global__ void fof_cell_sort_small_kernel(const uint32_t *__restrict__ cstart, int64_t ncell,
                                           uint32_t *__restrict__ sidx, uint32_t *__restrict__ big,
                                           uint32_t *__restrict__ nbig) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t b = cstart[c], m = cstart[c + 1] - b;
    if (m < 2) continue;
    if (m > (uint32_t)CELL_SORT_SMALL) {
      big[atomicAdd(nbig, 1u)] = (uint32_t)c;
      continue;
    }
    uint32_t *a = sidx + b;
    for (uint32_t i = 1; i < m; ++i) {
      const uint32_t v = a[i];
      uint32_t j = i;
      while (j > 0 && a[j - 1] > v) {
        a[j] = a[j - 1];
        --j;
      }
      a[j] = v;
    }
  }
}

__global__ void __launch_bounds__(1024) fof_cell_sort_big_kernel(const uint32_t *__restrict__ cstart,
                                                               const uint32_t *__restrict__ big,
                                                               const uint32_t *__restrict__ nbig,
                                                               uint32_t *__restrict__ sidx) {
  __shared__ uint32_t v[CELL_SORT_MAX];
  const uint32_t nb = *nbig;
  for (uint32_t j = blockIdx.x; j < nb; j += gridDim.x) {
    const uint32_t c = big[j];
    const uint32_t b = cstart[c], m = cstart[c + 1] - b;
    uint32_t np2 = 1;
    while (np2 < m) np2 <<= 1;
    for (uint32_t i = threadIdx.x; i < np2; i += blockDim.x) v[i] = i < m ? sidx[b + i] : 0xffffffffu;
    __syncthreads();
    for (uint32_t k = 2; k <= np2; k <<= 1)
      for (uint32_t h = k >> 1; h > 0; h >>= 1) {
        for (uint32_t i = threadIdx.x; i < np2; i += blockDim.x) {
          const uint32_t l = i ^ h;
          if (l > i) {
            const bool up = (i & k) == 0;
            const uint32_t x = v[i], y = v[l];
            if ((x > y) == up) {
              v[i] = y;
              v[l] = x;
            }
          }
        }
        __syncthreads();
      }
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) sidx[b + i] = v[i];
    __syncthreads();
  }
}

__global__ void __launch_bounds__(BLK) fof_gather_kernel(
    Coords xp, const RegionDev *__restrict__ R, const uint64_t *__restrict__ cell_off, int nreg,
    const uint32_t *__restrict__ skey, const uint32_t *__restrict__ sidx, int64_t n_active,
    double L, double half, float4 *__restrict__ pos, uint32_t *__restrict__ prid) {
  for (int64_t p = (int64_t)blockIdx.x * BLK + threadIdx.x; p < n_active;
       p += (int64_t)gridDim.x * BLK) {
    const int rid = nreg == 1 ? 0 : region_of_key(cell_off, nreg, skey[p]);
    const RegionDev &r = R[rid];
    const int64_t i = sidx[p];
    float v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
      v[d] = __double2float_rn(unwrap(xp.get(i, d), xp.get(r.start, d), half, L));
    pos[p] = make_float4(v[0], v[1], v[2], __int_as_float((int)i));
    if (prid) prid[p] = (uint32_t)rid;
  }
}

// ---- lock-free disjoint-set union over sorted positions -------------------
// parent[x] == x marks a root; parent pointers only ever point to smaller
// indices, so the root of every set is its minimum element, exactly as in
// atomic_dsu.c (a higher root is hung under a lower one by CAS).

__device__ __forceinline__ int dsu_find(int *parent, int x) {
  int y = __ldcg(parent + x);
  while (y != x) {
    int z = __ldcg(parent + y);
    if (z != y) parent[x] = z;  // path halving; z is an ancestor of x
    x = y;
    y = z;
  }
  return x;
}

__device__ __forceinline__ void dsu_union(int *parent, int a, int b, int32_t *flags) {
  for (int it = 0; it < (1 << 22); ++it) {
    a = dsu_find(parent, a);
    b = dsu_find(parent, b);
    if (a == b) return;
    if (a > b) { int t = a; a = b; b = t; }
    int old = atomicCAS(parent + b, b, a);
    if (old == b) return;
  }
  atomicExch(&flags[FLAG_ERR], kInvalid);  // unreachable: retry cap as a safety net
}

// Joins the sets of a and b; returns a root of the joined set.
__device__ __forceinline__ int dsu_join(int *parent, int a, int b, int32_t *flags) {
  for (int it = 0; it < (1 << 22); ++it) {
    a = dsu_find(parent, a);
    b = dsu_find(parent, b);
    if (a == b) return a;
    if (a > b) { int t = a; a = b; b = t; }
    if (atomicCAS(parent + b, b, a) == b) return a;
  }
  atomicExch(&flags[FLAG_ERR], kInvalid);  // unreachable: retry cap as a safety net
  return a;
}

struct LinkParams {
  double L, half, rp2;
  float rp2_open;   // largest float f with (double)f <= link^2
  float rp2_lo, rp2_hi;  // FP32 fast-path brackets of link^2 for periodic tests
  int fast_periodic;
};

// Exact reference distance tests.  Open regions: FP32 differences, squares
// and sum (fof_fortran.f90:636).  Periodic regions: dist2_pbc
// (fof_fortran.f90:483-491) in FP64; an FP32 estimate settles all pairs
// whose distance is far from the linking length and only the rest take the
// FP64 path, which decides them exactly.
__device__ __forceinline__ bool linked_open(float4 a, float4 b, float thr) {
  float d0 = __fsub_rn(a.x, b.x), d1 = __fsub_rn(a.y, b.y), d2 = __fsub_rn(a.z, b.z);
  float s = __fmul_rn(d0, d0);
  s = __fadd_rn(s, __fmul_rn(d1, d1));
  s = __fadd_rn(s, __fmul_rn(d2, d2));
  return s <= thr;
}

__device__ __forceinline__ bool linked_pbc(float4 a, float4 b, const LinkParams &P) {
  float d0 = __fsub_rn(a.x, b.x), d1 = __fsub_rn(a.y, b.y), d2 = __fsub_rn(a.z, b.z);
  if (P.fast_periodic) {
    const float hf = (float)P.half, Lf = (float)P.L;
    float e0 = fabsf(d0), e1 = fabsf(d1), e2 = fabsf(d2);
    e0 = e0 > hf ? Lf - e0 : e0;
    e1 = e1 > hf ? Lf - e1 : e1;
    e2 = e2 > hf ? Lf - e2 : e2;
    float s = e0 * e0 + e1 * e1 + e2 * e2;
    if (s < P.rp2_lo) return true;
    if (s > P.rp2_hi) return false;
  }
  double x = fabs((double)d0), y = fabs((double)d1), z = fabs((double)d2);
  if (x > P.half) x = __dadd_rn(P.L, -x);
  if (y > P.half) y = __dadd_rn(P.L, -y);
  if (z > P.half) z = __dadd_rn(P.L, -z);
  double r2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
  return r2 <= P.rp2;
}

// Which test a pair needs.  kNear: linked_pbc's answer for particles that are
// less than L/2 apart along every axis (RegionDev::near_ok), where the minimum
// image is the pair itself and the FP32 estimate needs no comparison with L/2.
enum LinkTest { kOpen = 0, kPeriodic = 1, kNear = 2 };

__device__ __forceinline__ bool linked_near(float4 a, float4 b, const LinkParams &P) {
  if (P.fast_periodic) {
    const float d0 = __fsub_rn(a.x, b.x), d1 = __fsub_rn(a.y, b.y), d2 = __fsub_rn(a.z, b.z);
    const float s = d0 * d0 + d1 * d1 + d2 * d2;
    if (s < P.rp2_lo) return true;
    if (s > P.rp2_hi) return false;
  }
  return linked_pbc(a, b, P);
}

__device__ __forceinline__ bool linked(int test, float4 a, float4 b, const LinkParams &P) {
  if (test == kNear) return linked_near(a, b, P);
  return test == kPeriodic ? linked_pbc(a, b, P) : linked_open(a, b, P.rp2_open);
}

// Cells with more than DENSE_T particles carry a sub-cell index (sub[d]
// slabs per axis, each at least one linking length wide; a single slab when
// the cell is narrower than two linking lengths): the particles of the cell
// are listed by sub-cell in dpos[], sub_tab holds the offsets.  A pair test
// against such a cell only visits the sub-cells that overlap the cube of
// half-width `reach` around the particle, which contains every partner the
// exact distance test can accept.  Their particles, and every pair between
// a dense and a sparse cell, are linked by the dense-cell kernel; pairs of
// sparse cells by the per-particle kernel.
constexpr int DENSE_T = 24;
constexpr int SUB_MAX = 216;

struct DenseIndex {
  const uint32_t *rank;  // number of each dense cell (set for dense cells only)
  const uint32_t *tab;   // per dense cell: S+1 offsets (relative to cell start)
  const float4 *dpos;    // dense cells' particles listed by sub-cell; .w = sorted position
  int stride;            // entries per dense cell in tab
  float reach;           // linking length plus FP32 rounding slack
};

// Sub-cell of a coordinate inside a cell whose lower corner is lo.  FP32,
// monotone in x; the same function places particles and bounds queries, and
// `reach` carries slack for the FP32 rounding of the query endpoints.
__device__ __forceinline__ int sub_of(float x, float lo, float inv_sub, int s) {
  float t = floorf(__fmul_rn(__fsub_rn(x, lo), inv_sub));
  if (!(t >= 0.0f)) t = 0.0f;
  if (t > (float)(s - 1)) t = (float)(s - 1);
  return (int)t;
}

// Sub-cell layout of a dense cell with n particles: about SUB_OCC particles
// per sub-cell (floor(cbrt(n / SUB_OCC)) slabs per axis), at most the
// region's sub[d] (slabs at least one linking length wide).  Few, well
// filled sub-cells keep the number of source ranges a query walks small.
// Build and queries use this one function, so they agree on every cell.
constexpr float SUB_OCC = 6.0f;

struct SubGrid {
  int s[3];
  float inv[3];  // sub-cells per unit length
};

// Very dense cell: a dense cell whose merge sub-cells hold VD_OCC particles
// or more on average.  All pairs inside one merge sub-cell are linked, so
// such cells are linked sub-cell by sub-cell (fof_vd_intra_kernel,
// fof_vd_inter_kernel) instead of pair by pair.
constexpr int VD_OCC = 4;
__device__ __forceinline__ bool is_vd(const RegionDev &r, int64_t n) {
  return r.vd_k[0] > 0 && n > DENSE_T && n >= (int64_t)VD_OCC * r.vd_k[0] * r.vd_k[1] * r.vd_k[2];
}

__device__ __forceinline__ SubGrid dense_sub(const RegionDev &r, int64_t n) {
  SubGrid g;
  if (is_vd(r, n)) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      g.s[d] = r.vd_k[d];
      g.inv[d] = r.vd_inv[d];
    }
    return g;
  }
  const int k = max(1, (int)cbrtf(__fdiv_rn((float)n, SUB_OCC)));
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    g.s[d] = min(k, r.sub[d]);
    g.inv[d] = g.s[d] == r.sub[d] ? r.inv_sub[d] : __double2float_rn((double)g.s[d] / r.size[d]);
  }
  return g;
}

__device__ __forceinline__ float cell_lower(const RegionDev &r, int d, int64_t i) {
  return __double2float_rn(__dadd_rn(r.origin[d], __dmul_rn((double)i, r.size[d])));
}

// Union of a linked pair (p, q); rp caches p's root between calls.
__device__ __forceinline__ void link_pair(int *parent, int p, int q, int &rp, int32_t *flags) {
  if (rp < 0) rp = dsu_find(parent, p);
  const int y = __ldcg(parent + q);
  if (y == rp) return;  // q already hangs directly under p's root
  const int rq = dsu_find(parent, q);
  if (rq != rp) {
    dsu_union(parent, rp, rq, flags);
    rp = dsu_find(parent, rp);
  }
}

// Sparse-cell particles, a warp per 32 consecutive sorted positions.  Each
// lane lists the source ranges of its particle: the sparse cells among the
// neighbour cells that the cube of half-width `reach` around it touches,
// from its own cell on (higher keys; in the own cell, the higher positions).
// Cells that are neighbours along x are consecutive in cell order, so a row
// of them is one range: at most five rows and as many wrapped cells.  Rows
// broken up by dense cells, and axes of one or two cells, can give more; a
// lane tests the ranges beyond the first MAX_RANGES itself, right away.  The warp then runs all pairs of all lanes
// in rounds of 32, one pair per lane (a lane finds its pair's particle by a
// count of the ends of the lanes' pairs and its source by walking that
// particle's ranges), so the lanes stay busy however unevenly the pairs are
// spread over the particles.  Pairs with dense-cell particles are the dense
// kernel's.
// Bound by instruction issue: what a particle costs before its first pair
// test.  So the cell is decoded by multiplication, the cells its reach
// touches follow from its FP32 place in the cell (RegionDev::near) and the
// rows need two loads each.
constexpr int MAX_RANGES = 10;
constexpr int kRounds = 2;

// Pairs of particle ip with the sorted positions [b, e), tested at once.
__device__ __noinline__ void link_range(const float4 *__restrict__ pos, float4 me, int ip, uint32_t b, uint32_t e,
                                        int periodic, const LinkParams &P, int *parent, int32_t *flags) {
  for (uint32_t q = b; q < e; ++q) {
    const float4 o = pos[q];
    const bool lk = periodic ? linked_pbc(me, o, P) : linked_open(me, o, P.rp2_open);
    if (lk) {
      int rp = -1;
      link_pair(parent, ip, (int)q, rp, flags);
    }
  }
}

__global__ void __launch_bounds__(BLK, 4) fof_link_kernel(
    const float4 *__restrict__ pos, const uint32_t *__restrict__ skey,
    const uint32_t *__restrict__ prid, const RegionDev *__restrict__ R,
    const uint32_t *__restrict__ cs, int *parent, int64_t n, LinkParams P, int32_t *flags) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ uint2 ranges[BLK][MAX_RANGES];  // (first source, count)
  __shared__ float4 target[BLK];
  // linked pairs of the warp, joined 32 at a time: a join is a chain of
  // dependent loads and a compare-and-swap, and only a few pairs of a round link
  __shared__ int2 joins[BLK / 32][32 + 32 * kRounds];
  __shared__ uint2 owners[BLK];
  int njoin = 0;
  const int lane = threadIdx.x & 31;
  uint2 *wowner = owners + (threadIdx.x & ~31);
  int2 *wjoin = joins[threadIdx.x >> 5];
  auto join_queue = [&](int m) {  // the first m pairs of the queue, a lane each
    if (lane < m) {
      const int2 e = wjoin[lane];
      int rp = -1;
      link_pair(parent, e.x, e.y, rp, flags);
    }
    __syncwarp();
  };
  const int wbase_t = threadIdx.x & ~31;
  const int64_t step_w = (int64_t)gridDim.x * BLK;
  int64_t wb = (((int64_t)blockIdx.x * BLK + threadIdx.x) >> 5) * 32;
  // the next particle's cell and position are loaded an iteration ahead
  uint32_t next_cell = wb + lane < n ? skey[wb + lane] : 0u;
  float4 next_me = wb + lane < n ? pos[wb + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  for (; wb < n; wb += step_w) {
    const int64_t w = wb + lane;
    const int ip = (int)w;
    uint32_t total = 0;
    int nr = 0;
    bool per = false, wrap = false;  // wrap: pairs across the box's faces, or too wide cells
    const uint32_t cell = next_cell;
    const float4 me = next_me;
    const uint32_t own_begin = cs[cell], own_end = cs[cell + 1];
    if (w + step_w < n) {
      next_cell = skey[w + step_w];
      next_me = pos[w + step_w];
    }
    if (w < n) {
      if (own_end - own_begin <= (uint32_t)DENSE_T) {
        const RegionDev &r = R[prid ? prid[w] : 0];
        per = r.periodic != 0;
        wrap = !r.near_ok;
        target[threadIdx.x] = me;
        const uint32_t coff = (uint32_t)r.cell_off, local = cell - coff;
        const int N0 = r.N[0], N1 = r.N[1], N2 = r.N[2];
        const uint32_t q0 = div_by(local, r.div[0]);
        const int ix = (int)(local - q0 * (uint32_t)N0);
        const int iz = (int)div_by(q0, r.div[1]);
        const int iy = (int)(q0 - (uint32_t)iz * (uint32_t)N1);
        // which neighbour cells the reach touches, per axis; both sides where
        // FP32 cannot tell the cell
        const float xyz[3] = {me.x, me.y, me.z};
        bool below[3], above[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float f = (xyz[d] - r.org[d]) * r.cinv[d];
          const float fr = f - floorf(f);
          below[d] = fr < r.near[d] || fr > 1.0f - r.slack[d];
          above[d] = fr > 1.0f - r.near[d] || fr < r.slack[d];
        }
        auto add = [&](uint32_t b, uint32_t e) {
          if (e <= b) return;
          if (nr < MAX_RANGES) {
            ranges[threadIdx.x][nr++] = make_uint2(b, e - b);
            total += e - b;
          } else {
            link_range(pos, me, ip, b, e, r.periodic, P, parent, flags);
          }
        };
        // the sparse cells among c0..c1, positions from `from` on; neighbours
        // in cell order are one range
        auto add_cells = [&](uint32_t c0, uint32_t c1, uint32_t from) {
          uint32_t run = cs[c0], end = run;
#pragma unroll 1
          for (uint32_t c = c0; c <= c1; ++c) {
            const uint32_t ce = cs[c + 1];
            if (ce - end > (uint32_t)DENSE_T) {
              add(max(run, from), end);
              run = ce;
            }
            end = ce;
          }
          add(max(run, from), end);
        };
        const bool px = r.pdim & 1;
        // rows by steps of the cell number wherever no row wraps around; at an
        // open face the rows outside the box are left out (a list of 20,000
        // small regions is mostly faces: 3.97 -> 2.45 ms with neighbouring sparse cells as one range)
        if ((!px || N0 >= 3) && (!(r.pdim & 2) || (iy > 0 && iy < N1 - 1)) &&
            (!(r.pdim & 4) || (iz > 0 && iz < N2 - 1))) {
          // x neighbours: a run of cells, and the cell around the box's edge
          const int x0 = below[0] && ix > 0 ? -1 : 0, x1 = above[0] && ix < N0 - 1 ? 1 : 0;
          const bool lo_wrap = px && below[0] && ix == 0, hi_wrap = px && above[0] && ix == N0 - 1;
          const bool up_y = above[1] && iy < N1 - 1, dn_y = below[1] && iy > 0, up_z = above[2] && iz < N2 - 1;
          // the rows to visit: own, then (y, z) = (+1, 0), (-1, +1), (0, +1),
          // (+1, +1); all their bounds are loaded before the first is used
          const bool need[5] = {true, up_y, up_z && dn_y, up_z, up_z && up_y};
          const int step[5] = {0, N0, N0 * (N1 - 1), N0 * N1, N0 * (N1 + 1)};
          uint32_t rb[5], re[5];
#pragma unroll
          for (int i = 0; i < 5; ++i) {
            const uint32_t c = cell + (uint32_t)step[i];
            rb[i] = i ? (need[i] ? cs[c + x0] : 0u) : own_begin;
            re[i] = need[i] ? cs[c + x1 + 1] : 0u;
          }
#pragma unroll
          for (int i = 0; i < 5; ++i) {
            if (re[i] == rb[i]) continue;
            if (re[i] - rb[i] <= (uint32_t)DENSE_T) {
              add(i ? rb[i] : (uint32_t)ip + 1, re[i]);
            } else {
              const uint32_t c = cell + (uint32_t)step[i];
              add_cells(i ? c + x0 : c, c + x1, i ? 0u : (uint32_t)ip + 1);
            }
          }
          if (lo_wrap || hi_wrap) {
            wrap = true;
#pragma unroll 1
            for (int i = lo_wrap ? 0 : 1; i < 5; ++i) {
              const int dz = i > 1 ? 1 : 0, dy = i > 1 ? i - 3 : i;
              if ((dz && !up_z) || (dy > 0 && !up_y) || (dy < 0 && !dn_y)) continue;
              const uint32_t c = cell + (uint32_t)(N0 * (dy + N1 * dz)) + (lo_wrap ? N0 - 1 : 1 - N0);
              add_cells(c, c, 0);
            }
          }
        } else {
          wrap = true;
          const int ic[3] = {ix, iy, iz}, Nd[3] = {N0, N1, N2};
          int lo[3], hi[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            if (Nd[d] == 1) { lo[d] = 0; hi[d] = 0; }
            else if (((r.pdim >> d) & 1) && Nd[d] == 2) { lo[d] = 0; hi[d] = (below[d] || above[d]) ? 1 : 0; }
            else { lo[d] = below[d] ? -1 : 0; hi[d] = above[d] ? 1 : 0; }
          }
          // (the distance test takes the minimum image itself: a wrapped cell
          // needs no coordinate shift)
          for (int dz = lo[2]; dz <= hi[2]; ++dz)
            for (int dy = lo[1]; dy <= hi[1]; ++dy)
              for (int dx = lo[0]; dx <= hi[0]; ++dx) {
                const int dd[3] = {dx, dy, dz};
                int j[3];
                bool in = true;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                  j[d] = ic[d] + dd[d];
                  if ((r.pdim >> d) & 1) {
                    if (j[d] < 0) j[d] += Nd[d]; else if (j[d] >= Nd[d]) j[d] -= Nd[d];
                  } else if (j[d] < 0 || j[d] >= Nd[d]) {
                    in = false;
                  }
                }
                if (!in) continue;
                const uint32_t jl = (uint32_t)j[0] + (uint32_t)N0 * ((uint32_t)j[1] + (uint32_t)N1 * (uint32_t)j[2]);
                if (jl < local) continue;
                add_cells(coff + jl, coff + jl, jl == local ? (uint32_t)ip + 1 : 0);
              }
        }
      }
    }
    // pair offsets of the lanes
    uint32_t incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += v;
    }
    const uint32_t T = __shfl_sync(FULL, incl, 31);
    const unsigned per_mask = __ballot_sync(FULL, per);
    const bool near = !__any_sync(FULL, wrap);  // of all the warp's periodic pairs
    // the lanes that have pairs, in order, and the first pair of each
    const unsigned some = __ballot_sync(FULL, total != 0);
    if (total != 0) wowner[__popc(some & lanemask_lt())] = make_uint2(incl - total, (uint32_t)lane);
    const uint32_t my_end = total != 0 ? incl : 0x7fffffffu;
    __syncwarp();
    // kRounds rounds at a time, so that their position loads overlap
    for (uint32_t g0 = 0; g0 < T; g0 += 32 * kRounds) {
      int own[kRounds], q[kRounds];
      float4 o[kRounds];
#pragma unroll
      for (int u = 0; u < kRounds; ++u) {
        const uint32_t g = g0 + 32 * u + (uint32_t)lane;
        // pair g's place in wowner: the number of those lanes whose pairs end at
        // or before g, by one bit per end within the round (a binary search of
        // five dependent shuffles over the ends took 21.9 ms of a 768^3 call, this 20.7)
        const int end = (int)(my_end - (g0 + 32 * u));
        const unsigned ends = __reduce_or_sync(FULL, (unsigned)(end - 1) < 31u ? 1u << end : 0u);
        const int at = __popc(__ballot_sync(FULL, end <= 0)) + __popc(ends & (2u * (1u << lane) - 1u));
        const uint2 ow = wowner[at & 31];
        const int owner = (int)ow.y;
        uint32_t j = g - ow.x;
        own[u] = owner;
        q[u] = -1;
        if (g < T) {
          const uint2 *rg = ranges[wbase_t + owner];
          int k = 0;
          while (j >= rg[k].y) {
            j -= rg[k].y;
            ++k;
          }
          q[u] = (int)(rg[k].x + j);
          o[u] = pos[q[u]];
        }
      }
#pragma unroll
      for (int u = 0; u < kRounds; ++u) {
        bool lk = false;
        if (q[u] >= 0) {
          const float4 pm = target[wbase_t + own[u]];
          lk = linked((per_mask >> own[u]) & 1 ? (near ? kNear : kPeriodic) : kOpen, pm, o[u], P);
        }
        const unsigned m = __ballot_sync(FULL, lk);
        if (lk) wjoin[njoin + __popc(m & lanemask_lt())] = make_int2((int)(wb + own[u]), q[u]);
        njoin += __popc(m);
      }
      __syncwarp();
      while (njoin >= 32) {
        join_queue(32);
        njoin -= 32;
        // (at most 32 kRounds pairs are left)
        int2 e[kRounds];
#pragma unroll
        for (int u = 0; u < kRounds; ++u) e[u] = wjoin[32 + 32 * u + lane];
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kRounds; ++u) wjoin[32 * u + lane] = e[u];
        __syncwarp();
      }
    }
    __syncwarp();
  }
  join_queue(njoin);
}

// Dense cells, warp-cooperative: a warp takes a chunk of up to 32 particles
// of one dense cell (consecutive in sub-cell order, so the chunk is
// compact) and walks the neighbour cells and sub-cell rows that the chunk's
// bounding box widened by `reach` can touch: a lane per neighbour cell, then
// a lane per row, whose source ranges are concatenated and read in full
// batches of 32 (row by row, most batches held a few sources and each cost a
// chain of dependent loads).  A source inside the widened box is tested by
// every lane against its own particle with the exact reference test.
//
// Few chunks leave the chip idle while each warp walks its chain of batches
// (2,000 particles, 60 chunks: 64 us), so up to eight warps share a chunk,
// every one taking every eighth batch (24 us; 64^3 particles: 117 -> 80 us).
// Once the chunks alone fill the blocks that run at a time it would only
// repeat the set-up.
//
// Which side tests a pair: two dense cells, this kernel from the lower cell
// (in one cell, from the lower sorted position); a dense and a sparse cell,
// this kernel from the dense cell, whichever key is lower; two sparse cells,
// the per-particle kernel.  Every pair within reach is tested once, and the
// reference test is symmetric (|a - b| = |b - a| in IEEE arithmetic), so
// the set of linked pairs, and with it the partition, equals the
// reference's.
struct DenseChunk {
  uint32_t cell, e0;  // dense cell (global cell index), first index in its dpos list
};

// A neighbour cell of a chunk: its particles, or the sub-cell rows of them
// that the chunk's widened box [wl, wh] overlaps (ny x nz rows of nx
// sub-cells, the first at s00; ny = 0: one range, all n particles).
struct NbCell {
  const uint32_t *tab;
  uint32_t b, n;
  float wl[3], wh[3];
  int s00, sy, sz, nx, ny;
  int dense, own;
};

// The warp's 32 particles against up to 32 sources, one per lane (o, q; hq a
// root of q's set found earlier in the call, or -2 for no source).  Sets only
// merge, so a source whose root is a particle's needs no test with it; and
// once all particles of the chunk share a root, sources of that set are
// dropped together.  A linked pair joins two whole sets: one lane joins them
// and the others take the new root over, so a set is joined once and not by
// every lane that links to it (in a dense core the kernel used to spend its
// time on those repeated finds and compare-and-swaps).
// rp: root of this lane's particle (-1: no particle).  own: the sources that
// are to be tested from the lower sorted position only, as a lane mask.
struct ChunkPair {
  float4 me;
  int ip, rp;
};

__device__ __forceinline__ void link_batch(ChunkPair &c, float4 o, int q, int hq, unsigned own, int test,
                                           const LinkParams &P, int *parent, int32_t *flags) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // the root the whole chunk shares, or -1 (invalid lanes agree with any)
  auto shared_root = [&]() -> int {
    const unsigned valid = __ballot_sync(FULL, c.rp >= 0);
    const int r0 = __shfl_sync(FULL, c.rp, __ffs(valid) - 1);
    return __all_sync(FULL, c.rp < 0 || c.rp == r0) ? r0 : -1;
  };
  int all = shared_root();
  unsigned mask = __ballot_sync(FULL, hq >= 0 && hq != all);
  while (mask) {
    const int src = __ffs(mask) - 1;
    mask &= mask - 1;
    int hs = __shfl_sync(FULL, hq, src);
    const int qs = __shfl_sync(FULL, q, src);
    bool lk = c.rp >= 0 && c.rp != hs && !(((own >> src) & 1) && qs <= c.ip);
    if (!__any_sync(FULL, lk)) continue;
    float4 so;
    so.x = __shfl_sync(FULL, o.x, src);
    so.y = __shfl_sync(FULL, o.y, src);
    so.z = __shfl_sync(FULL, o.z, src);
    so.w = 0.f;
    if (lk) lk = linked(test, c.me, so, P);
    unsigned m = __ballot_sync(FULL, lk);
    if (!m) continue;
    do {
      const int leader = __ffs(m) - 1;
      const int old = __shfl_sync(FULL, c.rp, leader);
      int r = 0;
      if (lane == leader) r = dsu_join(parent, old, hs, flags);
      r = __shfl_sync(FULL, r, leader);
      if (c.rp == old || c.rp == hs) c.rp = r;
      if (hq == old || hq == hs) hq = r;
      hs = r;
      m = __ballot_sync(FULL, lk && c.rp != r);
    } while (m);
    all = shared_root();
    mask &= __ballot_sync(FULL, hq >= 0 && hq != all);
  }
}

__global__ void __launch_bounds__(BLK, 4) fof_link_dense_kernel(
    const float4 *__restrict__ pos, const uint32_t *__restrict__ prid, const RegionDev *__restrict__ R,
    const uint32_t *__restrict__ cell_start, int *parent, const DenseChunk *__restrict__ chunks,
    int64_t nchunks, int lg_parts, LinkParams P, DenseIndex D, int32_t *flags) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ NbCell nb_cells[BLK / 32][27];
  const int lane = threadIdx.x & 31;
  NbCell *cells = nb_cells[threadIdx.x >> 5];
  const int64_t nw = ((int64_t)gridDim.x * BLK) >> 5;
  for (int64_t w = ((int64_t)blockIdx.x * BLK + threadIdx.x) >> 5; w < nchunks << lg_parts; w += nw) {
    const DenseChunk C = chunks[w >> lg_parts];
    const uint32_t part = (uint32_t)w & ((1u << lg_parts) - 1);
    uint32_t turn = 0;  // batches so far
    const int64_t cb = cell_start[C.cell];
    const int64_t cn = (int64_t)cell_start[C.cell + 1] - cb;
    const int64_t k = (int64_t)C.e0 + lane;
    const bool valid = k < cn;
    float4 me = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid) me = D.dpos[cb + k];
    const int ip = valid ? __float_as_int(me.w) : -1;
    const RegionDev &r = R[prid ? prid[cb] : 0];
    const bool my_vd = is_vd(r, cn);
    const int64_t local = (int64_t)C.cell - (int64_t)r.cell_off;
    const int64_t N0 = r.N[0], N1 = r.N[1], N2 = r.N[2];
    const int64_t ixyz[3] = {local % N0, (local / N0) % N1, local / (N0 * N1)};
    const int64_t Nd[3] = {N0, N1, N2};
    // a chunk whose cell is at no periodic face has no pairs around the box
    bool inner = r.near_ok;
#pragma unroll
    for (int d = 0; d < 3; ++d) inner = inner && (!((r.pdim >> d) & 1) || (ixyz[d] > 0 && ixyz[d] < Nd[d] - 1));
    const int test = r.periodic ? (inner ? kNear : kPeriodic) : kOpen;
    // chunk bounding box
    float bl[3] = {valid ? me.x : 3e38f, valid ? me.y : 3e38f, valid ? me.z : 3e38f};
    float bh[3] = {valid ? me.x : -3e38f, valid ? me.y : -3e38f, valid ? me.z : -3e38f};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        bl[d] = fminf(bl[d], __shfl_xor_sync(FULL, bl[d], o));
        bh[d] = fmaxf(bh[d], __shfl_xor_sync(FULL, bh[d], o));
      }
    int lo[3], hi[3];
    bool open_ax[3];  // periodic axes of one or two cells: no box along them
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const bool pd = (r.pdim >> d) & 1;
      open_ax[d] = pd && Nd[d] <= 2;
      if (Nd[d] == 1) { lo[d] = 0; hi[d] = 0; continue; }
      const float clo = cell_lower(r, d, ixyz[d]);
      const float chi = cell_lower(r, d, ixyz[d] + 1);
      const bool below = __fsub_rn(bl[d], D.reach) < clo;
      const bool above = __fadd_rn(bh[d], D.reach) >= chi;
      if (pd && Nd[d] == 2) { lo[d] = 0; hi[d] = (below || above) ? 1 : 0; }
      else { lo[d] = below ? -1 : 0; hi[d] = above ? 1 : 0; }
    }
    // --- neighbour cells, one per lane (lane = 9 (dz+1) + 3 (dy+1) + dx+1)
    uint32_t nrow = 0;  // source ranges of this lane's cell
    if (lane < 27) {
      const int off[3] = {lane % 3 - 1, (lane / 3) % 3 - 1, lane / 9 - 1};
      bool use = true;
      int64_t jcoord[3];
      NbCell &nc = cells[lane];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (off[d] < lo[d] || off[d] > hi[d]) use = false;
        int64_t j = ixyz[d] + off[d];
        float sh = 0.f;
        if ((r.pdim >> d) & 1) {
          if (j < 0) { j += Nd[d]; sh = (float)P.L; } else if (j >= Nd[d]) { j -= Nd[d]; sh = -(float)P.L; }
        } else if (j < 0 || j >= Nd[d]) use = false;
        jcoord[d] = j;
        // the widened box, in the neighbour's frame; none along periodic axes
        // of one or two cells
        nc.wl[d] = open_ax[d] ? -3e38f : __fsub_rn(__fadd_rn(bl[d], sh), D.reach);
        nc.wh[d] = open_ax[d] ? 3e38f : __fadd_rn(__fadd_rn(bh[d], sh), D.reach);
      }
      if (use) {
        const int64_t jl = jcoord[0] + N0 * (jcoord[1] + N1 * jcoord[2]);
        const uint64_t jc = r.cell_off + (uint64_t)jl;
        const uint32_t nb_b = cell_start[jc], n = cell_start[jc + 1] - nb_b;
        const bool dense = n > (uint32_t)DENSE_T;
        // pairs with a lower dense cell are that cell's; pairs with sparse
        // cells are all tested here; pairs of two very dense cells are the
        // merge kernels'
        if (n > 0 && !(dense && jl < local) && !(dense && my_vd && is_vd(r, n))) {
          nc.b = nb_b;
          nc.n = n;
          nc.dense = dense;
          nc.own = jl == local;
          nc.ny = 0;  // one range
          nrow = 1;
          if (dense) {
            const SubGrid g = dense_sub(r, n);
            if (g.s[0] * g.s[1] * g.s[2] > 1) {
              int slo[3], shi[3];
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                const float clo = cell_lower(r, d, jcoord[d]);
                slo[d] = sub_of(nc.wl[d], clo, g.inv[d], g.s[d]);
                shi[d] = sub_of(nc.wh[d], clo, g.inv[d], g.s[d]);
              }
              nc.tab = D.tab + (int64_t)D.rank[jc] * D.stride;
              nc.s00 = slo[0] + g.s[0] * (slo[1] + g.s[1] * slo[2]);
              nc.sy = g.s[0];
              nc.sz = g.s[0] * g.s[1];
              nc.nx = shi[0] - slo[0] + 1;
              nc.ny = shi[1] - slo[1] + 1;
              nrow = (uint32_t)(nc.ny * (shi[2] - slo[2] + 1));
            }
          }
        }
      }
    }
    uint32_t row_end = nrow;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(FULL, row_end, o);
      if (lane >= o) row_end += v;
    }
    const uint32_t rows = __shfl_sync(FULL, row_end, 31);
    __syncwarp();
    ChunkPair c{me, ip, valid ? dsu_find(parent, ip) : -1};
    for (uint32_t r0 = 0; r0 < rows; r0 += 32) {
      // --- a row per lane
      const uint32_t row = r0 + (uint32_t)lane;
      int cell = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const uint32_t v = __shfl_sync(FULL, row_end, cell + step - 1);
        if (v <= row) cell += step;
      }
      cell &= 31;
      const uint32_t cell_row0 = __shfl_sync(FULL, row_end - nrow, cell);
      uint32_t first = 0, cnt = 0;
      if (row < rows) {
        const NbCell &nc = cells[cell];
        if (nc.ny == 0) {
          first = nc.b;
          cnt = nc.n;
        } else {
          const int k = (int)(row - cell_row0), z = k / nc.ny, y = k - z * nc.ny;
          const uint32_t *t = nc.tab + nc.s00 + y * nc.sy + z * nc.sz;
          const uint32_t k0 = t[0];
          first = nc.b + k0;
          cnt = t[nc.nx] - k0;
        }
      }
      uint32_t incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
      }
      const uint32_t T = __shfl_sync(FULL, incl, 31);
      const uint32_t at = first - (incl - cnt);  // source of batch index g: at + g
      for (uint32_t g0 = 0; g0 < T; g0 += 32) {
        if ((turn++ & ((1u << lg_parts) - 1)) != part) continue;
        // --- a source per lane
        const uint32_t g = g0 + (uint32_t)lane;
        int owner = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
          const uint32_t v = __shfl_sync(FULL, incl, owner + step - 1);
          if (v <= g) owner += step;
        }
        owner &= 31;
        const uint32_t t = __shfl_sync(FULL, at, owner) + g;
        const NbCell &nc = cells[__shfl_sync(FULL, cell, owner)];
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        int q = -1, hq = -2;
        bool own = false;
        if (g < T) {
          if (nc.dense) {
            o = D.dpos[t];
            q = __float_as_int(o.w);
          } else {
            o = pos[t];
            q = (int)t;
          }
          own = nc.own != 0;
          if (o.x >= nc.wl[0] && o.x <= nc.wh[0] && o.y >= nc.wl[1] && o.y <= nc.wh[1] && o.z >= nc.wl[2] &&
              o.z <= nc.wh[2])
            hq = dsu_find(parent, q);
        }
        if (c.rp >= 0) c.rp = dsu_find(parent, c.rp);
        link_batch(c, o, q, hq, __ballot_sync(FULL, own), test, P, parent, flags);
      }
    }
    __syncwarp();
  }
}

// The cell of every sorted position (skey), the dense cells, their numbers and
// their chunks of up to 32 particles, in no particular order, and the
// fullest cell.  out: [0] dense cells, [1] chunks,
// [2] largest count (zeroed before).
__global__ void __launch_bounds__(BLK) fof_cells_kernel(const uint32_t *__restrict__ cs, int64_t ncell,
                                                        uint32_t *__restrict__ out, uint32_t *__restrict__ list,
                                                        uint32_t *__restrict__ rank, DenseChunk *__restrict__ chunks,
                                                        uint32_t *__restrict__ skey) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  uint32_t most = 0;
  for (int64_t base = (int64_t)blockIdx.x * BLK; base < ncell; base += (int64_t)gridDim.x * BLK) {
    const int64_t c = base + threadIdx.x;
    const uint32_t b = c < ncell ? cs[c] : 0u, n = c < ncell ? cs[c + 1] - b : 0u;
    most = max(most, n);
    // the cell of every sorted position: small cells by their lane, in step
    // with the neighbour lanes' stores, the others by the warp
    const unsigned m = __ballot_sync(FULL, n > (uint32_t)DENSE_T);
    for (uint32_t j = 0; j < n && n <= (uint32_t)DENSE_T; ++j) skey[b + j] = (uint32_t)c;
    for (unsigned k = m; k; k &= k - 1) {
      const int src = __ffs(k) - 1;
      const uint32_t sb = __shfl_sync(FULL, b, src), sn = __shfl_sync(FULL, n, src);
      for (uint32_t j = lane; j < sn; j += 32) skey[sb + j] = (uint32_t)(c - lane + src);
    }
    if (!m) continue;
    const uint32_t nch = n > (uint32_t)DENSE_T ? (n + 31u) / 32u : 0u;
    uint32_t incl = nch;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += v;
    }
    uint32_t r0 = 0, k0 = 0;
    if (lane == 31) {
      r0 = atomicAdd(&out[0], (uint32_t)__popc(m));
      k0 = atomicAdd(&out[1], incl);
    }
    r0 = __shfl_sync(FULL, r0, 31);
    k0 = __shfl_sync(FULL, k0, 31) + incl - nch;
    if (nch) {
      const uint32_t r = r0 + __popc(m & lanemask_lt());
      list[r] = (uint32_t)c;
      rank[c] = r;
      for (uint32_t j = 0; j < nch; ++j) chunks[k0 + j] = DenseChunk{(uint32_t)c, 32u * j};
    }
  }
  most = __reduce_max_sync(FULL, most);
  if (lane == 0 && most > 0) atomicMax(&out[2], most);
}

// The pairs inside one chunk: the warp's adjacency as a 32-bit mask per lane,
// its transitive closure (Warshall's algorithm, one lane per row), and every
// particle hung under its component's lowest sorted position.  No other
// thread touches these parents yet, so plain stores do.  Left to the linking
// kernel, these are up to 31 dependent joins by compare-and-swap per chunk,
// and every chunk nearby sees the members as separate sets meanwhile.
__device__ __forceinline__ void link_chunk(float4 me, int ip, int test, const LinkParams &P, int *parent) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // linked lanes relative to this one: bit k is lane + k.  The test is
  // symmetric, so half the pairs are tested and the other half read from the
  // votes:
  // the build of a 768^3 lognormal box 5.20 -> 4.47 ms, of a 251^3 box 273 ->
  // 219 us
  unsigned rel = 1;
#pragma unroll 4
  for (int k = 1; k <= 16; ++k) {
    float4 o;
    o.x = __shfl_sync(FULL, me.x, lane + k);
    o.y = __shfl_sync(FULL, me.y, lane + k);
    o.z = __shfl_sync(FULL, me.z, lane + k);
    o.w = 0.f;
    const int oip = __shfl_sync(FULL, ip, lane + k);
    const bool lk = ip >= 0 && oip >= 0 && linked(test, me, o, P);
    const unsigned m = __ballot_sync(FULL, lk);
    if (lk) rel |= 1u << k;
    rel |= __funnelshift_r(m, m, lane) & (1u << (32 - k));
  }
  unsigned comp = __funnelshift_l(rel, rel, lane);
  // (masks, not predicates: 32 of those do not fit)
#pragma unroll 8
  for (int j = 0; j < 32; ++j) comp |= __shfl_sync(FULL, comp, j) & (0u - ((comp >> j) & 1u));
  unsigned root = (unsigned)ip;
#pragma unroll 8
  for (int j = 0; j < 32; ++j) root = min(root, (unsigned)__shfl_sync(FULL, ip, j) | (((comp >> j) & 1u) - 1u));
  if ((int)root != ip) parent[ip] = (int)root;
}

// One block per dense cell: counting sort of its particles by sub-cell, then
// the pairs inside its chunks.
__global__ void __launch_bounds__(BLK) fof_dense_build_kernel(
    const uint32_t *__restrict__ list, const uint32_t *__restrict__ cs,
    const float4 *__restrict__ pos, const RegionDev *__restrict__ R,
    const uint64_t *__restrict__ cell_off, int nreg, int stride, uint32_t *__restrict__ tab,
    float4 *dpos, LinkParams P, int *parent) {
  __shared__ uint32_t hist[SUB_MAX + 1];
  __shared__ uint32_t cur[SUB_MAX + 1];
  const uint32_t c = list[blockIdx.x];
  const int rid = nreg == 1 ? 0 : region_of_key(cell_off, nreg, (uint64_t)c);
  const RegionDev &r = R[rid];
  const int64_t local = (int64_t)c - (int64_t)r.cell_off;
  const int64_t N0 = r.N[0], N1 = r.N[1];
  const int64_t ic[3] = {local % N0, (local / N0) % N1, local / (N0 * N1)};
  float clo[3];
  for (int d = 0; d < 3; ++d) clo[d] = cell_lower(r, d, ic[d]);
  for (int k = threadIdx.x; k <= SUB_MAX; k += BLK) hist[k] = 0;
  __syncthreads();
  const int64_t base = cs[c];
  const int64_t n = (int64_t)cs[c + 1] - base;
  const SubGrid g = dense_sub(r, n);
  const int S = g.s[0] * g.s[1] * g.s[2];
  for (int64_t k = threadIdx.x; k < n; k += BLK) {
    const float4 v = pos[base + k];
    const int sx = sub_of(v.x, clo[0], g.inv[0], g.s[0]);
    const int sy = sub_of(v.y, clo[1], g.inv[1], g.s[1]);
    const int sz = sub_of(v.z, clo[2], g.inv[2], g.s[2]);
    atomicAdd(&hist[sx + g.s[0] * (sy + g.s[1] * sz)], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    uint32_t run = 0;
    for (int k0 = 0; k0 < S; k0 += 32) {
      const int k = k0 + (int)threadIdx.x;
      const uint32_t h = k < S ? hist[k] : 0;
      uint32_t incl = h;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)threadIdx.x >= o) incl += v;
      }
      if (k < S) cur[k] = run + incl - h;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) cur[S] = run;
  }
  __syncthreads();
  uint32_t *t = tab + (int64_t)blockIdx.x * stride;
  for (int k = threadIdx.x; k <= S; k += BLK) t[k] = cur[k];
  __syncthreads();
  for (int64_t k = threadIdx.x; k < n; k += BLK) {
    const float4 v = pos[base + k];
    const int sx = sub_of(v.x, clo[0], g.inv[0], g.s[0]);
    const int sy = sub_of(v.y, clo[1], g.inv[1], g.s[1]);
    const int sz = sub_of(v.z, clo[2], g.inv[2], g.s[2]);
    const uint32_t slot = atomicAdd(&cur[sx + g.s[0] * (sy + g.s[1] * sz)], 1u);
    dpos[base + slot] = make_float4(v.x, v.y, v.z, __int_as_float((int)(base + k)));
  }
  __syncthreads();
  if (!is_vd(r, n)) {  // (very dense cells are joined sub-cell by sub-cell)
    const int lane = threadIdx.x & 31, m = (int)n;
    for (int e0 = 32 * (threadIdx.x >> 5); e0 < m; e0 += BLK) {
      const bool valid = e0 + lane < m;
      const float4 me = valid ? dpos[base + e0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
      link_chunk(me, valid ? __float_as_int(me.w) : -1, r.periodic ? (r.near_ok ? kNear : kPeriodic) : kOpen, P, parent);
    }
  }
}

// Very dense cells, step 1: every particle of a merge sub-cell joins the
// sub-cell's first particle (every pair inside one passes the exact test,
// see region_geometry).  One block per dense cell; the others return.  The
// very dense cells and their regions are listed for step 2 (in any order).
__global__ void __launch_bounds__(BLK) fof_vd_intra_kernel(
    const uint32_t *__restrict__ list, const uint32_t *__restrict__ cs, const RegionDev *__restrict__ R,
    const uint64_t *__restrict__ cell_off, int nreg, int stride, const uint32_t *__restrict__ tab,
    const float4 *__restrict__ dpos, int *parent, int2 *__restrict__ vd, int32_t *flags) {
  const uint32_t c = list[blockIdx.x];
  const int64_t base = cs[c];
  const int64_t n = (int64_t)cs[c + 1] - base;
  const int ri = nreg == 1 ? 0 : region_of_key(cell_off, nreg, (uint64_t)c);
  const RegionDev &r = R[ri];
  if (!is_vd(r, n)) return;
  if (threadIdx.x == 0) vd[atomicAdd(&flags[FLAG_VD], 1)] = make_int2((int)blockIdx.x, ri);
  const SubGrid g = dense_sub(r, n);
  const int S = g.s[0] * g.s[1] * g.s[2];
  const uint32_t *t = tab + (int64_t)blockIdx.x * stride;
  const int lane = threadIdx.x & 31;
  for (int sc = threadIdx.x >> 5; sc < S; sc += BLK / 32) {
    const int64_t m0 = base + t[sc], m1 = base + t[sc + 1];
    if (m1 - m0 < 2) continue;
    const int lead = __float_as_int(dpos[m0].w);
    int rp = -1;
    for (int64_t k = m0 + 1 + lane; k < m1; k += 32) link_pair(parent, lead, __float_as_int(dpos[k].w), rp, flags);
  }
}

// Very dense cells, step 2: merge sub-cells A (of cell c) and B (of c or of
// a neighbour very dense cell; pairs of cells from the lower cell, in one
// cell B > A) whose grid boxes come within `reach` are joined when any of
// their pairs passes the exact test.  The pairs are tested only while the
// two roots differ, 32 members of A at a time against the members of B
// inside A's widened box, up to the first link: linking one pair joins the
// whole of both.  A warp per sub-cell A, taken in turn by the warps of a full
// grid (with a block per cell, the few cells that hold most of the members of
// a cluster left most of the chip idle: 1 M zoom region 2.23 -> 1.0 to 1.75 ms,
// by the order the joins come in).  The
// sub-cells B of all neighbour cells are looked up 32 at a time, a lane each:
// most are joined to A already, and their tables and roots are chains of
// dependent loads (one after the other they were most of the kernel).
struct VdCell {
  const uint32_t *tab;
  uint32_t b;           // first particle
  float wl[3], wh[3];   // A's widened box
  int slo[3], nx, ny, s0, s01, own;
};

__global__ void __launch_bounds__(BLK) fof_vd_inter_kernel(
    const uint32_t *__restrict__ list, const uint32_t *__restrict__ cs, const RegionDev *__restrict__ R,
    const int2 *__restrict__ vd, int smax, int stride, const uint32_t *__restrict__ tab,
    const uint32_t *__restrict__ rank, const float4 *__restrict__ dpos, int *parent, LinkParams P,
    float reach, int32_t *flags) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ VdCell nb_cells[BLK / 32][27];
  const int lane = threadIdx.x & 31;
  VdCell *cells = nb_cells[threadIdx.x >> 5];
  const int64_t items = (int64_t)flags[FLAG_VD] * smax;
  for (int64_t item = ((int64_t)blockIdx.x * BLK + threadIdx.x) >> 5; item < items;
       item += ((int64_t)gridDim.x * BLK) >> 5) {
    const int2 e = vd[item / smax];
    const int A = (int)(item % smax);
    const RegionDev &r = R[e.y];
    const uint32_t c = list[e.x];
    const int64_t base = cs[c];
    const uint32_t *t = tab + (int64_t)e.x * stride;
    if (A >= r.vd_k[0] * r.vd_k[1] * r.vd_k[2]) continue;
    const int64_t a0 = base + t[A], a1 = base + t[A + 1];
    if (a1 == a0) continue;
    const int64_t local = (int64_t)c - (int64_t)r.cell_off;
    const int64_t Nd[3] = {r.N[0], r.N[1], r.N[2]};
    const int64_t ixyz[3] = {local % Nd[0], (local / Nd[0]) % Nd[1], local / (Nd[0] * Nd[1])};
    const bool per = r.periodic != 0;
    // A's bounding box from its members
    float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
    for (int64_t k = a0 + lane; k < a1; k += 32) {
      const float4 v = dpos[k];
      lo[0] = fminf(lo[0], v.x); lo[1] = fminf(lo[1], v.y); lo[2] = fminf(lo[2], v.z);
      hi[0] = fmaxf(hi[0], v.x); hi[1] = fmaxf(hi[1], v.y); hi[2] = fmaxf(hi[2], v.z);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        lo[d] = fminf(lo[d], __shfl_xor_sync(FULL, lo[d], o));
        hi[d] = fmaxf(hi[d], __shfl_xor_sync(FULL, hi[d], o));
      }
    // neighbour cells, a lane each
    uint32_t nsub = 0;
    if (lane < 27) {
      const int off[3] = {lane % 3 - 1, (lane / 3) % 3 - 1, lane / 9 - 1};
      VdCell &v = cells[lane];
      int64_t jcoord[3];
      bool ok = true;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        int64_t j = ixyz[d] + off[d];
        float sh = 0.f;
        if ((r.pdim >> d) & 1) {
          if (j < 0) { j += Nd[d]; sh = (float)P.L; } else if (j >= Nd[d]) { j -= Nd[d]; sh = -(float)P.L; }
        } else if (j < 0 || j >= Nd[d]) ok = false;
        jcoord[d] = j;
        v.wl[d] = __fsub_rn(__fadd_rn(lo[d], sh), reach);
        v.wh[d] = __fadd_rn(__fadd_rn(hi[d], sh), reach);
      }
      const int64_t jl = jcoord[0] + Nd[0] * (jcoord[1] + Nd[1] * jcoord[2]);
      if (ok && jl >= local) {
        const uint64_t jc = r.cell_off + (uint64_t)jl;
        const uint32_t jb = cs[jc], nj = cs[jc + 1] - jb;
        if (is_vd(r, nj)) {
          const SubGrid gj = dense_sub(r, nj);
          int shi[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const float cl = cell_lower(r, d, jcoord[d]);
            v.slo[d] = sub_of(v.wl[d], cl, gj.inv[d], gj.s[d]);
            shi[d] = sub_of(v.wh[d], cl, gj.inv[d], gj.s[d]);
          }
          v.tab = tab + (int64_t)rank[jc] * stride;
          v.b = jb;
          v.nx = shi[0] - v.slo[0] + 1;
          v.ny = shi[1] - v.slo[1] + 1;
          v.s0 = gj.s[0];
          v.s01 = gj.s[0] * gj.s[1];
          v.own = jl == local;
          nsub = (uint32_t)(v.nx * v.ny * (shi[2] - v.slo[2] + 1));
        }
      }
    }
    uint32_t sub_end = nsub;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(FULL, sub_end, o);
      if (lane >= o) sub_end += v;
    }
    const uint32_t total = __shfl_sync(FULL, sub_end, 31);
    __syncwarp();
    int ra = dsu_find(parent, __float_as_int(dpos[a0].w));  // the same on every lane
    ra = __shfl_sync(FULL, ra, 0);
    for (uint32_t t0 = 0; t0 < total; t0 += 32) {
      const uint32_t k = t0 + (uint32_t)lane;
      int cell = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const uint32_t v = __shfl_sync(FULL, sub_end, cell + step - 1);
        if (v <= k) cell += step;
      }
      cell &= 31;
      const uint32_t k0 = __shfl_sync(FULL, sub_end - nsub, cell);
      uint32_t b0 = 0, b1 = 0;
      int hb = -1;  // root of B's set; -1: no candidate
      if (k < total) {
        const VdCell &v = cells[cell];
        const int q = (int)(k - k0), z = q / (v.nx * v.ny), rem = q - z * (v.nx * v.ny), y = rem / v.nx,
                  x = rem - y * v.nx;
        const int B = (v.slo[0] + x) + v.s0 * (v.slo[1] + y) + v.s01 * (v.slo[2] + z);
        if (!(v.own && B <= A)) {
          b0 = v.b + v.tab[B];
          b1 = v.b + v.tab[B + 1];
          if (b1 > b0) hb = dsu_find(parent, __float_as_int(dpos[b0].w));
        }
      }
      unsigned mask = __ballot_sync(FULL, hb >= 0 && hb != ra);
      while (mask) {
        const int src = __ffs(mask) - 1;
        mask &= mask - 1;
        const int hs = __shfl_sync(FULL, hb, src);
        const uint32_t s0 = __shfl_sync(FULL, b0, src), s1 = __shfl_sync(FULL, b1, src);
        const VdCell &v = cells[__shfl_sync(FULL, cell, src)];
        bool linked = false;
        for (int64_t ka = a0; ka < a1 && !linked; ka += 32) {
          const bool valid = ka + lane < a1;
          const float4 me = valid ? dpos[ka + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
          for (uint32_t kb = s0; kb < s1 && !linked; kb += 32) {
            const float4 o = kb + lane < s1 ? dpos[kb + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
            unsigned in = __ballot_sync(FULL, kb + lane < s1 && o.x >= v.wl[0] && o.x <= v.wh[0] && o.y >= v.wl[1] &&
                                                  o.y <= v.wh[1] && o.z >= v.wl[2] && o.z <= v.wh[2]);
            while (in && !linked) {
              const int j = __ffs(in) - 1;
              in &= in - 1;
              float4 so;
              so.x = __shfl_sync(FULL, o.x, j);
              so.y = __shfl_sync(FULL, o.y, j);
              so.z = __shfl_sync(FULL, o.z, j);
              so.w = 0.f;
              linked = __any_sync(FULL, valid && (per ? linked_pbc(me, so, P) : linked_open(me, so, P.rp2_open)));
            }
          }
        }
        if (!linked) continue;
        int joined = 0;
        if (lane == 0) joined = dsu_join(parent, ra, hs, flags);
        joined = __shfl_sync(FULL, joined, 0);
        if (hb == hs || hb == ra) hb = joined;
        ra = joined;
        mask &= __ballot_sync(FULL, hb >= 0 && hb != ra);
      }
    }
    __syncwarp();
  }
}

__global__ void fof_init_kernel(int *__restrict__ parent, uint32_t *__restrict__ gsize, int64_t n) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x) {
    parent[p] = (int)p;
    gsize[p] = 0;
  }
}

// Final labels.  The forest is static after linking; find() may still
// shorten paths with halving stores (each store points a node at one of its
// ancestors, so concurrent finds stay correct), but the label of every
// particle goes to a separate array: a store into parent[] could be
// overwritten by another thread's halving store with a non-root ancestor.
__global__ void __launch_bounds__(BLK) fof_root_kernel(int *parent, int *lab, uint32_t *gsize,
                                                       int64_t n) {
  for (int64_t base = (int64_t)blockIdx.x * BLK; base < n; base += (int64_t)gridDim.x * BLK) {
    const int64_t p = base + threadIdx.x;
    int root = -1;
    if (p < n) {
      root = dsu_find(parent, (int)p);
      lab[p] = root;
    }
    // one add per run of lanes with the same root (a match over the warp
    // costs more than the adds it saves)
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(0xffffffffu, root, 1);
    const bool head = lane == 0 || prev != root;
    const unsigned later = __ballot_sync(0xffffffffu, head) & ~(0xffffffffu >> (31 - lane));
    if (root >= 0 && head) atomicAdd(&gsize[root], (uint32_t)((later ? __ffs(later) - 1 : 32) - lane));
  }
}

// Candidates: roots whose group has at least nmin members (gsize is 0 at
// every other position).  Compacted in position order, tile by tile: counts
// per tile, a scan of the tiles, then the fill.
constexpr int CTILE = 4096;

__global__ void __launch_bounds__(BLK) fof_cand_count_kernel(const uint32_t *__restrict__ gsize, int64_t n,
                                                             uint32_t nmin, uint32_t *__restrict__ cnt) {
  __shared__ uint32_t red[BLK / 32];
  uint32_t c = 0;
  const int64_t b = (int64_t)blockIdx.x * CTILE, e = min(n, b + CTILE);
#pragma unroll
  for (int k = 0; k < CTILE / BLK; ++k) {
    const int64_t p = b + k * BLK + threadIdx.x;
    c += p < e && gsize[p] >= nmin;
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < BLK / 32; ++w) t += red[w];
    cnt[blockIdx.x] = t;
    if (blockIdx.x == 0) cnt[gridDim.x] = 0;
  }
}

__global__ void __launch_bounds__(BLK) fof_cand_fill_kernel(const uint32_t *__restrict__ gsize, int64_t n,
                                                            uint32_t nmin, const uint32_t *__restrict__ off,
                                                            int32_t *__restrict__ root) {
  if (off[blockIdx.x + 1] == off[blockIdx.x]) return;  // no candidate in the tile
  __shared__ uint32_t wsum[BLK / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t at = off[blockIdx.x];
  const int64_t b = (int64_t)blockIdx.x * CTILE, e = min(n, b + CTILE);
  for (int k = 0; k < CTILE / BLK; ++k) {
    const int64_t p = b + k * BLK + threadIdx.x;
    const bool f = p < e && gsize[p] >= nmin;
    const unsigned m = __ballot_sync(0xffffffffu, f);
    __syncthreads();
    if (lane == 0) wsum[warp] = __popc(m);
    __syncthreads();
    uint32_t before = at;
    for (int w = 0; w < BLK / 32; ++w) {
      if (w < warp) before += wsum[w];
      at += wsum[w];
    }
    if (f) root[before + __popc(m & lanemask_lt())] = (int32_t)p;
  }
}

// First member of every candidate in the reference's order (cell, then
// ascending original index): the root is the lowest position, so it lies in
// the group's first cell, and the first member is the lowest index among the
// group's members there (they follow the root).  A warp per candidate, where
// at most kAnchorScan positions follow: 128 steps.  A cell with more of them
// would be walked by each of its candidates, so its positions are queued
// once, in pieces (`piece`, flags[FLAG_PIECES]), for
// fof_cand_anchor_large_kernel.  flags[FLAG_RUN]: more than kCandRun
// candidates share a cell; they are then sorted instead of counted (all after
// the linking, 1,000 counted take 0.17 ms, 1,728 0.27, sorted 0.14).  With a
// walk and a count by every candidate 64,000 groups of one cell took 9.4 ms and
// 512,000 270 ms, now 0.23 and 0.44 ms; one group of 10^6 members in a cell
// 1.86 -> 0.13 ms.
constexpr int kAnchorScan = 4096, kCandRun = 1024;

__global__ void __launch_bounds__(BLK) fof_cand_anchor_kernel(const int32_t *__restrict__ root, int64_t ncand,
                                                              const int *__restrict__ lab,
                                                              const uint32_t *__restrict__ skey,
                                                              const uint32_t *__restrict__ cs,
                                                              const float4 *__restrict__ pos,
                                                              uint32_t *__restrict__ first,
                                                              uint32_t *__restrict__ crank,
                                                              uint2 *__restrict__ piece, int32_t *__restrict__ flags) {
  const int lane = threadIdx.x & 31;
  for (int64_t c = ((int64_t)blockIdx.x * BLK + threadIdx.x) >> 5; c < ncand; c += ((int64_t)gridDim.x * BLK) >> 5) {
    const int r = root[c];
    const uint32_t cell = skey[r];
    const int64_t e = cs[cell + 1];
    uint32_t m = 0xffffffffu;
    if (e - r <= kAnchorScan) {
      for (int64_t q = (int64_t)r + lane; q < e; q += 32)
        if (lab[q] == r) m = min(m, (uint32_t)__float_as_int(pos[q].w));
      m = __reduce_min_sync(0xffffffffu, m);
    } else if (c == 0 || skey[root[c - 1]] != cell) {  // the cell's first candidate
      const uint32_t k = (uint32_t)((e - r + kAnchorScan - 1) / kAnchorScan);
      uint32_t at = 0;
      if (lane == 0) at = (uint32_t)atomicAdd(&flags[FLAG_PIECES], (int32_t)k);
      at = __shfl_sync(0xffffffffu, at, 0);
      for (uint32_t i = lane; i < k; i += 32) {
        const uint32_t b = (uint32_t)r + i * kAnchorScan;
        piece[at + i] = make_uint2(b, min((uint32_t)e, b + kAnchorScan));
      }
    }
    if (lane == 0) {
      first[c] = m;
      crank[r] = (uint32_t)c;
      if (c + kCandRun < ncand && skey[root[c + kCandRun]] == cell) flags[FLAG_RUN] = 1;
    }
  }
}

// The first members of the candidates that were not walked, position by
// position: a block per queued piece.  A warp whose positions all belong to one
// group adds one minimum.
__global__ void __launch_bounds__(BLK) fof_cand_anchor_large_kernel(
    const uint2 *__restrict__ piece, const int32_t *__restrict__ flags, const int *__restrict__ lab,
    const uint32_t *__restrict__ skey, const uint32_t *__restrict__ cs, const uint32_t *__restrict__ gsize,
    uint32_t nmin, const float4 *__restrict__ pos, const uint32_t *__restrict__ crank,
    uint32_t *__restrict__ first) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, np = flags[FLAG_PIECES];
  for (int i = blockIdx.x; i < np; i += gridDim.x) {
    const uint2 p = piece[i];
    const uint32_t cell = skey[p.x];
    const int64_t begin = cs[cell], end = cs[cell + 1];
    for (uint32_t q0 = p.x + threadIdx.x - lane; q0 < p.y; q0 += BLK) {
      const uint32_t q = q0 + lane;
      const int r = q < p.y ? lab[q] : -1;
      // a root of this cell, of a group large enough, and not walked
      const bool mine = r >= begin && end - r > kAnchorScan && gsize[r] >= nmin;
      const uint32_t idx = mine ? (uint32_t)__float_as_int(pos[q].w) : 0xffffffffu;
      const int r0 = __shfl_sync(FULL, r, 0);
      if (__all_sync(FULL, r == r0)) {
        const uint32_t m = __reduce_min_sync(FULL, idx);
        if (mine && lane == 0) atomicMin(&first[crank[r]], m);
      } else if (mine) {
        uint32_t *f = &first[crank[r]];
        if (idx < __ldcg(f)) atomicMin(f, idx);
      }
    }
  }
}

// Cells of the candidates in `order`.
__global__ void fof_cand_cell_kernel(const uint32_t *__restrict__ order, int64_t ncand,
                                     const int32_t *__restrict__ root, const uint32_t *__restrict__ skey,
                                     uint32_t *__restrict__ cell) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncand; c += (int64_t)gridDim.x * blockDim.x)
    cell[c] = skey[root[order[c]]];
}

// Candidate ids: position order, and by first member among candidates whose
// roots share a cell: counted among them or, where more than kCandRun do,
// taken from the candidates sorted that way (`order`).
__global__ void fof_cand_info_kernel(const int32_t *__restrict__ root, int64_t ncand,
                                     const uint32_t *__restrict__ first, const uint32_t *__restrict__ order,
                                     const uint32_t *__restrict__ skey,
                                     const uint32_t *__restrict__ prid, const uint32_t *__restrict__ gsize,
                                     uint32_t *__restrict__ crank, int64_t *__restrict__ cand_anchor,
                                     int32_t *__restrict__ cand_region, int32_t *__restrict__ cand_np,
                                     int32_t *__restrict__ cand_root) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < ncand;
       j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = order ? order[j] : j;
    const int r = root[c];
    const uint32_t f = first[c];
    int64_t id = j;
    if (!order) {
      const uint32_t cell = skey[r];
      for (int64_t k = c - 1; k >= 0 && skey[root[k]] == cell; --k) id -= first[k] > f;
      for (int64_t k = c + 1; k < ncand && skey[root[k]] == cell; ++k) id += first[k] < f;
    }
    crank[r] = (uint32_t)id;
    cand_anchor[id] = f;
    cand_region[id] = prid ? (int32_t)prid[r] : 0;
    cand_np[id] = (int32_t)gsize[r];
    cand_root[id] = r;
  }
}

// Candidate of every sorted particle (-1 if its group is too small), plus
// the no-unbinding outputs (fof_fortran.f90:207-222).
__global__ void fof_member_kernel(const int *lab, const uint32_t *gsize,
                                  const uint32_t *crank, const float4 *pos, int64_t n,
                                  uint32_t np_min, int write_out, int32_t *pcand,
                                  int32_t *in_halo, int32_t *halo_id) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int r = lab[p];
    int32_t c = -1;
    if (gsize[r] >= np_min) c = (int32_t)crank[r];
    pcand[p] = c;
    if (write_out && c >= 0) {
      const int i = __float_as_int(pos[p].w);
      if (in_halo) in_halo[i] = 1;
      halo_id[i] = c + 1;
    }
  }
}

// Per-candidate weighted sums for the centre of mass and mean velocity
// (fof_fortran.f90:225-238): acc[c] = {w, w*dx, w*dv}.
__global__ void __launch_bounds__(BLK) fof_com_kernel(Coords xp, Coords vp, const double *mp,
                                                      const float4 *pos, const int32_t *pcand,
                                                      const int64_t *cand_anchor, int64_t n,
                                                      double L, double half, double *acc) {
  for (int64_t base = (int64_t)blockIdx.x * BLK; base < n; base += (int64_t)gridDim.x * BLK) {
    const int64_t p = base + threadIdx.x;
    int32_t c = p < n ? pcand[p] : -1;
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    if (c >= 0) {
      const int64_t i = __float_as_int(pos[p].w);
      const int64_t a = cand_anchor[c];
      const double w = mp ? mp[i] : 1.0;
      v[0] = w;
      for (int d = 0; d < 3; ++d) {
        v[1 + d] = w * unwrap(xp.get(i, d), xp.get(a, d), half, L);
        v[4 + d] = w * vp.get(i, d);
      }
    }
    const unsigned peers = __match_any_sync(0xffffffffu, c);
    if (peers == 0xffffffffu) {
      for (int k = 0; k < 7; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
      if ((threadIdx.x & 31) == 0 && c >= 0)
        for (int k = 0; k < 7; ++k) atomicAdd(&acc[7 * (int64_t)c + k], v[k]);
    } else if (c >= 0) {
      for (int k = 0; k < 7; ++k) atomicAdd(&acc[7 * (int64_t)c + k], v[k]);
    }
  }
}

// Angular momentum about the candidate centre (fof_fortran.f90:239-247),
// accumulated per candidate.
__global__ void __launch_bounds__(BLK) fof_angmom_kernel(Coords xp, Coords vp, const double *mp,
                                                         const float4 *pos, const int32_t *pcand,
                                                         const int64_t *cand_anchor,
                                                         const double *acc, int64_t n, double L,
                                                         double half, double *am) {
  for (int64_t base = (int64_t)blockIdx.x * BLK; base < n; base += (int64_t)gridDim.x * BLK) {
    const int64_t p = base + threadIdx.x;
    int32_t c = p < n ? pcand[p] : -1;
    double v[3] = {0, 0, 0};
    if (c >= 0 && acc[7 * (int64_t)c] > 0.0) {
      const int64_t i = __float_as_int(pos[p].w);
      const int64_t a = cand_anchor[c];
      const double ws = acc[7 * (int64_t)c];
      const double w = mp ? mp[i] : 1.0;
      double dx[3], dv[3];
      for (int d = 0; d < 3; ++d) {
        dx[d] = unwrap(xp.get(i, d), xp.get(a, d), half, L) - acc[7 * (int64_t)c + 1 + d] / ws;
        dv[d] = vp.get(i, d) - acc[7 * (int64_t)c + 4 + d] / ws;
      }
      v[0] = w * (dx[1] * dv[2] - dx[2] * dv[1]);
      v[1] = w * (dx[2] * dv[0] - dx[0] * dv[2]);
      v[2] = w * (dx[0] * dv[1] - dx[1] * dv[0]);
    }
    const unsigned peers = __match_any_sync(0xffffffffu, c);
    if (peers == 0xffffffffu) {
      for (int k = 0; k < 3; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
      if ((threadIdx.x & 31) == 0 && c >= 0)
        for (int k = 0; k < 3; ++k) atomicAdd(&am[3 * (int64_t)c + k], v[k]);
    } else if (c >= 0) {
      for (int k = 0; k < 3; ++k) atomicAdd(&am[3 * (int64_t)c + k], v[k]);
    }
  }
}

int bits_for(uint64_t v) {
  int b = 0;
  while (b < 64 && (v >> b) != 0) ++b;
  return b;
}

}  // namespace

// ------------------------------------------------------- host geometry

// Half-width of the cube that holds every partner the distance test can
// accept: slack relative 1e-4 for the FP32 distance arithmetic, 8 FP32 ulps
// of the box size for the rounding of positions and query endpoints.
static double link_reach(double L, double link) {
  return link * (1.0 + 1e-4) + 8.0 * 1.1920928955078125e-07 * (std::fabs(L) + 1.0);
}

// Reference cell geometry of one region (fof_fortran.f90:528-570) from its
// unwrapped bounding box.  64-bit integers are used where the reference's
// default integers would overflow (N >= 2**29).
void region_geometry(double L, double link, int32_t np, const double *xmin, const double *xmax,
                     RegionDev &r) {
  const double half = 0.5 * L;
  double range[3];
  int pd = 0;
  for (int d = 0; d < 3; ++d) {
    range[d] = xmax[d] - xmin[d];
    if (range[d] + 2.0 * link >= L) pd |= 1 << d;
  }
  const double vol = std::max(range[0], link) * std::max(range[1], link) * std::max(range[2], link);
  auto geom = [&](double L_mesh, int64_t *N) {
    for (int d = 0; d < 3; ++d) {
      if ((pd >> d) & 1) {
        r.origin[d] = -half;
        int64_t a = (int64_t)(L / link), b = (int64_t)(L / L_mesh);
        N[d] = std::max<int64_t>(1, std::min(a, b));
        r.size[d] = L / (double)N[d];
      } else {
        r.origin[d] = xmin[d];
        N[d] = std::max<int64_t>(1, (int64_t)std::ceil(range[d] / L_mesh));
        r.size[d] = L_mesh;
      }
    }
  };
  int64_t N[3];
  double L_mesh = std::max(link, std::pow(vol / (double)std::max(1, np), 1.0 / 3.0));
  geom(L_mesh, N);
  const int64_t cap = std::max<int64_t>(262144, 4 * (int64_t)np);
  if ((double)N[0] * (double)N[1] * (double)N[2] > (double)cap) {
    L_mesh = std::pow(vol / (double)((int64_t)std::max(1, np) * 2), 1.0 / 3.0);
    L_mesh = std::max(link, L_mesh);
    geom(L_mesh, N);
  }
  for (int d = 0; d < 3; ++d) r.N[d] = (int32_t)std::min<int64_t>(N[d], INT32_MAX);
  r.pdim = pd;
  r.periodic = pd != 0;
  r.ncell = N[0] * N[1] * N[2];
  // sub-cells for dense cells: slabs at least one linking length wide; none
  // along periodic axes with fewer than 3 cells (both images are adjacent)
  for (int d = 0; d < 3; ++d) {
    int sd = (int)std::floor(r.size[d] / link);
    if (sd < 1 || !std::isfinite(r.size[d] / link)) sd = 1;
    if (sd > 6) sd = 6;
    if (((pd >> d) & 1) && N[d] < 3) sd = 1;
    r.sub[d] = sd;
  }
  r.near_ok = r.size[0] <= 0.24 * L && r.size[1] <= 0.24 * L && r.size[2] <= 0.24 * L;
  for (int d = 0; d < 3; ++d) r.inv_sub[d] = (float)((double)r.sub[d] / r.size[d]);
  const double reach = link_reach(L, link);
  for (int d = 0; d < 3; ++d) {
    r.inv_size[d] = 1.0 / r.size[d];
    r.org[d] = (float)r.origin[d];
    r.cinv[d] = (float)r.inv_size[d];
    // FP32 error of (x - org) * cinv: a few ulps of the coordinates, in
    // cells, and of the product (at most N)
    const double sl = 1e-4 + 4e-7 * (double)N[d] + 4e-7 * (std::fabs(L) + std::fabs(r.origin[d])) / r.size[d];
    r.slack[d] = (float)std::min(sl, 2.0);
    r.near[d] = (float)std::min(reach / r.size[d] + sl, 2.0);
    if (d < 2) r.div[d] = N[d] > 1 ? ~(uint64_t)0 / (uint64_t)N[d] + 1 : 0;
  }
  // merge sub-cells: width at most link/sqrt(3) * 0.999 less 8 FP32 ulps of
  // the box size (the rounding of positions and sub-cell boundaries), so the
  // largest distance inside one, as the FP32/FP64 test computes it, stays
  // below the linking length; only where a cell holds at most SUB_MAX of
  // them and no periodic axis has fewer than 3 cells
  const double mw = link / std::sqrt(3.0) * 0.999 - 8.0 * 1.1920928955078125e-07 * (std::fabs(L) + 1.0);
  int64_t km = 1;
  int k[3] = {0, 0, 0};
  bool vd = mw > 0.0 && std::isfinite(mw);
  for (int d = 0; d < 3 && vd; ++d) {
    const double kk = std::ceil(r.size[d] / mw);
    if (!(kk >= 1.0) || kk > (double)SUB_MAX || (((pd >> d) & 1) && N[d] < 3)) vd = false;
    else { k[d] = (int)kk; km *= k[d]; }
  }
  if (vd && km > SUB_MAX) vd = false;
  for (int d = 0; d < 3; ++d) {
    r.vd_k[d] = vd ? k[d] : 0;
    r.vd_inv[d] = vd ? (float)((double)k[d] / r.size[d]) : 0.0f;
  }
}

int32_t fof_link_stage(Context &ctx, const FofArgs &a, FofState &st) {
  cudaStream_t s = ctx.stream;
  Arena &W = ctx.work;
  const int64_t n = a.total_np;
  const int nreg = a.nhalo;
  const double L = a.L_Box, half = 0.5 * a.L_Box;
  st.n = n;
  st.nreg = nreg;
  Coords xp{a.xp, n, a.soa};

  // --- region table and tiles (host)
  const int64_t tile = n <= kTileSmallUpTo ? TILE_SMALL : TILE;
  int64_t total = 0, ntiles = 0;
  for (int r = 0; r < nreg; ++r) {
    total += a.np_halo[r];
    ntiles += a.np_halo[r] > 0 ? ceil_div(a.np_halo[r], tile) : 0;
  }
  if (total != n) {
    set_error("sum(np_halo)=%lld != total_np=%lld", (long long)total, (long long)n);
    return kInvalid;
  }
  // one block of tables: regions, cell offsets, bounding boxes, an error
  // word, tiles; uploaded together, the boxes and the error word read back
  // together, regions and offsets uploaded again with the geometry
  const size_t o_off = sizeof(RegionDev) * nreg, o_bb = o_off + sizeof(uint64_t) * (nreg + 1),
               o_err = o_bb + 6 * sizeof(uint64_t) * nreg, o_tile = o_err + sizeof(uint64_t),
               tab_bytes = o_tile + sizeof(Tile) * ntiles;
  static_assert(sizeof(RegionDev) % 8 == 0, "the tables that follow hold 64-bit values");
  uint8_t *dtab = W.carve<uint8_t>(tab_bytes);
  if (!dtab) { set_error("workspace exhausted (regions)"); return kAlloc; }
  RegionDev *dR = reinterpret_cast<RegionDev *>(dtab);
  uint64_t *dcoff = reinterpret_cast<uint64_t *>(dtab + o_off);
  unsigned long long *dbb = reinterpret_cast<unsigned long long *>(dtab + o_bb);
  int32_t *derr = reinterpret_cast<int32_t *>(dtab + o_err);
  Tile *dT = reinterpret_cast<Tile *>(dtab + o_tile);
  std::vector<uint64_t> large_tab;
  uint64_t *tab = ctx.host_words((tab_bytes + 7) / 8, large_tab);
  uint8_t *htab = reinterpret_cast<uint8_t *>(tab);
  RegionDev *reg = reinterpret_cast<RegionDev *>(htab);
  uint64_t *cell_off = tab + o_off / 8, *bb = tab + o_bb / 8;
  Tile *tiles = reinterpret_cast<Tile *>(htab + o_tile);
  memset(htab, 0, o_tile);
  int64_t start = 0;
  for (int r = 0; r < nreg; ++r) {
    RegionDev &R = reg[r];
    R.start = start;
    R.np = a.np_halo[r];
    R.active = (R.np >= a.np_halo_min && R.np > 0) ? 1 : 0;
    for (int64_t b = start; b < start + R.np; b += tile)
      *tiles++ = Tile{r, 0, b, std::min<int64_t>(start + R.np, b + tile)};
    start += R.np;
    for (int d = 0; d < 3; ++d) bb[6 * (size_t)r + d] = ~0ull;  // minima; maxima start at 0
  }
  PYFOF_TRY(upload(ctx, dtab, htab, tab_bytes, s));
  PYFOF_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(int32_t) * FLAG_COUNT, s));
  if (ntiles) {
    fof_bbox_kernel<<<(unsigned)ntiles, BLK, 0, s>>>(xp, dR, dT, L, half, dbb, derr);
    PYFOF_CHECK_LAUNCH();
  }
  PYFOF_CUDA(cudaMemcpyAsync(bb, dbb, sizeof(uint64_t) * (6 * (size_t)nreg + 1), cudaMemcpyDeviceToHost, s));
  PYFOF_CUDA(cudaStreamSynchronize(s));
  if (const int32_t err = (int32_t)bb[6 * (size_t)nreg]) {
    set_error("non-finite particle coordinates");
    return err;
  }

  // --- reference geometry per region (host)
  uint64_t total_cells = 0;
  int64_t n_active = 0;
  for (int r = 0; r < nreg; ++r) {
    RegionDev &R = reg[r];
    cell_off[r] = total_cells;
    R.cell_off = total_cells;
    if (!R.active) continue;
    double xmin[3], xmax[3];
    for (int d = 0; d < 3; ++d) {
      xmin[d] = ord_to_dbl(bb[6 * r + d]);
      xmax[d] = ord_to_dbl(bb[6 * r + 3 + d]);
    }
    region_geometry(L, a.link, R.np, xmin, xmax, R);
    total_cells += (uint64_t)R.ncell;
    n_active += R.np;
  }
  cell_off[nreg] = total_cells;
  if (total_cells >= 0xffffffffull) {
    set_error("total cell count %llu exceeds the 32-bit key range",
              (unsigned long long)total_cells);
    return kAlloc;
  }
  st.n_active = n_active;
  st.total_cells = total_cells;
  ctx.last_cells = (int64_t)total_cells;
  ctx.last_active = n_active;
  PYFOF_TRY(upload(ctx, dtab, htab, o_bb, s));
  uint32_t *keys = W.carve<uint32_t>(std::max<int64_t>(n, 1));
  uint32_t *cstart = W.carve<uint32_t>(total_cells + 2);
  if (!keys || !cstart) {
    set_error("workspace exhausted (keys)");
    return kAlloc;
  }
  PYFOF_CUDA(cudaMemsetAsync(cstart, 0, sizeof(uint32_t) * (total_cells + 2), s));
  // the particles' slots within their cells (sort scratch in the sorted modes)
  uint32_t *slot = W.carve<uint32_t>(std::max<int64_t>(n, 1));
  uint32_t *skey = W.carve<uint32_t>(std::max<int64_t>(n, 1));
  float4 *pos = W.carve<float4>(std::max<int64_t>(n_active, 1));
  uint32_t *prid = nreg > 1 ? W.carve<uint32_t>(std::max<int64_t>(n_active, 1)) : nullptr;
  if (!slot || !skey || !pos || (nreg > 1 && !prid)) { set_error("workspace exhausted (keys)"); return kAlloc; }
  const uint32_t sentinel = (uint32_t)total_cells;
  if (ntiles) {
    fof_key_kernel<<<(unsigned)ntiles, BLK, 0, s>>>(xp, dR, dT, L, half, sentinel, a.cell_order != 0,
                                                    (uint32_t)(total_cells / 64), keys, cstart, slot, ctx.d_flags);
    PYFOF_CHECK_LAUNCH();
  }
  PYFOF_TRY(exclusive_scan_u32(cstart, cstart, (int64_t)total_cells + 1, nullptr, W, s));
  // dense cells: at most n / (DENSE_T + 1); their chunks: one per 32
  // particles and one more per cell
  const size_t dense_cap = (size_t)n_active / (DENSE_T + 1) + 1;
  uint32_t *list = W.carve<uint32_t>(dense_cap);
  uint32_t *drank = W.carve<uint32_t>(total_cells + 1);
  DenseChunk *dchunks = W.carve<DenseChunk>((size_t)n_active / 32 + dense_cap);
  if (!list || !drank || !dchunks) { set_error("workspace exhausted (dense cells)"); return kAlloc; }
  uint32_t *dcells = reinterpret_cast<uint32_t *>(ctx.d_flags + FLAG_COUNT_A);  // A, B, C (zero)
  if (total_cells > 0) {
    const unsigned cgrid = (unsigned)std::min<int64_t>(ceil_div((int64_t)total_cells, (int64_t)BLK), (int64_t)kNumSMs * 16);
    fof_cells_kernel<<<cgrid, BLK, 0, s>>>(cstart, (int64_t)total_cells, dcells, list, drank, dchunks, skey);
    PYFOF_CHECK_LAUNCH();
  }
  PYFOF_CUDA(cudaMemcpyAsync(ctx.h_flags, ctx.d_flags, sizeof(int32_t) * FLAG_COUNT, cudaMemcpyDeviceToHost, s));
  ctx.last_cell_sorts = 0;
  PYFOF_CUDA(cudaStreamSynchronize(s));
  float4 *spare = nullptr;  // a float4 per particle, free after the scatter
  if (a.cell_order == 0 && n_active > 0) {
    if (use_partition(nreg, n_active, ntiles, ctx.h_flags[FLAG_SPREAD])) {
      spare = W.carve<float4>(n_active);
      uint2 *tkey = W.carve<uint2>(n_active);
      uint32_t *cursor = W.carve<uint32_t>(kBuckets);
      if (!spare || !tkey || !cursor) { set_error("workspace exhausted (scatter)"); return kAlloc; }
      fof_bucket_start_kernel<<<1, kBuckets, 0, s>>>(cstart, (uint32_t)total_cells, cursor);
      PYFOF_CHECK_LAUNCH();
      fof_partition_kernel<<<(unsigned)ceil_div(n, (int64_t)PTILE), BLK, 0, s>>>(xp, n, L, half, keys, slot,
                                                                                 (uint32_t)total_cells, cursor, spare,
                                                                                 tkey);
      PYFOF_CHECK_LAUNCH();
      fof_place_kernel<<<(unsigned)ceil_div(n, (int64_t)LU * BLK), BLK, 0, s>>>(spare, tkey, n, cstart, pos);
      PYFOF_CHECK_LAUNCH();
    } else {
      fof_scatter_kernel<<<(unsigned)ntiles, BLK, 0, s>>>(xp, dR, dT, L, half, keys, slot, cstart, pos, prid);
      PYFOF_CHECK_LAUNCH();
    }
  }
  const int64_t ndense = (uint32_t)ctx.h_flags[FLAG_COUNT_A], ndense_chunks = (uint32_t)ctx.h_flags[FLAG_COUNT_B];
  const uint32_t max_occ = (uint32_t)ctx.h_flags[FLAG_COUNT_C];
  ctx.last_max_cell = max_occ;
  ctx.last_dense = ndense;
  if (a.cell_order != 0) {
    // the reference's CRS order itself
    uint32_t *sidx = nullptr;
    uint32_t *ka = skey, *va = slot, *kb = W.carve<uint32_t>(std::max<int64_t>(n, 1)),
             *vb = W.carve<uint32_t>(std::max<int64_t>(n, 1));
    if (!kb || !vb) { set_error("workspace exhausted (cell order)"); return kAlloc; }
    if (a.cell_order == 1 && max_occ <= (uint32_t)CELL_SORT_MAX) {
      ctx.last_cell_sorts = 1;
      // cells of more than CELL_SORT_SMALL particles: at most n / (CELL_SORT_SMALL + 1)
      uint32_t *big = W.carve<uint32_t>(
          (size_t)std::min<int64_t>(n_active / (CELL_SORT_SMALL + 1) + 1, (int64_t)total_cells + 1));
      uint32_t *nbig = W.carve<uint32_t>(1);
      if (!big || !nbig) { set_error("workspace exhausted (cell sort)"); return kAlloc; }
      PYFOF_CUDA(cudaMemsetAsync(nbig, 0, sizeof(uint32_t), s));
      const unsigned sgrid = (unsigned)std::max<int64_t>(
          1, std::min<int64_t>(ceil_div(std::max<int64_t>(n, 1), (int64_t)BLK), (int64_t)kNumSMs * 16));
      fof_cell_scatter_kernel<<<sgrid, BLK, 0, s>>>(keys, slot, cstart, n, ka, vb);
      PYFOF_CHECK_LAUNCH();
      if (total_cells > 0) {
        const unsigned cgrid = (unsigned)std::min<int64_t>(ceil_div((int64_t)total_cells, (int64_t)BLK),
                                                           (int64_t)kNumSMs * 16);
        fof_cell_sort_small_kernel<<<cgrid, BLK, 0, s>>>(cstart, (int64_t)total_cells, vb, big, nbig);
        PYFOF_CHECK_LAUNCH();
        fof_cell_sort_big_kernel<<<kNumSMs * 2, 1024, 0, s>>>(cstart, big, nbig, vb);
        PYFOF_CHECK_LAUNCH();
      }
      sidx = vb;
    } else {
      const uint64_t max_key = (n_active < n) ? total_cells : (total_cells ? total_cells - 1 : 0);
      PYFOF_TRY(radix_sort_pairs(keys, nullptr, n, bits_for(max_key), ka, va, kb, vb, &skey, &sidx, W, s));
    }
    if (n_active > 0) {
      const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(n_active, BLK), (int64_t)kNumSMs * 16);
      fof_gather_kernel<<<grid, BLK, 0, s>>>(xp, dR, dcoff, nreg, skey, sidx, n_active, L, half, pos, prid);
      PYFOF_CHECK_LAUNCH();
    }
  }
  int *parent = W.carve<int>(std::max<int64_t>(n_active, 1));
  uint32_t *gsize = W.carve<uint32_t>(std::max<int64_t>(n_active, 1));
  if (!parent || !gsize) { set_error("workspace exhausted (link)"); return kAlloc; }
  const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(std::max<int64_t>(n_active, 1), BLK),
                                                    (int64_t)kNumSMs * 16);
  if (n_active > 0) {
    fof_init_kernel<<<grid, BLK, 0, s>>>(parent, gsize, n_active);
    PYFOF_CHECK_LAUNCH();
    LinkParams P;
    P.L = L;
    P.half = half;
    P.rp2 = a.link * a.link;
    {
      float f = (float)P.rp2;
      if ((double)f > P.rp2) f = std::nextafter(f, -INFINITY);
      P.rp2_open = f;
    }
    P.fast_periodic = (P.rp2 > 1e-20 && P.rp2 < 1e20 && L < 1e30) ? 1 : 0;
    P.rp2_lo = (float)(P.rp2 * (1.0 - 4e-6));
    P.rp2_hi = (float)(P.rp2 * (1.0 + 4e-6));
    DenseIndex D{};
    bool any_vd = false;               // a region where very dense cells can occur
    for (int r = 0; r < nreg; ++r) any_vd = any_vd || (reg[r].active && reg[r].vd_k[0] > 0);
    D.reach = (float)link_reach(L, a.link);
    if (ndense > 0) {
      int smax = 1;
      for (int r = 0; r < nreg; ++r)
        if (reg[r].active) {
          smax = std::max(smax, reg[r].sub[0] * reg[r].sub[1] * reg[r].sub[2]);
          smax = std::max(smax, reg[r].vd_k[0] * reg[r].vd_k[1] * reg[r].vd_k[2]);
        }
      D.stride = smax + 1;
      float4 *dpos = spare ? spare : W.carve<float4>(n_active);
      uint32_t *tab = W.carve<uint32_t>(ndense * D.stride);
      if (!dpos || !tab) { set_error("workspace exhausted (dense tables)"); return kAlloc; }
      fof_dense_build_kernel<<<(unsigned)ndense, BLK, 0, s>>>(list, cstart, pos, dR, dcoff, nreg, D.stride, tab,
                                                              dpos, P, parent);
      PYFOF_CHECK_LAUNCH();
      D.rank = drank;
      D.tab = tab;
      D.dpos = dpos;
    }
    // dense-cell particles and the rest as two launches: the long pair loops
    // of the dense part do not hold back blocks of the short sparse work
    if (ctx.timing) cudaEventRecord(ctx.ev[0], s);
    if (ctx.last_dense > 0 && any_vd) {
      int2 *vd = W.carve<int2>(ctx.last_dense);
      if (!vd) { set_error("workspace exhausted (very dense cells)"); return kAlloc; }
      int vd_max = 1;
      for (int r = 0; r < nreg; ++r)
        if (reg[r].active) vd_max = std::max(vd_max, reg[r].vd_k[0] * reg[r].vd_k[1] * reg[r].vd_k[2]);
      fof_vd_intra_kernel<<<(unsigned)ctx.last_dense, BLK, 0, s>>>(list, cstart, dR, dcoff, nreg, D.stride,
                                                                   D.tab, D.dpos, parent, vd, ctx.d_flags);
      PYFOF_CHECK_LAUNCH();
      const int64_t vd_blocks = ceil_div((int64_t)ctx.last_dense * vd_max, BLK / 32);
      fof_vd_inter_kernel<<<(unsigned)std::min<int64_t>(vd_blocks, kNumSMs * 5), BLK, 0, s>>>(
          list, cstart, dR, vd, vd_max, D.stride, D.tab, D.rank, D.dpos, parent, P, D.reach, ctx.d_flags);
      PYFOF_CHECK_LAUNCH();
    }
    if (ndense_chunks > 0) {
      // warps per chunk: up to 8 while the blocks all fit on the chip at once
      int lg = 0;
      while (lg < 3 && ndense_chunks << (lg + 1) <= (int64_t)kNumSMs * 4 * (BLK / 32)) ++lg;
      const unsigned dgrid = (unsigned)std::min<int64_t>(ceil_div((ndense_chunks << lg) * 32, BLK),
                                                         (int64_t)kNumSMs * 24);
      fof_link_dense_kernel<<<dgrid, BLK, 0, s>>>(pos, prid, dR, cstart, parent, dchunks, ndense_chunks, lg, P, D,
                                                  ctx.d_flags);
      PYFOF_CHECK_LAUNCH();
    }
    fof_link_kernel<<<grid, BLK, 0, s>>>(pos, skey, prid, dR, cstart, parent, n_active, P, ctx.d_flags);
    PYFOF_CHECK_LAUNCH();
    if (ctx.timing) cudaEventRecord(ctx.ev[1], s);
  }
  st.dR = dR;
  st.pos = pos;
  st.prid = prid;
  st.parent = parent;
  st.skey = skey;
  st.gsize = gsize;
  st.cell_start = cstart;
  st.keys_free = keys;
  return kOk;
}

int32_t fof_candidates_stage(Context &ctx, const FofArgs &a, FofState &st, bool write_plain) {
  cudaStream_t s = ctx.stream;
  Arena &W = ctx.work;
  const int64_t na = st.n_active;
  uint32_t *crank = W.carve<uint32_t>(std::max<int64_t>(na, 1));
  int32_t *pcand = W.carve<int32_t>(std::max<int64_t>(na, 1));
  const int64_t ntile = std::max<int64_t>(ceil_div(na, (int64_t)CTILE), 1);
  uint32_t *toff = W.carve<uint32_t>(ntile + 1);
  if (!crank || !pcand || !toff) { set_error("workspace exhausted (labels)"); return kAlloc; }
  // (every root has at least itself: a minimum of 0 takes all of them too)
  const uint32_t nmin = a.np_halo_min == 0 ? 1u : (uint32_t)a.np_halo_min;
  const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(std::max<int64_t>(na, 1), BLK), (int64_t)kNumSMs * 16);
  st.ncand = 0;
  if (na > 0) {
    st.lab = reinterpret_cast<int *>(st.keys_free);  // keys are dead after the scatter
    fof_root_kernel<<<grid, BLK, 0, s>>>(st.parent, st.lab, st.gsize, na);
    PYFOF_CHECK_LAUNCH();
    fof_cand_count_kernel<<<(unsigned)ntile, BLK, 0, s>>>(st.gsize, na, nmin, toff);
    PYFOF_CHECK_LAUNCH();
    PYFOF_TRY(exclusive_scan_u32(toff, toff, ntile + 1, reinterpret_cast<uint32_t *>(ctx.d_flags + FLAG_COUNT_A), W,
                                 s));
    PYFOF_CUDA(cudaMemcpyAsync(ctx.h_flags, ctx.d_flags, sizeof(int32_t) * FLAG_COUNT,
                               cudaMemcpyDeviceToHost, s));
    PYFOF_CUDA(cudaStreamSynchronize(s));
    if (ctx.h_flags[FLAG_ERR]) {
      set_error("linking failed (DSU retry cap)");
      return ctx.h_flags[FLAG_ERR];
    }
    st.ncand = (uint32_t)ctx.h_flags[FLAG_COUNT_A];
  }
  ctx.last_candidates = st.ncand;
  st.crank = crank;
  st.pcand = pcand;
  const int64_t nc = std::max<int64_t>(st.ncand, 1);
  st.cand_anchor = W.carve<int64_t>(nc);
  st.cand_np = W.carve<int32_t>(3 * nc);
  st.cand_region = st.cand_np + nc;
  st.cand_root = st.cand_np + 2 * nc;
  int32_t *root = W.carve<int32_t>(nc);
  uint32_t *first = W.carve<uint32_t>(nc);
  if (!st.cand_anchor || !st.cand_np || !root || !first) {
    set_error("workspace exhausted (candidates)");
    return kAlloc;
  }
  if (st.ncand > 0) {
    fof_cand_fill_kernel<<<(unsigned)ntile, BLK, 0, s>>>(st.gsize, na, nmin, toff, root);
    PYFOF_CHECK_LAUNCH();
    const unsigned gw = (unsigned)std::min<int64_t>(ceil_div(nc * 32, (int64_t)BLK), (int64_t)kNumSMs * 16);
    const unsigned gc = (unsigned)std::min<int64_t>(ceil_div(nc, (int64_t)BLK), (int64_t)kNumSMs * 16);
    const bool large = ctx.last_max_cell > kAnchorScan;  // (no candidate is left to the second kernel otherwise)
    uint2 *piece = nullptr;
    if (large) {
      // cells of more than kAnchorScan positions, ceil(size / kAnchorScan) pieces each
      piece = W.carve<uint2>(2 * (size_t)na / kAnchorScan + 1);
      if (!piece) { set_error("workspace exhausted (candidates)"); return kAlloc; }
    }
    fof_cand_anchor_kernel<<<gw, BLK, 0, s>>>(root, nc, st.lab, st.skey, st.cell_start, st.pos, first, crank, piece,
                                              ctx.d_flags);
    PYFOF_CHECK_LAUNCH();
    if (large) {
      fof_cand_anchor_large_kernel<<<kNumSMs * 4, BLK, 0, s>>>(piece, ctx.d_flags, st.lab, st.skey, st.cell_start,
                                                               st.gsize, nmin, st.pos, crank, first);
      PYFOF_CHECK_LAUNCH();
    }
    uint32_t *order = nullptr;
    const size_t before_sort = W.mark();
    if (ctx.last_max_cell > kCandRun && nc > kCandRun) {
      PYFOF_CUDA(cudaMemcpyAsync(ctx.h_flags, ctx.d_flags, sizeof(int32_t) * FLAG_COUNT, cudaMemcpyDeviceToHost, s));
      PYFOF_CUDA(cudaStreamSynchronize(s));
      if (ctx.h_flags[FLAG_RUN]) {
        // by first member, then (stable) by cell
        uint32_t *b[5];
        for (uint32_t *&p : b)
          if (!(p = W.carve<uint32_t>(nc))) { set_error("workspace exhausted (candidate order)"); return kAlloc; }
        uint32_t *k1, *v1, *k2;
        PYFOF_TRY(radix_sort_pairs(first, nullptr, nc, bits_for((uint64_t)a.total_np - 1), b[0], b[1], b[2], b[3], &k1,
                                   &v1, W, s));
        fof_cand_cell_kernel<<<gc, BLK, 0, s>>>(v1, nc, root, st.skey, b[4]);
        PYFOF_CHECK_LAUNCH();
        // the keys of the first sort are done with; its values are the input
        uint32_t *const spare = v1 == b[1] ? b[3] : b[1];
        uint32_t *const own = v1 == b[1] ? b[1] : b[3];
        PYFOF_TRY(radix_sort_pairs(b[4], v1, nc, bits_for(st.total_cells - 1), b[0], spare, b[2], own, &k2, &order, W,
                                   s));
      }
    }
    fof_cand_info_kernel<<<gc, BLK, 0, s>>>(root, nc, first, order, st.skey, st.prid, st.gsize, crank, st.cand_anchor,
                                            st.cand_region, st.cand_np, st.cand_root);
    PYFOF_CHECK_LAUNCH();
    W.release_to(before_sort);
    fof_member_kernel<<<grid, BLK, 0, s>>>(st.lab, st.gsize, crank, st.pos, na, nmin, write_plain ? 1 : 0, pcand,
                                           a.in_halo, a.halo_id);
    PYFOF_CHECK_LAUNCH();
  }
  return kOk;
}

// ang_mom per input region over all candidates (no unbinding):
// fof_fortran.f90:224-248.
int32_t fof_plain_angmom(Context &ctx, const FofArgs &a, FofState &st) {
  cudaStream_t s = ctx.stream;
  Arena &W = ctx.work;
  const int nreg = a.nhalo;
  std::vector<double> am_host(3 * (size_t)nreg, 0.0);
  if (st.ncand > 0 && a.vp) {
    const int64_t na = st.n_active, nc = st.ncand;
    double *acc = W.carve<double>(10 * (size_t)nc);
    if (!acc) { set_error("workspace exhausted (ang_mom)"); return kAlloc; }
    double *am = acc + 7 * (size_t)nc;
    PYFOF_CUDA(cudaMemsetAsync(acc, 0, sizeof(double) * 10 * nc, s));
    Coords xp{a.xp, a.total_np, a.soa}, vp{a.vp, a.total_np, a.soa};
    const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(na, BLK), (int64_t)kNumSMs * 16);
    fof_com_kernel<<<grid, BLK, 0, s>>>(xp, vp, a.mp, st.pos, st.pcand, st.cand_anchor, na,
                                        a.L_Box, 0.5 * a.L_Box, acc);
    PYFOF_CHECK_LAUNCH();
    fof_angmom_kernel<<<grid, BLK, 0, s>>>(xp, vp, a.mp, st.pos, st.pcand, st.cand_anchor, acc,
                                           na, a.L_Box, 0.5 * a.L_Box, am);
    PYFOF_CHECK_LAUNCH();
    std::vector<double> amc(3 * (size_t)nc);
    std::vector<int32_t> creg(nc, 0);
    PYFOF_CUDA(cudaMemcpyAsync(amc.data(), am, sizeof(double) * 3 * nc, cudaMemcpyDeviceToHost, s));
    if (nreg > 1)
      PYFOF_CUDA(cudaMemcpyAsync(creg.data(), st.cand_region, sizeof(int32_t) * nc, cudaMemcpyDeviceToHost, s));
    PYFOF_CUDA(cudaStreamSynchronize(s));
    for (int64_t c = 0; c < nc; ++c)
      for (int d = 0; d < 3; ++d) am_host[3 * (size_t)creg[c] + d] += amc[3 * c + d];
  }
  memcpy(a.ang_mom, am_host.data(), sizeof(double) * am_host.size());
  return kOk;
}

// Every mass positive and finite (py_fof/__init__.py:259-260); with
// m_div != 1 each checked mass is then converted to code units, mp / m_grid
// (py_fof/__init__.py:318-319), in the same pass.
__global__ void check_mass_kernel(double *__restrict__ mp, int64_t n, int32_t *__restrict__ bad, double m_div) {
  int found = 0;
  const bool conv = m_div != 1.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double m = mp[i];
    found |= !(m > 0.0 && m <= 1.7976931348623157e308);
    if (conv) mp[i] = m / m_div;
  }
  if (__syncthreads_or(found) && threadIdx.x == 0) atomicExch(bad, 1);
}

__global__ void divide_kernel(double *__restrict__ x, int64_t n, double d) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = x[i] / d;
}

__global__ void multiply_kernel(double *__restrict__ x, int64_t n, double f) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = x[i] * f;
}

__global__ void fill_kernel(double *__restrict__ x, int64_t n, double v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = v;
}

// mask[i] = halo_id[i] > 0 as 0/1 bytes, four particles per thread
__global__ void member_mask_kernel(const int32_t *__restrict__ id, int64_t n, uint8_t *__restrict__ mask) {
  const int64_t n4 = n / 4;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
    const int4 v = reinterpret_cast<const int4 *>(id)[i];
    const uint32_t w = (uint32_t)(v.x > 0) | ((uint32_t)(v.y > 0) << 8) | ((uint32_t)(v.z > 0) << 16) |
                       ((uint32_t)(v.w > 0) << 24);
    reinterpret_cast<uint32_t *>(mask)[i] = w;
  }
  if (blockIdx.x == 0 && threadIdx.x < (unsigned)(n - 4 * n4)) {
    const int64_t i = 4 * n4 + threadIdx.x;
    mask[i] = id[i] > 0 ? 1 : 0;
  }
}

static unsigned stream_grid(int64_t n) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, BLK), (int64_t)kNumSMs * 8));
}

int32_t divide_inplace(double *x, int64_t n, double d, cudaStream_t s) {
  if (n <= 0) return kOk;
  divide_kernel<<<stream_grid(n), BLK, 0, s>>>(x, n, d);
  PYFOF_CHECK_LAUNCH();
  return kOk;
}

int32_t multiply_inplace(double *x, int64_t n, double f, cudaStream_t s) {
  if (n <= 0) return kOk;
  multiply_kernel<<<stream_grid(n), BLK, 0, s>>>(x, n, f);
  PYFOF_CHECK_LAUNCH();
  return kOk;
}

int32_t fill_value(double *x, int64_t n, double v, cudaStream_t s) {
  if (n <= 0) return kOk;
  fill_kernel<<<stream_grid(n), BLK, 0, s>>>(x, n, v);
  PYFOF_CHECK_LAUNCH();
  return kOk;
}

int32_t member_mask(const int32_t *halo_id, int64_t n, uint8_t *mask, cudaStream_t s) {
  if (n <= 0) return kOk;
  member_mask_kernel<<<stream_grid(ceil_div(n, 4)), BLK, 0, s>>>(halo_id, n, mask);
  PYFOF_CHECK_LAUNCH();
  return kOk;
}

int32_t check_masses(Context &ctx, const double *mp, int64_t n, double m_div) {
  cudaStream_t s = ctx.stream;
  int32_t *bad = ctx.d_flags + FLAG_COUNT_C;
  PYFOF_CUDA(cudaMemsetAsync(bad, 0, sizeof(int32_t), s));
  // the mass array is only written when m_div != 1, and then it is the
  // library's own copy of the caller's masses
  check_mass_kernel<<<stream_grid(n), BLK, 0, s>>>(const_cast<double *>(mp), n, bad, m_div);
  PYFOF_CHECK_LAUNCH();
  PYFOF_CUDA(cudaMemcpyAsync(ctx.h_flags + FLAG_COUNT_C, bad, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  PYFOF_CUDA(cudaStreamSynchronize(s));
  if (ctx.h_flags[FLAG_COUNT_C]) {
    set_error("all particle masses must be positive and finite");
    return kMass;
  }
  return kOk;
}

int32_t fof_run(Context &ctx, const FofArgs &a) {
  FofState st;
  ctx.stage_reset();
  ctx.conv_timer.reset();
  ctx.gap_timer.reset();
  ctx.last_pm_passes = 0;
  ctx.side_timed = false;
  ctx.last_pm_solves = 0;
  ctx.last_pm_fft_bytes = 0.0;
  if (ctx.timing) cudaEventRecord(ctx.ev[2], ctx.stream);
  PYFOF_TRY(fof_link_stage(ctx, a, st));
  PYFOF_TRY(fof_candidates_stage(ctx, a, st, !a.bound_check));
  if (a.issue_masses) PYFOF_TRY(a.issue_masses());
  if (a.masses_ready) PYFOF_CUDA(cudaStreamWaitEvent(ctx.stream, a.masses_ready, 0));
  if (a.mp) PYFOF_TRY(check_masses(ctx, a.mp, a.total_np, a.m_div));
  if (ctx.timing) cudaEventRecord(ctx.ev[3], ctx.stream);
  if (!a.bound_check) {
    if (a.issue_inputs) PYFOF_TRY(a.issue_inputs());
    if (a.inputs_ready) PYFOF_CUDA(cudaStreamWaitEvent(ctx.stream, a.inputs_ready, 0));
    PYFOF_TRY(fof_plain_angmom(ctx, a, st));
  } else {
    // the velocities may still be copying: unbind_stage orders their use
    PYFOF_TRY(unbind_stage(ctx, a, st));
  }
  if (ctx.timing) cudaEventRecord(ctx.ev[4], ctx.stream);
  return kOk;
}

}  // namespace pyfof
