// Particle-mesh unbinding of candidates with more than 1000 members
// (bound_check_grid for gid >= 1, bound_fortran.f90:2436-2864).
//
// Per halo: TSC weights and self-potential of every member (:2558-2602),
// then up to 20 passes of
//   C1: TSC deposit of the kept members on the zero-padded n^3 grid, FFT,
//       multiplication by the optimal Green's function, inverse FFT, TSC
//       gather, self term and the far-field constant (:2657-2703);
//   C2: short-range residual between the spline-softened kernel and the C1
//       split kernel for pairs closer than 3.5 grid cells (:3403-3552),
//       evaluated over nodes of 3.5-cell neighbour cells: the kept set on the
//       first pass, the members removed since on the later ones;
//   removal: the inner loop of the direct path, with the top-2% selection
//       done by an in-block radix select (only the deleted set matters here).
// Halos are batched: one launch deposits and one gathers all of them, the
// transforms run per grid class and transform length.  R = float is the product path, R = double the plain
// FP64 path.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>

#include "context.cuh"
#include "fft.cuh"
#include "primitives.cuh"
#include "unbind_internal.cuh"

namespace pyfof {

namespace {

constexpr int BLK = 256;
constexpr int IBLK = 1024;  // inner-loop block
constexpr double kPi = 3.141592653589793238462643383279502884197;

// ---------------------------------------------------------------- Green

// bound_fft_wave_number (bound_fortran.f90:3563-3569)
__device__ __forceinline__ double wave_number(int i0, int n) {
  const int mode = ((i0 + n / 2) % n) - n / 2;
  return 2.0 * kPi * (double)mode / (double)n;
}

// bound_assignment_window_sq with assignment order 2 (:3571-3583)
__device__ __forceinline__ double window_sq(double k0, double k1, double k2) {
  double s = 1.0;
  double x = 0.5 * k0;
  if (x != 0.0) s = s * sin(x) / x;
  x = 0.5 * k1;
  if (x != 0.0) s = s * sin(x) / x;
  x = 0.5 * k2;
  if (x != 0.0) s = s * sin(x) / x;
  const double s2 = s * s, s3 = s2 * s;
  return s3 * s3;
}

// Alias-summed optimal Green's function (bound_calc_green_and_self,
// :2300-2371), one thread per half-spectrum point.
template <typename R>
__global__ void green_kernel(R *__restrict__ g, int n, double soft, double range, int truncated,
                             int32_t *flags) {
  const int nh = n / 2 + 1;
  const int64_t total = (int64_t)nh * n * n;
  const double radius = 0.5 * (double)n;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(t % nh);
    const int j = (int)((t / nh) % n);
    const int k = (int)(t / ((int64_t)nh * n));
    const double kv0 = wave_number(i, n), kv1 = wave_number(j, n), kv2 = wave_number(k, n);
    double asum = 0.0, bsum = 0.0;
    for (int ka = -2; ka <= 2; ++ka)
      for (int ja = -2; ja <= 2; ++ja)
        for (int ia = -2; ia <= 2; ++ia) {
          const double k0 = kv0 + 2.0 * kPi * (double)ia;
          const double k1 = kv1 + 2.0 * kPi * (double)ja;
          const double k2 = kv2 + 2.0 * kPi * (double)ka;
          const double kmag = sqrt(k0 * k0 + k1 * k1 + k2 * k2);
          const double uk2 = window_sq(k0, k1, k2);
          asum += uk2;
          double target;
          if (kmag == 0.0) {
            if (range == 0.0) target = -4.0 * kPi * radius * radius / 6.0;
            else if (truncated) target = 0.0;
            else target = -2.0 * kPi * (range * range - soft * soft) / 15.0;
          } else {
            double y = soft * kmag / 2.0;
            double y2 = y * y;
            const double ss = 12.0 * (1.0 / (y2 * y2)) * (2.0 - 2.0 * cos(y) - y * sin(y));
            double sr = 0.0;
            if (range != 0.0) {
              y = range * kmag / 2.0;
              y2 = y * y;
              sr = 12.0 * (1.0 / (y2 * y2)) * (2.0 - 2.0 * cos(y) - y * sin(y));
            }
            double cut = 1.0;
            if (truncated) {
              const double kr = kmag * radius;
              cut = 1.0 - sin(kr) / kr;
            }
            target = -4.0 * kPi * (ss * ss - sr * sr) * cut / (kmag * kmag);
          }
          bsum += uk2 * target;
        }
    if (!(asum > 2.2250738585072014e-308)) {
      atomicCAS(&flags[FLAG_ERR], 0, kInvalid);
      continue;
    }
    const double v = bsum / (asum * asum);
    g[t] = (R)v;  // FP32 path: the reference's complex(4) table
  }
}

template <typename R>
__global__ void self_extract_kernel(const R *__restrict__ grid, int n, R *__restrict__ self) {
  const int t = threadIdx.x;
  if (t >= 125) return;
  const int ox = t % 5 - 2, oy = (t / 5) % 5 - 2, oz = t / 25 - 2;
  const int x = (ox + n) % n, y = (oy + n) % n, z = (oz + n) % n;
  const R n3 = (R)((double)n * n * n);
  self[t] = grid[((int64_t)z * n + y) * n + x] / n3;
}

// The kernel on the m^3 lags of a shorter transform, as a half-spectrum shaped
// table (h[(z m + y)(m/2+1) + x]), from the n^3 grid of c2r_full.  Lag m/2
// stands for both signs and is never met.
__global__ void lag_crop_kernel(const double *__restrict__ grid, int n, double *__restrict__ h, int m) {
  const int mh = m / 2 + 1;
  const int64_t total = (int64_t)mh * m * m;
  const double n3 = (double)n * n * n;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(t % mh), y = (int)((t / mh) % m), z = (int)(t / ((int64_t)mh * m));
    const int ly = y <= m / 2 ? y : n - m + y, lz = z <= m / 2 ? z : n - m + z;
    h[t] = grid[((int64_t)lz * n + ly) * n + x] / n3;
  }
}

// The half of an m^3 grid that a table holds, with the 1/m^3 of a transform
// and its inverse.
__global__ void half_table_kernel(const double *__restrict__ grid, int m, double *__restrict__ g) {
  const int mh = m / 2 + 1;
  const int64_t total = (int64_t)mh * m * m;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x)
    g[t] = grid[(t / mh) * m + t % mh] / ((double)m * m * m);
}

}  // namespace

struct GreenTable {
  int n = 0;             // transform length
  void *g = nullptr;     // half-spectrum table (R)
  void *self = nullptr;  // 125 self-kernel values (R), device
  void *tw = nullptr;    // the transforms' twiddles (complex R), device
  bool fp64 = false, scaled = false;  // scaled: holds the transforms' 1/n^3
  std::vector<std::shared_ptr<GreenTable>> shorter;  // the same kernel at other conv_lengths (no self)
  const GreenTable *at(int m) const {
    for (const auto &t : shorter)
      if (t->n == m) return t.get();
    return this;
  }
  ~GreenTable() {
    if (g) cudaFree(g);
    if (self) cudaFree(self);
    if (tw) cudaFree(tw);
  }
};

namespace {

inline unsigned table_grid(int64_t n) { return (unsigned)std::min<int64_t>(ceil_div(n, 256), 148 * 16); }

// The tables of the n-point kernel (its real-space values in `grid`, n^3) at
// its shorter transform lengths.  The kernel is even along every axis, so its
// forward transform is the inverse one that c2r_full runs.  Once per process
// and grid size: about a millisecond for 256 points, all lengths together.
// Where the device has no room for a table (186 MB for the 256-point kernel,
// 166 MB more while they are made), it and the rest are left out, and their
// halos run at n points.
int32_t shorter_tables(GreenTable &t, const double *grid, double2 *spec, ConvBox *dbox, cudaStream_t s) {
  double *h = nullptr, *out = nullptr;
  int32_t r = kOk;
  auto one = [&](int m) -> int32_t {
    const int64_t cnt = (int64_t)(m / 2 + 1) * m * m;
    auto q = std::make_shared<GreenTable>();
    q->n = m;
    q->fp64 = q->scaled = true;
    if (cudaMalloc(&q->g, sizeof(double) * cnt) != cudaSuccess ||
        cudaMalloc(&q->tw, sizeof(double2) * m) != cudaSuccess) {
      cudaGetLastError();
      return kAlloc;
    }
    PYFOF_TRY(fill_twiddles<double>((double2 *)q->tw, m, s));
    ConvBox box{};
    for (int d = 0; d < 3; ++d) box.in[d] = box.out[d] = m;
    PYFOF_CUDA(cudaMemcpyAsync(dbox, &box, sizeof(ConvBox), cudaMemcpyHostToDevice, s));
    lag_crop_kernel<<<table_grid(cnt), 256, 0, s>>>(grid, t.n, h, m);
    PYFOF_CHECK_LAUNCH();
    PYFOF_TRY(c2r_full<double>(h, spec, out, (const double2 *)q->tw, dbox, m, s));
    half_table_kernel<<<table_grid(cnt), 256, 0, s>>>(out, m, (double *)q->g);
    PYFOF_CHECK_LAUNCH();
    t.shorter.push_back(std::move(q));
    return kOk;
  };
  const int *l = conv_lengths(t.n, true);
  if (*l == t.n) return kOk;
  int64_t top = 0;  // the longest of them
  for (const int *k = l; *k < t.n; ++k) top = *k;
  if (cudaMallocAsync(&h, sizeof(double) * (top / 2 + 1) * top * top, s) != cudaSuccess ||
      cudaMallocAsync(&out, sizeof(double) * top * top * top, s) != cudaSuccess) {
    cudaGetLastError();
    r = kAlloc;
  }
  for (; r == kOk && *l < t.n; ++l) r = one(*l);
  if (h) cudaFreeAsync(h, s);
  if (out) cudaFreeAsync(out, s);
  return r == kAlloc ? kOk : r;
}

// Green table of grid n for (soft, range, truncated), cached per device.  Its
// kernel has a status word of its own: the call's is being written by other
// streams (direct-summation halos) and may hold an error already.
template <typename R>
int32_t get_green(Context &ctx, int n, double soft, double range, int truncated,
                  std::shared_ptr<GreenTable> *out) {
  const int kind = range == 0.0 ? 0 : (range < 10.0 ? 1 : 2);
  const int64_t key = ((int64_t)n << 8) | (kind << 1) | (sizeof(R) == 8 ? 1 : 0);
  std::lock_guard<std::mutex> lk(ctx.green->mu);
  auto it = ctx.green->tables.find(key);
  if (it != ctx.green->tables.end()) { *out = it->second; return kOk; }
  auto t = std::make_shared<GreenTable>();
  t->n = n;
  t->fp64 = sizeof(R) == 8;
  const int nh = n / 2 + 1;
  const int64_t cnt = (int64_t)nh * n * n;
  cudaStream_t s = ctx.stream;
  PYFOF_CUDA(cudaMalloc(&t->g, sizeof(R) * cnt));
  PYFOF_CUDA(cudaMalloc(&t->self, sizeof(R) * 125));
  PYFOF_CUDA(cudaMalloc(&t->tw, sizeof(cplx_t<R>) * n));
  PYFOF_TRY(fill_twiddles<R>((cplx_t<R> *)t->tw, n, s));
  R *grid = nullptr;
  cplx_t<R> *spec = nullptr;
  ConvBox *dbox = nullptr;
  int32_t *status = nullptr;  // FLAG_ERR of the tables' kernel
  ConvBox box{};
  for (int d = 0; d < 3; ++d) box.in[d] = box.out[d] = n;
  PYFOF_CUDA(cudaMallocAsync(&grid, sizeof(R) * (size_t)n * n * n, s));
  PYFOF_CUDA(cudaMallocAsync(&spec, sizeof(cplx_t<R>) * spec_elems<R>(n, n), s));
  PYFOF_CUDA(cudaMallocAsync(&dbox, sizeof(ConvBox), s));
  PYFOF_CUDA(cudaMallocAsync(&status, sizeof(int32_t), s));
  static_assert(FLAG_ERR == 0, "the status word stands for the flags");
  PYFOF_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), s));
  green_kernel<R><<<(unsigned)std::min<int64_t>(ceil_div(cnt, 128), 148 * 64), 128, 0, s>>>(
      (R *)t->g, n, soft, range, truncated, status);
  PYFOF_CHECK_LAUNCH();
  PYFOF_CUDA(cudaMemcpyAsync(dbox, &box, sizeof(ConvBox), cudaMemcpyHostToDevice, s));
  int32_t r = c2r_full<R>((const R *)t->g, spec, grid, (const cplx_t<R> *)t->tw, dbox, n, s);
  if (r == kOk) {
    self_extract_kernel<R><<<1, 128, 0, s>>>(grid, n, (R *)t->self);
    PYFOF_CHECK_LAUNCH();
    if constexpr (sizeof(R) == 8) r = shorter_tables(*t, grid, spec, dbox, s);
  }
  int32_t bad = 0;
  PYFOF_CUDA(cudaMemcpyAsync(&bad, status, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  cudaFreeAsync(grid, s);
  cudaFreeAsync(spec, s);
  cudaFreeAsync(dbox, s);
  cudaFreeAsync(status, s);
  PYFOF_CUDA(cudaStreamSynchronize(s));
  if (r != kOk) return r;
  if (bad) {
    set_error("Green's function: zero assignment response");
    return kInvalid;
  }
  ctx.green->tables[key] = t;
  *out = t;
  return kOk;
}

// ---------------------------------------------------------------- setup

struct PmHalo {      // device copy of one PM halo's parameters
  int64_t off;       // first member
  int32_t np;
  int32_t n;         // grid size
  int32_t sup[3];    // nodes [0, sup) per axis the members' TSC clouds touch
  float spacing;
  float origin[3];
  int64_t cell_off;  // first C2 cell
  int64_t e0;        // first member in cell order (the halo's members are consecutive)
  int32_t nc[3];     // C2 cells per axis
  double u_min[3];   // C2 cell origin (q/spacing units)
  double mkeep;      // kept mass at the start of the pass (FP64)
  double cw_u;       // short-range cell width (grid units): 3.5, or 3.5/r_max two-level
  int32_t np_bound, status, pending;
  int32_t two_level; // dense regions refined on 128^3 / 216^3 inner grids
  int32_t r_max;     // largest refinement ratio of the halo's members
  int32_t pad;
};

// One refined region of a two-level halo (bound_fortran.f90:614-823)
struct TlRegion {
  int32_t h, b, r, n_in;
  float lo[3], hi[3];  // region bounds (grid units)
  float bo;            // source margin 3.5 + 3/r
  float u0[3];         // inner grid origin
};

// Nearest node f and TSC weights of one coordinate t (grid units): FP32 as in
// the reference (bound_fortran.f90:2562-2576).
__device__ __forceinline__ int tsc_axis(float t, float *w3) {
  const int nearest = (int)lroundf(t);
  const float dl = __fsub_rn(t, (float)nearest);
  const float a = __fsub_rn(0.5f, dl), b = __fadd_rn(0.5f, dl);
  w3[0] = __fmul_rn(0.5f, __fmul_rn(a, a));
  w3[1] = __fsub_rn(0.75f, __fmul_rn(dl, dl));
  w3[2] = __fmul_rn(0.5f, __fmul_rn(b, b));
  return nearest;
}

// The same for a member at q on its halo's grid.  Returns false outside the
// source domain.
__device__ __forceinline__ bool pm_tsc(const PmHalo &p, float4 q, int *f, float *w9) {
  const float x[3] = {q.x, q.y, q.z};
  bool ok = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float t = __fdiv_rn(__fsub_rn(x[d], p.origin[d]), p.spacing);
    if (!(t >= 0.0f) || t >= (float)(p.n / 2 - 1)) ok = false;
    f[d] = tsc_axis(t, w9 + 3 * d);
  }
  return ok;
}

// Self potential of a TSC cloud on a grid (bound_fortran.f90:2577-2602): FP32
// products, FP64 sum over the 27 x 27 pairs of its nodes, offset by offset.  The
// product of a pair is the same both ways round, so the two kernel values of
// an offset and its opposite are added and half the pairs are left.  Bound by
// the conversions of the products (71 % of the conversion units with all of
// them): 20,000 halos 1.14 -> 0.57 ms (refined regions 0.76 -> 0.34 ms), 256^3
// box 277 -> 139 us, FP32 203^3 box 199 -> 88 us.
template <typename R>
__device__ __forceinline__ R tsc_self(const float *w9, const R *__restrict__ sp) {
  float w[27];
#pragma unroll
  for (int j = 0; j < 27; ++j) w[j] = __fmul_rn(__fmul_rn(w9[j % 3], w9[3 + j / 3 % 3]), w9[6 + j / 9]);
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < 27; ++j) acc += (double)__fmul_rn(w[j], w[j]);
  acc *= (double)sp[62];
#pragma unroll
  for (int dz = 0; dz < 3; ++dz)
#pragma unroll
    for (int dy = -2; dy < 3; ++dy)
#pragma unroll
      for (int dx = -2; dx < 3; ++dx) {
        if (dz == 0 && (dy < 0 || (dy == 0 && dx <= 0))) continue;  // the opposite offset
        double t = 0.0;
#pragma unroll
        for (int j = 0; j < 27; ++j) {
          const int x = j % 3 + dx, y = j / 3 % 3 + dy, z = j / 9 + dz;
          if (x >= 0 && x < 3 && y >= 0 && y < 3 && z < 3) t += (double)__fmul_rn(w[j], w[x + 3 * (y + 3 * z)]);
        }
        const int k = ((dz + 2) * 5 + (dy + 2)) * 5 + (dx + 2);
        acc += t * ((double)sp[k] + (double)sp[124 - k]);
      }
  return (R)acc;
}

// Domain check and self potential of every PM member, in cell order.
template <typename R>
__global__ void pm_setup_kernel(const float4 *__restrict__ src4, const uint32_t *__restrict__ cmem, int64_t n,
                                const PmHalo *__restrict__ H, const int32_t *__restrict__ mhalo,
                                const R *const *__restrict__ selfs, R *__restrict__ selfe, int32_t *flags) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int h = mhalo[cmem[e]];
    int f[3];
    float w9[9];
    if (!pm_tsc(H[h], src4[e], f, w9)) {
      atomicCAS(&flags[FLAG_ERR], 0, kInvalid);
      continue;
    }
    selfe[e] = tsc_self<R>(w9, selfs[h]);
  }
}

// u = q/spacing extent of every PM halo (bound_build_cells :3134-3138).
// Division by the positive spacing is monotone and correctly rounded, so
// min_k (q_k / s) = (min_k q_k) / s exactly: the members' FP32 extremes are
// found first (order-free integer atomics on the ordered images of the
// floats, many blocks per halo), then divided once.
__device__ __forceinline__ uint32_t flt_to_ord(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord_to_flt(uint32_t o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

constexpr int64_t kExtentChunk = 16384;  // members per block

// One block per (halo, chunk of kExtentChunk members) of `work`; omin/omax
// (3 nh) start at 0xffffffff / 0
__global__ void __launch_bounds__(BLK) pm_extent_kernel(const Members m, const PmHalo *__restrict__ H,
                                                        const int2 *__restrict__ work,
                                                        uint32_t *__restrict__ omin, uint32_t *__restrict__ omax) {
  const int h = work[blockIdx.x].x;
  const PmHalo &p = H[h];
  const int64_t k0 = (int64_t)work[blockIdx.x].y * kExtentChunk;
  if (k0 >= p.np) return;
  const int64_t k1 = min((int64_t)p.np, k0 + kExtentChunk);
  uint32_t lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
  for (int64_t k = p.off + k0 + threadIdx.x; k < p.off + k1; k += BLK)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const uint32_t o = flt_to_ord(m.q[d][k]);
      lo[d] = min(lo[d], o);
      hi[d] = max(hi[d], o);
    }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = __reduce_min_sync(0xffffffffu, lo[d]);
    hi[d] = __reduce_max_sync(0xffffffffu, hi[d]);
  }
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      atomicMin(&omin[3 * h + d], lo[d]);
      atomicMax(&omax[3 * h + d], hi[d]);
    }
}

__global__ void pm_extent_final_kernel(const PmHalo *__restrict__ H, int nh, const uint32_t *__restrict__ omin,
                                       const uint32_t *__restrict__ omax, double *__restrict__ ext,
                                       int32_t *__restrict__ sup) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * nh) return;
  const int h = i / 3, d = i % 3;
  const PmHalo &p = H[h];
  if (p.np <= 0) {
    ext[6 * h + d] = 1e30;
    ext[6 * h + 3 + d] = -1e30;
    sup[i] = 3;
    return;
  }
  // the highest node of any member's TSC cloud (pm_setup_kernel's rounding
  // is monotone in q; members outside the domain are refused there)
  const float t = __fdiv_rn(__fsub_rn(ord_to_flt(omax[i]), p.origin[d]), p.spacing);
  sup[i] = t >= 0.0f && t < (float)(p.n / 2 - 1) ? max(3, min((int)lroundf(t) + 2, p.n / 2 + 1)) : p.n / 2 + 1;
  const double sp = (double)p.spacing;
  ext[6 * h + d] = (double)ord_to_flt(omin[i]) / sp;
  ext[6 * h + 3 + d] = (double)ord_to_flt(omax[i]) / sp;
}

// C2 cell key of every PM member (bound_build_cells :3166-3172), and a sort
// key that orders the members of a cell along a Morton curve of its
// (2^(sb/3))^3 sub-cells.
__device__ __forceinline__ uint32_t spread3(uint32_t v) {
  uint32_t r = 0;
  for (int b = 0; b < 3; ++b) r |= ((v >> b) & 1u) << (3 * b);
  return r;
}

// C2 cells are numbered brick by brick: a brick is 4^3 cells, its cells in
// Morton order, so the members of a whole brick, and of each aligned 2^3
// block of cells, are consecutive in cell order and can be read as one range
// (sr_gather_kernel picks the node size that fits a target's cutoff).
__device__ __forceinline__ uint32_t sr_cell(const PmHalo &p, int x, int y, int z) {
  const int bx = (p.nc[0] + 3) >> 2, by = (p.nc[1] + 3) >> 2;
  const int64_t brick = (x >> 2) + (int64_t)bx * ((y >> 2) + (int64_t)by * (z >> 2));
  const uint32_t m = spread3(x & 3) | (spread3(y & 3) << 1) | (spread3(z & 3) << 2);
  return (uint32_t)(p.cell_off + 64 * brick) + m;
}

__global__ void pm_cellkey_kernel(const Members m, const PmHalo *__restrict__ H,
                                  const int32_t *__restrict__ mhalo, int64_t M,
                                  uint32_t *__restrict__ key, uint32_t sentinel, int sb,
                                  uint32_t *__restrict__ skey) {
  const int sub = 1 << (sb / 3);
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < M;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int h = mhalo[k];
    if (h < 0) {
      key[k] = sentinel;
      skey[k] = sentinel << sb;
      continue;
    }
    const PmHalo &p = H[h];
    int64_t c[3];
    uint32_t f[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double u = (double)m.q[d][k] / (double)p.spacing;
      const double g = (u - p.u_min[d]) / p.cw_u;
      double v = floor(g) + 1.0;
      if (!(v >= 1.0)) v = 1.0;
      if (v > (double)p.nc[d]) v = (double)p.nc[d];
      c[d] = (int64_t)v - 1;
      double fr = (g - (double)c[d]) * (double)sub;
      fr = fr < 0.0 ? 0.0 : (fr > (double)(sub - 1) ? (double)(sub - 1) : fr);
      f[d] = (uint32_t)fr;
    }
    const uint32_t cell = sr_cell(p, (int)c[0], (int)c[1], (int)c[2]);
    key[k] = cell;
    skey[k] = (cell << sb) | (spread3(f[0]) | (spread3(f[1]) << 1) | (spread3(f[2]) << 2));
  }
}

__global__ void pm_cellcount_kernel(const uint32_t *__restrict__ key, int64_t M,
                                    uint32_t sentinel, uint32_t *__restrict__ cnt) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < M;
       k += (int64_t)gridDim.x * blockDim.x)
    if (key[k] != sentinel) atomicAdd(&cnt[key[k]], 1u);
}

// ---------------------------------------------------------------- passes

// Deterministic deposit.  The TSC contributions (the reference's FP32
// products w*wx*wy*wz, bound_fortran.f90:2657-2672) are added as 64-bit
// fixed-point integers: integer addition is associative, so the deposited
// grid does not depend on the order in which threads add, and every run
// gives the same bits.  The scale 2^(61 - e), e = ilogb(kept mass), keeps
// the sum of a halo's contributions below 2^62 (TSC weights sum to one per
// member); one unit is 2^-61 of the kept mass, far below FP32 rounding.
__device__ __forceinline__ int fx_exp(double mass) {
  return (mass > 0.0 && isfinite(mass)) ? ilogb(mass) : 0;
}

// v 2^k rounded to the nearest integer, 2^k as a product of two floats (a
// product of a float and either is exact, unless it is far below 1).
__device__ __forceinline__ unsigned long long fx_quantum(float v, float2 sc) {
  return __float2ull_rn(__fmul_rn(__fmul_rn(v, sc.x), sc.y));
}
__device__ __forceinline__ float2 fx_scale(int k) {
  return make_float2(__int_as_float((k / 2 + 127) << 23), __int_as_float((k - k / 2 + 127) << 23));
}

// Last entry e0 of the ascending array off[0..n] with off[e0] <= idx.
__device__ __forceinline__ int seg_of(const uint32_t *__restrict__ off, int n, uint32_t idx) {
  int lo = 0, hi = n;  // off[lo] <= idx < off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= idx) lo = mid;
    else hi = mid;
  }
  return lo;
}

// The deposits and gathers run a block per chunk of up to kDepChunk members
// consecutive in cell order, so that a block's members are close together:
// bpre = prefix of the chunk counts of a batch's grids.
constexpr int kDepChunk = BLK;
constexpr int kDepNodes = 4096;

constexpr int kDepWords = 11;  // (odd: members' words fall in different banks)
struct DepositTile {
  union {
    struct {
      unsigned lo[kDepNodes], hi[kDepNodes];
    };
    float member[BLK][kDepWords];  // weights, mass and first node of the block's members
  };
  int box[6];
};

// Adds one member's 27 contributions per thread (act: the thread has one; f,
// w9, wk its node, weights and mass) to the grid g with rows of nx and planes
// of ny rows.  The members of a chunk share most of their nodes, so they
// are summed in shared memory over the box of the chunk's nodes where it has
// at most kDepNodes (two 32-bit words and a carry per node), and each node
// goes out once; a wider box goes to the grid directly.  Neighbour threads
// start at different nodes: in a cusp all of them add to the same 27.
// Bound by instruction issue.  Refined grids of 1 M members 2.16 ms with the
// fixed-point conversion through FP64, divisions in the flush and a node per
// lane and instruction in the direct adds (32 sectors each), 1.57 ms so.
__device__ __forceinline__ void deposit_chunk(bool act, const int (&f)[3], const float (&w9)[9], float wk, float2 sc,
                                              unsigned long long *__restrict__ g, int nx, int ny, DepositTile &S) {
  constexpr unsigned FULL = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < 6) S.box[tid] = tid < 3 ? INT_MAX : INT_MIN;
  __syncthreads();
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int mn = __reduce_min_sync(FULL, act ? f[d] : INT_MAX), mx = __reduce_max_sync(FULL, act ? f[d] : INT_MIN);
    if (lane == 0) {
      atomicMin(&S.box[d], mn);
      atomicMax(&S.box[3 + d], mx);
    }
  }
  __syncthreads();
  if (S.box[0] > S.box[3]) return;  // nothing to add
  const int x0 = S.box[0] - 1, y0 = S.box[1] - 1, z0 = S.box[2] - 1;
  const int bx = S.box[3] - x0 + 2, by = S.box[4] - y0 + 2, bz = S.box[5] - z0 + 2;
  const int64_t vol = (int64_t)bx * by * bz;
  const bool tile = vol <= kDepNodes;
  if (tile) {
    for (int i = tid; i < (int)vol; i += BLK) S.lo[i] = S.hi[i] = 0;
    __syncthreads();
  }
  if (!tile) {
    // member by member, a node per lane: a row's three nodes go to L2 as one
    // request where they fall in one 32-byte sector
    float *mine = S.member[tid];
#pragma unroll
    for (int j = 0; j < 9; ++j) mine[j] = w9[j];
    mine[9] = wk;
    mine[10] = __int_as_float(act ? (f[0] - 1) + nx * ((f[1] - 1) + ny * (f[2] - 1)) : -1);
    __syncwarp();
    const float(*members)[kDepWords] = &S.member[tid - lane];
    const int jz = lane / 9, jy = lane / 3 - 3 * jz, jx = lane - 9 * jz - 3 * jy;
    const int off = jx + nx * (jy + ny * jz);
    if (lane < 27) {
#pragma unroll 4
      for (int i = 0; i < 32; ++i) {
        const float *c = members[i];
        const int at = __float_as_int(c[10]);
        if (at < 0) continue;
        const float v = __fmul_rn(__fmul_rn(__fmul_rn(c[9], c[jx]), c[3 + jy]), c[6 + jz]);
        atomicAdd(&g[at + off], fx_quantum(v, sc));
      }
    }
    return;
  }
  if (act) {
    // this thread's order of the three nodes of each axis
    const int r[3] = {lane % 3, (lane / 3) % 3, (lane / 9) % 3};
    int o[3][3];
    float w[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int k = j + r[d] < 3 ? j + r[d] : j + r[d] - 3;
        o[d][j] = k;
        w[d][j] = k == 0 ? w9[3 * d] : (k == 1 ? w9[3 * d + 1] : w9[3 * d + 2]);
      }
    const int plane = bx * by, at = (f[0] - 1 - x0) + bx * (f[1] - 1 - y0) + plane * (f[2] - 1 - z0);
#pragma unroll
    for (int jz = 0; jz < 3; ++jz)
#pragma unroll
      for (int jy = 0; jy < 3; ++jy)
#pragma unroll
        for (int jx = 0; jx < 3; ++jx) {
          const float v = __fmul_rn(__fmul_rn(__fmul_rn(wk, w[0][jx]), w[1][jy]), w[2][jz]);
          const unsigned long long u = fx_quantum(v, sc);
          const int i = at + o[0][jx] + bx * o[1][jy] + plane * o[2][jz];
          const unsigned l = (unsigned)u, old = atomicAdd(&S.lo[i], l);
          const unsigned hi = (unsigned)(u >> 32) + (old + l < l ? 1u : 0u);
          if (hi) atomicAdd(&S.hi[i], hi);
        }
  }
  __syncthreads();
  // (i / bx and r / by as high products: exact below 2^12)
  const unsigned inv_bx = 0xffffffffu / (unsigned)bx + 1u, inv_by = 0xffffffffu / (unsigned)by + 1u;
  g += x0 + (int64_t)nx * (y0 + (int64_t)ny * z0);
  for (int i = tid; i < (int)vol; i += BLK) {
    const unsigned long long u = ((unsigned long long)S.hi[i] << 32) | S.lo[i];
    if (!u) continue;
    const int r = (int)__umulhi((unsigned)i, inv_bx), z = (int)__umulhi((unsigned)r, inv_by), y = r - z * by;
    atomicAdd(&g[(i - r * bx) + nx * (y + ny * z)], u);
  }
}

// Deposit of the kept members of a batch of halos (batch[j] = halo of
// grid j, boxes[j] its support box).  Block 0 also writes the grids' inverse
// scales inv[j] = 2^(e - 61).
__global__ void __launch_bounds__(BLK) pm_deposit_kernel(const float4 *__restrict__ src4,
                                                         const uint32_t *__restrict__ cmem,
                                                         const PmHalo *__restrict__ H,
                                                         const ConvBox *__restrict__ boxes,
                                                         const int32_t *__restrict__ batch,
                                                         const uint32_t *__restrict__ bpre, int nb,
                                                         const uint8_t *__restrict__ keep,
                                                         unsigned long long *__restrict__ acc,
                                                         double *__restrict__ inv) {
  __shared__ DepositTile S;
  if (blockIdx.x == 0)
    for (int j = threadIdx.x; j < nb; j += blockDim.x) inv[j] = scalbn(1.0, fx_exp(H[batch[j]].mkeep) - 61);
  const int j = seg_of(bpre, nb, blockIdx.x);
  const PmHalo &p = H[batch[j]];
  const int64_t i = (int64_t)(blockIdx.x - bpre[j]) * kDepChunk + threadIdx.x;
  const bool act = i < p.np && keep[cmem[p.e0 + i]];
  int f[3] = {0, 0, 0};
  float w9[9] = {}, wk = 0.f;
  if (act) {
    const float4 q = src4[p.e0 + i];
    pm_tsc(p, q, f, w9);
    wk = q.w;
  }
  deposit_chunk(act, f, w9, wk, fx_scale(61 - fx_exp(p.mkeep)), acc + boxes[j].in_off, boxes[j].in[0],
                boxes[j].in[1], S);
}

// Value of the convolved grid g (rows of nx, planes of ny rows) at a TSC cloud.
template <typename R>
__device__ __forceinline__ R tsc_gather(const R *__restrict__ g, int nx, int ny, const float (&w9)[9]) {
  R raw = 0;
  for (int sz = 0; sz < 3; ++sz)
    for (int sy = 0; sy < 3; ++sy)
      for (int sx = 0; sx < 3; ++sx)
        raw += g[((int64_t)sz * ny + sy) * nx + sx] * (R)w9[sx] * (R)w9[3 + sy] * (R)w9[6 + sz];
  return raw;
}

// TSC gather and the C1 potential (bound_fortran.f90:2681-2703) at the kept
// members of a batch; grid j holds the potential of halo batch[j].
template <typename R>
__global__ void __launch_bounds__(BLK) pm_gather_kernel(
    const float4 *__restrict__ src4, const uint32_t *__restrict__ cmem, const PmHalo *__restrict__ H,
    const ConvBox *__restrict__ boxes, const int32_t *__restrict__ batch, const uint32_t *__restrict__ bpre, int nb,
    const uint8_t *__restrict__ keep, const R *__restrict__ selfe, const R *__restrict__ rho, double a_val,
    R *__restrict__ phi_c1) {
  const int j = seg_of(bpre, nb, blockIdx.x);
  const PmHalo &p = H[batch[j]];
  const int64_t i = (int64_t)(blockIdx.x - bpre[j]) * kDepChunk + threadIdx.x;
  if (i >= p.np) return;
  const int64_t e = p.e0 + i, k = cmem[e];
  if (!keep[k]) return;
  const float4 q = src4[e];
  int f[3];
  float w9[9];
  pm_tsc(p, q, f, w9);
  const int nx = boxes[j].out[0], ny = boxes[j].out[1];  // the window starts at node 0
  const R raw = tsc_gather<R>(rho + boxes[j].out_off + (((int64_t)(f[2] - 1) * ny + (f[1] - 1)) * nx + (f[0] - 1)), nx,
                              ny, w9);
  const R wk = (R)q.w;
  const double rest = p.mkeep - (double)q.w;
  const R radius = (R)p.n / (R)2;
  const R dz0 = (R)(rest > 0.0 ? rest : 0.0) / radius;
  const R pref = (R)(a_val / (6.0 * kPi * (double)p.spacing));
  phi_c1[k] = pref * ((raw - wk * selfe[e]) - dz0);
}

// Short-range residual of every kept member: the spline-softened kernel
// minus the split kernel its potential already contains, over the kept
// members within the member's own cutoff a_i = 3.5 spacing / r_i, where
// r_i = 1 for plain C2 halos (bound_c2_calc_cells, :3403-3483; in grid
// units there) and the region refinement ratio for two-level halos
// (bound_two_level_pp_full, :1088-1343).  Both are
//     phi_i += w_j * -(a/(6 pi)) * (D(d, eps) - D(d, a_i)),  d < a_i.
// After a refresh the members removed since the previous pass take their
// terms back out (bound_c2_update_incremental_cells :3490-3552,
// bound_two_level_pp_update :1345-1498): UPDATE sums over those sources only
// and subtracts.
//
// FP32 product path: the spline-softened 1/r, D(r, h) (bound_depth_continuous,
// :3080-3102), with its divisions replaced by products with per-h reciprocals
// and 1/r from rsqrtf (a few ulps).  FP32 sums are compensated (Kahan); FP64 sums are plain, which
// keeps the dependent chain per pair to one add.
struct DepthConst {
  float h, two_over_h, inv70h, six_h;
};
__device__ __forceinline__ DepthConst depth_const(float h) {
  return DepthConst{h, 2.0f / h, 1.0f / (70.0f * h), 6.0f * h};
}
__device__ __forceinline__ float depth_fast(float r, float rinv, const DepthConst &c) {
  if (r >= c.h) return rinv;
  const float e = r * c.two_over_h;
  if (e <= 1.0f) {
    const float prim = e * e * (112.0f + e * e * (-56.0f + e * (14.0f + e * (8.0f - 3.0f * e))));
    return (208.0f - prim) * c.inv70h;
  }
  // 12/e = 6 h / r
  const float prim = e * e * (448.0f + e * (-280.0f + e * (56.0f + e * (14.0f + e * (-8.0f + e))))) -
                     224.0f * e - c.six_h * rinv;
  return (128.0f - prim) * c.inv70h;
}

// FP64 path: a pair's term D(r, a) - D(r, eps) as one polynomial.  Between the
// break points h/2 and h of the two kernels each is a polynomial in r, or that
// plus a multiple of 1/r (the outer piece's 12/e is 6 h / r), and so
// is their difference: k / r + c0 + c1 u + .. + c7 u^7, u = r - m, with the
// coefficients and the middle m of the zone the pair is in.  Where both are on
// the same piece the 1/r cancels.  A table per halo and refinement ratio
// (SrSpline) holds the four zones; the pieces join smoothly, so the upper half
// of the squared distance is enough to pick one.  About the middle the terms do not cancel:
// the largest error against quadruple precision over d < a, for a = 1.2 to 17
// eps and eps = 0.05, is 1.1e-14 on values up to 56 (splines evaluated in
// e = 2 r / h, as the oracle's formula is written: 1.0e-13).  Two splines per
// pair took 45 FP64 operations, this takes 22.
struct alignas(16) SrSpline {
  double c[4][10];  // per zone: c0..c7, k, m
  int b2[4];        // squared distances at which zones 1, 2, 3 begin (upper halves)
};

// a b + c with a and c as unevaluated sums of two doubles.
struct Two {
  double hi, lo;
};
__device__ __forceinline__ Two two_fma(Two a, double b, Two c) {
  const double p = __dmul_rn(a.hi, b), e = fma(a.hi, b, -p) + a.lo * b;
  const double s = __dadd_rn(p, c.hi), t = __dadd_rn(s, -p);
  const double r = __dadd_rn(__dadd_rn(p, -__dadd_rn(s, -t)), __dadd_rn(c.hi, -t)) + (e + c.lo);
  const double h = __dadd_rn(s, r);
  return Two{h, __dadd_rn(r, -__dadd_rn(h, -s))};
}

// The piece of D(., h) around distance m: Taylor coefficients of its
// polynomial about m, and the factor of 1/r.  At and beyond h (always, for
// h = 0) it is 1/r alone.
__device__ __forceinline__ void spline_piece(double h, double m, double *c) {
  if (m >= h) {
#pragma unroll
    for (int j = 0; j < 8; ++j) c[j] = 0.0;
    c[8] = 1.0;
    return;
  }
  const double s = 2.0 / h, u = 1.0 / (70.0 * h), e0 = s * m;
  const double inner[8] = {208.0, 0.0, -112.0, 0.0, 56.0, -14.0, -8.0, 3.0};
  const double outer[8] = {128.0, 224.0, -448.0, 280.0, -56.0, -14.0, 8.0, -1.0};
  Two d[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) d[j] = Two{m < 0.5 * h ? inner[j] : outer[j], 0.0};
#pragma unroll
  for (int i = 0; i < 7; ++i)
#pragma unroll
    for (int j = 6; j >= i; --j) d[j] = two_fma(d[j + 1], e0, d[j]);
  double p = u;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    c[j] = d[j].hi * p;
    p *= s;
  }
  c[8] = m < 0.5 * h ? 0.0 : 6.0 / 70.0;
}

// A thread per (halo, ratio 1, 2, 4).  A softening of 0 has no zones of its
// own: the first one then holds distance 0 only, where D(0, h) = 208 / (70 h)
// is infinite.
__global__ void sr_spline_kernel(const PmHalo *__restrict__ H, int nh, double app, SrSpline *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * nh) return;
  const double eps = (double)(float)app, a = 3.5 * (double)H[i / 3].spacing / (double)(1 << (i % 3));
  const double soft = eps > 0.0 ? eps : 0.0;
  double b[4] = {0.5 * soft, 0.5 * a, soft, a};  // ascending below
  for (int j = 0; j < 3; ++j)
    for (int k = j + 1; k < 4; ++k)
      if (b[k] < b[j]) {
        const double t = b[j];
        b[j] = b[k];
        b[k] = t;
      }
  SrSpline &S = out[i];
  for (int z = 0; z < 4; ++z) {
    const double mid = 0.5 * ((z ? b[z - 1] : 0.0) + b[z]);
    double ca[9], ce[9];
    spline_piece(a, mid, ca);
    spline_piece(eps, mid, ce);
    for (int j = 0; j < 9; ++j) S.c[z][j] = ca[j] - ce[j];
    if (b[z] == 0.0) {  // distance 0
      S.c[z][0] = 208.0 / (70.0 * a) - 208.0 / (70.0 * eps);
      S.c[z][8] = 0.0;
    }
    S.c[z][9] = mid;
    S.b2[z] = z < 3 ? max(__double2hiint(b[z] * b[z]), 1) : 0;
  }
}

// 1/r: the hardware's reciprocal square root of a double's upper half as the
// seed y and one step of the binomial series 1/sqrt(r2) = y (1 - g)^(-1/2) =
// y (1 + g/2 + 3 g^2/8 + ..), g = 1 - r2 y^2.  The argument is kept above
// 2^-300, for a finite 1/r of coincident members; distinct FP32 coordinates
// are at least 2^-149 apart.
__device__ __forceinline__ double rsqrt_series64(double r2) {
  const double a = __hiloint2double(max(__double2hiint(r2), 0x2d300000), __double2loint(r2));
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double g = fma(-(r2 * y), y, 1.0);
  return fma(y * g, fma(0.375, g, 0.5), y);
}

// A target chunk: up to 32 members of one brick, consecutive in cell order
// (along the brick's Morton curve, so they are spatially compact), with the
// range of source nodes its widened bounding box touches.  A node is an
// aligned block of 2^level cells per axis.
struct SrChunk {
  uint32_t e0;       // first member (position in cell order)
  int32_t h;         // halo
  float lo[3], hi[3];  // bounding box of the targets
  float amax;        // largest cutoff of the targets, a little widened
  uint32_t nsrc;     // members of all its nodes
  int16_t x0[3];     // first node per axis
  uint16_t nx[3];    // nodes per axis
  uint8_t cnt, level;
};

// Chunks whose nodes hold this many members or more are summed by the eight
// warps of a block together.  The rule looks at the chunk alone, so the order
// of its sum does not depend on what else is in the call.  Where the line
// lies: a full chip likes it higher (20,000 halos: 21.2 ms at 512, 20.6 at
// 1024, 19.9 at 2048), a call of middle-sized halos lower, since its last
// chunks run alone (1000 halos: 0.67, 0.79, 0.92 ms).
// Update passes sum over the removed members only, a few per cent of them.
constexpr uint32_t kSrHeavy = 1024, kSrHeavyUpdate = 16384;
constexpr int kSrWarps = 8;

__global__ void sr_chunk_count_kernel(const uint32_t *__restrict__ cstart, int64_t nbrick,
                                      uint32_t *__restrict__ cnt) {
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nbrick;
       b += (int64_t)gridDim.x * blockDim.x)
    cnt[b] = (cstart[64 * (b + 1)] - cstart[64 * b] + 31u) / 32u;
}

__global__ void sr_chunk_fill_kernel(const uint32_t *__restrict__ cstart, const uint32_t *__restrict__ coff,
                                     int64_t nbrick, uint2 *__restrict__ span) {
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nbrick;
       b += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t e0 = cstart[64 * b], e1 = cstart[64 * (b + 1)];
    const uint32_t n = (e1 - e0 + 31u) / 32u;
    for (uint32_t i = 0; i < n; ++i) span[coff[b] + i] = make_uint2(e0 + 32u * i, min(32u, e1 - e0 - 32u * i));
  }
}

// First member of node (x, y, z) of `level` and the one after its last.
__device__ __forceinline__ uint2 sr_node_range(const PmHalo &p, const uint32_t *__restrict__ cstart, int x, int y,
                                               int z, int level) {
  const uint32_t c = sr_cell(p, x << level, y << level, z << level);
  return make_uint2(cstart[c], cstart[c + (1u << (3 * level))]);
}

// Chunk records, a warp per chunk, and their sort keys: most sources first,
// so that the dynamically fetched chunks end together.
__global__ void __launch_bounds__(BLK) sr_chunk_setup_kernel(
    const uint2 *__restrict__ span, int64_t nchunk, const PmHalo *__restrict__ H,
    const int32_t *__restrict__ mhalo, const uint32_t *__restrict__ cmem, const float4 *__restrict__ src4,
    const uint8_t *__restrict__ pr, const uint32_t *__restrict__ cstart, SrChunk *__restrict__ out,
    uint32_t *__restrict__ key, uint32_t *__restrict__ nheavy) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  for (int64_t ch = ((int64_t)blockIdx.x * BLK + threadIdx.x) >> 5; ch < nchunk;
       ch += ((int64_t)gridDim.x * BLK) >> 5) {
    const uint2 sp = span[ch];
    const bool valid = lane < (int)sp.y;
    float4 me = make_float4(0.f, 0.f, 0.f, 0.f);
    int ri = 64;
    if (valid) {
      me = src4[sp.x + lane];
      ri = pr[cmem[sp.x + lane]];
    }
    const int h = mhalo[cmem[sp.x]];
    const PmHalo &p = H[h];
    SrChunk C;
    C.e0 = sp.x;
    C.h = h;
    C.cnt = (uint8_t)sp.y;
    const float m3[3] = {me.x, me.y, me.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      C.lo[d] = ord_to_flt(__reduce_min_sync(FULL, valid ? flt_to_ord(m3[d]) : 0xffffffffu));
      C.hi[d] = ord_to_flt(__reduce_max_sync(FULL, valid ? flt_to_ord(m3[d]) : 0u));
    }
    const int rmin = __reduce_min_sync(FULL, ri);
    const double spc = (double)p.spacing;
    // conservative filter radius (a little above every target's cutoff)
    C.amax = (float)(3.5 * spc / (double)rmin) * 1.0001f + 1e-30f;
    // nodes about as wide as the cutoff; wider ones for a chunk that a
    // sparse brick spreads over many
    int level = p.two_level ? (p.r_max >= 4 * rmin ? 2 : (p.r_max >= 2 * rmin ? 1 : 0)) : 0;
    int nodes;
    for (;; ++level) {
      nodes = 1;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double gl = (((double)C.lo[d] - (double)C.amax) / spc - p.u_min[d]) / p.cw_u - 1e-4;
        const double gh = (((double)C.hi[d] + (double)C.amax) / spc - p.u_min[d]) / p.cw_u + 1e-4;
        const int top = p.nc[d] - 1;
        const int a = gl <= 0.0 ? 0 : (gl >= (double)top ? top : (int)gl);
        const int b = gh <= 0.0 ? 0 : (gh >= (double)top ? top : (int)gh);
        C.x0[d] = (int16_t)(a >> level);
        C.nx[d] = (uint16_t)((b >> level) - (a >> level) + 1);
        nodes *= C.nx[d];
      }
      if (level == 2 || nodes <= 128) break;
    }
    C.level = (uint8_t)level;
    uint32_t t = 0;
    for (int j = lane; j < nodes; j += 32) {
      const int w0 = C.nx[0], w1 = C.nx[1];
      const uint2 r = sr_node_range(p, cstart, C.x0[0] + j % w0, C.x0[1] + (j / w0) % w1,
                                    C.x0[2] + j / (w0 * w1), level);
      t += r.y - r.x;
    }
    C.nsrc = __reduce_add_sync(FULL, t);
    if (lane == 0) {
      out[ch] = C;
      key[ch] = 65535u - min(C.nsrc >> 2, 65535u);
      if (C.nsrc >= kSrHeavy) atomicAdd(&nheavy[0], 1u);
      if (C.nsrc >= kSrHeavyUpdate) atomicAdd(&nheavy[1], 1u);
    }
  }
}

__global__ void sr_chunk_order_kernel(const SrChunk *__restrict__ chunks, const uint32_t *__restrict__ idx,
                                      int64_t n, SrChunk *__restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = chunks[idx[i]];
}

// What a warp needs of its targets to test and add pairs.
template <typename R>
struct SrTarget {
  float4 me;
  uint32_t e0;    // the chunk's first target (position in cell order)
  float a2f;      // FP32 bound of the pair test, a little above a2; < 0: no target
  R a2;
  bool tl;
  DepthConst eps, ai;      // FP32 path
  const SrSpline *spline;  // FP64 path: the halo's table of this target's ratio
  R acc, comp;
};

// A warp's 32 sources: FP32 coordinates by axis for the marks, and (FP64 path)
// all of them in FP64, converted once for all its targets.
template <typename R>
struct SrStage {
  alignas(16) float x[32], y[32], z[32];
};
template <>
struct SrStage<double> {
  alignas(16) float x[32], y[32], z[32];
  double2 xy[32], zw[32];
};

// The sources within FP32 distance^2 a2f of `me`, two per instruction: a third
// of the kernel's instructions were the marks, one
// source at a time; 20,000 halos 18.9 -> 17.8 ms, one halo of 30,000 222 -> 200 us.
template <typename R>
__device__ __forceinline__ unsigned sr_mark(const SrStage<R> &S, float4 me, float a2f) {
  auto both = [](float v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
  };
  const unsigned long long mx = both(-me.x), my = both(-me.y), mz = both(-me.z);
  unsigned mask = 0;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    const ulonglong2 X = reinterpret_cast<const ulonglong2 *>(S.x)[g];
    const ulonglong2 Y = reinterpret_cast<const ulonglong2 *>(S.y)[g];
    const ulonglong2 Z = reinterpret_cast<const ulonglong2 *>(S.z)[g];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      unsigned long long dx, dy, dz, q;
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(dx) : "l"(h ? X.y : X.x), "l"(mx));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(dy) : "l"(h ? Y.y : Y.x), "l"(my));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(dz) : "l"(h ? Z.y : Z.x), "l"(mz));
      asm("mul.rn.f32x2 %0, %1, %1;" : "=l"(q) : "l"(dx));
      asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(q) : "l"(dy), "l"(q));
      asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(q) : "l"(dz), "l"(q));
      float lo, hi;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(q));
      if (lo <= a2f) mask |= 1u << (4 * g + 2 * h);
      if (hi <= a2f) mask |= 2u << (4 * g + 2 * h);
    }
  }
  return mask;
}

// The terms of a target's marked sources.  The conversion units were the
// busiest part of a pair (59 %: three coordinates, the weight and both ways
// around the seed of 1/r): with sources converted once per warp and a seed from
// the FP64 word they do one operation per pair of a two-level halo
// (DIFF64: differences in FP64) and four where the differences are FP32's.
template <bool DIFF64>
__device__ __forceinline__ void sr_marked64(const float4 *__restrict__ buf, const SrStage<double> &wide, unsigned mask,
                                            SrTarget<double> &t) {
  const SrSpline &S = *t.spline;
  const double mx = (double)t.me.x, my = (double)t.me.y, mz = (double)t.me.z;
  const int none = __ffs(mask) - 1;  // a mark to stand in for a missing second one
  while (mask) {
    // two pairs at a time, for their dependent chains to overlap
    int j[2];
    j[0] = __ffs(mask) - 1;
    mask &= mask - 1;
    const bool two = mask != 0;
    j[1] = two ? __ffs(mask) - 1 : none;
    mask &= mask - 1;
    double v[2], w[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      double dx, dy, dz;
      if (DIFF64) {
        const double2 xy = wide.xy[j[e]], zw = wide.zw[j[e]];
        dx = xy.x - mx; dy = xy.y - my; dz = zw.x - mz;
        w[e] = zw.y;
      } else {
        const float4 s = buf[j[e]];
        dx = (double)(s.x - t.me.x); dy = (double)(s.y - t.me.y); dz = (double)(s.z - t.me.z);
        w[e] = wide.zw[j[e]].y;
      }
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (!(r2 < t.a2 && (e == 0 || two))) w[e] = 0.0;
      const int r2h = __double2hiint(r2);
      const int z = (r2h >= S.b2[0]) + (r2h >= S.b2[1]) + (r2h >= S.b2[2]);
      const double2 *c = reinterpret_cast<const double2 *>(S.c[z]);
      // (coincident members: a finite 1/r with coefficient 0, u = -m)
      const double rinv = rsqrt_series64(r2);
      const double2 km = c[4], c67 = c[3], c45 = c[2], c23 = c[1], c01 = c[0];
      const double u = fma(r2, rinv, -km.y);
      double f = fma(c67.y, u, c67.x);
      f = fma(f, u, c45.y);
      f = fma(f, u, c45.x);
      f = fma(f, u, c23.y);
      f = fma(f, u, c23.x);
      f = fma(f, u, c01.y);
      f = fma(f, u, c01.x);
      v[e] = fma(km.x, rinv, f);
    }
    t.acc = fma(w[0], v[0], t.acc);
    t.acc = fma(w[1], v[1], t.acc);
  }
}

// Up to 32 staged sources against the warp's 32 targets.  Every lane first
// marks the sources inside its own cutoff with an FP32 test (the box filter
// in front of it keeps a chunk's union, of which a target needs a third or
// less), then walks its own marks, so the long pair arithmetic runs on
// interacting pairs only, in ascending source order per target.
template <typename R, bool UPDATE>
__device__ __forceinline__ void sr_pairs(const float4 *__restrict__ buf, const uint32_t *__restrict__ idx, int cnt,
                                         SrStage<R> *stage, SrTarget<R> &t) {
  const int lane = threadIdx.x & 31;
  const float4 mine = buf[lane];
  // (a place without a source is out of every reach)
  stage->x[lane] = lane < cnt ? mine.x : 3e38f;
  stage->y[lane] = mine.y;
  stage->z[lane] = mine.z;
  if constexpr (sizeof(R) == 8) {
    stage->xy[lane] = make_double2((double)mine.x, (double)mine.y);
    stage->zw[lane] = make_double2((double)mine.z, (double)mine.w);
  }
  __syncwarp();
  unsigned mask = sr_mark(*stage, t.me, t.a2f);
  if constexpr (!UPDATE) {  // a target is not its own source
    const uint32_t own = lane < cnt ? idx[lane] - t.e0 : 32u;
    unsigned self = __ballot_sync(0xffffffffu, own < 32u);
    while (self) {
      const int j = __ffs(self) - 1;
      self &= self - 1;
      if (__shfl_sync(0xffffffffu, own, j) == (uint32_t)lane) mask &= ~(1u << j);
    }
  }
  if constexpr (sizeof(R) == 8) {
    if (t.tl) sr_marked64<true>(buf, *stage, mask, t);
    else sr_marked64<false>(buf, *stage, mask, t);
  } else {
    const int none = __ffs(mask) - 1;  // a mark to stand in for a missing second one
    while (mask) {
      // two pairs at a time, for their dependent chains to overlap
      int j[2];
      j[0] = __ffs(mask) - 1;
      mask &= mask - 1;
      const bool two = mask != 0;
      j[1] = two ? __ffs(mask) - 1 : none;
      mask &= mask - 1;
      R v[2], w[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float4 s = buf[j[e]];
        const R dx = s.x - t.me.x, dy = s.y - t.me.y, dz = s.z - t.me.z;
        const R r2 = dx * dx + dy * dy + dz * dz;
        w[e] = r2 < t.a2 && (e == 0 || two) ? s.w : (R)0;
        // (coincident members: 1/r is infinite, and not needed within a softening)
        const float rinv = rsqrtf(r2), d = r2 > 0.0f ? r2 * rinv : 0.0f;
        v[e] = depth_fast(d, rinv, t.eps) - depth_fast(d, rinv, t.ai);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {  // compensated sum of the negated terms
        if (w[e] == 0.0f) continue;
        const float y = -(w[e] * v[e]) - t.comp;
        const float sum = t.acc + y;
        t.comp = (sum - t.acc) - y;
        t.acc = sum;
      }
    }
  }
}

// The sum of one chunk by a warp.  Nodes are taken 32 at a time: a lane loads
// one node's member range, the ranges are concatenated by a warp prefix sum and read in batches of 32 (a lane finds
// its source's node by a binary search over the prefix); sources within the
// largest cutoff of the targets' bounding box are staged, and every 32
// staged sources go to sr_pairs.
template <typename R, bool UPDATE>
__device__ __forceinline__ void sr_chunk_sum(const SrChunk &C, const PmHalo &p, const uint32_t *__restrict__ cstart,
                                             const float4 *__restrict__ src4, const uint32_t *__restrict__ rpos,
                                             const uint32_t *__restrict__ rsrc, float4 *buf, uint32_t *idx,
                                             SrStage<R> *stage, SrTarget<R> &t) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  const float amax2 = C.amax * C.amax;
  const int w0 = C.nx[0], w1 = C.nx[1], nodes = w0 * w1 * C.nx[2];
  int fill = 0, n0 = -32;
  uint32_t T = 0, g0 = 0, incl = 0, first = 0;  // the 32 nodes in hand
  for (;;) {
    bool more = true;
    while (fill < 32) {
      if (g0 >= T) {
        n0 += 32;
        more = n0 < nodes;
        if (!more) break;
        const int j = n0 + lane;
        uint32_t s0 = 0, cnt = 0;
        if (j < nodes) {
          uint2 r = sr_node_range(p, cstart, C.x0[0] + j % w0, C.x0[1] + (j / w0) % w1, C.x0[2] + j / (w0 * w1),
                                  C.level);
          if (UPDATE && r.y > r.x) r = make_uint2(rpos[r.x], rpos[r.y]);
          s0 = r.x;
          cnt = r.y - r.x;
        }
        incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(FULL, incl, o);
          if (lane >= o) incl += v;
        }
        first = s0 - (incl - cnt);  // source of batch index g: first + g
        T = __shfl_sync(FULL, incl, 31);
        g0 = 0;
        continue;
      }
      const uint32_t g = g0 + (uint32_t)lane;
      g0 += 32;
      int owner = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const uint32_t v = __shfl_sync(FULL, incl, owner + step - 1);
        if (v <= g) owner += step;
      }
      owner &= 31;
      const uint32_t of = __shfl_sync(FULL, first, owner);
      uint32_t se = 0;
      float4 sv = make_float4(0.f, 0.f, 0.f, 0.f);
      bool cand = false;
      if (g < T) {
        se = UPDATE ? rsrc[of + g] : of + g;
        sv = src4[se];
        const float bx = fmaxf(fmaxf(C.lo[0] - sv.x, sv.x - C.hi[0]), 0.f);
        const float by = fmaxf(fmaxf(C.lo[1] - sv.y, sv.y - C.hi[1]), 0.f);
        const float bz = fmaxf(fmaxf(C.lo[2] - sv.z, sv.z - C.hi[2]), 0.f);
        cand = bx * bx + by * by + bz * bz <= amax2;
      }
      const unsigned m = __ballot_sync(FULL, cand);
      if (cand) {
        const int q = fill + __popc(m & lt);
        buf[q] = sv;
        idx[q] = se;
      }
      fill += __popc(m);
      __syncwarp();
    }
    if (fill) sr_pairs<R, UPDATE>(buf, idx, min(fill, 32), stage, t);
    __syncwarp();
    if (!more) break;
    fill -= 32;
    if (lane < fill) {
      buf[lane] = buf[32 + lane];
      idx[lane] = idx[32 + lane];
    }
    __syncwarp();
  }
}

// The sum of a heavy chunk by a block: the ranges of 256 nodes at a time are
// loaded and concatenated by all threads, and every warp takes the source
// batches of 32 in turn.
struct SrNodes {
  uint32_t incl[32 * kSrWarps], first[32 * kSrWarps], total[kSrWarps];
};

template <typename R, bool UPDATE>
__device__ __forceinline__ void sr_block_sum(const SrChunk &C, const PmHalo &p, const uint32_t *__restrict__ cstart,
                                             const float4 *__restrict__ src4, const uint32_t *__restrict__ rpos,
                                             const uint32_t *__restrict__ rsrc, SrNodes &N, float4 *buf,
                                             uint32_t *idx, SrStage<R> *stage, SrTarget<R> &t) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int NT = 32 * kSrWarps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float amax2 = C.amax * C.amax;
  const int w0 = C.nx[0], w1 = C.nx[1], nodes = w0 * w1 * C.nx[2];
  int fill = 0;
  for (int n0 = 0; n0 < nodes; n0 += NT) {
    const int j = n0 + (int)threadIdx.x;
    uint32_t s0 = 0, cnt = 0;
    if (j < nodes) {
      uint2 r = sr_node_range(p, cstart, C.x0[0] + j % w0, C.x0[1] + (j / w0) % w1, C.x0[2] + j / (w0 * w1), C.level);
      if (UPDATE && r.y > r.x) r = make_uint2(rpos[r.x], rpos[r.y]);
      s0 = r.x;
      cnt = r.y - r.x;
    }
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) N.total[warp] = incl;
    __syncthreads();
    uint32_t T = 0;
#pragma unroll
    for (int w = 0; w < kSrWarps; ++w) {
      if (w == warp) incl += T;
      T += N.total[w];
    }
    N.incl[threadIdx.x] = incl;
    N.first[threadIdx.x] = s0 - (incl - cnt);  // source of batch index g: first + g
    __syncthreads();
    for (uint32_t g0 = 32 * (uint32_t)warp; g0 < T; g0 += NT) {
      const uint32_t g = g0 + (uint32_t)lane;
      int owner = 0;  // nodes that end at or before g
#pragma unroll
      for (int step = NT / 2; step > 0; step >>= 1)
        if (N.incl[owner + step - 1] <= g) owner += step;
      uint32_t se = 0;
      float4 sv = make_float4(0.f, 0.f, 0.f, 0.f);
      bool cand = false;
      if (g < T) {
        const uint32_t e = N.first[owner] + g;
        se = UPDATE ? rsrc[e] : e;
        sv = src4[se];
        const float bx = fmaxf(fmaxf(C.lo[0] - sv.x, sv.x - C.hi[0]), 0.f);
        const float by = fmaxf(fmaxf(C.lo[1] - sv.y, sv.y - C.hi[1]), 0.f);
        const float bz = fmaxf(fmaxf(C.lo[2] - sv.z, sv.z - C.hi[2]), 0.f);
        cand = bx * bx + by * by + bz * bz <= amax2;
      }
      const unsigned m = __ballot_sync(FULL, cand);
      if (cand) {
        const int q = fill + __popc(m & lanemask_lt());
        buf[q] = sv;
        idx[q] = se;
      }
      fill += __popc(m);
      __syncwarp();
      if (fill < 32) continue;
      sr_pairs<R, UPDATE>(buf, idx, 32, stage, t);
      __syncwarp();
      fill -= 32;
      if (lane < fill) {
        buf[lane] = buf[32 + lane];
        idx[lane] = idx[32 + lane];
      }
      __syncwarp();
    }
    __syncthreads();
  }
  if (fill) sr_pairs<R, UPDATE>(buf, idx, fill, stage, t);
  __syncwarp();
}

// Bound by instruction issue per interacting pair (FP64 and conversions) once
// enough warps have work.  Persistent blocks: first the heavy chunks, a
// block each (the node ranges are found once for its eight warps, which take
// the source batches in turn; their sums are added in warp order, the FP32
// ones compensated like the sums themselves), then the others, a warp each;
// both most sources first, fetched from a counter.  Two pairs in flight per
// lane and the shared node ranges: 1 M zoom region 3.72 ->
// 3.37 ms, 20,000 halos 22.6 -> 20.6 ms.
template <typename R, bool UPDATE>
__global__ void __launch_bounds__(32 * kSrWarps, sizeof(R) == 4 ? 4 : 3) sr_gather_kernel(
    const PmHalo *__restrict__ H, const uint8_t *__restrict__ keep, const uint8_t *__restrict__ pr,
    const SrChunk *__restrict__ chunks, uint32_t nchunks, const uint32_t *__restrict__ nheavy_p,
    const uint32_t *__restrict__ cstart, const uint32_t *__restrict__ cmem, const float4 *__restrict__ src4,
    const uint32_t *__restrict__ rpos, const uint32_t *__restrict__ rsrc, const SrSpline *__restrict__ splines,
    double a_val, double app, R *__restrict__ phi_sr, unsigned *__restrict__ next) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ float4 buf[kSrWarps][64];
  __shared__ uint32_t idx[kSrWarps][64];
  __shared__ R part[kSrWarps][32], pcomp[sizeof(R) == 4 ? kSrWarps : 1][32];
  __shared__ SrNodes nodes;
  __shared__ unsigned s_ch;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the spline tables of the halo in hand (FP64), one copy per warp
  __shared__ SrSpline tables[sizeof(R) == 8 ? kSrWarps : 1][3];
  __shared__ SrStage<R> stages[kSrWarps];
  int table_h = -1;
  const uint32_t nheavy = nheavy_p[UPDATE ? 1 : 0];
  const R fac = (R)(a_val / (6.0 * kPi));
  SrTarget<R> t;
  t.eps = depth_const((float)(double)(float)app);
  // the chunk's targets; false when it has nothing to do
  auto begin = [&](const SrChunk &C, const PmHalo &p, int64_t &k) -> bool {
    if (!p.pending) return false;
    const bool valid = lane < (int)C.cnt;
    t.e0 = C.e0;
    k = valid ? (int64_t)cmem[C.e0 + lane] : -1;
    const bool active = valid && (!UPDATE || keep[k] != 0);
    if (!__any_sync(FULL, active)) return false;
    t.me = valid ? src4[C.e0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int ri = active ? (int)pr[k] : 1;
    const R ai = (R)(3.5 * (double)p.spacing / (double)ri);
    t.a2 = ai * ai;
    // the FP32 distance of a pair is within 1e-6 of the exact one
    t.a2f = active ? (float)t.a2 * 1.00001f + 1e-37f : -1.0f;
    t.ai = depth_const((float)ai);
    if constexpr (sizeof(R) == 8) {
      if (C.h != table_h) {
        __syncwarp();
        const uint4 *from = reinterpret_cast<const uint4 *>(splines + 3 * (int64_t)C.h);
        uint4 *to = reinterpret_cast<uint4 *>(tables[warp]);
        for (int i = lane; i < (int)(3 * sizeof(SrSpline) / 16); i += 32) to[i] = from[i];
        __syncwarp();
        table_h = C.h;
      }
      t.spline = &tables[warp][ri == 4 ? 2 : ri - 1];
    }
    t.tl = p.two_level != 0;
    t.acc = t.comp = (R)0;
    if (!active) k = -1;
    return true;
  };
  bool heavy = true;  // the same for every warp of the block at its barriers
  for (;;) {
    unsigned ch = 0;
    if (heavy) {
      if (threadIdx.x == 0) s_ch = atomicAdd(&next[0], 1u);
      __syncthreads();
      ch = s_ch;
      if (ch >= nheavy) {
        heavy = false;
        continue;
      }
    } else {
      if (lane == 0) ch = nheavy + atomicAdd(&next[1], 1u);
      ch = __shfl_sync(FULL, ch, 0);
      if (ch >= nchunks) break;
    }
    const SrChunk &C = chunks[ch];  // read where needed (L1), not held in registers
    const PmHalo &p = H[C.h];
    int64_t k;
    const bool some = begin(C, p, k);
    if (!heavy) {
      if (some) sr_chunk_sum<R, UPDATE>(C, p, cstart, src4, rpos, rsrc, buf[warp], idx[warp], &stages[warp], t);
    } else {
      if (some) {  // the same for every warp
        sr_block_sum<R, UPDATE>(C, p, cstart, src4, rpos, rsrc, nodes, buf[warp], idx[warp], &stages[warp], t);
        part[warp][lane] = t.acc;
        if (sizeof(R) == 4) pcomp[warp][lane] = t.comp;
      }
      __syncthreads();
      if (warp != 0 || !some) continue;
      if constexpr (sizeof(R) == 8) {
#pragma unroll
        for (int w = 1; w < kSrWarps; ++w) t.acc += part[w][lane];
      } else {
        // the warps' sums with what they left out (comp: the excess of a sum)
        // and what each addition here leaves out
        R low = -t.comp;
#pragma unroll
        for (int w = 1; w < kSrWarps; ++w) {
          const R x = part[w][lane], sum = __fadd_rn(t.acc, x), bb = __fsub_rn(sum, t.acc);
          low += __fadd_rn(__fsub_rn(t.acc, __fsub_rn(sum, bb)), __fsub_rn(x, bb)) - pcomp[w][lane];
          t.acc = sum;
        }
        t.acc += low;
      }
    }
    if (some && k >= 0) {
      const R v = fac * t.acc;
      if (UPDATE) phi_sr[k] -= v;
      else phi_sr[k] = v;
    }
  }
}

// Cell-ordered copy of the members' positions and weights, and every
// member's position in cell order.
__global__ void sr_pack_kernel(const Members m, const uint32_t *__restrict__ cmem, int64_t n,
                               float4 *__restrict__ src4, uint32_t *__restrict__ epos) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t k = cmem[e];
    src4[e] = make_float4(m.q[0][k], m.q[1][k], m.q[2][k], m.w[k]);
    epos[k] = (uint32_t)e;
  }
}

// The members removed since the previous pass (flagged per cell-ordered
// position by the removal kernels), compacted in cell order; clears the flags.
__global__ void sr_removed_fill_kernel(uint32_t *__restrict__ flag, const uint32_t *__restrict__ rpos,
                                       int64_t n, uint32_t *__restrict__ rsrc) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    if (flag[e]) {
      rsrc[rpos[e]] = (uint32_t)e;
      flag[e] = 0;
    }
}

// ---------------------------------------------------------------- two-level

// One refined region: halo h, region b (8x8x8 regions of 16 grid cells),
// ratio r, inner grid n_in (bound_two_level_build_halo, :614-823).
__device__ __forceinline__ void tl_t(const PmHalo &p, float x, float y, float z, float *t) {
  const float q[3] = {x, y, z};
#pragma unroll
  for (int d = 0; d < 3; ++d) t[d] = (float)(((double)q[d] - (double)p.origin[d]) / (double)p.spacing);
}

__device__ __forceinline__ int tl_region(const float *t, int *bxyz) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int c = (int)floor((double)t[d]) / 16;
    bxyz[d] = c < 0 ? 0 : (c > 7 ? 7 : c);
  }
  return bxyz[0] + 8 * bxyz[1] + 64 * bxyz[2];
}

// fine-grid TSC of a coordinate relative to region R; false if the nodes
// leave the first half of the inner grid
__device__ __forceinline__ bool tl_tsc(const TlRegion &R, const float *t, int *f, float *w9) {
  bool ok = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    f[d] = tsc_axis(__fmul_rn(__fsub_rn(t[d], R.u0[d]), (float)R.r), w9 + 3 * d);
    if (f[d] < 1 || f[d] + 2 > R.n_in / 2) ok = false;
  }
  return ok;
}

// Refinement ratio of every member (1 without refinement).
__global__ void tl_particle_kernel(const Members m, const PmHalo *__restrict__ H,
                                   const int32_t *__restrict__ mhalo, int64_t M,
                                   const uint8_t *__restrict__ region_r, uint8_t *__restrict__ pr) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < M;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int h = mhalo[k];
    if (h < 0) continue;
    const PmHalo &p = H[h];
    if (!p.two_level) { pr[k] = 1; continue; }
    float t[3];
    int bx[3];
    tl_t(p, m.q[0][k], m.q[1][k], m.q[2][k], t);
    pr[k] = region_r[(int64_t)h * 512 + tl_region(t, bx)];
  }
}

// A region's sources are the members inside its box widened by 3.5 + 3/r grid
// cells (:685-745), its targets the members inside it.  Neither is listed:
// the bricks that the (widened) box touches are whole rows of consecutive
// members in cell order, cut into chunks of kDepChunk, and a chunk's members
// test the box themselves.  A warp per region counts its chunks (fill = 0:
// cnt[a]) or writes them (fill = 1: from start[a] on); widen = 0 for targets.
__global__ void __launch_bounds__(BLK) tl_chunk_kernel(const PmHalo *__restrict__ H, const TlRegion *__restrict__ A,
                                                       int na, int widen, const uint32_t *__restrict__ cstart,
                                                       uint32_t *__restrict__ cnt, const uint32_t *__restrict__ start,
                                                       uint2 *__restrict__ chunk, int fill) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  for (int a = (int)(((int64_t)blockIdx.x * BLK + threadIdx.x) >> 5); a < na; a += (int)((gridDim.x * BLK) >> 5)) {
    const TlRegion &Rg = A[a];
    const PmHalo &p = H[Rg.h];
    int b0[3], nbk[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double mrg = widen ? (double)Rg.bo : 0.0, off = (double)p.origin[d] / (double)p.spacing - p.u_min[d];
      // (the FP32 grid units of a member are within 1e-5 of these)
      const double gl = ((double)Rg.lo[d] - mrg + off) / p.cw_u - 1e-3;
      const double gh = ((double)Rg.lo[d] + 16.0 + mrg + off) / p.cw_u + 1e-3;
      const int top = p.nc[d] - 1;
      const int c0 = gl <= 0.0 ? 0 : (gl >= (double)top ? top : (int)gl);
      const int c1 = gh <= 0.0 ? 0 : (gh >= (double)top ? top : (int)gh);
      b0[d] = c0 >> 2;
      nbk[d] = (c1 >> 2) - b0[d] + 1;
    }
    uint32_t run = 0;
    const int rows = nbk[1] * nbk[2];
    for (int r0 = 0; r0 < rows; r0 += 32) {
      const int r = r0 + lane;
      uint32_t e0 = 0, e1 = 0;
      if (r < rows) {
        const int y = b0[1] + r % nbk[1], z = b0[2] + r / nbk[1];
        e0 = cstart[sr_cell(p, 4 * b0[0], 4 * y, 4 * z)];
        e1 = cstart[sr_cell(p, 4 * (b0[0] + nbk[0] - 1), 4 * y, 4 * z) + 64];
      }
      const uint32_t n = (e1 - e0 + kDepChunk - 1) / kDepChunk;
      uint32_t incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
      }
      if (fill)
        for (uint32_t i = 0; i < n; ++i)
          chunk[start[a] + run + incl - n + i] =
              make_uint2(e0 + kDepChunk * i, min((uint32_t)kDepChunk, e1 - e0 - kDepChunk * i));
      run += __shfl_sync(FULL, incl, 31);
    }
    if (!fill && lane == 0) cnt[a] = run;
  }
}

// Whether a member at t is a target of region R.
__device__ __forceinline__ bool tl_is_target(const TlRegion &R, const float *t) {
  int bx[3];
  return tl_region(t, bx) == R.b;
}

// Inner self term of every target (:772-800); a block per target chunk.
template <typename R>
__global__ void __launch_bounds__(BLK) tl_self_kernel(const float4 *__restrict__ src4, const PmHalo *__restrict__ H,
                                                      const TlRegion *__restrict__ A, int na,
                                                      const uint32_t *__restrict__ start,
                                                      const uint2 *__restrict__ chunk, const R *__restrict__ self2,
                                                      const R *__restrict__ self4, R *__restrict__ self_in,
                                                      int32_t *flags) {
  const TlRegion &Rg = A[seg_of(start, na, blockIdx.x)];
  const uint2 c = chunk[blockIdx.x];
  if (threadIdx.x >= c.y) return;
  const int64_t e = (int64_t)c.x + threadIdx.x;
  const float4 q = src4[e];
  float t[3], w9[9];
  int f[3];
  tl_t(H[Rg.h], q.x, q.y, q.z, t);
  if (!tl_is_target(Rg, t)) return;
  if (!tl_tsc(Rg, t, f, w9)) {
    atomicCAS(&flags[FLAG_ERR], 0, kInvalid);
    return;
  }
  self_in[e] = tsc_self<R>(w9, Rg.r == 2 ? self2 : self4);
}

// Inner PM of a batch of refined regions of one inner grid size
// (bound_two_level_run_pm, :825-942): deposit of the kept sources, a block per
// source chunk ...
__global__ void __launch_bounds__(BLK) tl_deposit_kernel(const float4 *__restrict__ src4,
                                                         const uint32_t *__restrict__ cmem,
                                                         const PmHalo *__restrict__ H, const TlRegion *__restrict__ A,
                                                         const ConvBox *__restrict__ boxes,
                                                         const int32_t *__restrict__ batch,
                                                         const uint32_t *__restrict__ bpre, int nb,
                                                         const uint32_t *__restrict__ start,
                                                         const uint2 *__restrict__ chunk,
                                                         const uint8_t *__restrict__ keep,
                                                         unsigned long long *__restrict__ acc,
                                                         double *__restrict__ inv) {
  __shared__ DepositTile S;
  if (blockIdx.x == 0)
    for (int j = threadIdx.x; j < nb; j += blockDim.x) inv[j] = scalbn(1.0, fx_exp(H[A[batch[j]].h].mkeep) - 61);
  const int j = seg_of(bpre, nb, blockIdx.x);
  const int a = batch[j];
  const TlRegion &Rg = A[a];
  const PmHalo &p = H[Rg.h];
  const uint2 c = chunk[start[a] + (blockIdx.x - bpre[j])];
  int f[3] = {0, 0, 0};
  float w9[9] = {}, wk = 0.f;
  bool act = false;
  if (threadIdx.x < c.y) {
    const float4 q = src4[c.x + threadIdx.x];
    float t[3];
    tl_t(p, q.x, q.y, q.z, t);
    act = true;
#pragma unroll
    for (int d = 0; d < 3; ++d)
      act = act && t[d] >= __fsub_rn(Rg.lo[d], Rg.bo) && t[d] <= __fadd_rn(Rg.hi[d], Rg.bo);
    act = act && keep[cmem[c.x + threadIdx.x]];
    // (a source inside the widened box is inside the inner grid's half)
    if (act) act = tl_tsc(Rg, t, f, w9);
    wk = q.w;
  }
  deposit_chunk(act, f, w9, wk, fx_scale(61 - fx_exp(p.mkeep)), acc + boxes[j].in_off, boxes[j].in[0],
                boxes[j].in[1], S);
}

// ... and gather at the kept targets: phi_in = a r/(6 pi sp) (raw - w self_in)
template <typename R>
__global__ void __launch_bounds__(BLK) tl_gather_kernel(
    const float4 *__restrict__ src4, const uint32_t *__restrict__ cmem, const PmHalo *__restrict__ H,
    const TlRegion *__restrict__ A, const ConvBox *__restrict__ boxes, const int32_t *__restrict__ batch,
    const uint32_t *__restrict__ bpre, int nb, const uint32_t *__restrict__ start, const uint2 *__restrict__ chunk,
    const uint8_t *__restrict__ keep, const R *__restrict__ self_in, const R *__restrict__ rho, double a_val,
    R *__restrict__ phi_in) {
  const int j = seg_of(bpre, nb, blockIdx.x);
  const int a = batch[j];
  const TlRegion &Rg = A[a];
  const PmHalo &p = H[Rg.h];
  const uint2 c = chunk[start[a] + (blockIdx.x - bpre[j])];
  if (threadIdx.x >= c.y) return;
  const int64_t e = (int64_t)c.x + threadIdx.x;
  const float4 q = src4[e];
  float t[3], w9[9];
  int f[3];
  tl_t(p, q.x, q.y, q.z, t);
  if (!tl_is_target(Rg, t)) return;
  const int64_t k = cmem[e];
  if (!keep[k]) return;
  tl_tsc(Rg, t, f, w9);
  const ConvBox &bx = boxes[j];
  const int nx = bx.out[0], ny = bx.out[1];
  const R raw = tsc_gather<R>(rho + bx.out_off +
                                  (((int64_t)(f[2] - 1 - bx.out0[2]) * ny + (f[1] - 1 - bx.out0[1])) * nx +
                                   (f[0] - 1 - bx.out0[0])),
                              nx, ny, w9);
  const R pref = (R)(a_val * (double)Rg.r / (6.0 * kPi * (double)p.spacing));
  phi_in[k] = pref * (raw - (R)q.w * self_in[e]);
}

// ---------------------------------------------------------------- removal

__device__ __forceinline__ double bsum_d(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
  __syncthreads();
  return t;
}

// Seven block sums at once, for 32 warps or fewer: each is reduced as by
// bsum_d (warp butterfly, then the warp partials in warp order), so the
// results are bit-identical.  The butterfly's first three steps exchange
// halves: at each a lane hands over the values it does not go on with (18
// shuffles instead of 70), and one lane per value adds the partials, not
// every thread all of them.  Afterwards lane j of warp 0 holds sum j (j < 7);
// the other threads hold nothing.  red: 7 * 33 doubles.
__device__ __forceinline__ double block_sum7(const double *a, double *red) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const double hi = j < 3 ? a[j + 4] : 0.0;
    const double got = __shfl_xor_sync(FULL, lane & 16 ? a[j] : hi, 16);
    v[j] = (lane & 16 ? hi : a[j]) + got;
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const double got = __shfl_xor_sync(FULL, lane & 8 ? v[j] : v[j + 2], 8);
    v[j] = (lane & 8 ? v[j + 2] : v[j]) + got;
  }
  const double got = __shfl_xor_sync(FULL, lane & 4 ? v[0] : v[1], 4);
  double t = (lane & 4 ? v[1] : v[0]) + got;
  t += __shfl_xor_sync(FULL, t, 2);
  t += __shfl_xor_sync(FULL, t, 1);
  const int j = (lane & 16) / 4 + (lane & 8) / 4 + (lane & 4) / 4;
  if ((lane & 3) == 0 && j < 7) red[33 * j + warp] = t;
  __syncthreads();
  t = 0.0;
  if (warp == 0 && lane < 7) {
#pragma unroll 8
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[33 * lane + w];
  }
  return t;
}

// Centre and mean velocity from the seven sums in the lanes of warp 0, to
// c6[6].  All threads of warp 0 call it.
__device__ __forceinline__ void centre_of(double t, float *c6) {
  const int lane = threadIdx.x & 31;
  const double w = __shfl_sync(0xffffffffu, t, 0);
  if (lane >= 1 && lane < 7) c6[lane - 1] = __double2float_rn(t / w);
}

// The digit of the need-th largest key, from a 256-bin histogram of one digit
// of the keys: bins are summed from the top by one warp (eight bins per lane, a suffix
// scan over the lanes).  Returns the digit; above =
// keys in higher bins, count = keys in it.
__device__ __forceinline__ int digit_of(const unsigned *hist, int need, int &above, int &count) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int c[8], sum = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    c[j] = (int)hist[8 * lane + j];
    sum += c[j];
  }
  int suffix = sum;  // this lane's bins and all higher ones
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_down_sync(FULL, suffix, o);
    if (lane + o < 32) suffix += v;
  }
  // the highest lane whose suffix reaches `need` holds the digit
  const int src = 31 - __clz(__ballot_sync(FULL, suffix >= need));
  int ab = suffix - sum, digit = 0, cnt = 0;
  bool found = false;
#pragma unroll
  for (int j = 7; j >= 0; --j) {
    if (!found && ab + c[j] >= need) {
      digit = 8 * lane + j;
      cnt = c[j];
      found = true;
    }
    if (!found) ab += c[j];
  }
  above = __shfl_sync(FULL, ab, src);
  count = __shfl_sync(FULL, cnt, src);
  return __shfl_sync(FULL, digit, src);
}

// The unbound members leave most energetic first; equal energies: lower index
// first.  As one 64-bit key (the bits of E + 0, which order like E >= 0,
// then ~index) they are distinct; 0 is no key.
__device__ __forceinline__ unsigned long long removal_key(float e, uint32_t i) {
  return ((unsigned long long)__float_as_uint(e + 0.0f) << 32) | (0xffffffffu - i);
}

// The need-th largest of the keys key(0) .. key(nu - 1) up to the digits that
// do not matter: exactly `need` keys are at or above the value returned.
// Radix select by the block, from the exponent down, until the keys of the
// last digit's bin are all taken (three digits, usually).  Energies have few
// exponents, so that digit is counted per warp first.  hist: 2 x 256.
template <typename Key>
__device__ __forceinline__ unsigned long long nth_largest(Key key, int nu, int need, unsigned (*hist)[256],
                                                          int *s_digit) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nt = (int)blockDim.x;
  unsigned long long prefix = 0, mask = 0;
  for (int t = threadIdx.x; t < 512; t += nt) (&hist[0][0])[t] = 0;
  __syncthreads();
  for (int step = 0; step < 8; ++step) {
    // bits 62..55, 54..47, .., 14..7, 6..0
    const int shift = step < 7 ? 55 - 8 * step : 0;
    const unsigned dm = step < 7 ? 255u : 127u;
    unsigned *h = hist[step & 1];
    if (step == 0) {
      for (int t0 = 32 * warp; t0 < nu; t0 += nt) {
        const unsigned long long k = t0 + lane < nu ? key(t0 + lane) : 0;
        const unsigned d = k ? (unsigned)(k >> 55) & 255u : 256u;
        const unsigned same = __match_any_sync(FULL, d);
        if (k && lane == __ffs(same) - 1) atomicAdd(&h[d], (unsigned)__popc(same));
      }
    } else {
#pragma unroll 4
      for (int t = threadIdx.x; t < nu; t += nt) {
        const unsigned long long k = key(t);
        if (k && (k & mask) == prefix) atomicAdd(&h[(unsigned)(k >> shift) & dm], 1u);
      }
    }
    __syncthreads();
    if (warp == 0) {
      int above, count;
      const int digit = digit_of(h, need, above, count);
      if (lane == 0) {
        s_digit[0] = digit;
        s_digit[1] = need - above;
        s_digit[2] = count;
      }
    } else if (step > 0) {  // the previous step's bins, for the next step
      for (int t = threadIdx.x - 32; t < 256; t += nt - 32) hist[(step + 1) & 1][t] = 0;
    }
    __syncthreads();
    need = s_digit[1];
    prefix |= (unsigned long long)s_digit[0] << shift;
    mask |= (unsigned long long)dm << shift;
    if (need == s_digit[2]) break;
  }
  return prefix;
}

// One block per pending halo: combine the potential, then the inner
// removal loop of bound_check_grid (:2739-2855).  Leaves status -1 when the
// potential must be refreshed (next pass).
//
// A chain of sweeps over the members with a barrier between them, bound by
// latency.  An iteration sweeps all members twice (centre, energies) with the
// loads of four members in flight; the unbound ones go as removal keys to
// shared memory, where the nb-th largest is found.  Only when more than KCAP
// are unbound are the keys made again from memory, by sweeps over all members.
// (256^3 box, 17 passes: 1.79 ms with every thread adding all warps' partial
// sums, dividing for the centre and looking for the digit, 1.23 ms with one
// warp doing so.)
constexpr int KCAP = 4096;

template <typename R>
__global__ void __launch_bounds__(IBLK) pm_inner_kernel(const Members m, PmHalo *__restrict__ H,
                                                        const int32_t *__restrict__ list, int nlist,
                                                        uint8_t *__restrict__ keep,
                                                        const uint32_t *__restrict__ epos,
                                                        uint32_t *__restrict__ rflag,
                                                        const R *__restrict__ phi_c1,
                                                        const R *__restrict__ phi_in,
                                                        const R *__restrict__ phi_c2,
                                                        float *__restrict__ phi,
                                                        float *__restrict__ en, float b_val, int nmin,
                                                        int phi_only, int32_t *flags) {
  const int h = list[blockIdx.x];
  PmHalo &p = H[h];
  if (!p.pending) return;
  __shared__ double red7[7 * 33];
  __shared__ unsigned hist[2][256];
  __shared__ unsigned long long ukey[KCAP];
  __shared__ float s_c[6];
  __shared__ int s_err, s_nu, s_digit[3];
  const int64_t b0 = p.off;
  const int np = p.np;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_err = 0;
  int np_bound = p.np_bound;
  const int n_source = np_bound;
  for (int i = threadIdx.x; i < np; i += IBLK) {
    const int64_t k = b0 + i;
    if (!keep[k]) continue;
    float v = (float)((phi_c1[k] + phi_in[k]) + phi_c2[k]);
    if (np_bound == 1 || n_source == 1) v = 0.0f;
    if (!isfinite(v)) s_err = kNonFinite;
    phi[k] = v;
  }
  __syncthreads();
  if (s_err) {
    if (threadIdx.x == 0) atomicCAS(&flags[FLAG_ERR], 0, s_err);
    return;
  }
  if (phi_only) {
    if (threadIdx.x == 0) { p.status = 0; p.pending = 0; }
    return;
  }
  auto remove = [&](int i) {
    const int64_t k = b0 + i;
    keep[k] = 0;
    rflag[epos[k]] = 1;
  };
  int deleted = 0, status = -1;
  for (;;) {
    double a7[7] = {0, 0, 0, 0, 0, 0, 0};
    if (threadIdx.x == 0) s_nu = 0;
#pragma unroll 4
    for (int i = threadIdx.x; i < np; i += IBLK) {
      const int64_t k = b0 + i;
      const bool in = keep[k];
      const double wi = (double)m.w[k];
      a7[0] += in ? wi : 0.0;
      for (int d = 0; d < 3; ++d) {
        const double q = wi * (double)m.q[d][k], v = wi * (double)m.v[d][k];
        a7[1 + d] += in ? q : 0.0;
        a7[4 + d] += in ? v : 0.0;
      }
    }
    const double sum = block_sum7(a7, red7);
    if (threadIdx.x < 32) centre_of(sum, s_c);
    __syncthreads();
    const float qc[3] = {s_c[0], s_c[1], s_c[2]}, vc[3] = {s_c[3], s_c[4], s_c[5]};
#pragma unroll 4
    for (int i0 = threadIdx.x - lane; i0 < np; i0 += IBLK) {
      const int i = i0 + lane;
      const int64_t k = b0 + min(i, np - 1);
      const bool in = i < np && keep[k];
      float s = 0.f;
      for (int d = 0; d < 3; ++d) {
        const float dv = __fadd_rn(__fsub_rn(m.v[d][k], vc[d]), __fmul_rn(b_val, __fsub_rn(m.q[d][k], qc[d])));
        s = d == 0 ? __fmul_rn(dv, dv) : __fadd_rn(s, __fmul_rn(dv, dv));
      }
      float e = __fadd_rn(__fdiv_rn(s, 2.0f), phi[k]);
      if (in) {
        if (!isfinite(e)) s_err = kInvalid;
        en[k] = e;
      } else {
        e = -1.0f;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, e >= 0.0f);
      if (bal) {
        int at = 0;
        if (lane == 0) at = atomicAdd(&s_nu, __popc(bal));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(bal & lanemask_lt());
        if (e >= 0.0f && at < KCAP) ukey[at] = removal_key(e, (uint32_t)i);
      }
    }
    __syncthreads();
    const int nu = s_nu;
    if (s_err) break;
    if (nu == 0) {
      if (deleted == 0) status = 0;
      break;
    }
    const int nb = min(nu, max(1, (int)ceil(0.02 * (double)np_bound)));
    if (nu <= KCAP) {
      const unsigned long long least = nth_largest([&](int t) { return ukey[t]; }, nu, nb, hist, s_digit);
      for (int t = threadIdx.x; t < nu; t += IBLK) {
        const unsigned long long key = ukey[t];
        if (key >= least) remove((int)(0xffffffffu - (unsigned)key));
      }
    } else {
      auto key = [&](int i) -> unsigned long long {
        const int64_t k = b0 + i;
        const float e = keep[k] ? en[k] : -1.0f;
        return e >= 0.0f ? removal_key(e, (uint32_t)i) : 0ull;
      };
      const unsigned long long least = nth_largest(key, np, nb, hist, s_digit);
      for (int i = threadIdx.x; i < np; i += IBLK) {
        const unsigned long long v = key(i);
        if (v && v >= least) remove(i);
      }
    }
    __syncthreads();
    np_bound -= nb;
    deleted += nb;
    if (np_bound < nmin) { status = 1; break; }
    if ((double)deleted >= 0.2 * (double)np_bound) break;
  }
  __syncthreads();
  if (s_err) {
    if (threadIdx.x == 0) atomicCAS(&flags[FLAG_ERR], 0, s_err);
    return;
  }
  if (threadIdx.x == 0) {
    p.np_bound = np_bound;
    p.status = status;
    if (status >= 0) p.pending = 0;
  }
}

// ------------------------------------------------- removal of large halos
// Halos above kBigNp members run the same removal loop as pm_inner_kernel,
// but spread over the whole GPU: their members are cut into chunks of
// kChunk, every sweep is a grid of chunk blocks, and the per-halo decisions
// (selection, stop conditions) are small kernels between sweeps,
// driven by a host loop.  The unbound members of an iteration are compacted
// into a per-halo list of removal keys, so the selection runs over that list
// only.
// Bound by the latency of three small launches per iteration: one halo of
// 0.6 M members 29 us, in four launches with the centre by one thread and
// half as many blocks per sweep 62 us.

constexpr int64_t kBigNp = 32768;  // default; option "unbind_big_np" overrides
constexpr int kChunk = 8192;
// blocks per chunk of the sweeps that sum nothing
constexpr int kBigSplit = 4;

struct BigHalo {
  int32_t h;          // index into the PM halo table
  int32_t active;     // still in this pass's inner loop
  int64_t off, np;    // members
  int64_t uoff;       // first slot of the halo's unbound list
  int32_t chunk0, nchunk;
  int32_t np_bound, deleted, n_source, status;
};

struct BigChunk {
  int32_t b;          // big halo
  int64_t start, end; // member range
};

// phi = (c1 + in) + c2 of the kept members at the start of a pass
template <typename R>
__global__ void big_phi_kernel(const BigChunk *__restrict__ ch, int nch, const BigHalo *__restrict__ B,
                               const uint8_t *__restrict__ keep, const R *__restrict__ c1,
                               const R *__restrict__ in, const R *__restrict__ c2, float *__restrict__ phi,
                               int32_t *flags) {
  const BigChunk c = ch[blockIdx.x / kBigSplit];
  const BigHalo &bh = B[c.b];
  if (!bh.active) return;
  bool bad = false;
  const int64_t k0 = c.start + (int64_t)(blockIdx.x % kBigSplit) * (kChunk / kBigSplit);
  const int64_t k1 = min(c.end, k0 + kChunk / kBigSplit);
#pragma unroll 4
  for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
    if (!keep[k]) continue;
    float v = (float)((c1[k] + in[k]) + c2[k]);
    if (bh.np_bound == 1 || bh.n_source == 1) v = 0.0f;
    bad |= !isfinite(v);
    phi[k] = v;
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicCAS(&flags[FLAG_ERR], 0, kNonFinite);
}

// per-chunk sums of w, w q, w v over the kept members
__global__ void big_com_kernel(const Members m, const BigChunk *__restrict__ ch, const BigHalo *__restrict__ B,
                               const uint8_t *__restrict__ keep, double *__restrict__ part) {
  const BigChunk c = ch[blockIdx.x];
  if (!B[c.b].active) return;
  double a7[7] = {0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
  for (int64_t k = c.start + threadIdx.x; k < c.end; k += blockDim.x) {
    const bool in = keep[k];
    const double wi = (double)m.w[k];
    a7[0] += in ? wi : 0.0;
    for (int d = 0; d < 3; ++d) {
      const double q = wi * (double)m.q[d][k], v = wi * (double)m.v[d][k];
      a7[1 + d] += in ? q : 0.0;
      a7[4 + d] += in ? v : 0.0;
    }
  }
  __shared__ double red[7 * 33];
  const double t = block_sum7(a7, red);
  if (threadIdx.x < 7) part[7 * (int64_t)blockIdx.x + threadIdx.x] = t;
}

// Energies of the kept members; the unbound ones join the halo's list.  Every
// block adds up the halo's chunk sums (in chunk order) for the centre itself.
__global__ void big_energy_kernel(const Members m, const BigChunk *__restrict__ ch, const BigHalo *__restrict__ B,
                                  const uint8_t *__restrict__ keep, const float *__restrict__ phi,
                                  const double *__restrict__ part, float b_val, int32_t *__restrict__ ucount,
                                  unsigned long long *__restrict__ ulist, int32_t *flags) {
  const BigChunk c = ch[blockIdx.x / kBigSplit];
  const BigHalo &bh = B[c.b];
  if (!bh.active) return;
  const int lane = threadIdx.x & 31;
  __shared__ float s_c[6];
  if (threadIdx.x < 32) {
    double t = 0.0;
    if (lane < 7) {
#pragma unroll 8
      for (int j = bh.chunk0; j < bh.chunk0 + bh.nchunk; ++j) t += part[7 * (int64_t)j + lane];
    }
    centre_of(t, s_c);
  }
  __syncthreads();
  const float qc[3] = {s_c[0], s_c[1], s_c[2]}, vc[3] = {s_c[3], s_c[4], s_c[5]};
  bool bad = false;
  const int64_t k0 = c.start + (int64_t)(blockIdx.x % kBigSplit) * (kChunk / kBigSplit);
  const int64_t k1 = min(c.end, k0 + kChunk / kBigSplit);
#pragma unroll 4
  for (int64_t base = k0; base < k1; base += blockDim.x) {
    const int64_t i = base + threadIdx.x, k = min(i, k1 - 1);
    const bool in = i < k1 && keep[k];
    float s = 0.f;
    for (int d = 0; d < 3; ++d) {
      const float dv = __fadd_rn(__fsub_rn(m.v[d][k], vc[d]), __fmul_rn(b_val, __fsub_rn(m.q[d][k], qc[d])));
      s = d == 0 ? __fmul_rn(dv, dv) : __fadd_rn(s, __fmul_rn(dv, dv));
    }
    const float e = __fadd_rn(__fdiv_rn(s, 2.0f), phi[k]);
    if (in) bad |= !isfinite(e);
    const bool unb = in && e >= 0.0f;
    // warp-aggregated append
    const unsigned bal = __ballot_sync(0xffffffffu, unb);
    int at = 0;
    if (lane == 0 && bal) at = atomicAdd(&ucount[c.b], __popc(bal));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (unb) ulist[bh.uoff + at + __popc(bal & lanemask_lt())] = removal_key(e, (uint32_t)(k - bh.off));
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicCAS(&flags[FLAG_ERR], 0, kInvalid);
}

// per big halo, one block: the nb most unbound members leave, then the stop
// conditions of the inner loop; the count starts again
__global__ void __launch_bounds__(IBLK) big_select_kernel(BigHalo *__restrict__ B, int32_t *__restrict__ ucount,
                                                          const unsigned long long *__restrict__ ulist,
                                                          uint8_t *__restrict__ keep,
                                                          const uint32_t *__restrict__ epos,
                                                          uint32_t *__restrict__ rflag,
                                                          int nmin, int32_t *__restrict__ nactive,
                                                          const int32_t *flags) {
  BigHalo &bh = B[blockIdx.x];
  if (!bh.active) return;
  __shared__ unsigned hist[2][256];
  __shared__ int s_digit[3];
  if (flags[FLAG_ERR]) {  // a sweep failed: stop, the host reports it
    if (threadIdx.x == 0) { bh.active = 0; atomicSub(nactive, 1); }
    return;
  }
  const int nu = ucount[blockIdx.x];
  if (nu == 0) {
    if (threadIdx.x == 0) {
      if (bh.deleted == 0) bh.status = 0;
      bh.active = 0;
      atomicSub(nactive, 1);
    }
    return;
  }
  const int nb = min(nu, max(1, (int)ceil(0.02 * (double)bh.np_bound)));
  const unsigned long long *L = ulist + bh.uoff;
  const unsigned long long least = nth_largest([&](int t) { return L[t]; }, nu, nb, hist, s_digit);
#pragma unroll 4
  for (int t = threadIdx.x; t < nu; t += IBLK) {
    const unsigned long long key = L[t];
    if (key < least) continue;
    const int64_t k = bh.off + (0xffffffffu - (unsigned)key);
    keep[k] = 0;
    rflag[epos[k]] = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ucount[blockIdx.x] = 0;
    bh.np_bound -= nb;
    bh.deleted += nb;
    if (bh.np_bound < nmin) {
      bh.status = 1;
      bh.active = 0;
      atomicSub(nactive, 1);
    } else if ((double)bh.deleted >= 0.2 * (double)bh.np_bound) {
      bh.active = 0;
      atomicSub(nactive, 1);
    }
  }
}

// the pass's outcome back into the PM halo table
__global__ void big_finish_kernel(const BigHalo *__restrict__ B, int nbig, PmHalo *__restrict__ H) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbig) return;
  const BigHalo &bh = B[b];
  PmHalo &p = H[bh.h];
  if (!p.pending) return;
  p.np_bound = bh.np_bound;
  p.status = bh.status;
  if (bh.status >= 0) p.pending = 0;
}

// start of a pass: the pending big halos enter the inner loop
__global__ void big_start_kernel(BigHalo *__restrict__ B, int nbig, const PmHalo *__restrict__ H, int phi_only,
                                 int32_t *__restrict__ nactive, int32_t *__restrict__ ucount) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbig) return;
  BigHalo &bh = B[b];
  ucount[b] = 0;
  const PmHalo &p = H[bh.h];
  bh.active = p.pending ? 1 : 0;
  bh.np_bound = p.np_bound;
  bh.n_source = p.np_bound;
  bh.deleted = 0;
  bh.status = -1;
  if (bh.active) atomicAdd(nactive, 1);
  (void)phi_only;
}

__global__ void big_phi_only_kernel(BigHalo *__restrict__ B, int nbig) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbig || !B[b].active) return;
  B[b].status = 0;
  B[b].active = 0;
}

// pm_mkeep_kernel of the big halos: chunk sums of the kept mass, then the
// ordered sum per halo
__global__ void big_mass_kernel(const Members m, const BigChunk *__restrict__ ch, const BigHalo *__restrict__ B,
                                const PmHalo *__restrict__ H, const uint8_t *__restrict__ keep,
                                double *__restrict__ part) {
  const BigChunk c = ch[blockIdx.x];
  if (!H[B[c.b].h].pending) return;
  double s = 0.0;
#pragma unroll 8
  for (int64_t k = c.start + threadIdx.x; k < c.end; k += blockDim.x) {
    const double w = (double)m.w[k];
    s += keep[k] ? w : 0.0;
  }
  __shared__ double red[32];
  s = bsum_d(s, red);
  if (threadIdx.x == 0) part[7 * (int64_t)blockIdx.x] = s;
}

__global__ void big_mass_sum_kernel(const BigHalo *__restrict__ B, int nbig, const double *__restrict__ part,
                                    PmHalo *__restrict__ H) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbig) return;
  const BigHalo &bh = B[b];
  PmHalo &p = H[bh.h];
  if (!p.pending) return;
  double s = 0.0;
  for (int c = bh.chunk0; c < bh.chunk0 + bh.nchunk; ++c) s += part[7 * (int64_t)c];
  p.mkeep = s;
}

__global__ void pm_mkeep_kernel(const Members m, PmHalo *__restrict__ H, const int32_t *list, int nlist,
                                const uint8_t *__restrict__ keep) {
  const int h = list[blockIdx.x];
  PmHalo &p = H[h];
  if (!p.pending) return;
  double s = 0.0;
#pragma unroll 8
  for (int64_t i = threadIdx.x; i < p.np; i += blockDim.x) {
    const int64_t k = p.off + i;
    const double w = (double)m.w[k];
    s += keep[k] ? w : 0.0;
  }
  __shared__ double red[32];
  s = bsum_d(s, red);
  if (threadIdx.x == 0) p.mkeep = s;
}

// Members of every PM halo: their halo, and kept.
__global__ void pm_mark_halo_kernel(const PmHalo *__restrict__ H, int nh, int32_t *__restrict__ mhalo,
                                    uint8_t *__restrict__ keep) {
  const int h = blockIdx.x;
  if (h >= nh) return;
  for (int64_t i = threadIdx.x; i < H[h].np; i += blockDim.x) {
    mhalo[H[h].off + i] = h;
    keep[H[h].off + i] = 1;
  }
}

// Results of the PM halos into the candidates' table.
__global__ void pm_result_kernel(const PmHalo *__restrict__ H, const int32_t *__restrict__ cand, int nh,
                                 HaloResult *__restrict__ res) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= nh) return;
  res[cand[h]].status = H[h].pending ? 5 : H[h].status;
  res[cand[h]].np_bound = H[h].np_bound;
}

__global__ void pm_fill_i32(int32_t *a, int64_t n, int32_t v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    a[i] = v;
}

// Members per 16-cell region of every 256-grid halo
// (bound_two_level_setup_ratios, bound_fortran.f90:551-568).
__global__ void pm_region_count_kernel(const Members m, const PmHalo *__restrict__ H,
                                       const int32_t *__restrict__ mhalo, int64_t M,
                                       uint32_t *__restrict__ cnt) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < M;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int h = mhalo[k];
    if (h < 0 || H[h].n != 256) continue;
    const PmHalo &p = H[h];
    int b[3];
    for (int d = 0; d < 3; ++d) {
      const float t = (float)(((double)m.q[d][k] - (double)p.origin[d]) / (double)p.spacing);
      const int c = (int)floor((double)t) / 16;
      b[d] = c < 0 ? 0 : (c > 7 ? 7 : c);
    }
    atomicAdd(&cnt[(int64_t)h * 512 + b[0] + 8 * b[1] + 64 * b[2]], 1u);
  }
}

int bits_for(uint64_t v) {
  int b = 0;
  while (b < 64 && (v >> b) != 0) ++b;
  return b;
}

// One pass of the removal loop of the large halos (see BigHalo).
template <typename R>
int32_t big_removal(Context &ctx, const Members &m, BigHalo *dB, int nbig, const BigChunk *dCh, int nchb,
                    PmHalo *dH, uint8_t *keep, const uint32_t *epos, uint32_t *rflag, const R *c1, const R *phi_in, const R *c2,
                    float *phi, double *part, int32_t *ucount, unsigned long long *ulist, int32_t *nactive, float b_val, int nmin, int phi_only) {
  cudaStream_t s = ctx.stream;
  const unsigned gb = (unsigned)ceil_div(nbig, 128);
  PYFOF_CUDA(cudaMemsetAsync(nactive, 0, sizeof(int32_t), s));
  big_start_kernel<<<gb, 128, 0, s>>>(dB, nbig, dH, phi_only, nactive, ucount);
  PYFOF_CHECK_LAUNCH();
  big_phi_kernel<R><<<nchb * kBigSplit, 256, 0, s>>>(dCh, nchb, dB, keep, c1, phi_in, c2, phi, ctx.d_flags);
  PYFOF_CHECK_LAUNCH();
  if (phi_only) {
    big_phi_only_kernel<<<gb, 128, 0, s>>>(dB, nbig);
    PYFOF_CHECK_LAUNCH();
  } else {
    // iterations until every big halo left the inner loop; the host looks
    // every few iterations (an iteration removes >= 2 % of a halo, and a pass
    // ends after 20 %)
    PYFOF_CUDA(wait_velocities(ctx, s));
    for (int it = 0; it < 1 << 20; it += 4) {
      for (int j = 0; j < 4; ++j) {
        big_com_kernel<<<nchb, 256, 0, s>>>(m, dCh, dB, keep, part);
        PYFOF_CHECK_LAUNCH();
        big_energy_kernel<<<nchb * kBigSplit, 256, 0, s>>>(m, dCh, dB, keep, phi, part, b_val, ucount, ulist,
                                                           ctx.d_flags);
        PYFOF_CHECK_LAUNCH();
        big_select_kernel<<<nbig, IBLK, 0, s>>>(dB, ucount, ulist, keep, epos, rflag, nmin, nactive, ctx.d_flags);
        PYFOF_CHECK_LAUNCH();
      }
      PYFOF_CUDA(cudaMemcpyAsync(ctx.h_flags + FLAG_COUNT_B, nactive, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
      PYFOF_CUDA(cudaStreamSynchronize(s));
      if (ctx.h_flags[FLAG_COUNT_B] <= 0) break;
    }
  }
  big_finish_kernel<<<gb, 128, 0, s>>>(dB, nbig, dH);
  PYFOF_CHECK_LAUNCH();
  return kOk;
}

template <typename R>
int32_t run_pm(Context &ctx, const FofArgs &a, const GridRules &rules, const Members &m,
               const std::vector<HaloTask> &tasks, const std::vector<int32_t> &list,
               HaloResult *res, uint8_t *keep, float *phi_out, int phi_only) {
  (void)rules;
  cudaStream_t s = ctx.stream;
  Arena &W = ctx.work;
  const int nh = (int)list.size();
  const int64_t M = tasks.back().off + tasks.back().np;  // all packed members
  // Green tables of the grid classes in use
  std::shared_ptr<GreenTable> green_of[257];
  std::vector<PmHalo> H(nh);
  std::vector<const R *> selfs(nh);
  for (int h = 0; h < nh; ++h) {
    const HaloTask &t = tasks[list[h]];
    PmHalo &p = H[h];
    std::memset(&p, 0, sizeof(p));
    p.off = t.off;
    p.np = t.np;
    p.n = t.n;
    p.spacing = t.spacing;
    for (int d = 0; d < 3; ++d) p.origin[d] = t.origin[d];
    p.np_bound = t.np;
    p.status = -1;
    p.pending = 1;
    if (!green_of[t.n]) PYFOF_TRY(get_green<R>(ctx, t.n, 3.5, 0.0, 1, &green_of[t.n]));
    selfs[h] = (const R *)green_of[t.n]->self;
  }
  PmHalo *dH = W.carve<PmHalo>(nh);
  int32_t *dlist = W.carve<int32_t>(nh);
  const R **dselfs = W.carve<const R *>(nh);
  int32_t *mhalo = W.carve<int32_t>(M);
  R *selfe = W.carve<R>(M), *c1 = W.carve<R>(M), *c2 = W.carve<R>(M);
  float *phi = W.carve<float>(M), *en = W.carve<float>(M);
  R *tl_self_in = nullptr;
  uint32_t *epos = W.carve<uint32_t>(M);  // positions in cell order (PM members)
  if (!epos) { set_error("workspace exhausted (cell positions)"); return kAlloc; }
  double *ext = W.carve<double>(6 * (size_t)nh);
  int32_t *dsup = W.carve<int32_t>(3 * (size_t)nh);
  if (!dH || !dlist || !dselfs || !mhalo || !selfe || !c1 || !c2 || !phi || !en || !ext || !dsup) {
    set_error("workspace exhausted (PM members)");
    return kAlloc;
  }
  PYFOF_TRY(upload(ctx, dH, H.data(), sizeof(PmHalo) * nh, s));
  PYFOF_TRY(upload(ctx, dlist, list.data(), sizeof(int32_t) * nh, s));
  PYFOF_TRY(upload(ctx, dselfs, selfs.data(), sizeof(R *) * nh, s));
  const unsigned gM = (unsigned)std::min<int64_t>(ceil_div(M, BLK), (int64_t)kNumSMs * 16);
  pm_fill_i32<<<gM, BLK, 0, s>>>(mhalo, M, -1);
  PYFOF_CHECK_LAUNCH();
  pm_mark_halo_kernel<<<nh, BLK, 0, s>>>(dH, nh, mhalo, keep);
  PYFOF_CHECK_LAUNCH();
  // two-level refinement of dense 16-cell regions of 256-grid halos
  // (bound_two_level_setup_ratios / build_halo, bound_fortran.f90:551-823)
  std::vector<TlRegion> act;
  std::vector<uint8_t> region_r((size_t)nh * 512, 1);
  {
    uint32_t *rc = W.carve<uint32_t>((size_t)nh * 512);
    if (!rc) { set_error("workspace exhausted (regions)"); return kAlloc; }
    PYFOF_CUDA(cudaMemsetAsync(rc, 0, sizeof(uint32_t) * nh * 512, s));
    pm_region_count_kernel<<<gM, BLK, 0, s>>>(m, dH, mhalo, M, rc);
    PYFOF_CHECK_LAUNCH();
    std::vector<uint32_t> hrc((size_t)nh * 512);
    PYFOF_CUDA(cudaMemcpyAsync(hrc.data(), rc, sizeof(uint32_t) * nh * 512, cudaMemcpyDeviceToHost, s));
    PYFOF_CUDA(cudaStreamSynchronize(s));
    const double app_f = (double)(float)a.softening;
    for (int h = 0; h < nh; ++h) {
      if (H[h].n != 256) continue;
      const double sp = (double)H[h].spacing;
      int rmax = 1;
      for (int b = 0; b < 512; ++b) {
        const uint32_t c = hrc[(size_t)h * 512 + b];
        int r = c < 3926u ? 1 : (c < 14688u ? 2 : 4);
        if (r == 4 && 3.5 * (sp / 4.0) < app_f) r = 2;
        if (r == 2 && 3.5 * (sp / 2.0) < app_f) r = 1;
        region_r[(size_t)h * 512 + b] = (uint8_t)r;
        if (c > 0 && r > rmax) rmax = r;
      }
      if (rmax == 1) continue;
      H[h].two_level = 1;
      H[h].r_max = rmax;
      for (int b = 0; b < 512; ++b) {
        const uint32_t c = hrc[(size_t)h * 512 + b];
        const int r = region_r[(size_t)h * 512 + b];
        if (c == 0 || r == 1) continue;
        TlRegion Rg;
        Rg.h = h;
        Rg.b = b;
        Rg.r = r;
        Rg.n_in = r == 2 ? 128 : 216;
        const int bb[3] = {b % 8, (b / 8) % 8, b / 64};
        Rg.bo = 3.5f + 3.0f / (float)r;
        for (int d = 0; d < 3; ++d) {
          Rg.lo[d] = (float)(bb[d] * 16);
          Rg.hi[d] = std::min(Rg.lo[d] + 16.0f, 127.0f);
          Rg.u0[d] = ((Rg.lo[d] - Rg.bo) - (1.0f / (float)r)) + (0.0f / (float)r);
        }
        act.push_back(Rg);
      }
    }
    ctx.last_tl_regions = (int64_t)act.size();
  }
  // C2 cells (3.5 grid cells)
  {
    uint32_t *omin = W.carve<uint32_t>(3 * (size_t)nh), *omax = W.carve<uint32_t>(3 * (size_t)nh);
    if (!omin || !omax) { set_error("workspace exhausted (extents)"); return kAlloc; }
    std::vector<int2> work;
    for (int h = 0; h < nh; ++h)
      for (int64_t c = 0; c * kExtentChunk < std::max<int64_t>(H[h].np, 1); ++c) work.push_back(make_int2(h, (int)c));
    int2 *dwork = W.carve<int2>(work.size());
    if (!dwork) { set_error("workspace exhausted (extents)"); return kAlloc; }
    PYFOF_TRY(upload(ctx, dwork, work.data(), sizeof(int2) * work.size(), s));
    PYFOF_CUDA(cudaMemsetAsync(omin, 0xff, sizeof(uint32_t) * 3 * nh, s));
    PYFOF_CUDA(cudaMemsetAsync(omax, 0, sizeof(uint32_t) * 3 * nh, s));
    if (!work.empty()) {
      pm_extent_kernel<<<(unsigned)work.size(), BLK, 0, s>>>(m, dH, dwork, omin, omax);
      PYFOF_CHECK_LAUNCH();
    }
    pm_extent_final_kernel<<<(unsigned)ceil_div(3 * (int64_t)nh, 128), 128, 0, s>>>(dH, nh, omin, omax, ext,
                                                                                       dsup);
    PYFOF_CHECK_LAUNCH();
  }
  std::vector<double> hext(6 * (size_t)nh);
  std::vector<int32_t> hsup(3 * (size_t)nh);
  PYFOF_CUDA(cudaMemcpyAsync(hext.data(), ext, sizeof(double) * 6 * nh, cudaMemcpyDeviceToHost, s));
  PYFOF_CUDA(cudaMemcpyAsync(hsup.data(), dsup, sizeof(int32_t) * 3 * nh, cudaMemcpyDeviceToHost, s));
  PYFOF_CUDA(cudaStreamSynchronize(s));
  int64_t ncell = 0, first_e = 0;
  for (int h = 0; h < nh; ++h) {
    PmHalo &p = H[h];
    p.cell_off = ncell;
    p.e0 = first_e;
    first_e += p.np;
    p.cw_u = p.two_level ? 3.5 / (double)p.r_max : 3.5;
    int64_t c = 1;
    for (int d = 0; d < 3; ++d) {
      p.u_min[d] = hext[6 * h + d];
      p.sup[d] = hsup[3 * h + d];
      const double span = hext[6 * h + 3 + d] - hext[6 * h + d];
      p.nc[d] = std::max(1, (int)std::floor(span / p.cw_u) + 1);
      c *= 4 * (((int64_t)p.nc[d] + 3) / 4);  // whole bricks of 4^3 cells
    }
    ncell += c;
  }
  if (ncell >= 0xffffffffll) { set_error("too many C2 cells"); return kAlloc; }
  PYFOF_TRY(upload(ctx, dH, H.data(), sizeof(PmHalo) * nh, s));
  uint32_t *ckey = W.carve<uint32_t>(M), *cstart = W.carve<uint32_t>(ncell + 2);
  uint32_t *ka = W.carve<uint32_t>(M), *va = W.carve<uint32_t>(M), *kb = W.carve<uint32_t>(M),
           *vb = W.carve<uint32_t>(M);
  if (!ckey || !cstart || !ka || !va || !kb || !vb) { set_error("workspace exhausted (C2 cells)"); return kAlloc; }
  const uint32_t sentinel = (uint32_t)ncell;
  // Morton sub-key bits inside a cell (a multiple of 3, the key within 32 bits)
  const int sb = std::max(0, std::min(9, 32 - bits_for((uint64_t)ncell))) / 3 * 3;
  uint32_t *skey = W.carve<uint32_t>(M);
  if (!skey) { set_error("workspace exhausted (C2 cells)"); return kAlloc; }
  pm_cellkey_kernel<<<gM, BLK, 0, s>>>(m, dH, mhalo, M, ckey, sentinel, sb, skey);
  PYFOF_CHECK_LAUNCH();
  PYFOF_CUDA(cudaMemsetAsync(cstart, 0, sizeof(uint32_t) * (ncell + 2), s));
  pm_cellcount_kernel<<<gM, BLK, 0, s>>>(ckey, M, sentinel, cstart);
  PYFOF_CHECK_LAUNCH();
  PYFOF_TRY(exclusive_scan_u32(cstart, cstart, ncell + 1, nullptr, W, s));
  uint32_t *sk, *cmem;
  PYFOF_TRY(radix_sort_pairs(skey, nullptr, M, bits_for((uint64_t)sentinel << sb), ka, va, kb, vb, &sk, &cmem,
                             W, s));
  // cell-ordered positions and weights, target chunks, removal lists
  uint32_t npm = 0;
  PYFOF_CUDA(cudaMemcpyAsync(&npm, cstart + ncell, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  const int64_t nbrick = ncell / 64;
  uint32_t *chcnt = W.carve<uint32_t>(nbrick + 1);
  if (!chcnt) { set_error("workspace exhausted (C2 chunks)"); return kAlloc; }
  PYFOF_CUDA(cudaMemsetAsync(chcnt, 0, sizeof(uint32_t) * (nbrick + 1), s));
  const unsigned gC = (unsigned)std::min<int64_t>(ceil_div(std::max<int64_t>(nbrick, 1), BLK), 148 * 16);
  sr_chunk_count_kernel<<<gC, BLK, 0, s>>>(cstart, nbrick, chcnt);
  PYFOF_CHECK_LAUNCH();
  PYFOF_TRY(exclusive_scan_u32(chcnt, chcnt, nbrick + 1, nullptr, W, s));
  uint32_t nchunk = 0;
  PYFOF_CUDA(cudaMemcpyAsync(&nchunk, chcnt + nbrick, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  PYFOF_CUDA(cudaStreamSynchronize(s));
  float4 *src4 = W.carve<float4>(std::max<uint32_t>(npm, 1));
  SrChunk *chunks = W.carve<SrChunk>(std::max<uint32_t>(nchunk, 1));
  uint2 *chspan = W.carve<uint2>(std::max<uint32_t>(nchunk, 1));
  uint32_t *rflag = W.carve<uint32_t>((size_t)npm + 1), *rpos = W.carve<uint32_t>((size_t)npm + 1);
  uint32_t *rsrc = W.carve<uint32_t>(std::max<uint32_t>(npm, 1));
  // [0..1] the chunk counters of a pass, [2..3] the heavy chunks (first pass, updates)
  unsigned *sr_next = W.carve<unsigned>(4);
  if (!src4 || !chunks || !chspan || !rflag || !rpos || !rsrc || !sr_next) {
    set_error("workspace exhausted (C2 sources)");
    return kAlloc;
  }
  PYFOF_CUDA(cudaMemsetAsync(sr_next, 0, 4 * sizeof(unsigned), s));
  PYFOF_CUDA(cudaMemsetAsync(rflag, 0, sizeof(uint32_t) * ((size_t)npm + 1), s));
  const unsigned gP = (unsigned)std::min<int64_t>(ceil_div(std::max<uint32_t>(npm, 1), BLK), 148 * 16);
  sr_pack_kernel<<<gP, BLK, 0, s>>>(m, cmem, npm, src4, epos);
  PYFOF_CHECK_LAUNCH();
  pm_setup_kernel<R><<<gP, BLK, 0, s>>>(src4, cmem, npm, dH, mhalo, dselfs, selfe, ctx.d_flags);
  PYFOF_CHECK_LAUNCH();
  sr_chunk_fill_kernel<<<gC, BLK, 0, s>>>(cstart, chcnt, nbrick, chspan);
  PYFOF_CHECK_LAUNCH();
  SrSpline *splines = W.carve<SrSpline>(3 * (size_t)nh);
  if (!splines) { set_error("workspace exhausted (C2 splines)"); return kAlloc; }
  static_assert(sizeof(SrSpline) % 16 == 0, "copied as 16-byte words");
  if (sizeof(R) == 8) {
    sr_spline_kernel<<<(unsigned)ceil_div(3 * (int64_t)nh, 128), 128, 0, s>>>(dH, nh, a.softening, splines);
    PYFOF_CHECK_LAUNCH();
  }
  // persistent blocks: those that fit on the GPU at once, if there is work for
  // them; with fewer chunks than the warps of two blocks per SM, no more than
  // two (one halo of 30,000 members: 0.32 ms against 0.39 with three, where
  // most blocks take two chunks and some a third)
  const int per_sm = nchunk <= 148 * 2 * kSrWarps ? 2 : (sizeof(R) == 4 ? 4 : 3);
  const unsigned gS = (unsigned)std::min<int64_t>(std::max<uint32_t>(nchunk, 1), 148 * per_sm);
  // per-member refinement ratio, refined-region sources and targets
  const int na = (int)act.size();
  uint8_t *pr = W.carve<uint8_t>(M);
  R *phi_in = W.carve<R>(M);
  if (!pr || !phi_in) { set_error("workspace exhausted (two-level)"); return kAlloc; }
  PYFOF_CUDA(cudaMemsetAsync(phi_in, 0, sizeof(R) * M, s));
  PYFOF_CUDA(cudaMemsetAsync(pr, 1, M, s));
  TlRegion *dA = nullptr;
  // source and target chunks of the refined regions (tl_chunk_kernel)
  uint32_t *src_start = nullptr, *tgt_start = nullptr;
  uint2 *src = nullptr, *tgt = nullptr;
  std::vector<uint32_t> hsrc, htgt;
  std::shared_ptr<GreenTable> g_r2, g_r4;
  {
    uint8_t *dregr = W.carve<uint8_t>((size_t)nh * 512);
    if (!dregr) { set_error("workspace exhausted (two-level)"); return kAlloc; }
    PYFOF_TRY(upload(ctx, dregr, region_r.data(), (size_t)nh * 512, s));
    tl_particle_kernel<<<gM, BLK, 0, s>>>(m, dH, mhalo, M, dregr, pr);
    PYFOF_CHECK_LAUNCH();
    {
      // chunk records, then most sources first (a stable sort on a 16-bit key)
      const int64_t nc = std::max<uint32_t>(nchunk, 1);
      uint32_t *ck = W.carve<uint32_t>(nc), *c1k = W.carve<uint32_t>(nc), *c1v = W.carve<uint32_t>(nc),
               *c2k = W.carve<uint32_t>(nc), *c2v = W.carve<uint32_t>(nc);
      SrChunk *sorted = W.carve<SrChunk>(nc);
      if (!ck || !c1k || !c1v || !c2k || !c2v || !sorted) { set_error("workspace exhausted (C2 chunks)"); return kAlloc; }
      const unsigned gW = (unsigned)std::min<int64_t>(ceil_div(nc * 32, BLK), 148 * 16);
      sr_chunk_setup_kernel<<<gW, BLK, 0, s>>>(chspan, nchunk, dH, mhalo, cmem, src4, pr, cstart, chunks, ck,
                                               sr_next + 2);
      PYFOF_CHECK_LAUNCH();
      const unsigned gK = (unsigned)std::min<int64_t>(ceil_div(nc, BLK), 148 * 16);
      uint32_t *sk2, *order;
      PYFOF_TRY(radix_sort_pairs(ck, nullptr, nchunk, 16, c1k, c1v, c2k, c2v, &sk2, &order, W, s));
      sr_chunk_order_kernel<<<gK, BLK, 0, s>>>(chunks, order, nchunk, sorted);
      PYFOF_CHECK_LAUNCH();
      chunks = sorted;
    }
    if (na > 0) {
      dA = W.carve<TlRegion>(na);
      uint32_t *cnt = W.carve<uint32_t>(na + 1);
      src_start = W.carve<uint32_t>(na + 1);
      tgt_start = W.carve<uint32_t>(na + 1);
      if (!dA || !cnt || !src_start || !tgt_start) { set_error("workspace exhausted (two-level)"); return kAlloc; }
      PYFOF_TRY(upload(ctx, dA, act.data(), sizeof(TlRegion) * na, s));
      const unsigned gA = (unsigned)std::min<int64_t>(ceil_div((int64_t)na * 32, BLK), 148 * 8);
      for (int w = 0; w < 2; ++w) {  // sources (the widened box), then targets
        uint32_t *st = w == 0 ? src_start : tgt_start;
        std::vector<uint32_t> &hs = w == 0 ? hsrc : htgt;
        PYFOF_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * (na + 1), s));
        tl_chunk_kernel<<<gA, BLK, 0, s>>>(dH, dA, na, w == 0, cstart, cnt, nullptr, nullptr, 0);
        PYFOF_CHECK_LAUNCH();
        PYFOF_TRY(exclusive_scan_u32(cnt, st, na + 1, nullptr, W, s));
        hs.resize(na + 1);
        PYFOF_CUDA(cudaMemcpyAsync(hs.data(), st, sizeof(uint32_t) * (na + 1), cudaMemcpyDeviceToHost, s));
      }
      PYFOF_CUDA(cudaStreamSynchronize(s));
      src = W.carve<uint2>(std::max<uint32_t>(hsrc[na], 1));
      tgt = W.carve<uint2>(std::max<uint32_t>(htgt[na], 1));
      if (!src || !tgt) { set_error("workspace exhausted (two-level chunks)"); return kAlloc; }
      tl_chunk_kernel<<<gA, BLK, 0, s>>>(dH, dA, na, 1, cstart, cnt, src_start, src, 1);
      PYFOF_CHECK_LAUNCH();
      tl_chunk_kernel<<<gA, BLK, 0, s>>>(dH, dA, na, 0, cstart, cnt, tgt_start, tgt, 1);
      PYFOF_CHECK_LAUNCH();
      bool need2 = false, need4 = false;
      for (auto &Rg : act) { need2 |= Rg.r == 2; need4 |= Rg.r == 4; }
      if (need2) PYFOF_TRY(get_green<R>(ctx, 128, 3.5, 7.0, 0, &g_r2));
      if (need4) PYFOF_TRY(get_green<R>(ctx, 216, 3.5, 14.0, 0, &g_r4));
      R *self_in = W.carve<R>(M);
      if (!self_in) { set_error("workspace exhausted (two-level self)"); return kAlloc; }
      if (htgt[na] > 0) {
        tl_self_kernel<R><<<htgt[na], BLK, 0, s>>>(src4, dH, dA, na, tgt_start, tgt,
                                                   g_r2 ? (const R *)g_r2->self : nullptr,
                                                   g_r4 ? (const R *)g_r4->self : nullptr, self_in, ctx.d_flags);
        PYFOF_CHECK_LAUNCH();
      }
      tl_self_in = self_in;
    }
  }
  PYFOF_CUDA(cudaMemcpyAsync(ctx.h_flags, ctx.d_flags, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  PYFOF_CUDA(cudaStreamSynchronize(s));
  if (ctx.h_flags[FLAG_ERR]) {
    set_error("particle outside the PM source domain or non-finite grid coordinate");
    return ctx.h_flags[FLAG_ERR];
  }

  // One batch deposits and gathers grids of every class together, and runs
  // the convolutions of each class and transform length (a run) one after the
  // other.  The grids have an area each and the runs share one for their
  // spectra, both bounded by half the budget and reused by every pass.
  const size_t budget = std::max<size_t>(ctx.pm_budget / 2, 1);
  auto round256 = [](size_t b) { return (b + 255) & ~(size_t)255; };
  auto waves = [&](int n) { return a.tiles.conv_waves[kGridIndex(n)]; };
  auto run_cap = [&](int n) {
    const int cap = a.tiles.pm_batch[kGridIndex(n)];
    return (size_t)(cap > 0 ? std::min(cap, 65535) : 65535);
  };
  // the box of a halo's own grid, and of a region's inner grid: its sources
  // lie within 3.5 + 3/r grid cells of the region, its targets inside it
  // (tl_deposit_kernel, tl_gather_kernel), one node of slack each side
  auto halo_box = [&](int h) {
    ConvBox b{};
    for (int d = 0; d < 3; ++d) b.in[d] = b.out[d] = H[h].sup[d];
    return b;
  };
  auto region_box = [&](int ia) {
    const TlRegion &Rg = act[ia];
    ConvBox b{};
    for (int d = 0; d < 3; ++d) {
      b.in[d] = std::min(Rg.n_in / 2 + 1, (int)((16.0f + 2.0f * Rg.bo) * Rg.r + 1.0f) + 3);
      b.out0[d] = (int)(Rg.bo * Rg.r + 1.0f) - 2;
      b.out[d] = 16 * Rg.r + 5;
    }
    return b;
  };
  // bytes of a grid: the fixed-point deposit nodes (8 B each; the convolved
  // potential, R, is written back over them) and the half spectrum
  auto acc_bytes = [&](const ConvBox &b) {
    return round256(sizeof(unsigned long long) * b.in[0] * (size_t)b.in[1] * b.in[2]);
  };
  auto spec_bytes = [&](int n, const ConvBox &b) { return sizeof(cplx_t<R>) * (size_t)spec_elems<R>(n, b.in[2]); };
  // grids in batch order: class, length, boxes of similar size together (a
  // launch is shaped by the largest)
  struct Grid {
    ConvBox box;
    int32_t id, n, len;
  };
  auto order = [](std::vector<Grid> &g) {
    std::stable_sort(g.begin(), g.end(), [](const Grid &x, const Grid &y) {
      if (x.n != y.n) return x.n < y.n;
      if (x.len != y.len) return x.len < y.len;
      return (int64_t)x.box.in[1] * x.box.in[2] > (int64_t)y.box.in[1] * y.box.in[2];
    });
  };
  std::vector<Grid> hgrid, rgrid;
  for (int h = 0; h < nh; ++h) {
    const ConvBox b = halo_box(h);
    hgrid.push_back(Grid{b, h, H[h].n, green_of[H[h].n]->at(conv_length(H[h].n, sizeof(R) == 8, b))->n});
  }
  for (int ia = 0; ia < na; ++ia) {
    const ConvBox b = region_box(ia);
    const int n = act[ia].n_in;
    rgrid.push_back(Grid{b, ia, n, (n == 128 ? g_r2 : g_r4)->at(conv_length(n, sizeof(R) == 8, b))->n});
  }
  order(hgrid);
  order(rgrid);
  size_t acc_cap = 256, spec_cap = 256;
  for (const auto *gs : {&hgrid, &rgrid}) {
    size_t need = 0, largest = 0;
    for (size_t i = 0; i < gs->size(); ++i) {
      const size_t ab = acc_bytes((*gs)[i].box);
      need += ab;
      largest = std::max(largest, ab);
    }
    acc_cap = std::max(acc_cap, std::min(need, std::max(budget, largest)));
    for (size_t i = 0; i < gs->size();) {
      const Grid &g = (*gs)[i];
      std::vector<size_t> sizes;
      for (; i < gs->size() && (*gs)[i].n == g.n && (*gs)[i].len == g.len; ++i)
        sizes.push_back(spec_bytes(g.len, (*gs)[i].box));
      std::sort(sizes.begin(), sizes.end(), std::greater<size_t>());
      size_t sum = 0;
      for (size_t j = 0; j < sizes.size() && j < run_cap(g.n); ++j) sum += sizes[j];
      spec_cap = std::max(spec_cap, std::min(sum, std::max(budget, sizes[0])));
    }
  }
  acc_cap = round256(acc_cap);
  const size_t scratch_bytes = acc_cap + spec_cap;
  const int64_t nbat = std::max<int64_t>(nh, na);
  unsigned char *scratch = W.carve<unsigned char>(scratch_bytes);
  int32_t *dpend = W.carve<int32_t>(nh);
  // a batch's tables, uploaded together: boxes, ids, member prefixes
  unsigned char *dmeta = W.carve<unsigned char>((size_t)nbat * (sizeof(ConvBox) + 12) + 64);
  double *dinv = W.carve<double>(nbat);
  if (!scratch || !dpend || !dmeta || !dinv) {
    set_error("workspace exhausted (PM grids)");
    return kAlloc;
  }
  struct Run {  // grids [first, first + count) of a batch
    int n, len, first, count;
    ConvExtent ext;
  };
  struct Batch {
    std::vector<int32_t> ids;
    std::vector<ConvBox> boxes;
    std::vector<Run> runs;
    size_t acc = 0;  // bytes
    const ConvBox *dbox;
    const int32_t *did;
    const uint32_t *dpre0, *dpre1;
    uint32_t n0, n1;  // chunks of sources and of targets (the same for a halo's own grid)
  };
  // takes grids from items[at..] while they fit, and uploads the tables
  std::vector<unsigned char> meta;
  auto next_batch = [&](const std::vector<const Grid *> &items, size_t &at, bool region, Batch &B) -> int32_t {
    B = Batch();
    std::vector<uint32_t> p0(1, 0), p1(1, 0);
    size_t spec = 0;
    for (; at < items.size(); ++at) {
      const Grid &g = *items[at];
      ConvBox b = g.box;
      const size_t ab = acc_bytes(b), sb = spec_bytes(g.len, b);
      if (!B.ids.empty() && B.acc + ab > acc_cap) break;
      if (B.runs.empty() || B.runs.back().n != g.n || B.runs.back().len != g.len || spec + sb > spec_cap ||
          (size_t)B.runs.back().count >= run_cap(g.n)) {
        B.runs.push_back(Run{g.n, g.len, (int)B.ids.size(), 0, ConvExtent()});
        spec = 0;
      }
      b.in_off = (int64_t)(B.acc / sizeof(unsigned long long));
      b.out_off = (int64_t)(B.acc / sizeof(R));
      b.spec_off = (int64_t)(spec / sizeof(cplx_t<R>));
      B.acc += ab;
      spec += sb;
      B.runs.back().ext.add(b);
      ++B.runs.back().count;
      ctx.last_pm_fft_bytes += conv_bytes<R>(g.len, b);
      B.ids.push_back(g.id);
      B.boxes.push_back(b);
      if (region) {
        p0.push_back(p0.back() + (hsrc[g.id + 1] - hsrc[g.id]));
        p1.push_back(p1.back() + (htgt[g.id + 1] - htgt[g.id]));
      } else {
        p0.push_back(p0.back() + (uint32_t)ceil_div(H[g.id].np, kDepChunk));
      }
    }
    const size_t nb = B.ids.size(), ob = sizeof(ConvBox) * nb, oi = ob + 4 * nb, op = oi + 4 * (nb + 1);
    meta.resize(op + (region ? 4 * (nb + 1) : 0));
    std::memcpy(meta.data(), B.boxes.data(), ob);
    std::memcpy(meta.data() + ob, B.ids.data(), 4 * nb);
    std::memcpy(meta.data() + oi, p0.data(), 4 * (nb + 1));
    if (region) std::memcpy(meta.data() + op, p1.data(), 4 * (nb + 1));
    PYFOF_TRY(upload(ctx, dmeta, meta.data(), meta.size(), s));
    B.dbox = reinterpret_cast<const ConvBox *>(dmeta);
    B.did = reinterpret_cast<const int32_t *>(dmeta + ob);
    B.dpre0 = reinterpret_cast<const uint32_t *>(dmeta + oi);
    B.dpre1 = region ? reinterpret_cast<const uint32_t *>(dmeta + op) : B.dpre0;
    B.n0 = p0.back();
    B.n1 = region ? p1.back() : p0.back();
    ctx.last_pm_solves += (int64_t)nb;
    PYFOF_CUDA(cudaMemsetAsync(scratch, 0, B.acc, s));
    return kOk;
  };
  unsigned long long *const acc = reinterpret_cast<unsigned long long *>(scratch);
  R *const rho = reinterpret_cast<R *>(scratch);  // the convolved grids overwrite acc
  auto convolve = [&](const Batch &B, auto &&table) -> int32_t {
    if (ctx.timing) ctx.conv_timer.begin(s);
    for (const Run &r : B.runs) {
      const GreenTable *g = table(r.n)->at(r.len);
      PYFOF_TRY(pm_convolve_batch<R>(acc, dinv + r.first, rho, reinterpret_cast<cplx_t<R> *>(scratch + acc_cap),
                                     (const R *)g->g, (const cplx_t<R> *)g->tw, r.len, B.dbox + r.first, r.ext,
                                     r.count, g->scaled, s, waves(r.n)));
    }
    if (ctx.timing) ctx.conv_timer.end(s);
    return kOk;
  };
  // halos above kBigNp members: chunked removal loop
  std::vector<BigHalo> hbig;
  std::vector<BigChunk> hch;
  std::vector<char> is_big(nh, 0);
  int64_t ubig = 0;
  for (int h = 0; h < nh; ++h) {
    if (H[h].np <= (a.big_np > 0 ? a.big_np : kBigNp)) continue;
    is_big[h] = 1;
    BigHalo bh{};
    bh.h = h;
    bh.off = H[h].off;
    bh.np = H[h].np;
    bh.uoff = ubig;
    bh.chunk0 = (int32_t)hch.size();
    for (int64_t st0 = 0; st0 < bh.np; st0 += kChunk)
      hch.push_back(BigChunk{(int32_t)hbig.size(), bh.off + st0, bh.off + std::min<int64_t>(bh.np, st0 + kChunk)});
    bh.nchunk = (int32_t)hch.size() - bh.chunk0;
    ubig += bh.np;
    hbig.push_back(bh);
  }
  const int nbig = (int)hbig.size(), nchb = (int)hch.size();
  BigHalo *dB = nullptr;
  BigChunk *dCh = nullptr;
  double *bpart = nullptr;
  int32_t *bucount = nullptr;
  unsigned long long *bulist = nullptr;
  int32_t *nactive = ctx.d_flags + FLAG_COUNT_B;
  if (nbig) {
    dB = W.carve<BigHalo>(nbig);
    dCh = W.carve<BigChunk>(nchb);
    bpart = W.carve<double>(7 * (size_t)nchb);
    bucount = W.carve<int32_t>(nbig);
    bulist = W.carve<unsigned long long>(ubig);
    if (!dB || !dCh || !bpart || !bucount || !bulist) {
      set_error("workspace exhausted (large halos)");
      return kAlloc;
    }
    PYFOF_TRY(upload(ctx, dB, hbig.data(), sizeof(BigHalo) * nbig, s));
    PYFOF_TRY(upload(ctx, dCh, hch.data(), sizeof(BigChunk) * nchb, s));
  }
  for (int pass = 1; pass <= kMaxPasses; ++pass) {
    std::vector<int32_t> pend;
    for (int h = 0; h < nh; ++h) if (H[h].pending) pend.push_back(h);
    if (pend.empty()) break;
    std::vector<int32_t> pend_small;
    for (int h : pend) if (!is_big[h]) pend_small.push_back(h);
    ++ctx.last_pm_passes;
    if (ctx.timing && pass > 1) ctx.gap_timer.end(s);
    if (!pend_small.empty()) {
      PYFOF_TRY(upload(ctx, dpend, pend_small.data(), sizeof(int32_t) * pend_small.size(), s));
      pm_mkeep_kernel<<<(unsigned)pend_small.size(), 256, 0, s>>>(m, dH, dpend, (int)pend_small.size(), keep);
      PYFOF_CHECK_LAUNCH();
    }
    if (nbig) {
      big_mass_kernel<<<nchb, 256, 0, s>>>(m, dCh, dB, dH, keep, bpart);
      PYFOF_CHECK_LAUNCH();
      big_mass_sum_kernel<<<(unsigned)ceil_div(nbig, 128), 128, 0, s>>>(dB, nbig, bpart, dH);
      PYFOF_CHECK_LAUNCH();
    }
    Batch B;
    std::vector<const Grid *> todo;
    for (const Grid &g : hgrid)
      if (H[g.id].pending) todo.push_back(&g);
    for (size_t at = 0; at < todo.size();) {
      PYFOF_TRY(next_batch(todo, at, false, B));
      const int nb = (int)B.ids.size();
      pm_deposit_kernel<<<B.n0, BLK, 0, s>>>(src4, cmem, dH, B.dbox, B.did, B.dpre0, nb, keep, acc, dinv);
      PYFOF_CHECK_LAUNCH();
      PYFOF_TRY(convolve(B, [&](int n) { return green_of[n].get(); }));
      pm_gather_kernel<R><<<B.n0, BLK, 0, s>>>(src4, cmem, dH, B.dbox, B.did, B.dpre0, nb, keep, selfe, rho,
                                               a.a_val, c1);
      PYFOF_CHECK_LAUNCH();
    }
    // refined regions of pending halos
    todo.clear();
    for (const Grid &g : rgrid)
      if (H[act[g.id].h].pending) todo.push_back(&g);
    for (size_t at = 0; at < todo.size();) {
      PYFOF_TRY(next_batch(todo, at, true, B));
      const int nb = (int)B.ids.size();
      tl_deposit_kernel<<<B.n0, BLK, 0, s>>>(src4, cmem, dH, dA, B.dbox, B.did, B.dpre0, nb, src_start, src, keep,
                                             acc, dinv);
      PYFOF_CHECK_LAUNCH();
      PYFOF_TRY(convolve(B, [&](int n) { return (n == 128 ? g_r2 : g_r4).get(); }));
      if (B.n1 > 0) {
        tl_gather_kernel<R><<<B.n1, BLK, 0, s>>>(src4, cmem, dH, dA, B.dbox, B.did, B.dpre1, nb, tgt_start, tgt,
                                                 keep, tl_self_in, rho, a.a_val, phi_in);
        PYFOF_CHECK_LAUNCH();
      }
    }
    PYFOF_CUDA(cudaMemsetAsync(sr_next, 0, 2 * sizeof(unsigned), s));
    if (pass == 1) {
      sr_gather_kernel<R, false><<<gS, 32 * kSrWarps, 0, s>>>(dH, keep, pr, chunks, nchunk, sr_next + 2, cstart,
                                                              cmem, src4, nullptr, nullptr, splines, a.a_val,
                                                              a.softening, c2, sr_next);
      PYFOF_CHECK_LAUNCH();
    } else {
      PYFOF_TRY(exclusive_scan_u32(rflag, rpos, (int64_t)npm + 1, nullptr, W, s));
      sr_removed_fill_kernel<<<gP, BLK, 0, s>>>(rflag, rpos, npm, rsrc);
      PYFOF_CHECK_LAUNCH();
      sr_gather_kernel<R, true><<<gS, 32 * kSrWarps, 0, s>>>(dH, keep, pr, chunks, nchunk, sr_next + 2, cstart,
                                                             cmem, src4, rpos, rsrc, splines, a.a_val, a.softening,
                                                             c2, sr_next);
      PYFOF_CHECK_LAUNCH();
    }
    if (!pend_small.empty()) {
      PYFOF_CUDA(wait_velocities(ctx, s));
      pm_inner_kernel<R><<<(unsigned)pend_small.size(), IBLK, 0, s>>>(m, dH, dpend, (int)pend_small.size(), keep,
                                                                     epos, rflag, c1, phi_in, c2, phi, en,
                                                                     (float)a.b_val, a.np_halo_min, phi_only,
                                                                     ctx.d_flags);
      PYFOF_CHECK_LAUNCH();
    }
    if (nbig) PYFOF_TRY(big_removal<R>(ctx, m, dB, nbig, dCh, nchb, dH, keep, epos, rflag, c1, phi_in, c2, phi, bpart,
                                       bucount, bulist, nactive, (float)a.b_val, a.np_halo_min, phi_only));
    if (ctx.timing) ctx.gap_timer.begin(s);
    PYFOF_CUDA(cudaMemcpyAsync(H.data(), dH, sizeof(PmHalo) * nh, cudaMemcpyDeviceToHost, s));
    PYFOF_CUDA(cudaMemcpyAsync(ctx.h_flags, ctx.d_flags, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    PYFOF_CUDA(cudaStreamSynchronize(s));
    if (ctx.timing) ctx.conv_timer.collect();
    if (ctx.h_flags[FLAG_ERR]) {
      set_error("particle-mesh unbinding failed (error %d)", ctx.h_flags[FLAG_ERR]);
      return ctx.h_flags[FLAG_ERR];
    }
  }
  pm_result_kernel<<<(unsigned)ceil_div(nh, 128), 128, 0, s>>>(dH, dlist, nh, res);
  PYFOF_CHECK_LAUNCH();
  if (phi_out) PYFOF_CUDA(cudaMemcpyAsync(phi_out, phi, sizeof(float) * M, cudaMemcpyDeviceToDevice, s));
  PYFOF_CUDA(cudaStreamSynchronize(s));
  return kOk;
}

}  // namespace

int32_t unbind_pm(Context &ctx, const FofArgs &a, const GridRules &rules, const Members &m,
                  const std::vector<HaloTask> &tasks, const std::vector<int32_t> &list,
                  HaloResult *res, uint8_t *keep, float *phi_out, int phi_only) {
  if (a.bound_fp64 || a.bound_per_halo) return run_pm<double>(ctx, a, rules, m, tasks, list, res, keep, phi_out, phi_only);
  return run_pm<float>(ctx, a, rules, m, tasks, list, res, keep, phi_out, phi_only);
}

}  // namespace pyfof
