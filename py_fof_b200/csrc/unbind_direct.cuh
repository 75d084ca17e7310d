// Direct-summation solver of the unbinding removal loop (bound_check_grid
// for gid 0, bound_fortran.f90:2611-2864), shared by the batched stage
// (unbind.cu) and the static-scratch entry point (direct_static.cu).
#pragma once

#include "unbind_internal.cuh"

namespace pyfof {
namespace direct {

constexpr int BLK = 256;

// bound_depth_continuous (bound_fortran.f90:3080-3102): spline-softened 1/r.
template <typename T>
__device__ __forceinline__ T depth_continuous(T r, T h);

template <>
__device__ __forceinline__ double depth_continuous<double>(double r, double h) {
  if (r <= 0.0) return __ddiv_rn(208.0, __dmul_rn(70.0, h));
  if (r >= h) return __ddiv_rn(1.0, r);
  const double e = __ddiv_rn(__dmul_rn(2.0, r), h);
  if (e <= 1.0) {
    double t = __dadd_rn(8.0, __dmul_rn(-3.0, e));
    t = __dadd_rn(14.0, __dmul_rn(e, t));
    t = __dadd_rn(-56.0, __dmul_rn(e, t));
    t = __dadd_rn(112.0, __dmul_rn(__dmul_rn(e, e), t));
    const double prim = __dmul_rn(__dmul_rn(e, e), t);
    return __ddiv_rn(__dadd_rn(208.0, -prim), __dmul_rn(70.0, h));
  }
  double t = __dadd_rn(-8.0, e);
  t = __dadd_rn(14.0, __dmul_rn(e, t));
  t = __dadd_rn(56.0, __dmul_rn(e, t));
  t = __dadd_rn(-280.0, __dmul_rn(e, t));
  t = __dadd_rn(448.0, __dmul_rn(e, t));
  double prim = __dmul_rn(__dmul_rn(e, e), t);
  prim = __dadd_rn(prim, -__dmul_rn(224.0, e));
  prim = __dadd_rn(prim, -__ddiv_rn(12.0, e));
  return __ddiv_rn(__dadd_rn(128.0, -prim), __dmul_rn(70.0, h));
}

// FP32 product-path kernel: same piecewise polynomial, with the
// reciprocals precomputed by the caller (inv70h = 1/(70h), inv_h = 1/h).
__device__ __forceinline__ float depth_f32(float r2, float h, float inv_h, float inv70h) {
  if (r2 >= h * h) return rsqrtf(r2);
  const float r = sqrtf(r2);
  const float e = 2.0f * r * inv_h;
  if (e <= 1.0f) {
    const float e2 = e * e;
    const float prim = e2 * (112.0f + e2 * (-56.0f + e * (14.0f + e * (8.0f - 3.0f * e))));
    return (208.0f - prim) * inv70h;
  }
  const float prim = e * e * (448.0f + e * (-280.0f + e * (56.0f + e * (14.0f + e * (-8.0f + e))))) -
                     224.0f * e - 12.0f / e;
  return (128.0f - prim) * inv70h;
}

// Compensated (Fast2Sum/Kahan) FP32 accumulator.
struct Kahan {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
};

__device__ __forceinline__ int block_sum_i(int v, int *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  int t = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
  return t;
}

struct DirectParams {
  double fac;     // a / (6 pi)
  double app;     // softening (standard grid units)
  float b;        // real(b_bound, 4)
  int nmin;       // np_halo_min
  int phi_only;   // stop after the first potential
};

// One FP64 pair term of the first pass, -(w_j * fac D(r)), with the
// reference's operations (bound_fortran.f90:2619-2640).
__device__ __forceinline__ double pair_depth64(float xj, float yj, float zj, float xi, float yi, float zi, double app) {
  const double dx = (double)__fsub_rn(xj, xi);
  const double dy = (double)__fsub_rn(yj, yi);
  const double dz = (double)__fsub_rn(zj, zi);
  const double r = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
  return depth_continuous<double>(r, app);
}

// Adds the terms t of a group of G lanes to acc in lane order, the same on
// every lane of the group: a serial sum whose terms were computed in parallel.
template <int G>
__device__ __forceinline__ void add_in_order(double &acc, double t, int n, unsigned group) {
  if constexpr (G == 1) {
    acc = __dadd_rn(acc, t);
  } else {
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const double v = __shfl_sync(group, t, u, G);
      if (u < n) acc = __dadd_rn(acc, v);
    }
  }
}

// The first-pass potentials of many direct-summation halos, spread over the
// whole GPU: block b takes the kPhi1Targets<G> targets tiles[b] = (entry of list, first
// target) of one halo and streams the halo's members through shared memory
// in ascending order.  Each target adds its sources in ascending index,
// skipping itself: the reference's accumulation order (bound_fortran.f90:
// 2619-2640; its i<j loop adds each pair term to both ends) with the
// operations of the in-kernel first pass of ub_direct_kernel, so the results
// are the same bits; the removal loop then starts from phi1.
// G lanes share a target: they compute G terms at once and add them in order
// (add_in_order).  An FP64 term is a square root and a division in one
// dependent chain per target, so a few targets (fewer than the chip has
// thread slots) are latency-bound and take G = 8: a halo of 450 members takes
// 41 us, with a lane per target 184.  With more targets the chains hide one
// another and the ordered adds are only extra work, so G = 1: 20,000 halos of
// 20 to 1000 members 2.6 ms, with eight lanes 3.7.  FP32 terms are as short
// as the ordered adds: always G = 1.
constexpr int kPhi1Lanes = 8;
template <int G>
constexpr int kPhi1Targets = G == 1 ? 64 : 32;
template <bool FP64, int G>
__global__ void __launch_bounds__(kPhi1Targets<G> * G) ub_direct_phi1_kernel(
    Members m, const int64_t *__restrict__ off, const int32_t *__restrict__ list, const int2 *__restrict__ tiles,
    DirectParams P, double *__restrict__ phi1) {
  constexpr int NT = kPhi1Targets<G> * G;
  __shared__ float4 src[NT];
  const int2 t = tiles[blockIdx.x];
  const int c = list[t.x];
  const int64_t b0 = off[c];
  const int np = (int)(off[c + 1] - b0);
  const int i = t.y + threadIdx.x / G, gl = threadIdx.x % G;
  const bool act = i < np;
  const unsigned group = G == 1 ? 0u : ((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1));
  const float xi = act ? m.q[0][b0 + i] : 0.f, yi = act ? m.q[1][b0 + i] : 0.f,
              zi = act ? m.q[2][b0 + i] : 0.f;
  const float h32 = (float)P.app, inv_h = (float)(1.0 / P.app), inv70h = (float)(1.0 / (70.0 * P.app));
  double acc64 = 0.0;
  Kahan acc32;
  for (int j0 = 0; j0 < np; j0 += NT) {
    const int j = j0 + threadIdx.x;
    __syncthreads();
    if (j < np) src[threadIdx.x] = make_float4(m.q[0][b0 + j], m.q[1][b0 + j], m.q[2][b0 + j], m.w[b0 + j]);
    __syncthreads();
    const int cnt = min(NT, np - j0);
    if (FP64) {
      if (act)
        for (int k0 = 0; k0 < cnt; k0 += G) {
          const int k = k0 + gl;
          double v = 0.0;  // adding +0 leaves the sum as it is: the target itself
          if (k < cnt && j0 + k != i) {
            const float4 s = src[k];
            v = -__dmul_rn((double)s.w, __dmul_rn(P.fac, pair_depth64(s.x, s.y, s.z, xi, yi, zi, P.app)));
          }
          add_in_order<G>(acc64, v, cnt - k0, group);
        }
    } else if (act) {
      for (int k = 0; k < cnt; ++k) {
        if (j0 + k == i) continue;
        const float4 s = src[k];
        const float dx = s.x - xi, dy = s.y - yi, dz = s.z - zi;
        acc32.add(-s.w * depth_f32(dx * dx + dy * dy + dz * dz, h32, inv_h, inv70h));
      }
    }
  }
  if (act && gl == 0) phi1[b0 + i] = FP64 ? acc64 : (double)((float)P.fac * acc32.s);
}

// Dynamic shared memory of ub_direct_kernel for halos of up to cap members
// (cap a multiple of 32): eight float arrays and one int array, two 64-bit
// arrays and the keep flags.
__host__ __device__ constexpr size_t direct_smem(int cap) { return (size_t)cap * (11 * 4 + 8 + 1); }

// One block of NT threads per halo: bound_check_grid for gid 0
// (:2611-2864).  FP64=true is the plain FP64 path, bit-exact with the
// reference arithmetic; FP64=false the FP32 product path with compensated
// sums.  phi1 (optional): the first-pass potentials from
// ub_direct_phi1_kernel; null computes them here.  Every halo of the launch
// has at most cap members.  No result depends on NT: every sum is the one of
// an order fixed by the member indices alone (per-target serial sums; for the
// centre sums see s_amax below).
//
// One block per halo is a chain of short steps, so what counts is their
// latency.  The centre sums in their fixed order cost one dependent add per
// member and iteration (8 ms of a 128^3 box for its largest halos); here the
// block sums them in parallel, bounds the distance to the ordered sums, and
// runs the ordered sums only if that bound leaves the FP32 centre open.  The
// refresh of the potential shares a target among eight lanes as
// ub_direct_phi1_kernel does, and the removal order is a count over 64-bit
// keys (energy, then index).
template <bool FP64, int NT = BLK>
__global__ void __launch_bounds__(NT) ub_direct_kernel(Members m, const int64_t *__restrict__ off,
                                                       const int32_t *__restrict__ list,
                                                       DirectParams P, HaloResult *__restrict__ res,
                                                       uint8_t *__restrict__ keep_out,
                                                       float *__restrict__ phi_out,
                                                       int32_t *flags,
                                                       const double *__restrict__ phi1 = nullptr,
                                                       int cap = kDirectMax) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int c = list[blockIdx.x];
  const int64_t b0 = off[c];
  const int np = (int)(off[c + 1] - b0);
  float *qx = reinterpret_cast<float *>(smem);
  float *qy = qx + cap, *qz = qy + cap;
  float *vx = qz + cap, *vy = vx + cap, *vz = vy + cap;
  float *w = vz + cap, *phi = w + cap;
  int *jdel = reinterpret_cast<int *>(phi + cap);
  // unbound members: bits of E (E >= 0, so they order like E) over ~index, so
  // that a larger key is removed first (equal energies: lower index first)
  unsigned long long *ukey = reinterpret_cast<unsigned long long *>(jdel + cap);
  double *phid = reinterpret_cast<double *>(ukey + cap);
  unsigned char *keep = reinterpret_cast<unsigned char *>(phid + cap);
  constexpr int G = FP64 ? kPhi1Lanes : 1;
  __shared__ int red_i[NT / 32];
  __shared__ double red_d[7][NT / 32];
  __shared__ double s_sum[7];
  __shared__ float s_c[6];          // centre and mean velocity
  __shared__ unsigned s_amax[6];    // largest |component| of q and v over the members
  __shared__ int s_nu, s_err, s_open;

  if (threadIdx.x < 6) s_amax[threadIdx.x] = 0;
  __syncthreads();
  float am[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int i = threadIdx.x; i < np; i += NT) {
    const int64_t k = b0 + i;
    qx[i] = m.q[0][k]; qy[i] = m.q[1][k]; qz[i] = m.q[2][k];
    vx[i] = m.v[0][k]; vy[i] = m.v[1][k]; vz[i] = m.v[2][k];
    w[i] = m.w[k];
    keep[i] = 1;
    phid[i] = 0.0;
    const float v6[6] = {qx[i], qy[i], qz[i], vx[i], vy[i], vz[i]};
#pragma unroll
    for (int d = 0; d < 6; ++d) am[d] = fmaxf(am[d], fabsf(v6[d]));
  }
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    const unsigned o = __reduce_max_sync(0xffffffffu, __float_as_uint(am[d]));
    if ((threadIdx.x & 31) == 0) atomicMax(&s_amax[d], o);
  }
  if (threadIdx.x == 0) s_err = 0;
  __syncthreads();
  const float h32 = (float)P.app, inv_h = (float)(1.0 / P.app), inv70h = (float)(1.0 / (70.0 * P.app));
  const float fac32 = (float)P.fac;
  int np_bound = np, njd = 0, status = 5;

  for (int pass = 1; pass <= kMaxPasses; ++pass) {
    int ks = 0;
    for (int i = threadIdx.x; i < np; i += NT) ks += keep[i];
    const int n_source = block_sum_i(ks, red_i);
    // potential: full sum on the first pass, later passes add back the
    // sources removed since the previous refresh, in removal order; G lanes
    // per target (the same targets for every lane of a group)
    const int gl = threadIdx.x % G;
    const unsigned group = G == 1 ? 0u : ((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1));
    for (int i = threadIdx.x / G; i < np; i += NT / G) {
      if (pass == 1 && phi1) {
        if (gl == 0) phid[i] = phi1[b0 + i];
      } else if (FP64 && (pass == 1 || keep[i])) {
        const float xi = qx[i], yi = qy[i], zi = qz[i];
        const int nk = pass == 1 ? np : njd;
        double acc = pass == 1 ? 0.0 : phid[i];
        for (int k0 = 0; k0 < nk; k0 += G) {
          const int k = k0 + gl;
          double v = 0.0;
          if (pass == 1) {
            if (k < nk && k != i)
              v = -__dmul_rn((double)w[k], __dmul_rn(P.fac, pair_depth64(qx[k], qy[k], qz[k], xi, yi, zi, P.app)));
          } else if (k < nk) {
            const int j = jdel[k];
            v = __dmul_rn(__dmul_rn((double)w[j], P.fac), pair_depth64(qx[j], qy[j], qz[j], xi, yi, zi, P.app));
          }
          add_in_order<G>(acc, v, nk - k0, group);
        }
        __syncwarp(group);  // every lane has read phid[i]
        if (gl == 0) phid[i] = acc;
      } else if (!FP64 && (pass == 1 || keep[i])) {
        Kahan acc;
        const float xi = qx[i], yi = qy[i], zi = qz[i];
        const int nk = pass == 1 ? np : njd;
        for (int k = 0; k < nk; ++k) {
          const int j = pass == 1 ? k : jdel[k];
          if (pass == 1 && j == i) continue;
          const float dx = qx[j] - xi, dy = qy[j] - yi, dz = qz[j] - zi;
          const float t = w[j] * depth_f32(dx * dx + dy * dy + dz * dz, h32, inv_h, inv70h);
          acc.add(pass == 1 ? -t : t);
        }
        phid[i] = (pass == 1 ? 0.0 : phid[i]) + (double)(fac32 * acc.s);
      }
    }
    __syncthreads();
    njd = 0;
    for (int i = threadIdx.x; i < np; i += NT) {
      if (!keep[i]) continue;
      float v = FP64 ? __double2float_rn(phid[i]) : (float)phid[i];
      if (np_bound == 1 || n_source == 1) v = 0.0f;
      if (!isfinite(v)) s_err = kNonFinite;
      phi[i] = v;
    }
    __syncthreads();
    if (s_err) break;
    if (P.phi_only) { status = 0; break; }
    int deleted = 0;
    for (;;) {
      // centre of mass and mean velocity of the kept set.  The FP64 sums of
      // w, w q and w v over n members in two orders, here this block's and
      // the fixed one, differ by at most 2 (n-1) u sum |terms| (u = 2^-53), and
      // sum |w x| <= max |x| sum w; so the two quotients differ by less than
      // err = 5 (n + 4) u max |x|.  If q - err and q + err round to the same
      // FP32 value, that is the fixed order's; if not (about one iteration in
      // a hundred), the sums are run in the fixed order.
      {
        double a[7] = {0, 0, 0, 0, 0, 0, 0};
        for (int i = threadIdx.x; i < np; i += NT) {
          if (!keep[i]) continue;
          const double wi = (double)w[i];
          a[0] += wi;
          a[1] += wi * (double)qx[i]; a[2] += wi * (double)qy[i]; a[3] += wi * (double)qz[i];
          a[4] += wi * (double)vx[i]; a[5] += wi * (double)vy[i]; a[6] += wi * (double)vz[i];
        }
#pragma unroll
        for (int k = 0; k < 7; ++k)
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
        if ((threadIdx.x & 31) == 0)
#pragma unroll
          for (int k = 0; k < 7; ++k) red_d[k][threadIdx.x >> 5] = a[k];
        if (threadIdx.x == 0) s_nu = 0;
        __syncthreads();
        if (threadIdx.x < 32) {
          double v = 0.0;
          if (threadIdx.x < 7)
#pragma unroll
            for (int u = 0; u < NT / 32; ++u) v += red_d[threadIdx.x][u];
          const double ws = __shfl_sync(0xffffffffu, v, 0);
          bool open = false;
          if (threadIdx.x >= 1 && threadIdx.x < 7) {
            const double q = v / ws;
            const double err = 5.0 * (double)(np + 4) * 1.1102230246251566e-16 *
                               (double)__uint_as_float(s_amax[threadIdx.x - 1]);
            const float lo = __double2float_rn(q - err), hi = __double2float_rn(q + err);
            open = !(lo == hi);
            s_c[threadIdx.x - 1] = hi;
          }
          open = __any_sync(0xffffffffu, open);
          if (threadIdx.x == 0) s_open = open;
        }
        __syncthreads();
      }
      if (s_open) {
        if (FP64) {
          // seven sequential sums in ascending index (the reference's order),
          // one per lane of warp 0
          if (threadIdx.x < 7) {
            const int qi = threadIdx.x;
            const float *src = qi == 1 ? qx : qi == 2 ? qy : qi == 3 ? qz : qi == 4 ? vx : qi == 5 ? vy : vz;
            double acc = 0.0;
#pragma unroll 4
            for (int i = 0; i < np; ++i) {
              if (!keep[i]) continue;
              const double wi = (double)w[i];
              acc = __dadd_rn(acc, qi == 0 ? wi : __dmul_rn(wi, (double)src[i]));
            }
            s_sum[qi] = acc;
          }
        } else if (threadIdx.x < 32) {
          // warp 0: lane l sums the members l, l+32, ...; then a butterfly
          double a[7] = {0, 0, 0, 0, 0, 0, 0};
          for (int i = threadIdx.x; i < np; i += 32) {
            if (!keep[i]) continue;
            const double wi = (double)w[i];
            a[0] += wi;
            a[1] += wi * qx[i]; a[2] += wi * qy[i]; a[3] += wi * qz[i];
            a[4] += wi * vx[i]; a[5] += wi * vy[i]; a[6] += wi * vz[i];
          }
          for (int k = 0; k < 7; ++k)
            for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
          if (threadIdx.x == 0)
            for (int k = 0; k < 7; ++k) s_sum[k] = a[k];
        }
        __syncthreads();
        if (threadIdx.x < 6) s_c[threadIdx.x] = __double2float_rn(__ddiv_rn(s_sum[1 + threadIdx.x], s_sum[0]));
        __syncthreads();
      }
      const float qc0 = s_c[0], qc1 = s_c[1], qc2 = s_c[2], vc0 = s_c[3], vc1 = s_c[4], vc2 = s_c[5];
      // specific energies (bound_fortran.f90:2773-2786), FP32
      for (int i = threadIdx.x; i < np; i += NT) {
        if (!keep[i]) continue;
        const float d0 = __fadd_rn(__fsub_rn(vx[i], vc0), __fmul_rn(P.b, __fsub_rn(qx[i], qc0)));
        const float d1 = __fadd_rn(__fsub_rn(vy[i], vc1), __fmul_rn(P.b, __fsub_rn(qy[i], qc1)));
        const float d2 = __fadd_rn(__fsub_rn(vz[i], vc2), __fmul_rn(P.b, __fsub_rn(qz[i], qc2)));
        float s = __fmul_rn(d0, d0);
        s = __fadd_rn(s, __fmul_rn(d1, d1));
        s = __fadd_rn(s, __fmul_rn(d2, d2));
        const float e = __fadd_rn(__fdiv_rn(s, 2.0f), phi[i]);
        if (!isfinite(e)) s_err = kInvalid;
        if (e >= 0.0f)
          ukey[atomicAdd(&s_nu, 1)] =
              ((unsigned long long)__float_as_uint(e + 0.0f) << 32) | (0xffffffffu - (unsigned)i);
      }
      __syncthreads();
      if (s_err) break;
      const int nu = s_nu;
      if (nu == 0) {
        if (deleted == 0) { status = 0; break; }
        break;
      }
      // delete the nb highest energies; ties go to the lower local index
      // first (bound_fortran.f90:2808-2844)
      int nb = (int)ceil(0.02 * (double)np_bound);
      nb = max(1, nb);
      nb = min(nu, nb);
      for (int t = threadIdx.x; t < nu; t += NT) {
        const unsigned long long key = ukey[t];
        int rank = 0;
#pragma unroll 8
        for (int u = 0; u < nu; ++u) rank += ukey[u] > key;
        if (rank < nb) {
          const int i = (int)(0xffffffffu - (unsigned)key);
          keep[i] = 0;
          jdel[njd + rank] = i;
        }
      }
      __syncthreads();
      njd += nb;
      np_bound -= nb;
      deleted += nb;
      if (np_bound < P.nmin) { status = 1; break; }
      if ((double)deleted >= 0.2 * (double)np_bound) break;
    }
    __syncthreads();
    if (s_err || status != 5) break;
    if (pass == kMaxPasses) break;
  }
  if (s_err) {
    if (threadIdx.x == 0) atomicCAS(&flags[FLAG_ERR], 0, s_err);
    return;
  }
  for (int i = threadIdx.x; i < np; i += NT) {
    keep_out[b0 + i] = keep[i];
    if (phi_out) phi_out[b0 + i] = phi[i];
  }
  if (threadIdx.x == 0) {
    res[c].status = status;
    res[c].np_bound = np_bound;
  }
}

}  // namespace direct
}  // namespace pyfof
