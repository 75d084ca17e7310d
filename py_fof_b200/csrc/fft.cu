// Batched zero-padded 3-D FFT convolution for the particle-mesh solver.
// See fft.cuh for layouts.
//
// Every line transform of length N = N1 * N2 runs as two register-resident
// DFTs with one shared-memory exchange between them (Cooley-Tukey with the
// input index e = s + N2 q and the output index k = k1 + N1 k2):
//   stage A  thread (line, s):  Y[s][k1] = sum_q x[s + N2 q] W_N1^(q k1),
//            times the twiddle W_N^(s k1), written to shared memory;
//   stage B  thread (line, k1): X[k1 + N1 k2] = sum_s Y[s][k1] W_N2^(s k2).
// The register DFTs are mixed-radix (4, 2, 3, 5) decompositions unrolled at
// compile time with constant twiddles.  A block works on a tile of W lines
// that are adjacent in memory (consecutive kx), so every global access of a
// warp covers whole 128-byte segments.  The z pass does forward transform,
// Green multiplication and inverse transform in one kernel (stage B holds a
// full frequency line per thread; the inverse walks the same stages back),
// and loops over the halos of a batch with the Green values held in
// registers, so the table is read once per block.
#include <utility>

#include "fft.cuh"
#include "per_device.cuh"

namespace pyfof {

namespace {

// ------------------------------------------------------------ compile time

template <class F, int... I>
__device__ __forceinline__ void sfor_impl(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void sfor(F &&f) {
  sfor_impl(static_cast<F &&>(f), std::make_integer_sequence<int, N>{});
}

constexpr double kQuarterPi = 0.785398163397448309615660845819875721;

__host__ __device__ constexpr double taylor_sin(double x) {
  double x2 = x * x, term = x, sum = x;
  for (int k = 1; k < 12; ++k) {
    term *= -x2 / (double)((2 * k) * (2 * k + 1));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double taylor_cos(double x) {
  double x2 = x * x, term = 1.0, sum = 1.0;
  for (int k = 1; k < 12; ++k) {
    term *= -x2 / (double)((2 * k - 1) * (2 * k));
    sum += term;
  }
  return sum;
}

struct CosSin {
  double c, s;
};

// cos and sin of the angle 2 pi num / den: exact octant reduction of the
// rational angle, then Taylor series on [0, pi/4].
__host__ __device__ constexpr CosSin turn(int num, int den) {
  num %= den;
  if (num < 0) num += den;
  const long long e = 8LL * num;
  const int o = (int)(e / den);
  const long long r = e - (long long)o * den;
  const double th = kQuarterPi * (double)r / (double)den;          // [0, pi/4)
  const double ph = kQuarterPi * (double)(den - r) / (double)den;  // pi/4 - th
  switch (o) {
    case 0: return {taylor_cos(th), taylor_sin(th)};
    case 1: return {taylor_sin(ph), taylor_cos(ph)};
    case 2: return {-taylor_sin(th), taylor_cos(th)};
    case 3: return {-taylor_cos(ph), taylor_sin(ph)};
    case 4: return {-taylor_cos(th), -taylor_sin(th)};
    case 5: return {-taylor_sin(ph), -taylor_cos(ph)};
    case 6: return {taylor_sin(th), -taylor_cos(th)};
    default: return {taylor_cos(ph), -taylor_sin(ph)};
  }
}

// ---------------------------------------------------------------- complex

template <typename C>
__device__ __forceinline__ C mk(decltype(C{}.x) x, decltype(C{}.x) y) {
  C r;
  r.x = x;
  r.y = y;
  return r;
}
template <typename C>
__device__ __forceinline__ C cadd(C a, C b) { return mk<C>(a.x + b.x, a.y + b.y); }
template <typename C>
__device__ __forceinline__ C csub(C a, C b) { return mk<C>(a.x - b.x, a.y - b.y); }
template <typename C>
__device__ __forceinline__ C cmul(C a, C b) {
  return mk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
template <typename C>
__device__ __forceinline__ C cmulc(C a, C b) {
  return mk<C>(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

// v * exp(SIGN 2 pi i J / M), J and M known at compile time
template <int SIGN, int J, int M, typename C>
__device__ __forceinline__ C twc(C v) {
  constexpr int j = J % M;
  if constexpr (j == 0) {
    return v;
  } else if constexpr (2 * j == M) {
    return mk<C>(-v.x, -v.y);
  } else if constexpr (4 * j == M) {  // times SIGN i
    return SIGN < 0 ? mk<C>(v.y, -v.x) : mk<C>(-v.y, v.x);
  } else if constexpr (4 * j == 3 * M) {  // times -SIGN i
    return SIGN < 0 ? mk<C>(-v.y, v.x) : mk<C>(v.y, -v.x);
  } else {
    using R = decltype(v.x);
    constexpr CosSin w = turn(j, M);
    constexpr R c = (R)w.c;
    constexpr R s = (R)(SIGN * w.s);
    return mk<C>(v.x * c - v.y * s, v.x * s + v.y * c);
  }
}

// In-register DFT of length M: v[k] <- sum_e v[e] exp(SIGN 2 pi i e k / M).
// Only the first NI inputs are read, the others are zero.  (Outputs nobody
// reads cost nothing: the compiler drops their arithmetic.)
template <int M, int SIGN, int NI = M, typename C>
__device__ __forceinline__ void dft(C (&v)[M]) {
  using R = decltype(v[0].x);
  static_assert(NI >= 1 && NI <= M, "nonzero inputs");
  if constexpr (NI == 1) {
#pragma unroll
    for (int k = 1; k < M; ++k) v[k] = v[0];
  } else if constexpr (M == 2) {
    const C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (M == 3) {
    const R h = (R)0.866025403784438646763723170752936183;  // sqrt(3)/2
    C t1 = v[1], d = v[1];
    if constexpr (NI == 3) {
      t1 = cadd(v[1], v[2]);
      d = csub(v[1], v[2]);
    }
    const C t2 = mk<C>(v[0].x - (R)0.5 * t1.x, v[0].y - (R)0.5 * t1.y);
    const C t3 = SIGN < 0 ? mk<C>(h * d.y, -h * d.x) : mk<C>(-h * d.y, h * d.x);
    v[0] = cadd(v[0], t1);
    v[1] = cadd(t2, t3);
    v[2] = csub(t2, t3);
  } else if constexpr (M == 4) {
    C t0 = v[0], t1 = v[0], t2 = v[1], d = v[1];
    if constexpr (NI >= 3) {
      t0 = cadd(v[0], v[2]);
      t1 = csub(v[0], v[2]);
    }
    if constexpr (NI == 4) {
      t2 = cadd(v[1], v[3]);
      d = csub(v[1], v[3]);
    }
    const C t3 = SIGN < 0 ? mk<C>(d.y, -d.x) : mk<C>(-d.y, d.x);
    v[0] = cadd(t0, t2);
    v[1] = cadd(t1, t3);
    v[2] = csub(t0, t2);
    v[3] = csub(t1, t3);
  } else if constexpr (M == 5) {
    constexpr CosSin w1 = turn(1, 5), w2 = turn(2, 5);
    constexpr R c1 = (R)w1.c, c2 = (R)w2.c, s1 = (R)w1.s, s2 = (R)w2.s;
    C a1 = v[1], d1 = v[1], a2 = mk<C>(0, 0), d2 = a2;
    if constexpr (NI == 5) {
      a1 = cadd(v[1], v[4]);
      d1 = csub(v[1], v[4]);
    }
    if constexpr (NI == 3) a2 = d2 = v[2];
    if constexpr (NI >= 4) {
      a2 = cadd(v[2], v[3]);
      d2 = csub(v[2], v[3]);
    }
    C e1, e2, o1, o2;  // o1, o2: SIGN i times the odd parts
    if constexpr (NI >= 3) {
      e1 = mk<C>(v[0].x + c1 * a1.x + c2 * a2.x, v[0].y + c1 * a1.y + c2 * a2.y);
      e2 = mk<C>(v[0].x + c2 * a1.x + c1 * a2.x, v[0].y + c2 * a1.y + c1 * a2.y);
      o1 = mk<C>((R)-SIGN * (s1 * d1.y + s2 * d2.y), (R)SIGN * (s1 * d1.x + s2 * d2.x));
      o2 = mk<C>((R)-SIGN * (s2 * d1.y - s1 * d2.y), (R)SIGN * (s2 * d1.x - s1 * d2.x));
      v[0] = cadd(v[0], cadd(a1, a2));
    } else {
      e1 = mk<C>(v[0].x + c1 * a1.x, v[0].y + c1 * a1.y);
      e2 = mk<C>(v[0].x + c2 * a1.x, v[0].y + c2 * a1.y);
      o1 = mk<C>((R)-SIGN * (s1 * d1.y), (R)SIGN * (s1 * d1.x));
      o2 = mk<C>((R)-SIGN * (s2 * d1.y), (R)SIGN * (s2 * d1.x));
      v[0] = cadd(v[0], a1);
    }
    v[1] = cadd(e1, o1);
    v[2] = cadd(e2, o2);
    v[3] = csub(e2, o2);
    v[4] = csub(e1, o1);
  } else {
    // decimation in time: e = p + P q, k = k' + Q j
    constexpr int P = (M % 4 == 0) ? 4 : ((M % 2 == 0) ? 2 : (M % 3 == 0) ? 3 : 5);
    constexpr int Q = M / P;
    constexpr int NP = NI < P ? NI : P;  // nonzero sub-transforms
    static_assert(P * Q == M, "DFT length must be 2^a 3^b 5^c");
    C sub[P][Q];
    sfor<NP>([&](auto pc) {
      constexpr int p = decltype(pc)::value;
#pragma unroll
      for (int q = 0; q < Q; ++q) sub[p][q] = v[p + P * q];
      dft<Q, SIGN, (NI - p + P - 1) / P>(sub[p]);
    });
    sfor<Q>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      C t[P];
      sfor<NP>([&](auto pc) {
        constexpr int p = decltype(pc)::value;
        t[p] = twc<SIGN, p * k, M>(sub[p][k]);
      });
      dft<P, SIGN, NP>(t);
#pragma unroll
      for (int j = 0; j < P; ++j) v[k + Q * j] = t[j];
    });
  }
}

// ------------------------------------------------------------------ plans

// Lines per tile: 128 bytes of complex values per row of the tile.
template <typename R>
constexpr int kW = sizeof(R) == 4 ? 16 : 8;

// N = N1 * N2 and threads per block (T units of stage B, W N1, in one go).
template <typename R, int N>
struct Cfg;
template <> struct Cfg<float, 48> { static constexpr int N1 = 8, N2 = 6, T = 128; };
template <> struct Cfg<float, 64> { static constexpr int N1 = 8, N2 = 8, T = 128; };
template <> struct Cfg<float, 128> { static constexpr int N1 = 16, N2 = 8, T = 128; };
template <> struct Cfg<float, 216> { static constexpr int N1 = 12, N2 = 18, T = 96; };
template <> struct Cfg<float, 256> { static constexpr int N1 = 16, N2 = 16, T = 256; };
template <> struct Cfg<double, 48> { static constexpr int N1 = 8, N2 = 6, T = 64; };
template <> struct Cfg<double, 64> { static constexpr int N1 = 8, N2 = 8, T = 64; };
template <> struct Cfg<double, 96> { static constexpr int N1 = 12, N2 = 8, T = 96; };
template <> struct Cfg<double, 108> { static constexpr int N1 = 12, N2 = 9, T = 96; };
template <> struct Cfg<double, 128> { static constexpr int N1 = 16, N2 = 8, T = 64; };
template <> struct Cfg<double, 144> { static constexpr int N1 = 12, N2 = 12, T = 96; };
template <> struct Cfg<double, 160> { static constexpr int N1 = 16, N2 = 10, T = 128; };
template <> struct Cfg<double, 180> { static constexpr int N1 = 15, N2 = 12, T = 128; };
template <> struct Cfg<double, 192> { static constexpr int N1 = 16, N2 = 12, T = 128; };
template <> struct Cfg<double, 216> { static constexpr int N1 = 12, N2 = 18, T = 144; };
template <> struct Cfg<double, 240> { static constexpr int N1 = 16, N2 = 15, T = 128; };
template <> struct Cfg<double, 256> { static constexpr int N1 = 16, N2 = 16, T = 128; };

// What of a line a convolution can read and write: stage A's nonzero inputs
// (e = s + N2 q < conv_in_max) and the elements that stage A' (e = s + N2 q)
// and stage B (e = k1 + N1 k2) of the inverse transforms produce (e <
// conv_out_end), out of N1, N1 and N2.  About half of each; leaving out the
// rest took 5 to 13 % off the FP64 passes (fused z pass of 180 points, 282
// refined regions: 3.37 -> 2.96 ms; 96 points: 3.92 -> 3.63 ms).  FP32 keeps all of them (and with them its bits).
template <typename R, int N>
constexpr int kInA = sizeof(R) == 8 ? (conv_in_max(N) + Cfg<R, N>::N2 - 1) / Cfg<R, N>::N2 : Cfg<R, N>::N1;
template <typename R, int N>
constexpr int kOutA = sizeof(R) == 8 ? (conv_out_end(N) + Cfg<R, N>::N2 - 1) / Cfg<R, N>::N2 : Cfg<R, N>::N1;
template <typename R, int N>
constexpr int kOutB = sizeof(R) == 8 ? (conv_out_end(N) + Cfg<R, N>::N1 - 1) / Cfg<R, N>::N1 : Cfg<R, N>::N2;

// Threads of the fused z pass: as above, but 216 points do better with two
// rounds of stage A than with fewer registers (18.7 us a grid against 23; the
// other passes of 216 points take a seventh less time at 144 threads).
template <typename R, int N>
constexpr int kConvT = Cfg<R, N>::T;
template <>
constexpr int kConvT<double, 216> = 96;

// Shared memory of the line kernels: twiddles and one tile of N rows of W+1
// complex (one pad column).  Every stage runs in place: stage B rewrites
// exactly the column each thread read, stage A reads all its inputs into
// registers before a barrier (x passes); the plain y passes write stage B
// straight to the spectrum.
template <typename R, int N>
constexpr size_t smem_lines_bytes() {
  return sizeof(cplx_t<R>) * (size_t)(N + (kW<R> + 1) * N);
}

// Shared memory of the fused z pass: the tile plus a staging buffer of `rows`
// rows for the next grid's input.
template <typename R, int N>
constexpr size_t smem_conv_bytes(int rows) {
  return smem_lines_bytes<R, N>() + sizeof(cplx_t<R>) * (size_t)(rows * kW<R>);
}

// Blocks per SM the registers of a line kernel are limited for.  The FP64 z
// pass is bound by the latency between dependent operations (FP64 units 48 to
// 56 % busy, issue 44 to 46 %, three warps per scheduler), so a few more warps
// help until the registers spill (256: 2.97 ms a call of
// the 256^3 box at 3 blocks, 3.28 at 4; 216: 6.7 -> 4.5 ms of the NFW list at
// 3 instead of 2).  The y passes go without a staging buffer: with one their
// registers left 2 blocks per SM and they ran a quarter slower.
template <typename R, int N, bool CONV>
constexpr int kMinBlocks = 0;  // the compiler's choice
template <> constexpr int kMinBlocks<double, 256, true> = 3;
template <> constexpr int kMinBlocks<double, 216, true> = 3;
template <> constexpr int kMinBlocks<double, 128, true> = 7;

// 16-byte asynchronous copy global -> shared (completion by wait_group)
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory"); }

// tw[j] = exp(-2 pi i j / N), from double-precision sincospi, computed once
// per grid size: a block's own N calls would be a tenth of its FP64 work.
template <typename R>
__global__ void k_twiddles(cplx_t<R> *tw, int n) {
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    double s, c;
    sincospi(2.0 * (double)j / (double)n, &s, &c);
    tw[j] = mk<cplx_t<R>>((R)c, (R)-s);
  }
}

template <typename R, int N, int T>
__device__ __forceinline__ void load_twiddles(cplx_t<R> *tw, const cplx_t<R> *__restrict__ table) {
#pragma unroll
  for (int j = threadIdx.x; j < N; j += T) tw[j] = table[j];
}

// Stage A in place on `buf`: every thread first reads all the elements of
// its units into registers, then (after a barrier) writes the results over
// the tile.
template <typename R, int N, int SIGN, int NI>
__device__ __forceinline__ void stage_a_inplace(cplx_t<R> *buf, const cplx_t<R> *tw, int in_lim) {
  using C = cplx_t<R>;
  constexpr int N1 = Cfg<R, N>::N1, N2 = Cfg<R, N>::N2, T = Cfg<R, N>::T;
  constexpr int W = kW<R>, WP = W + 1, UA = W * N2, IA = (UA + T - 1) / T;
  C v[IA][N1];
#pragma unroll
  for (int it = 0; it < IA; ++it) {
    const int u = threadIdx.x + it * T;
    const int li = u % W, s = u / W;
#pragma unroll
    for (int q = 0; q < NI; ++q) {
      const int e = s + N2 * q;
      v[it][q] = (u < UA && e < in_lim) ? buf[li + WP * e] : mk<C>(0, 0);
    }
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < IA; ++it) {
    const int u = threadIdx.x + it * T;
    if (u < UA) {
      const int li = u % W, s = u / W;
      dft<N1, SIGN, NI>(v[it]);
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1)
        buf[li + WP * (k1 + N1 * s)] = SIGN < 0 ? cmul(v[it][k1], tw[s * k1]) : cmulc(v[it][k1], tw[s * k1]);
    }
  }
}

// Stage B from `src` (stage A layout) into tile layout `dst` (li + (W+1) k).
// Unit (li, k1) reads and writes only the elements li + (W+1) (k1 + N1 j),
// so src may equal dst.  The outputs k2 < NO are written.
template <typename R, int N, int SIGN, int NO>
__device__ __forceinline__ void stage_b_smem(const cplx_t<R> *src, cplx_t<R> *dst) {
  using C = cplx_t<R>;
  constexpr int N1 = Cfg<R, N>::N1, N2 = Cfg<R, N>::N2, T = Cfg<R, N>::T;
  constexpr int W = kW<R>, WP = W + 1, UB = W * N1;
#pragma unroll
  for (int it = 0; it < (UB + T - 1) / T; ++it) {
    const int u = threadIdx.x + it * T;
    if (u < UB) {
      const int li = u % W, k1 = u / W;
      C v[N2];
#pragma unroll
      for (int s = 0; s < N2; ++s) v[s] = src[li + WP * (k1 + N1 * s)];
      dft<N2, SIGN>(v);
#pragma unroll
      for (int k2 = 0; k2 < NO; ++k2) dst[li + WP * (k1 + N1 * k2)] = v[k2];
    }
  }
}

// ------------------------------------------------------------------ kernels

// Grid of every pass but the fused z pass: blockIdx.y = grid of the batch,
// blockIdx.x = tile within it; a grid with fewer tiles than the largest
// leaves the rest of its blocks at once (the host batches grids of similar
// size).

// Spectrum offset of line (y, z), z-major over ny lines per plane.
template <int N>
__device__ __forceinline__ int64_t line_off(int line, int ny, int y0, int z0, int nhp) {
  const int z = line / ny, y = line - z * ny;
  return ((int64_t)(z0 + z) * N + (y0 + y)) * nhp;
}

// x pass, forward r2c.  The in[1] x in[2] real lines of a grid (in[0]
// fixed-point values each, scaled by the grid's inv_scale) are taken in
// pairs as one complex line (a + i b); the two half spectra are separated
// with the Hermitian symmetry of real transforms.  All loops have
// compile-time trip counts, so every thread issues its loads before the
// first one returns.
template <typename R, int N>
__global__ void __launch_bounds__(Cfg<R, N>::T) k_x_r2c(const unsigned long long *__restrict__ acc,
                                                        const double *__restrict__ inv_scale,
                                                        cplx_t<R> *__restrict__ spec,
                                                        const cplx_t<R> *__restrict__ twt,
                                                        const ConvBox *__restrict__ boxes, int nhp) {
  using C = cplx_t<R>;
  constexpr int T = Cfg<R, N>::T, W = kW<R>, WP = W + 1, NH = N / 2 + 1, SUP = conv_in_max(N);
  const ConvBox &bx = boxes[blockIdx.y];
  const int sx = bx.in[0], sy = bx.in[1];
  const int L0 = blockIdx.x * (2 * W);
  const int nl = min(2 * W, sy * bx.in[2] - L0);
  if (nl <= 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int64_t loff[2 * W];
  C *tw = reinterpret_cast<C *>(smem_raw);
  C *t0 = tw + N;
  load_twiddles<R, N, T>(tw, twt);
  if (threadIdx.x < 2 * W) loff[threadIdx.x] = bx.spec_off + line_off<N>(L0 + threadIdx.x, sy, 0, 0, nhp);
  const double inv = inv_scale[blockIdx.y];
  const unsigned long long *src = acc + bx.in_off + (int64_t)L0 * sx;
#pragma unroll
  for (int it = 0; it < (W * SUP + T - 1) / T; ++it) {
    const int idx = threadIdx.x + it * T;
    const int p = idx / SUP, x = idx - p * SUP;
    if (idx < W * SUP && x < sx) {
      const R va = 2 * p < nl ? (R)((double)src[(2 * p) * sx + x] * inv) : (R)0;
      const R vb = 2 * p + 1 < nl ? (R)((double)src[(2 * p + 1) * sx + x] * inv) : (R)0;
      t0[p + WP * x] = mk<C>(va, vb);
    }
  }
  __syncthreads();
  stage_a_inplace<R, N, -1, kInA<R, N>>(t0, tw, sx);
  __syncthreads();
  stage_b_smem<R, N, -1, Cfg<R, N>::N2>(t0, t0);
  __syncthreads();
#pragma unroll
  for (int it = 0; it < (2 * W * NH + T - 1) / T; ++it) {
    const int idx = threadIdx.x + it * T;
    const int lr = idx / NH, kx = idx - lr * NH;
    if (lr < nl) {
      const int p = lr >> 1;
      const C zk = t0[p + WP * kx];
      const C zm = t0[p + WP * ((N - kx) % N)];
      C out;
      if ((lr & 1) == 0) out = mk<C>((R)0.5 * (zk.x + zm.x), (R)0.5 * (zk.y - zm.y));
      else out = mk<C>((R)0.5 * (zk.y + zm.y), (R)0.5 * (zm.x - zk.x));
      spec[loff[lr] + kx] = out;
    }
  }
}

// x pass, c2r of the lines (y, z) of a grid's output window; the values
// [out0[0], out0[0] + out[0]) of each, divided by `scale`, go to the compact
// output.  Two Hermitian half spectra become one complex line (a + i b); only
// the real parts of the DC and Nyquist bins are used.  SUP: the largest
// out[0] of the launch.
template <typename R, int N, int SUP>
__global__ void __launch_bounds__(Cfg<R, N>::T) k_x_c2r(const cplx_t<R> *__restrict__ spec, R *__restrict__ phi,
                                                        const cplx_t<R> *__restrict__ twt,
                                                        const ConvBox *__restrict__ boxes, int nhp, R scale) {
  using C = cplx_t<R>;
  constexpr int T = Cfg<R, N>::T, W = kW<R>, WP = W + 1, NH = N / 2 + 1;
  const ConvBox &bx = boxes[blockIdx.y];
  const int ox = bx.out[0], x0 = bx.out0[0], oy = bx.out[1];
  const int L0 = blockIdx.x * (2 * W);
  const int nl = min(2 * W, oy * bx.out[2] - L0);
  if (nl <= 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int64_t loff[2 * W];
  C *tw = reinterpret_cast<C *>(smem_raw);
  C *t0 = tw + N;
  load_twiddles<R, N, T>(tw, twt);
  if (threadIdx.x < 2 * W)
    loff[threadIdx.x] = bx.spec_off + line_off<N>(L0 + threadIdx.x, oy, bx.out0[1], bx.out0[2], nhp);
  __syncthreads();
#pragma unroll
  for (int it = 0; it < (W * NH + T - 1) / T; ++it) {
    const int idx = threadIdx.x + it * T;
    if (idx < W * NH) {
      const int p = idx / NH, kx = idx - p * NH;
      C a = mk<C>(0, 0), b = mk<C>(0, 0);
      if (2 * p < nl) a = spec[loff[2 * p] + kx];
      if (2 * p + 1 < nl) b = spec[loff[2 * p + 1] + kx];
      if (kx == 0 || kx == N / 2) {
        a.y = 0;
        b.y = 0;
      }
      t0[p + WP * kx] = mk<C>(a.x - b.y, a.y + b.x);
      if (kx > 0 && kx < N / 2) t0[p + WP * (N - kx)] = mk<C>(a.x + b.y, b.x - a.y);
    }
  }
  __syncthreads();
  stage_a_inplace<R, N, +1, Cfg<R, N>::N1>(t0, tw, N);
  __syncthreads();
  stage_b_smem<R, N, +1, SUP == N ? Cfg<R, N>::N2 : kOutB<R, N>>(t0, t0);
  __syncthreads();
  R *dst = phi + bx.out_off + (int64_t)L0 * ox;
  // a power of two divides exactly as its reciprocal multiplies
  constexpr bool pow2 = (N & (N - 1)) == 0;
  const bool plain = scale == (R)1;
  const R inv = (R)1 / scale;
  auto scaled = [&](R v) { return pow2 ? v * inv : (plain ? v : v / scale); };
#pragma unroll
  for (int it = 0; it < (W * SUP + T - 1) / T; ++it) {
    const int idx = threadIdx.x + it * T;
    const int p = idx / SUP, x = idx - p * SUP;
    if (idx < W * SUP && x < ox) {
      const C v = t0[p + WP * (x0 + x)];
      if (2 * p < nl) dst[(2 * p) * ox + x] = scaled(v.x);
      if (2 * p + 1 < nl) dst[(2 * p + 1) * ox + x] = scaled(v.y);
    }
  }
}

// Strided passes over tiles of W consecutive kx.
enum { kYForward = 0, kZConv = 1, kYInverse = 2, kZInverse = 3, kYInverseAll = 4 };

// kYForward: lines (kx, z < in[2]), values y < in[1] in, all N out.
// kZConv: lines (kx, ky), values z < in[2] in, forward transform,
//   multiplication by the real Green table (index ((kz*N + ky)*NH + kx)),
//   inverse transform, the output window's z out; a block handles the grids
//   [b0, b0 + nbb) of the batch with its Green values in registers.
// kYInverse: lines (kx, z of the output window), all N in, its y out.
// kZInverse: lines (kx, ky), all N in and out, kYInverseAll: lines (kx, z) of
//   all z, all N in and out (c2r_full).
template <typename R, int N, int PASS>
__global__ void __launch_bounds__(PASS == kZConv ? kConvT<R, N> : Cfg<R, N>::T, kMinBlocks<R, N, PASS == kZConv>) k_lines(cplx_t<R> *__restrict__ spec, const R *__restrict__ green,
                                                        const cplx_t<R> *__restrict__ twt,
                                                        const ConvBox *__restrict__ boxes, int nhp, int ntiles,
                                                        int nbb, int batch) {
  using C = cplx_t<R>;
  constexpr bool CONV = PASS == kZConv, FWD = PASS == kYForward || CONV, ZLINE = CONV || PASS == kZInverse;
  constexpr int N1 = Cfg<R, N>::N1, N2 = Cfg<R, N>::N2, T = CONV ? kConvT<R, N> : Cfg<R, N>::T;
  constexpr int W = kW<R>, WP = W + 1, NH = N / 2 + 1;
  constexpr int UA = W * N2, UB = W * N1;
  constexpr int IA = (UA + T - 1) / T, IB = (UB + T - 1) / T;
  constexpr int NI = FWD ? kInA<R, N> : N1;
  constexpr int NOA = kOutA<R, N>, NOB = PASS == kYInverse ? kOutB<R, N> : N2;
  const int tile = (int)(blockIdx.x % (unsigned)ntiles);
  const int other = (int)(blockIdx.x / (unsigned)ntiles);
  const int kx0 = tile * W;
  const int b0 = (int)blockIdx.y * nbb;
  const int b1 = CONV ? min(batch, b0 + nbb) : b0 + 1;
  if constexpr (PASS == kYForward) {
    if (other >= boxes[b0].in[2]) return;
  } else if constexpr (PASS == kYInverse) {
    if (other >= boxes[b0].out[2]) return;
  }
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *tw = reinterpret_cast<C *>(smem_raw);
  C *const buf0 = tw + N;
  load_twiddles<R, N, T>(tw, twt);
  R g[CONV ? IB : 1][CONV ? N2 : 1];
  if constexpr (CONV) {
#pragma unroll
    for (int it = 0; it < IB; ++it) {
      const int u = threadIdx.x + it * T;
      const int li = u % W, k1 = u / W, kx = kx0 + li;
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) {
        const int e = k1 + N1 * k2;
        g[it][k2] = (u < UB && kx < NH) ? green[((int64_t)e * N + other) * NH + kx] : (R)0;
      }
    }
  }
  __syncthreads();
  const int64_t estride = ZLINE ? (int64_t)N * nhp : nhp;
  // first element of the line tile of grid b
  auto tile_base = [&](int b) -> C * {
    const int64_t o = ZLINE ? other : (int64_t)N * (other + (PASS == kYInverse ? boxes[b].out0[2] : 0));
    return spec + boxes[b].spec_off + o * nhp + kx0;
  };
  // CONV: the input rows of the next grid are copied into a staging buffer
  // while the current one is transformed, from the end of its stage A (which
  // empties the buffer) on
  constexpr int CPR = (int)(W * sizeof(C) / 16);
  C *const stg = buf0 + WP * N;
  auto prefetch = [&](int b) {
    const C *src = tile_base(b);
    const int rows = boxes[b].in[2];
    for (int c = threadIdx.x; c < rows * CPR; c += T) {
      const int e = c / CPR, part = c - e * CPR;
      cp_async16(reinterpret_cast<char *>(stg + e * W) + 16 * part,
                 reinterpret_cast<const char *>(src + (int64_t)e * estride) + 16 * part);
    }
    cp_async_commit();
  };
  if constexpr (CONV) {
    if (b0 < b1) prefetch(b0);
  }
  for (int b = b0; b < b1; ++b) {
    C *const base = tile_base(b);
    const ConvBox &bx = boxes[b];
    const int in_lim = CONV ? bx.in[2] : (PASS == kYForward ? bx.in[1] : N);
    // values [lo, lo + cnt) are written
    const int lo = CONV ? bx.out0[2] : (PASS == kYInverse ? bx.out0[1] : 0);
    const unsigned cnt = CONV ? bx.out[2] : (PASS == kYInverse ? bx.out[1] : N);
    C *bA = buf0;
    if constexpr (CONV) {
      cp_async_wait<0>();
      __syncthreads();
    }
    // stage A: input -> registers -> DFT over q -> twiddle -> shared
#pragma unroll
    for (int it = 0; it < IA; ++it) {
      const int u = threadIdx.x + it * T;
      if (u < UA) {
        const int li = u % W, s = u / W;
        const bool col = kx0 + li < NH;
        C v[N1];
#pragma unroll
        for (int q = 0; q < NI; ++q) {
          const int e = s + N2 * q;
          if constexpr (CONV) v[q] = (col && e < in_lim) ? stg[e * W + li] : mk<C>(0, 0);
          else v[q] = (col && e < in_lim) ? base[(int64_t)e * estride + li] : mk<C>(0, 0);
        }
        dft<N1, FWD ? -1 : +1, NI>(v);
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) {
          const C w = tw[s * k1];
          bA[li + WP * (k1 + N1 * s)] = FWD ? cmul(v[k1], w) : cmulc(v[k1], w);
        }
      }
    }
    __syncthreads();
    if constexpr (CONV) {
      if (b + 1 < b1) prefetch(b + 1);
    }
    // stage B: DFT over s (and for CONV: Green, inverse DFT over k2, twiddle,
    // written back in place: unit (li, k1) reads and rewrites only its own
    // elements li + WP (k1 + N1 s))
    C *bB = buf0;
#pragma unroll
    for (int it = 0; it < IB; ++it) {
      const int u = threadIdx.x + it * T;
      if (u < UB) {
        const int li = u % W, k1 = u / W;
        C v[N2];
#pragma unroll
        for (int s = 0; s < N2; ++s) v[s] = bA[li + WP * (k1 + N1 * s)];
        dft<N2, FWD ? -1 : +1>(v);
        if constexpr (CONV) {
#pragma unroll
          for (int k2 = 0; k2 < N2; ++k2) {
            v[k2].x *= g[it][k2];
            v[k2].y *= g[it][k2];
          }
          dft<N2, +1>(v);
#pragma unroll
          for (int s = 0; s < N2; ++s) bB[li + WP * (k1 + N1 * s)] = cmulc(v[s], tw[s * k1]);
        } else {
          if (kx0 + li < NH) {
#pragma unroll
            for (int k2 = 0; k2 < NOB; ++k2) {
              const int e = k1 + N1 * k2;
              if ((unsigned)(e - lo) < cnt) base[(int64_t)e * estride + li] = v[k2];
            }
          }
        }
      }
    }
    if constexpr (CONV) {
      __syncthreads();
      // stage A': inverse DFT over k1 -> element s + N2 q
#pragma unroll
      for (int it = 0; it < IA; ++it) {
        const int u = threadIdx.x + it * T;
        if (u < UA) {
          const int li = u % W, s = u / W;
          C v[N1];
#pragma unroll
          for (int k1 = 0; k1 < N1; ++k1) v[k1] = bB[li + WP * (k1 + N1 * s)];
          dft<N1, +1>(v);
          if (kx0 + li < NH) {
#pragma unroll
            for (int q = 0; q < NOA; ++q) {
              const int e = s + N2 * q;
              if ((unsigned)(e - lo) < cnt) base[(int64_t)e * estride + li] = v[q];
            }
          }
        }
      }
    }
    // the next grid's stage A rewrites the tile: every thread has finished
    // reading it at the barrier at the top of the loop
  }
}

template <typename R>
__global__ void k_real_to_cplx(const R *__restrict__ g, cplx_t<R> *__restrict__ spec, int n, int nhp) {
  const int nh = n / 2 + 1;
  const int64_t cnt = (int64_t)nh * n * n;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / nh;
    const int kx = (int)(i - row * nh);
    spec[row * nhp + kx] = mk<cplx_t<R>>(g[i], (R)0);
  }
}

template <typename K>
int32_t allow_smem(K kernel, size_t bytes) {
  PYFOF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return kOk;
}

// Shared-memory limits of every kernel of grid N, set once per device.
template <typename R, int N>
int32_t prepare() {
  static PerDeviceOnce once;
  int dev = 0;
  PYFOF_CUDA(cudaGetDevice(&dev));
  return once.run(dev, [] {
    const size_t sm = smem_lines_bytes<R, N>();
    int32_t r = kOk;
    if (r == kOk) r = allow_smem(k_x_r2c<R, N>, sm);
    if (r == kOk) r = allow_smem(k_x_c2r<R, N, N / 2 + 1>, sm);
    if (r == kOk) r = allow_smem(k_x_c2r<R, N, N>, sm);
    if (r == kOk) r = allow_smem(k_lines<R, N, kYForward>, sm);
    if (r == kOk) r = allow_smem(k_lines<R, N, kYInverse>, sm);
    if (r == kOk) r = allow_smem(k_lines<R, N, kYInverseAll>, sm);
    if (r == kOk) r = allow_smem(k_lines<R, N, kZInverse>, sm);
    if (r == kOk) r = allow_smem(k_lines<R, N, kZConv>, smem_conv_bytes<R, N>(conv_in_max(N)));
    return r;
  });
}

template <typename R, int N>
int32_t convolve_n(const unsigned long long *acc, const double *inv_scale, R *phi, cplx_t<R> *spec, const R *green,
                   const cplx_t<R> *tw, const ConvBox *boxes, const ConvExtent &ext, int batch, bool scaled,
                   cudaStream_t s, int waves) {
  PYFOF_TRY((prepare<R, N>()));
  constexpr int W = kW<R>, T = Cfg<R, N>::T;
  const int nhp = (int)spec_row<R>(N);
  const int ntiles = nhp / W;
  const size_t sm = smem_lines_bytes<R, N>();
  const dim3 gx_in((unsigned)ceil_div(ext.in_lines, 2 * W), (unsigned)batch);
  const dim3 gx_out((unsigned)ceil_div(ext.out_lines, 2 * W), (unsigned)batch);
  k_x_r2c<R, N><<<gx_in, T, sm, s>>>(acc, inv_scale, spec, tw, boxes, nhp);
  PYFOF_CHECK_LAUNCH();
  k_lines<R, N, kYForward><<<dim3((unsigned)(ntiles * ext.in_z), (unsigned)batch), T, sm, s>>>(
      spec, nullptr, tw, boxes, nhp, ntiles, 1, batch);
  PYFOF_CHECK_LAUNCH();
  // z: grids split into chunks so that the launch is at least `waves` full waves
  const int64_t per = (int64_t)ntiles * N;
  const size_t smc = smem_conv_bytes<R, N>(ext.in_z);
  int conv_blocks_per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&conv_blocks_per_sm, k_lines<R, N, kZConv>, kConvT<R, N>, smc) !=
          cudaSuccess || conv_blocks_per_sm < 1)
    conv_blocks_per_sm = 1;
  const int64_t slots = (int64_t)conv_blocks_per_sm * kNumSMs;
  const int nchunk = (int)std::max<int64_t>(1, std::min<int64_t>(batch, ceil_div((int64_t)waves * slots, per)));
  const int nbb = (int)ceil_div(batch, nchunk);
  const int nchunk_used = (int)ceil_div(batch, nbb);
  k_lines<R, N, kZConv><<<dim3((unsigned)per, (unsigned)nchunk_used), kConvT<R, N>, smc, s>>>(
      spec, green, tw, boxes, nhp, ntiles, nbb, batch);
  PYFOF_CHECK_LAUNCH();
  k_lines<R, N, kYInverse><<<dim3((unsigned)(ntiles * ext.out_z), (unsigned)batch), T, sm, s>>>(
      spec, nullptr, tw, boxes, nhp, ntiles, 1, batch);
  PYFOF_CHECK_LAUNCH();
  const R n3 = scaled ? (R)1 : (R)((double)N * N * N);
  k_x_c2r<R, N, N / 2 + 1><<<gx_out, T, sm, s>>>(spec, phi, tw, boxes, nhp, n3);
  PYFOF_CHECK_LAUNCH();
  return kOk;
}

template <typename R, int N>
int32_t c2r_full_n(const R *green, cplx_t<R> *spec, R *out, const cplx_t<R> *tw, const ConvBox *box, cudaStream_t s) {
  PYFOF_TRY((prepare<R, N>()));
  constexpr int W = kW<R>, T = Cfg<R, N>::T;
  const int nhp = (int)spec_row<R>(N);
  const int ntiles = nhp / W;
  const size_t sm = smem_lines_bytes<R, N>();
  const int64_t cnt = (int64_t)(N / 2 + 1) * N * N;
  k_real_to_cplx<R><<<(unsigned)std::min<int64_t>(ceil_div(cnt, 256), 4096), 256, 0, s>>>(green, spec, N, nhp);
  PYFOF_CHECK_LAUNCH();
  // z inverse over all ky, then y inverse over all z
  k_lines<R, N, kZInverse><<<(unsigned)(ntiles * N), T, sm, s>>>(spec, nullptr, tw, box, nhp, ntiles, 1, 1);
  PYFOF_CHECK_LAUNCH();
  k_lines<R, N, kYInverseAll><<<(unsigned)(ntiles * N), T, sm, s>>>(spec, nullptr, tw, box, nhp, ntiles, 1, 1);
  PYFOF_CHECK_LAUNCH();
  k_x_c2r<R, N, N><<<(unsigned)ceil_div((int64_t)N * N, 2 * W), T, sm, s>>>(spec, out, tw, box, nhp, (R)1);
  PYFOF_CHECK_LAUNCH();
  return kOk;
}

}  // namespace

template <typename R>
int32_t fill_twiddles(cplx_t<R> *tw, int n, cudaStream_t s) {
  k_twiddles<R><<<1, 256, 0, s>>>(tw, n);
  PYFOF_CHECK_LAUNCH();
  return kOk;
}

template <typename R>
int32_t pm_convolve_batch(const unsigned long long *acc, const double *inv_scale, R *phi, cplx_t<R> *spec,
                          const R *green, const cplx_t<R> *tw, int n, const ConvBox *boxes, const ConvExtent &ext,
                          int batch, bool scaled, cudaStream_t s, int waves) {
  const int in_max = conv_in_max(n), out_max = conv_out_end(n);
  if (batch < 1 || batch > 65535 || ext.in_lines < 1 || ext.out_lines < 1 || ext.in_x > in_max ||
      ext.in_y > in_max || ext.in_z > in_max || ext.out_end > out_max) {
    set_error("invalid convolution batch (n %d, batch %d)", n, batch);
    return kInvalid;
  }
#define PYFOF_CONV(N) return convolve_n<R, N>(acc, inv_scale, phi, spec, green, tw, boxes, ext, batch, scaled, s, waves)
  if constexpr (sizeof(R) == 8) {
    switch (n) {
      case 96: PYFOF_CONV(96);
      case 108: PYFOF_CONV(108);
      case 144: PYFOF_CONV(144);
      case 160: PYFOF_CONV(160);
      case 180: PYFOF_CONV(180);
      case 192: PYFOF_CONV(192);
      case 240: PYFOF_CONV(240);
      default: break;
    }
  }
  switch (n) {
    case 48: PYFOF_CONV(48);
    case 64: PYFOF_CONV(64);
    case 128: PYFOF_CONV(128);
    case 216: PYFOF_CONV(216);
    case 256: PYFOF_CONV(256);
    default: set_error("unsupported FFT size %d", n); return kInvalid;
  }
#undef PYFOF_CONV
}

template <typename R>
int32_t c2r_full(const R *green, cplx_t<R> *spec, R *out, const cplx_t<R> *tw, const ConvBox *box, int n,
                 cudaStream_t s) {
  if constexpr (sizeof(R) == 8) {
    switch (n) {
      case 96: return c2r_full_n<R, 96>(green, spec, out, tw, box, s);
      case 108: return c2r_full_n<R, 108>(green, spec, out, tw, box, s);
      case 144: return c2r_full_n<R, 144>(green, spec, out, tw, box, s);
      case 160: return c2r_full_n<R, 160>(green, spec, out, tw, box, s);
      case 180: return c2r_full_n<R, 180>(green, spec, out, tw, box, s);
      case 192: return c2r_full_n<R, 192>(green, spec, out, tw, box, s);
      case 240: return c2r_full_n<R, 240>(green, spec, out, tw, box, s);
      default: break;
    }
  }
  switch (n) {
    case 48: return c2r_full_n<R, 48>(green, spec, out, tw, box, s);
    case 64: return c2r_full_n<R, 64>(green, spec, out, tw, box, s);
    case 128: return c2r_full_n<R, 128>(green, spec, out, tw, box, s);
    case 216: return c2r_full_n<R, 216>(green, spec, out, tw, box, s);
    case 256: return c2r_full_n<R, 256>(green, spec, out, tw, box, s);
    default: set_error("unsupported FFT size %d", n); return kInvalid;
  }
}

template int32_t fill_twiddles<float>(float2 *, int, cudaStream_t);
template int32_t fill_twiddles<double>(double2 *, int, cudaStream_t);
template int32_t pm_convolve_batch<float>(const unsigned long long *, const double *, float *, float2 *, const float *,
                                          const float2 *, int, const ConvBox *, const ConvExtent &, int, bool, cudaStream_t,
                                          int);
template int32_t pm_convolve_batch<double>(const unsigned long long *, const double *, double *, double2 *,
                                           const double *, const double2 *, int, const ConvBox *, const ConvExtent &,
                                           int, bool, cudaStream_t, int);
template int32_t c2r_full<float>(const float *, float2 *, float *, const float2 *, const ConvBox *, int, cudaStream_t);
template int32_t c2r_full<double>(const double *, double2 *, double *, const double2 *, const ConvBox *, int,
                                  cudaStream_t);

}  // namespace pyfof
