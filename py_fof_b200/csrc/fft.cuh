// Batched 3-D real<->complex FFTs of zero-padded cubic grids, for the
// isolated particle-mesh convolution (replaces FFTW3f at
// bound_fortran.f90:2166-2169, :2675-2677, :894-906).
//
// Grids: n points per axis, n = 2^a 3^b 5^c <= 256 (48, 64, 128, 216, 256; in
// FP64 also 96, 108, 144, 160, 180, 192, 240).
// Every grid of a batch comes with its support box (ConvBox): the density is
// nonzero only on the nodes [0, in) of the zero-padded half of the isolated
// convolution, and the potential is wanted only on the nodes
// [out0, out0 + out).  Both real grids are compact arrays of those nodes, x
// fastest.  The spectrum keeps the in[2] planes of nonzero z, x halved, rows
// padded to a whole number of 128-byte line tiles (spec_row):
//     spec[spec_off + (z*n + y)*spec_row(n) + kx],  kx < n/2+1, z < in[2]
// Line transforms are register-resident mixed-radix DFTs (fft.cu).  Lines
// that are zero, and lines none of whose values are wanted, are neither read
// nor transformed; what is computed is the same operations on the same
// values as over the whole grid.  The inverse follows FFTW's c2r definition
// (complex inverse transforms along z and y, then a Hermitian c2r along x
// that uses only the real parts of the DC and Nyquist bins) and is
// unnormalised.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace pyfof {

template <typename R>
using cplx_t = typename std::conditional<std::is_same<R, float>::value, float2, double2>::type;

// Row length (complex elements) of the half spectrum of an n-point axis.
template <typename R>
constexpr int64_t spec_row(int n) {
  return (int64_t)((n / 2 + 1 + (sizeof(R) == 4 ? 15 : 7)) / (sizeof(R) == 4 ? 16 : 8)) *
         (sizeof(R) == 4 ? 16 : 8);
}

// Complex elements of the first nz planes of a half spectrum of an n^3 grid.
template <typename R>
constexpr int64_t spec_elems(int n, int nz) {
  return spec_row<R>(n) * n * nz;
}

// Lengths a convolution on the n-point grid may run at, ascending, n last.
// The grid is a zero-padded one: between the nodes of a box a convolution only
// meets the lags |d| <= reach, so any transform of 2 reach + 1 points or more
// gives the same potential, with the kernel cut to the lags of its length.
// A 256-point grid whose halo fills half of what it may costs a sixth at 128
// points; calls: 256^3 box 27.7 -> 25.5 ms, 20,000 halos 108.6 -> 93.7 ms, 1 M
// zoom region 19.4 -> 16.7 ms.  The list is coarse, since every length in a call is five more launches.  A
// halo's length follows from its own box alone, so its bits do not depend on
// what else is in the call.  FP32 stays at n: there the rounding of another
// length (1e-7) could show in who is bound.
inline const int *conv_lengths(int n, bool fp64) {
  static const int own[5][2] = {{48, 0}, {64, 0}, {128, 0}, {216, 0}, {256, 0}};
  static const int l64[] = {48, 64, 0}, l128[] = {96, 108, 128, 0}, l216[] = {180, 216, 0};
  static const int l256[] = {128, 144, 160, 180, 192, 216, 240, 256, 0};
  if (fp64) {
    if (n == 64) return l64;
    if (n == 128) return l128;
    if (n == 216) return l216;
    if (n == 256) return l256;
  }
  return own[n == 48 ? 0 : n == 64 ? 1 : n == 128 ? 2 : n == 216 ? 3 : 4];
}

// Nonzero input nodes per axis that a transform of n points takes, and the end
// of the nodes it can put out.  A box that fits a shorter transform is at most
// half of it; a whole grid's may have one node more, a refined region's sources
// reach beyond half of its 96 or 180 points.
__host__ __device__ constexpr bool conv_shorter(int n) {
  return n == 96 || n == 108 || n == 144 || n == 160 || n == 180 || n == 192 || n == 240;
}
__host__ __device__ constexpr int conv_out_end(int n) { return conv_shorter(n) ? n / 2 : n / 2 + 1; }
__host__ __device__ constexpr int conv_in_max(int n) { return n == 96 ? 56 : n == 180 ? 108 : conv_out_end(n); }

// One grid of a batch (see above).  Offsets in elements; out0 + out <= in.
struct ConvBox {
  int64_t in_off;    // density (64-bit fixed-point nodes)
  int64_t out_off;   // potential (R nodes)
  int64_t spec_off;  // half spectrum (complex)
  int32_t in[3];
  int32_t out0[3], out[3];
  int32_t pad;
};

// Transform length for a box on the n-point grid.
inline int conv_length(int n, bool fp64, const ConvBox &b) {
  int reach = 0, in = 0, end = 0;
  for (int d = 0; d < 3; ++d) {
    const int back = b.in[d] - 1 - b.out0[d], ahead = b.out0[d] + b.out[d] - 1;
    reach = back > reach ? back : reach;
    reach = ahead > reach ? ahead : reach;
    in = b.in[d] > in ? b.in[d] : in;
    end = ahead + 1 > end ? ahead + 1 : end;
  }
  const int *l = conv_lengths(n, fp64);
  while (*l < n && (*l < 2 * reach + 1 || conv_in_max(*l) < in || conv_out_end(*l) < end)) ++l;
  return *l;
}

// Bytes the five passes of one grid's convolution read and write (x, y,
// fused z, y, x), each line once.
template <typename R>
inline double conv_bytes(int n, const ConvBox &b) {
  const double c = 2.0 * sizeof(R) * (n / 2 + 1), ix = b.in[0], iy = b.in[1], iz = b.in[2];
  const double ox = b.out[0], oy = b.out[1], oz = b.out[2];
  return 8.0 * ix * iy * iz + 2.0 * c * iy * iz + 2.0 * c * n * iz + 2.0 * c * n * oz + 2.0 * c * oy * oz +
         sizeof(R) * ox * oy * oz;
}

// Largest extents over the boxes of a batch (launch shapes).
struct ConvExtent {
  int in_x = 0, in_y = 0, in_z = 0, out_y = 0, out_z = 0, out_end = 0;
  int64_t in_lines = 0, out_lines = 0;
  void add(const ConvBox &b) {
    in_x = b.in[0] > in_x ? b.in[0] : in_x;
    for (int d = 0; d < 3; ++d) out_end = b.out0[d] + b.out[d] > out_end ? b.out0[d] + b.out[d] : out_end;
    in_y = b.in[1] > in_y ? b.in[1] : in_y;
    in_z = b.in[2] > in_z ? b.in[2] : in_z;
    out_y = b.out[1] > out_y ? b.out[1] : out_y;
    out_z = b.out[2] > out_z ? b.out[2] : out_z;
    const int64_t li = (int64_t)b.in[1] * b.in[2], lo = (int64_t)b.out[1] * b.out[2];
    in_lines = li > in_lines ? li : in_lines;
    out_lines = lo > out_lines ? lo : out_lines;
  }
};

// twiddle table exp(-2 pi i j / n), j < n, into tw (device, n elements)
template <typename R>
int32_t fill_twiddles(cplx_t<R> *tw, int n, cudaStream_t s);

// Runs out = G * FFT(rho) and phi <- iFFT(out) / n^3 over a batch:
//   acc, inv_scale  the densities as 64-bit fixed-point nodes (value of grid
//         j = acc * inv_scale[j])
//   phi   the potentials divided by n^3 in R precision (as the reference's
//         rho/real(n**3)), or as they are where the table holds the factor
//         (scaled); may alias acc when every out_off is at its grid's
//         in_off or below it in bytes
//   boxes, ext  the batch's boxes (device) and their largest extents
//   spec  half spectra (scratch)
//   green half-spectrum table of real values, unpadded rows:
//         green[((kz*n + ky)*(n/2+1) + kx]
//   tw    fill_twiddles' table
//   waves the fused z pass splits the batch so that its grid covers at
//         least this many full waves of the GPU (a launch shape only)
template <typename R>
int32_t pm_convolve_batch(const unsigned long long *acc, const double *inv_scale, R *phi, cplx_t<R> *spec,
                          const R *green, const cplx_t<R> *tw, int n, const ConvBox *boxes, const ConvExtent &ext,
                          int batch, bool scaled, cudaStream_t s, int waves = 4);

// FFTW-style c2r of a real half-spectrum table (the Green's function) into a
// full n^3 real grid (unnormalised); used once per table to extract the
// self-potential kernel.  box (device): in = out = n, everything else 0.
template <typename R>
int32_t c2r_full(const R *green, cplx_t<R> *spec, R *out, const cplx_t<R> *tw, const ConvBox *box, int n,
                 cudaStream_t s);

}  // namespace pyfof
