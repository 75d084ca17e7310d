// Batched 3-D real<->complex FFTs of zero-padded cubic grids, for the
// isolated particle-mesh convolution (replaces FFTW3f at
// bound_fortran.f90:2166-2169, :2675-2677, :894-906).
//
// Grids: n points per axis, n = 2^a 3^b <= 256 (48, 64, 128, 216, 256).
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

// One grid of a batch (see above).  Offsets in elements; out0 + out <= in.
struct ConvBox {
  int64_t in_off;    // density (64-bit fixed-point nodes)
  int64_t out_off;   // potential (R nodes)
  int64_t spec_off;  // half spectrum (complex)
  int32_t in[3];
  int32_t out0[3], out[3];
  int32_t pad;
};

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
  int in_y = 0, in_z = 0, out_y = 0, out_z = 0;
  int64_t in_lines = 0, out_lines = 0;
  void add(const ConvBox &b) {
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
//         rho/real(n**3)); may alias acc when every out_off is at its grid's
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
                          int batch, cudaStream_t s, int waves = 4);

// FFTW-style c2r of a real half-spectrum table (the Green's function) into a
// full n^3 real grid (unnormalised); used once per table to extract the
// self-potential kernel.  box (device): in = out = n, everything else 0.
template <typename R>
int32_t c2r_full(const R *green, cplx_t<R> *spec, R *out, const cplx_t<R> *tw, const ConvBox *box, int n,
                 cudaStream_t s);

}  // namespace pyfof
