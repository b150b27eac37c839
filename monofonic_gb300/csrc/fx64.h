// Transforms of the plain FP64 form in 64-bit fixed point (fx64.cuh): what the
// engine launches.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "pdl.cuh"

namespace fx {

// a length the transforms are built for: even, no prime factor above 7
bool length_supported(int L);
// twiddle tables of a length (host memory, kept for the process: some KB for
// each length that was asked for)
const void *twiddles(int L);
inline size_t twiddle_bytes(int L) { return (size_t(L) * 24 + 15) / 16 * 16; }
// device tables of a grid: mode[0..1][n] (Strided::mode), mode[2][n] the
// fractional part and mode[4][n] (as int) the integer part of the PLT table
// coordinate x = i * (64 / n), mode[3][n] the signed mode index that x stands for,
// (x - 64 (x > 32)) / (64 / n), all evaluated in double as particle_plt.hh:551-585
// does (where 64 / n is rounded, so are the small negative indices); rinv[q] = 1 / q and root[q] = sqrt(q) for
// q = 1 .. 3 (n/2)^2 (zero at q = 0)
cudaError_t fill_tables(int n, double *mode, double *rinv, double *root, cudaStream_t st);
inline size_t rinv_len(int n) { return 3 * size_t(n / 2) * (n / 2) + 1; }
// the kernels' shared memory limits on the current device `dev`, once (before
// any capture)
cudaError_t prepare_device(int dev);

// One pass over pencils along x or y of k-space arrays, 8 (or 4) adjacent kz a
// CTA.  A pencil element (outer o, row r, kz) lies at base + o * outer + r *
// row + kz (complex elements).
struct Strided {
  int L;                  // transform length
  const void *tw;         // its twiddles on the device (twiddles / twiddles32)
  bool inverse;
  int n;                  // N (the unpadded grid) for padded or cut rows
  bool pad_in;            // rows r < n go to the padded positions of a length-L pencil (else r < L)
  bool cut_out;           // the padded positions of r < n are stored as rows r, Nyquist row zero (else r < L)
  int outer, kc;          // outer indices, kz values
  long long in_outer, in_row, out_outer, out_row;
  // up to 6 outputs in `groups` groups of consecutive ones: a CTA makes the
  // outputs of one group in turn, so that the last may overwrite their source
  int ops, groups, first[7];
  const void *src[6];
  void *dst[6];
  // factors of an output's input: (row index)^pr (kz)^pk, signed mode indices
  // with the Nyquist index n / 2 zero where the power is positive
  int pr[6], pk[6];
  const double *mode;     // [2][n]: signed index and its square, Nyquist zero (padded rows)
  // cut_out: output factor.  inv_lap: times -fac / (i^2 + j^2 + k^2) with the
  // Nyquist indices and k = 0 zero, outer index = mode index (rinv[q] = 1 / q),
  // and the kz = kc column (Nyquist) zeroed
  bool inv_lap;
  const double *rinv;
  double fac;
  double in_fac;          // single precision: factor of the inputs (0: one); mode and rinv are not read
  // forward transform, rows cut to n (Nyquist zero), factor fac, transformed
  // back: convolve3's truncation between its two products
  bool truncate;
};
cudaError_t run_strided(const Strided &s, cudaStream_t st);

// Real rows: `rows` consecutive rows of L reals, `pitch` reals apart, in place
// with their spectra (kz < kc complex values); two rows share a transform.
struct Rows {
  int L;
  const void *tw;
  int kc;                 // kz values of the spectrum (read or written); 2 (kc - 1) == L: with the Nyquist one
  long long rows, pitch;
  int count;              // fields
  void *field[6];
};
cudaError_t run_c2r(const Rows &r, cudaStream_t st);
cudaError_t run_r2c(const Rows &r, cudaStream_t st);

// The same passes on single-precision fields (fs32.cu), for the lengths that
// length_supported names
cudaError_t run_strided32(const Strided &s, cudaStream_t st);
cudaError_t run_c2r32(const Rows &r, cudaStream_t st);
cudaError_t run_r2c32(const Rows &r, cudaStream_t st);
// float2 (cos, -sin)(2 pi t / L), t < L (host memory, kept for the process)
const float2 *twiddles32(int L);
cudaError_t prepare_device32(int dev);
// lengths whose single-precision passes beat cuFFT: the instances, and short ones
// with the run-time kernels (36^3 3LPT 0.24 against 0.43 ms; without instances
// 300^3 2LPT would take 16.4 ms against 9.3, 400^3 26.0 against 25.8)
bool length_fast32(int L, bool padded);

}  // namespace fx
