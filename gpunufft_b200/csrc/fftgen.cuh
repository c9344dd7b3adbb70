// Pruned transform passes for line lengths up to 1024 that split into two or
// three factors of at most 16 (the power-of-two lengths have kernels of their
// own in fftpass.cu).  Conventions as there: FFT input n reads source row
// (n + in_add) mod L when < in_count (else zero), FFT output k goes to row
// (k + out_add) mod L when < out_count.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "geometry.hpp"

namespace gnufft
{

// L = R[0] R[1] R[2] with factors in [2, 16] (R[1] 1: two factors); false
// when there is no such split.
bool gen_split(int L, int R[3]);

// Columns per tile of a listed, paired column pass.
constexpr int kGenTileCols = 8;

// Lines along a strided axis: src planes of src_rows x ncols, dst planes of
// dst_rows x ncols, columns contiguous.  `paired`: coil pairs interleaved in
// the output (plane c: ((c / 2) * dst_rows * ncols + row * ncols + col) * 2 +
// c % 2).  `colrange`: per column the output rows to write.  `tiles` (paired):
// the n_tiles tiles of kGenTileCols columns to transform (NULL: all).
void gen_cols(bool inverse, int L, const float2 *src, float2 *dst,
              long long ncols, int src_rows, int dst_rows, long long planes,
              int in_add, int in_count, int out_add, int out_count,
              const float2 *roots, const uint2 *colrange, bool paired,
              const uint32_t *tiles, int n_tiles, cudaStream_t s);

// Forward rows: image (x maps) x deapodization -> A [C][rows][L].
void gen_rows_fwd(int L, const float2 *image, const float2 *sens,
                  const float *deapo, int Nx, long long rows, long long N,
                  int C, int in_add, int out_add, const float2 *roots,
                  float2 *A, cudaStream_t s);

// Last adjoint pass (inverse lines along a strided axis, crop, scale,
// deapodization, conj(maps) coil sum per group of cpb coils, or per coil
// without maps): as k_fft_cols_sum in fftpass.cu.
void gen_cols_sum(int L, const float2 *src, long long ncols,
                  long long coil_stride, const float *deapo,
                  const float2 *sens, int n_out, long long N, int C, int cpb,
                  int groups, int out_add, float scale, int stage,
                  int accumulate, const float2 *roots, float2 *out,
                  float2 *partial, cudaStream_t s);

// Inverse x transform of the column spread's grid (layout and occupancy of
// tilespread.cuh): out [C][G_z][G_y][N_x].  tile_x, tile_y, tile_z: log2 of
// the columns' extents.
void gen_xpass(const float2 *grid, const uint32_t *occ, int occ_words,
               int tile_x, int tile_y, int tile_z, int tiles_y, const Geo &g,
               int C, const float2 *roots, float2 *out, cudaStream_t s);

}  // namespace gnufft
