// Adjoint spread by register columns, and the inverse x transform that reads
// its coil-interleaved grid.
//
// The grid is cut into columns: 3-D 4 (x) x 2 (y) x 16 (z) cells, 2-D 8 (x) x
// 8 (y) cells.  A plan-time record per (sample, column) pair
// holds the sample's weights clipped to the column; a column's records are
// ordered by the first plane (z in 3-D, y in 2-D) they meet.  One warp walks
// a run of a column's records ("chunk") with the sums of the few planes that
// the current footprints meet in registers -- lanes over coils -- and writes
// each plane once, coil-interleaved.  No atomics; the summation order is
// fixed.
//
// The grid of C coils: groups of 16 coils, each [G_z][G_y][G_x][16], then a
// last group of C mod 16 coils with 4, 8 or 16 coils of storage per cell.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "binning.cuh"
#include "devutil.hpp"
#include "geometry.hpp"
#include "tma.cuh"

namespace gnufft
{

// A run of one column's records that meets planes [p0, p1); slot >= 0: the
// column has several runs, this one's sums go to partial column `slot`.
struct TileChunk
{
  uint32_t tile, begin, end;
  int32_t slot;
  uint32_t p0, p1, pad[2];
};

// Plan-time tables (built by build_tile_tables).
struct TileTables
{
  DeviceBuffer recs;    // records, sorted by column and first plane
  DeviceBuffer chunks;  // TileChunk
  DeviceBuffer multi;   // uint4 (column, first slot, slots, first
                        // chunk) of columns with several chunks
  DeviceBuffer occ;     // per row of columns: bit per column along x
  int n_chunks = 0, n_few = 0, n_many = 0, n_slots = 0;
  size_t bytes() const
  {
    return recs.bytes() + chunks.bytes() + multi.bytes() + occ.bytes();
  }
  bool ready() const { return n_chunks > 0; }
};

// Grids the spread takes: every axis longer than a column by a footprint (up
// to 8 cells), so that a wrapped footprint meets each column once.
bool tile_spread_supported(const Geo &g);

void build_tile_tables(const float *traj_sorted, const uint32_t *sector_sorted,
                       uint32_t M, const Geo &g, const float *lut,
                       TileTables &t, BuildWork &work, cudaStream_t s);

// Coil lanes per group of the tile spread for CP k-space lanes (0: CP is
// not a multiple of 4).
int tile_coil_lanes(int CP);

// Coils of storage per grid cell of a call with C coils, all groups.
int tile_grid_pitch(int C);

// Partial columns (complex elements) of a call with C coils.
size_t tile_partial_elems(const TileTables &t, const Geo &g, int C);

// grid (layout above) = spread of the coil-interleaved sorted k-space ks
// [M][CP] (coils from C on are zero); only columns with
// records are written (see TileTables::occ).  Returns the launches made.
int launch_tile_spread(const TileTables &t, const float2 *ks, int CP,
                       const Geo &g, int C, float2 *grid, float2 *partial,
                       cudaStream_t s);

// The inverse x transform of the spread's grid: out [C][G_z][G_y][N_x]
// (rows in the INVERSE-shifted frame the next passes expect), for
// power-of-two rows of 16 to 1024 cells and those of the general passes.
bool tile_xpass_supported(const Geo &g);
void launch_tile_xpass(const TileTables &t, const float2 *grid,
                       const Geo &g, int C, const float2 *roots_x,
                       float2 *out, tma::CopyWait cw, cudaStream_t s);

}  // namespace gnufft
