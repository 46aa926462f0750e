// tb_cells.cuh -- cell list shared by the neighbour searches (tb_cells.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace tb {

struct CellGrid {
    int nc[3];                // cells along each edge
    double box[3], lo[3], scale[3];  // box[d] > 0: periodic; cell = (x - lo) scale
    // the atoms cell by cell, ascending within a cell
    const int32_t *start = nullptr, *atom = nullptr;
    const float4 *pos = nullptr;  // position, species (as bits)

    __host__ __device__ int index(int d, double x) const
    {
        if (box[d] > 0) x -= box[d] * floor(x / box[d]);
        const int c = (int)((x - lo[d]) * scale[d]);
        return c < 0 ? 0 : c < nc[d] ? c : nc[d] - 1;
    }
};

// The cells (at least rc wide) of natoms host positions; false, and one cell
// for all, if a position is not finite or absurdly far out.
bool cell_grid(int natoms, const double *xyz, const double box[3], double rc, CellGrid &g);
size_t cell_bytes(int natoms, const CellGrid &g);
// Sorts the atoms into cells on the device; scratch: cell_bytes, 16-byte aligned.
void cell_build(cudaStream_t st, int natoms, const double *d_xyz, const int32_t *d_species, CellGrid &g, void *scratch);

// Calls f(first, end) for the sorted atoms of each cell around position x
// (its own and the adjoining ones, every cell once).
template <typename F>
__device__ __forceinline__ void cell_around(const CellGrid &g, const double x[3], F f)
{
    int c[3], n[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        c[d] = g.index(d, x[d]);
        n[d] = g.nc[d] > 1 ? 3 : 1;
    }
    for (int a = 0; a < n[0]; a++) {
        int ca = c[0] + (n[0] > 1 ? a - 1 : 0);
        if (ca < 0 || ca >= g.nc[0]) {
            if (!(g.box[0] > 0)) continue;
            ca += ca < 0 ? g.nc[0] : -g.nc[0];
        }
        for (int b = 0; b < n[1]; b++) {
            int cb = c[1] + (n[1] > 1 ? b - 1 : 0);
            if (cb < 0 || cb >= g.nc[1]) {
                if (!(g.box[1] > 0)) continue;
                cb += cb < 0 ? g.nc[1] : -g.nc[1];
            }
            for (int e = 0; e < n[2]; e++) {
                int ce = c[2] + (n[2] > 1 ? e - 1 : 0);
                if (ce < 0 || ce >= g.nc[2]) {
                    if (!(g.box[2] > 0)) continue;
                    ce += ce < 0 ? g.nc[2] : -g.nc[2];
                }
                const int id = (ca * g.nc[1] + cb) * g.nc[2] + ce;
                f(__ldg(g.start + id), __ldg(g.start + id + 1));
            }
        }
    }
}

}  // namespace tb
