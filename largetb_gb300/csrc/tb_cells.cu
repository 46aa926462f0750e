// tb_cells.cu -- cell list of an orthorhombic box on the GPU: the atoms within
// a cutoff of an atom lie in its own and the adjoining cells, so that the
// neighbour searches of the geometry (tb_geom.cu, the reference's getHaloAtoms,
// withSP2_deltaH.cpp:372-501) and of the charge model's features (tb_mlp.cu)
// look at tens of candidates instead of at every atom.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <cmath>

#include "tb_cells.cuh"

namespace tb {

namespace {

__global__ void k_cell_of(int natoms, const double *__restrict__ xyz, const CellGrid g, int32_t *__restrict__ cell,
                          int32_t *__restrict__ count)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= natoms) return;
    int c[3];
    for (int d = 0; d < 3; d++) c[d] = g.index(d, xyz[3 * i + d]);
    const int id = (c[0] * g.nc[1] + c[1]) * g.nc[2] + c[2];
    cell[i] = id;
    atomicAdd(count + id, 1);
}

// start[c] = atoms in the cells before c; count is left as each cell's cursor
__global__ void __launch_bounds__(1024) k_cell_scan(int ncells, int32_t *__restrict__ count, int32_t *__restrict__ start)
{
    __shared__ int32_t part[1024];
    const int t = threadIdx.x, len = (ncells + 1023) / 1024, c0 = min(ncells, t * len), c1 = min(ncells, c0 + len);
    int32_t s = 0;
    for (int c = c0; c < c1; c++) s += count[c];
    part[t] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int32_t v = t >= o ? part[t - o] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int32_t at = part[t] - s;
    for (int c = c0; c < c1; c++) {
        const int32_t k = count[c];
        start[c] = at;
        count[c] = at;
        at += k;
    }
    if (t == 1023) start[ncells] = part[1023];
}

__global__ void k_cell_fill(int natoms, const int32_t *__restrict__ cell, int32_t *__restrict__ cursor,
                            int32_t *__restrict__ atom)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < natoms) atom[atomicAdd(cursor + cell[i], 1)] = i;
}

// each cell's atoms in ascending order (the sums over neighbours then have one
// order), with their positions and species beside them: an atom's place is the
// number of smaller ones in its cell
__global__ void k_cell_sort(int natoms, const int32_t *__restrict__ cell, const int32_t *__restrict__ start,
                            const int32_t *__restrict__ unsorted, const double *__restrict__ xyz,
                            const int32_t *__restrict__ species, int32_t *__restrict__ atom, float4 *__restrict__ pos)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= natoms) return;
    const int s = start[cell[i]], e = start[cell[i] + 1];
    int at = s;
    for (int k = s; k < e; k++) at += unsorted[k] < i;
    atom[at] = i;
    pos[at] = make_float4((float)xyz[3 * i], (float)xyz[3 * i + 1], (float)xyz[3 * i + 2],
                          __int_as_float(species ? species[i] : 0));
}

}  // namespace

bool cell_grid(int natoms, const double *xyz, const double box[3], double rc, CellGrid &g)
{
    double lo[3], hi[3];
    for (int d = 0; d < 3; d++) {
        lo[d] = INFINITY;
        hi[d] = -INFINITY;
        g.box[d] = box[d];
        g.nc[d] = 1;  // one cell, should the positions not sort into more
        g.lo[d] = g.scale[d] = 0.0;
    }
    for (int i = 0; i < natoms; i++)
        for (int d = 0; d < 3; d++) {
            const double v = xyz[3 * i + d];
            if (!(std::fabs(v) < 1e9)) return false;  // NaN, infinite or absurd: no cells
            lo[d] = std::min(lo[d], v);
            hi[d] = std::max(hi[d], v);
        }
    const double side = rc * (1.0 + 1e-6);
    // no more cells than a few per atom, however far apart the atoms are
    const double most = 4.0 * natoms + 64;
    double want[3];
    for (int d = 0; d < 3; d++) {
        const double span = box[d] > 0 ? box[d] : hi[d] - lo[d];
        if (!(span < 1e12)) return false;
        want[d] = std::min(std::floor(span / side), most);  // span / side may be infinite
    }
    while (std::max(1.0, want[0]) * std::max(1.0, want[1]) * std::max(1.0, want[2]) > most)
        for (int d = 0; d < 3; d++) want[d] = std::floor(want[d] / 1.5);
    for (int d = 0; d < 3; d++) {
        // a periodic edge with fewer than three cells would meet the same cell
        // on both sides: one cell then, all of whose atoms are candidates
        const double span = box[d] > 0 ? box[d] : hi[d] - lo[d];
        g.nc[d] = box[d] > 0 && want[d] < 3 ? 1 : std::max(1, (int)want[d]);
        g.lo[d] = box[d] > 0 ? 0.0 : lo[d];
        g.scale[d] = span > 0 ? g.nc[d] / span : 0.0;
    }
    return true;
}

size_t cell_bytes(int natoms, const CellGrid &g)
{
    const size_t nc = (size_t)g.nc[0] * g.nc[1] * g.nc[2];
    return sizeof(float4) * natoms + sizeof(int32_t) * (3 * (size_t)natoms + 2 * nc + 1);
}

void cell_build(cudaStream_t st, int natoms, const double *d_xyz, const int32_t *d_species, CellGrid &g, void *scratch)
{
    const int nc = g.nc[0] * g.nc[1] * g.nc[2];
    float4 *pos = reinterpret_cast<float4 *>(scratch);
    int32_t *atom = reinterpret_cast<int32_t *>(pos + natoms), *cell = atom + natoms, *unsorted = cell + natoms,
            *count = unsorted + natoms, *start = count + nc;
    cudaMemsetAsync(count, 0, sizeof(int32_t) * nc, st);
    k_cell_of<<<(natoms + 255) / 256, 256, 0, st>>>(natoms, d_xyz, g, cell, count);
    k_cell_scan<<<1, 1024, 0, st>>>(nc, count, start);
    k_cell_fill<<<(natoms + 255) / 256, 256, 0, st>>>(natoms, cell, count, unsorted);
    k_cell_sort<<<(natoms + 255) / 256, 256, 0, st>>>(natoms, cell, start, unsorted, d_xyz, d_species, atom, pos);
    g.start = start;
    g.atom = atom;
    g.pos = pos;
}

}  // namespace tb
