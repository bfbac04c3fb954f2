// Periodic ghost-cell refresh of a padded field on the device.
//
// Reference: for one rank with periodic boundaries the halo exchange packs each face, sends it
// to itself through MPI and unpacks it into the opposite ghost layers, axis by axis
// (Appfis/Communication.hpp:612-678, pack/unpack Appfis/Runtime.hpp:916-1173; on GPU builds via
// pinned host buffers every iteration, Appfis/Runtime_CUDA.hpp:743-1198).  Axis a's low ghost
// layer g takes interior layer dim-2G+g and its high ghost layer dim-G+g takes layer G+g, over
// the full extent of the other axes, X first, then Y, then Z, so edges and corners come out as
// in the reference.  Every ghost cell so ends up with the interior cell that it wraps to in all its
// axes (each axis is at least 3G long, so that cell is no ghost itself): here one launch writes all of
// them, reading interior cells only.  200 x 190 x 180 FP32, G = 1: axis by axis in three launches
// 12.3 us, so 3.4; 512^3 29 -> 9.
#include "gb_common.cuh"

namespace {

// Padded extents and the ghost width per axis (0 on an axis the field does not have).
struct Ghosts {
    int dx, dy, dz, gx, gy, gz;
};

__device__ __forceinline__ int wrapped(int c, int d, int g) { return c < g ? c + d - 2 * g : (c >= d - g ? c - d + 2 * g : c); }

constexpr int SEG = 256;  // cells of a row per warp

// Blocks 0 .. row_blocks - 1: whole rows of the y and z ghost layers, a warp per segment of a row (z layers
// first, then the y layers of the planes between them).  The others: the x ghosts of the interior
// rows, one cell per thread, the 2 gx cells of a row side by side.
template <class E>
__global__ void __launch_bounds__(256) periodic_ghosts(E* __restrict__ f, Ghosts g, unsigned row_blocks, long long rows, int segs, long long cells)
{
    const gb::BlockId bid = gb::grid_wait();
    const size_t plane = (size_t)g.dx * g.dy;
    if (bid.x < row_blocks) {
        const int lane = threadIdx.x & 31;
        const long long task = (long long)bid.x * 8 + (threadIdx.x >> 5), r = task / segs;
        if (r >= rows) return;
        const int x0 = (int)(task - r * segs) * SEG, x1 = min(x0 + SEG, g.dx);
        int y, z;
        const long long zrows = 2LL * g.gz * g.dy;
        if (r < zrows) {
            const int layer = (int)(r / g.dy);
            y = (int)(r - (long long)layer * g.dy);
            z = layer < g.gz ? layer : g.dz - 2 * g.gz + layer;
        } else {
            const long long q = r - zrows;
            const int k = (int)(q / (2 * g.gy)), layer = (int)(q - (long long)k * 2 * g.gy);
            z = g.gz + k;
            y = layer < g.gy ? layer : g.dy - 2 * g.gy + layer;
        }
        E* __restrict__ d = f + (size_t)z * plane + (size_t)y * g.dx;
        const E* __restrict__ s = f + (size_t)wrapped(z, g.dz, g.gz) * plane + (size_t)wrapped(y, g.dy, g.gy) * g.dx;
#pragma unroll 8
        for (int x = x0 + lane; x < x1; x += 32) d[x] = s[wrapped(x, g.dx, g.gx)];
    } else {
        const long long t = (long long)(bid.x - row_blocks) * 256 + threadIdx.x;
        if (t >= cells) return;
        const unsigned per = 2u * (unsigned)g.gx, ny = (unsigned)(g.dy - 2 * g.gy);
        const long long r = t / per;
        const int layer = (int)(t - r * per), k = (int)(r / ny), j = (int)(r - (long long)k * ny);
        const int x = layer < g.gx ? layer : g.dx - 2 * g.gx + layer;
        E* row = f + (size_t)(g.gz + k) * plane + (size_t)(g.gy + j) * g.dx;
        row[x] = row[wrapped(x, g.dx, g.gx)];
    }
}

template <class E>
int fill(void* field, int ndim, const int* pd, int G, cudaStream_t st)
{
    const Ghosts g = {pd[0], ndim > 1 ? pd[1] : 1, ndim > 2 ? pd[2] : 1, G, ndim > 1 ? G : 0, ndim > 2 ? G : 0};
    const long long rows = 2LL * g.gz * g.dy + 2LL * g.gy * (g.dz - 2 * g.gz);
    const long long cells = 2LL * g.gx * (g.dy - 2 * g.gy) * (g.dz - 2 * g.gz);
    const int segs = (g.dx + SEG - 1) / SEG;
    const unsigned row_blocks = gb::ceil_div((size_t)rows * segs, 8), cell_blocks = gb::ceil_div((size_t)cells, 256);
    gb::launch(periodic_ghosts<E>, row_blocks + cell_blocks, 256, 0, st, reinterpret_cast<E*>(field), g, row_blocks, rows, segs, cells);
    return gb::launched("periodic_ghosts");
}

}  // namespace

extern "C" {

int appfis_gb_ghost_periodic(void* field, int elem_size, int ndim, const int* padded_dims, int ghost, void* stream)
{
    if (!field || !padded_dims || ndim < 1 || ndim > 3 || ghost < 0) return gb::fail(APPFIS_GB_EINVAL, "ghost_periodic: bad arguments");
    if (ghost == 0) return APPFIS_GB_OK;
    for (int a = 0; a < ndim; a++)
        if (padded_dims[a] < 3 * ghost) return gb::fail(APPFIS_GB_EINVAL, "ghost_periodic: axis %d too small for %d ghost layers", a, ghost);
    cudaStream_t st = gb::as_stream(stream);
    switch (elem_size) {
    case 1: return fill<uint8_t>(field, ndim, padded_dims, ghost, st);
    case 2: return fill<uint16_t>(field, ndim, padded_dims, ghost, st);
    case 4: return fill<uint32_t>(field, ndim, padded_dims, ghost, st);
    case 8: return fill<unsigned long long>(field, ndim, padded_dims, ghost, st);
    default: return gb::fail(APPFIS_GB_EINVAL, "ghost_periodic: element size %d", elem_size);
    }
}

}  // extern "C"
