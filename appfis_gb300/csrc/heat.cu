// 2-D heat (explicit 5-point Jacobi, FP32) on a DUAL grid with a Dirichlet ghost ring.
//
// Reference functor: HeatDiffusion/src/heat_appfis.hpp:166-174 (3-D FP64), restated in 2-D FP32:
//     next = c + cx*((l + r) - 2c) + cy*((u + d) - 2c)
// driven once per iteration by Execute2D -> Kernel2D (Appfis/Runtime_CUDA.hpp:345-369,1217-1230).
// The arithmetic below uses explicit round-to-nearest intrinsics in exactly that order (no FMA
// contraction), so every point is bit-identical to the reference's CPU path.
//
// The 1024^2 workload is 8.4 MB for both buffers, so it lives in L2; one launch per sweep would
// be launch-bound.  heat2d_bands therefore runs 8 sweeps per launch on a tile held on chip
// (overlapped tiling: the tile plus an 8-deep halo is loaded once, each sweep shrinks the valid
// region by one cell, the centre tile is written back).  Ghost-ring cells are loaded and held
// constant, so Dirichlet boundaries are exact for any number of sweeps.
#include <cmath>

#include "f32x2.cuh"
#include "gb_common.cuh"

namespace {

__device__ __forceinline__ float heat_point(float c, float l, float r, float u, float d, float cx, float cy)
{
    float two_c = __fmul_rn(2.0f, c);
    float x = __fmul_rn(cx, __fsub_rn(__fadd_rn(l, r), two_c));
    float y = __fmul_rn(cy, __fsub_rn(__fadd_rn(u, d), two_c));
    return __fadd_rn(__fadd_rn(c, x), y);
}

__global__ void __launch_bounds__(256) heat2d_sweep_k(const float* __restrict__ cur, float* __restrict__ nxt, int nx,
                                                       int ny, int pitch, float cx, float cy)
{
    const gb::BlockId bid = gb::grid_wait();
    const int i = 1 + bid.x * blockDim.x + threadIdx.x;
    const int j = 1 + bid.y * blockDim.y + threadIdx.y;
    if (i > nx || j > ny) return;
    const size_t c = (size_t)j * pitch + i;
    nxt[c] = heat_point(__ldg(cur + c), __ldg(cur + c - 1), __ldg(cur + c + 1), __ldg(cur + c - pitch), __ldg(cur + c + pitch),
                        cx, cy);
}

// Two points of a row at once, each lane's operations those of heat_point: packed additions and
// subtractions, except the x sums, whose operands straddle register pairs.  2c is c + c (the same value),
// and the products are scalar, because the code generator contracts a packed product into the packed
// addition that takes it.  12 instructions for two points instead of 18.
__device__ __forceinline__ float2 heat_pair(float2 c, float2 l, float2 r, float2 u, float2 d, float cx, float cy)
{
    namespace f2 = gb::f2;
    const float2 two_c = f2::add(c, c);
    const float2 tx = f2::sub(make_float2(__fadd_rn(l.x, r.x), __fadd_rn(l.y, r.y)), two_c);
    const float2 ty = f2::sub(f2::add(u, d), two_c);
    const float2 x = make_float2(__fmul_rn(cx, tx.x), __fmul_rn(cx, tx.y));
    const float2 y = make_float2(__fmul_rn(cy, ty.x), __fmul_rn(cy, ty.y));
    return f2::add(f2::add(c, x), y);
}

// Overlapped tiling: a CTA of W warps holds a 128 x (HR W) region in registers for up to 8 sweeps and writes
// the 112 x (HR W - 16) tile in its middle.  A warp owns a band of HR rows, a lane 4 columns of it, so that the
// x neighbours at a lane's edges come by shuffle and only a band's first and last row go through shared
// memory (one 16-byte vector each per lane and sweep, one barrier).  A sweep works down the band and
// replaces the rows as it goes, keeping one old row.  Ghost-ring cells and cells outside the field
// keep their values; every other cell of the region is updated each sweep (those outside the shrinking
// valid window only feed cells that are not written back).
constexpr int HS = 8;             // sweeps per launch, and halo width
constexpr int HTX = 128 - 2 * HS;  // output columns

template <int G> struct HeatVec;  // G floats that are aligned together
template <> struct HeatVec<1> { typedef float type; };
template <> struct HeatVec<2> { typedef float2 type; };
template <> struct HeatVec<4> { typedef float4 type; };

// MASK: the region reaches the ghost ring or beyond the field: loads are guarded and only interior cells
// are updated and stored.
template <int W, int HR, int G, bool MASK>
__device__ __forceinline__ void heat_tile(const float* __restrict__ cur, float* __restrict__ nxt, int nx, int ny, int pitch, int ns, float cx,
                                          float cy, int bx, int by, float4 (&top)[2][W][32], float4 (&bot)[2][W][32])
{
    typedef typename HeatVec<G>::type V;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int x = bx * HTX - HS + 4 * lane, y0 = 1 + by * (HR * W - 2 * HS) - HS + HR * w;  // padded coordinates of the first cell
    float v[HR][4];
    bool in[4];  // MASK: an interior column
#pragma unroll
    for (int c = 0; c < 4; c++) in[c] = !MASK || (x + c >= 1 && x + c <= nx);
#pragma unroll
    for (int r = 0; r < HR; r++) {
        const float* row = cur + (ptrdiff_t)(y0 + r) * pitch + x;
        if (MASK) {
            const bool yin = y0 + r >= 0 && y0 + r <= ny + 1;
#pragma unroll
            for (int c = 0; c < 4; c++) v[r][c] = yin && x + c >= 0 && x + c <= nx + 1 ? __ldg(row + c) : 0.0f;
        } else {
#pragma unroll
            for (int c = 0; c < 4; c += G) *reinterpret_cast<V*>(&v[r][c]) = __ldg(reinterpret_cast<const V*>(row + c));
        }
    }
    const float4 z4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
    for (int s = 0; s < ns; s++) {
        // one barrier per sweep: a half is rewritten two sweeps later, after every thread has passed the
        // next sweep's barrier and so finished reading it
        const int q = s & 1;
        top[q][w][lane] = make_float4(v[0][0], v[0][1], v[0][2], v[0][3]);
        bot[q][w][lane] = make_float4(v[HR - 1][0], v[HR - 1][1], v[HR - 1][2], v[HR - 1][3]);
        __syncthreads();
        const float4 up = w > 0 ? bot[q][w - 1][lane] : z4;
        const float4 dn = w < W - 1 ? top[q][w + 1][lane] : z4;
        float2 u01 = make_float2(up.x, up.y), u23 = make_float2(up.z, up.w);  // the row above, before this sweep
#pragma unroll
        for (int r = 0; r < HR; r++) {
            const float lf = __shfl_up_sync(0xffffffffu, v[r][3], 1), rt = __shfl_down_sync(0xffffffffu, v[r][0], 1);
            const float2 c01 = make_float2(v[r][0], v[r][1]), c23 = make_float2(v[r][2], v[r][3]);
            const float2 d01 = r < HR - 1 ? make_float2(v[r < HR - 1 ? r + 1 : 0][0], v[r < HR - 1 ? r + 1 : 0][1]) : make_float2(dn.x, dn.y);
            const float2 d23 = r < HR - 1 ? make_float2(v[r < HR - 1 ? r + 1 : 0][2], v[r < HR - 1 ? r + 1 : 0][3]) : make_float2(dn.z, dn.w);
            const float2 h01 = heat_pair(c01, make_float2(lf, c01.x), make_float2(c01.y, c23.x), u01, d01, cx, cy);
            const float2 h23 = heat_pair(c23, make_float2(c01.y, c23.x), make_float2(c23.y, rt), u23, d23, cx, cy);
            if (!MASK || (y0 + r >= 1 && y0 + r <= ny)) {  // uniform in the warp
                v[r][0] = in[0] ? h01.x : c01.x;
                v[r][1] = in[1] ? h01.y : c01.y;
                v[r][2] = in[2] ? h23.x : c23.x;
                v[r][3] = in[3] ? h23.y : c23.y;
            }
            u01 = c01;
            u23 = c23;
        }
    }
    if (lane < HS / 4 || lane >= 32 - HS / 4) return;
#pragma unroll
    for (int r = 0; r < HR; r++) {
        if (HR * w + r < HS || HR * w + r >= HR * W - HS) continue;
        float* row = nxt + (ptrdiff_t)(y0 + r) * pitch + x;
        if (MASK) {
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (in[c] && y0 + r <= ny) row[c] = v[r][c];
        } else {
#pragma unroll
            for (int c = 0; c < 4; c += G) *reinterpret_cast<V*>(row + c) = *reinterpret_cast<V*>(&v[r][c]);
        }
    }
}

template <int W, int HR, int G>
__global__ void __launch_bounds__(32 * W, HR == 8 ? 24 / W : 4) heat2d_bands(const float* __restrict__ cur, float* __restrict__ nxt, int nx, int ny, int pitch,
                                                            int ns, float cx, float cy)
{
    const gb::BlockId bid = gb::grid_wait();
    __shared__ float4 top[2][W][32], bot[2][W][32];
    const int bx = (int)bid.x, by = (int)bid.y, x0 = bx * HTX - HS, y0 = 1 + by * (HR * W - 2 * HS) - HS;
    if (x0 >= 1 && y0 >= 1 && x0 + 127 <= nx && y0 + HR * W - 1 <= ny)  // the whole region lies on interior cells
        heat_tile<W, HR, G, false>(cur, nxt, nx, ny, pitch, ns, cx, cy, bx, by, top, bot);
    else
        heat_tile<W, HR, G, true>(cur, nxt, nx, ny, pitch, ns, cx, cy, bx, by, top, bot);
}

long long heat_tiles(int rows, int nx, int ny) { return (long long)gb::ceil_div(nx + 1, HTX) * gb::ceil_div(ny, rows - 2 * HS); }

// Rows of a CTA's region: 64 (8 warps of 8 rows, 112 x 48 tiles: 1.5 points computed per point written), unless a
// small grid's launch is shorter with 32 (8 warps of 4 rows: 2.3, but a third as long), 20 (10 warps of 2 rows: 5.7)
// or 96 (12 warps of 8 rows: 1.4).  A launch lasts about 3.2 us and 3.3 for each tile of the fullest SM, 2.4 and 1.6
// with 32 rows, 2.1 and 1.15 with 20; 96 rows 9 us if every SM has one tile at most.  Us per 8 sweeps with 20 / 32 / 64 /
// 96 rows: 64^2 3.2 / 3.7 / 5.7 / 7.3; 250 x 190 3.4 / 3.9; 512^2 7.9 / 5.7 / 6.4 / 8.7; 777 x 900 14.8 / 7.5 / 6.5 / 8.8; 1024^2
// 21.7 / 9.9 / 9.6 / 8.8; 1500^2 42 / 16.7 / 13.4 / 14.9; 2048^2 75 / 28 / 22.4 / 23.8; 4096^2 283 / 98 / 72 / 72.  32 rows as 4 warps
// of 8: 4.6, 4.7, 6.0, 7.8, 10.6; 64 rows as 16 warps of 4: 5.8, 6.5, 6.6, 6.7, 10.8.
// The 4 x 4 register blocks that this replaced (48 x 32 tiles, four edge vectors per thread and sweep through
// shared memory): 64^2 6.4, 512^2 8.4, 777 x 900 14.5, 1024^2 15.7, 1500^2 26.4, 2048^2 40.5, 4096^2 139.  Bound by
// instruction issue and the sweep's barrier; 16 warps of 8 rows 10.7 and more up to 1024^2.
int heat_region(int nx, int ny)
{
    const double sms = gb::sm_count();
    auto full = [&](int rows) { return std::ceil((double)heat_tiles(rows, nx, ny) / sms); };
    const int rows[4] = {64, 32, 20, 96};
    const double cost[4] = {3.2 + 3.3 * full(64), 2.4 + 1.6 * full(32), 2.1 + 1.15 * full(20), full(96) <= 1 ? 9.0 : 1e30};
    return rows[std::min_element(cost, cost + 4) - cost];
}

// The copies' width goes by the alignment of the rows (region rows start on 4-element boundaries).
template <int W, int HR>
void launch_bands(const float* cur, float* nxt, int nx, int ny, int pitch, int ns, float cx, float cy, cudaStream_t st)
{
    const dim3 grd(gb::ceil_div(nx + 1, HTX), gb::ceil_div(ny, HR * W - 2 * HS));
    const unsigned long long align = (unsigned long long)pitch * sizeof(float) | reinterpret_cast<uintptr_t>(cur) | reinterpret_cast<uintptr_t>(nxt);
    auto kern = align % 16 == 0 ? heat2d_bands<W, HR, 4> : (align % 8 == 0 ? heat2d_bands<W, HR, 2> : heat2d_bands<W, HR, 1>);
    gb::launch(kern, grd, 32 * W, 0, st, cur, nxt, nx, ny, pitch, ns, cx, cy);
}

int check_heat(const void* a, const void* b, int nx, int ny, int pitch)
{
    if (!a || !b || a == b) return gb::fail(APPFIS_GB_EINVAL, "heat2d: null or aliased buffers");
    if (nx < 1 || ny < 1 || pitch < nx + 2) return gb::fail(APPFIS_GB_EINVAL, "heat2d: bad size %d x %d pitch %d", nx, ny, pitch);
    return APPFIS_GB_OK;
}

}  // namespace

extern "C" {

int appfis_gb_heat2d_sweep(const float* cur, float* next, int nx, int ny, int pitch, float cx, float cy, void* stream)
{
    GB_TRY(check_heat(cur, next, nx, ny, pitch));
    dim3 blk(64, 4), grd(gb::ceil_div(nx, 64), gb::ceil_div(ny, 4));
    gb::launch(heat2d_sweep_k, grd, blk, 0, gb::as_stream(stream), cur, next, nx, ny, pitch, cx, cy);
    return gb::launched("heat2d_sweep");
}

int appfis_gb_heat2d(float* a, float* b, int nx, int ny, int pitch, int iters, float cx, float cy, int* cur_index,
                     void* stream)
{
    GB_TRY(check_heat(a, b, nx, ny, pitch));
    if (iters < 0) return gb::fail(APPFIS_GB_EINVAL, "heat2d: negative iteration count");
    cudaStream_t st = gb::as_stream(stream);
    const int rows = heat_region(nx, ny);
    float* buf[2] = {a, b};
    int ci = 0;
    for (int done = 0; done < iters;) {
        const int ns = std::min(HS, iters - done);
        auto launch = rows == 64 ? launch_bands<8, 8> : rows == 32 ? launch_bands<8, 4> : rows == 20 ? launch_bands<10, 2> : launch_bands<12, 8>;
        launch(buf[ci], buf[1 - ci], nx, ny, pitch, ns, cx, cy, st);
        ci = 1 - ci;
        done += ns;
    }
    GB_TRY(gb::launched("heat2d_bands"));
    if (cur_index) *cur_index = ci;
    return APPFIS_GB_OK;
}

int appfis_gb_heat2d_job(float* field, int nx, int ny, int iters, float cx, float cy, double* stats)
{
    if (!field || nx < 1 || ny < 1 || iters < 0) return gb::fail(APPFIS_GB_EINVAL, "heat2d_job: bad arguments");
    cudaStream_t st;
    GB_TRY(gb::job_stream(&st));
    const int px = nx + 2, py = ny + 2;
    const size_t bytes = sizeof(float) * (size_t)px * py;
    void *a, *b, *res;
    GB_TRY(gb::workspace(gb::WS_JOB_A, bytes, &a));
    GB_TRY(gb::workspace(gb::WS_JOB_B, bytes, &b));
    GB_TRY(gb::workspace(gb::WS_JOB_F, 64, &res));
    GB_CUDA(cudaMemcpyAsync(a, field, bytes, cudaMemcpyHostToDevice, st));
    GB_CUDA(cudaMemcpyAsync(b, a, bytes, cudaMemcpyDeviceToDevice, st));  // ghost ring in both buffers
    int ci = 0;
    GB_TRY(appfis_gb_heat2d((float*)a, (float*)b, nx, ny, px, iters, cx, cy, &ci, st));
    float* latest = ci == 0 ? (float*)a : (float*)b;
    double s[3] = {0, 0, 0};
    if (stats) {
        const int box[6] = {1, nx + 1, 1, ny + 1, 0, 1};
        for (int op = 0; op < 3; op++) {
            GB_TRY(appfis_gb_reduce(latest, APPFIS_GB_F32, px, py, box, op, (char*)res + 8 * op, st));
        }
        GB_CUDA(cudaMemcpyAsync(s, res, sizeof s, cudaMemcpyDeviceToHost, st));
    }
    GB_CUDA(cudaMemcpyAsync(field, latest, bytes, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    if (stats) for (int k = 0; k < 3; k++) stats[k] = s[k];
    return APPFIS_GB_OK;
}

}  // extern "C"
