// FP64 sweeps: the heat, Himeno and radius-4 star functors instantiated with double.
//
// The reference's functors are templates on the element type, and two of its applications run
// in double (HeatDiffusion: Grid<double>, HeatDiffusion/src/heat_appfis.hpp:72; Triton:
// Triton/src/triton_appfis.hpp:108-122).  These kernels are those functors in double with every
// multiply and add rounded separately in the reference's order (explicit __d*_rn, no FMA
// contraction), so they reproduce the reference's CPU path built with double bit for bit.  They
// are also the precision reference of the engine: the FP32, FP16-storage, mixed-precision and
// time-blocked forms state their error against these results.
//
// FP64 arithmetic on a GB300 runs at a small fraction of the FP32 rate (2 lanes per SM and clock, a warp
// instruction every 16 cycles), so these sweeps are bounded by the FP64 pipe, not by HBM; they are not
// a fast path.  What counts is the number of FP64 warp instructions: interior points are numbered along
// their rows and dealt to threads in that order, so every lane has a point whatever the row length (a
// 32-wide block left a quarter of them idle at nx = 65), and nothing that can be done exactly in
// integers is done in FP64.  Neighbours come through the read-only cache.  G points/s before and now: heat
// 1000 x 777 45.4 / 57.5 (8 FP64 instructions a point), Himeno 65 x 65 x 129 7.1 / 11.6 with gosa, 8.3 / 13.9
// without, 257 x 257 x 129 11.6 / 14.4, star 100^3 15.1 / 19.7, 255 x 256 x 200 18.0 / 18.1.
#include "gb_common.cuh"

namespace {

constexpr int NT = 256;  // threads per block

// 2 v, the same value as the product: an exponent step in the integer pipe, but for zeros, subnormals,
// values next to overflow, infinities and NaN (out of line: inlined, the product would be formed for
// every value and then selected).
__device__ __noinline__ double twice_product(double v) { return __dmul_rn(2.0, v); }
__device__ __forceinline__ double twice(double v)
{
    const int hi = __double2hiint(v);
    if ((unsigned)((hi & 0x7ff00000) - 0x00100000) >= 0x7fd00000u) return twice_product(v);
    return __hiloint2double(hi + 0x00100000, __double2loint(v));
}

// The thread's place among the rows of nx points: row and column from 0, or row >= rows when it has none.
__device__ __forceinline__ void place(size_t q, unsigned nx, size_t points, unsigned* row, unsigned* col)
{
    if (points <= 0xffffffffu) {  // uniform
        const unsigned p = (unsigned)q;
        *row = p / nx;
        *col = p - *row * nx;
    } else {
        *row = (unsigned)(q / nx);
        *col = (unsigned)(q - (size_t)*row * nx);
    }
}

__global__ void __launch_bounds__(NT) heat2d_f64(const double* __restrict__ cur, double* __restrict__ nxt, int nx, int ny, int px, double cx,
                                                 double cy)
{
    const gb::BlockId bid = gb::grid_wait();
    const size_t points = (size_t)nx * ny, q = (size_t)bid.x * NT + threadIdx.x;
    if (q >= points) return;
    unsigned row, col;
    place(q, nx, points, &row, &col);
    const size_t c = (size_t)(row + 1) * px + col + 1;
    const double v = __ldg(cur + c), two_c = twice(v);
    const double x = __dmul_rn(cx, __dsub_rn(__dadd_rn(__ldg(cur + c - 1), __ldg(cur + c + 1)), two_c));
    const double y = __dmul_rn(cy, __dsub_rn(__dadd_rn(__ldg(cur + c - px), __ldg(cur + c + px)), two_c));
    nxt[c] = __dadd_rn(__dadd_rn(v, x), y);
}

struct CoefF64 {
    const double* f[12];  // a0 a1 a2 a3 b0 b1 b2 c0 c1 c2 bnd wrk1
};

// Himeno/src/himeno_appfis.hpp:178-198 in double, hk planes per thread; ss^2 summed per thread and block
// (fixed order) where gosa is asked for, the block partials folded in block order by fold_f64 into
// gosa[it].  The sum over a warp takes 5 FP64 instructions, as many as 5 points' operations: one plane per
// thread spent 39 instructions per point, 33 without the sum, this 35.5 with 4.
__global__ void __launch_bounds__(NT) himeno_f64(CoefF64 cf, const double* __restrict__ p, double* __restrict__ w2, int nx, int ny, int nz, int px,
                                                 int py, int hk, unsigned plane_blocks, double omega, double* __restrict__ partials)
{
    const gb::BlockId bid = gb::grid_wait();
    const unsigned zc = bid.x / plane_blocks;
    const size_t points = (size_t)nx * ny, q = (size_t)(bid.x - zc * plane_blocks) * NT + threadIdx.x;
    double g = 0.0;
    if (q < points) {
        unsigned row, col;
        place(q, nx, points, &row, &col);
        const long long sy = px, sz = (long long)px * py;
        size_t c = (size_t)(1 + zc * hk) * sz + (size_t)(row + 1) * sy + col + 1;
#pragma unroll 1
        for (int k = 1 + (int)zc * hk; k < 1 + (int)(zc + 1) * hk && k <= nz; k++, c += sz) {
            auto P = [&](int di, int dj, int dk) { return __ldg(p + c + di + dj * sy + dk * sz); };
            auto C = [&](int n) { return __ldg(cf.f[n] + c); };
            double s0 = __dmul_rn(C(0), P(1, 0, 0));
            s0 = __dadd_rn(s0, __dmul_rn(C(1), P(0, 1, 0)));
            s0 = __dadd_rn(s0, __dmul_rn(C(2), P(0, 0, 1)));
            s0 = __dadd_rn(s0, __dmul_rn(C(4), __dadd_rn(__dsub_rn(__dsub_rn(P(1, 1, 0), P(1, -1, 0)), P(-1, 1, 0)), P(-1, -1, 0))));
            s0 = __dadd_rn(s0, __dmul_rn(C(5), __dadd_rn(__dsub_rn(__dsub_rn(P(0, 1, 1), P(0, -1, 1)), P(0, 1, -1)), P(0, -1, -1))));
            s0 = __dadd_rn(s0, __dmul_rn(C(6), __dadd_rn(__dsub_rn(__dsub_rn(P(1, 0, 1), P(-1, 0, 1)), P(1, 0, -1)), P(-1, 0, -1))));
            s0 = __dadd_rn(s0, __dmul_rn(C(7), P(-1, 0, 0)));
            s0 = __dadd_rn(s0, __dmul_rn(C(8), P(0, -1, 0)));
            s0 = __dadd_rn(s0, __dmul_rn(C(9), P(0, 0, -1)));
            s0 = __dadd_rn(s0, C(11));
            const double p0 = P(0, 0, 0);
            const double ss = __dmul_rn(__dsub_rn(__dmul_rn(s0, C(3)), p0), C(10));
            w2[c] = __dadd_rn(p0, __dmul_rn(omega, ss));
            if (partials) g = __dadd_rn(g, __dmul_rn(ss, ss));
        }
    }
    if (!partials) return;
    // block sum in a fixed order: warp shuffles, then the warp sums by another
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g = __dadd_rn(g, __shfl_down_sync(0xffffffffu, g, o));
    __shared__ double ws[NT / 32];
    const int t = threadIdx.x;
    if ((t & 31) == 0) ws[t >> 5] = g;
    __syncthreads();
    if (t < 32) {
        double s = t < NT / 32 ? ws[t] : 0.0;
#pragma unroll
        for (int o = NT / 64; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_down_sync(0xffffffffu, s, o));
        if (t == 0) partials[bid.x] = s;
    }
}

// Planes per thread: more share a sum, but a small grid then has too few blocks.  The fullest SM's blocks follow one
// another on its FP64 pipe, 2.5 us for a plane of a block and 0.5 for its sum.  Us per sweep with 1 / 2 / 3 / 4 planes,
// with gosa (without, 1 is the fastest or as fast): 24^3 9.3 / 12.0 / 14.6 / 17.2; 33 x 33 x 65 15.3 / 17.1 / 14.7 / 17.3;
// 300 x 24 x 24 21.8 / 23.0 / 22.4 / 27.3; 65^3 30.5 / 28.8 / 30.6 / 27.5; 64 x 64 x 128 48.5 / 45.4 / 46.8 / 48.7;
// 100^3 84.6 / 81.2 / 81.6 / 82.7; 257 x 257 x 129 656 / 608 / 597 / 588; without 552 / 553 / 559 / 558.
int planes_per_thread(size_t plane_blocks, int nz, bool gosa)
{
    const size_t sms = gb::sm_count();
    int best = 1;
    double cost = 1e30;
    for (int hk = 1; hk <= 4; hk++) {
        const size_t blocks = plane_blocks * ((nz + hk - 1) / hk);
        const double c = (double)((blocks + sms - 1) / sms) * (2.5 * hk + (gosa ? 0.5 : 0.0));
        if (c < cost) {
            cost = c;
            best = hk;
        }
    }
    return best;
}

// One block folds n partials: each thread a contiguous run in order, then the runs in thread order.
__global__ void __launch_bounds__(1024) fold_f64(const double* part, size_t n, double* out)
{
    gb::grid_wait();
    __shared__ double sh[1024];
    const size_t per = (n + 1023) / 1024, b = (size_t)threadIdx.x * per, e = b + per < n ? b + per : n;
    double s = 0.0;
    for (size_t q = b; q < e; q++) s = __dadd_rn(s, part[q]);
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = 512; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) sh[threadIdx.x] = __dadd_rn(sh[threadIdx.x], sh[threadIdx.x + w]);
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0];
}

struct StarWeightsF64 {
    double w[5];
};

// FDTD3d/src/fdtd3d_appfis.hpp:129-143 (mode 0) and the weighted form (mode 1) in double.
template <int MODE>
__global__ void __launch_bounds__(NT) star_r4_f64(const double* __restrict__ cur, double* __restrict__ nxt, int nx, int ny, int px, int py,
                                                  unsigned plane_blocks, double coeff, StarWeightsF64 wt)
{
    const gb::BlockId bid = gb::grid_wait();
    constexpr int R = 4;
    const unsigned k = bid.x / plane_blocks;
    const size_t points = (size_t)nx * ny, q = (size_t)(bid.x - k * plane_blocks) * NT + threadIdx.x;
    if (q >= points) return;
    unsigned row, col;
    place(q, nx, points, &row, &col);
    const long long sy = px, sz = (long long)px * py;
    const size_t c = (size_t)(R + k) * sz + (size_t)(R + row) * sy + R + col;
    double v = MODE == 0 ? __ldg(cur + c) : __dmul_rn(wt.w[0], __ldg(cur + c));
#pragma unroll
    for (int s = 1; s <= R; s++) {
        const double sx = __dadd_rn(__ldg(cur + c - s), __ldg(cur + c + s));
        const double syy = __dadd_rn(__ldg(cur + c - s * sy), __ldg(cur + c + s * sy));
        const double szz = __dadd_rn(__ldg(cur + c - s * sz), __ldg(cur + c + s * sz));
        const double ring = __dadd_rn(__dadd_rn(sx, syy), szz);
        v = MODE == 0 ? __dadd_rn(v, ring) : __dadd_rn(v, __dmul_rn(wt.w[s], ring));
    }
    if (MODE == 0) v = __dmul_rn(v, coeff);
    nxt[c] = v;
}

}  // namespace

extern "C" {

int appfis_gb_heat2d_f64(double* a, double* b, int nx, int ny, int pitch, int iters, double cx, double cy, int* cur_index,
                         void* stream)
{
    if (!a || !b || a == b) return gb::fail(APPFIS_GB_EINVAL, "heat2d_f64: null or aliased buffers");
    if (nx < 1 || ny < 1 || pitch < nx + 2 || iters < 0) return gb::fail(APPFIS_GB_EINVAL, "heat2d_f64: bad dims");
    cudaStream_t st = gb::as_stream(stream);
    double* buf[2] = {a, b};
    const size_t blocks = ((size_t)nx * ny + NT - 1) / NT;
    if (blocks > 0x7fffffffu) return gb::fail(APPFIS_GB_EINVAL, "heat2d_f64: grid too large");
    int ci = 0;
    for (int it = 0; it < iters; it++, ci = 1 - ci) gb::launch(heat2d_f64, (unsigned)blocks, NT, 0, st, buf[ci], buf[1 - ci], nx, ny, pitch, cx, cy);
    GB_TRY(gb::launched("heat2d_f64"));
    if (cur_index) *cur_index = ci;
    return APPFIS_GB_OK;
}

int appfis_gb_himeno_f64(const double* const* coef, double* p, double* wrk2, int nx, int ny, int nz, int pitch, int iters,
                         double omega, double* dev_gosa, int* cur_index, void* stream)
{
    if (!coef || !p || !wrk2 || p == wrk2) return gb::fail(APPFIS_GB_EINVAL, "himeno_f64: null or aliased buffers");
    if (nx < 1 || ny < 1 || nz < 1 || nz > 65535 || pitch < nx + 2 || iters < 0)
        return gb::fail(APPFIS_GB_EINVAL, "himeno_f64: bad dims");
    CoefF64 cf;
    for (int n = 0; n < 12; n++) {
        if (!coef[n]) return gb::fail(APPFIS_GB_EINVAL, "himeno_f64: null coefficient field %d", n);
        cf.f[n] = coef[n];
    }
    cudaStream_t st = gb::as_stream(stream);
    const size_t pb = ((size_t)nx * ny + NT - 1) / NT;
    const int hk = planes_per_thread(pb, nz, dev_gosa != nullptr);
    const size_t nblk = pb * ((nz + hk - 1) / hk);
    if (nblk > 0x7fffffffu) return gb::fail(APPFIS_GB_EINVAL, "himeno_f64: grid too large");
    void* ws = nullptr;
    if (dev_gosa) GB_TRY(gb::workspace(gb::WS_F64_PARTIALS, sizeof(double) * nblk, &ws));
    double* part = reinterpret_cast<double*>(ws);
    double* buf[2] = {p, wrk2};
    int ci = 0;
    for (int it = 0; it < iters; it++, ci = 1 - ci) {
        gb::launch(himeno_f64, (unsigned)nblk, NT, 0, st, cf, buf[ci], buf[1 - ci], nx, ny, nz, pitch, ny + 2, hk, (unsigned)pb, omega, part);
        if (dev_gosa) gb::launch(fold_f64, 1, 1024, 0, st, part, nblk, dev_gosa + it);
    }
    GB_TRY(gb::launched("himeno_f64"));
    if (cur_index) *cur_index = ci;
    return APPFIS_GB_OK;
}

int appfis_gb_star_r4_f64(double* a, double* b, int nx, int ny, int nz, int pitch, int iters, int mode, double coeff,
                          const double* weights, int* cur_index, void* stream)
{
    if (!a || !b || a == b) return gb::fail(APPFIS_GB_EINVAL, "star_r4_f64: null or aliased buffers");
    if (nx < 1 || ny < 1 || nz < 1 || nz > 65535 || pitch < nx + 8 || iters < 0)
        return gb::fail(APPFIS_GB_EINVAL, "star_r4_f64: bad dims");
    if (mode != 0 && mode != 1) return gb::fail(APPFIS_GB_EINVAL, "star_r4_f64: mode %d", mode);
    if (mode == 1 && !weights) return gb::fail(APPFIS_GB_EINVAL, "star_r4_f64: weighted mode needs 5 weights");
    StarWeightsF64 w = {{0, 0, 0, 0, 0}};
    if (weights)
        for (int n = 0; n < 5; n++) w.w[n] = weights[n];
    cudaStream_t st = gb::as_stream(stream);
    double* buf[2] = {a, b};
    const size_t pb = ((size_t)nx * ny + NT - 1) / NT;
    if (pb * nz > 0x7fffffffu) return gb::fail(APPFIS_GB_EINVAL, "star_r4_f64: grid too large");
    const unsigned grd = (unsigned)(pb * nz);
    int ci = 0;
    for (int it = 0; it < iters; it++, ci = 1 - ci) {
        if (mode == 0) gb::launch(star_r4_f64<0>, grd, NT, 0, st, buf[ci], buf[1 - ci], nx, ny, pitch, ny + 8, (unsigned)pb, coeff, w);
        else gb::launch(star_r4_f64<1>, grd, NT, 0, st, buf[ci], buf[1 - ci], nx, ny, pitch, ny + 8, (unsigned)pb, coeff, w);
    }
    GB_TRY(gb::launched("star_r4_f64"));
    if (cur_index) *cur_index = ci;
    return APPFIS_GB_OK;
}

}  // extern "C"
