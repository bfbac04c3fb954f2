// Box reductions MAX / MIN / SUM over a padded field (the reference's Execute{1,2,3}DReduce).
//
// Reference: GPU path Appfis/Runtime_CUDA.hpp:554-740 launches one thread per element of the
// WHOLE padded array masked by the Config box, writes block partials into the grid's `next`
// buffer (so a SINGLE grid's input is overwritten), loops multi-pass kernels, then copies one
// scalar to the host and synchronises; CPU path Appfis/Runtime.hpp:597-913.  Seeds: MAX starts
// from numeric_limits<T>::min(), MIN from max(), SUM from 0 (kept here, including MAX's
// smallest-positive seed for floating types).
//
// Here: the box's elements are numbered along its rows and dealt to threads round robin, so a warp
// reads 32 neighbours whatever the row length, eight loads in flight per thread; the position moves
// by fixed steps and two carries, no division per element.  Each block leaves one partial and a
// second launch folds them in block order (a box of up to 4096 elements is one block and one
// launch): fixed grid, fixed order, deterministic, and nothing kept between calls.
// This part has 2 FP64 lanes per SM and clock, so FP32 elements are compared as floats, and summed
// as three floats in packed pairs (FloatSum) that reach a double once per 128 elements: FP32 SUM of 200 x 190 x 180
// 38 us with a double add and conversion per element, 12.1 so (MAX 38 -> 10.2); 512^3 547 -> 135 us.
// Bound there by the index arithmetic (a third of the instructions) and HBM (4.7 TB/s MAX); FP64 by
// its pipe (272 us at 512^3).  The input is never written.
#include <cfloat>
#include <climits>
#include <mutex>
#include <type_traits>

#include "f32x2.cuh"
#include "gb_common.cuh"

namespace {

template <class T> __device__ __forceinline__ T max_seed();
template <> __device__ __forceinline__ float max_seed<float>() { return FLT_MIN; }
template <> __device__ __forceinline__ double max_seed<double>() { return DBL_MIN; }
template <> __device__ __forceinline__ int32_t max_seed<int32_t>() { return INT_MIN; }
template <class T> __device__ __forceinline__ T min_seed();
template <> __device__ __forceinline__ float min_seed<float>() { return FLT_MAX; }
template <> __device__ __forceinline__ double min_seed<double>() { return DBL_MAX; }
template <> __device__ __forceinline__ int32_t min_seed<int32_t>() { return INT_MAX; }

// The type a thread hands to its block: the element's own for MAX and MIN, double or int64 for SUM.
template <class T, int OP> struct Acc { typedef T type; };
template <> struct Acc<float, APPFIS_GB_SUM> { typedef double type; };
template <> struct Acc<int32_t, APPFIS_GB_SUM> { typedef long long type; };
// The type of a partial and of the result.
template <class T> struct Wide { typedef double type; };
template <> struct Wide<int32_t> { typedef long long type; };

template <class T, int OP>
__device__ __forceinline__ typename Acc<T, OP>::type seed()
{
    typedef typename Acc<T, OP>::type A;
    return OP == APPFIS_GB_MAX ? (A)max_seed<T>() : (OP == APPFIS_GB_MIN ? (A)min_seed<T>() : (A)0);
}

template <int OP, class A>
__device__ __forceinline__ A combine(A a, A b)
{
    return OP == APPFIS_GB_MAX ? (b > a ? b : a) : (OP == APPFIS_GB_MIN ? (b < a ? b : a) : a + b);
}

template <int OP, class A>
__device__ __forceinline__ A block_reduce(A v, A neutral, A* sh)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = combine<OP>(v, __shfl_down_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : neutral;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = combine<OP>(v, __shfl_down_sync(0xffffffffu, v, o));
    }
    return v;
}

using gb::f2::two_sum;

// A thread's running sum of floats, in two lanes: hi takes the element, mid what hi rounds off and lo what mid
// rounds off.  Of n elements of a lane (n <= 64) and the sum S of their magnitudes, mid holds at most n 2^-24 S and
// lo n^2 2^-48 S, so only lo's own roundings are lost, at most n^3 2^-72 S <= 2^-54 S, whatever the values: less
// than one rounding of a double sum, and 128 elements reach the thread's double in one addition.
// Infinities, NaN and sums beyond the float range leave a component that is not finite: the thread
// then starts again in doubles.
struct FloatSum {
    static constexpr int BATCH = 128;
    float2 hi = {0.0f, 0.0f}, mid = {0.0f, 0.0f}, lo = {0.0f, 0.0f};
    double total = 0.0;
    bool finite = true;
    __device__ __forceinline__ void add(float2 v)
    {
        float2 e, r;
        hi = two_sum(hi, v, e);
        mid = two_sum(mid, e, r);
        lo = gb::f2::add(lo, r);
    }
    __device__ __forceinline__ void flush()
    {
        float e, f, g;
        const float h = two_sum(hi.x, hi.y, e), m = two_sum(two_sum(mid.x, mid.y, f), e, g);
        finite = finite && fabsf(h) <= FLT_MAX && fabsf(m) <= FLT_MAX;
        total += (double)h + ((double)m + (double)__fadd_rn(__fadd_rn(lo.x, lo.y), __fadd_rn(f, g)));
        hi = mid = lo = make_float2(0.0f, 0.0f);
    }
};

// The box: W x ny x nz elements from `first` (element offset of its corner), and what one stride of
// all threads moves a position by.
struct Box {
    size_t first, n;          // elements
    unsigned W, ny;           // row length, rows per plane
    unsigned dcol, drow;      // the stride's columns, rows within a plane
    long long step;           // and as an element offset
    long long row_end, plane_end;  // offsets added when a row or a plane is passed
};

// A position in the box; Off: 32-bit offsets where the box spans less than 2^31 elements.
template <class Off>
struct Cursor {
    Off at;
    unsigned col, row;  // their sums with the stride's may pass 2^31
    __device__ __forceinline__ void to(const Box& b, size_t e, int px, size_t plane)
    {
        const size_t r = e / b.W, k = r / b.ny;
        col = (unsigned)(e - r * b.W);
        row = (unsigned)(r - k * b.ny);
        at = (Off)(k * plane + (size_t)row * px + col);
    }
    __device__ __forceinline__ void next(const Box& b)
    {
        at += (Off)b.step;
        col += b.dcol;
        row += b.drow;
        if (col >= b.W) {
            col -= b.W;
            row += 1;
            at += (Off)b.row_end;
        }
        if (row >= b.ny) {
            row -= b.ny;
            at += (Off)b.plane_end;
        }
    }
};

constexpr int RED_THREADS = 256;
constexpr int RED_PER_SM = 4;        // blocks per SM (3 to 8, and 12 or 16 loads in flight, measured within 5%)
constexpr int RED_ONE_BLOCK = 4096;  // elements up to which one block does it all

template <class W>
__device__ __forceinline__ void put_result(void* result, W w)
{
    *reinterpret_cast<W*>(result) = w;
}

template <class T, int OP, class Off>
__global__ void __launch_bounds__(RED_THREADS, RED_PER_SM) reduce_part(const T* __restrict__ field, Box b, int px, size_t plane,
                                                          typename Wide<T>::type* __restrict__ partials, void* __restrict__ result)
{
    const gb::BlockId bid = gb::grid_wait();
    typedef typename Acc<T, OP>::type A;
    typedef typename Wide<T>::type Wd;
    constexpr int U = 8;  // loads in flight
    __shared__ A sh[32];
    const size_t stride = (size_t)gridDim.x * RED_THREADS, e0 = (size_t)bid.x * RED_THREADS + threadIdx.x;
    const T* __restrict__ f = field + b.first;
    A v = seed<T, OP>();
    if (e0 < b.n) {
        Cursor<Off> c;
        c.to(b, e0, px, plane);
        size_t left = (b.n - e0 + stride - 1) / stride;  // this thread's elements
        if constexpr (std::is_same<T, float>::value && OP == APPFIS_GB_SUM) {
            FloatSum t;
            int m = 0;
            size_t q = left;
            for (; q >= U; q -= U) {
                float x[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    x[u] = __ldg(f + c.at);
                    c.next(b);
                }
#pragma unroll
                for (int u = 0; u < U; u += 2) t.add(make_float2(x[u], x[u + 1]));
                if ((m += U) == FloatSum::BATCH) {
                    t.flush();
                    m = 0;
                }
            }
            for (; q > 0; q--) {
                t.add(make_float2(__ldg(f + c.at), 0.0f));
                c.next(b);
            }
            t.flush();
            v = t.total;
            if (!t.finite) {
                v = 0.0;
                c.to(b, e0, px, plane);
                for (; left > 0; left--) {
                    v += (double)__ldg(f + c.at);
                    c.next(b);
                }
            }
        } else {
            for (; left >= U; left -= U) {
                T x[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    x[u] = __ldg(f + c.at);
                    c.next(b);
                }
                A w[U];
#pragma unroll
                for (int u = 0; u < U; u++) w[u] = (A)x[u];
                if (OP == APPFIS_GB_SUM) {
#pragma unroll
                    for (int o = U / 2; o > 0; o /= 2)
#pragma unroll
                        for (int u = 0; u < o; u++) w[u] += w[u + o];
                    v += w[0];
                } else {
#pragma unroll
                    for (int u = 0; u < U; u++) v = combine<OP>(v, w[u]);
                }
            }
            for (; left > 0; left--) {
                v = combine<OP>(v, (A)__ldg(f + c.at));
                c.next(b);
            }
        }
    }
    v = block_reduce<OP>(v, seed<T, OP>(), sh);
    if (threadIdx.x == 0) {
        if (result) put_result(result, (Wd)v);
        else partials[bid.x] = (Wd)v;
    }
}

template <class T, int OP>
__global__ void __launch_bounds__(RED_THREADS) reduce_fold(const typename Wide<T>::type* partials, int n, void* result)
{
    gb::grid_wait();
    typedef typename Wide<T>::type Wd;
    __shared__ Wd sh[32];
    const Wd neutral = (Wd)seed<T, OP>();
    Wd v = neutral;
    for (int k = threadIdx.x; k < n; k += RED_THREADS) v = combine<OP>(v, partials[k]);
    v = block_reduce<OP>(v, neutral, sh);
    if (threadIdx.x == 0) put_result(result, v);
}

int reduce_blocks(long long n)
{
    if (n <= RED_ONE_BLOCK) return 1;
    return (int)std::min<long long>((n + RED_THREADS * 16 - 1) / (RED_THREADS * 16), (long long)RED_PER_SM * gb::sm_count());
}

// partials: one value per block, for grids of more than one
template <class T, int OP>
int launch_op(const T* f, int px, int py, const int* x, int grid, void* partials, void* res, cudaStream_t st)
{
    Box b;
    const size_t plane = (size_t)px * py;
    b.W = x[1] - x[0];
    b.ny = x[3] - x[2];
    b.first = x[4] * plane + (size_t)x[2] * px + x[0];
    b.n = (size_t)b.W * b.ny * (x[5] - x[4]);
    const size_t stride = (size_t)grid * RED_THREADS, srow = stride / b.W;
    b.dcol = (unsigned)(stride % b.W);
    b.drow = (unsigned)(srow % b.ny);
    b.step = (long long)(srow / b.ny * plane) + (long long)b.drow * px + b.dcol;
    b.row_end = px - (long long)b.W;
    b.plane_end = (long long)plane - (long long)b.ny * px;
    typedef typename Wide<T>::type Wd;
    Wd* part = reinterpret_cast<Wd*>(partials);
    // the last offset a cursor can reach: one stride past the box
    const bool small = (double)plane * (x[5] - x[4] + 2) + (double)b.step < 2147483647.0;
    auto kern = small ? reduce_part<T, OP, int> : reduce_part<T, OP, long long>;
    gb::launch(kern, grid, RED_THREADS, 0, st, f, b, px, plane, part, grid == 1 ? res : nullptr);
    if (grid > 1) gb::launch(reduce_fold<T, OP>, 1, RED_THREADS, 0, st, part, grid, res);
    return gb::launched("reduce");
}

template <class T>
int launch_reduce(const void* field, int px, int py, const int* b, int op, int grid, void* partials, void* res, cudaStream_t st)
{
    const T* f = reinterpret_cast<const T*>(field);
    switch (op) {
    case APPFIS_GB_MAX: return launch_op<T, APPFIS_GB_MAX>(f, px, py, b, grid, partials, res, st);
    case APPFIS_GB_MIN: return launch_op<T, APPFIS_GB_MIN>(f, px, py, b, grid, partials, res, st);
    default: return launch_op<T, APPFIS_GB_SUM>(f, px, py, b, grid, partials, res, st);
    }
}

int launch_reduce(int dtype, const void* field, int px, int py, const int* b, int op, int grid, void* partials, void* res, cudaStream_t st)
{
    switch (dtype) {
    case APPFIS_GB_F32: return launch_reduce<float>(field, px, py, b, op, grid, partials, res, st);
    case APPFIS_GB_F64: return launch_reduce<double>(field, px, py, b, op, grid, partials, res, st);
    default: return launch_reduce<int32_t>(field, px, py, b, op, grid, partials, res, st);
    }
}

long long box_elements(const int* b) { return (long long)(b[1] - b[0]) * (b[3] - b[2]) * (b[5] - b[4]); }

// ---------------------------------------------------------------- allocation-free variant
// Some callers cannot allocate device memory at the moment they need a reduction: a host
// framework whose caching allocator has reserved the device memory, a library embedded in a
// runtime that owns every allocation, or a latency-critical loop that cannot take the implicit
// synchronisation of a first cudaMalloc/cudaFree.  For them the same reduction kernel can take
// its scratch (one partial per block) from a fixed array that is part of the library image instead of
// the grow-only workspace.  Of its 64 KiB 8160 partials are used; the kernel has at most 4 blocks per
// SM (608 on a GB300), so every box fits on current GPUs.  Every device that loads the library keeps this array until the process exits
// (under lazy module loading the runtime commits it on the first use of the module on a device).
constexpr size_t NOALLOC_SCRATCH_BYTES = 64 * 1024;
constexpr size_t NOALLOC_MAX_PARTIALS = (NOALLOC_SCRATCH_BYTES - 256) / sizeof(double);
static __device__ __align__(256) unsigned char g_reduce_scratch[NOALLOC_SCRATCH_BYTES];

constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};

// Device address of the scratch array on the current device.  On the host the array's name
// only stands for the symbol, so its address is looked up once per device (first call on that
// device, with it current) and cached.
int noalloc_scratch(void** out)
{
    int dev = 0;
    GB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return gb::fail(APPFIS_GB_EINVAL, "reduce_noalloc: device %d out of range", dev);
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_reduce_scratch);
        if (e != cudaSuccess || !p) return gb::cuda_status(e != cudaSuccess ? e : cudaErrorInvalidSymbol, "cudaGetSymbolAddress(reduce scratch)");
        g_noalloc_addr[dev] = p;
    }
    *out = g_noalloc_addr[dev];
    return APPFIS_GB_OK;
}

}  // namespace

extern "C" {

int appfis_gb_reduce_noalloc(const void* field, int dtype, int px, int py, const int* box, int op, void* dev_result,
                             void* stream)
{
    if (!field || !box || !dev_result) return gb::fail(APPFIS_GB_EINVAL, "reduce_noalloc: null argument");
    if (op < APPFIS_GB_MAX || op > APPFIS_GB_SUM) return gb::fail(APPFIS_GB_EINVAL, "reduce_noalloc: unknown op %d", op);
    for (int a = 0; a < 3; a++)
        if (box[2 * a] < 0 || box[2 * a + 1] < box[2 * a]) return gb::fail(APPFIS_GB_EINVAL, "reduce_noalloc: bad box axis %d", a);
    if (box[1] > px || box[3] > py || px < 1 || py < 1) return gb::fail(APPFIS_GB_EINVAL, "reduce_noalloc: box outside the field");
    if (box[0] == box[1] || box[2] == box[3] || box[4] == box[5]) return gb::fail(APPFIS_GB_EINVAL, "reduce_noalloc: empty box");
    if (dtype != APPFIS_GB_F32 && dtype != APPFIS_GB_F64 && dtype != APPFIS_GB_I32)
        return gb::fail(APPFIS_GB_EINVAL, "reduce_noalloc: unknown dtype %d", dtype);
    const int grid = reduce_blocks(box_elements(box));
    if ((size_t)grid > NOALLOC_MAX_PARTIALS)
        return gb::fail(APPFIS_GB_EINVAL, "reduce_noalloc: %d partial sums needed, the fixed scratch holds %zu", grid,
                        NOALLOC_MAX_PARTIALS);
    void* part = nullptr;
    GB_TRY(noalloc_scratch(&part));
    return launch_reduce(dtype, field, px, py, box, op, grid, part, dev_result, gb::as_stream(stream));
}

int appfis_gb_reduce(const void* field, int dtype, int px, int py, const int* box, int op, void* dev_result, void* stream)
{
    if (!field || !box || !dev_result) return gb::fail(APPFIS_GB_EINVAL, "reduce: null argument");
    if (op < APPFIS_GB_MAX || op > APPFIS_GB_SUM) return gb::fail(APPFIS_GB_EINVAL, "reduce: unknown op %d", op);
    for (int a = 0; a < 3; a++)
        if (box[2 * a] < 0 || box[2 * a + 1] < box[2 * a]) return gb::fail(APPFIS_GB_EINVAL, "reduce: bad box axis %d", a);
    if (box[1] > px || box[3] > py || px < 1 || py < 1) return gb::fail(APPFIS_GB_EINVAL, "reduce: box outside the field");
    if (box[0] == box[1] || box[2] == box[3] || box[4] == box[5])
        return gb::fail(APPFIS_GB_EINVAL, "reduce: empty box");
    if (dtype != APPFIS_GB_F32 && dtype != APPFIS_GB_F64 && dtype != APPFIS_GB_I32)
        return gb::fail(APPFIS_GB_EINVAL, "reduce: unknown dtype %d", dtype);
    const int grid = reduce_blocks(box_elements(box));
    void* part;
    GB_TRY(gb::workspace(gb::WS_REDUCE, sizeof(double) * (size_t)grid, &part));
    return launch_reduce(dtype, field, px, py, box, op, grid, part, dev_result, gb::as_stream(stream));
}

int appfis_gb_reduce_host(const void* field, int dtype, int px, int py, const int* box, int op, double* result, void* stream)
{
    if (!result) return gb::fail(APPFIS_GB_EINVAL, "reduce_host: null result");
    void* d;
    GB_TRY(gb::workspace(gb::WS_JOB_F, 64, &d));
    cudaStream_t st = gb::as_stream(stream);
    GB_TRY(appfis_gb_reduce(field, dtype, px, py, box, op, d, st));
    union { double f; long long i; } u;
    GB_CUDA(cudaMemcpyAsync(&u, d, 8, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    *result = dtype == APPFIS_GB_I32 ? (double)u.i : u.f;
    return APPFIS_GB_OK;
}

}  // extern "C"
