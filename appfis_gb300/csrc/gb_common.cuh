// Shared plumbing of the C-ABI library: status codes, the last-error message, argument checks,
// CUDA error capture and a grow-only per-device workspace.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <string>

#include "appfis_gb.h"

namespace gb {

// Records msg as this thread's last error and returns `code`.
int fail(int code, const char* fmt, ...);
// Returns OK, or records the CUDA error of `e` (with `what`) and returns APPFIS_GB_ECUDA.
int cuda_status(cudaError_t e, const char* what);
// Checks the launch that just happened on this thread.
inline int launched(const char* what) { return cuda_status(cudaGetLastError(), what); }

// Launch on `st` as a programmatic dependent of what runs before it there.  None of the kernels lets
// its dependents start early, so a kernel still starts when the one before has finished; but the
// stream then goes from one to the next in ~1.4 us instead of 3.1-4.1 (a plain launch waits for the
// finished grid's completion to be polled, in steps of ~2 us; an empty kernel of 608 blocks, 200 in
// a row: 4.10 -> 1.45 us each, recorded in a graph 1.22 -> 0.97).  Every kernel launched this way begins
// with grid_wait(), which costs a block a little: a kernel of hundreds of thousands of small blocks is
// launched plainly (the FP16 coefficient copies of the Himeno set-up took 870 -> 1208 us with it).
template <class... P, class... A>
cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args)
{
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Waits until everything before this kernel on its stream has finished and its writes are visible;
// every thread calls it before its first access to global memory.  The block's index is read behind
// the wait, in the same statement, so that no load whose address comes from it can be moved ahead
// (and as the special register, so that it stays uniform: an index that went through an ordinary
// register cost the heat tiles 12%).  A kernel that has no use for the index declares no pointer
// __restrict__: its loads are then ordinary ones, which are not moved across the wait, where one of data that is
// promised constant for the kernel's time may be.
struct BlockId {
    unsigned x, y, z;
};
__device__ __forceinline__ BlockId grid_wait()
{
    BlockId b;
    asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, %%ctaid.x;\n\tmov.u32 %1, %%ctaid.y;\n\tmov.u32 %2, %%ctaid.z;"
                 : "=r"(b.x), "=r"(b.y), "=r"(b.z)::"memory");
    return b;
}

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Device workspace: one grow-only allocation per (device, slot), reused across calls.  Calls
// that use the same slot on the same device must not overlap on the GPU.
enum Slot { WS_REDUCE = 0, WS_JOB_A, WS_JOB_B, WS_JOB_C, WS_JOB_D, WS_JOB_E, WS_JOB_F, WS_LIFE_C, WS_LIFE_D, WS_LIFE_E, WS_LIFE_F, WS_FLOOD_Z, WS_FLOOD_SRC, WS_F64_PARTIALS, WS_FLOOD_MAPS, WS_FLOOD_ORDER, WS_SLOTS };
int workspace(int slot, size_t bytes, void** out);
// True if that slot holds at least `bytes` already, so that workspace() will not allocate.
bool workspace_holds(int slot, size_t bytes);
// Gives that slot's memory back.
void workspace_drop(int slot);
// Device memory for one call, ordered on `st` (allocated and freed by the stream, so calls on other
// streams and threads never share it): from a pool per device that keeps up to 256 MB between
// calls and gives back what is over that when the device is next synchronised.  False, with no error
// left behind, if there is none (the caller then takes a path without it).
bool scratch_alloc(size_t bytes, cudaStream_t st, void** out);
void scratch_free(void* p, cudaStream_t st);
// True while `st` records a graph (or cannot tell): a call then allocates nothing of its own.
bool capturing(cudaStream_t st);
// Copies a host table to the device on `st`; the source may go as soon as it returns, and the host does not wait
// for earlier work of the stream.  Through pinned memory of the library's own: whether a copy from
// pageable memory has been read when the call returns is the platform's choice, and one whose GPU reads pageable
// memory itself need not have.  Up to 6 copies a device are under way, then the oldest is waited for.
int upload(void* dst, const void* src, size_t bytes, cudaStream_t st);

inline unsigned ceil_div(size_t a, size_t b) { return (unsigned)((a + b - 1) / b); }

// Splits n planes into the fewest chunks of at most `target` planes, all of (nearly) equal size,
// and returns the chunk size.
inline int balanced_chunk(int n, int target)
{
    const int chunks = (n + target - 1) / target;
    return (n + chunks - 1) / chunks;
}

// Chunk size for a grid with `per_chunk` CTAs per chunk of planes: among the balanced chunks of
// about lo..hi planes (steps of 8), the one whose grid fills `slots` resident CTAs best over its
// waves, counting the `halo` planes each chunk reads beyond its own as waste.
inline int wave_chunk(int n, int lo, int hi, long long per_chunk, long long slots, int halo)
{
    int best = balanced_chunk(n, lo);
    double score = -1.0;
    for (int t = lo; t <= hi; t += 8) {
        const int kz = balanced_chunk(n, t), chunks = (n + kz - 1) / kz;
        const long long ctas = per_chunk * chunks, waves = (ctas + slots - 1) / slots;
        const double sc = (double)ctas / (double)(waves * slots) * kz / (kz + halo);
        if (sc > score + 1e-9) {
            score = sc;
            best = kz;
        }
    }
    return best;
}

// Number of SMs of the current device (cached).
int sm_count();

// The non-blocking stream the _job entry points run on, one per device (created on first use).
int job_stream(cudaStream_t* out);

// Test plan of the bounded device-side waits (set by appfis_gb_test_stall_next): returns true,
// with the plan's limit, once for the next call of the given kind, and clears the plan.
enum TestStall { TEST_NONE = 0, TEST_FLOOD_BARRIER = 1, TEST_TMA_SHORTFALL = 2 };
bool take_test_stall(int kind, unsigned long long* limit);

#define GB_TRY(expr)                 \
    do {                             \
        int _st = (expr);            \
        if (_st != APPFIS_GB_OK)     \
            return _st;              \
    } while (0)

#define GB_CUDA(expr) GB_TRY(::gb::cuda_status((expr), #expr))

}  // namespace gb
