// GameOfLife on a periodic grid: byte-per-cell (SWAR, 16 cells per thread per row) and
// bit-packed (32 cells per word) sweeps, pack/unpack, population count, whole-run job.
//
// Reference semantics (GameOfLife/src/game_appfis.hpp:121-135): a live cell whose 8-neighbour
// count is < 2 or > 4 is cleared in `next`; a dead cell with count 3 is set in `next`; any
// other cell leaves `next` untouched, so `next` keeps the state of two generations back (the
// DUAL grid's buffers swap every generation, Appfis/Runtime.hpp:318-319).  In bit-slice form:
//     new = (cur & keep & old) | (~cur & (birth | old)),  keep = (cnt in 2..4), birth = (cnt == 3).
// The periodic halo refresh of the reference (pack, MPI self-exchange, unpack every
// generation, Appfis/Communication.hpp:612-678) becomes index wrap-around inside the sweep.
//
// Layout: interior cells only, x fastest, row pitch nx bytes (u8) or nx/32 words (bits).
// The byte-per-cell sweep (life_u8_bulk) stages its rows in shared memory with bulk copies; the
// one-generation bit-packed sweep (life_bits_sweep) marches down a strip of rows per warp,
// keeping the row above / at / below in registers and exchanging the words at lane boundaries
// with warp shuffles.  Runs of 3 or more bit-packed generations (while a stream is recorded: 16), and byte
// runs that are worth the conversion to words and back, use life_bits_tb, which advances a region held in
// registers by up to 16 generations per launch.
#include "gb_common.cuh"
#include "tma.cuh"

namespace {

constexpr uint32_t FULL = 0xffffffffu;
constexpr uint32_t LSB = 0x01010101u;  // bit 0 of each byte
constexpr int LIFE_ROWS = 32;           // rows per warp task (bit-packed sweep)

// ------------------------------------------------------------------------------ rule logic
// Per byte lane (u8 form): cnt in 0..8 in each byte, c/o in {0,1} per byte.
template <int RULE>
__device__ __forceinline__ uint32_t rule_bytes(uint32_t cnt, uint32_t c, uint32_t o)
{
    uint32_t b0 = cnt & LSB, b1 = (cnt >> 1) & LSB, b2 = (cnt >> 2) & LSB, b3 = (cnt >> 3) & LSB;
    if (RULE == APPFIS_GB_LIFE_REFERENCE) {
        uint32_t birth = b0 & b1 & ~(b2 | b3);
        uint32_t keep = ~b3 & ((~b2 & b1) | (b2 & ~b1 & ~b0));
        return ((c & keep & o) | (~c & (birth | o))) & LSB;
    } else {
        return (b1 & ~(b2 | b3) & (b0 | c)) & LSB;
    }
}


// ------------------------------------------------------------------------------ generic form
// One thread per cell, any nx, ny (a few generations of rows that are not whole 16-byte vectors, or of
// a small grid).
template <int RULE>
__global__ void life_u8_generic(const uint8_t* __restrict__ cur, uint8_t* __restrict__ out, int nx, int ny)
{
    const gb::BlockId bid = gb::grid_wait();
    int i = bid.x * blockDim.x + threadIdx.x;
    int j = bid.y * blockDim.y + threadIdx.y;
    if (i >= nx || j >= ny) return;
    int im = i == 0 ? nx - 1 : i - 1, ip = i == nx - 1 ? 0 : i + 1;
    size_t rm = (size_t)(j == 0 ? ny - 1 : j - 1) * nx, r0 = (size_t)j * nx, rp = (size_t)(j == ny - 1 ? 0 : j + 1) * nx;
    uint32_t cnt = cur[rm + im] + cur[rm + i] + cur[rm + ip] + cur[r0 + im] + cur[r0 + ip] + cur[rp + im] + cur[rp + i] +
                   cur[rp + ip];
    uint32_t c = cur[r0 + i];
    uint32_t o = out[r0 + i];
    out[r0 + i] = (uint8_t)rule_bytes<RULE>(cnt, c, RULE == APPFIS_GB_LIFE_REFERENCE ? o : 0u);
}

// ------------------------------------------------------------------------------ u8 form, bulk-staged
struct RowU8 {         // 16 cells of one row, one per byte (SWAR)
    uint32_t w[4];     // the cells
    uint32_t s3[4];    // per byte: left + self + right
};

// A CTA owns a strip of UB_W cells (256 threads x 16) of UB_ROWS consecutive rows.  Each row it
// needs arrives in a shared-memory slot by bulk copies (the cur row with a 16-byte periodic halo
// on each side, and for output rows the t-1 row), UB_RING - 1 rows ahead of the row it computes,
// signalled on the slot's mbarrier: every copy is a contiguous run of up to 4 KB, and the rows in
// flight need no registers.  Each thread carries the row summaries of the rows above and at its
// output row and reads the row below from the slot (one 16-byte vector and the two neighbour
// words), so every row is summarised once.  Waits are bounded; a wait that gives up sets the
// device status word.
constexpr int UB_W = 4096;      // strip width in cells (bytes)
constexpr int UB_ROWS = 32;     // output rows per CTA
constexpr int UB_RING = 6;      // row slots
constexpr int UB_OLD = 16 + UB_W + 16;      // offset of the t-1 row in a slot
constexpr int UB_SLOT = UB_OLD + UB_W;      // 8224 bytes
constexpr int UB_SMEM = UB_RING * UB_SLOT + UB_RING * 8;

__device__ __forceinline__ RowU8 slot_row_u8(const unsigned char* s, int t)
{
    const unsigned char* p = s + 16 + 16 * t;
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t lw = *reinterpret_cast<const uint32_t*>(p - 4);   // cell x-1 in the top byte
    const uint32_t rw = *reinterpret_cast<const uint32_t*>(p + 16);  // cell x+16 in the low byte
    RowU8 r;
    r.w[0] = v.x;
    r.w[1] = v.y;
    r.w[2] = v.z;
    r.w[3] = v.w;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t prev = k == 0 ? lw : r.w[k - 1];
        const uint32_t next = k == 3 ? rw : r.w[k + 1];
        r.s3[k] = __funnelshift_l(prev, r.w[k], 8) + r.w[k] + __funnelshift_r(r.w[k], next, 8);
    }
    return r;
}

template <int RULE>
__global__ void __launch_bounds__(256) life_u8_bulk(const uint8_t* __restrict__ cur, uint8_t* __restrict__ out, int nx, int ny,
                                                     int strips, unsigned* __restrict__ status)
{
    const gb::BlockId bid = gb::grid_wait();
    extern __shared__ __align__(128) unsigned char ub[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(ub + UB_RING * UB_SLOT);
    const int t = threadIdx.x;
    const int strip = bid.x % strips, band = bid.x / strips;
    const int x0 = strip * UB_W, w = min(UB_W, nx - x0);
    const int j0 = band * UB_ROWS, j1 = min(j0 + UB_ROWS, ny);
    const int rbase = j0 - 1;  // row of slot 0, first use
    const bool active = 16 * t < w;
    if (gb::tma::smem_u32(ub) & 15u) {
        if (t == 0) atomicOr(status, (unsigned)gb::ST_SMEM_ALIGN);
        return;
    }
    if (t == 0) {
        for (int n = 0; n < UB_RING; n++) gb::tma::bar_init(&bar[n], 1);
        gb::tma::fence_init();
    }
    __syncthreads();
    int last_issued = rbase - 1;  // thread 0 only
    auto issue = [&](int r) {     // cur row r (periodic) with its halos; the t-1 row if r is an output row
        last_issued = r;
        const int n = (r - rbase) % UB_RING;
        unsigned char* d = ub + n * UB_SLOT;
        const int rr = r < 0 ? r + ny : (r >= ny ? r - ny : r);
        const uint8_t* row = cur + (size_t)rr * nx;
        const bool oldrow = RULE == APPFIS_GB_LIFE_REFERENCE && r >= j0 && r < j1;
        gb::tma::arrive_expect(&bar[n], 32 + w + (oldrow ? w : 0));
        gb::tma::load_1d(d, row + (x0 == 0 ? nx - 16 : x0 - 16), 16, &bar[n]);
        gb::tma::load_1d(d + 16, row + x0, w, &bar[n]);
        gb::tma::load_1d(d + 16 + w, row + (x0 + w == nx ? 0 : x0 + w), 16, &bar[n]);
        if (oldrow) gb::tma::load_1d(d + UB_OLD, out + (size_t)r * nx + x0, w, &bar[n]);
    };
    auto ready = [&](int r, uint64_t limit = 1000000000ull) {
        return gb::tma::wait(&bar[(r - rbase) % UB_RING], (unsigned)((r - rbase) / UB_RING) & 1u, limit);
    };
    auto slot = [&](int r) { return ub + ((r - rbase) % UB_RING) * UB_SLOT; };
    if (t == 0)
        for (int r = rbase; r < rbase + UB_RING && r <= j1; r++) issue(r);
    bool bad = !ready(rbase) || !ready(j0);
    RowU8 up = slot_row_u8(slot(rbase), t);
    RowU8 mid = slot_row_u8(slot(j0), t);
    bad = __syncthreads_or(bad);  // row j0-1 is read: its slot takes row j0-1+UB_RING
    if (t == 0 && !bad && rbase + UB_RING <= j1) issue(rbase + UB_RING);
    for (int j = j0; j < j1 && !bad; j++) {
        if (!ready(j + 1)) bad = true;
        const RowU8 dn = slot_row_u8(slot(j + 1), t);
        const uint4 o = RULE == APPFIS_GB_LIFE_REFERENCE ? *reinterpret_cast<const uint4*>(slot(j) + UB_OLD + 16 * t)
                                                         : make_uint4(0, 0, 0, 0);
        if (active && !bad) {
            const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
            uint32_t nw[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t cnt = up.s3[k] + (mid.s3[k] - mid.w[k]) + dn.s3[k];
                nw[k] = rule_bytes<RULE>(cnt, mid.w[k], ow[k]);
            }
            *reinterpret_cast<uint4*>(out + (size_t)j * nx + x0 + 16 * t) = make_uint4(nw[0], nw[1], nw[2], nw[3]);
        }
        up = mid;
        mid = dn;
        // row j's slot (cur read at step j-1, t-1 read now) takes row j + UB_RING
        bad = __syncthreads_or(bad);
        if (t == 0 && !bad && j + UB_RING <= j1) issue(j + UB_RING);
    }
    if (bad && t == 0) {  // a wait gave up: report and let the copies still in flight land
        atomicOr(status, (unsigned)gb::ST_TMA_TIMEOUT);
        for (int r = max(rbase, last_issued - UB_RING + 1); r <= last_issued; r++) ready(r, gb::tma::DRAIN_NS);
    }
}

// ------------------------------------------------------------------------------ bit-packed form
struct RowBits {
    uint32_t w;       // 32 cells
    uint32_t a0, a1;  // left + self + right as 2-bit slices
};

// New word from the row sums of the rows above, at and below (each left + self + right, 0..3).
// S = up + mid + dn is the 3x3 sum including the cell, so the neighbour count is S - c:
//   reference rule (S234 with the stale carry): a live cell keeps o when S is 3, 4 or 5 and dies
//     otherwise; a dead cell is born when S is 3 and otherwise keeps o;
//   B3/S23: a live cell survives when S is 3 or 4; a dead cell is born when S is 3.
// Every step is one explicit 3-input logic instruction (lop3).  The reference rule takes 8: 4 for the count,
// S = s0 + 2 (c1 + x + 2 y), 3 for the rule and 1 for the keep / birth select with the stale value; B3/S23 takes 6 in
// all.  S in binary is not formed: the tables are what an exhaustive search over networks of such
// instructions gave for the rule at every S that a cell can have (a live cell counts itself, so a live
// cell's S is never 0 and a dead one's never 9); it has no shorter one for the reference rule with s0 and c1.
// With S's bits and a window on them it was one more and two more: 16384^2, 64 generations 541 against 518 us
// (reference rule); B3/S23 455 with 7, 411 with 6.
// One 3-input logic instruction; LUT = f(0xF0, 0xCC, 0xAA) for the function f(a, b, c).
template <unsigned LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c)
{
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT));
    return d;
}
constexpr unsigned XOR3 = 0x96, MAJ3 = 0xE8;

template <int RULE>
__device__ __forceinline__ uint32_t life_combine(const RowBits& up, const RowBits& mid, const RowBits& dn, uint32_t o)
{
    const uint32_t s0 = lop3<XOR3>(up.a0, mid.a0, dn.a0);
    const uint32_t c = mid.w;
    if (RULE == APPFIS_GB_LIFE_REFERENCE) {
        const uint32_t c1 = lop3<MAJ3>(up.a0, mid.a0, dn.a0);
        const uint32_t x = lop3<XOR3>(up.a1, mid.a1, dn.a1);
        const uint32_t y = lop3<MAJ3>(up.a1, mid.a1, dn.a1);
        const uint32_t p = lop3<0x17>(s0, c1, x);  // not the majority
        const uint32_t q = lop3<0x42>(c1, x, c);   // c1 == x, and c the other way
        const uint32_t d = lop3<0x81>(y, p, q);    // all equal: live: S in 3..5; dead: S == 3
        return lop3<0x8E>(c, o, d);                // c ? o & d : o | d
    } else {
        const uint32_t e = lop3<0x7E>(up.a0, mid.a0, dn.a0);  // one or two
        const uint32_t p = lop3<0x17>(s0, up.a1, dn.a1);
        const uint32_t q = lop3<0x61>(e, up.a1, dn.a1);
        const uint32_t r = lop3<0x4A>(mid.a1, p, q);
        return lop3<0xE0>(r, s0, c);  // r & (s0 | c): live: S in 3..4; dead: S == 3
    }
}
struct RawBits {
    uint32_t w, lw, rw;
};

__device__ __forceinline__ RawBits load_raw_bits(const uint32_t* __restrict__ bits, int nw, int row, int xw, bool active,
                                                 int lane)
{
    const uint32_t* p = bits + (size_t)row * nw;
    RawBits r;
    r.w = active ? __ldg(p + xw) : 0u;
    r.lw = lane == 0 ? __ldg(p + (xw == 0 ? nw - 1 : xw - 1)) : 0u;
    r.rw = (active && (lane == 31 || xw + 1 >= nw)) ? __ldg(p + (xw + 1 >= nw ? 0 : xw + 1)) : 0u;
    return r;
}

__device__ __forceinline__ RowBits finish_row_bits(const RawBits& raw, int xw, int nw, int lane)
{
    uint32_t lw = __shfl_up_sync(FULL, raw.w, 1);
    uint32_t rw = __shfl_down_sync(FULL, raw.w, 1);
    if (lane == 0) lw = raw.lw;
    if (lane == 31 || xw + 1 >= nw) rw = raw.rw;
    const uint32_t w = raw.w;
    const uint32_t L = __funnelshift_l(lw, w, 1);  // bit b = cell x-1
    const uint32_t R = __funnelshift_r(w, rw, 1);  // bit b = cell x+1
    RowBits r;
    r.w = w;
    r.a0 = L ^ w ^ R;
    r.a1 = (L & w) | (R & (L ^ w));
    return r;
}

// Warp tasks: 32 words (1024 cells) per row over LIFE_ROWS rows, grid-stride, one row prefetched.
template <int RULE>
__global__ void __launch_bounds__(256) life_bits_sweep(const uint32_t* __restrict__ cur, uint32_t* __restrict__ out,
                                                        int nw, int ny, int strips, int rows, int tasks)
{
    const gb::BlockId bid = gb::grid_wait();
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int task = (bid.x * blockDim.x + threadIdx.x) >> 5; task < tasks; task += nwarps) {
        const int strip = task % strips, seg = task / strips;
        const int xw = strip * 32 + lane;
        const bool active = xw < nw;
        const int j0 = seg * rows, j1 = min(j0 + rows, ny);
        RowBits up = finish_row_bits(load_raw_bits(cur, nw, j0 == 0 ? ny - 1 : j0 - 1, xw, active, lane), xw, nw, lane);
        RowBits mid = finish_row_bits(load_raw_bits(cur, nw, j0, xw, active, lane), xw, nw, lane);
        RawBits rdn = load_raw_bits(cur, nw, j0 == ny - 1 ? 0 : j0 + 1, xw, active, lane);
        uint32_t o = (RULE == APPFIS_GB_LIFE_REFERENCE && active) ? out[(size_t)j0 * nw + xw] : 0u;
        for (int j = j0; j < j1; j++) {
            RawBits rnext = {0u, 0u, 0u};
            uint32_t onext = 0u;
            if (j + 1 < j1) {
                const int r2 = j + 2 >= ny ? j + 2 - ny : j + 2;
                rnext = load_raw_bits(cur, nw, r2, xw, active, lane);
                if (RULE == APPFIS_GB_LIFE_REFERENCE && active) onext = out[(size_t)(j + 1) * nw + xw];
            }
            const RowBits dn = finish_row_bits(rdn, xw, nw, lane);
            if (active) out[(size_t)j * nw + xw] = life_combine<RULE>(up, mid, dn, o);
            up = mid;
            mid = dn;
            rdn = rnext;
            o = onext;
        }
    }
}

// ------------------------------------------------------------------------------ bit-packed, time-blocked
// Up to TB_STEPS generations per launch on a region held in registers.  A CTA of 8 warps owns a region of
// 32 words x 8R rows (periodic wrap at load time, so it is a consistent periodic window even on the
// grid's last tiles) and writes the 30 words x (8R - 32) rows in its middle; a warp owns a band of R
// rows, a lane a column of words, both states of it (t and t-1) in registers.  x neighbours come by
// shuffle; of a band only the first and last row of a generation go through shared memory, one barrier a
// generation.  A generation works down the band and leaves the new state over the t-1 state (new(x) reads
// only old(x) and the current state), then the two change roles.  Lane 0 / 31 hold the halo words: their
// outer bits go stale by one cell per generation, which never reaches the output words for up to 31
// generations; rows go stale from the region's top and bottom by one row per generation, which never
// reaches the output rows for up to TB_STEPS generations.  The launch reads two planes and writes two planes
// (the next launch needs both), so global traffic per generation drops by ~TB_STEPS/1.5.
//
// Bound by the logic pipe (86% of its issue slots; 13.0 instructions executed per word and generation): a
// word costs its 10 lop3 (B3/S23: 8) and two funnel shifts and two shuffles, and no address, load or
// store.  (With the planes in shared memory, two loads and a store per word and generation and their
// loop: 17.8 there for 11 lop3, and 256-row tiles even on small grids.)
//
// Ragged rows: nw words whose last word holds only v = nx - 32*(nw - 1) cells (the rest of its
// bits 0).  Interior words are loaded as they are; the words past a row's end are put together
// from the two words that hold their 32 cells after the periodic wrap.  Needs nx >= 64.
constexpr int TB_STEPS = 16;  // generations per launch (max)
constexpr int TB_WARPS = 8;

// The tiles of a grid of nw words a row: `cols` columns of 30 words, and (rest > 0) one of the `rest` words that
// are left, `side` tiles of which, one above the other in the grid, stand side by side in a warp, each with its
// own two halo words: nothing but the lanes' places differs, as a stale outer bit is all that lanes of
// different tiles give each other.  A column of its own for the rest, us for 64 generations against this:
// 2080 x 30000 178 / 133, 4096^2 46.2 / 44.3, 6016 x 5000 76.6 / 73.4 (B3/S23 143 / 109, 40.0 / 37.4, 62.9 / 58.2).
struct LifeTiles {
    unsigned whole;  // tiles of whole columns, dealt along the rows
    int cols, rest, side;
};

// One lane's words of a region: word `q` of every row, or (general) the 32 cells that start r bits
// into word q, of which only `cnt` lie before the row's end and the others are the row's first.
struct WordSource {
    int q, r, cnt, nw;
    __device__ __forceinline__ void at(int word, int nx, int nwords)
    {
        nw = nwords;
        long long s = (32LL * word) % nx;
        if (s < 0) s += nx;
        q = (int)(s >> 5);
        r = (int)(s & 31);
        cnt = nx - (int)s;
    }
    __device__ __forceinline__ bool whole() const { return r == 0 && cnt >= 32; }  // the word as it is stored
    struct Parts {
        uint32_t lo, hi, first;
    };
    __device__ __forceinline__ Parts fetch(const uint32_t* __restrict__ row) const
    {
        Parts v = {__ldg(row + q), 0u, 0u};
        if (q + 1 < nw) v.hi = __ldg(row + q + 1);
        if (cnt < 32) v.first = __ldg(row);
        return v;
    }
    __device__ __forceinline__ uint32_t join(const Parts& v) const
    {
        const uint32_t w = __funnelshift_r(v.lo, v.hi, r);
        return cnt >= 32 ? w : (w & ((1u << cnt) - 1u)) | (v.first << cnt);
    }
};

// Row summary of one word for the bit-sliced neighbour count.  Lanes 0 / 31 get their own word
// back from the shuffles, so their outer bit is wrong; those lanes are the stale halo, whose
// wrong bits travel one cell per generation and never reach an output word.
__device__ __forceinline__ RowBits tile_row(uint32_t w)
{
    const uint32_t lw = __shfl_up_sync(FULL, w, 1);
    const uint32_t rw = __shfl_down_sync(FULL, w, 1);
    const uint32_t L = __funnelshift_l(lw, w, 1), R = __funnelshift_r(w, rw, 1);
    RowBits r;
    r.w = w;
    r.a0 = lop3<XOR3>(L, w, R);
    r.a1 = lop3<MAJ3>(L, w, R);
    return r;
}

// One generation of a band: c = state at t, o = state at t-1 and then at t+1; up / dn: the rows around it.
template <int RULE, int R>
__device__ __forceinline__ void band_generation(const uint32_t (&c)[R], uint32_t (&o)[R], uint32_t upw, uint32_t dnw)
{
    RowBits up = tile_row(upw), mid = tile_row(c[0]);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const RowBits dn = tile_row(r + 1 < R ? c[r + 1 < R ? r + 1 : 0] : dnw);
        o[r] = life_combine<RULE>(up, mid, dn, o[r]);
        up = mid;
        mid = dn;
    }
}

template <int RULE, int R, bool RAGGED, bool BESIDE>
__global__ void __launch_bounds__(TB_WARPS * 32, 2) life_bits_tb(const uint32_t* __restrict__ curG, const uint32_t* __restrict__ oldG,
                                                                 uint32_t* __restrict__ outCur, uint32_t* __restrict__ outOld, int nx, int nw,
                                                                 int ny, LifeTiles tiles, int steps)
{
    const gb::BlockId bid = gb::grid_wait();
    constexpr int W = TB_WARPS, RR = R * W, ROWS = RR - 2 * TB_STEPS;  // rows of the region, of the tile
    __shared__ uint32_t top[2][W][32], bot[2][W][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int ty, word;
    bool mine;  // this lane's words are written
    if (!BESIDE || bid.x < tiles.whole) {
        ty = (int)(bid.x / (unsigned)tiles.cols);
        word = ((int)bid.x - ty * tiles.cols) * 30 - 1 + lane;
        mine = lane >= 1 && lane <= 30 && word < nw;
    } else {  // the words left over
        const int g = lane / (tiles.rest + 2), at = lane - g * (tiles.rest + 2);
        ty = (int)(bid.x - tiles.whole) * tiles.side + g;
        word = 30 * tiles.cols + at - 1;
        mine = g < tiles.side && at >= 1 && at <= tiles.rest;
    }
    int wx = word % nw;
    if (wx < 0) wx += nw;
    WordSource src;
    if (RAGGED) src.at(word, nx, nw);
    const int y0 = ty * ROWS - TB_STEPS + R * w;  // the band's first row
    uint32_t c[R], o[R];
    {
        int gy = y0 % ny;
        if (gy < 0) gy += ny;
        const size_t plane = (size_t)ny * nw;
        const uint32_t* pc = curG + (size_t)gy * nw;
        const ptrdiff_t old = oldG - curG;
        int wrap = ny - gy;  // the band's row at which the grid begins again
        auto at_row = [&](int r) {
            if (r == wrap) {
                pc -= plane;
                wrap += ny;
            }
        };
        if (!RAGGED || __all_sync(FULL, src.whole())) {
            pc += RAGGED ? src.q : wx;
#pragma unroll
            for (int r = 0; r < R; r++) {
                at_row(r);
                c[r] = __ldg(pc);
                o[r] = RULE == APPFIS_GB_LIFE_REFERENCE ? __ldg(pc + old) : 0u;
                pc += nw;
            }
        } else {
            // four rows' loads before their words are put together: row by row, the warps at a row's end took
            // 90 loads one after the other (3001 x 3000, 64 generations with the bytes' conversion 64 us, now 50)
            constexpr int B = 4;
#pragma unroll
            for (int r0 = 0; r0 < R; r0 += B) {
                WordSource::Parts a[B], b[B];
#pragma unroll
                for (int k = 0; k < B; k++)
                    if (r0 + k < R) {
                        at_row(r0 + k);
                        a[k] = src.fetch(pc);
                        if (RULE == APPFIS_GB_LIFE_REFERENCE) b[k] = src.fetch(pc + old);
                        pc += nw;
                    }
#pragma unroll
                for (int k = 0; k < B; k++)
                    if (r0 + k < R) {
                        c[r0 + k] = src.join(a[k]);
                        o[r0 + k] = RULE == APPFIS_GB_LIFE_REFERENCE ? src.join(b[k]) : 0u;
                    }
            }
        }
    }
    const int above = w > 0 ? w - 1 : 0, below = w < W - 1 ? w + 1 : W - 1;  // the region's outer rows go stale
    int t = 0;
    for (; t + 2 <= steps; t += 2) {
        top[0][w][lane] = c[0];
        bot[0][w][lane] = c[R - 1];
        __syncthreads();
        band_generation<RULE, R>(c, o, bot[0][above][lane], top[0][below][lane]);
        top[1][w][lane] = o[0];
        bot[1][w][lane] = o[R - 1];
        __syncthreads();
        band_generation<RULE, R>(o, c, bot[1][above][lane], top[1][below][lane]);
    }
    const bool odd = t < steps;
    if (odd) {
        top[0][w][lane] = c[0];
        bot[0][w][lane] = c[R - 1];
        __syncthreads();
        band_generation<RULE, R>(c, o, bot[0][above][lane], top[0][below][lane]);
    }
    // the newest state is in o after an odd number of generations
    uint32_t* __restrict__ outC = odd ? outOld : outCur;
    uint32_t* __restrict__ outO = odd ? outCur : outOld;
    const uint32_t keep = RAGGED && word == nw - 1 ? (1u << (nx & 31)) - 1u : FULL;
    if (BESIDE ? !mine : lane < 1 || lane > 30 || word >= nw) return;
    const int first = TB_STEPS - R * w, end = min(RR - TB_STEPS - R * w, ny - y0);  // the band's rows to be written
    uint32_t* pc = outC + (ptrdiff_t)y0 * nw + word;
    uint32_t* po = outO + (ptrdiff_t)y0 * nw + word;
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (r >= first && r < end) {
            *pc = RAGGED ? c[r] & keep : c[r];
            *po = RAGGED ? o[r] & keep : o[r];
        }
        pc += nw;
        po += nw;
    }
}

// ------------------------------------------------------------------------------ bytes <-> words
__device__ __forceinline__ uint32_t four_bits(uint32_t v)  // bit 0 of bytes 0..3 -> bits 0..3
{
    uint32_t x = v & LSB;
    x = (x | (x >> 7)) & 0x00030003u;  // bytes 0,1 -> bits 0,1 ; bytes 2,3 -> bits 16,17
    return (x | (x >> 14)) & 0x0000000fu;
}

__device__ __forceinline__ uint32_t four_bytes(uint32_t b)  // bits 0..3 -> bytes 0..3
{
    uint32_t x = b & 0xfu;
    x = (x | (x << 14)) & 0x00030003u;
    return (x | (x << 7)) & LSB;
}

// Whole words (nx a multiple of 32), one or two planes per launch (blockIdx.y).
__global__ void life_pack(const uint8_t* __restrict__ cellsA, const uint8_t* __restrict__ cellsB, uint32_t* __restrict__ bitsA,
                          uint32_t* __restrict__ bitsB, size_t nwords)
{
    const gb::BlockId bid = gb::grid_wait();
    const uint8_t* __restrict__ cells = bid.y ? cellsB : cellsA;
    uint32_t* __restrict__ bits = bid.y ? bitsB : bitsA;
    size_t w = (size_t)bid.x * blockDim.x + threadIdx.x;
    if (w >= nwords) return;
    const uint4* p = reinterpret_cast<const uint4*>(cells + w * 32);
    uint4 a = __ldg(p), b = __ldg(p + 1);
    uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}, out = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) out |= four_bits(v[k]) << (4 * k);
    bits[w] = out;
}

__global__ void life_unpack(const uint32_t* __restrict__ bitsA, const uint32_t* __restrict__ bitsB, uint8_t* __restrict__ cellsA,
                            uint8_t* __restrict__ cellsB, size_t nwords)
{
    const gb::BlockId bid = gb::grid_wait();
    const uint32_t* __restrict__ bits = bid.y ? bitsB : bitsA;
    uint8_t* __restrict__ cells = bid.y ? cellsB : cellsA;
    size_t w = (size_t)bid.x * blockDim.x + threadIdx.x;
    if (w >= nwords) return;
    uint32_t b = __ldg(bits + w), v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = four_bytes(b >> (4 * k));
    uint4* p = reinterpret_cast<uint4*>(cells + w * 32);
    p[0] = make_uint4(v[0], v[1], v[2], v[3]);
    p[1] = make_uint4(v[4], v[5], v[6], v[7]);
}

// Byte rows of any length (nx >= 64) to and from rows of nw = ceil(nx / 32) words, two planes per
// launch (blockIdx.y).  Bytes move as aligned words whatever the rows' alignment: packing, a thread
// puts its 32 cells together from nine aligned words; unpacking, a thread writes one aligned
// 16-byte piece of the plane, which may hold the end of a row and the start of the next.
// Row and column of the block's first item, items numbered along rows of `per`; the threads then
// need no 64-bit division.
__device__ __forceinline__ size_t block_origin(size_t first, int per, int* col)
{
    __shared__ size_t row;
    __shared__ int c;
    if (threadIdx.x == 0) {
        row = first / per;
        c = (int)(first - row * per);
    }
    __syncthreads();
    *col = c;
    return row;
}

__global__ void __launch_bounds__(256) life_pack_rows(const uint8_t* __restrict__ cellsA, const uint8_t* __restrict__ cellsB,
                                                      uint32_t* __restrict__ bitsA, uint32_t* __restrict__ bitsB, int nx, int nw,
                                                      size_t nwords, size_t ncells)
{
    const gb::BlockId bid = gb::grid_wait();
    const uint8_t* __restrict__ cells = bid.y ? cellsB : cellsA;
    uint32_t* __restrict__ bits = bid.y ? bitsB : bitsA;
    int col;
    const size_t first = (size_t)bid.x * 256, row0 = block_origin(first, nw, &col);
    const size_t id = first + threadIdx.x;
    if (id >= nwords) return;
    const unsigned q = (unsigned)(col + threadIdx.x) / (unsigned)nw, w = (unsigned)(col + threadIdx.x) - q * (unsigned)nw;
    const size_t at = (row0 + q) * (size_t)nx + 32 * (size_t)w;
    const int n = min(32, nx - (int)(32 * w));
    const uint8_t* p = cells + at;
    const unsigned off = (unsigned)(reinterpret_cast<uintptr_t>(p) & 3u);
    uint32_t out = 0u;
    if (at >= off && at - off + 36 <= ncells) {  // the nine words lie inside the plane
        const uint32_t* a = reinterpret_cast<const uint32_t*>(p - off);
        uint32_t u[9];
#pragma unroll
        for (int k = 0; k < 9; k++) u[k] = __ldg(a + k);
#pragma unroll
        for (int k = 0; k < 8; k++) out |= four_bits(__funnelshift_r(u[k], u[k + 1], 8 * off)) << (4 * k);
        if (n < 32) out &= (1u << n) - 1u;
    } else {
        for (int k = 0; k < n; k++) out |= (uint32_t)(__ldg(p + k) & 1u) << k;
    }
    bits[id] = out;
}

__global__ void __launch_bounds__(256) life_unpack_rows(const uint32_t* __restrict__ bitsA, const uint32_t* __restrict__ bitsB,
                                                        uint8_t* __restrict__ cellsA, uint8_t* __restrict__ cellsB, int nx, int nw,
                                                        size_t ncells)
{
    const gb::BlockId bid = gb::grid_wait();
    const uint32_t* __restrict__ bits = bid.y ? bitsB : bitsA;
    uint8_t* __restrict__ cells = bid.y ? cellsB : cellsA;
    // the block's 4096 cells start at the plane's byte 4096 * bid.x - lead, a 16-byte boundary
    const int lead = (int)(reinterpret_cast<uintptr_t>(cells) & 15u);
    const size_t begin = (size_t)bid.x * 4096;
    const int skip = begin == 0 ? lead : 0;  // bytes of the first block that lie before the plane
    int col;
    const size_t row0 = block_origin(begin + skip - lead, nx, &col);
    const int from = max(16 * (int)threadIdx.x, skip);  // this thread's cells of the block: from .. to
    const size_t cell = begin + from - lead;
    if (cell >= ncells) return;
    const int to = (int)min((size_t)(16 * (threadIdx.x + 1)), ncells + lead - begin);
    if (from >= to) return;
    const unsigned x0 = (unsigned)(col + from - skip), q = x0 / (unsigned)nx, x = x0 - q * (unsigned)nx;
    const uint32_t* row = bits + (row0 + q) * (size_t)nw;
    const unsigned w = x >> 5;
    uint32_t v = __funnelshift_r(__ldg(row + w), (int)w + 1 < nw ? __ldg(row + w + 1) : 0u, x & 31u);
    const int here = nx - (int)x;  // cells of this row from x on
    if (here < to - from) v = (v & ((1u << here) - 1u)) | (__ldg(row + nw) << here);
    uint8_t* d = cells + cell;
    if (to - from == 16) {
        *reinterpret_cast<uint4*>(d) = make_uint4(four_bytes(v), four_bytes(v >> 4), four_bytes(v >> 8), four_bytes(v >> 12));
    } else {
        for (int k = 0; k < to - from; k++) d[k] = (uint8_t)((v >> k) & 1u);
    }
}

// The reference's layout: int cells 0/1 on a (nx + 2g) x (ny + 2g) grid with a periodic ghost
// ring of width g (GameOfLife/src/game_appfis.hpp:58-62).  From it: the u8 interior; into it:
// every padded cell from the interior cell it wraps to (the ghost ring as the periodic exchange
// leaves it, corners included).
__global__ void life_from_i32(const int32_t* __restrict__ f, int px, int g, uint8_t* __restrict__ cells, int nx, int ny)
{
    const gb::BlockId bid = gb::grid_wait();
    const int i = bid.x * blockDim.x + threadIdx.x;
    if (i >= nx) return;
    for (int j = bid.y; j < ny; j += gridDim.y) cells[(size_t)j * nx + i] = __ldg(f + (size_t)(j + g) * px + i + g) != 0;
}

__global__ void life_to_i32(const uint8_t* __restrict__ cells, int nx, int ny, int32_t* __restrict__ f, int px, int g)
{
    const gb::BlockId bid = gb::grid_wait();
    const int i = bid.x * blockDim.x + threadIdx.x;
    if (i >= nx + 2 * g) return;
    int si = (i - g) % nx;
    if (si < 0) si += nx;
    for (int j = bid.y; j < ny + 2 * g; j += gridDim.y) {
        int sj = (j - g) % ny;
        if (sj < 0) sj += ny;
        f[(size_t)j * px + i] = __ldg(cells + (size_t)sj * nx + si);
    }
}

// Population: popcount over 32-bit words (u8 cells are 0/1, so popc of 4 bytes = live bytes).
__global__ void popcount_words(const uint32_t* __restrict__ words, size_t n, unsigned long long* __restrict__ out)
{
    const gb::BlockId bid = gb::grid_wait();
    unsigned long long s = 0;
    for (size_t i = (size_t)bid.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        s += __popc(__ldg(words + i));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(FULL, s, o);
    __shared__ unsigned long long part[32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(FULL, s, o);
        if (threadIdx.x == 0) atomicAdd(out, s);
    }
}

// tail of a byte array whose length is not a multiple of 4
__global__ void popcount_tail(const uint8_t* p, int n, unsigned long long* out)
{
    gb::grid_wait();
    unsigned long long s = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += p[i];
    if (s) atomicAdd(out, s);
}

// Blocks of 256 threads: as many as are resident at once, but no more than the warp tasks need.
template <class K>
unsigned resident_grid(K kernel, int tasks)
{
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0) != cudaSuccess || per_sm < 1) per_sm = 4;
    const size_t need = gb::ceil_div((size_t)tasks * 32, 256);
    return (unsigned)std::max<size_t>(1, std::min<size_t>(need, (size_t)per_sm * gb::sm_count()));
}

// ------------------------------------------------------------------------------ time-blocked runs
struct TbPair {
    uint32_t* p[2];  // state at t, state at t-1
};

#define LIFE_BANDS(F) F(5) F(6) F(7) F(8) F(10) F(12) F(14) F(16) F(18) F(20) F(22) F(24) F(26) F(28) F(30) F(33) F(36) F(39) F(41) F(43) F(45)

unsigned life_tiles(int nw, int ny, int rows, bool beside, LifeTiles& t)
{
    const unsigned high = gb::ceil_div(ny, rows);
    t.cols = beside ? nw / 30 : (nw + 29) / 30;
    t.rest = beside ? nw % 30 : 0;
    t.side = 32 / (t.rest + 2);
    t.whole = (unsigned)t.cols * high;
    return t.whole + (t.rest ? gb::ceil_div(high, t.side) : 0u);
}

struct LifePlan {
    int band;
    bool beside;
};

// Rows per band, and whether the words left over from whole columns go side by side: what takes the least time
// with the tiles dealt to the SMs; the fullest SM's tiles follow one another on its logic pipe, 0.47 us per band
// row (and 0.2) for 16 generations, whatever is resident together.  Tall bands compute less halo (45 rows:
// 10%, 8: half, 5: four fifths), but a small grid needs many tiles, and a step in the fullest SM's tiles separates
// neighbouring heights: us per 64 generations (four launches of 16), reference rule, in columns of their own,
//   rows             5    6    7    8   10   12   14   16   18   20   22   24   26   28   30   33   36   39   41   43   45
//   256^2           17   18   19   20   23   26   30   33   36   39   43   46   49   53   57   67   71   77   84   85   92
//   1024 x 1000     26   19   19   21   24   28   31   35   38   41   45   48   51   56   60   70   74   82   89   90   98
//   1440 x 1500     36   30   20   21   24   28   32   35   39   42   46   49   52   57   61   71   75   83   90   91   98
//   2048^2          66   41   32   36   24   28   32   36   39   43   46   50   53   57   61   72   76   83   90   91   99
//   3072 x 3000    106   65   58   50   42   49   33   36   39   43   46   50   53   58   62   72   76   84   91   92   99
//   4096^2         177  112   85   80   60   71   57   64   71   78   48   51   54   58   62   73   77   84   92   93  100
//   5760 x 6000    306  182  138  125   97   94   83   93  102   79   86   92   98  106  114  129   78   85   92   93  100
//   8192^2         615  367  282  242  203  179  181  175  165  148  163  171  145  157  169  187  142  155  164  169  179
//   11520 x 12000 1194  705  531  448  365  330  308  289  291  286  279  257  279  256  277  307  272  295  311  319  264
//   15904 x 12000 1683  986  742  626  509  478  432  401  414  390  394  379  371  397  384  371  399  367  388  403  423
//   16384^2       2431 1426 1070  906  743  675  632  595  573  562  550  542  547  546  545  553  537  517  545  565  519
// (planes in shared memory, tiles of 32 to 256 rows: 1024 x 1000 49, 2048^2 66, 4096^2 107, 8192^2 211, 16384^2 706).
// The rule takes the fastest of them, 45 rows at 11520 x 12000 within 3% of it; a run of 8 generations (two
// launches of 4, more load than generations) within 9% (1024 x 1000 6.6 against 6.1 us, 4096^2 11.4 against 10.9).
// Side by side costs its warps scattered loads (1024 x 1000, where whole columns leave SMs idle anyway: 20.6 against
// 18.6 with 6 rows; 4096^2 with 20 rows 45.5, the fastest), so it has to save 0.8 us and 5% (16384^2, 4% fewer tiles with
// 45 rows: 546 against 519; with 30 rows 510), and half a column or more is a column.
LifePlan tb_plan(int nw, int ny)
{
    const unsigned sms = gb::sm_count();
    LifePlan best = {8, false};
    double cost = 1e30;
    LifeTiles t;
    for (int beside = 0; beside < (nw % 30 && nw % 30 <= 14 ? 2 : 1); beside++) {
#define LIFE_COST(R)                                                                                                             \
    {                                                                                                                            \
        const unsigned tiles = life_tiles(nw, ny, 8 * R - 2 * TB_STEPS, beside != 0, t);                                         \
        double c = (double)gb::ceil_div(tiles, sms) * (0.47 * R + 0.2);                                                          \
        if (beside) c = std::max(1.05 * c, c + 0.8);                                                                             \
        if (c < cost || (c == cost && !beside)) {                                                                                \
            cost = c;                                                                                                            \
            best = {R, beside != 0};                                                                                             \
        }                                                                                                                        \
    }
        LIFE_BANDS(LIFE_COST)
#undef LIFE_COST
    }
    return best;
}

template <int RULE, int R>
void launch_tb(TbPair in, TbPair out, int nx, int nw, int ny, int steps, bool beside, cudaStream_t st)
{
    static_assert(TB_WARPS == 8, "bands of 8 warps");
    LifeTiles t;
    const unsigned tiles = life_tiles(nw, ny, R * TB_WARPS - 2 * TB_STEPS, beside, t);
    auto kernel = nx % 32 ? life_bits_tb<RULE, R, true, true> : beside ? life_bits_tb<RULE, R, false, true> : life_bits_tb<RULE, R, false, false>;
    gb::launch(kernel, tiles, TB_WARPS * 32, 0, st, in.p[0], in.p[1], out.p[0], out.p[1], nx, nw, ny, t, steps);
}

template <int RULE>
void tb_step(LifePlan plan, TbPair in, TbPair out, int nx, int nw, int ny, int steps, cudaStream_t st)
{
    switch (plan.band) {
#define LIFE_CASE(R) \
    case R: return launch_tb<RULE, R>(in, out, nx, nw, ny, steps, plan.beside, st);
        LIFE_BANDS(LIFE_CASE)
#undef LIFE_CASE
    }
}

// `gens` generations in `launches` launches of nearly equal length, from pair[0] and back into
// `last`; a launch cannot write the pair it reads (its tiles read their neighbours' halo rows).
// An odd number of launches goes round three pairs once, so it needs pair[2].
template <int RULE>
int run_tb(const TbPair (&pair)[3], TbPair last, int nx, int ny, int gens, int launches, cudaStream_t st)
{
    const int nw = (nx + 31) / 32;
    const LifePlan plan = tb_plan(nw, ny);
    int at = 0, done = 0;
    for (int n = 0; n < launches; n++) {
        const int next = (pair[2].p[0] && n < 3) ? (n + 1) % 3 : 1 - at;
        const int upto = (int)((long long)gens * (n + 1) / launches);
        tb_step<RULE>(plan, pair[at], n + 1 == launches ? last : pair[next], nx, nw, ny, upto - done, st);
        done = upto;
        at = next;
    }
    return gb::launched("life_bits_tb");
}

template <int RULE>
int run_u8(uint8_t* buf[2], int nx, int ny, int gens, int* cur_index, cudaStream_t st)
{
    int ci = 0;
    const size_t cells = (size_t)nx * ny;
    // bulk: rows of whole 16-byte vectors and enough of them; 64 x 32-row CTAs at 4 M cells take the
    // 18.4 us of one CTA's march, which the one-thread-per-cell form takes there too (701 x 700: 5.4)
    const bool bulk = nx % 16 == 0 && cells >= ((size_t)1 << 22);
    // Packed: bytes to words, the time-blocked kernel, words to bytes.  The conversions and launches cost
    // 7-9 us and 0.8-1.6 us per M cells, a generation next to nothing; a sweep costs 3.0 us (0.1 M cells),
    // 4.6 (1 M), 14 (4 M, either form), 60 / 19 (17 M, one thread per cell / bulk), 244 / 30-47 (67 M).
    // Us for 20 generations, sweeps -> packed: 301 x 300 82 -> 17, 2050 x 1999 366 -> 26, 8192^2 697 -> 105,
    // 8200 x 8192 4878 -> 150.
    const bool packed = bulk ? gens >= 2 || cells < ((size_t)1 << 23)
                             : gens >= 4 || (gens >= 2 && (size_t)gens * cells >= 3000000) || cells >= 6000000;
    if (nx >= 64 && gens > 0 && packed && !gb::capturing(st)) {
        const int nw = (nx + 31) / 32;
        const size_t words = (size_t)nw * ny, plane = (words + 63) / 64 * 64;
        void* ws = nullptr;
        if (gb::scratch_alloc(4 * sizeof(uint32_t) * plane, st, &ws)) {
            uint32_t* w = reinterpret_cast<uint32_t*>(ws);
            const TbPair pair[3] = {{{w, w + plane}}, {{w + 2 * plane, w + 3 * plane}}, {{nullptr, nullptr}}};
            const unsigned planes = RULE == APPFIS_GB_LIFE_REFERENCE ? 2 : 1;  // B3/S23 does not read the state at t-1
            const int launches = (gens + TB_STEPS - 1) / TB_STEPS;
            const TbPair last = pair[launches & 1];
            const dim3 wgrid(gb::ceil_div(words, 256), planes);
            ci = gens & 1;
            int rc;
            if (nx % 32) {
                gb::launch(life_pack_rows, wgrid, 256, 0, st, buf[0], buf[1], w, w + plane, nx, nw, words, cells);
                rc = run_tb<RULE>(pair, last, nx, ny, gens, launches, st);
                gb::launch(life_unpack_rows, dim3(gb::ceil_div(cells + 15, 4096), 2), 256, 0, st, last.p[0], last.p[1], buf[ci], buf[1 - ci], nx, nw, cells);
            } else {
                gb::launch(life_pack, wgrid, 256, 0, st, buf[0], buf[1], w, w + plane, words);
                rc = run_tb<RULE>(pair, last, nx, ny, gens, launches, st);
                gb::launch(life_unpack, dim3(wgrid.x, 2), 256, 0, st, last.p[0], last.p[1], buf[ci], buf[1 - ci], words);
            }
            gb::scratch_free(ws, st);
            GB_TRY(rc);
            GB_TRY(gb::launched("life_u8 (packed)"));
            if (cur_index) *cur_index = ci;
            return APPFIS_GB_OK;
        }
    }
    if (bulk) {
        unsigned* status;
        GB_TRY(gb::status_word(&status));
        GB_CUDA(cudaFuncSetAttribute(life_u8_bulk<RULE>, cudaFuncAttributeMaxDynamicSharedMemorySize, UB_SMEM));
        const int strips = (nx + UB_W - 1) / UB_W;
        const unsigned grid = (unsigned)strips * gb::ceil_div(ny, UB_ROWS);
        for (int g = 0; g < gens; g++) {
            gb::launch(life_u8_bulk<RULE>, grid, 256, UB_SMEM, st, buf[ci], buf[1 - ci], nx, ny, strips, status);
            ci = 1 - ci;
        }
    } else {
        dim3 blk(32, 8), grd(gb::ceil_div(nx, 32), gb::ceil_div(ny, 8));
        for (int g = 0; g < gens; g++) {
            gb::launch(life_u8_generic<RULE>, grd, blk, 0, st, buf[ci], buf[1 - ci], nx, ny);
            ci = 1 - ci;
        }
    }
    GB_TRY(gb::launched("life_u8 sweep"));
    if (cur_index) *cur_index = ci;
    return APPFIS_GB_OK;
}

// Bit-packed run.  Three or more generations take the time-blocked kernel, at least two launches so that
// the state comes back into (a, b): as sweeps / tiles, us: 1024 x 1000 4 generations 9.3 / 5.7; 4096^2 3
// 10.7 / 9.8, 8 28 / 12.8; 16384^2 3 84 / 75, 8 226 / 113.  The newest state is in a after an even number of
// generations, else in b, as it is when every generation is a sweep.
template <int RULE>
int run_bits(uint32_t* buf[2], int nx, int ny, int gens, int* cur_index, cudaStream_t st)
{
    const int nw = nx / 32, ci = gens & 1;
    const size_t plane = (size_t)nw * ny, bytes = sizeof(uint32_t) * plane;
    const TbPair own = {{buf[0], buf[1]}}, last = {{buf[ci], buf[1 - ci]}};
    if (cur_index) *cur_index = ci;
    if (gens >= TB_STEPS) {
        // the long runs' pairs stay in the workspace, so that a run can be recorded in a graph after a
        // first one has sized them; a recording that would need more, or a full device, takes one more, shorter,
        // launch and no third pair
        int launches = std::max(2, (gens + TB_STEPS - 1) / TB_STEPS);
        void *wc, *wd, *we = nullptr, *wf = nullptr;
        GB_TRY(gb::workspace(gb::WS_LIFE_C, bytes, &wc));
        GB_TRY(gb::workspace(gb::WS_LIFE_D, bytes, &wd));
        if (launches % 2) {
            const bool held = gb::workspace_holds(gb::WS_LIFE_E, bytes) && gb::workspace_holds(gb::WS_LIFE_F, bytes);
            int rc = !held && gb::capturing(st) ? (int)APPFIS_GB_ENOMEM : gb::workspace(gb::WS_LIFE_E, bytes, &we);
            if (rc == APPFIS_GB_OK && (rc = gb::workspace(gb::WS_LIFE_F, bytes, &wf)) == APPFIS_GB_ENOMEM) gb::workspace_drop(gb::WS_LIFE_E);
            if (rc == APPFIS_GB_ENOMEM) {
                launches++;
                we = wf = nullptr;
            } else if (rc != APPFIS_GB_OK) {
                return rc;
            }
        }
        const TbPair pair[3] = {own, {{(uint32_t*)wc, (uint32_t*)wd}}, {{(uint32_t*)we, (uint32_t*)wf}}};
        return run_tb<RULE>(pair, last, nx, ny, gens, launches, st);
    }
    void* ws = nullptr;
    if (gens >= 3 && !gb::capturing(st) && gb::scratch_alloc(2 * bytes, st, &ws)) {
        const TbPair pair[3] = {own, {{(uint32_t*)ws, (uint32_t*)ws + plane}}, {{nullptr, nullptr}}};
        const int rc = run_tb<RULE>(pair, last, nx, ny, gens, 2, st);
        gb::scratch_free(ws, st);
        return rc;
    }
    // one launch per generation; rows per warp so that every SM has 24 warps' work if the grid has it
    // (1024 x 1000: 4.1 us with 4 rows, 10.3 with 32; 16384^2: 37.9 and 30.7)
    const int strips = (nw + 31) / 32;
    int srows = LIFE_ROWS;
    while (srows > 4 && (long long)strips * ((ny + srows - 1) / srows) < 24LL * gb::sm_count()) srows /= 2;
    const int tasks = strips * ((ny + srows - 1) / srows);
    const unsigned grid = resident_grid(life_bits_sweep<RULE>, tasks);
    for (int g = 0; g < gens; g++) gb::launch(life_bits_sweep<RULE>, grid, 256, 0, st, buf[g & 1], buf[1 - (g & 1)], nw, ny, strips, srows, tasks);
    return gb::launched("life_bits sweep");
}

int check_life(const void* a, const void* b, int nx, int ny, int gens, int rule)
{
    if (!a || !b) return gb::fail(APPFIS_GB_EINVAL, "life: null buffer");
    if (a == b) return gb::fail(APPFIS_GB_EINVAL, "life: the two buffers must differ");
    if (nx < 1 || ny < 1) return gb::fail(APPFIS_GB_EINVAL, "life: bad size %d x %d", nx, ny);
    if ((size_t)nx * (size_t)ny > ((size_t)1 << 40)) return gb::fail(APPFIS_GB_EINVAL, "life: grid too large");
    if (gens < 0) return gb::fail(APPFIS_GB_EINVAL, "life: negative generation count");
    if (rule != APPFIS_GB_LIFE_REFERENCE && rule != APPFIS_GB_LIFE_B3S23)
        return gb::fail(APPFIS_GB_EINVAL, "life: unknown rule %d", rule);
    return APPFIS_GB_OK;
}

int population_u8(const uint8_t* cells, int64_t n, int64_t* dev_count, cudaStream_t st)
{
    GB_CUDA(cudaMemsetAsync(dev_count, 0, sizeof(int64_t), st));
    size_t nw = (size_t)n / 4;
    if (nw) {
        unsigned grid = (unsigned)std::min<size_t>(gb::ceil_div(nw, 256), (size_t)gb::sm_count() * 8);
        gb::launch(popcount_words, grid, 256, 0, st, reinterpret_cast<const uint32_t*>(cells), nw,
                                             reinterpret_cast<unsigned long long*>(dev_count));
    }
    if (n % 4)
        gb::launch(popcount_tail, 1, 32, 0, st, cells + nw * 4, (int)(n % 4), reinterpret_cast<unsigned long long*>(dev_count));
    return gb::launched("life population");
}

}  // namespace

extern "C" {

int appfis_gb_life_u8(uint8_t* a, uint8_t* b, int nx, int ny, int gens, int rule, int* cur_index, void* stream)
{
    GB_TRY(check_life(a, b, nx, ny, gens, rule));
    if (nx % 16 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15))
        return gb::fail(APPFIS_GB_EINVAL, "life_u8: buffers must be 16-byte aligned");
    uint8_t* buf[2] = {a, b};
    cudaStream_t st = gb::as_stream(stream);
    return rule == APPFIS_GB_LIFE_REFERENCE ? run_u8<APPFIS_GB_LIFE_REFERENCE>(buf, nx, ny, gens, cur_index, st)
                                            : run_u8<APPFIS_GB_LIFE_B3S23>(buf, nx, ny, gens, cur_index, st);
}

int appfis_gb_life_bits(uint32_t* a, uint32_t* b, int nx, int ny, int gens, int rule, int* cur_index, void* stream)
{
    GB_TRY(check_life(a, b, nx, ny, gens, rule));
    if (nx % 32) return gb::fail(APPFIS_GB_EINVAL, "life_bits: nx (%d) must be a multiple of 32", nx);
    uint32_t* buf[2] = {a, b};
    cudaStream_t st = gb::as_stream(stream);
    return rule == APPFIS_GB_LIFE_REFERENCE ? run_bits<APPFIS_GB_LIFE_REFERENCE>(buf, nx, ny, gens, cur_index, st)
                                            : run_bits<APPFIS_GB_LIFE_B3S23>(buf, nx, ny, gens, cur_index, st);
}

int appfis_gb_life_pack(const uint8_t* cells, uint32_t* bits, int nx, int ny, void* stream)
{
    if (!cells || !bits || nx < 1 || ny < 1 || nx % 32) return gb::fail(APPFIS_GB_EINVAL, "life_pack: bad arguments");
    if (reinterpret_cast<uintptr_t>(cells) & 15) return gb::fail(APPFIS_GB_EINVAL, "life_pack: cells must be 16-byte aligned");
    size_t nw = (size_t)nx * ny / 32;
    gb::launch(life_pack, gb::ceil_div(nw, 256), 256, 0, gb::as_stream(stream), cells, cells, bits, bits, nw);
    return gb::launched("life_pack");
}

int appfis_gb_life_unpack(const uint32_t* bits, uint8_t* cells, int nx, int ny, void* stream)
{
    if (!cells || !bits || nx < 1 || ny < 1 || nx % 32) return gb::fail(APPFIS_GB_EINVAL, "life_unpack: bad arguments");
    if (reinterpret_cast<uintptr_t>(cells) & 15) return gb::fail(APPFIS_GB_EINVAL, "life_unpack: cells must be 16-byte aligned");
    size_t nw = (size_t)nx * ny / 32;
    gb::launch(life_unpack, gb::ceil_div(nw, 256), 256, 0, gb::as_stream(stream), bits, bits, cells, cells, nw);
    return gb::launched("life_unpack");
}

int appfis_gb_life_from_i32(const int32_t* padded, int px, int ghost, uint8_t* cells, int nx, int ny, void* stream)
{
    if (!padded || !cells || nx < 1 || ny < 1 || ghost < 0 || ghost > nx || ghost > ny || px < nx + 2 * ghost)
        return gb::fail(APPFIS_GB_EINVAL, "life_from_i32: bad arguments");
    dim3 grd(gb::ceil_div(nx, 256), std::min(ny, 65535));
    gb::launch(life_from_i32, grd, 256, 0, gb::as_stream(stream), padded, px, ghost, cells, nx, ny);
    return gb::launched("life_from_i32");
}

int appfis_gb_life_to_i32(const uint8_t* cells, int nx, int ny, int32_t* padded, int px, int ghost, void* stream)
{
    if (!padded || !cells || nx < 1 || ny < 1 || ghost < 0 || ghost > nx || ghost > ny || px < nx + 2 * ghost)
        return gb::fail(APPFIS_GB_EINVAL, "life_to_i32: bad arguments");
    dim3 grd(gb::ceil_div(nx + 2 * ghost, 256), std::min(ny + 2 * ghost, 65535));
    gb::launch(life_to_i32, grd, 256, 0, gb::as_stream(stream), cells, nx, ny, padded, px, ghost);
    return gb::launched("life_to_i32");
}

int appfis_gb_life_population_u8(const uint8_t* cells, int64_t n, int64_t* dev_count, void* stream)
{
    if (!cells || !dev_count || n < 0) return gb::fail(APPFIS_GB_EINVAL, "life_population_u8: bad arguments");
    if (reinterpret_cast<uintptr_t>(cells) & 3) return gb::fail(APPFIS_GB_EINVAL, "life_population_u8: cells must be 4-byte aligned");
    return population_u8(cells, n, dev_count, gb::as_stream(stream));
}

int appfis_gb_life_population_bits(const uint32_t* bits, int64_t nwords, int64_t* dev_count, void* stream)
{
    if (!bits || !dev_count || nwords < 0) return gb::fail(APPFIS_GB_EINVAL, "life_population_bits: bad arguments");
    cudaStream_t st = gb::as_stream(stream);
    GB_CUDA(cudaMemsetAsync(dev_count, 0, sizeof(int64_t), st));
    if (nwords) {
        unsigned grid = (unsigned)std::min<size_t>(gb::ceil_div((size_t)nwords, 256), (size_t)gb::sm_count() * 8);
        gb::launch(popcount_words, grid, 256, 0, st, bits, (size_t)nwords, reinterpret_cast<unsigned long long*>(dev_count));
    }
    return gb::launched("life_population_bits");
}

int appfis_gb_life_job(const uint8_t* cells_in, uint8_t* cells_out, int nx, int ny, int gens, int rule, int form,
                       int64_t* population)
{
    if (!cells_in) return gb::fail(APPFIS_GB_EINVAL, "life_job: null input");
    if (form != APPFIS_GB_FORM_U8 && form != APPFIS_GB_FORM_BITS) return gb::fail(APPFIS_GB_EINVAL, "life_job: form %d", form);
    GB_TRY(check_life(cells_in, cells_in + 1, nx, ny, gens, rule));
    if (form == APPFIS_GB_FORM_BITS && nx % 32) return gb::fail(APPFIS_GB_EINVAL, "life_job: bit form needs nx %% 32 == 0");
    cudaStream_t st;
    GB_TRY(gb::job_stream(&st));
    const size_t n = (size_t)nx * ny;
    const size_t nbytes = (n + 15) & ~(size_t)15;
    void *ua, *ub, *cnt;
    GB_TRY(gb::workspace(gb::WS_JOB_A, nbytes, &ua));
    GB_TRY(gb::workspace(gb::WS_JOB_F, 64, &cnt));
    GB_CUDA(cudaMemcpyAsync(ua, cells_in, n, cudaMemcpyHostToDevice, st));
    uint8_t* latest = nullptr;
    if (form == APPFIS_GB_FORM_U8) {
        GB_TRY(gb::workspace(gb::WS_JOB_B, nbytes, &ub));
        GB_CUDA(cudaMemsetAsync(ub, 0, n, st));
        int ci = 0;
        GB_TRY(appfis_gb_life_u8((uint8_t*)ua, (uint8_t*)ub, nx, ny, gens, rule, &ci, st));
        latest = ci == 0 ? (uint8_t*)ua : (uint8_t*)ub;
        GB_TRY(appfis_gb_life_population_u8(latest, (int64_t)n, (int64_t*)cnt, st));
    } else {
        void *wa, *wb;
        const size_t wbytes = n / 8;
        GB_TRY(gb::workspace(gb::WS_JOB_C, wbytes, &wa));
        GB_TRY(gb::workspace(gb::WS_JOB_D, wbytes, &wb));
        GB_TRY(appfis_gb_life_pack((const uint8_t*)ua, (uint32_t*)wa, nx, ny, st));
        GB_CUDA(cudaMemsetAsync(wb, 0, wbytes, st));
        int ci = 0;
        GB_TRY(appfis_gb_life_bits((uint32_t*)wa, (uint32_t*)wb, nx, ny, gens, rule, &ci, st));
        uint32_t* lw = ci == 0 ? (uint32_t*)wa : (uint32_t*)wb;
        GB_TRY(appfis_gb_life_population_bits(lw, (int64_t)(n / 32), (int64_t*)cnt, st));
        if (cells_out) GB_TRY(appfis_gb_life_unpack(lw, (uint8_t*)ua, nx, ny, st));
        latest = (uint8_t*)ua;
    }
    if (cells_out) GB_CUDA(cudaMemcpyAsync(cells_out, latest, n, cudaMemcpyDeviceToHost, st));
    int64_t pop = 0;
    GB_CUDA(cudaMemcpyAsync(&pop, cnt, sizeof pop, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    if (population) *population = pop;
    return gb::check_status("life_job");  // a bounded wait of the u8 sweep that gave up
}

}  // extern "C"
