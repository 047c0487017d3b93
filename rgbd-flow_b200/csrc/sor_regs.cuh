// sor_regs.cuh — red-black SOR with the linear system held in registers (FP32): the default for levels
// that fit the device's register files.
//
// The tile and strip SOR of kernels.cuh keep the 12-float system in shared memory and read 31 values
// a pixel update there: at 128 bytes a clock those reads alone take about a clock per update and SM,
// and the kernels run at a third of that rate.  Here a thread owns a block of 2 columns x 4 rows of a
// region 64 columns wide (a warp: 64 columns x 4 rows, warps stacked downwards) and keeps the
// block's system, its edge weights and its unknowns in registers for the whole launch:
//   * horizontal neighbours are the thread's own other column or one lane away (3 shuffles an update),
//   * vertical neighbours are the thread's own rows, except across warps (each warp publishes the
//     unknowns of its first and last row in shared memory after every half-sweep).
// Every register index is a compile-time constant, because a block starts on an even row and column and
// so the colour of each of its pixels is fixed.  Every pixel's operations and their order are the tile kernel's
// (the negated weights negate exactly), so the results are the same bit for bit.  (The packed FP32 instructions
// were tried for pairs of rows: two operations in one take the register reads of two.)
#pragma once
#include "kernels.cuh"

namespace rgbdflow {

// A thread's block: V rows (a) x 2 columns (e).
template <int V>
struct RegBlock {
    float c[V][2][9];              // reciprocal diagonal, couplings, right-hand sides (sys planes 0..8)
    float R[V][2], Rs[V][2];       // right edge's weight, and times the pixel's depth-smoothness weight
    float L[V], Ls[V];             // left edge of the even column (the left lane's odd column's R)
    float D[V][2], Ds[V][2];       // lower edge
    float U[2], Us[2];             // upper edge of row 0 (the row above's D)
    float x[V][2][3];              // the increment
};

// The unknowns a warp publishes for its neighbours: [first / last row][u, v, w][column parity][lane].
constexpr int kRegEx = 2 * 3 * 2 * 32;

// One half-sweep (colour C) of a warp's block (its first row is even).  up / down: the other pixels' unknowns of the row
// above / below the block, of this lane ([u, v, w], 64 elements apart); own: where this lane publishes.
// Pixels outside the image have a system of zeros and start at 0, so they stay 0: 0 times a finite
// neighbour adds nothing, and every unknown is finite while the steps add up to a finite number (an update is
// clamped to +-step around the old value, which also turns a NaN into one).  CHK: md takes the largest |change|
// over the pixels of `mine` (bit 2 a + e: row a, column parity e).  MASK, for unknowns that may be infinite: `in` (same
// bits) keeps pixels outside the image at 0, and what lies beside the region, with an edge of weight 0 (a shuffle
// there gives the lane's own column), is taken as 0.
template <int V, int C, bool CHK, bool MASK>
__device__ __forceinline__ void reg_half_sweep(RegBlock<V>& b, const float* up, const float* down, float* own, float omega,
                                               float step, unsigned in, unsigned mine, float& md)
{
    constexpr unsigned full = 0xffffffffu;
    constexpr int eV = (C + V - 1) & 1;  // the column parity of the last row's pixel
    float xu0[3], xdV[3];
#pragma unroll
    for (int v = 0; v < 3; v++) {
        xu0[v] = up[(v * 2 + C) * 32];
        xdV[v] = down[(v * 2 + eV) * 32];
    }
#pragma unroll
    for (int a = 0; a < V; a++) {
        const int e = (a + C) & 1;
        float xl[3], xr[3], xu[3], xd[3], nv[3];
#pragma unroll
        for (int v = 0; v < 3; v++) {
            if (e == 0) {
                xl[v] = __shfl_up_sync(full, b.x[a][1][v], 1);
                xr[v] = b.x[a][1][v];
            } else {
                xl[v] = b.x[a][0][v];
                xr[v] = __shfl_down_sync(full, b.x[a][0][v], 1);
            }
            xu[v] = a > 0 ? b.x[a > 0 ? a - 1 : 0][e][v] : xu0[v];
            xd[v] = a < V - 1 ? b.x[a < V - 1 ? a + 1 : a][e][v] : xdV[v];
            if (MASK && e == 0) xl[v] = (threadIdx.x & 31) != 0 ? xl[v] : 0.f;
            if (MASK && e == 1) xr[v] = (threadIdx.x & 31) != 31 ? xr[v] : 0.f;
        }
        const float aL = e == 0 ? b.L[a] : b.R[a][0], wL = e == 0 ? b.Ls[a] : b.Rs[a][0];
        const float aU = a > 0 ? b.D[a > 0 ? a - 1 : 0][e] : b.U[e], wU = a > 0 ? b.Ds[a > 0 ? a - 1 : 0][e] : b.Us[e];
        sor_point_w<float>(b.c[a][e], aL, aU, b.R[a][e], b.D[a][e], wL, wU, b.Rs[a][e], b.Ds[a][e], xl, xu, xr, xd,
                           b.x[a][e], omega, step, nv);
        if (MASK) {
            const bool ok = (in >> (2 * a + e)) & 1;
#pragma unroll
            for (int v = 0; v < 3; v++) nv[v] = ok ? nv[v] : 0.f;
        }
        if (CHK) {
            const bool cnt = (mine >> (2 * a + e)) & 1;
#pragma unroll
            for (int v = 0; v < 3; v++) md = cnt ? fmaxf(md, fabsf(nv[v] - b.x[a][e][v])) : md;
        }
#pragma unroll
        for (int v = 0; v < 3; v++) b.x[a][e][v] = nv[v];
    }
#pragma unroll
    for (int v = 0; v < 3; v++) {
        own[(v * 2 + C) * 32] = b.x[0][C][v];
        own[(6 + v * 2 + eV) * 32] = b.x[V - 1][eV][v];
    }
}

// Publishes the first and last row before the first half-sweep.
template <int V>
__device__ __forceinline__ void reg_publish(const RegBlock<V>& b, float* own)
{
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
        for (int v = 0; v < 3; v++) {
            own[(v * 2 + e) * 32] = b.x[0][e][v];
            own[(6 + v * 2 + e) * 32] = b.x[V - 1][e][v];
        }
}

// Fills a block from the planes of an item in the checkerboard layout:
// sys + z stride the 12 system planes, x + v stride the increment's (xzero: it starts at 0).  off: the element
// of the block's first row, colour 0, this lane's position; hw: elements between half-rows; row a is read
// where ok[a] (zeros elsewhere; positions of a half-row past its last pixel hold zeros).  top: read the
// weights of the edge to the row above.
template <int V>
__device__ __forceinline__ void reg_block_load(RegBlock<V>& b, int lane, const float* __restrict__ sys,
                                               const float* __restrict__ x, long long stride, int off, int hw,
                                               const bool* ok, bool xzero, bool top)
{
    int o[2 * V];
#pragma unroll
    for (int q = 0; q < 2 * V; q++) o[q] = off + q * hw;  // half-row q: row q / 2, colour q & 1
    auto at = [&](int a, int e) { return o[2 * a + ((a + e) & 1)]; };
#pragma unroll
    for (int z = 0; z < 12; z++) {
        const float* p = sys + z * stride;
#pragma unroll
        for (int a = 0; a < V; a++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float q = ok[a] ? __ldg(p + at(a, e)) : 0.f;
                if (z < 9) b.c[a][e][z] = q;
                else if (z == 9) b.R[a][e] = q;
                else if (z == 10) b.D[a][e] = q;
                else b.Rs[a][e] = q;  // the depth-smoothness weight, multiplied out below
            }
    }
    float us[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int oa = off + (((e + 1) & 1) - 2) * hw;  // the row above
        b.U[e] = top ? __ldg(sys + 10 * stride + oa) : 0.f;
        us[e] = top ? __ldg(sys + 11 * stride + oa) : 0.f;
    }
#pragma unroll
    for (int v = 0; v < 3; v++) {
        const float* p = x + v * stride;
#pragma unroll
        for (int a = 0; a < V; a++)
#pragma unroll
            for (int e = 0; e < 2; e++) b.x[a][e][v] = ok[a] && !xzero ? __ldg(p + at(a, e)) : 0.f;
    }
#pragma unroll
    for (int a = 0; a < V; a++) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const float s = b.Rs[a][e];
            b.Rs[a][e] = mulR(b.R[a][e], s);
            b.Ds[a][e] = mulR(b.D[a][e], s);
        }
        // the left lane's odd column; the region's first column has no left neighbour
        const float l = __shfl_up_sync(0xffffffffu, b.R[a][1], 1), ls = __shfl_up_sync(0xffffffffu, b.Rs[a][1], 1);
        b.L[a] = lane == 0 ? 0.f : l;
        b.Ls[a] = lane == 0 ? 0.f : ls;
    }
#pragma unroll
    for (int e = 0; e < 2; e++) b.Us[e] = mulR(b.U[e], us[e]);
}

// Stores the increment's pixels of `mine` (bit 2 a + e).
template <int V>
__device__ __forceinline__ void reg_block_store(const RegBlock<V>& b, float* x, long long stride, int off, int hw, unsigned mine)
{
#pragma unroll
    for (int a = 0; a < V; a++)
#pragma unroll
        for (int e = 0; e < 2; e++)
            if ((mine >> (2 * a + e)) & 1) {
#pragma unroll
                for (int v = 0; v < 3; v++) x[v * stride + off + (2 * a + ((a + e) & 1)) * hw] = b.x[a][e][v];
            }
}

// ------------------------------------------------------------------------------------------
// Resident SOR: levels of several CTAs' registers.
//
// The level is cut into tiles of 64 x 48 pixels (12 warps of 4 rows; one CTA per SM) that overlap by 4 K
// pixels, and every tile stays in its CTA's registers for all the iterations of an inner iteration.  After
// K iterations a tile is right except within 2 K pixels of a side that is not the image's edge: there
// its neighbours own the pixels.  So every K iterations a CTA sends its pixels within 2 K of such a side and
// reads its neighbours': a pixel travels as one 16-byte word (u, v, w, tag) stored and loaded whole, and
// the reader polls the word itself until it carries the round's tag, so an exchange costs one trip through
// L2 and no fence.  Two sets of words alternate between rounds: who sends round r + 1 has read round r, and
// sends round r + 2 only after it has read its neighbours' round r + 1.  Tags do not repeat within a level,
// and k_level_setup clears the words before it.  A convergence check ends a round and counts the item's CTAs
// in, so that all take the same decision.  Launched cooperatively (the CTAs wait for one another), every
// wait bounded.
//
// What bounds it: the half-sweeps (0.65 us; 106 cycles of a scheduler per warp and pixel update, for which a launch
// executes 91 instructions, load and exchange included, 42 of them the update's arithmetic), then the exchange (1.8 us:
// half of it the way through L2; by flags -- store, barrier, fence, flag; poll with acquire loads, barrier, load -- it
// took 4.8 us).  Of the 168 registers a thread may have 96 bytes more are in local memory (spill stores 156 bytes, loads
// 216).
// Measured, 30 iterations of one level (one pair): 640x480 91 us (tile SOR 261), 320x240 64 (108), 160x120 63
// and 80x60 63 (cluster whole-level kernel 126 and 105); 16 pairs: 640x480 15.4 -> 9.1 ms of SOR a solve (strip
// SOR), 320x240 3.3 -> 1.6 (strips), 160x120 0.81 -> 0.44 (cluster).  Levels of more than 148 tiles (about
// 390,000 pixels) stay on the strip and tile SOR, steps of few small levels go to k_level_bands.
//
// Items take the launch's CTAs in order, as many together as fit; a CTA goes through its items in order,
// so an item waits for nothing but earlier items.
constexpr int kResW = 12, kResV = 4, kResRows = kResW * kResV, kResCols = 64, kResNT = 32 * kResW;
constexpr int kResMaxK = 5;
constexpr int kResItems = 64;  // items a launch serves
// Measured cost of K iterations: a half-sweep, and an exchange with the neighbours (thousands of cycles).
constexpr double kResHalfSweep = 1.25, kResExchange = 3.6;

struct ResItem {
    PairCtl* ctl;
    float* x;          // x[0][0]; the six increment planes, then the 12 system planes, stride elements apart
    long long stride;  // (checkerboard layout)
    ulonglong2* exch;  // exchange words: two sets of one per element of a plane
    int W, H, hw;
    int K;             // iterations between exchanges
    int nx, ny;        // tiles across and down
    int item, fold0;   // its LevelItem; the first of its blocks in the fold's grid
};

__host__ __device__ constexpr int res_tiles(int size, int region, int K)
{
    return size <= region ? 1 : (size - 4 * K + region - 4 * K - 1) / (region - 4 * K);
}
// Tile i of n along one axis (region pixels wide, size pixels in all): its first pixel and the pixels it owns.
__host__ __device__ inline void res_tile(int i, int n, int size, int region, int K, int& first, int& lo, int& hi)
{
    first = i * (region - 4 * K);
    lo = i == 0 ? 0 : first + 2 * K;
    hi = i == n - 1 ? size : first + region - 2 * K;
}

// A tile of an item: the first pixel of its region and the pixels it owns.
struct ResTile {
    int tx, ty, c0, x0, x1, r0, y0, y1;
};
__host__ __device__ inline ResTile res_tile_of(const ResItem& it, int tile)
{
    ResTile t;
    t.tx = tile % it.nx;
    t.ty = tile / it.nx;
    res_tile(t.tx, it.nx, it.W, kResCols, it.K, t.c0, t.x0, t.x1);
    res_tile(t.ty, it.ny, it.H, kResRows, it.K, t.r0, t.y0, t.y1);
    return t;
}
// What a pixel of the image or of its half-rows' padding is to a tile: 1 inside the image, 2 owned (the
// padding, which holds zeros, by the last tile of its row), 4 owned and read by a neighbour.
__host__ __device__ inline int res_pixel(const ResItem& it, const ResTile& t, int i, int j)
{
    int f = 0;
    if (i < it.H && j < it.W) f |= 1;
    if (i >= t.y0 && i < t.y1 && j >= t.x0 && (j < t.x1 || (t.x1 == it.W && j < 2 * it.hw))) {
        f |= 2;
        const int r = 2 * it.K;
        if ((t.tx > 0 && j < t.x0 + r) || (t.tx < it.nx - 1 && j >= t.x1 - r) || (t.ty > 0 && i < t.y0 + r) ||
            (t.ty < it.ny - 1 && i >= t.y1 - r))
            f |= 4;
    }
    return f;
}

// One pixel's exchange word, stored and loaded as a single 128-bit access.
__device__ __forceinline__ void send_word(ulonglong2* p, const float* x, unsigned tag)
{
    const unsigned long long lo = (unsigned long long)__float_as_uint(x[1]) << 32 | __float_as_uint(x[0]);
    const unsigned long long hi = (unsigned long long)tag << 32 | __float_as_uint(x[2]);
    asm volatile("{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}\n" ::"l"(p), "l"(lo), "l"(hi)
                 : "memory");
}
// Loads a word where `want` is set (0 elsewhere), without a branch: several loads are in flight together.
__device__ __forceinline__ void load_word(const ulonglong2* p, bool want, unsigned long long& lo, unsigned long long& hi)
{
    asm volatile("{\n .reg .pred w;\n .reg .b128 q;\n setp.ne.u32 w, %3, 0;\n mov.b128 q, {%4, %4};\n"
                 " @w ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}\n"
                 : "=l"(lo), "=l"(hi) : "l"(p), "r"((unsigned)want), "l"(0ull) : "memory");
}
// Polls of a word or counter before a wait gives up (0.35 us or more each, so a third of a second at least), and what
// a launch adds for each SOR iteration of each item but one: a tile's neighbours may still be at earlier items, and
// an iteration takes them up to 5 us.
constexpr int kResPolls = 1 << 20, kResPollsIteration = 16;
static inline int resident_polls(int n_items, int n_sor)
{
    const double p = kResPolls + (double)kResPollsIteration * (n_items - 1) * n_sor;
    return p < (1 << 30) ? (int)p : 1 << 30;
}

// tag0: the launch's first tag less one; a launch uses at most n_sor of them.  MASK: unknowns may overflow (a kernel of
// its own: in one with the other, what it adds to the half-sweeps cost a solve 1.6 %).
template <bool MASK>
__global__ void __launch_bounds__(kResNT, 1)
k_sor_resident(const ResItem* __restrict__ items, int n_items, SolveConst<float> k, SorLaunch L, unsigned tag0,
               int polls, int* status)
{
    __shared__ float ex[(kResW + 2) * kRegEx];  // slot w + 1: warp w; slots 0 and 13 stay 0
    __shared__ int s_first[kResItems], s_tiles[kResItems];  // the CTAs of each item: first and number (0: done)
    __shared__ unsigned s_max;
    // what only the exchange needs stays out of the registers: re-read from here after a barrier
    __shared__ struct {
        PairCtl* ctl;
        float* planes;
        ulonglong2* exch;
        long long stride;
        int hw, off0, K, tiles, tile, words;
    } t;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int e = tid; e < (kResW + 2) * kRegEx; e += kResNT) ex[e] = 0.f;
    if (tid < n_items) s_tiles[tid] = items[tid].ctl->level_done ? 0 : items[tid].nx * items[tid].ny;
    __syncthreads();
    if (tid == 0) {
        int used = 0;
        for (int i = 0; i < n_items; i++) {
            const int n = s_tiles[i];
            if (used + n > (int)gridDim.x) used = 0;
            s_first[i] = used;
            used += n;
        }
    }
    __syncthreads();
    float* const own = ex + (w + 1) * kRegEx + lane;
    const float *const up = own - kRegEx + 6 * 32, *const down = own + kRegEx;
    RegBlock<kResV> b;
    for (int i = 0; i < n_items; i++) {
        const int tile = (int)blockIdx.x - s_first[i];
        if (tile < 0 || tile >= s_tiles[i]) continue;
        // per pixel (bit 2 a + e): inside the image / owned / owned and read by a neighbour.  A half-row's
        // padding counts as owned by the last tile (it holds zeros)
        unsigned in = 0, mine = 0, ring = 0;
        int buf;  // the planes of the result
        {
            const ResItem* const it = &items[i];
            const ResTile g = res_tile_of(*it, tile);
            const int H = it->H, hw = it->hw;
            const int row0 = g.r0 + w * kResV, m = g.c0 / 2 + lane;
            bool ok[kResV];
#pragma unroll
            for (int a = 0; a < kResV; a++) {
                ok[a] = row0 + a < H && m < hw;
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int f = res_pixel(*it, g, row0 + a, 2 * m + e);
                    in |= (unsigned)(f & 1) << (2 * a + e);
                    mine |= (unsigned)(f >> 1 & 1) << (2 * a + e);
                    ring |= (unsigned)(f >> 2 & 1) << (2 * a + e);
                }
            }
            const int xin = L.xin_zero ? 0 : it->ctl->x_in;
            buf = xin ^ 1;
            reg_block_load<kResV>(b, lane, it->x + 6 * it->stride, it->x + 3 * xin * it->stride, it->stride, row0 * 2 * hw + m, hw,
                                  ok, L.xin_zero != 0, row0 > 0 && row0 <= H && m < hw);
            __syncthreads();  // the warps have left the last item's published rows and `t`
            if (tid == 0) {
                t.ctl = it->ctl;
                t.planes = it->x;
                t.stride = it->stride;
                t.hw = hw;
                t.off0 = g.r0 * 2 * hw + g.c0 / 2;
                t.exch = it->exch;
                t.words = 2 * hw * H;
                t.K = it->K;
                t.tiles = it->nx * it->ny;
                t.tile = tile;
                s_max = 0;
            }
        }
        reg_publish(b, own);
        __syncthreads();
        unsigned round = 0;
        for (int itn = 0; itn < k.n_sor;) {
            int nit = min(t.K, k.n_sor - itn);
            if (!k.fixed) nit = min(nit, k.period - itn % k.period);
            const bool chk = !k.fixed && (itn + nit) % k.period == 0;
            float md = 0.f;
#pragma unroll 1
            for (int h = 0; h < 2 * nit; h++) {
                // a check is of its own iteration (masked, every half-sweep takes the variant that can count)
                const bool last = h >= 2 * nit - 2;
                if (MASK || (chk && last)) {
                    const unsigned cnt = last ? mine : 0u;
                    if (h & 1) reg_half_sweep<kResV, 1, true, MASK>(b, up, down, own, k.omega, k.step, in, cnt, md);
                    else reg_half_sweep<kResV, 0, true, MASK>(b, up, down, own, k.omega, k.step, in, cnt, md);
                } else {
                    if (h & 1) reg_half_sweep<kResV, 1, false, MASK>(b, up, down, own, k.omega, k.step, in, mine, md);
                    else reg_half_sweep<kResV, 0, false, MASK>(b, up, down, own, k.omega, k.step, in, mine, md);
                }
                __syncthreads();
            }
            itn += nit;
            if (itn == k.n_sor && !chk) break;
            if (chk) {
                for (int o = 16; o > 0; o >>= 1) md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, o));
                if (lane == 0 && md > 0) atomicMax(&s_max, __float_as_uint(md));
            }
            // the exchange: send the ring, then fetch the pixels that the neighbours own
            ulonglong2* const words = t.exch + (round & 1) * t.words + t.off0 + w * kResV * 2 * t.hw + lane;
            const unsigned tag = tag0 + round + 1;
#pragma unroll
            for (int a = 0; a < kResV; a++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    if ((ring >> (2 * a + e)) & 1) send_word(words + (2 * a + ((a + e) & 1)) * t.hw, b.x[a][e], tag);
            bool ok = true;
            if (chk) {
                // the item's largest change: every CTA's into the control block, then all counted in
                const int ci = min(itn / k.period - 1, kMaxChecks - 1);
                __syncthreads();
                if (tid == 0) {
                    PairCtl* const ctl = t.ctl;
                    if (s_max) atomicMax(&ctl->maxdiff[ci], s_max);
                    __threadfence();
                    atomicAdd(&ctl->arrived, 1u);
                    const unsigned want = (unsigned)t.tiles * (unsigned)(itn / k.period);
                    int p = 0;
                    while (*(volatile unsigned*)&ctl->arrived < want && ++p < polls) {}
                    ok = p < polls;
                    __threadfence();
                    s_max = __ldcg(&ctl->maxdiff[ci]);
                }
                if (__syncthreads_or(!ok)) {
                    report_wait_failure(status);
                    return;
                }
                const float g = __uint_as_float(s_max);
                const bool stop = (double)g < k.sor_tol || g >= k.step;
                __syncthreads();  // every thread has read it
                if (tid == 0) {
                    s_max = 0;
                    if (stop && t.tile == 0) {
                        t.ctl->sor_stop_iter = itn;
                        t.ctl->sor_stop = 1;
                    }
                }
                if (stop || itn == k.n_sor) break;
            }
            // all of a thread's words in flight together (two at a time took 2.1 us instead of 0.9)
            unsigned halo = in & ~mine;
            for (int p = 0; __any_sync(0xffffffffu, halo != 0) && p < polls; p++) {
                unsigned long long lo[2 * kResV], hi[2 * kResV];
#pragma unroll
                for (int q = 0; q < 2 * kResV; q++)
                    load_word(words + (q & ~1) * t.hw + (((q >> 1) + q) & 1) * t.hw, (halo >> q) & 1, lo[q], hi[q]);
#pragma unroll
                for (int q = 0; q < 2 * kResV; q++) {
                    const bool got = ((halo >> q) & 1) && (unsigned)(hi[q] >> 32) == tag;
                    float* const x = b.x[q >> 1][q & 1];
                    x[0] = got ? __uint_as_float((unsigned)lo[q]) : x[0];
                    x[1] = got ? __uint_as_float((unsigned)(lo[q] >> 32)) : x[1];
                    x[2] = got ? __uint_as_float((unsigned)hi[q]) : x[2];
                    halo &= ~((unsigned)got << q);
                }
            }
            reg_publish(b, own);
            if (__syncthreads_or(halo != 0)) {
                report_wait_failure(status);
                return;
            }
            round++;
        }
        // the result: the owned pixels
        reg_block_store<kResV>(b, t.planes + 3 * buf * t.stride, t.stride, t.off0 + w * kResV * 2 * t.hw + lane, t.hw, mine);
        if (t.tile == 0 && tid == 0) t.ctl->x_stop = buf;
    }
}

// ------------------------------------------------------------------------------------------
// The fold after the last inner iteration of the resident items: u += x and the early-termination
// statistic, one 512-thread CTA per 32 x 32 tile in the tile kernel's order; the item's last tile takes
// the outer iteration's control (k_control's work).
template <class S>
__global__ void __launch_bounds__(512)
k_sor_fold(const LevelItem<float, S>* items, const ResItem* res, int n_res, SolveConst<float> k, int outer, int n_checks)
{
    int lo = 0, hi = n_res - 1;  // the resident item whose tiles this block is among
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (res[mid].fold0 <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const LevelItem<float, S>& it = items[res[lo].item];
    const int idx = (int)blockIdx.x - res[lo].fold0, sx = (it.W + kSorTW - 1) / kSorTW;
    const int ix0 = idx % sx * kSorTW, iy0 = idx / sx * kSorTH;
    PairCtl* ctl = it.ctl;
    if (ctl->level_done) return;
    __shared__ float red[16];
    __shared__ int s_last;
    const int xb = ctl->x_stop;
    const float *x0 = it.x[xb][0], *x1 = it.x[xb][1], *x2 = it.x[xb][2];
    float part = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int q = threadIdx.x + 512 * h;
        const int gi = iy0 + q / kSorTW, gj = ix0 + q % kSorTW;
        if (gi >= it.H || gj >= it.W) continue;
        const int lc = cs_idx(gi, gj, it.hwp);
        const float a = x0[lc], bq = x1[lc], cz = x2[lc];
        const size_t lp = (size_t)gi * it.pitch + gj;
        it.u[0][lp] = addR(it.u[0][lp], a);
        it.u[1][lp] = addR(it.u[1][lp], bq);
        it.u[2][lp] = addR(it.u[2][lp], cz);
        part = addR(part, stat_px<float>(a, bq, cz, it.f_level, it.pyr[6][(size_t)gi * it.W + gj]));
    }
    for (int off = 16; off > 0; off >>= 1) part += __shfl_down_sync(0xffffffffu, part, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        float tot = 0;
        for (int w = 0; w < 16; w++) tot += red[w];
        it.stat_part[idx] = tot;
        __threadfence();
        s_last = atomicAdd(&ctl->tiles_done, 1) == it.n_sor_tiles - 1;
    }
    __syncthreads();
    if (s_last && threadIdx.x < 32) {
        __threadfence();
        if (threadIdx.x == 0) ctl->tiles_done = 0;
        control_item(it, k, outer, n_checks, threadIdx.x);
    }
}

}  // namespace rgbdflow
