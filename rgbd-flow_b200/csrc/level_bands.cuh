// level_bands.cuh — the whole solve of a small level in one launch (FP32).
//
// A level of a few thousand pixels is latency: linearisation, SOR, fold and control as launches of their own
// each pay a start, and after an early stop the rest of the schedule is launches that do nothing.  Here a
// thread-block cluster takes a level through all its outer iterations (sceneFlowSingleScale's loop,
// sceneFlowSingleScaleJacobiCUDA.cu:755-954) and leaves the loop when the outer iterations have converged.
// CTA r of C holds a band of rows, a thread one position of it: one pixel of each colour, whose system it
// linearises into its own registers.  The flow, the increment and the linearisation's planes live in shared
// memory. What a band needs of its neighbours they store into it: of every half-sweep the increment's
// boundary row, by stores that count in at an mbarrier, so that only the band's own boundary rows wait for them
// and the rest of a half-sweep is an update and a block barrier; of every outer iteration the flow's two boundary
// rows, before a cluster barrier.
//
// What bounds it: the half-sweep's latency.  Cycles of one, 30 iterations of it and of the rest of an outer iteration:
//   10x7, 1 CTA    370; SOR 22 K, linearisation 8 K, fold 0.8 K
//   80x60, 16      840; SOR 50 K, linearisation 11 K, fold 5 K (a cluster barrier a half-sweep: 1060)
//   160x120, 16   1330; SOR 79 K, linearisation 22 K, fold 11 K (1720)
// (the form for 640 threads, which 160x120 takes, has 96 registers a thread and spills: 188 bytes of stores, 224 of loads)
// against 60, 120 and 120 K for the SOR alone as launches of k_sor_level_reg and k_sor_resident, and 25 to 40 us an
// outer iteration for the rest.  A half-sweep of 80x60 is 370 cycles of update and block barrier and the way of the
// neighbours' rows (about 470).  A 160x120 solve 1.17 -> 0.89 ms, one of 320x240 without allocations 1.63 -> 1.30.
//
// Every pixel's operations and their order are k_linearize's, the tile SOR's and control_item's, and the
// statistic is summed in the 32 x 32 tiles' order: the results are theirs bit for bit.
#pragma once
#include "kernels.cuh"

namespace rgbdflow {

constexpr int kBandMax = 640;    // positions of a band (threads of a CTA)
constexpr int kBandSmall = 256;  // threads up to which a thread may keep 255 registers
constexpr size_t kBandSmem = 200 * 1024;
// Sets of the CTAs' largest changes that the convergence checks alternate between.  A check's barrier orders the
// stores of the check after the next behind its reads, but not the next one's: until then only the neighbours' rows
// tie the CTAs together, so that one d bands away may be d half-sweeps ahead of a warp that still reads.
constexpr int kBandCheckSets = 2;

// Row pitch (positions) of a half-row of the increment: a zero position each side, and the threads of a warp, which
// span rows where hw < 32, on different banks.
__host__ __device__ constexpr int band_rp(int hw)
{
    int rp = hw + 2;
    while (((2 * rp - hw) & 30) != 0) rp++;
    return rp;
}
// Rows of band r of C: [band_row(r), band_row(r + 1)).
__host__ __device__ inline int band_row(int r, int H, int C) { return (int)((unsigned)(r * H) / (unsigned)C); }
// The band of row i.
__host__ __device__ inline int band_of(int i, int H, int C) { return (int)((unsigned)((i + 1) * C - 1) / (unsigned)H); }
__host__ __device__ inline int band_rows(int H, int C) { return (H + C - 1) / C; }
__host__ __device__ inline size_t band_smem_bytes(int W, int H, int C)
{
    const int B = band_rows(H, C), hw = (W + 1) / 2;
    const size_t tiles = (size_t)((W + kSorTW - 1) / kSorTW) * ((H + kSorTH - 1) / kSorTH);
    return sizeof(float) * ((size_t)kLinN * (B + 4) * W + (size_t)3 * (B + 2) * 2 * band_rp(hw) + 17 * tiles);
}

__device__ __forceinline__ unsigned cluster_addr(const void* p, int rank)
{
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_store(unsigned a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ float cluster_load(unsigned a)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
// A store into another CTA's shared memory that counts its bytes in at that CTA's mbarrier.
__device__ __forceinline__ void cluster_send(unsigned a, float v, unsigned mbar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(a), "f"(v), "r"(mbar) : "memory");
}
__device__ __forceinline__ void mbar_init(unsigned mbar)
{
    asm volatile("mbarrier.init.shared.b64 [%0], 1;\n fence.mbarrier_init.release.cluster;" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned mbar, int bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
// Waits (`polls` tries) for the phase of the given parity; false: it gave up.  A try that fails has blocked for 4 us
// (measured), so that a wait gives up after a second.
constexpr int kBandPolls = 1 << 18;
__device__ __forceinline__ bool mbar_wait(unsigned mbar, int parity, int polls)
{
    for (int p = 0; p < polls; p++) {
        int ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// All CTAs of the cluster (one: a block barrier); the shared and global memory written before is visible.
template <bool CL>
__device__ __forceinline__ void cluster_sync()
{
    if (CL) {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// The end of a block (all its threads) of which some may have lost a wait: reports it, and stays for a millisecond so
// that rows the neighbours sent before the last cluster barrier land in shared memory that is still this block's.
__device__ __forceinline__ void report_lost(bool lost, int* status)
{
    if (!__syncthreads_or(lost)) return;
    report_wait_failure(status);
    for (int q = 0; q < 16; q++) __nanosleep(65536);
}

// NTM: most threads of a CTA.  CL: more than one CTA an item.
template <class S, int NTM, bool CL>
__global__ void __launch_bounds__(NTM, 1)
k_level_bands(const LevelItem<float, S>* items, SolveConst<float> k, int C, int n_outer, int n_inner, int polls, int* status)
{
    extern __shared__ __align__(16) float band_smem[];
    __shared__ float s_all[kBandCheckSets][16], red[32];
    __shared__ __align__(8) unsigned long long s_mbar[2];  // the neighbours' rows of even and odd half-sweeps
    const int rank = CL ? (int)blockIdx.x % C : 0;
    // the item from shared memory: a cluster barrier drops what L1 holds of global memory
    __shared__ LevelItem<float, S> it;
    static_assert(sizeof(it) % 4 == 0, "copied by words");
    for (int q = threadIdx.x; q < (int)(sizeof(it) / 4); q += blockDim.x)
        reinterpret_cast<unsigned*>(&it)[q] = reinterpret_cast<const unsigned*>(items + blockIdx.x / C)[q];
    __syncthreads();
    const int W = it.W, H = it.H, hw = (W + 1) / 2, RP = band_rp(hw);
    const int B = band_rows(H, C), r0 = band_row(rank, H, C), nr = band_row(rank + 1, H, C) - r0;
    const int tid = threadIdx.x, NT = (int)blockDim.x, lane = tid & 31, warp = tid >> 5, n_warps = NT >> 5;
    const int tx = (W + kSorTW - 1) / kSorTW, tiles = it.n_sor_tiles;
    const LinPlanes<float, 0> sv{band_smem, r0 - 2, 0, W, (B + 4) * W};
    const int PLS = (B + 2) * 2 * RP;
    float* const xs = band_smem + kLinN * sv.n;  // the increment: [u, v, w][row + 1][colour][position + 1], zeros around
    float* const part = xs + 3 * PLS;            // the statistic of each tile's 16 warps, then of the tiles
    const bool stat = it.allow_early && !k.fixed;
    // this thread's position: local row li, half-row index m
    const int li = tid / hw, m = tid % hw, i = r0 + li;
    const bool inpos = tid < nr * hw;
    const int odd = i & 1;                        // colour c's pixel of the position is in column 2 m + (c ^ odd)
    const bool valid[2] = {inpos && 2 * m + odd < W, inpos && 2 * m + (odd ^ 1) < W};
    float* const xo = xs + (li + 1) * 2 * RP + m + 1;  // the increment of colour 0 (1: RP further)
    // where the neighbours keep this thread's increment and flow: the halo rows of the bands above and below
    const bool to_up = CL && rank > 0, to_dn = CL && rank < C - 1;
    const int nr_up = to_up ? r0 - band_row(rank - 1, H, C) : 0;
    const unsigned base_up = to_up ? cluster_addr(band_smem, rank - 1) : 0, base_dn = to_dn ? cluster_addr(band_smem, rank + 1) : 0;
    const int xs0 = kLinN * sv.n;
    const unsigned mbar = (unsigned)__cvta_generic_to_shared(s_mbar);
    const unsigned mbar_up = to_up ? cluster_addr(s_mbar, rank - 1) : 0, mbar_dn = to_dn ? cluster_addr(s_mbar, rank + 1) : 0;
    if (CL && tid == 0) {
        mbar_init(mbar);
        mbar_init(mbar + 8);
    }
    unsigned sweeps = 0;  // half-sweeps so far
    int set = 0;          // of the next check's changes
    // the thread's row goes to the band above / below; it arrives at the block's barriers (a thread that also waits)
    bool send_up = to_up && li == 0, send_dn = to_dn && li == nr - 1, expects = CL && tid == (to_up ? 0 : (nr - 1) * hw);
    // A wait gave up: from then on the thread neither waits nor sends nor arrives (the barrier's last phase may be
    // open), and only the cluster barriers go on.
    bool lost = false;
    auto await = [&](unsigned n) {
        if (!lost && !mbar_wait(mbar + 8 * (n & 1), (n >> 1) & 1, polls)) {
            lost = true;
            send_up = send_dn = expects = false;
        }
    };

    for (int q = tid; q < (nr + 4) * W; q += NT) {
        const int gi = r0 - 2 + q / W, gj = q % W;
        if (gi < 0 || gi >= H) continue;
        for (int c = 0; c < 3; c++) sv.at(kLinU + c, gi, gj) = it.u[c][(size_t)gi * it.pitch + gj];
    }
    // f / depth of the two pixels (the statistic's weight of w^2)
    float fz[2];
#pragma unroll
    for (int c = 0; c < 2; c++)
        fz[c] = stat && valid[c] ? divR(it.f_level, it.pyr[6][(size_t)i * W + 2 * m + (c ^ odd)]) : 0.f;
    float cf[2][9], aL[2], aU[2], aR[2], aD[2], wL[2], wU[2], wR[2], wD[2], xp[2][3];
    bool ran = false;
    for (int outer = 0; outer < n_outer; outer++) {
        for (int e = tid; e < 3 * PLS; e += NT) xs[e] = 0.f;
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
            for (int v = 0; v < 3; v++) xp[c][v] = 0.f;
        __syncthreads();
        int iters = 0;         // SOR iterations of the inner iteration
        float maxdiff = -1.f;  // its last check's change, as control_item reads it
        for (int hh = 0; hh < n_inner; hh++) {
            // ---- linearise about u + x (k_linearize)
            iters = k.n_sor;
            maxdiff = -1.f;
            for (int q = tid; q < (nr + 4) * W; q += NT) {
                const int gi = r0 - 2 + q / W, gj = q % W;
                if (gi < 0 || gi >= H) continue;
                float U[3];
                const int lr = gi - r0 + 1;  // the increment's row
                const bool du = hh > 0 && lr >= 0 && lr <= nr + 1;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    U[c] = sv.at(kLinU + c, gi, gj);
                    const float D = du ? xs[c * PLS + (lr * 2 + ((gi + gj) & 1)) * RP + (gj >> 1) + 1] : 0.f;
                    sv.at(kLinUD + c, gi, gj) = U[c] + D;
                }
                lin_warp_px<float, S>(it, sv, gi, gj, U);
            }
            __syncthreads();
            for (int q = tid; q < (nr + 1) * W; q += NT) {
                const int gi = r0 - 1 + q / W, gj = q % W;
                if (gi >= 0) lin_phi_px<float, S>(it, k, sv, gi, gj);
            }
            __syncthreads();
            {
                // both pixels at once (a missing one is computed as some other pixel and not used): a
                // pixel is a long chain of divisions and square roots
                float o[2][12], e[2][4];
#pragma unroll
                for (int c = 0; c < 2; c++)
                    lin_system_px<float, S>(it, k, sv, inpos ? i : r0, !inpos ? 0 : 2 * m + (valid[c] ? c ^ odd : 0), o[c], e[c]);
#pragma unroll
                for (int c = 0; c < 2; c++) {
#pragma unroll
                    for (int z = 0; z < 9; z++) cf[c][z] = o[c][z];
                    aR[c] = o[c][9];
                    aD[c] = o[c][10];
                    aL[c] = e[c][0];
                    aU[c] = e[c][1];
                    wR[c] = mulR(o[c][9], o[c][11]);
                    wD[c] = mulR(o[c][10], o[c][11]);
                    wL[c] = mulR(e[c][0], e[c][2]);
                    wU[c] = mulR(e[c][1], e[c][3]);
                }
            }
            ran = true;
            // every CTA has zeroed its increment, or read it; nobody sends into it before this
            cluster_sync<CL>();
            // ---- the SOR iterations
            for (int itn = 0; itn < k.n_sor; itn++) {
                const bool chk = !k.fixed && (itn % k.period == k.period - 1);
                float md = 0.f;
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    if (CL) {
                        // the row of a neighbour that the half-sweep before has sent
                        if (itn + c > 0 && (send_up || send_dn)) await(sweeps - 1);
                        if (expects)
                            mbar_expect(mbar + 8 * (sweeps & 1), 12 * ((to_up ? (W + 1 - (c ^ ((r0 + 1) & 1))) / 2 : 0) +
                                                                      (to_dn ? (W + 1 - (c ^ ((r0 + nr) & 1))) / 2 : 0)));
                    }
                    if (valid[c]) {
                        const float* const xn = xo + (1 - c) * RP;  // the other colour's pixel of the position
                        const float* const xh = xn + (c ^ odd);     // the right neighbour
                        float xl[3], xu[3], xr[3], xd[3], nv[3];
#pragma unroll
                        for (int v = 0; v < 3; v++) {
                            const float* const xv = xn + v * PLS;
                            xl[v] = xh[v * PLS - 1];
                            xr[v] = xh[v * PLS];
                            xu[v] = xv[-2 * RP];
                            xd[v] = xv[2 * RP];
                        }
                        sor_point_w<float>(cf[c], aL[c], aU[c], aR[c], aD[c], wL[c], wU[c], wR[c], wD[c], xl, xu, xr, xd, xp[c],
                                           k.omega, k.step, nv);
#pragma unroll
                        for (int v = 0; v < 3; v++) {
                            xo[v * PLS + c * RP] = nv[v];
                            if (chk) md = fmaxf(md, fabsf(nv[v] - xp[c][v]));
                            xp[c][v] = nv[v];
                        }
                        if (send_up) {
                            const int o = xs0 + ((nr_up + 1) * 2 + c) * RP + m + 1;
#pragma unroll
                            for (int v = 0; v < 3; v++) cluster_send(base_up + 4 * (o + v * PLS), nv[v], mbar_up + 8 * (sweeps & 1));
                        }
                        if (send_dn) {
                            const int o = xs0 + c * RP + m + 1;
#pragma unroll
                            for (int v = 0; v < 3; v++) cluster_send(base_dn + 4 * (o + v * PLS), nv[v], mbar_dn + 8 * (sweeps & 1));
                        }
                    }
                    sweeps++;
                    __syncthreads();
                }
                if (chk) {
                    // the largest change of this iteration over the level, in every CTA
                    for (int o = 16; o > 0; o >>= 1) md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, o));
                    if (lane == 0) red[warp] = md;
                    __syncthreads();
                    if (tid < C) {
                        float g = 0.f;
                        for (int w = 0; w < n_warps; w++) g = fmaxf(g, red[w]);
                        if (CL) cluster_store(cluster_addr(&s_all[set][rank], tid), g);
                        else s_all[set][0] = g;
                    }
                    cluster_sync<CL>();
                    float g = 0.f;
                    for (int r = 0; r < C; r++) g = fmaxf(g, s_all[set][r]);
                    set = (set + 1) % kBandCheckSets;
                    const bool stop = (double)g < k.sor_tol || g >= k.step;
                    if (g > 0) maxdiff = g;
                    if (stop) iters = itn + 1;
                    if (stop) break;
                }
            }
            if (CL && k.n_sor > 0) await(sweeps - 1);
        }
        // ---- u += x, the statistic's terms, and the neighbours' copies of the flow's boundary rows
#pragma unroll
        for (int c = 0; c < 2; c++)
            if (valid[c]) {
                const int j = 2 * m + (c ^ odd);
                float u[3];
#pragma unroll
                for (int v = 0; v < 3; v++) {
                    u[v] = addR(sv.at(kLinU + v, i, j), xp[c][v]);
                    sv.at(kLinU + v, i, j) = u[v];
                }
                if (stat)
                    sv.at(kLinPhi, i, j) = addR(addR(mulR(xp[c][0], xp[c][0]), mulR(xp[c][1], xp[c][1])),
                                                mulR(mulR(xp[c][2], xp[c][2]), fz[c]));
                if (to_up && li < 2)
#pragma unroll
                    for (int v = 0; v < 3; v++)
                        cluster_store(base_up + 4 * ((kLinU + v) * sv.n + (nr_up + 2 + li) * W + j), u[v]);
                if (to_dn && li >= nr - 2)
#pragma unroll
                    for (int v = 0; v < 3; v++) cluster_store(base_dn + 4 * ((kLinU + v) * sv.n + (li - nr + 2) * W + j), u[v]);
            }
        cluster_sync<CL>();
        float tot = 0.f;  // the statistic, on one lane
        if (stat) {
            // in the tile kernels' order: virtual thread vt (0..511) takes pixels vt and vt + 512 of the 32 x 32
            // tile, a warp tree per virtual warp, then the 16 virtual warps in order; every CTA gets every warp's
            for (int q = rank * n_warps + warp; q < tiles * 16; q += C * n_warps) {
                const int ty = (q >> 4) / tx, gj = ((q >> 4) - ty * tx) * kSorTW + lane;
                bool ok[2];
                float t[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int gi = ty * kSorTH + (q & 15) + 16 * h;
                    ok[h] = gi < H && gj < W;
                    const int r = CL ? band_of(min(gi, H - 1), H, C) : 0;
                    const int o = kLinPhi * sv.n + (min(gi, H - 1) - band_row(r, H, C) + 2) * W + min(gj, W - 1);
                    t[h] = CL ? cluster_load(cluster_addr(band_smem + o, r)) : band_smem[o];
                }
                float p = ok[0] ? addR(0.f, t[0]) : 0.f;
                p = ok[1] ? addR(p, t[1]) : p;
                for (int o = 16; o > 0; o >>= 1) p += __shfl_down_sync(0xffffffffu, p, o);
                p = __shfl_sync(0xffffffffu, p, 0);
                if (CL && lane < C) cluster_store(cluster_addr(part + q, lane), p);
                if (!CL && lane == 0) part[q] = p;
            }
            cluster_sync<CL>();
            for (int ti = tid; ti < tiles; ti += NT) {
                float sum = 0.f;
#pragma unroll
                for (int w = 0; w < 16; w++) sum += part[ti * 16 + w];
                part[tiles * 16 + ti] = sum;
            }
            __syncthreads();
            for (int t = lane; t < tiles; t += 32) tot += part[tiles * 16 + t];
            for (int o = 16; o > 0; o >>= 1) tot += __shfl_down_sync(0xffffffffu, tot, o);
            tot = __shfl_sync(0xffffffffu, tot, 0);
        }
        const bool done = control_decide(it, k, tot);
        if (rank == 0 && tid == 0) control_record(it, k, outer, tot, iters, maxdiff, done);
        if (done) break;
    }
    if (CL) report_lost(lost, status);
    if (!ran) return;
    // ---- the flow, and the last system for rgbdflow_debug_read_plane
#pragma unroll
    for (int c = 0; c < 2; c++)
        if (valid[c]) {
            const int j = 2 * m + (c ^ odd), lp = cs_idx(i, j, it.hwp);
#pragma unroll
            for (int v = 0; v < 3; v++) it.u[v][(size_t)i * it.pitch + j] = sv.at(kLinU + v, i, j);
#pragma unroll
            for (int z = 0; z < 9; z++) it.sys[z][lp] = cf[c][z];
            it.sys[9][lp] = aR[c];
            it.sys[10][lp] = aD[c];
            it.sys[11][lp] = it.pyr[9][(size_t)i * W + j];
        }
}

}  // namespace rgbdflow
