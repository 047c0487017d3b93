// Host-side check of the resident SOR's tiles (rgbd-flow_b200/csrc/sor_regs.cuh) and of the rule that picks
// the iterations between exchanges (resident_k, resident_fit in pipeline.cuh).  For levels at the edges of
// the tiling and every K, each tile's pixels are walked as its threads own them, and
//   * every pixel of the image (and of the half-rows' padding a region reaches) is owned by exactly one tile,
//   * owned pixels are at least 2 K pixels inside their region on every side that is not the image's edge,
//   * every other image pixel of a region is owned by one of the tile's 8 neighbours, which stores it for
//     its neighbours,
//   * every thread's element is its pixel's place in the checkerboard layout.
// Runs on the host only (no kernel is launched).
#include <cstdio>
#include <vector>

#include "../../rgbd-flow_b200/csrc/pipeline.cuh"

using namespace rgbdflow;

#define CHECK(c)                                                                                              \
    do {                                                                                                      \
        if (!(c)) {                                                                                           \
            std::printf("FAIL %s (line %d): %dx%d K %d tile %d\n", #c, __LINE__, it.W, it.H, it.K, tile);      \
            return 1;                                                                                         \
        }                                                                                                     \
    } while (0)

static int check(int W, int H, int K)
{
    ResItem it{};
    it.W = W; it.H = H; it.hw = hwp_of(W); it.K = K;
    it.nx = res_tiles(W, kResCols, K);
    it.ny = res_tiles(H, kResRows, K);
    const int P = 2 * it.hw, n = it.nx * it.ny;
    std::vector<int> owner((size_t)P * H, -1), stored((size_t)P * H, 0);
    for (int tile = 0; tile < n; tile++) {
        const ResTile t = res_tile_of(it, tile);
        CHECK(t.c0 % 2 == 0 && t.r0 % 2 == 0 && t.c0 < W && t.r0 < H && t.c0 / 2 < it.hw);
        CHECK(t.x0 < t.x1 && t.x1 <= W && t.y0 < t.y1 && t.y1 <= H);
        CHECK(t.x0 >= t.c0 && t.x1 <= t.c0 + kResCols && t.y0 >= t.r0 && t.y1 <= t.r0 + kResRows);
        CHECK(t.c0 == 0 || t.x0 - t.c0 >= 2 * K);
        CHECK(t.x1 == W || t.c0 + kResCols - t.x1 >= 2 * K);
        CHECK(t.r0 == 0 || t.y0 - t.r0 >= 2 * K);
        CHECK(t.y1 == H || t.r0 + kResRows - t.y1 >= 2 * K);
        for (int w = 0; w < kResW; w++)
            for (int lane = 0; lane < 32; lane++)
                for (int a = 0; a < kResV; a++)
                    for (int e = 0; e < 2; e++) {
                        const int row0 = t.r0 + w * kResV, m = t.c0 / 2 + lane, i = row0 + a, j = 2 * m + e;
                        const int f = res_pixel(it, t, i, j);
                        CHECK((f & 1) == (i < H && j < W));
                        if (f & 3) {
                            CHECK(i < H && m < it.hw);
                            CHECK((long)row0 * 2 * it.hw + m + (2 * a + ((a + e) & 1)) * it.hw == cs_idx(i, j, it.hw));
                        }
                        if (f & 2) {
                            CHECK(owner[(size_t)i * P + j] < 0);
                            owner[(size_t)i * P + j] = tile;
                            stored[(size_t)i * P + j] = f & 4;
                        }
                        CHECK(!(f & 4) || (f & 2));
                    }
    }
    int tile = -1;
    for (int i = 0; i < H; i++)
        for (int j = 0; j < W; j++) CHECK(owner[(size_t)i * P + j] >= 0);
    for (tile = 0; tile < n; tile++) {
        const ResTile t = res_tile_of(it, tile);
        for (int i = t.r0; i < t.r0 + kResRows; i++)
            for (int j = t.c0; j < t.c0 + kResCols; j++) {
                const int f = res_pixel(it, t, i, j);
                if ((f & 3) != 1) continue;  // not a pixel the exchange brings
                const int o = owner[(size_t)i * P + j], dx = o % it.nx - t.tx, dy = o / it.nx - t.ty;
                CHECK(o != tile && dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1 && stored[(size_t)i * P + j]);
            }
    }
    return 0;
}

int main()
{
    int cases = 0;
    for (int K = 1; K <= kResMaxK; K++)
        for (int W : {2, 3, 40, 63, 64, 65, 66, 80, 107, 108, 109, 116, 117, 124, 125, 160, 320, 501, 640, 801})
            for (int H : {2, 3, 47, 48, 49, 58, 59, 76, 77, 92, 93, 120, 240, 377, 480}) {
                if (check(W, H, K)) return 1;
                cases++;
            }
    struct It { int W, H; };
    for (const It& z : {It{640, 480}, It{501, 377}, It{320, 240}, It{160, 120}, It{80, 60}, It{66, 50}})
        for (int c : {1, 4, 16}) {
            std::vector<It> v(c, z);
            std::vector<int> w;
            for (int i = 0; i < c; i++) w.push_back(i);
            const int k = resident_k(v, w, 148), f = resident_fit(z.W, z.H, k, 148);
            if (k < 1 || f < 1 || f > k || res_tiles(z.W, kResCols, f) * res_tiles(z.H, kResRows, f) > 148) return 1;
            std::printf("rule %d x %dx%d: exchange every %d\n", c, z.W, z.H, f);
            cases++;
        }
    if (resident_fit(1280, 960, 5, 148) != 0) return 1;
    std::printf("ok resident tiles: %d cases\n", cases);
    return 0;
}
