// Checks of the row bands of k_level_bands (rgbd-flow_b200/csrc/level_bands.cuh) and of the rule for the CTAs an
// item gets (band_ctas in pipeline.cuh), on the CPU: no kernel is launched.
#include "../../rgbd-flow_b200/csrc/pipeline.cuh"

#include <cstdio>

using namespace rgbdflow;

struct Size {
    int W, H;
};
static int fail(const char* what, int a, int b, int c)
{
    std::printf("%s: %d %d %d\n", what, a, b, c);
    return 1;
}

int main()
{
    for (int C : {1, 2, 4, 8, 16})
        for (int H = C > 1 ? 2 * C : 1; H < 700; H++) {
            const int B = band_rows(H, C);
            if (band_row(0, H, C) != 0 || band_row(C, H, C) != H) return fail("ends", H, C, 0);
            for (int r = 0; r < C; r++) {
                const int n = band_row(r + 1, H, C) - band_row(r, H, C);
                if (n > B || n < (C > 1 ? 2 : 1)) return fail("rows", H, C, r);
            }
            for (int i = 0; i < H; i++) {
                const int r = band_of(i, H, C);
                if (i < band_row(r, H, C) || i >= band_row(r + 1, H, C)) return fail("band_of", H, C, i);
            }
        }
    for (int hw = 1; hw < 400; hw++)
        if (band_rp(hw) < hw + 2 || ((2 * band_rp(hw) - hw) & 30)) return fail("pitch", hw, band_rp(hw), 0);
    const Size sizes[] = {{2, 2}, {10, 7}, {20, 15}, {40, 30}, {75, 56}, {80, 60}, {101, 75}, {160, 120}, {161, 120}, {12, 900},
                          {900, 12}, {240, 180}, {640, 480}};
    for (const Size& a : sizes)
        for (const Size& b : sizes)
            for (int n : {1, 2, 7, 8, 16, 17, 35, 36, 74, 75, 148, 149}) {
                std::vector<Size> items(n, a);
                items.back() = b;
                const int C = band_ctas(items, 148);
                if (!C) continue;
                if (n * C > 148) return fail("CTAs", n, C, 0);
                for (const Size& s : items)
                    if (band_rows(s.H, C) * ((s.W + 1) / 2) > kBandMax || (C > 1 && s.H < 2 * C) ||
                        band_smem_bytes(s.W, s.H, C) > kBandSmem)
                        return fail("fit", s.W, s.H, C);
            }
    std::vector<Size> one = {{640, 480}};
    if (band_ctas(one, 148)) return fail("640x480 on bands", 0, 0, 0);
    std::printf("ok level bands\n");
    return 0;
}
