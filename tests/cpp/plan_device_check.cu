// Plans for devices of other sizes (make_plan, rgbd-flow_b200/csrc/pipeline.cuh), on the CPU: no kernel is launched.
//
// The CTAs of a resident SOR item wait for one another, so its tiles have to fit the launch, which has at most a CTA
// a multiprocessor; the clusters of a step on level bands have to run together.
#include "../../rgbd-flow_b200/csrc/pipeline.cuh"

#include <cstdio>

using namespace rgbdflow;

static HostParams params(int n_outer)
{
    HostParams h;
    std::memset(&h, 0, sizeof(h));
    h.color_w = h.dvc = 1;
    h.alpha = 0.02; h.gamma = 1e-5; h.ratio = 0.5; h.min_width = -16;
    h.n_outer = n_outer; h.n_inner = 1; h.n_sor = 30; h.period = 25;
    h.omega = 0.7; h.step = 0.3; h.sor_tol = 1e-5; h.outer_tol = 4e-4;
    h.sor_strip = 1; h.sor_level = 1; h.level_reg = 1; h.fill_rounds = 253; h.wait_polls = -1;
    return h;
}

int main()
{
    const int sizes[][2] = {{640, 480}, {501, 377}, {320, 240}, {160, 120}, {64, 48}};
    int resident = 0, banded = 0, older = 0;
    for (int sms : {1, 2, 8, 20, 64, 100, 132, 144, 148, 160})
        for (const auto& s : sizes)
            for (int n : {1, 3}) {
                std::vector<PairSpec> pairs(n);
                for (auto& q : pairs) {
                    q.W = s[0];
                    q.H = s[1];
                    q.f_full = 0.8f * s[0];
                    q.xres_full = s[0];
                }
                PlanDevice dev;
                dev.sms = sms;
                const Plan<float, float> P = make_plan<float, float>(pairs, params(10), nullptr, dev);
                for (const auto& d : P.steps) {
                    const ResItem* ri = (const ResItem*)(P.desc.data() + d.res_items_off);
                    for (int i = 0; i < d.n_res; i++)
                        if (ri[i].nx * ri[i].ny > std::min(sms, d.res_tiles)) {
                            std::printf("%d multiprocessors: a %dx%d item of %d tiles\n", sms, ri[i].W, ri[i].H, ri[i].nx * ri[i].ny);
                            return 1;
                        }
                    if (d.band_c && d.n_items * d.band_c > sms) {
                        std::printf("%d multiprocessors: %d items on bands of %d\n", sms, d.n_items, d.band_c);
                        return 1;
                    }
                    resident += d.n_res > 0;
                    banded += d.band_c > 0;
                    older += !d.regs;
                }
            }
    // a device that holds no clusters above a size (or none): smaller ones, or the launches of their own
    for (int most : {8, 4, 2, 1}) {
        PlanDevice dev;
        for (int q = 0; q < 4; q++)
            if (kClusterSizes[q] > most) dev.clusters[q] = 0;
        for (const auto& s : sizes) {
            std::vector<PairSpec> pairs(1);
            pairs[0].W = s[0];
            pairs[0].H = s[1];
            pairs[0].f_full = 0.8f * s[0];
            pairs[0].xres_full = s[0];
            const Plan<float, float> P = make_plan<float, float>(pairs, params(10), nullptr, dev);
            for (const auto& d : P.steps)
                if (d.band_c > most) {
                    std::printf("clusters of up to %d: bands of %d\n", most, d.band_c);
                    return 1;
                }
        }
    }
    if (!resident || !banded || !older) return 1;
    std::printf("ok plans\n");
    return 0;
}
