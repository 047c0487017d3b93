// The longest wait between the CTAs of a resident SOR launch (k_sor_resident, rgbd-flow_b200/csrc/sor_regs.cuh)
// against the polls after which it gives up (resident_polls), on the CPU: no kernel is launched.
//
// Items take the launch's CTAs in order, as many together as fit, and a CTA goes through its items in
// order; so an item runs from when the last of its CTAs has left the item before, and the others wait for that.
#include "../../rgbd-flow_b200/csrc/pipeline.cuh"

#include <cstdio>

using namespace rgbdflow;

struct Size {
    int W, H;
};

// Seconds of the longest wait, without early stops.
static double longest_wait(const std::vector<Size>& items, int n_sor, int ctas)
{
    std::vector<int> which(items.size());
    for (size_t i = 0; i < items.size(); i++) which[i] = (int)i;
    const int kmax = resident_k(items, which, ctas);
    std::vector<double> ready(ctas, 0.0);
    double longest = 0;
    int used = 0;
    for (const Size& s : items) {
        const int K = resident_fit(s.W, s.H, kmax, ctas);
        const int n = res_tiles(s.W, kResCols, K) * res_tiles(s.H, kResRows, K);
        if (used + n > ctas) used = 0;
        double start = 0, first = 1e30;
        for (int c = used; c < used + n; c++) {
            start = std::max(start, ready[c]);
            first = std::min(first, ready[c]);
        }
        longest = std::max(longest, start - first);
        const double it = (2 * kResHalfSweep + (n > 1 ? kResExchange / K : 0.0)) * 1e3 / 1.965e9;
        for (int c = used; c < used + n; c++) ready[c] = start + n_sor * it;
        used += n;
    }
    return longest;
}

int main()
{
    const double poll = 0.35e-6;
    std::vector<std::vector<Size>> batches(3);
    for (int i = 0; i < 16; i++) batches[0].push_back({640, 480});
    for (int i = 0; i < 24; i++) batches[0].push_back({320, 240});
    for (int i = 0; i < 24; i++) batches[0].push_back({160, 120});
    batches[1].push_back({640, 480});
    for (int i = 0; i < 63; i++) batches[1].push_back({200, 150});
    batches[2].push_back({640, 480});
    bool beyond = false;  // a wait longer than the limit of a single item
    for (const auto& b : batches)
        for (int n_sor : {1, 30, 1000, 10000, 100000, 400000}) {
            const double w = longest_wait(b, n_sor, 148);
            beyond = beyond || w > kResPolls * poll;
            if (w > 0.8 * resident_polls((int)b.size(), n_sor) * poll) {
                std::printf("%zu items, %d iterations: a wait of %g s, given up after %g s\n", b.size(), n_sor, w,
                            resident_polls((int)b.size(), n_sor) * poll);
                return 1;
            }
        }
    if (!beyond) {
        std::printf("no batch here waits for earlier items\n");
        return 1;
    }
    if (resident_polls(64, 2000000000) != 1 << 30 || resident_polls(1, 2000000000) != kResPolls) return 1;
    std::printf("ok resident waits\n");
    return 0;
}
