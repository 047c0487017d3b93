// The order between the CTAs of a level's cluster (k_level_bands, rgbd-flow_b200/csrc/level_bands.cuh) around its
// convergence checks, on the CPU: no kernel is launched.
//
// A check's largest changes go into one of kBandCheckSets arrays of every CTA, whose threads read it after the
// check's cluster barrier.  The array is written again kBandCheckSets checks later; here it is shown that
// every such store comes after those reads, for every cluster size, period and reading CTA.
#include "../../rgbd-flow_b200/csrc/level_bands.cuh"

#include <cstdio>

using namespace rgbdflow;

// Whether every CTA's store for the check `sets` checks after check 0 comes after a read of check 0 by a warp of
// CTA `reader`.  after[c]: the block barrier that ends CTA c's half-sweep h comes after the read; sent[c]: so do
// the rows it sends in half-sweep h + 1.
static bool ordered(int C, int period, int reader, int sets)
{
    if (sets > 1) return true;  // the warp takes part in the next check's cluster barrier, and the store follows that
    bool after[16] = {}, sent[16] = {};
    for (int h = 0; h < 2 * period; h++) {  // the half-sweeps between the two checks
        bool now[16];
        for (int c = 0; c < C; c++) {
            // the read precedes its own CTA's next block barrier; the first half-sweep of an iteration waits
            // for the rows that the neighbours sent in the one before (the very first: sent before the check)
            now[c] = c == reader || after[c];
            if (h > 0 && c > 0) now[c] = now[c] || sent[c - 1];
            if (h > 0 && c < C - 1) now[c] = now[c] || sent[c + 1];
        }
        for (int c = 0; c < C; c++) {
            sent[c] = after[c];  // the rows of half-sweep h leave before its block barrier, after the last one's
            after[c] = now[c];
        }
    }
    // a store of the check comes after the CTA's own last block barrier, and before the check's cluster barrier
    for (int c = 0; c < C; c++)
        if (!after[c]) return false;
    return true;
}

int main()
{
    // the model finds the race of a single array, at the periods where it is one, and none at the default's
    if (ordered(16, 1, 0, 1) || ordered(2, 1, 0, 1) || ordered(16, 7, 0, 1) || !ordered(16, 25, 0, 1)) {
        std::printf("the model does not tell a race from an order\n");
        return 1;
    }
    for (int C : {1, 2, 4, 8, 16})
        for (int period = 1; period <= 64; period++)
            for (int reader = 0; reader < C; reader++)
                if (!ordered(C, period, reader, kBandCheckSets)) {
                    std::printf("race: %d CTAs, period %d, a reader in CTA %d\n", C, period, reader);
                    return 1;
                }
    std::printf("ok band checks\n");
    return 0;
}
