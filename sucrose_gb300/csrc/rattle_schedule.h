// The schedule of one molecule's RATTLE sweeps (k_rattle_wave; host code).
#pragma once
#include <algorithm>
#include <cstddef>
#include <vector>

struct WaveSlot {
    int x, y;   // a constraint's atoms, or a slot: atom i | atom j << 8 | sweep lag << 16, constraint
};

// slots[t mod period][lane], -1: empty. Constraint k of sweep s is visited at time
// o_k + period * s, o_k past that of every earlier constraint that shares an atom
// with it and the period larger than every such difference: any two visits that
// share an atom keep the list order, and those of one time share none.
struct WaveSchedule {
    int lanes = 0, period = 0;
    std::vector<WaveSlot> slots;
};

// loc: the constraints in list order, by their atoms' places in the molecule.
inline WaveSchedule wave_schedule(const std::vector<WaveSlot>& loc) {
    const int nc = (int)loc.size();
    auto share = [&](int a, int b) {
        return loc[a].x == loc[b].x || loc[a].x == loc[b].y || loc[a].y == loc[b].x || loc[a].y == loc[b].y;
    };
    std::vector<int> off(nc, 0);
    WaveSchedule w;
    w.period = 1;
    for (int k = 0; k < nc; ++k)
        for (int e = 0; e < k; ++e)
            if (share(e, k)) off[k] = std::max(off[k], off[e] + 1);
    for (int k = 0; k < nc; ++k)
        for (int e = 0; e < k; ++e)
            if (share(e, k)) w.period = std::max(w.period, off[k] - off[e] + 1);
    std::vector<int> used(w.period, 0);
    for (int k = 0; k < nc; ++k) w.lanes = std::max(w.lanes, ++used[off[k] % w.period]);
    w.slots.assign((size_t)w.period * w.lanes, WaveSlot{-1, -1});
    std::fill(used.begin(), used.end(), 0);
    for (int k = 0; k < nc; ++k) {
        const int r = off[k] % w.period;
        w.slots[(size_t)r * w.lanes + used[r]++] = {loc[k].x | loc[k].y << 8 | (off[k] / w.period) << 16, k};
    }
    return w;
}
