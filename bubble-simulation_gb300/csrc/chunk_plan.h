// Plan of the z chunks of lattices that share a persistent launch (batch.h).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <functional>
#include <utility>
#include <vector>

namespace bubble {

struct ChunkPlanGrid {
    uint32_t nx, ny, nz;
};

// Equal chunks no longer than the cap: nz cut into as few as that takes.
inline int equal_chunk(int nz, int cap) {
    const int pieces = (nz + cap - 1) / cap;
    return (nz + pieces - 1) / pieces;
}

// Chunks of the shared lattices in the strict arithmetic: one cap, the one of
// least cost, the item-planes (each chunk's planes and 2 of warm-up) spread
// over the persistent grid plus the longest item.  The IEEE divisions of the
// strict kernel leave their fast path on a fluid at rest, so items of one
// length differ up to twofold in time and balanced_chunks, which counts planes,
// cuts too coarsely: 40 steps of a 128^3 lattice are served in 28.4 ms with
// these chunks and took 38.6 with balanced_chunks', 16 of 48^3 .. 128^3 in 128 and
// 143 ms; where a round of balanced_chunks' happens to be one wave of short
// items it is ahead (96^3 8.3 ms, 9.0 here).  The fast arithmetic has no such
// path (128^3 8.5 ms with balanced_chunks, 9.0 with these, 96^3 3.9 and 4.5).
inline std::vector<int> spread_chunks(const std::vector<ChunkPlanGrid> &grids, int tx, int ty, int max_grid, int cap_max) {
    if (max_grid < 1) max_grid = 1;
    double best = 1e300;
    int best_cap = cap_max;
    for (int cap : {cap_max, 48, 32, 24, 16, 12, 8, 6, 4}) {
        if (cap > cap_max) continue;
        double planes = 0.0;
        int longest = 0;
        for (const ChunkPlanGrid &g : grids) {
            const long tiles = (long)((g.nx + tx - 1) / tx) * (long)((g.ny + ty - 1) / ty);
            const int lz = equal_chunk((int)g.nz, cap);
            const long chunks = ((long)g.nz + lz - 1) / lz;
            planes += (double)tiles * (double)(g.nz + 2 * chunks);
            longest = std::max(longest, lz + 2);
        }
        const double cost = planes / (double)max_grid + (double)longest;
        if (cost < best * (1.0 - 1e-9)) {
            best = cost;
            best_cap = cap;
        }
    }
    std::vector<int> lz;
    for (const ChunkPlanGrid &g : grids) lz.push_back(equal_chunk((int)g.nz, best_cap));
    return lz;
}

// Chunks of the shared lattices for the shortest round, in the fast arithmetic.
// Equal chunks per lattice, no longer than one cap for the first (largest)
// lattices and a smaller one for the rest, whose short items fill the round's
// end; among such plans with caps up to cap_max, the one whose round ends first
// when its items, each its planes and its warm-up's, are handed out in order to
// the persistent CTAs as they come free.  Any chunking gives the same bits.
// spread_chunks counts every round's end as a whole item, so it cuts too finely
// here, and knows one cap: 16 short solves of 48^3 .. 128^3 were served in 60.8 ms
// with it, in 57.5 ms with this, a light stream of 24 at 9.35 and 10.08 solves/s.
//
// It runs at each change of membership, while the GPU waits.  Simulating every
// plan took 0.1 ms for 16 lattices of different ragged sizes and 1.2 ms for 64
// (21 ms for 256); with the plans in the order of their lower bounds, each
// left at the time of the best, 0.02 and 0.1 ms (0.35), with the same choice.
// `grids`: the lattices, largest first.  Returns each one's chunk.
inline std::vector<int> balanced_chunks(const std::vector<ChunkPlanGrid> &grids, int tx, int ty, bool pair, int max_grid,
                                        int cap_max) {
    if (max_grid < 1) max_grid = 1;
    const double warm_up = pair ? 1.6 : 2.0;  // planes, as in the launch cost models (params.h)
    const size_t n = grids.size();
    // tiles and the items of the lattices under each cap
    struct Cut {
        int lz;
        long items;
    };
    const std::vector<int> caps = [&] {
        std::vector<int> c{cap_max};
        for (int cap : {48, 32, 24, 16, 12, 8, 6, 4})
            if (cap < cap_max) c.push_back(cap);
        return c;
    }();
    std::vector<Cut> cuts(caps.size() * n);
    std::vector<double> work(caps.size() * (n + 1), 0.0);  // plane times of the lattices before q
    std::vector<long> items(caps.size() * (n + 1), 0);
    for (size_t c = 0; c < caps.size(); ++c) {
        for (size_t q = 0; q < n; ++q) {
            const ChunkPlanGrid &g = grids[q];
            const long tiles = (long)((g.nx + tx - 1) / tx) * (long)((g.ny + ty - 1) / ty);
            const int lz = equal_chunk((int)g.nz, caps[c]);
            const long k = tiles * (((long)g.nz + lz - 1) / lz);
            cuts[c * n + q] = {lz, k};
            items[c * (n + 1) + q + 1] = items[c * (n + 1) + q] + k;
            work[c * (n + 1) + q + 1] = work[c * (n + 1) + q] + (double)k * (lz + warm_up);
        }
    }
    struct Plan {
        double bound;  // no round with these cuts ends sooner: the work spread evenly
        double pace;
        size_t a, b, split;  // caps, first lattice of the second one
        size_t rank;         // of equally short plans the first listed is taken
    };
    std::vector<Plan> plans;
    auto add = [&](size_t a, size_t b, size_t split) {
        const size_t m = n + 1;
        const long total = items[a * m + split] + (items[b * m + n] - items[b * m + split]);
        const double all = work[a * m + split] + (work[b * m + n] - work[b * m + split]);
        // CTAs with an SM to themselves, or shared by two, are faster
        const double pace = !pair ? 1.0 : 3 * total <= max_grid ? 0.57 : 3 * total <= 2 * (long)max_grid ? 0.77 : 1.0;
        plans.push_back({pace * all / max_grid, pace, a, b, split, plans.size()});
    };
    for (size_t c = 0; c < caps.size(); ++c) {
        add(c, c, n);
        for (size_t r = c + 1; r < caps.size(); ++r)
            if (caps[r] == 16 || caps[r] == 8 || caps[r] == 4)
                for (size_t split : {n / 4, n / 2, 3 * n / 4})
                    if (split > 0) add(c, r, split);
    }
    // The round of a plan in plane times, or any time beyond `stop`.
    std::vector<std::pair<double, int>> busy;  // (time, CTAs that come free then), a heap
    auto round_time = [&](const Plan &p, double stop) {
        const auto later = std::greater<std::pair<double, int>>();
        busy.assign(1, {0.0, max_grid});
        double end = 0.0;
        for (size_t q = 0; q < n && end <= stop;) {
            const size_t c = q < p.split ? p.a : p.b;
            const Cut cut = cuts[c * n + q];
            const double t_item = cut.lz + warm_up;
            long left = 0;  // items of this lattice and of those cut alike behind it
            for (; q < n && (q < p.split ? p.a : p.b) == c && cuts[c * n + q].lz == cut.lz; ++q) left += cuts[c * n + q].items;
            while (left > 0) {
                std::pop_heap(busy.begin(), busy.end(), later);
                const auto [t, ctas] = busy.back();
                busy.pop_back();
                const int take = (int)std::min<long>(left, ctas);
                left -= take;
                end = std::max(end, t + t_item);
                busy.emplace_back(t + t_item, take);
                std::push_heap(busy.begin(), busy.end(), later);
                if (take < ctas) {
                    busy.emplace_back(t, ctas - take);
                    std::push_heap(busy.begin(), busy.end(), later);
                }
            }
        }
        return end;
    };
    // the plans likely to be short first: the others are then ruled out by their
    // bound or on the way
    std::stable_sort(plans.begin(), plans.end(), [](const Plan &x, const Plan &y) { return x.bound < y.bound; });
    const Plan *best = nullptr;
    double shortest = 1e300;
    for (const Plan &p : plans) {
        const double tie = shortest * (1.0 + 1e-9);
        if (p.bound > tie) break;
        const double cost = p.pace * round_time(p, tie / p.pace);
        if (cost < shortest * (1.0 - 1e-9) || (cost <= tie && p.rank < best->rank)) {
            shortest = cost;
            best = &p;
        }
    }
    std::vector<int> lz(n);
    for (size_t q = 0; q < n; ++q) lz[q] = cuts[(q < best->split ? best->a : best->b) * n + q].lz;
    return lz;
}

}  // namespace bubble
