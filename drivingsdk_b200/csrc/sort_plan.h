// How the counting sort of cell_sort.cuh divides its work: what the launch decides from sizes, and what
// each CTA decides from the size of its map.
#pragma once

#include <algorithm>
#include <cstdint>

namespace msda {

constexpr int kSortThreads = 1024;
constexpr uint32_t kMaxSortParts = 8;        // most CTAs per map
constexpr uint32_t kSortCells = 24 * 1024;   // counters of one CTA: 96 KB, two CTAs per SM
constexpr uint32_t kSortRoom = 28 * 1024;    // ... and the most that two CTAs per SM may have

// How the counters of a map are kept (cell_sort.cuh).
enum class Counters { kSplit, kMerged, kAlone };

// Two levels of 14 and 53 samples per cell in two parts took 80 us split, 32 merged; at 5 per cell the two
// are equal. Alone from 16 samples per cell and CTA on.
__host__ __device__ __forceinline__ Counters counters_of(uint32_t parts, uint32_t samples, uint32_t cells) {
    const bool fits = cells <= kSortCells;
    if (parts == 1 || (fits && samples / parts >= 16u * cells)) return Counters::kAlone;
    return fits && 2u * samples >= parts * cells ? Counters::kMerged : Counters::kSplit;
}

// Maps of `samples` samples each; cells of a map on average, and at most.
struct SortShape {
    uint32_t maps, samples, mean_cells, most_cells;
};
struct SortChoice {
    uint32_t parts;   // CTAs per map
    uint32_t room;    // words of shared memory of each
    double ns;        // about how long it takes
};

// alike: all maps have the same cells, and a kernel with their one way of keeping counters is launched.
inline SortChoice choose_sort(const SortShape& s, uint32_t sm_count, bool alike) {
    SortChoice r{};
    // The cluster that is done first, by a model of the time in ns: an SM works on two CTAs at a time, 1.5
    // per sample of both (one alone takes 0.65 of the time of two); a cluster costs 8 us, and 3.1 per
    // cell and other CTA (merged) or 2.8 per sample (split). More parts have to gain a tenth: apart,
    // they leave shorter runs. (Samples alone, us: 256 maps of 80 K 258 / 227 / 208 in 1 / 4 / 8 parts,
    // 192 of 20 K 67 / 56 / 57 in 1 / 2 / 4, 96 of 107 K 111 / 127 / 95 / 84 in 1 / 2 / 4 / 8; 144 of
    // 5 K, whole sort: 17 / 28 in 1 / 2.) In a kernel that holds one way only a cluster costs 5 us (12 and 18
    // maps of 13 K samples on 1.5 K cells: 15.6 and 15.5 us in 1 part, 11.5 and 11.6 in 4, 10.2 and 13.5 in 8).
    const double cluster = alike ? 5000.0 : 8000.0;
    for (uint32_t parts = 1; parts <= kMaxSortParts; parts *= 2) {
        const uint32_t per_sm = (s.maps * parts + sm_count - 1) / sm_count;
        const double share = (per_sm / 2 + 0.65 * (per_sm % 2)) / parts;
        const double between = std::min(3.1 * s.mean_cells * (parts - 1), 2.8 * s.samples);
        const double ns = share * (1.5 * s.samples + (parts > 1 ? between : 0.0)) + (parts > 1 ? cluster : 0.0);
        if (parts == 1 || ns < 0.9 * r.ns) {
            r.ns = ns;
            r.parts = parts;
        }
    }
    // more room only where that lets every map's samples be staged (it costs L1: the encoder shape's
    // sort takes 82 instead of 69 us; one in a hundred of the whole backward where it is not needed)
    const uint32_t part = (s.samples - 1) / r.parts + 1, staged = part + s.most_cells;
    r.room = staged > kSortCells && staged <= kSortRoom && part >= 16u * s.most_cells ? kSortRoom : kSortCells;
    return r;
}

}  // namespace msda
