// group.cuh -- interface of the grouped neighbour search (group.cu).
#pragma once

#include "kernels.cuh"

namespace pgeof {

// Queries a row of cells must hold to be searched as a group.
constexpr int kGroupMin = 8;
constexpr uint32_t kGroupMaxK = 128;
constexpr uint64_t kGroupMinQueries = 150000;

struct GroupSearch {
    GridParams g;  // single cloud
    const uint32_t* cell_start = nullptr;
    const SPoint<float>* pts = nullptr;
    CloudTable ct;                 // several clouds: ct.n > 0, g unused
    const SPoint<float>* queries = nullptr;
    uint64_t m = 0;
    int mode = MODE_KNN;
    uint32_t k = 0;
    float radius = 0.0f;
    float occupancy = 1.0f;  // points per cell around an average point, roughly
    uint32_t* counters = nullptr;  // device: two zeroed words
    void* groups = nullptr;        // device: group_scratch_bytes(m)
    // device: the zeroed length of the list of queries left over, and the list
    // (m entries: positions in `queries`)
    uint32_t* rest_count = nullptr;
    uint32_t* rest = nullptr;
    // device: group_block_words(g) words, and the list in spatial order (m
    // entries); nullptr: the list stays as it comes
    uint32_t* block_counts = nullptr;
    uint32_t* rest_sorted = nullptr;
};
size_t group_scratch_bytes(uint64_t m);
uint64_t group_block_words(const GridParams& g);  // 0: too many to put in order
// Whether a search of m queries over n points goes by groups, on any cloud or on one of
// surfaces alone (GridIndex::volume tells them apart). Without and with groups, ms:
//  * below 150k queries the groups are too few to fill the GPU (100k points, k = 32: 0.265
//    and 0.387), above 64 neighbours, which leave an SM four blocks or three, below 200k
//    (scene of 150k points, k = 80 / 100: 0.635 and 0.676 / 0.678 and 0.749; of 200k, k = 100:
//    0.881 and 0.798);
//  * queries much sparser than the points find little company in their cells (100k over
//    400k, k = 16: 0.355 and 0.444), in a volume sooner (150k over 300k uniform points, k =
//    1 / 50 / 100: 0.300 and 0.362 / 0.371 and 0.405 / 0.502 and 0.680; the scene 0.311 and
//    0.249 / 0.473 and 0.454 / 0.634 and 0.639);
//  * above 64 neighbours a volume gains nothing (200k / 1M uniform points, k = 100: 0.551 and
//    0.604 / 2.17 and 2.16), above 100 only large searches of surfaces (scene of 300k / 700k /
//    1.5M points, k = 128: 1.05 and 1.06 / 2.14 and 1.87 / 4.01 and 3.78; radii, 30 found:
//    1M points 1.11 and 1.33).
enum Groups { GROUPS_NONE = 0, GROUPS_SURFACES, GROUPS_ALL };
inline Groups use_groups(uint64_t n, uint64_t m, uint32_t k, int mode) {
    if (k > kGroupMaxK || m < (k <= 64 ? kGroupMinQueries : 200000) || 2 * m < n) return GROUPS_NONE;
    if (k > 100 && (mode == MODE_RADIUS || m < 500000 || m < n)) return GROUPS_NONE;
    return k > 64 || 4 * m < 3 * n ? GROUPS_SURFACES : GROUPS_ALL;
}
// A radius search's cells end at the radius: where a group's width of them holds fewer than
// the members a group must have, groups are not worth their cutting (1M uniform points, 5
// found, 30 kept: 0.778 and 0.939 ms without and with; the scene, whose cells hold more, 0.797
// and 0.681). A volume takes more of them (uniform points, 8 / 15 found, 30 kept: 0.85 and 0.95 /
// 0.908 and 0.888; 15 / 30 found, 64 kept: 0.923 and 1.000 / 1.066 and 1.011), and so do more than
// 64 neighbours (the scene, 100 kept, 15 / 100 found: 0.977 and 1.085 / 1.659 and 1.439).
constexpr float kRadiusWidth = 6.0f;  // x extent of a radius group, in cell edges
inline bool radius_groups_fill(double occupancy, bool volume, uint32_t k) {
    const int members = volume ? (k > 32 ? 32 : 16) : (k > 64 ? 64 : kGroupMin);
    return kRadiusWidth * (occupancy - 1.0) >= members;
}
// The cell occupancy (points sharing a cell with an average point) that suits
// it: cells of a few dozen points fill groups (1M-point scene, k = 16: 8 points
// 1.10 ms, 15 0.869 ms, 19 0.790 ms; k = 50: 25 1.29 ms, 27 1.26 ms, 31 1.21 ms).
inline double group_occupancy(uint32_t k) { return 14.0 + 0.33 * k; }
int launch_group_search(const GroupSearch& q, const SearchOut<float>& out, cudaStream_t s);

}  // namespace pgeof
