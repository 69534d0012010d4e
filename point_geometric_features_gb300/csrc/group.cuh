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
// Whether a search of m queries over n points goes by groups: below 150k
// queries the groups are too few to fill the GPU (100k points, k = 32: 0.265 ms
// without, 0.387 ms with), and queries much sparser than the points find little
// company in their cells (100k queries over 400k points, k = 16: 0.355 ms
// without, 0.444 ms with).
inline bool use_groups(uint64_t n, uint64_t m, uint32_t k) {
    return k <= kGroupMaxK && m >= kGroupMinQueries && 2 * m >= n;
}
// The cell occupancy (points sharing a cell with an average point) that suits
// it: cells of a few dozen points fill groups (1M-point scene, k = 16: 8 points
// 1.10 ms, 15 0.869 ms, 19 0.790 ms; k = 50: 25 1.29 ms, 27 1.26 ms, 31 1.21 ms).
inline double group_occupancy(uint32_t k) { return 14.0 + 0.33 * k; }
int launch_group_search(const GroupSearch& q, const SearchOut<float>& out, cudaStream_t s);

}  // namespace pgeof
