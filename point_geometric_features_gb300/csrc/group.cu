// group.cu -- the neighbour search of compact query groups, one query per lane
// (include/nn_search.hpp:31-132 for float clouds, k <= kGroupMaxK).
//
// Up to 32 consecutive queries in cell order that lie in one row of cells form
// a group: one block, one query per lane. Their neighbourhoods overlap, so the
// points within R of the group's box are staged in shared memory once and each
// lane takes the distance to its own query, with addresses that are the same
// for all lanes: a candidate costs ~20 warp instructions for the whole group
// (both passes), against ~45 for 32 candidates of one query when a warp owns a
// single query.
//
//  1. R: the largest k-th distance of the group solved before, with slack (a
//     radius search has its radius).
//  2. First pass: every lane counts its d^2 in a histogram of its own, one
//     column of shared memory per lane (no bank conflicts, whatever the bins).
//     The bin that reaches k bounds the k-th distance; a lane whose R-sphere
//     holds fewer than k points fails.
//  3. Second pass: candidates up to that bin go to the lane's key column at
//     their bin's cursor, so that the column is sorted but for the handful of
//     keys inside each bin, whose ranks a few comparisons give.
//  4. The columns are turned through padded tiles and leave as whole rows.
//
// The block's four warps hold the same 32 queries and split the candidates:
// key columns and histograms take ~25 KB at k = 50, and one warp per group left
// 9 warps on an SM, each waiting on itself (1M-point scene, k = 50: 2.1 ms;
// with four warps 1.0 ms, and 0.68 ms once ranks, cursors and the cut into
// groups were cheap). Bound now by instruction issue (70% of slots, ~600 warp
// instructions per query against 1,320).
//
// Queries without company (sparse regions) and lanes that fail go to a list for
// the one-query-per-warp kernel: 10% of the scene's queries, 0.30 ms. Whole
// search, scene: 1.42 -> 1.01 ms at k = 50, 1.07 -> 0.70 ms at k = 16, 2.17 ->
// 1.80 ms at k = 100; radius 0.5 / 64 on 4M points 5.81 -> 4.25 ms.
//
// Two candidates share one packed instruction (add/fma.rn.f32x2). Every packed
// operation rounds as its scalar form does, and (p - q)^2 is (q - p)^2, so
// distances are nanoflann's, bit for bit.
#include <algorithm>
#include <cmath>

#include "group.cuh"

namespace pgeof {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kBins = 64;
constexpr uint32_t kEmptyKey = 0x7f900000u;
constexpr uint32_t kMagic = 0x4b000000u;  // bits of 2^23: adding it leaves a rounded integer in the low bits
constexpr int kWarps = 4;
constexpr int kBinsPerWarp = kBins / kWarps;
// What a group may be: x gaps between consecutive members up to kGroupGap cell
// edges, about kGroupWidth wide (twice that at most).
// (1M-point scene, widths 1.5 / 2: 0.830 / 0.804 ms at k = 16, 1.211 / 1.199 ms
// at k = 50; gaps 0.75 / 1.5: 1.297 / 1.328 ms at k = 50.)
constexpr float kGroupGap = 0.75f;
constexpr float kGroupWidth = 2.0f;
// A radius search's edge is at most the radius, which in sparse clouds leaves a
// cell few points; its R does not grow with the group's own k-th distances either,
// so wider groups only bring more company (2.6M points, 33 per square metre, radius
// 0.56 / 64: one query per warp 2.35 ms, gap / width 0.75 / 2 2.42, 1 / 4 2.19, 1 / 6
// 2.18, 1.5 / 8 2.16; 400k points, 0.4 / 30: 0.41, 0.46, 0.40, 0.39, 0.38; dense
// clouds cut their runs at 32 members first: 4M points, 0.5 / 64 4.39, 4.40, 4.40, 4.41).
constexpr float kRadiusGap = 1.0f;
// (1.06 / 1.1: 1.190 / 1.211 ms on the scene, k = 50, 1.196 / 1.211 ms on
// a uniform cube.)
constexpr float kGroupSlack = 1.07f;  // R over the largest k-th distance of the group before
// An SM's shared memory, and what each resident block takes of it besides its own.
constexpr uint32_t kSmSharedBytes = 228 * 1024, kBlockSharedBytes = 1024;
constexpr uint32_t kItemGroups = 8;  // groups per work item, at most

// A group of queries: positions [first, first + len) of the sorted queries,
// their bounding box, and (several clouds) the cloud.
struct __align__(16) Group {
    uint32_t first, len_cloud;  // len | cloud << 8
    float x0, x1, y0, y1, z0, z1;
};

// Blocks of kBlockEdge cells a side, in which the queries left over are put in
// order (single clouds; counts == nullptr: no order).
constexpr int kBlockEdge = 4;
struct Blocks {
    float ox, oy, oz, inv;
    int nx, ny, nz;
    uint32_t* counts;
    __device__ __forceinline__ uint32_t of(float x, float y, float z) const {
        const int bx = (int)fminf(fmaxf((x - ox) * inv, 0.0f), (float)(nx - 1));
        const int by = (int)fminf(fmaxf((y - oy) * inv, 0.0f), (float)(ny - 1));
        const int bz = (int)fminf(fmaxf((z - oz) * inv, 0.0f), (float)(nz - 1));
        return ((uint32_t)bz * ny + by) * nx + bx;
    }
};

struct SplitArgs {
    GridParams g;
    CloudTable ct;
    const SPoint<float>* queries;
    uint64_t m;
    float gap, width;  // largest x gap between consecutive members and x extent of a group, in cell edges (y / z)
    Group* groups;
    uint32_t* group_count;
    uint32_t* rest;
    uint32_t* rest_count;
    Blocks blocks;
};

struct GroupArgs {
    GridParams g;
    const uint32_t* cell_start;
    const SPoint<float>* pts;
    CloudTable ct;
    const SPoint<float>* queries;
    uint32_t k;
    float r2;                  // radius mode
    unsigned long long zero2;  // -0 twice (see dist2x2)
    float slack;               // R over the largest k-th distance of the group before
    float first;               // R of an item's first group, in cell edges
    uint32_t cap;              // keys per lane
    uint32_t stage;            // candidates staged at once (a multiple of 32)
    const Group* groups;
    const uint32_t* group_count;
    uint32_t* work;
    uint32_t* rest;  // queries left to the one-query-per-warp kernel
    uint32_t* rest_count;
    Blocks blocks;
    void* out_idx;
    float* out_d2;
    uint32_t* out_found;
    int fill_last;
    int rows_sorted;
};

__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    return ((unsigned long long)__float_as_uint(b) << 32) | __float_as_uint(a);
}
__device__ __forceinline__ uint32_t lo32(unsigned long long v) { return (uint32_t)v; }
__device__ __forceinline__ uint32_t hi32(unsigned long long v) { return (uint32_t)(v >> 32); }

__device__ __forceinline__ int cell_floor(float v, int gdim) {
    return (int)floorf(fminf(fmaxf(v, -1.0f), (float)gdim));
}

// The rows of cells that may hold points within R of the group's box.
struct RowBox {
    float x0, x1, y0, y1, z0, z1;  // the queries' bounding box
    float R;                       // with the index margin
    int cy0, cz0, ny, rows;
};

__device__ __forceinline__ void set_radius(const GridParams& g, RowBox& b, float R) {
    b.R = R * 1.000001f + g.margin;
    b.cy0 = max(0, cell_floor((b.y0 - b.R - g.oy) * g.inv_h, g.gy));
    b.cz0 = max(0, cell_floor((b.z0 - b.R - g.oz) * g.inv_h, g.gz));
    const int cy1 = min(g.gy - 1, cell_floor((b.y1 + b.R - g.oy) * g.inv_h, g.gy));
    const int cz1 = min(g.gz - 1, cell_floor((b.z1 + b.R - g.oz) * g.inv_h, g.gz));
    b.ny = max(0, cy1 - b.cy0 + 1);
    b.rows = b.ny * max(0, cz1 - b.cz0 + 1);
}

// Points of row `row` of the box: [st, en) of the cell-ordered array.
__device__ __forceinline__ void row_run(const GridParams& g, const uint32_t* cell_start, const RowBox& b, int row,
                                        uint32_t& st, uint32_t& en) {
    st = en = 0;
    if (row >= b.rows) return;
    const int dz = row / b.ny, cy = b.cy0 + row - dz * b.ny, cz = b.cz0 + dz;
    const float ya = g.oy + (float)cy * g.h, za = g.oz + (float)cz * g.h;
    const float yb = g.oy + (float)(cy + 1) * g.h, zb = g.oz + (float)(cz + 1) * g.h;
    const float gy = fmaxf(0.0f, fmaxf(ya - b.y1, b.y0 - yb) - g.margin);
    const float gz = fmaxf(0.0f, fmaxf(za - b.z1, b.z0 - zb) - g.margin);
    const float rest = b.R * b.R - gy * gy - gz * gz;
    if (rest < 0.0f) return;
    const float bx = sqrtf(rest) + g.margin;
    const int xa = max(0, cell_floor((b.x0 - bx - g.ox) * g.inv_hx, g.gx));
    const int xb = min(g.gx - 1, cell_floor((b.x1 + bx - g.ox) * g.inv_hx, g.gx));
    if (xa > xb) return;
    const uint32_t base = ((uint32_t)cz * (uint32_t)g.gy + (uint32_t)cy) * (uint32_t)g.gx;
    st = __ldg(cell_start + base + xa);
    en = __ldg(cell_start + base + xb + 1);
}

// d^2 of two candidates: ((dx dx) + (dy dy)) + (dz dz), each operation rounded.
// A square is a fused multiply-add with -0 (`zero2`, a value the compiler does
// not know): a packed multiply that feeds a packed add is contracted with it,
// seen as last-bit differences, and a constant -0 is folded away first.
__device__ __forceinline__ unsigned long long dist2x2(unsigned long long x, unsigned long long y, unsigned long long z,
                                                      unsigned long long nx, unsigned long long ny,
                                                      unsigned long long nz, unsigned long long zero2) {
    unsigned long long t = add2(x, nx);
    unsigned long long d = fma2(t, t, zero2);
    t = add2(y, ny);
    d = add2(d, fma2(t, t, zero2));
    t = add2(z, nz);
    return add2(d, fma2(t, t, zero2));
}

// (The shared-memory assembly below names no memory clobber: its words are
// read by C++ code only across barriers.)
template <bool RADIUS>
__device__ __forceinline__ void count_one(uint32_t bits, uint32_t lim, uint32_t d2, float r2, uint32_t hbase) {
    if (RADIUS)
        asm volatile(
            "{.reg .pred p; setp.lt.u32 p, %2, %3; setp.lt.and.f32 p, %4, %5, p; @p red.shared.add.u32 [%0], %1;}" ::"r"(
                hbase + (bits << 7)),
            "r"(1u), "r"(bits), "r"(lim), "f"(__uint_as_float(d2)), "f"(r2));
    else
        asm volatile("{.reg .pred p; setp.lt.u32 p, %2, %3; @p red.shared.add.u32 [%0], %1;}" ::"r"(hbase + (bits << 7)),
                     "r"(1u), "r"(bits), "r"(lim));
}
// Four candidates: those accepted take the slot (byte address) at their bin's
// cursor, which advances, and leave d^2 and index there.
template <bool RADIUS>
__device__ __forceinline__ void take_four(const uint32_t (&bits)[4], const uint32_t (&d2)[4], const uint4& idx,
                                          uint32_t lim, float r2, uint32_t hbase) {
    if (RADIUS)
        asm volatile(
            "{.reg .pred p, q, r, s; .reg .b32 a, b, c, d;"
            "setp.lt.u32 p, %0, %12; setp.lt.and.f32 p, %4, %13, p; setp.lt.u32 q, %1, %12; setp.lt.and.f32 q, %5, %13, q;"
            "setp.lt.u32 r, %2, %12; setp.lt.and.f32 r, %6, %13, r; setp.lt.u32 s, %3, %12; setp.lt.and.f32 s, %7, %13, s;"
            "mad.lo.u32 a, %0, 128, %14; mad.lo.u32 b, %1, 128, %14; mad.lo.u32 c, %2, 128, %14; mad.lo.u32 d, %3, 128, %14;"
            "@p atom.shared.add.u32 a, [a], 256; @q atom.shared.add.u32 b, [b], 256;"
            "@r atom.shared.add.u32 c, [c], 256; @s atom.shared.add.u32 d, [d], 256;"
            "@p st.shared.f32 [a], %4; @p st.shared.u32 [a + 128], %8; @q st.shared.f32 [b], %5; @q st.shared.u32 [b + 128], %9;"
            "@r st.shared.f32 [c], %6; @r st.shared.u32 [c + 128], %10; @s st.shared.f32 [d], %7; @s st.shared.u32 [d + 128], %11;}" ::
                "r"(bits[0]), "r"(bits[1]), "r"(bits[2]), "r"(bits[3]), "f"(__uint_as_float(d2[0])),
            "f"(__uint_as_float(d2[1])), "f"(__uint_as_float(d2[2])), "f"(__uint_as_float(d2[3])), "r"(idx.x), "r"(idx.y),
            "r"(idx.z), "r"(idx.w), "r"(lim), "f"(r2), "r"(hbase));
    else
        asm volatile(
            "{.reg .pred p, q, r, s; .reg .b32 a, b, c, d;"
            "setp.lt.u32 p, %0, %12; setp.lt.u32 q, %1, %12; setp.lt.u32 r, %2, %12; setp.lt.u32 s, %3, %12;"
            "mad.lo.u32 a, %0, 128, %13; mad.lo.u32 b, %1, 128, %13; mad.lo.u32 c, %2, 128, %13; mad.lo.u32 d, %3, 128, %13;"
            "@p atom.shared.add.u32 a, [a], 256; @q atom.shared.add.u32 b, [b], 256;"
            "@r atom.shared.add.u32 c, [c], 256; @s atom.shared.add.u32 d, [d], 256;"
            "@p st.shared.f32 [a], %4; @p st.shared.u32 [a + 128], %8; @q st.shared.f32 [b], %5; @q st.shared.u32 [b + 128], %9;"
            "@r st.shared.f32 [c], %6; @r st.shared.u32 [c + 128], %10; @s st.shared.f32 [d], %7; @s st.shared.u32 [d + 128], %11;}" ::
                "r"(bits[0]), "r"(bits[1]), "r"(bits[2]), "r"(bits[3]), "f"(__uint_as_float(d2[0])),
            "f"(__uint_as_float(d2[1])), "f"(__uint_as_float(d2[2])), "f"(__uint_as_float(d2[3])), "r"(idx.x), "r"(idx.y),
            "r"(idx.z), "r"(idx.w), "r"(lim), "r"(hbase));
}

// The block's shared memory.
struct Smem {
    uint32_t* hist;   // [kBins][32] counts, then cursors; later the turned d^2, [32][T]
    uint32_t* keys;   // [cap][2][32]: d^2 bits, index; and a row after (kEmptyKey)
    float* x;         // staged candidates, [stage] each; later the turned indices, [32][T]
    float* y;
    float* z;
    uint32_t* idx;
    uint32_t* part;   // [kWarps][32]
    uint32_t* last;   // [32]
    uint32_t* take;   // [32]
    uint32_t* ctl;    // staged candidates, work item start and length, the widest bin
};
__host__ __device__ inline uint32_t tile_width(uint32_t k) { return (k + 1) | 1u; }
__host__ __device__ inline uint32_t hist_words(uint32_t k) {
    return kBins * 32 > 32 * tile_width(k) ? kBins * 32 : 32 * tile_width(k);
}
__host__ __device__ inline size_t group_smem_bytes(uint32_t k, uint32_t cap, uint32_t stage) {
    return 4 * ((size_t)hist_words(k) + 64 * ((size_t)cap + 1) + 4 * (size_t)stage + 32 * kWarps + 64 + 8);
}
__device__ __forceinline__ Smem carve(uint32_t* base, uint32_t k, uint32_t cap, uint32_t stage) {
    Smem m;
    m.hist = base;
    m.keys = m.hist + hist_words(k);
    m.x = reinterpret_cast<float*>(m.keys + 64 * (cap + 1));
    m.y = m.x + stage;
    m.z = m.y + stage;
    m.idx = reinterpret_cast<uint32_t*>(m.z + stage);
    m.part = m.idx + stage;
    m.last = m.part + 32 * kWarps;
    m.take = m.last + 32;
    m.ctl = m.take + 32;
    return m;
}

// Stages the points of the box's rows that lie within its radius of the
// queries' box; each warp takes every kWarps-th row, of them the `part`-th of
// each `parts`. More than `cap` are counted but not kept, and beyond `give_up` the
// count itself is left incomplete. (Block-wide between
// barriers; m.ctl[0] is the zeroed count.)
__device__ __forceinline__ void stage_rows(const GridParams& g, const uint32_t* cell_start, const SPoint<float>* pts,
                                           const RowBox& b, const Smem& m, uint32_t cap, int part, int parts,
                                           uint32_t give_up) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float lim = b.R * b.R * 1.00001f;
    const int rows = (b.rows + parts - 1) / parts;
    for (int rg = 0; rg < rows; rg += 32 * kWarps) {
        uint32_t st, en;
        row_run(g, cell_start, b, (rg + lane * kWarps + w) * parts + part, st, en);
        uint32_t live = __ballot_sync(FULL, en > st);
        while (live) {
            const int r = __ffs(live) - 1;
            live &= live - 1;
            const uint32_t s = __shfl_sync(FULL, st, r), e = __shfl_sync(FULL, en, r);
            for (uint32_t base = s; base < e; base += 32) {
                const bool in = base + lane < e;
                const SPoint<float> p = pts[in ? base + lane : s];
                const float dx = fmaxf(0.0f, fmaxf(b.x0 - p.x, p.x - b.x1));
                const float dy = fmaxf(0.0f, fmaxf(b.y0 - p.y, p.y - b.y1));
                const float dz = fmaxf(0.0f, fmaxf(b.z0 - p.z, p.z - b.z1));
                const bool near = in && dx * dx + dy * dy + dz * dz <= lim;
                const uint32_t mask = __ballot_sync(FULL, near);
                if (!mask) continue;
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(m.ctl, (uint32_t)__popc(mask));
                at = __shfl_sync(FULL, at, 0);
                if (at > give_up) return;
                at += __popc(mask & ((1u << lane) - 1u));
                if (near && at < cap) {
                    m.x[at] = p.x;
                    m.y[at] = p.y;
                    m.z[at] = p.z;
                    m.idx[at] = p.idx;
                }
            }
        }
    }
}

// (The last four candidates end in points at infinity.)
__device__ __forceinline__ void clear_stage(const Smem& m, uint32_t stage) {
    for (uint32_t t = threadIdx.x; t < stage / 4; t += 32 * kWarps)
        reinterpret_cast<float4*>(m.x)[t] = make_float4(INFINITY, INFINITY, INFINITY, INFINITY);
}
// One part of the rows in place of what is staged: their number in n. False
// (n = 0) when they do not fit.
__device__ __forceinline__ bool restage(const GridParams& g, const uint32_t* cell_start, const SPoint<float>* pts,
                                     const RowBox& b, const Smem& m, uint32_t stage, int part, int parts, uint32_t& n) {
    __syncthreads();
    if (threadIdx.x == 0) m.ctl[0] = 0;
    clear_stage(m, stage);
    __syncthreads();
    stage_rows(g, cell_start, pts, b, m, stage, part, parts, 0xffffffffu);
    __syncthreads();
    n = m.ctl[0];
    if (n <= stage) return true;
    n = 0;
    return false;
}

struct Four {  // four staged candidates: d^2 and histogram values, two by two
    unsigned long long d0, d1, h0, h1;
};
__device__ __forceinline__ Four eval_four(const Smem& m, uint32_t c, unsigned long long nx,
                                          unsigned long long ny, unsigned long long nz, unsigned long long zero2,
                                          unsigned long long sb2) {
    const unsigned long long magic2 = pack2(__uint_as_float(kMagic), __uint_as_float(kMagic));
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(m.x + c);
    const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(m.y + c);
    const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(m.z + c);
    Four f;
    f.d0 = dist2x2(x.x, y.x, z.x, nx, ny, nz, zero2);
    f.d1 = dist2x2(x.y, y.y, z.y, nx, ny, nz, zero2);
    f.h0 = fma2(f.d0, sb2, magic2);
    f.h1 = fma2(f.d1, sb2, magic2);
    return f;
}

// Moves rows j0 .. j0 + 3 of the lane's key column (n keys) to their
// ranks in the turned tiles. The column is sorted by bins of at most `widest`
// keys, so a key is out of place by less than that: its rank is its row, plus
// the smaller keys among the next widest - 1 rows, minus the larger ones among
// the last widest - 1; each of those rows is read once for all four. Rows behind the
// column hold larger values (kEmptyKey) than any key; as signed integers d^2 bits
// keep their order. Keys that tie keep the order of their rows (order_ties).
struct Turn {
    uint32_t* tile_d;
    uint32_t* tile_i;
    uint32_t at;    // the lane's first tile word
    uint32_t want;  // ranks that are wanted
};
constexpr int kRankRows = 4;
__device__ __forceinline__ void rank_rows(const uint32_t* col, int j0, int n, int cap, int widest, const Turn& turn) {
    int d[kRankRows], r[kRankRows];
#pragma unroll
    for (int t = 0; t < kRankRows; ++t) {
        d[t] = (int)col[64 * min(j0 + t, cap)];
        r[t] = j0 + t;
    }
#pragma unroll
    for (int t = 0; t < kRankRows; ++t)
#pragma unroll
        for (int o = t + 1; o < kRankRows; ++o) {
            const int swap = d[o] < d[t];
            r[t] += swap;
            r[o] -= swap;
        }
    const int first = max(j0 - widest + 1, 0), last = min(j0 + kRankRows + widest - 2, cap);
#pragma unroll 2
    for (int o = j0 - 1; o >= first; --o) {
        const int e = (int)col[64 * o];
#pragma unroll
        for (int t = 0; t < kRankRows; ++t) r[t] -= e > d[t];
    }
#pragma unroll 2
    for (int o = j0 + kRankRows; o <= last; ++o) {
        const int e = (int)col[64 * o];
#pragma unroll
        for (int t = 0; t < kRankRows; ++t) r[t] += e < d[t];
    }
#pragma unroll
    for (int t = 0; t < kRankRows; ++t)
        if (j0 + t < n && (uint32_t)r[t] < turn.want) {
            turn.tile_d[turn.at + r[t]] = (uint32_t)d[t];
            turn.tile_i[turn.at + r[t]] = col[64 * (j0 + t) + 32];
        }
}

// Puts the indices of a row in which distances tie in their order: among equal
// distances the smaller index comes first. td / ti: the row's keys by distance, `have`
// of them, and one more if the column has (all > have); col: the column, whose last
// `widest` keys hold the k-th distance's bin; out: the row, written by distance already.
// A run of equal distances sorts itself by counting, passed from lane to lane. One that
// the row's end cuts through takes its indices from the column. (Warp-wide call. Every key
// against all of the column took as long as a row's search: a million points on a 5 cm
// grid, k = 32 / 50: 1.64 / 2.59 ms, now 1.06 / 1.35; without ties 0.94 / 1.14.)
__device__ __noinline__ void order_ties(const uint32_t* td, const uint32_t* ti, const uint32_t* col, int have, int all,
                                        int widest, uint32_t* out) {
    const int lane = threadIdx.x & 31;
    const uint32_t dk = td[have - 1];
    const bool cut = have < all && td[have] == dk;
    int before = 0;  // the lane's keys nearer than dk
    for (int base = 0; base < have; base += 32) {
        const int j = base + lane;
        const uint32_t d = j < have ? td[j] : 0xffffffffu, i = ti[min(j, have - 1)];
        const bool in = j < have && !(cut && d == dk);
        before += in;
        const uint32_t left = __shfl_up_sync(FULL, d, 1);
        const uint32_t heads = ~__ballot_sync(FULL, lane > 0 && left == d);  // of runs of one distance
        const int start = 31 - __clz(heads & (FULL >> (31 - lane)));
        const uint32_t after = lane == 31 ? 0u : heads & (FULL << (lane + 1));
        const int stop = after ? __ffs(after) - 1 : 32;
        const int longest = __reduce_max_sync(FULL, in ? stop - start : 0);
        int r = j;
        for (int o = 1; o < longest; ++o) {
            const uint32_t up = __shfl_up_sync(FULL, i, o), down = __shfl_down_sync(FULL, i, o);
            if (lane - o >= start) r -= up > i;
            if (lane + o < stop) r += down < i;
        }
        // runs that reach beyond these 32
        if (in && start == 0)
            for (int o = base - 1; o >= 0 && td[o] == d; --o) r -= ti[o] > i;
        if (in && stop == 32)
            for (int o = base + 32; o < have && td[o] == d; ++o) r += ti[o] < i;
        if (in && r != j) out[r] = i;
    }
    __syncwarp();
    if (!cut) return;
    before = __reduce_add_sync(FULL, before);
    const int lo = max(0, all - widest);
    for (int base = lo; base < all; base += 32) {
        const int t = base + lane;
        const bool mine = t < all && col[64 * min(t, all - 1)] == dk;
        const uint32_t i = col[64 * min(t, all - 1) + 32];
        int r = before;
        if (all - lo <= 32) {
            for (uint32_t left = __ballot_sync(FULL, mine); left; left &= left - 1) r += __shfl_sync(FULL, i, __ffs(left) - 1) < i;
        } else {
            for (int o = lo; o < all; ++o) r += col[64 * o] == dk && col[64 * o + 32] < i;
        }
        if (mine && r < have) out[r] = i;
    }
}

// Cuts the sorted queries into groups, each warp kWindow consecutive ones: a
// run of queries in one row of cells, without an x gap of more than `gap` cell
// edges, is cut into equal groups of at most 32, about `width` cell edges wide;
// groups of fewer than kGroupMin, or wider than twice that, are left to the
// other kernel.
constexpr int kWindow = 256;
constexpr int kWords = kWindow / 32;
template <bool MULTI>
__global__ void __launch_bounds__(32) group_split_kernel(const __grid_constant__ SplitArgs a) {
    __shared__ float sx[kWindow], sy[kWindow], sz[kWindow];
    __shared__ uint32_t shead[kWindow];  // groups: first | len << 16, then what becomes of them
    const int lane = threadIdx.x & 31;
    const uint64_t base = (uint64_t)blockIdx.x * kWindow;
    const int n = (int)min((uint64_t)kWindow, a.m - base);
    GridParams g = a.g;
    // heads of runs: a bit each, the same on every lane
    uint32_t head[kWords + 1];
    uint32_t prev_row = 0xffffffffu;
    float prev_x = 0.0f;
    int prev_cloud = -1;
#pragma unroll
    for (int t = 0; t < kWords; ++t) {
        const int i = t * 32 + lane;
        const SPoint<float> q = a.queries[base + min(i, n - 1)];
        int ci = 0;
        if (MULTI) {
            ci = cloud_of(a.ct, base + min(i, n - 1));
            g = a.ct.g[ci];
        }
        const int cy = (int)floorf(fminf(fmaxf((q.y - g.oy) * g.inv_h, 0.0f), (float)(g.gy - 1)));
        const int cz = (int)floorf(fminf(fmaxf((q.z - g.oz) * g.inv_h, 0.0f), (float)(g.gz - 1)));
        sx[i] = q.x;
        sy[i] = q.y;
        sz[i] = q.z;
        // (a query beyond the cloud shares the border cells, however far it is: those by more than an edge stay alone)
        const float dy = fmaxf(g.oy - q.y, q.y - (g.oy + (float)g.gy * g.h));
        const float dz = fmaxf(g.oz - q.z, q.z - (g.oz + (float)g.gz * g.h));
        const bool sane = dy <= g.h && dz <= g.h && fabsf(q.x) < INFINITY;
        const uint32_t row = sane ? (uint32_t)cz * (uint32_t)g.gy + (uint32_t)cy : 0xffffffffu;
        const uint32_t up_row = __shfl_up_sync(FULL, row, 1);
        const float up_x = __shfl_up_sync(FULL, q.x, 1);
        const int up_cloud = __shfl_up_sync(FULL, ci, 1);
        const uint32_t row_before = lane ? up_row : prev_row;
        const float x_before = lane ? up_x : prev_x;
        const int cloud_before = lane ? up_cloud : prev_cloud;
        const bool same = i > 0 && i < n && row == row_before && row != 0xffffffffu && fabsf(q.x - x_before) <= a.gap * g.h &&
                          (!MULTI || ci == cloud_before);
        head[t] = __ballot_sync(FULL, !same);
        prev_row = __shfl_sync(FULL, row, 31);
        prev_x = __shfl_sync(FULL, q.x, 31);
        prev_cloud = __shfl_sync(FULL, ci, 31);
    }
    head[kWords] = FULL;
    // every query's run, and whether it heads a group of it
    int n_groups = 0;
    uint32_t rest[kWords];
    int run0 = 0;  // the run that reaches into this word from before
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kWords; ++t) {
        const int i = t * 32 + lane;
        const uint32_t at_or_before = head[t] & (FULL >> (31 - lane));
        const int first = at_or_before ? 32 * t + 31 - __clz(at_or_before) : run0;
        int next = kWindow;
#pragma unroll
        for (int u = kWords - 1; u >= t; --u) {
            const uint32_t after = u > t ? head[u] : (lane == 31 ? 0u : head[u] & (FULL << (lane + 1)));
            if (after) next = 32 * u + __ffs(after) - 1;
        }
        next = min(next, n);
        run0 = head[t] ? 32 * t + 31 - __clz(head[t]) : run0;
        const int size = max(next - first, 1);
        float h = a.g.h;
        if (MULTI) h = a.ct.g[cloud_of(a.ct, base + min(i, n - 1))].h;
        const float extent = fabsf(sx[min(first + size, n) - 1] - sx[min(first, n - 1)]);
        const int parts = min(max((size + 31) / 32, (int)ceilf(fminf(extent / (a.width * h), (float)kWindow))), size);
        const int part = (size + parts - 1) / parts;
        const int off = i - first, len = min(part, size - off);
        const bool in = i < n, lone = size < kGroupMin;
        const bool is_head = in && !lone && off % part == 0 && len >= kGroupMin;
        const bool few = min(part, size - off / part * part) < kGroupMin;  // of a part that is too short
        const uint32_t heads = __ballot_sync(FULL, is_head);
        if (is_head) shead[n_groups + __popc(heads & ((1u << lane) - 1u))] = (uint32_t)i | (uint32_t)len << 16;
        n_groups += __popc(heads);
        rest[t] = __ballot_sync(FULL, in && (lone || few));
    }
    __syncwarp();
    // one group per lane: its box (at most kWindow / kGroupMin groups)
    Group gr{};
    bool keep = false;
    int first = 0, len = 0;
    if (lane < n_groups) {
        first = (int)(shead[lane] & 0xffffu);
        len = (int)(shead[lane] >> 16);
        gr.first = (uint32_t)(base + first);
        float h = a.g.h;
        int ci = 0;
        if (MULTI) {
            ci = cloud_of(a.ct, base + first);
            h = a.ct.g[ci].h;
        }
        gr.len_cloud = (uint32_t)len | (uint32_t)ci << 8;
        gr.x0 = gr.x1 = sx[first];
        gr.y0 = gr.y1 = sy[first];
        gr.z0 = gr.z1 = sz[first];
        for (int t = 1; t < len; ++t) {
            gr.x0 = fminf(gr.x0, sx[first + t]);
            gr.x1 = fmaxf(gr.x1, sx[first + t]);
            gr.y0 = fminf(gr.y0, sy[first + t]);
            gr.y1 = fmaxf(gr.y1, sy[first + t]);
            gr.z0 = fminf(gr.z0, sz[first + t]);
            gr.z1 = fmaxf(gr.z1, sz[first + t]);
        }
        keep = gr.x1 - gr.x0 <= 2.0f * a.width * h;
    }
    const uint32_t kept = __ballot_sync(FULL, keep), wide = __ballot_sync(FULL, lane < n_groups && !keep);
    uint32_t n_rest = (lane < n_groups && !keep) ? (uint32_t)len : 0u;
    uint32_t wide_at = n_rest;  // (inclusive) prefix of the wide groups' members
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, wide_at, o);
        if (lane >= o) wide_at += y;
    }
    uint32_t total = __shfl_sync(FULL, wide_at, 31);
    wide_at -= n_rest;
    const uint32_t wide_total = total;
#pragma unroll
    for (int t = 0; t < kWords; ++t) total += __popc(rest[t]);
    uint32_t at = 0, rest_at = 0;
    if (lane == 0) {
        if (kept) at = atomicAdd(a.group_count, (uint32_t)__popc(kept));
        if (total) rest_at = atomicAdd(a.rest_count, total);
    }
    at = __shfl_sync(FULL, at, 0);
    rest_at = __shfl_sync(FULL, rest_at, 0);
    if (keep) a.groups[at + __popc(kept & ((1u << lane) - 1u))] = gr;
    if ((wide >> lane) & 1u)
        for (int t = 0; t < len; ++t) {
            a.rest[rest_at + wide_at + t] = (uint32_t)(base + first + t);
            if (a.blocks.counts) atomicAdd(a.blocks.counts + a.blocks.of(sx[first + t], sy[first + t], sz[first + t]), 1u);
        }
    rest_at += wide_total;
#pragma unroll
    for (int t = 0; t < kWords; ++t) {
        if ((rest[t] >> lane) & 1u) {
            a.rest[rest_at + __popc(rest[t] & ((1u << lane) - 1u))] = (uint32_t)(base + 32 * t + lane);
            if (a.blocks.counts)
                atomicAdd(a.blocks.counts + a.blocks.of(sx[32 * t + lane], sy[32 * t + lane], sz[32 * t + lane]), 1u);
        }
        rest_at += __popc(rest[t]);
    }
}

template <int MODE, bool MULTI>
__global__ void __launch_bounds__(32 * kWarps, 6) group_search_kernel(const __grid_constant__ GroupArgs a) {
    constexpr bool RADIUS = MODE == MODE_RADIUS;
    extern __shared__ __align__(16) uint32_t smem[];
    const Smem m = carve(smem, a.k, a.cap, a.stage);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t keys_addr = (uint32_t)__cvta_generic_to_shared(m.keys) + 4u * lane;
    const uint32_t hbase = (uint32_t)__cvta_generic_to_shared(m.hist) + 4u * lane - (kMagic << 7);
    const uint32_t k = a.k, T = tile_width(a.k);
    const uint32_t n_groups = *a.group_count;
    const unsigned long long zero2 = a.zero2;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            // items of consecutive groups, shrinking towards the end
            const uint32_t seen = __ldcg(a.work);
            const uint32_t part = (n_groups - min(seen, n_groups)) / (4 * gridDim.x);
            const uint32_t n = min(max(part, 1u), kItemGroups);
            m.ctl[1] = atomicAdd(a.work, n);
            m.ctl[2] = n;
        }
        __syncthreads();
        const uint32_t start = m.ctl[1];
        if (start >= n_groups) break;
        const uint32_t stop = min(start + m.ctl[2], n_groups);
        float r_last = -1.0f;  // the largest k-th distance of the group before
        for (uint32_t at = start; at < stop; ++at) {
            const Group gr = a.groups[at];
            const int len = (int)(gr.len_cloud & 255u);
            const uint64_t q0 = gr.first;
            const bool valid = lane < len;
            const SPoint<float> qp = a.queries[q0 + (valid ? lane : 0)];
            GridParams g = a.g;
            const uint32_t* cell_start = a.cell_start;
            uint64_t row_base = 0;
            if (MULTI) {
                const int ci = (int)(gr.len_cloud >> 8);
                g = a.ct.g[ci];
                cell_start = a.cell_start + a.ct.cell_base[ci];
                row_base = a.ct.off[ci];
            }
            uint32_t rest = len == 32 ? FULL : (1u << len) - 1u;  // members left to the other kernel
            RowBox b;
            b.x0 = gr.x0;
            b.x1 = gr.x1;
            b.y0 = gr.y0;
            b.y1 = gr.y1;
            b.z0 = gr.z0;
            b.z1 = gr.z1;
            {
                const unsigned long long nx = pack2(-qp.x, -qp.x), ny = pack2(-qp.y, -qp.y), nz = pack2(-qp.z, -qp.z);
                // ---- first pass: the bin of the k-th distance
                float R = RADIUS ? sqrtf(a.r2) : (r_last > 0.0f ? r_last * a.slack : a.first * g.h);
                bool ok = false;
                float sb = 0.0f;
                uint32_t n = 0, n_take = 0, found = 0, lim = 0;
                int parts = 1;
                float too_small = 0.0f;  // a radius known to be short
                // A radius carried from a sparse place may take in a whole dense
                // one; counted to the end, a few such groups took 1 to 3 million
                // cycles each and were the kernel's tail (256 scenes: 9.9 -> 7.4
                // ms; 33 scenes, k = 20: 2.8 -> 1.1 ms; 2 x, 4 x and 8 x alike).
                // A radius search cannot shrink: where its 64 parts could not hold
                // it, the group is left to the other kernel, as is one whose
                // rows turn out not to fit a part.
                const uint32_t give_up = a.stage * (RADIUS ? 64u : 4u);
                for (int attempt = 0; attempt < 4; ++attempt) {
                    ok = false;
                    set_radius(g, b, R);
                    __syncthreads();  // the group before has left
                    if (threadIdx.x == 0) m.ctl[0] = m.ctl[3] = 0;
                    for (uint32_t j = w; j <= a.cap; j += kWarps) m.keys[64 * j + lane] = kEmptyKey + j;
                    clear_stage(m, a.stage);
#pragma unroll
                    for (int t = 0; t < kBins * 32 / 4 / (32 * kWarps); ++t)
                        reinterpret_cast<uint4*>(m.hist)[t * 32 * kWarps + threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
                    __syncthreads();
                    parts = 1;
                    stage_rows(g, cell_start, a.pts, b, m, a.stage, 0, 1, give_up);
                    __syncthreads();
                    n = m.ctl[0];
                    if (n > a.stage) {
                        // too many: a smaller radius, unless that would be short;
                        // otherwise the rows in several parts (if all were counted)
                        float less = R * 0.95f * cbrtf((float)a.stage / (float)n);
                        if (!RADIUS && n > give_up) less = fminf(less, a.first * g.h);
                        if (!RADIUS && attempt < 2 && less > too_small * 1.02f) {
                            R = less;
                            continue;
                        }
                        if (n > give_up) break;
                        parts = (int)min((n + n / 4) / a.stage + 1, 64u);
                    }
                    if (!RADIUS && n < k) {
                        too_small = R;
                        R *= 1.4f;
                        continue;
                    }
                    sb = (float)(kBins - 1) / (R * R);
                    const unsigned long long sb2 = pack2(sb, sb);
                    // bins below the last lie wholly inside the R-sphere
                    lim = valid ? kMagic + (uint32_t)(RADIUS ? kBins : kBins - 1) : 0u;
                    bool fits = true;
                    for (int part = 0; part < parts && fits; ++part) {
                        if (parts > 1) fits = restage(g, cell_start, a.pts, b, m, a.stage, part, parts, n);
#pragma unroll 2
                        for (uint32_t c = 4 * w; c < n; c += 4 * kWarps) {
                            const Four f = eval_four(m, c, nx, ny, nz, zero2, sb2);
                            count_one<RADIUS>(lo32(f.h0), lim, lo32(f.d0), a.r2, hbase);
                            count_one<RADIUS>(hi32(f.h0), lim, hi32(f.d0), a.r2, hbase);
                            count_one<RADIUS>(lo32(f.h1), lim, lo32(f.d1), a.r2, hbase);
                            count_one<RADIUS>(hi32(f.h1), lim, hi32(f.d1), a.r2, hbase);
                        }
                    }
                    __syncthreads();
                    if (!fits) break;
                    // cursors: every bin's first slot; the bin that reaches k
                    uint32_t cnt[kBinsPerWarp], sum = 0;
#pragma unroll
                    for (int t = 0; t < kBinsPerWarp; ++t) {
                        cnt[t] = m.hist[(w * kBinsPerWarp + t) * 32 + lane];
                        sum += cnt[t];
                    }
                    m.part[w * 32 + lane] = sum;
                    __syncthreads();
                    uint32_t cum = 0;
                    found = 0;
#pragma unroll
                    for (int v = 0; v < kWarps; ++v) {
                        const uint32_t c = m.part[v * 32 + lane];
                        if (v < w) cum += c;
                        found += c;
                    }
                    const uint32_t before = cum;
                    uint32_t widest = 0, reach = cum, below = 0;  // the count through the bin that reaches k, bins below it
#pragma unroll
                    for (int t = 0; t < kBinsPerWarp; ++t) {
                        m.hist[(w * kBinsPerWarp + t) * 32 + lane] = keys_addr + 256u * cum;
                        const bool open = cum < k;
                        cum += cnt[t];
                        widest = open ? max(widest, cnt[t]) : widest;
                        reach = open ? cum : reach;
                        below += cum < k;
                    }
                    if (before < k && cum >= k) {
                        m.last[lane] = w * kBinsPerWarp + below;
                        m.take[lane] = reach;
                    }
                    widest = __reduce_max_sync(FULL, valid ? widest : 0u);
                    if (lane == 0) atomicMax(m.ctl + 3, widest);
                    __syncthreads();
                    ok = valid && (RADIUS || found >= k);
                    n_take = found >= k ? m.take[lane] : found;
                    lim = kMagic + 1u + (found >= k ? m.last[lane] : (uint32_t)kBins - 1u);
                    const uint32_t fail = __ballot_sync(FULL, valid && !ok);
                    if (RADIUS || __popc(fail) * 8 <= len) break;
                    // the shortest lane's count says how much is missing
                    const uint32_t least = __reduce_min_sync(FULL, valid ? found : 0xffffffffu);
                    too_small = R;
                    R *= fminf(fmaxf(1.06f * cbrtf((float)k / (float)max(least, 1u)), 1.1f), 1.5f);
                }
                ok = ok && n_take <= a.cap;
                if (!ok) lim = 0u;
                const uint32_t good = __ballot_sync(FULL, ok);
                rest &= ~good;
                if (good) {
                    // ---- second pass: candidates up to that bin into the key columns
                    const unsigned long long sb2 = pack2(sb, sb);
                    for (int part = 0; part < parts; ++part) {
                        if (parts > 1) restage(g, cell_start, a.pts, b, m, a.stage, part, parts, n);
#pragma unroll 2
                        for (uint32_t c = 4 * w; c < n; c += 4 * kWarps) {
                            const Four f = eval_four(m, c, nx, ny, nz, zero2, sb2);
                            const uint4 i4 = *reinterpret_cast<const uint4*>(m.idx + c);
                            const uint32_t bits[4] = {lo32(f.h0), hi32(f.h0), lo32(f.h1), hi32(f.h1)};
                            const uint32_t d2[4] = {lo32(f.d0), hi32(f.d0), lo32(f.d1), hi32(f.d1)};
                            take_four<RADIUS>(bits, d2, i4, lim, a.r2, hbase);
                        }
                    }
                    __syncthreads();
                    // ---- ranks inside the bins; keys go to their turned place
                    const uint32_t n_sel = min(n_take, k);
                    const int most = (int)__reduce_max_sync(FULL, ok ? n_take : 0u);
                    const int n_mine = ok ? (int)n_take : 0, widest = (int)m.ctl[3];
                    uint32_t* tile_i = reinterpret_cast<uint32_t*>(m.x);
                    uint32_t* tile_d = m.hist;
                    const uint32_t* col = m.keys + lane;  // row j: col[64 j] (d^2 bits), col[64 j + 32] (index)
                    // (one more than the row needs, to see a tie at its end)
                    const Turn turn{tile_d, tile_i, lane * T, ok ? n_sel + 1 : 0u};
                    for (int j0 = kRankRows * w; j0 < most; j0 += kRankRows * kWarps)
                        rank_rows(col, j0, n_mine, (int)a.cap, widest, turn);
                    __syncthreads();
                    if (!RADIUS) {
                        const uint32_t dk = ok ? tile_d[lane * T + k - 1] : 0u;
                        r_last = sqrtf(__uint_as_float(__reduce_max_sync(FULL, dk)));
                    }
                    // ---- rows out
                    const uint64_t row = a.rows_sorted ? q0 + lane : row_base + qp.idx;
                    uint32_t* out_idx = static_cast<uint32_t*>(a.out_idx);
                    const uint64_t first = reinterpret_cast<uint64_t>(out_idx) + row * k * 4;  // the row's indices
                    const ptrdiff_t to_d2 = reinterpret_cast<char*>(a.out_d2) - reinterpret_cast<char*>(out_idx);
                    uint32_t mine = good & (0x11111111u << w);  // every fourth query
                    while (mine) {
                        const int q = __ffs(mine) - 1;
                        mine &= mine - 1;
                        uint32_t* o = reinterpret_cast<uint32_t*>(__shfl_sync(FULL, first, q)) + lane;
                        const uint32_t have = RADIUS ? __shfl_sync(FULL, n_sel, q) : k;
                        const uint32_t* ti = tile_i + q * T;
                        const uint32_t* td = tile_d + q * T;
                        const uint32_t all = __shfl_sync(FULL, n_take, q);
                        bool tie = false;
                        for (uint32_t j = lane; j < k; j += 32, o += 32) {
                            uint32_t i = 0xffffffffu, d = 0u;
                            if (!RADIUS || j < have) {
                                i = ti[j];
                                d = td[j];
                                tie = tie || (j + 1 < all && td[j + 1] == d);
                            } else if (a.fill_last && j == k - 1) {
                                d = __float_as_uint(a.r2);
                            }
                            *o = i;
                            if (a.out_d2) *reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(o) + to_d2) = d;
                        }
                        if (__any_sync(FULL, tie)) {
                            __syncwarp();  // (the row as written above)
                            order_ties(td, ti, m.keys + q, (int)have, (int)all, widest,
                                       reinterpret_cast<uint32_t*>(__shfl_sync(FULL, first, q)));
                        }
                    }
                    if (RADIUS && a.out_found && ok && w == 0) a.out_found[row] = found;
                }
            }
            if (rest && w == 0) {
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(a.rest_count, (uint32_t)__popc(rest));
                at = __shfl_sync(FULL, at, 0);
                if ((rest >> lane) & 1u) {
                    a.rest[at + __popc(rest & ((1u << lane) - 1u))] = gr.first + lane;
                    if (a.blocks.counts) atomicAdd(a.blocks.counts + a.blocks.of(qp.x, qp.y, qp.z), 1u);
                }
            }
        }
    }
}

// The queries left over in the order of their blocks: neighbours in the list
// are then neighbours in space, whose k-th distances bound each other's (in
// cell order consecutive queries of a sparse region lie several of those
// distances apart along x). 4M points, radius: their search 0.607 -> 0.388 ms for 0.030 ms.
__global__ void __launch_bounds__(1024) rest_scan_kernel(uint32_t* counts, uint32_t n) {
    __shared__ uint32_t warp_sums[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < n; base += 4096) {
        uint32_t v[4], sum = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t i = base + threadIdx.x * 4 + q;
            v[q] = i < n ? counts[i] : 0u;
            sum += v[q];
        }
        uint32_t x = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sums[w] = x;
        __syncthreads();
        uint32_t all = warp_sums[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, all, o);
            if (lane >= o) all += y;
        }
        const uint32_t before = w ? __shfl_sync(FULL, all, w - 1) : 0u;
        uint32_t run = carry + before + x - sum;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t i = base + threadIdx.x * 4 + q;
            if (i < n) counts[i] = run;
            run += v[q];
        }
        carry += __shfl_sync(FULL, all, 31);
        __syncthreads();
    }
}

__global__ void rest_scatter_kernel(Blocks blocks, const SPoint<float>* __restrict__ queries,
                                    const uint32_t* __restrict__ rest, const uint32_t* __restrict__ rest_count,
                                    uint32_t* __restrict__ sorted) {
    const uint32_t n = *rest_count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t p = rest[i];
        const SPoint<float> q = queries[p];
        sorted[atomicAdd(blocks.counts + blocks.of(q.x, q.y, q.z), 1u)] = p;
    }
}

uint64_t block_count(const GridParams& g, Blocks* b) {
    const int ex = kBlockEdge * g.xsub, nx = (g.gx + ex - 1) / ex;
    const int ny = (g.gy + kBlockEdge - 1) / kBlockEdge, nz = (g.gz + kBlockEdge - 1) / kBlockEdge;
    if (b) {
        b->ox = g.ox;
        b->oy = g.oy;
        b->oz = g.oz;
        b->inv = g.inv_h / kBlockEdge;
        b->nx = nx;
        b->ny = ny;
        b->nz = nz;
    }
    return (uint64_t)nx * ny * nz;
}
// One block of threads scans them, 0.2 to 0.3 ms of a 16M-point search; without the order that
// takes 14.08 instead of 13.57 ms at k = 16, 20.37 instead of 19.72 at k = 50.
constexpr uint64_t kMaxBlocks = 1u << 20;

}  // namespace

// Largest number of groups of m queries.
uint64_t group_cap(uint64_t m) { return m / kGroupMin + 1; }
size_t group_scratch_bytes(uint64_t m) { return group_cap(m) * sizeof(Group); }
uint64_t group_block_words(const GridParams& g) {
    const uint64_t n = block_count(g, nullptr);
    return n <= kMaxBlocks ? n : 0;
}

int launch_group_search(const GroupSearch& q, const SearchOut<float>& out, cudaStream_t s) {
    const DeviceInfo* di;
    PGEOF_TRY(current_device_info(&di));
    const bool multi = q.ct.n > 0, rad = q.mode == MODE_RADIUS;
    SplitArgs sp{};
    sp.g = q.g;
    sp.ct = q.ct;
    sp.queries = q.queries;
    sp.m = q.m;
    sp.gap = rad ? kRadiusGap : kGroupGap;
    sp.width = rad ? kRadiusWidth : kGroupWidth;
    sp.groups = static_cast<Group*>(q.groups);
    sp.group_count = q.counters + 1;
    sp.rest = q.rest;
    sp.rest_count = q.rest_count;
    const uint64_t n_blocks = q.block_counts ? block_count(q.g, &sp.blocks) : 0;
    sp.blocks.counts = q.block_counts;
    if (n_blocks) PGEOF_CUDA_TRY(cudaMemsetAsync(q.block_counts, 0, n_blocks * sizeof(uint32_t), s));
    {
        KernelTimer kt("group_split_kernel", s);
        auto split = multi ? group_split_kernel<true> : group_split_kernel<false>;
        split<<<ceil_div_u(q.m, kWindow), 32, 0, s>>>(sp);
    }
    count_launch();
    PGEOF_TRY(check_launch("group_split_kernel"));
    GroupArgs a{};
    a.g = q.g;
    a.cell_start = q.cell_start;
    a.pts = q.pts;
    a.ct = q.ct;
    a.queries = q.queries;
    a.k = q.k;
    a.r2 = q.radius * q.radius;  // sq_search_radius in real_t, nn_search.hpp:98
    a.zero2 = 0x8000000080000000ull;
    a.slack = kGroupSlack;
    // k points at `occupancy` points per cell, between a surface's and a volume's
    a.first = powf((float)q.k / (2.0f * q.occupancy), 0.4f);
    a.cap = (q.k + 12 + 1) / 2 * 2;
    // At least so much room for candidates; groups beyond it go in parts. (The turned
    // indices take the same place: 32 rows of tile_width(k) words.)
    a.stage = (std::max<uint32_t>({256u, (q.k <= 64 ? 12u : 8u) * q.k + 63u, 8 * tile_width(q.k)}) + 31) / 32 * 32;
    a.groups = sp.groups;
    a.group_count = sp.group_count;
    a.work = q.counters;
    a.rest = q.rest;
    a.rest_count = q.rest_count;
    a.blocks = sp.blocks;
    a.out_idx = out.indices;
    a.out_d2 = out.sqr_dist;
    a.out_found = out.found;
    a.fill_last = out.radius_fill_last ? 1 : 0;
    a.rows_sorted = out.rows_in_query_order ? 1 : 0;
    auto kern = rad ? group_search_kernel<MODE_RADIUS, false>
                    : (multi ? group_search_kernel<MODE_KNN, true> : group_search_kernel<MODE_KNN, false>);
    int smem = (int)group_smem_bytes(a.k, a.cap, a.stage);
    int per_sm = 0;
    PGEOF_TRY(kernel_blocks_per_sm((const void*)kern, 32 * kWarps, smem, &per_sm));
    // Then all the shared memory that costs no resident block, but no more than kNN
    // groups use (a radius search stages whatever its spheres hold). Restaging parts is what
    // volumes and large radii paid before: 1M uniform points, k = 16 / 24 / 32 1.007 / 0.936 /
    // 0.974 ms with the minimum, 0.781 / 0.862 / 0.936 with 448 / 608 / 768; half as many
    // queries as points, k = 16 / 32 / 64 0.976 / 0.932 / 1.076 and 0.683 / 0.777 / 1.003;
    // radius, 180 found / 10 kept 2.293 and 1.362. The scene, k = 16 / 50: 0.812 / 1.137 and
    // 0.812 / 1.137. (One block less costs 6 to 12%.)
    const uint32_t room = kSmSharedBytes / (uint32_t)per_sm - kBlockSharedBytes;
    if (room > (uint32_t)smem) {
        const uint32_t most = a.stage + (room - (uint32_t)smem) / 16;
        const uint32_t want = std::min(rad ? most : std::min(most, 20 * q.k + 192), 2048u) / 32 * 32;
        const int larger = (int)group_smem_bytes(a.k, a.cap, std::max(a.stage, want));
        int blocks_then = 0;
        PGEOF_TRY(kernel_blocks_per_sm((const void*)kern, 32 * kWarps, larger, &blocks_then));
        if (blocks_then == per_sm) {
            a.stage = std::max(a.stage, want);
            smem = larger;
        }
    }
    const uint64_t blocks = std::min<uint64_t>(group_cap(q.m), (uint64_t)di->sm_count * per_sm);
    {
        KernelTimer kt("group_search_kernel", s);
        kern<<<(unsigned)blocks, 32 * kWarps, smem, s>>>(a);
    }
    count_launch();
    PGEOF_TRY(check_launch("group_search_kernel"));
    if (!n_blocks) return PGEOF_OK;
    KernelTimer kt("rest_order_kernels", s);
    rest_scan_kernel<<<1, 1024, 0, s>>>(q.block_counts, (uint32_t)n_blocks);
    rest_scatter_kernel<<<(unsigned)di->sm_count * 2, 256, 0, s>>>(sp.blocks, q.queries, q.rest, q.rest_count,
                                                                   q.rest_sorted);
    count_launch(2);
    return check_launch("rest_order_kernels");
}

}  // namespace pgeof
