// features.cu -- fused CSR gather -> covariance -> eigen -> feature kernels for
// compute_features, compute_features_multiscale and compute_features_optimal
// (include/pgeof.hpp:75-117, 123-211, 243-310).
//
// One thread owns one point. Its neighbours are swept twice in CSR order: the
// first sweep forms the float mean, the second the centred float products, the
// exact operation order of include/pca.hpp:75-76 (Eigen's column sums run
// sequentially), so the covariance is the one the reference forms. Multiscale
// fills every scale prefix in the same two sweeps (the reference re-gathers
// each prefix): the first keeps one running sum and takes each scale's mean
// after that scale's last neighbour -- the value the reference's own sum over
// the prefix produces -- the second keeps one product accumulator set per
// scale; the scales' covariances then wait in shared memory and one copy of
// the eigen solver handles them in turn. A warp's output rows are staged in
// its shared memory and leave as one coalesced run. The few neighbourhoods
// whose float eigenvectors are ill-conditioned are queued and solved exactly
// afterwards by features_exact_kernel.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>

#include "eig3.cuh"
#include "kernels.cuh"

namespace pgeof {

namespace {

constexpr int kFeatThreads = 128;
constexpr int kMaxScalesPerLaunch = 8;
constexpr int kSlabLoads = 8;  // index loads in flight per lane
constexpr uint32_t kApartMax = 128;  // longest rows kept an odd number of words apart in the slab
// Words between a warp's staged columns: with 33, a lane's column and a row's
// features are both free of bank conflicts (with 128 a row's features were all
// in one bank).
constexpr int kStageCol = 33;

struct FeatArgs {
    const float4* xyz4;
    uint32_t n_xyz;
    const uint32_t* nn;
    uint64_t nnz;
    const uint32_t* ptr;
    uint32_t n_points;
    uint32_t k_min;      // FULL mode gate
    int full;            // 1: compute_features (one scale = all neighbours)
    int n_scales;        // scales handled by this launch
    int scale_offset;    // first output scale column of this launch
    int out_scales;      // scales per output row
    uint32_t scales[kMaxScalesPerLaunch];
    int order;
    float* out;
    uint32_t* err;
    // multi-cloud batches: row r belongs to the cloud c with off[c] <= r < off[c+1];
    // its neighbour indices are local to that cloud's slice of xyz4
    const uint64_t* cloud_off;
    int n_clouds;
    const SPoint<float>* row_map;  // optional: row r's output row is row_map[r].idx
    uint32_t uniform_k;            // ptr == nullptr: row r is nn[r * uniform_k, (r + 1) * uniform_k)
    uint32_t row_base;             // this launch covers rows [row_base, row_base + n_points)
    int row_map_input;             // with row_map: row r also reads CSR row row_map[r].idx
    uint32_t slab_words;           // SLAB kernel: index words per warp in shared memory
    uint32_t warp_words;           // shared memory words per warp (set at the launch)
    // neighbourhoods left to the exact solve: defer[0] counts them, defer[1 ..]
    // holds their output blocks (row * out_scales + scale), whose first six
    // floats carry the covariance until features_exact_kernel replaces them
    unsigned long long* defer;
    uint64_t defer_cap;
};

// Float solve and features of one neighbourhood into f[0..10]; a neighbourhood
// that needs the exact solve gets its covariance in f[0..5] and its output
// block queued for features_exact_kernel. EXACT_INLINE runs the exact solve in
// place instead (callers without a queue).
template <bool EXACT_INLINE>
__device__ __forceinline__ void solve_or_defer(const FeatArgs& a, const Cov<float>& c, uint64_t block, float (&f)[11],
                                               uint32_t& flags) {
    Pca<float> p;
    if constexpr (EXACT_INLINE) {
        bool res;
        pca_solve_f32(c, a.order, p, res);
        features11(p, f);
        return;
    }
    if (pca_solve_f32_fast(c, a.order, p)) {
        features11(p, f);
        return;
    }
    f[0] = c.xx;
    f[1] = c.xy;
    f[2] = c.xz;
    f[3] = c.yy;
    f[4] = c.yz;
    f[5] = c.zz;
#pragma unroll
    for (int q = 6; q < 11; ++q) f[q] = 0.0f;
    const unsigned long long slot = atomicAdd(a.defer, 1ull);
    if (slot < a.defer_cap) a.defer[1 + slot] = block;
    else flags |= ERR_INTERNAL;
}

struct RowCloud {
    const float4* xyz4;
    uint32_t n;
};

__device__ __forceinline__ float4 gather_nb(const float4* xyz4, uint32_t n_xyz, uint32_t id, uint32_t& flags) {
    if (id >= n_xyz) {
        flags |= ERR_NN_RANGE;
        id = 0;
    }
    return __ldg(xyz4 + id);
}

// Calls f(j, point) for the neighbours j = 0 .. count-1 of the CSR row at
// nn + b, in order. Indices are read four at a time (16-byte loads once the
// row pointer is aligned), which quarters the L1 requests for them, and each
// group's four gathers are issued before any is used.
template <typename F>
__device__ __forceinline__ void gather_row(const uint32_t* nn_all, uint64_t b, uint32_t count, const float4* xyz4,
                                           uint32_t n_xyz, uint32_t& flags, F&& f) {
    const uint32_t* nn = nn_all + b;
    uint32_t j = 0;
    while (j < count && (reinterpret_cast<uintptr_t>(nn + j) & 15u)) {
        f(j, gather_nb(xyz4, n_xyz, __ldg(nn + j), flags));
        ++j;
    }
    for (; j + 4 <= count; j += 4) {
        const uint4 ids = __ldg(reinterpret_cast<const uint4*>(nn + j));
        const float4 p0 = gather_nb(xyz4, n_xyz, ids.x, flags), p1 = gather_nb(xyz4, n_xyz, ids.y, flags);
        const float4 p2 = gather_nb(xyz4, n_xyz, ids.z, flags), p3 = gather_nb(xyz4, n_xyz, ids.w, flags);
        f(j, p0);
        f(j + 1, p1);
        f(j + 2, p2);
        f(j + 3, p3);
    }
    for (; j < count; ++j) f(j, gather_nb(xyz4, n_xyz, __ldg(nn + j), flags));
}

// A word that is read once: not kept in L1, which the gathers need.
__device__ __forceinline__ uint32_t load_once(const uint32_t* p) {
    uint32_t v;
    asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// gather_row over indices already in shared memory (idx[0 .. count)).
template <typename F>
__device__ __forceinline__ void gather_row_slab(const uint32_t* idx, uint32_t count, const float4* xyz4,
                                                uint32_t n_xyz, uint32_t& flags, F&& f) {
    uint32_t j = 0;
    for (; j + 4 <= count; j += 4) {
        const uint32_t i0 = idx[j], i1 = idx[j + 1], i2 = idx[j + 2], i3 = idx[j + 3];
        const float4 p0 = gather_nb(xyz4, n_xyz, i0, flags), p1 = gather_nb(xyz4, n_xyz, i1, flags);
        const float4 p2 = gather_nb(xyz4, n_xyz, i2, flags), p3 = gather_nb(xyz4, n_xyz, i3, flags);
        f(j, p0);
        f(j + 1, p1);
        f(j + 2, p2);
        f(j + 3, p3);
    }
    for (; j < count; ++j) f(j, gather_nb(xyz4, n_xyz, idx[j], flags));
}

// What bounds it: the scattered 16-byte gathers, two per neighbour, of which an
// SM serves 0.9 a cycle from L1 and L2; the solver and the output hide under them.
//
// SLAB: the CSR indices of a warp's 32 consecutive rows (one contiguous range
// of nn when the rows are in CSR order) are read once into shared memory with
// coalesced loads, eight in flight per lane, and both sweeps take them from
// there -- instead of each thread reading its own row's indices from global
// memory in both sweeps, which took an L1 request per row for every four
// neighbours. Rows outside the slab (too long, out of order) read global memory.
// The staged features take the slab's place after the sweeps. (Keeping the
// first sweep's coordinates in shared memory as well, so that the second does
// not gather, left 8 to 16 warps per SM and little L1: 0.77 ms instead of 0.52 on
// three scales of 50 neighbours.)
//
// EXACT_INLINE: neighbourhoods that need the exact solve get it in place.
// Otherwise they are queued for features_exact_kernel, which keeps the rare
// exact solve (and the stack frame its call needs) out of this kernel: on the
// 1M-point scene the k = 50 single-scale kernel drops from 76 to 44 registers
// and from 0.449 to 0.387 ms, and the few hundred queued solves take one
// double-float solve's latency (~0.016 ms) in features_exact_kernel.
template <int S, bool MULTI, bool SLAB = false, bool EXACT_INLINE = false>
__device__ __forceinline__ void features_body(const FeatArgs& a) {
    extern __shared__ __align__(16) float smem_f[];
    const int tid = threadIdx.x, lane = tid & 31;
    // a warp's words: its index slab (SLAB) until both sweeps are done, then its
    // rows' features, one column per lane, columns of kStageCol words apart
    float* stage = smem_f + (size_t)(tid >> 5) * a.warp_words;
    const uint32_t i = a.row_base + blockIdx.x * kFeatThreads + tid;
    const int row_w = a.n_scales * 11;

    uint32_t flags = 0;
    const bool row_ok = i < a.row_base + a.n_points;
    uint64_t b = 0, e = 0;
    if (row_ok) {
        const uint32_t ri = a.row_map_input ? a.row_map[i].idx : i;
        if (a.ptr) {
            b = __ldg(a.ptr + ri);
            e = __ldg(a.ptr + ri + 1);
        } else {
            b = (uint64_t)i * a.uniform_k;
            e = b + a.uniform_k;
        }
    }
    const uint32_t* slab_idx = nullptr;  // this row's indices in shared memory
    if constexpr (SLAB) {
        const uint32_t vmask = __ballot_sync(0xffffffffu, row_ok);
        if (vmask && !a.row_map_input) {
            const int last = 31 - __clz(vmask);  // valid rows are a prefix of the warp
            const uint64_t s0 = __shfl_sync(0xffffffffu, b, 0), s1 = __shfl_sync(0xffffffffu, e, last);
            // rows of one even length are kept an odd number of words apart: end to
            // end, the lanes' reads meet in a few banks (rows of 32: in one, and two
            // scales took 0.42 ms)
            const uint32_t len0 = (uint32_t)__shfl_sync(0xffffffffu, e - b, 0);
            // (longer ones end to end: the last warp of a pass may hold a few rows of thousands,
            // for which the quotient below is not exact)
            const bool apart = __all_sync(0xffffffffu, !row_ok || e - b == len0) && len0 > 0 && len0 <= kApartMax &&
                               (len0 & 1u) == 0;
            if (s1 >= s0 && s1 - s0 + (apart ? 32u : 0u) <= a.slab_words && s1 <= a.nnz) {
                uint32_t* to = reinterpret_cast<uint32_t*>(stage);
                const uint32_t* from = a.nn + s0;
                const uint32_t words = (uint32_t)(s1 - s0);
                // w / len0 = w * inv >> 22 while w * len0 < 2^22 (w < 32 * len0, len0 <= kApartMax)
                const uint32_t inv = apart ? ((1u << 22) + len0 - 1) / len0 : 0u;
                uint32_t w = lane;
                for (; w + 32 * (kSlabLoads - 1) < words; w += 32 * kSlabLoads) {
                    uint32_t v[kSlabLoads];
#pragma unroll
                    for (int q = 0; q < kSlabLoads; ++q) v[q] = load_once(from + w + 32 * q);
#pragma unroll
                    for (int q = 0; q < kSlabLoads; ++q) to[w + 32 * q + ((w + 32 * q) * inv >> 22)] = v[q];
                }
                if (w < words) {
                    uint32_t v[kSlabLoads - 1];
#pragma unroll
                    for (int q = 0; q < kSlabLoads - 1; ++q)
                        if (w + 32 * q < words) v[q] = load_once(from + w + 32 * q);
#pragma unroll
                    for (int q = 0; q < kSlabLoads - 1; ++q)
                        if (w + 32 * q < words) to[w + 32 * q + ((w + 32 * q) * inv >> 22)] = v[q];
                }
                __syncwarp();
                if (row_ok && b >= s0 && e <= s1 && e >= b) slab_idx = to + (b - s0) + (apart ? lane : 0);
            }
        }
    }
    uint32_t k_nn = 0;
    uint32_t ks[S];
    int n_active = 0;
    float cxx[S], cxy[S], cxz[S], cyy[S], cyz[S], czz[S];
#pragma unroll
    for (int s = 0; s < S; ++s) cxx[s] = cxy[s] = cxz[s] = cyy[s] = cyz[s] = czz[s] = 0.0f;
    if (row_ok) {
        if (e < b || e > a.nnz) {
            flags |= ERR_PTR_RANGE;
        } else {
            k_nn = (uint32_t)(e - b);
        }
        RowCloud rc{a.xyz4, a.n_xyz};
        if (MULTI) {
            int lo = 0, hi = a.n_clouds - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (a.cloud_off[mid] <= i) lo = mid;
                else hi = mid - 1;
            }
            rc.xyz4 = a.xyz4 + a.cloud_off[lo];
            rc.n = (uint32_t)(a.cloud_off[lo + 1] - a.cloud_off[lo]);
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
            ks[s] = a.full ? k_nn : a.scales[s];
            bool act;
            if (a.full) {
                act = s == 0 && k_nn >= a.k_min;
            } else {
                act = s < a.n_scales && k_nn >= ks[s] && n_active == s;  // break at the first short scale
            }
            if (act) n_active = s + 1;
        }
        if (n_active > 0) {
            // neighbours [j0, j1) of the row in order, indices from the slab or global memory
            const auto sweep = [&](uint32_t j0, uint32_t j1, auto&& f) {
                if (SLAB && slab_idx) {
                    gather_row_slab(slab_idx + j0, j1 - j0, rc.xyz4, rc.n, flags, f);
                } else {
                    gather_row(a.nn, b + j0, j1 - j0, rc.xyz4, rc.n, flags, f);
                }
            };
            // sweep 1: one sequential float sum over the neighbours; every scale
            // is a prefix of the same list summed from the first neighbour, so
            // its sum is this running sum after its last neighbour
            float rx = 0.0f, ry = 0.0f, rz = 0.0f;
            float mx[S], my[S], mz[S];
#pragma unroll
            for (int s = 0; s < S; ++s) mx[s] = my[s] = mz[s] = 0.0f;
            // both sweeps run in segments [ks[t-1], ks[t]) between the (ascending)
            // scale sizes, so each neighbour updates only the scales that contain it
            uint32_t j0 = 0;
#pragma unroll
            for (int t = 0; t < S; ++t) {
                if (t < n_active) {
                    const uint32_t j1 = ks[t];
                    sweep(j0, j1, [&](uint32_t, const float4& p) {
                        rx = FADD(rx, p.x);
                        ry = FADD(ry, p.y);
                        rz = FADD(rz, p.z);
                    });
                    const float kk = (float)j1;
                    mx[t] = FDIV(rx, kk);
                    my[t] = FDIV(ry, kk);
                    mz[t] = FDIV(rz, kk);
                    j0 = j1;
                }
            }
            // sweep 2: centred products, sequential sums
            j0 = 0;
#pragma unroll
            for (int t = 0; t < S; ++t) {
                if (t < n_active) {
                    const uint32_t j1 = ks[t];
                    sweep(j0, j1, [&](uint32_t, const float4& p) {
#pragma unroll
                        for (int s = t; s < S; ++s) {
                            if (s < n_active) {
                                const float dx = FSUB(p.x, mx[s]);
                                const float dy = FSUB(p.y, my[s]);
                                const float dz = FSUB(p.z, mz[s]);
                                cxx[s] = FADD(cxx[s], FMUL(dx, dx));
                                cxy[s] = FADD(cxy[s], FMUL(dx, dy));
                                cxz[s] = FADD(cxz[s], FMUL(dx, dz));
                                cyy[s] = FADD(cyy[s], FMUL(dy, dy));
                                cyz[s] = FADD(cyz[s], FMUL(dy, dz));
                                czz[s] = FADD(czz[s], FMUL(dz, dz));
                            }
                        }
                    });
                    j0 = j1;
                }
            }
        }
    }
    // output block of scale s of this row
    const uint64_t dst = a.row_map && row_ok ? (uint64_t)a.row_map[i].idx : (uint64_t)i;
    const auto out_block = [&](int s) -> uint64_t { return dst * (uint64_t)a.out_scales + (uint64_t)(a.scale_offset + s); };
    __syncwarp();  // the slab is done with
    if constexpr (S == 1) {
        float f[11];
#pragma unroll
        for (int q = 0; q < 11; ++q) f[q] = 0.0f;
        if (n_active > 0) {
            const float kk = (float)ks[0];
            Cov<float> c;
            c.xx = FDIV(cxx[0], kk);
            c.xy = FDIV(cxy[0], kk);
            c.xz = FDIV(cxz[0], kk);
            c.yy = FDIV(cyy[0], kk);
            c.yz = FDIV(cyz[0], kk);
            c.zz = FDIV(czz[0], kk);
            solve_or_defer<EXACT_INLINE>(a, c, out_block(0), f, flags);
        }
#pragma unroll
        for (int q = 0; q < 11; ++q) stage[q * kStageCol + lane] = f[q];
    } else {
        // park each scale's covariance in its staging slot, then solve the
        // scales one at a time (one copy of the solver, not S)
#pragma unroll
        for (int s = 0; s < S; ++s) {
            if (s < n_active) {
                const float kk = (float)ks[s];
                float* st = stage + (s * 11) * kStageCol + lane;
                st[0 * kStageCol] = FDIV(cxx[s], kk);
                st[1 * kStageCol] = FDIV(cxy[s], kk);
                st[2 * kStageCol] = FDIV(cxz[s], kk);
                st[3 * kStageCol] = FDIV(cyy[s], kk);
                st[4 * kStageCol] = FDIV(cyz[s], kk);
                st[5 * kStageCol] = FDIV(czz[s], kk);
            }
        }
#pragma unroll 1
        for (int s = 0; s < a.n_scales; ++s) {
            float* st = stage + (s * 11) * kStageCol + lane;
            float f[11];
#pragma unroll
            for (int q = 0; q < 11; ++q) f[q] = 0.0f;
            if (s < n_active) {
                Cov<float> c;
                c.xx = st[0 * kStageCol];
                c.xy = st[1 * kStageCol];
                c.xz = st[2 * kStageCol];
                c.yy = st[3 * kStageCol];
                c.yz = st[4 * kStageCol];
                c.zz = st[5 * kStageCol];
                solve_or_defer<EXACT_INLINE>(a, c, out_block(s), f, flags);
            }
#pragma unroll
            for (int q = 0; q < 11; ++q) st[q * kStageCol] = f[q];
        }
    }
    if (flags) atomicOr(a.err, flags);
    __syncwarp();
    // the warp's rows leave in runs of row_w consecutive floats each (rows
    // processed in another order, row_map, go each to their own place)
    const uint32_t vrows = __ballot_sync(0xffffffffu, row_ok);
    const int total = __popc(vrows) * row_w;  // (valid rows are a prefix of the warp)
    const uint64_t out_w = (uint64_t)a.out_scales * 11;
    const uint64_t mine = dst * out_w + (uint64_t)a.scale_offset * 11;
    int r = 0, c = lane;
    while (c >= row_w) {
        c -= row_w;
        ++r;
    }
    const bool runs = !a.row_map && a.n_scales == a.out_scales;  // rows side by side: one run of all
    float* run = a.out + __shfl_sync(0xffffffffu, mine, 0);
    for (int t0 = 0; t0 < total; t0 += 32) {
        const uint64_t at = runs ? 0 : __shfl_sync(0xffffffffu, mine, r & 31);
        if (t0 + lane < total) {
            const float v = stage[c * kStageCol + r];
            if (runs) run[t0 + lane] = v;
            else a.out[at + c] = v;
        }
        c += 32;
        while (c >= row_w) {
            c -= row_w;
            ++r;
        }
    }
}

template <int S, bool MULTI, bool SLAB = false, bool EXACT_INLINE = false>
__global__ void __launch_bounds__(kFeatThreads) features_kernel(const __grid_constant__ FeatArgs a) {
    features_body<S, MULTI, SLAB, EXACT_INLINE>(a);
}

// The 3-scale pass compiled for 8 resident blocks per SM: 64 registers and a
// small spill instead of 76 registers and 6 blocks (1M-point scene, 50
// neighbours: 0.52 and 0.54 ms).
template <bool MULTI, bool SLAB>
__global__ void __launch_bounds__(kFeatThreads, 8) features3_kernel(const __grid_constant__ FeatArgs a) {
    features_body<3, MULTI, SLAB, false>(a);
}

// Coordinates of each CSR row's first neighbour (point 0's for an empty or
// invalid row): the key by which rows are ordered in space.
__global__ void first_nb_kernel(const float* __restrict__ xyz, uint64_t n_xyz, const uint32_t* __restrict__ nn,
                                uint64_t nnz, const uint32_t* __restrict__ ptr, uint64_t n_rows,
                                float* __restrict__ out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n_rows;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = ptr[i], e = ptr[i + 1];
        uint64_t id = 0;
        if (e > b && b < nnz) {
            id = nn[b];
            if (id >= n_xyz) id = 0;
        }
        out[3 * i] = xyz[3 * id];
        out[3 * i + 1] = xyz[3 * id + 1];
        out[3 * i + 2] = xyz[3 * id + 2];
    }
}

// The exact (float64) solve of the neighbourhoods features_kernel queued: each
// queued output block holds its float covariance in its first six floats and
// gets its 11 features in their place.
__global__ void __launch_bounds__(128) features_exact_kernel(float* __restrict__ out,
                                                             const unsigned long long* __restrict__ defer,
                                                             uint64_t cap, int order, unsigned long long* resolved) {
    const uint64_t n = min((uint64_t)defer[0], cap);
    if (resolved && blockIdx.x == 0 && threadIdx.x == 0 && n) atomicAdd(resolved, (unsigned long long)n);
    // one solve per thread: the kernel's time is one solve's latency
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x) {
        float* o = out + defer[1 + t] * 11;
        const Cov<float> c{o[0], o[1], o[2], o[3], o[4], o[5]};
        Pca<float> p;
        pca_solve_refined(c, order, p);
        float f[11];
        features11(p, f);
#pragma unroll
        for (int q = 0; q < 11; ++q) o[q] = f[q];
    }
}

__global__ void pad_xyz_kernel(const float* __restrict__ xyz, uint64_t n, float4* __restrict__ out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        out[i] = make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], 0.0f);
    }
}

// ------------------------------------------------------------------ optimal
constexpr int kOptThreads = 64;
constexpr int kOptCands = 11;      // near-tied sizes kept per point: what its output row holds beside their number
constexpr uint32_t kOptSizes = 64;  // (a bit each) points with more candidate sizes have all of them evaluated exactly

struct OptArgs {
    const float4* xyz4;
    uint32_t n_xyz;
    const uint32_t* nn;
    uint64_t nnz;
    const uint32_t* ptr;
    uint32_t n_points;
    uint32_t k_min, k_step, k_min_search;
    int order;
    float* out;  // (n, 12)
    uint32_t* err;
    unsigned long long* stats;  // [0] exact tie re-evaluations, [1] double re-solves
    // rows left to optimal_exact_kernel: their number, then the rows; a queued
    // output row carries the number of near-tied sizes and the sizes themselves
    uint32_t* queue;
};

// Packed pairs of floats: one instruction for two values, each rounded as its
// scalar form.
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float lo, float hi) {
    return ((F2)__float_as_uint(hi) << 32) | __float_as_uint(lo);
}
__device__ __forceinline__ float f2_lo(F2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float f2_hi(F2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) {  // a - b
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xbf800000bf800000ull), "l"(a));
    return r;
}

// Two Kahan-compensated running sums.
struct KSum2 {
    F2 s = 0, c = 0;
    __device__ __forceinline__ void add(F2 x) {
        const F2 y = f2_sub(x, c);
        const F2 t = f2_add(s, y);
        c = f2_sub(f2_sub(t, s), y);
        s = t;
    }
};

// The two smaller eigenvalues, about zero and about equal beside the largest one, e2:
// those of A with its principal axis v taken out, C = A - e2 v v', from the trace of C
// and the sum of its squares. v is the cross product of two rows of A - e2, scaled to
// about 1 by `scale`.
__device__ __noinline__ float2 smaller_two(const Cov<float> c, float e2, float scale) {
    const bool y = c.yy > c.xx, z = c.zz > fmaxf(c.xx, c.yy);  // the largest diagonal's row is left out
    const float xx = (c.xx - e2) * scale, yy = (c.yy - e2) * scale, zz = (c.zz - e2) * scale;
    const float xy = c.xy * scale, xz = c.xz * scale, yz = c.yz * scale;
    const float ax = z || y ? xx : xy, ay = z || y ? xy : yy, az = z || y ? xz : yz;  // row x, or y
    const float bx = z ? xy : xz, by = z ? yy : yz, bz = z ? yz : zz;                 // row z, or y
    const float vx = ay * bz - az * by, vy = az * bx - ax * bz, vz = ax * by - ay * bx;
    const float n = vx * vx + vy * vy + vz * vz;
    const float s = n > 1e-30f ? __fdividef(e2, n) : 0.0f;
    const float dx = c.xx - s * vx * vx, dy = c.yy - s * vy * vy, dz = c.zz - s * vz * vz;
    const float ex = c.xy - s * vx * vy, ey = c.xz - s * vx * vz, ez = c.yz - s * vy * vz;
    const float half = 0.5f * (dx + dy + dz), squares = dx * dx + dy * dy + dz * dz + 2.0f * (ex * ex + ey * ey + ez * ez);
    const float apart = sqrtf(fmaxf(0.5f * squares - half * half, 0.0f));
    return make_float2(half - apart, half + apart);
}

// Eigentropy (include/pca.hpp:140-150) of a covariance for ranking candidate
// sizes: the trigonometric closed form of the eigenvalues (O. K. Smith,
// "Eigenvalues of a symmetric 3x3 matrix", CACM 4(4), 1961). Every size within
// kTieBand (3e-5) of the minimum is re-evaluated exactly, so these values need
// only stay within half the band of the exact ones. The arc cosine is
// Abramowitz & Stegun 4.4.46 (error <= 2e-8) and the other functions are the
// hardware's (__cosf: absolute error < 2^-21 on [-pi, pi]; __logf): ~1e-6 in the
// eigentropy, with an exact arc cosine as with this one (300k covariances each of
// planes, volumes, isotropic and mixed points). Where the two smaller eigenvalues
// nearly meet (r near 1) the arc cosine magnifies r's rounding to 1e-4 of the largest
// one; where they are next to nothing as well, on a line, that is up to 1.4e-3 in the
// eigentropy and chose other sizes. There they come from smaller_two (6e-6 at most); the
// scan of all rows, which has no registers for it (4M rows: 3.38 -> 3.52 ms), asks for
// no more than `line`, and leaves such rows to optimal_exact_kernel.
constexpr float kLine = 0.999f;
constexpr float kThin = 0.02f;
__device__ __forceinline__ float eigentropy_scan(const Cov<float>& c) {
    const float q = (c.xx + c.yy + c.zz) * (1.0f / 3.0f);
    const float b00 = c.xx - q, b11 = c.yy - q, b22 = c.zz - q;
    const float off = c.xy * c.xy + c.xz * c.xz + c.yz * c.yz;
    const float p2 = fmaxf((b00 * b00 + b11 * b11 + b22 * b22 + 2.0f * off) * (1.0f / 6.0f), 1e-36f);
    float inv_p = rsqrtf(p2);
    inv_p *= fmaf(-0.5f * p2 * inv_p, inv_p, 1.5f);  // (its cube goes into r, which near 1 loses half its digits below)
    const float p = p2 * inv_p;
    const float det = b00 * (b11 * b22 - c.yz * c.yz) - c.xy * (c.xy * b22 - c.yz * c.xz) +
                      c.xz * (c.xy * c.yz - b11 * c.xz);
    const float r = fminf(1.0f, fmaxf(-1.0f, det * (0.5f * inv_p) * inv_p * inv_p));
    const float x = fabsf(r);
    float a = -0.0012624911f;
    a = fmaf(a, x, 0.0066700901f);
    a = fmaf(a, x, -0.0170881256f);
    a = fmaf(a, x, 0.0308918810f);
    a = fmaf(a, x, -0.0501743046f);
    a = fmaf(a, x, 0.0889789874f);
    a = fmaf(a, x, -0.2145988016f);
    a = fmaf(a, x, 1.5707963050f);
    const float y = 1.0f - x;
    a *= y > 0.0f ? y * rsqrtf(y) : 0.0f;
    const float phi = (r < 0.0f ? 3.14159265f - a : a) * (1.0f / 3.0f);
    const float e2 = q + 2.0f * p * __cosf(phi);
    float e0 = q + 2.0f * p * __cosf(phi + 2.0943951023931953f);
    float e1 = 3.0f * q - e0 - e2;
    if (r > kLine && e0 + e1 <= kThin * e2) {
        const float2 e = smaller_two(c, e2, inv_p);
        e0 = e.x;
        e1 = e.y;
    }
    const float v0 = fmaxf(e0, 0.0f), v1 = fmaxf(e1, 0.0f), v2 = fmaxf(e2, 0.0f);
    const float eps = 1e-3f;
    const float inv = __fdividef(1.0f, v0 + v1 + v2 + eps);
    const float f0 = v0 * inv, f1 = v1 * inv, f2 = v2 * inv;
    return -(f0 * __logf(f0 + eps) + f1 * __logf(f1 + eps) + f2 * __logf(f2 + eps));
}

// Covariance of the first k neighbours exactly as include/pca.hpp:75-76.
__device__ __forceinline__ Cov<float> literal_cov(const OptArgs& a, uint32_t b, uint32_t k, uint32_t& flags) {
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    gather_row(a.nn, b, k, a.xyz4, a.n_xyz, flags, [&](uint32_t, const float4& p) {
        sx = FADD(sx, p.x);
        sy = FADD(sy, p.y);
        sz = FADD(sz, p.z);
    });
    const float kk = (float)k;
    const float mx = FDIV(sx, kk), my = FDIV(sy, kk), mz = FDIV(sz, kk);
    float xx = 0.0f, xy = 0.0f, xz = 0.0f, yy = 0.0f, yz = 0.0f, zz = 0.0f;
    gather_row(a.nn, b, k, a.xyz4, a.n_xyz, flags, [&](uint32_t, const float4& p) {
        const float dx = FSUB(p.x, mx), dy = FSUB(p.y, my), dz = FSUB(p.z, mz);
        xx = FADD(xx, FMUL(dx, dx));
        xy = FADD(xy, FMUL(dx, dy));
        xz = FADD(xz, FMUL(dx, dz));
        yy = FADD(yy, FMUL(dy, dy));
        yz = FADD(yz, FMUL(dy, dz));
        zz = FADD(zz, FMUL(dz, dz));
    });
    Cov<float> c;
    c.xx = FDIV(xx, kk);
    c.xy = FDIV(xy, kk);
    c.xz = FDIV(xz, kk);
    c.yy = FDIV(yy, kk);
    c.yz = FDIV(yz, kk);
    c.zz = FDIV(zz, kk);
    return c;
}

// The reference's float eigentropy of the first k neighbours: its own
// covariance, an exact eigen solve.
__device__ __noinline__ float exact_eigentropy(const OptArgs& a, uint32_t b, uint32_t k, uint32_t& flags) {
    Pca<float> p;
    pca_solve_f64<float>(literal_cov(a, b, k, flags), a.order, &p);
    return eigentropy_of<float>(p.val);
}

// Calls f(k, dx, dy, dz) for k = 1 .. k_nn: neighbour k's offset from the first
// one. Neighbours go by aligned groups of four indices (one 16-byte read where
// the group lies inside nn), and the next group's points are on their way while
// four are handled. f appears once in the code: four copies of a scan's step
// ran out of the instruction cache (3.4 of 9 stall cycles per instruction).
template <typename F>
__device__ __forceinline__ void offset_row(const OptArgs& a, uint32_t b, uint32_t k_nn, uint32_t& flags, F&& f) {
    const uint32_t* row = a.nn + b;
    const uint32_t id0 = __ldg(row);
    const float4 p0 = gather_nb(a.xyz4, a.n_xyz, id0, flags);
    const int skip = (int)((reinterpret_cast<uintptr_t>(row) >> 2) & 3u);  // places of the first group before the row
    const int end = (int)k_nn;
    const auto indices = [&](int j) {  // of places j .. j + 3 of the row (j + skip a multiple of 4)
        const uint32_t* g = row + j;
        if (g >= a.nn && g + 4 <= a.nn + a.nnz) {
            uint4 v = __ldg(reinterpret_cast<const uint4*>(g));
            if (j < 0 || j + 4 > end) {
                if (j < 0) v.x = id0;
                if ((uint32_t)(j + 1) >= k_nn) v.y = id0;
                if ((uint32_t)(j + 2) >= k_nn) v.z = id0;
                if ((uint32_t)(j + 3) >= k_nn) v.w = id0;
            }
            return v;
        }
        uint4 v;
        v.x = (uint32_t)j < k_nn ? __ldg(g) : id0;
        v.y = (uint32_t)(j + 1) < k_nn ? __ldg(g + 1) : id0;
        v.z = (uint32_t)(j + 2) < k_nn ? __ldg(g + 2) : id0;
        v.w = (uint32_t)(j + 3) < k_nn ? __ldg(g + 3) : id0;
        return v;
    };
    uint4 ids = indices(-skip);
    float4 q0 = gather_nb(a.xyz4, a.n_xyz, ids.x, flags), q1 = gather_nb(a.xyz4, a.n_xyz, ids.y, flags);
    float4 q2 = gather_nb(a.xyz4, a.n_xyz, ids.z, flags), q3 = gather_nb(a.xyz4, a.n_xyz, ids.w, flags);
    if (4 - skip < end) ids = indices(4 - skip);
    for (int j = -skip; j < end;) {
        float4 c0 = q0, c1 = q1, c2 = q2, c3 = q3;
        if (j + 4 < end) {
            q0 = gather_nb(a.xyz4, a.n_xyz, ids.x, flags);
            q1 = gather_nb(a.xyz4, a.n_xyz, ids.y, flags);
            q2 = gather_nb(a.xyz4, a.n_xyz, ids.z, flags);
            q3 = gather_nb(a.xyz4, a.n_xyz, ids.w, flags);
            if (j + 8 < end) ids = indices(j + 8);
        }
#pragma unroll 1
        for (int t = 0; t < 4; ++t, ++j) {
            if ((uint32_t)j < k_nn) f((uint32_t)j + 1, c0.x - p0.x, c0.y - p0.y, c0.z - p0.z);
            c0 = c1;
            c1 = c2;
            c2 = c3;
        }
    }
}

// The compensated prefix moments of offset_row's points.
struct Moments {
    KSum2 s_xy, s_z, s_xx_xy, s_xz_yz, s_yy_zz;
    __device__ __forceinline__ void add(float dx, float dy, float dz) {
        const F2 d01 = f2(dx, dy), d12 = f2(dy, dz);
        s_xy.add(d01);
        s_z.add(f2(dz, 0.0f));
        s_xx_xy.add(f2_mul(f2(dx, dx), d01));
        s_xz_yz.add(f2_mul(d01, f2(dz, dz)));
        s_yy_zz.add(f2_mul(d12, d12));
    }
    __device__ __forceinline__ Cov<float> cov(uint32_t k) const {
        const float inv = __fdividef(1.0f, (float)k);
        const float mx = f2_lo(s_xy.s) * inv, my = f2_hi(s_xy.s) * inv, mz = f2_lo(s_z.s) * inv;
        Cov<float> c;
        c.xx = f2_lo(s_xx_xy.s) * inv - mx * mx;
        c.xy = f2_hi(s_xx_xy.s) * inv - mx * my;
        c.xz = f2_lo(s_xz_yz.s) * inv - mx * mz;
        c.yy = f2_lo(s_yy_zz.s) * inv - my * my;
        c.yz = f2_hi(s_xz_yz.s) * inv - my * mz;
        c.zz = f2_hi(s_yy_zz.s) * inv - mz * mz;
        return c;
    }
};

// The sizes of a row: k0, the multiples of k_step above it, and k_nn.
struct Sizes {
    uint32_t k0, step, k_nn, due;
    __device__ __forceinline__ Sizes(const OptArgs& a, uint32_t k_nn_)
        : k0(min(max(a.k_min, a.k_min_search), k_nn_)), step(a.k_step), k_nn(k_nn_), due(k0) {}
    __device__ __forceinline__ uint32_t count() const {
        const uint32_t multiples = k_nn / step - k0 / step;  // in (k0, k_nn]
        return 1 + multiples + (k_nn > k0 && k_nn % step != 0);
    }
    __device__ __forceinline__ uint32_t at(uint32_t t) const {  // the t-th of count()
        const uint64_t k = ((uint64_t)(k0 / step) + t) * step;
        return t == 0 ? k0 : (uint32_t)(k < k_nn ? k : k_nn);
    }
    __device__ __forceinline__ bool take(uint32_t k) {  // (called for k = 1, 2, ...)
        if (k == due) {
            due = step == 1 ? k + 1 : (k / step + 1) * step;
            return true;
        }
        return k == k_nn;
    }
};

constexpr float kTieBand = 3e-5f;

// include/pgeof.hpp:264-299. Candidate sizes are ranked by eigentropy from
// compensated prefix moments (O(k) gathers instead of the reference's O(k^2));
// every size whose fast eigentropy lies within kTieBand of the fast minimum is
// then re-evaluated from the reference's own covariance and an exact eigen
// solve, and the smallest exact eigentropy wins (first k on equality -- the
// reference's strict '<' scan). Features come from the winning size's
// reference covariance. Rows that need an exact solve (near-tied sizes, 0.4% of
// a scene's; small eigen-gaps) are queued for optimal_exact_kernel.
//
// What bounds it: instruction issue (72% of slots, 23 of 32 threads), after the gathers' latency
// and L1 look-ups in the scan (one random 16-byte read per neighbour). So four
// points are in flight per thread while four are handled, indices come four at
// a time, moments are summed in packed pairs, and only near-tied sizes are kept
// (one eigentropy per size took 32 KB of shared memory a block and half the
// resident warps). 4M rows of up to 64 neighbours: 5.98 -> 3.18 ms, and 0.15 ms
// for the queue. Blocks of 64 x 12 / 128 x 6 / 128 x 5 / 32 x 20 per SM: 3.16 /
// 3.20 / 3.29 / 3.22 ms.
__global__ void __launch_bounds__(kOptThreads, 12) optimal_kernel(const __grid_constant__ OptArgs a) {
    __shared__ float cand_e[kOptCands * kOptThreads];
    __shared__ uint32_t cand_k[kOptCands * kOptThreads];
    __shared__ float stage[12 * kOptThreads];
    const int tid = threadIdx.x;
    const uint32_t i = blockIdx.x * kOptThreads + tid;
#pragma unroll
    for (int f = 0; f < 12; ++f) stage[f * kOptThreads + tid] = 0.0f;
    uint32_t flags = 0;
    if (i < a.n_points) {
        const uint32_t b = __ldg(a.ptr + i), e = __ldg(a.ptr + i + 1);
        uint32_t k_nn = 0;
        bool ok = true;
        if (e < b || (uint64_t)e > a.nnz) {
            flags |= ERR_PTR_RANGE;
            ok = false;
        } else {
            k_nn = e - b;
        }
        if (ok && k_nn >= a.k_min && k_nn >= a.k_min_search && k_nn > 0) {
            Sizes sizes(a, k_nn);
            int cands = kOptCands + 1;
            if (sizes.count() <= kOptSizes) {
                cands = 0;
                float best = INFINITY;
                Moments m;
                offset_row(a, b, k_nn, flags, [&](uint32_t k, float dx, float dy, float dz) {
                    m.add(dx, dy, dz);
                    if (!sizes.take(k)) return;
                    const float ent = eigentropy_scan(m.cov(k));
                    if (!(ent <= best + kTieBand)) return;
                    if (ent < best) {
                        const bool far = !(best <= ent + kTieBand);  // no earlier size is near-tied any more
                        best = ent;
                        int kept = 0;
                        for (int t = 0; t < min(cands, kOptCands); ++t) {
                            const float et = cand_e[t * kOptThreads + tid];
                            if (et <= best + kTieBand) {
                                cand_e[kept * kOptThreads + tid] = et;
                                cand_k[kept * kOptThreads + tid] = cand_k[t * kOptThreads + tid];
                                ++kept;
                            }
                        }
                        cands = cands > kOptCands && !far ? kOptCands + 1 : kept;
                    }
                    if (cands < kOptCands) {
                        cand_e[cands * kOptThreads + tid] = ent;
                        cand_k[cands * kOptThreads + tid] = k;
                    }
                    cands = min(cands + 1, kOptCands + 1);
                });
            }
            bool queued = cands > 1;
            if (!queued) {
                const uint32_t k_opt = cands == 1 ? cand_k[tid] : sizes.k0;
                Pca<float> p;
                queued = !pca_solve_f32_fast(literal_cov(a, b, k_opt, flags), a.order, p);
                if (queued) {
                    cands = 1;
                    cand_k[tid] = k_opt;
                } else {
                    float f[11];
                    features11(p, f);
#pragma unroll
                    for (int q = 0; q < 11; ++q) stage[q * kOptThreads + tid] = f[q];
                    stage[11 * kOptThreads + tid] = (float)k_opt;
                }
            }
            if (queued) {
                a.queue[1 + atomicAdd(a.queue, 1u)] = i;
                stage[tid] = __uint_as_float((uint32_t)cands);
                for (int t = 0; t < min(cands, kOptCands); ++t)
                    stage[(1 + t) * kOptThreads + tid] = __uint_as_float(cand_k[t * kOptThreads + tid]);
            }
        }
    }
    if (flags) atomicOr(a.err, flags);
    __syncthreads();
    const uint32_t row0 = blockIdx.x * kOptThreads;
    const uint32_t rows = min((uint32_t)kOptThreads, a.n_points - row0);
    float* dst = a.out + (uint64_t)row0 * 12;
    for (int t = tid; t < (int)rows * 12; t += kOptThreads) {
        const int r = t / 12, c = t - r * 12;
        dst[t] = stage[c * kOptThreads + r];
    }
}

// The rows optimal_kernel queued, 2 to 16 lanes per row: exact eigentropies of the
// near-tied sizes (found again by a scan where they had no room; every size of
// rows with more than kOptSizes), dealt out to the lanes, which solve together, and
// an exact solve of the winner where its eigen-gap is small. What bounds it: a float64 solve is a ~40 us chain of dependent
// operations, so a row's few solves run side by side, and the queue's do instead of
// holding up one warp in eight of optimal_kernel (4M rows: 0.77 ms there, 0.23 ms
// here with one lane per row, 0.15 ms now; 17k rows: 0.07 ms, and 0.145 with two
// lanes solving in turn; 65 sizes of each of 200k rows 36.7 ms, and 74.2). More lanes
// only where rows are few: a long queue is bound by the float64 pipe (4M rows at
// kExactLanes = 64: 0.26 ms).
constexpr uint32_t kExactLanes = 16;  // per block
__global__ void __launch_bounds__(64) optimal_exact_kernel(const __grid_constant__ OptArgs a) {
    const uint32_t n = a.queue[0];
    uint32_t lanes = 16;  // per row
    while (lanes > 2 && (uint64_t)n * lanes > (uint64_t)gridDim.x * kExactLanes) lanes /= 2;
    const uint32_t part = threadIdx.x & (lanes - 1), rows = blockDim.x / lanes;
    for (uint32_t q0 = blockIdx.x * rows; q0 < n; q0 += gridDim.x * rows) {
        const uint32_t q = q0 + threadIdx.x / lanes;
        const bool valid = q < n;
        const uint32_t i = a.queue[1 + (valid ? q : q0)];
        float* out = a.out + (uint64_t)i * 12;
        const uint32_t b = __ldg(a.ptr + i), k_nn = __ldg(a.ptr + i + 1) - b;
        uint32_t flags = 0, n_exact = 0;
        const int cands = valid ? (int)__float_as_uint(out[0]) : 0;
        Sizes sizes(a, k_nn);
        uint32_t k_opt = 0xffffffffu;
        float best = INFINITY;
        if (cands == 1) {
            k_opt = __float_as_uint(out[1]);
        } else if (cands > 1) {
            const auto eval = [&](uint32_t k) {
                const float ent = exact_eigentropy(a, b, k, flags);
                ++n_exact;
                if (k_opt == 0xffffffffu || ent < best) {
                    best = ent;
                    k_opt = k;
                }
            };
            if (cands <= kOptCands) {
                for (int t = (int)part; t < cands; t += (int)lanes) eval(__float_as_uint(out[1 + t]));
            } else if (sizes.count() > kOptSizes) {
                for (uint32_t t = part; t < sizes.count(); t += lanes) eval(sizes.at(t));
            } else {
                // the scan again for its minimum, then once more for the sizes near it, a
                // bit each; the lane's own are solved after the scan, where the warp's
                // lanes solve together (solved at their place in it, they waited for one
                // another: 200k rows of a 0.5 m voxel grid, 64 neighbours, 5.2 ms)
                float low = INFINITY;
                uint64_t near = 0, mine = 0;
                for (int pass = 0; pass < 2; ++pass) {
                    Moments m;
                    Sizes each(a, k_nn);
                    uint32_t t = 0;
                    offset_row(a, b, k_nn, flags, [&](uint32_t k, float dx, float dy, float dz) {
                        m.add(dx, dy, dz);
                        if (!each.take(k)) return;
                        const float ent = eigentropy_scan(m.cov(k));
                        if (pass == 0) low = fminf(low, ent);
                        else if (ent <= low + kTieBand) near |= 1ull << t;
                        ++t;
                    });
                }
                for (uint32_t t = 0; near; near &= near - 1, ++t)
                    if ((t & (lanes - 1)) == part) mine |= near & (0ull - near);
                for (; mine; mine &= mine - 1) eval(sizes.at((uint32_t)__ffsll((long long)mine) - 1));
            }
        }
        __syncwarp();
        // the smallest eigentropy of the lanes', the smaller size on equality (a
        // NaN never replaces what came before it)
        for (uint32_t d = 1; d < lanes; d *= 2) {
            const float other = __shfl_xor_sync(0xffffffffu, best, d);
            const uint32_t other_k = __shfl_xor_sync(0xffffffffu, k_opt, d);
            const uint32_t first_k = min(k_opt, other_k), last_k = max(k_opt, other_k);
            const float first = k_opt <= other_k ? best : other, last = k_opt <= other_k ? other : best;
            const bool take = last_k != 0xffffffffu && last < first;
            k_opt = take ? last_k : first_k;
            best = take ? last : first;
        }
        if (flags) atomicOr(a.err, flags);
        if (a.stats && n_exact) atomicAdd(a.stats, (unsigned long long)n_exact);
        if (valid && part == 0) {
            flags = 0;
            if (k_opt == 0xffffffffu) k_opt = sizes.k0;
            Pca<float> p;
            bool res;
            pca_solve_f32(literal_cov(a, b, k_opt, flags), a.order, p, res);
            float f[11];
            features11(p, f);
#pragma unroll
            for (int t = 0; t < 11; ++t) out[t] = f[t];
            out[11] = (float)k_opt;
            if (flags) atomicOr(a.err, flags);
            if (a.stats && res) atomicAdd(a.stats + 1, 1ull);
        }
    }
}

}  // namespace

int pad_xyz(const float* xyz, uint64_t n, float4* out, cudaStream_t s) {
    if (n == 0) return PGEOF_OK;
    const DeviceInfo* di;
    PGEOF_TRY(current_device_info(&di));
    const unsigned blocks = (unsigned)std::min<uint64_t>(ceil_div_u(n, 256), (uint64_t)di->sm_count * 8);
    KernelTimer kt("pad_xyz_kernel", s);
    pad_xyz_kernel<<<blocks, 256, 0, s>>>(xyz, n, out);
    count_launch();
    return check_launch("pad_xyz_kernel");
}

// Index slabs (SLAB kernel); PGEOF_FEATURE_SLAB=0 turns them off.
bool use_index_slab() {
    static const bool v = [] {
        const char* e = getenv("PGEOF_FEATURE_SLAB");
        return e ? atoi(e) != 0 : true;
    }();
    return v;
}

template <int S>
static int launch_features_s(FeatArgs& a, cudaStream_t s) {
    const uint32_t stage_words = (uint32_t)a.n_scales * 11 * kStageCol;
    a.warp_words = (std::max(a.slab_words, stage_words) + 3) / 4 * 4;
    const unsigned blocks = ceil_div_u(a.n_points, kFeatThreads);
    KernelTimer kt("features_kernel", s);
    const bool slab = a.slab_words > 0;
    using Kern = void (*)(const FeatArgs);
    Kern kern = slab ? (a.n_clouds > 0 ? features_kernel<S, true, true> : features_kernel<S, false, true>)
                     : (a.n_clouds > 0 ? features_kernel<S, true> : features_kernel<S, false>);
    if constexpr (S == 3) {
        kern = slab ? (a.n_clouds > 0 ? features3_kernel<true, true> : features3_kernel<false, true>)
                    : (a.n_clouds > 0 ? features3_kernel<true, false> : features3_kernel<false, false>);
    }
    const size_t smem = (size_t)(kFeatThreads / 32) * a.warp_words * sizeof(uint32_t);
    PGEOF_TRY(cap_smem_carveout((const void*)kern, kFeatThreads, (int)smem));
    kern<<<blocks, kFeatThreads, smem, s>>>(a);
    count_launch();
    return check_launch("features_kernel");
}

static int launch_features_exact(float* out, const unsigned long long* defer, uint64_t cap,
                                 unsigned long long* resolved, cudaStream_t s) {
    const DeviceInfo* di;
    PGEOF_TRY(current_device_info(&di));
    const unsigned blocks = (unsigned)std::min<uint64_t>(ceil_div_u(cap, 128), (uint64_t)di->sm_count * 2);
    KernelTimer kt("features_exact_kernel", s);
    features_exact_kernel<<<blocks, 128, 0, s>>>(out, defer, cap, eig_order(), resolved);
    count_launch();
    return check_launch("features_exact_kernel");
}

static int launch_features_impl(FeatArgs& a, uint64_t n_points, bool full, uint64_t k_min, const uint32_t* scales,
                                int n_scales, uint64_t nnz, uint32_t uniform_k, cudaStream_t s);

int launch_features(const float4* xyz4, uint64_t n_xyz, const uint32_t* nn, uint64_t nnz, const uint32_t* ptr,
                    uint64_t n_points, bool full, uint64_t k_min, const uint32_t* scales, int n_scales,
                    float* out, unsigned long long* resolved, cudaStream_t s, const uint64_t* cloud_off,
                    int n_clouds, const SPoint<float>* row_map, uint32_t uniform_k, uint64_t row_base,
                    bool row_map_input, unsigned long long* defer, uint64_t slice_nnz) {
    if (n_points == 0) return PGEOF_OK;
    if (!full && n_scales <= 0) return PGEOF_OK;
    // queue for the exact solves: a count and one slot per output block
    const uint64_t cap = n_points * (uint64_t)(full ? 1 : n_scales);
    Scratch own;
    if (!defer) {
        PGEOF_TRY(own.alloc((cap + 1) * sizeof(unsigned long long), s));
        defer = own.as<unsigned long long>();
    }
    PGEOF_CUDA_TRY(cudaMemsetAsync(defer, 0, sizeof(unsigned long long), s));
    FeatArgs a{};
    a.defer = defer;
    a.defer_cap = cap;
    a.row_map = row_map;
    a.row_map_input = row_map && row_map_input ? 1 : 0;
    a.uniform_k = uniform_k;
    a.row_base = (uint32_t)row_base;
    a.cloud_off = cloud_off;
    a.n_clouds = cloud_off ? n_clouds : 0;
    a.xyz4 = xyz4;
    a.n_xyz = (uint32_t)n_xyz;
    a.nn = nn;
    a.nnz = nnz;
    a.ptr = ptr;
    a.n_points = (uint32_t)n_points;
    a.order = eig_order();
    a.err = device_error_word();
    a.out = out;
    PGEOF_TRY(launch_features_impl(a, n_points, full, k_min, scales, n_scales, slice_nnz ? slice_nnz : nnz, uniform_k, s));
    return launch_features_exact(out, defer, cap, resolved, s);
}

// Words of a warp's index slab, 0 for none. It holds rows of the average length
// (warps whose rows run longer read global memory), each one word further apart
// if that is even. `nnz`: the neighbours of the rows of this launch.
//
// Up to which length: while its blocks leave warps enough to hide the gathers.
// Without and with it, 1M-point scene, one scale of 50 / 80 / 100 / 128 neighbours
// 0.484 and 0.420 / 0.717 and 0.648 / 0.904 and 0.856 ms / (200k points) 0.291 and
// 0.309; two of 50 / 64 / 80 0.546 and 0.477 / 0.612 and 0.590 / 0.743 and 0.732 (200k
// points, 64 / 80: 0.178 and 0.184 / 0.203 and 0.214); three of 50 / 60 / 64 / 80 0.639 and
// 0.572 / 0.689 and 0.659 / 0.669 and 0.682 / 0.805 and 0.838; four of 50 / 80 / 100 0.780 and 0.619 / 0.903 and 0.865 / 1.074 and
// 1.156.
//
// Rows of different lengths fill it badly: half of the warps go without, and all
// pay for its room. A mean that is no whole number tells them (on kNN rows it
// is one); they have a slab while it is small. Radius rows of the same scene, mean 19 /
// 29 / 33 / 52 neighbours, two scales: 0.287 and 0.279 / 0.340 and 0.365 / 0.332 and 0.354 /
// 0.397 and 0.454 ms; three of mean 19 / 52 0.429 and 0.394 / 0.524 and 0.596.
//
// Several scales of fewer rows than one block per SM go without: there the time is one
// warp's chain of loads, to which the slab adds its own (5848 rows, two scales:
// 0.019 and 0.022 ms); the full pass of so few rows takes the same either way.
constexpr uint64_t kSlabRagged = 24;
static uint32_t index_slab_words(const FeatArgs& a, uint64_t nnz, uint32_t uniform_k, int sm_count) {
    const uint64_t k = uniform_k ? uniform_k : (nnz + a.n_points - 1) / a.n_points;
    const bool even_rows = uniform_k || nnz % a.n_points == 0;
    const uint64_t limit = !even_rows ? kSlabRagged : a.out_scales == 1 ? 100 : a.out_scales <= 3 ? 60 : 80;
    if (!a.full && a.n_points < (uint32_t)sm_count * kFeatThreads) return 0;
    if (!use_index_slab() || a.row_map_input || k < 1 || k > limit) return 0;
    return 32u * ((uint32_t)k | 1u) + 4u;
}

static int launch_features_impl(FeatArgs& a, uint64_t n_points, bool full, uint64_t k_min, const uint32_t* scales,
                                int n_scales, uint64_t nnz, uint32_t uniform_k, cudaStream_t s) {
    const DeviceInfo* di;
    PGEOF_TRY(current_device_info(&di));
    if (full) {
        a.full = 1;
        a.k_min = (uint32_t)std::min<uint64_t>(k_min, 0xffffffffull);
        a.n_scales = 1;
        a.out_scales = 1;
        a.scale_offset = 0;
        a.slab_words = index_slab_words(a, nnz, uniform_k, di->sm_count);
        return launch_features_s<1>(a, s);
    }
    a.full = 0;
    a.out_scales = n_scales;
    a.slab_words = index_slab_words(a, nnz, uniform_k, di->sm_count);
    for (int s0 = 0; s0 < n_scales; s0 += kMaxScalesPerLaunch) {
        const int cnt = std::min(kMaxScalesPerLaunch, n_scales - s0);
        a.n_scales = cnt;
        a.scale_offset = s0;
        for (int q = 0; q < cnt; ++q) a.scales[q] = scales[s0 + q];
        int st;
        if (cnt == 1) st = launch_features_s<1>(a, s);
        else if (cnt == 2) st = launch_features_s<2>(a, s);
        else if (cnt == 3) st = launch_features_s<3>(a, s);
        else if (cnt == 4) st = launch_features_s<4>(a, s);
        else if (cnt <= 6) st = launch_features_s<6>(a, s);
        else st = launch_features_s<8>(a, s);
        if (st != PGEOF_OK) return st;
    }
    return PGEOF_OK;
}

int first_neighbour_xyz(const float* xyz, uint64_t n_xyz, const uint32_t* nn, uint64_t nnz, const uint32_t* ptr,
                        uint64_t n_rows, float* out, cudaStream_t s) {
    if (n_rows == 0) return PGEOF_OK;
    const DeviceInfo* di;
    PGEOF_TRY(current_device_info(&di));
    KernelTimer kt("row_order_kernels", s);
    first_nb_kernel<<<std::min<unsigned>(ceil_div_u(n_rows, 256), (unsigned)di->sm_count * 8), 256, 0, s>>>(
        xyz, n_xyz, nn, nnz, ptr, n_rows, out);
    count_launch();
    return check_launch("first_nb_kernel");
}

int launch_optimal(const float4* xyz4, uint64_t n_xyz, const uint32_t* nn, uint64_t nnz, const uint32_t* ptr,
                   uint64_t n_points, uint32_t k_min, uint32_t k_step, uint32_t k_min_search, float* out,
                   unsigned long long* stats, cudaStream_t s) {
    if (n_points == 0) return PGEOF_OK;
    OptArgs a{};
    a.xyz4 = xyz4;
    a.n_xyz = (uint32_t)n_xyz;
    a.nn = nn;
    a.nnz = nnz;
    a.ptr = ptr;
    a.n_points = (uint32_t)n_points;
    a.k_min = k_min;
    a.k_step = k_step;
    a.k_min_search = k_min_search;
    a.order = eig_order();
    a.out = out;
    a.err = device_error_word();
    a.stats = stats;
    Scratch queue;
    PGEOF_TRY(queue.alloc((n_points + 1) * sizeof(uint32_t), s));
    a.queue = queue.as<uint32_t>();
    PGEOF_CUDA_TRY(cudaMemsetAsync(a.queue, 0, sizeof(uint32_t), s));
    const DeviceInfo* di;
    PGEOF_TRY(current_device_info(&di));
    {
        KernelTimer kt("optimal_kernel", s);
        optimal_kernel<<<ceil_div_u(n_points, kOptThreads), kOptThreads, 0, s>>>(a);
    }
    count_launch();
    PGEOF_TRY(check_launch("optimal_kernel"));
    KernelTimer kt("optimal_exact_kernel", s);
    optimal_exact_kernel<<<std::min<unsigned>(ceil_div_u(n_points, 4), (unsigned)di->sm_count * 8), 64, 0, s>>>(a);
    count_launch();
    return check_launch("optimal_exact_kernel");
}

}  // namespace pgeof

// ===========================================================================
// compute_features without any allocation (pgeof_compute_features_f32_noalloc)
//
// Some callers cannot allocate GPU memory while they call us: code running
// under a fixed device-memory budget that was reserved up front (a serving
// process that pre-sizes every buffer so it can never fail mid-request), hosts
// whose own allocator owns the device heap and forbids foreign cudaMalloc /
// pool traffic, and real-time loops where an allocation's latency or
// implicit synchronisation is not acceptable. For them this entry point
// keeps its only scratch -- the float4-padded copy of xyz that the feature
// kernel gathers from -- in the fixed array below instead of in freshly
// allocated memory. The caller still owns and passes every input and output.
//
// The array is file-scope device memory: every GPU that loads this library
// holds it (16 MiB) until the process exits, and every call shares it. Calls
// that overlap on the GPU (two streams, or two host threads) race on it and
// must be serialised by the caller. Host code only ever sees a host-side
// stand-in for the array's name, so the device address is fetched with
// cudaGetSymbolAddress on the first call on each device, with that device
// current; make that first call before any stream capture.
// ===========================================================================
static __device__ __align__(256) float4 g_noalloc_xyz4[1u << 20];
static __device__ __align__(256) uint32_t g_noalloc_err[64];

namespace pgeof {
namespace {

constexpr uint64_t kNoAllocMaxPoints = 1u << 20;  // capacity of g_noalloc_xyz4, in points
constexpr int kNoAllocMaxDevices = 64;

struct NoAllocSetup {
    std::mutex mu;
    std::atomic<bool> ready{false};
    float4* xyz4 = nullptr;   // device address of g_noalloc_xyz4
    uint32_t* err = nullptr;  // device address of g_noalloc_err
};
NoAllocSetup g_noalloc_setup[kNoAllocMaxDevices];

// Looks the arrays' device addresses up once per device. Only success is
// cached: a failed lookup (e.g. attempted during a stream capture) clears the
// error it left and is retried by the next call.
cudaError_t noalloc_setup(NoAllocSetup& st) {
    if (st.ready.load(std::memory_order_acquire)) return cudaSuccess;
    std::lock_guard<std::mutex> lk(st.mu);
    if (st.ready.load(std::memory_order_relaxed)) return cudaSuccess;
    float4* xyz4 = nullptr;
    uint32_t* err = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&xyz4, g_noalloc_xyz4);
    if (e == cudaSuccess) e = cudaGetSymbolAddress((void**)&err, g_noalloc_err);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return e;
    }
    st.xyz4 = xyz4;
    st.err = err;
    st.ready.store(true, std::memory_order_release);
    return cudaSuccess;
}

}  // namespace
}  // namespace pgeof

namespace pgeof {
int noalloc_take_errors(uint32_t* bits) {
    *bits = 0;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) {
        (void)cudaGetLastError();
        return PGEOF_OK;  // no device: nothing was ever recorded
    }
    NoAllocSetup& st = g_noalloc_setup[dev];
    if (!st.ready.load(std::memory_order_acquire)) return PGEOF_OK;  // no call on this device yet
    PGEOF_CUDA_TRY(cudaMemcpy(bits, st.err, sizeof(uint32_t), cudaMemcpyDeviceToHost));
    if (*bits) PGEOF_CUDA_TRY(cudaMemset(st.err, 0, sizeof(uint32_t)));
    return PGEOF_OK;
}
}  // namespace pgeof

extern "C" int pgeof_compute_features_f32_noalloc(const float* xyz, int64_t n_xyz, const uint32_t* nn, int64_t nnz,
                                                  const uint32_t* nn_ptr, int64_t n_points, uint64_t k_min,
                                                  float* features, uint32_t* error_bits, pgeof_stream_t stream) {
    using namespace pgeof;
    // the same argument checks as pgeof_compute_features_f32, then the capacity
    if (k_min < 1) return fail(PGEOF_ERR_INVALID_ARGUMENT, "k_min should be > 1");
    if (n_xyz < 0 || nnz < 0) return fail(PGEOF_ERR_INVALID_ARGUMENT, "negative size");
    if (n_points < 0) return fail(PGEOF_ERR_INVALID_ARGUMENT, "nn_ptr must hold at least one entry");
    if ((uint64_t)n_xyz > kNoAllocMaxPoints)
        return fail(PGEOF_ERR_INVALID_ARGUMENT,
                    "xyz has " + std::to_string(n_xyz) + " points; pgeof_compute_features_f32_noalloc holds at most " +
                        std::to_string(kNoAllocMaxPoints) + " (use pgeof_compute_features_f32)");
    if ((uint64_t)n_points > 0xfffffffeull) return fail(PGEOF_ERR_INVALID_ARGUMENT, "nn_ptr is too long");
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) {
        (void)cudaGetLastError();
        return fail(PGEOF_ERR_NO_DEVICE, std::string("no CUDA device: ") + cudaGetErrorString(e));
    }
    NoAllocSetup& st = g_noalloc_setup[dev];
    e = noalloc_setup(st);
    if (e != cudaSuccess) return fail(PGEOF_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    const cudaStream_t s = (cudaStream_t)stream;
    // without a caller word the bits accumulate in the library's word for this
    // device until pgeof_take_device_errors reads and clears it
    uint32_t* err = error_bits ? error_bits : st.err;
    if (n_points == 0) return PGEOF_OK;
    if (n_xyz > 0) {
        const unsigned blocks = (unsigned)std::min<uint64_t>(ceil_div_u((uint64_t)n_xyz, 256), 4096);
        pad_xyz_kernel<<<blocks, 256, 0, s>>>(xyz, (uint64_t)n_xyz, st.xyz4);
        count_launch();
        PGEOF_TRY(check_launch("pad_xyz_kernel (noalloc)"));
    }
    FeatArgs a{};
    a.xyz4 = st.xyz4;
    a.n_xyz = (uint32_t)n_xyz;
    a.nn = nn;
    a.nnz = (uint64_t)nnz;
    a.ptr = nn_ptr;
    a.n_points = (uint32_t)n_points;
    a.k_min = (uint32_t)std::min<uint64_t>(k_min, 0xffffffffull);
    a.full = 1;
    a.n_scales = 1;
    a.scale_offset = 0;
    a.out_scales = 1;
    a.order = eig_order();
    a.out = features;
    a.err = err;
    a.warp_words = 11 * kStageCol + 1;  // (a multiple of 4)
    const size_t smem = (size_t)(kFeatThreads / 32) * a.warp_words * sizeof(float);
    features_kernel<1, false, false, true><<<ceil_div_u((uint64_t)n_points, kFeatThreads), kFeatThreads, smem, s>>>(a);
    count_launch();
    return check_launch("features_kernel (noalloc)");
}
