// The drainage tree on the device: FlowRouting.drainageOrder and accumulate
// (FlowRouting.kt:485-511, 695-729), HydraulicErosion.incise (HydraulicErosion.kt:2298-2390) and
// FlowRouting.spillways (FlowRouting.kt:573-677), each reproducing the reference's result exactly.
//
// Kahn order without a queue. The reference seeds a FIFO with the land sources in index order and
// appends a cell when its last donor leaves the queue, so the queue is sorted by level (the longest
// donor chain into a cell) and, within a level, by the position of the last donor to leave. By
// induction that is the order of the chain of "deepest latest" donors back to a source, i.e. of
// that source's index. So a cell's place is the key (level, s), s the largest source index among the
// sources farthest upstream of it, and key(r) = max over donors of key(d) + (1, 0): a tree
// reduction from the leaves. It runs as a last-arriver walk: one thread per source climbs down its
// receivers; at each cell the thread that brings the donor count to zero computes the cell's key and
// its accumulation (its weight plus its donors' areas in key order, the reference's float
// additions in the reference's order) and carries on; the others stop. No barrier, O(N) work.
//
// Incision needs each receiver final before its donors: cells are bucketed by their Kahn level (a
// receiver's level is always higher than its donors') and one cooperative kernel gathers what the sweep
// cannot change and then sweeps the levels from the top down with a grid barrier between them. Every order with receivers first gives the
// same bits, because a cell reads only its receiver's final state.
#include <cooperative_groups.h>
#include <cuda/atomic>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <utility>
#include <vector>

#include "cg_common.cuh"
#include "cg_internal.h"
#include "cg_util.h"

namespace cg {

namespace cgr = cooperative_groups;

namespace {

constexpr long long LEVEL_ONE = 1LL << 32;

__device__ __forceinline__ bool is_land_receiver(const uint8_t* land, int r) { return r >= 0 && land[r]; }

// Neighbour directions in stencil order (rows -1..1, then columns -1..1, the cell itself left out).
__device__ __forceinline__ int dir_row(int t) { return t < 3 ? -1 : (t < 5 ? 0 : 1); }
__device__ __forceinline__ int dir_col(int t) { return t < 3 ? t - 1 : (t < 5 ? (t == 3 ? -1 : 1) : t - 6); }
__device__ __forceinline__ int dir_of(int rs, int cs) { return (rs + 1) * 3 + (cs + 1) - ((rs > 0 || (rs == 0 && cs > 0)) ? 1 : 0); }
__device__ __forceinline__ int step_to(int W, int c, int t) {
    const int row = pdiv(c, W), col = pmod(c, W);
    return (row + dir_row(t)) * W + wrap_col(col + dir_col(t), W);
}

// The tree's links, one byte each per cell: down[c] the direction from c to its receiver when that
// receiver is land (0xFF otherwise), and mask[r] bit t set when the neighbour of r in direction t
// drains into r. The mask bytes are set with a 32-bit atomicOr on the word holding them.
__global__ void k_links(const uint8_t* __restrict__ land, const int32_t* __restrict__ recv, int W, int H,
                        uint8_t* __restrict__ down, uint8_t* __restrict__ mask) {
    const size_t N = (size_t)W * H;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        uint8_t d = 0xFF;
        if (land[i]) {
            const int r = recv[i];
            if (is_land_receiver(land, r)) {
                const int c = (int)i;
                int rs = pdiv(r, W) - pdiv(c, W);
                int cs = pmod(r, W) - pmod(c, W);
                if (cs > 1) cs -= W;
                if (cs < -1) cs += W;
                d = (uint8_t)dir_of(rs, cs);
                const int up = dir_of(-rs, -cs);   // from r back to c
                atomicOr(reinterpret_cast<unsigned*>(mask + (r & ~3)), 1u << (up + 8 * (r & 3)));
            }
        }
        down[i] = d;
    }
}

// Donor counts, the pending counts of the walk, and the list of land sources (cells no land cell
// drains into). A CTA takes SRC_PER cells per thread at a time and reserves its sources' slots with
// one atomic (a per-warp atomic on the one counter was the kernel's cost); the list's order does not
// matter, since the walk's results do not depend on which thread reaches a cell first.
constexpr int SRC_PER = 8;

__global__ void __launch_bounds__(256) k_sources(const uint8_t* __restrict__ land, const uint8_t* __restrict__ mask,
                                                 size_t N, int32_t* __restrict__ donors,
                                                 int32_t* __restrict__ pending, int* __restrict__ sources,
                                                 int* __restrict__ n_sources) {
    const unsigned FULL = 0xFFFFFFFFu;
    __shared__ int warp_tot[8];
    __shared__ int s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t chunk = (size_t)blockDim.x * SRC_PER;
    for (size_t cb = (size_t)blockIdx.x * chunk; cb < N; cb += (size_t)gridDim.x * chunk) {
        unsigned bits = 0;
        int cnt = 0;
#pragma unroll
        for (int k = 0; k < SRC_PER; ++k) {
            const size_t i = cb + (size_t)k * blockDim.x + threadIdx.x;
            if (i >= N) continue;
            const int n = __popc((unsigned)mask[i]);
            donors[i] = n;
            pending[i] = n;
            if (land[i] && n == 0) {
                bits |= 1u << k;
                ++cnt;
            }
        }
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        if (threadIdx.x == 0) {
            int run = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
                const int t = warp_tot[w];
                warp_tot[w] = run;
                run += t;
            }
            s_base = run ? atomicAdd(n_sources, run) : 0;
        }
        __syncthreads();
        int slot = s_base + warp_tot[warp] + incl - cnt;
#pragma unroll
        for (int k = 0; k < SRC_PER; ++k)
            if (bits & (1u << k)) sources[slot++] = (int)(cb + (size_t)k * blockDim.x + threadIdx.x);
        __syncthreads();
    }
}

struct WalkArgs {
    int W, H;
    const uint8_t* down;
    const uint8_t* mask;
    int32_t* pending;
    long long* key;
    const float* weights;
    float* area;
    const double* inflow;
    double* flow;
    const int* sources;
    const int* n_sources;
    unsigned long long* max_key;
};

// What a walk adds up beside the keys: nothing, areas (float weights), discharges (weights and the
// inflows from off the tree, in double), or, over a tree whose keys are known, flows that start as each
// cell's own.
enum { WALK_KEYS, WALK_AREA, WALK_DISCHARGE, WALK_FLOW };

template <int M>
struct WalkValue {
    using type = double;
};
template <>
struct WalkValue<WALK_AREA> {
    using type = float;
};
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

// One thread per source climbs down its receivers while it is the last donor into each. At a cell
// r it already holds the key and value of the cell it came from; r's donor mask and own value are
// loaded beside the atomic that decides whether it goes on, so a step costs the atomic and one
// round of loads of the other donors' keys and values. The counts end at 0, so a second walk over
// the same tree counts up to the donors again.
template <int M>
__global__ void __launch_bounds__(64) k_walk(WalkArgs a) {
    using V = typename WalkValue<M>::type;
    V* const val = M == WALK_AREA ? (V*)a.area : (V*)a.flow;
    auto own = [&](int c) -> V {
        if (M == WALK_AREA) return (V)a.weights[c];
        if (M == WALK_DISCHARGE) return (V)__dadd_rn((double)a.weights[c], a.inflow[c]);
        if (M == WALK_FLOW) return (V)a.flow[c];
        return (V)0;
    };
    unsigned long long local_max = 0;
    const int n_sources = *a.n_sources;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n_sources; idx += gridDim.x * blockDim.x) {
        int c = a.sources[idx];
        long long kc = (long long)c;   // a source: level 0, its own index
        V vc = own(c);
        if (M != WALK_FLOW) a.key[c] = kc;
        if (M == WALK_AREA || M == WALK_DISCHARGE) val[c] = vc;
        if ((unsigned long long)kc > local_max) local_max = (unsigned long long)kc;
        while (true) {
            const int d = a.down[c];
            if (d == 0xFF) break;
            const int r = step_to(a.W, c, d);
            const unsigned m = a.mask[r];
            const V vr = own(r);
            const long long kr = M == WALK_FLOW ? a.key[r] : 0;
            // Release: this cell's key and value are visible before its arrival is counted. Acquire:
            // the last donor in sees every other donor's.
            cuda::atomic_ref<int, cuda::thread_scope_device> pend(a.pending[r]);
            if (M == WALK_FLOW) {
                if (pend.fetch_add(1, cuda::memory_order_acq_rel) + 1 != __popc(m)) break;
            } else {
                if (pend.fetch_sub(1, cuda::memory_order_acq_rel) != 1) break;   // not the last donor in
            }
            // The donors' keys and values (the cell just left from registers). Keys are distinct, so
            // each donor's rank is the number of smaller keys; the values are added in rank order.
            long long kt[8];
            V vt[8];
            long long kmax = LLONG_MIN;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                kt[t] = LLONG_MAX;
                vt[t] = (V)0;
                if (!(m & (1u << t))) continue;
                const int dn = step_to(a.W, r, t);
                if (dn == c) {
                    kt[t] = kc;
                    vt[t] = vc;
                } else {
                    kt[t] = *((volatile long long*)&a.key[dn]);
                    if (M != WALK_KEYS) vt[t] = *((volatile V*)&val[dn]);
                }
                kmax = kt[t] > kmax ? kt[t] : kmax;
            }
            kc = M == WALK_FLOW ? kr : kmax + LEVEL_ONE;
            if (M != WALK_FLOW) a.key[r] = kc;
            if (M != WALK_KEYS) {
                int rank[8];
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    rank[t] = 0;
#pragma unroll
                    for (int u = 0; u < 8; ++u) rank[t] += (kt[u] < kt[t]) ? 1 : 0;
                }
                const int n = __popc(m);
                V sum = vr;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (j >= n) break;
                    V pick = (V)0;
#pragma unroll
                    for (int t = 0; t < 8; ++t) pick = rank[t] == j && (m & (1u << t)) ? vt[t] : pick;
                    sum = add_rn(sum, pick);
                }
                vc = sum;
                val[r] = sum;
            }
            if ((unsigned long long)kc > local_max) local_max = (unsigned long long)kc;
            c = r;
        }
    }
    if constexpr (M != WALK_FLOW) {
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xFFFFFFFFu, local_max, o);
            if (other > local_max) local_max = other;
        }
        if ((threadIdx.x & 31) == 0 && local_max) atomicMax(a.max_key, local_max);
    }
}

// Areas of land cells are the weights where no walk reached (sea cells hold 0).
__global__ void k_area_sea(const uint8_t* __restrict__ land, size_t N, float* __restrict__ area) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        if (!land[i]) area[i] = 0.0f;
}

__global__ void k_land_flags(const uint8_t* __restrict__ land, size_t N, int* __restrict__ flag) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        flag[i] = land[i] ? 1 : 0;
}

// The drainage order as a stable LSD radix sort of the land cells' compact keys, level N + deepest
// source (distinct, ordered as the drainage keys are), 8 bits a pass over the bits they use. A CTA
// takes a tile of cells: it counts its digits, the counts are scanned digit-major over the
// tiles, and the CTA scatters its tile in order, 256 cells at a time, each cell's place among the
// chunk's cells of its digit found with __match_any_sync within its warp and per-warp counts across
// warps, so cells of one digit keep their order. A tile is 4096 cells, or fewer (whole chunks) where that
// would leave SMs without two: the chunks of a tile follow one another, and at 60,000 cells 15 CTAs of 16
// chunks took 14 us a pass.
constexpr int kRsTile = 4096;
constexpr int kRsOneLaunch = 2048;   // cells an SM up to which the passes share one launch

__global__ void k_land_compact_ck(const uint8_t* __restrict__ land, const int* __restrict__ pos,
                                  const long long* __restrict__ key, size_t N, unsigned long long* __restrict__ ck,
                                  int* __restrict__ vals, unsigned long long* __restrict__ kmax) {   // kmax or null
    unsigned long long m = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        if (land[i]) {
            const unsigned long long k = (unsigned long long)key[i];
            const unsigned long long c = (k >> 32) * (unsigned long long)N + (k & 0xFFFFFFFFull);
            ck[pos[i]] = c;
            vals[pos[i]] = (int)i;
            m = c > m ? c : m;
        }
    if (!kmax) return;
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_down_sync(0xFFFFFFFFu, m, o);
        m = t > m ? t : m;
    }
    if ((threadIdx.x & 31) == 0 && m) atomicMax(kmax, m);
}

// The same from a list of the cells (in any order: the keys are distinct).
__global__ void k_list_ck(const int* __restrict__ cells, int n, const long long* __restrict__ key, size_t N,
                          unsigned long long* __restrict__ ck, int* __restrict__ vals) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int c = cells[i];
        const unsigned long long k = (unsigned long long)key[c];
        ck[i] = (k >> 32) * (unsigned long long)N + (k & 0xFFFFFFFFull);
        vals[i] = c;
    }
}

__global__ void __launch_bounds__(256) k_rs_hist(const unsigned long long* __restrict__ keys, int n, int shift,
                                                 int tile, int tiles, int* __restrict__ hist) {
    __shared__ int h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int lo = blockIdx.x * tile, hi = min(n, lo + tile);
    for (int i = lo + (int)threadIdx.x; i < hi; i += 256) atomicAdd(&h[(int)((keys[i] >> shift) & 255ull)], 1);
    __syncthreads();
    hist[threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

struct RsSmem {
    int base[256];
    int wcnt[8][256];
};

// A CTA's tile [lo, hi) scattered in order, its digits' first places in sh.base.
__device__ __forceinline__ void rs_scatter_tile(const unsigned long long* __restrict__ kin, const int* __restrict__ vin,
                                                int lo, int hi, int shift, RsSmem& sh,
                                                unsigned long long* __restrict__ kout, int* __restrict__ vout) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int w = 0; w < 8; ++w) sh.wcnt[w][tid] = 0;
    __syncthreads();
    for (int c = lo; c < hi; c += 256) {
        const int i = c + tid;
        const bool valid = i < hi;
        const unsigned long long k = valid ? __ldcg(kin + i) : 0ull;
        const int v = valid ? __ldcg(vin + i) : 0;
        const int d = valid ? (int)((k >> shift) & 255ull) : 256;
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank == 0) sh.wcnt[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            int before = 0;
            for (int w = 0; w < warp; ++w) before += sh.wcnt[w][d];
            const int p = sh.base[d] + before + rank;
            kout[p] = k;
            vout[p] = v;
        }
        __syncthreads();
        int sum = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            sum += sh.wcnt[w][tid];
            sh.wcnt[w][tid] = 0;
        }
        sh.base[tid] += sum;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) k_rs_scatter(const unsigned long long* __restrict__ kin,
                                                    const int* __restrict__ vin, int n, int shift, int tile,
                                                    int tiles, const int* __restrict__ off, unsigned long long* __restrict__ kout,
                                                    int* __restrict__ vout) {
    __shared__ RsSmem sh;
    sh.base[threadIdx.x] = off[threadIdx.x * tiles + blockIdx.x];
    const int lo = blockIdx.x * tile;
    rs_scatter_tile(kin, vin, lo, min(n, lo + tile), shift, sh, kout, vout);
}

// Every pass in one cooperative launch, a CTA a tile, where the tiles are no more than the SMs: the counts,
// a warp a digit scanning them over the tiles, and the scatter, a grid barrier after each. Four launches a
// pass took 16 us at 50,000 cells, mostly between them; a pass here takes 10.
struct RsArgs {
    unsigned long long* keys[2];
    int* vals[2];
    int n, tile, tiles, bits;
    int* hist;     // [tiles][256]
    int* before;   // [tiles][256]: the cells of the digit in the tiles before
    int* total;    // [256]
    int* out;
};
__global__ void __launch_bounds__(256) k_rs_sort(RsArgs a) {
    cgr::grid_group grid = cgr::this_grid();
    __shared__ RsSmem sh;
    __shared__ int warp_sum[8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lo = blockIdx.x * a.tile, hi = min(a.n, lo + a.tile);
    int pass = 0;
    for (int shift = 0; shift < a.bits; shift += 8, ++pass) {
        const unsigned long long* kin = a.keys[pass & 1];
        sh.base[tid] = 0;
        __syncthreads();
        for (int i = lo + tid; i < hi; i += 256) atomicAdd(&sh.base[(int)((__ldcg(kin + i) >> shift) & 255ull)], 1);
        __syncthreads();
        __stcg(a.hist + blockIdx.x * 256 + tid, sh.base[tid]);
        grid.sync();
        for (int d = blockIdx.x * 8 + warp; d < 256; d += gridDim.x * 8) {
            int run = 0;
            for (int t0 = 0; t0 < a.tiles; t0 += 32) {
                const int v = t0 + lane < a.tiles ? __ldcg(a.hist + (t0 + lane) * 256 + d) : 0;
                int x = v;
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                    if (lane >= o) x += y;
                }
                if (t0 + lane < a.tiles) __stcg(a.before + (t0 + lane) * 256 + d, run + x - v);
                run += __shfl_sync(0xFFFFFFFFu, x, 31);
            }
            if (lane == 0) __stcg(a.total + d, run);
        }
        grid.sync();
        const int all = __ldcg(a.total + tid);
        int x = all;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
        __syncthreads();
        for (int w = 0; w < warp; ++w) x += warp_sum[w];
        sh.base[tid] = x - all + __ldcg(a.before + blockIdx.x * 256 + tid);
        const bool last = shift + 8 >= a.bits;
        rs_scatter_tile(kin, a.vals[pass & 1], lo, hi, shift, sh, a.keys[(pass & 1) ^ 1], last ? a.out : a.vals[(pass & 1) ^ 1]);
        if (!last) grid.sync();
    }
}

__global__ void k_level_bounds(const int* __restrict__ order, const long long* __restrict__ key, int n, int levels,
                               int* __restrict__ level_start) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int L = (int)(key[order[k]] >> 32);
        const int prev = k > 0 ? (int)(key[order[k - 1]] >> 32) : -1;
        for (int l = prev + 1; l <= L; ++l) level_start[l] = k;
        if (k == n - 1)
            for (int l = L + 1; l <= levels; ++l) level_start[l] = n;
    }
}

// ---- incise

// Cells bucketed by their Kahn level (the high half of their drainage key). A cell's receiver sits
// on a strictly higher level, so sweeping the levels from the top down reaches every receiver
// before its donors. Warp-aggregated atomics: lanes sharing a level take one atomic between them.
// Cells per Kahn level, and the cells bucketed by level. A CTA counts its cells per level in shared
// memory and adds each nonzero count to the global one with a single atomic; the scatter does the
// same per chunk of LVL_PER cells per thread, a cell's slot being its rank within the chunk's level
// (a shared-memory atomic) after the chunk's base for that level. Level 0 holds millions of cells,
// so atomics per warp on its cursor were the kernels' cost. Worlds with more than LVL_SMEM levels
// take the per-warp kernels.
constexpr int kLevelThreads = 1024;   // k_incise_levels's CTAs, one an SM: a shorter grid barrier than many
constexpr int LVL_SMEM = 4096;
constexpr int LVL_PER = 8;

__device__ __forceinline__ int level_of(const uint8_t* land, const long long* key, size_t i, size_t N, int levels) {
    if (i >= N || !land[i]) return -1;
    const int L = (int)(key[i] >> 32);
    return (L < 0 || L >= levels) ? -1 : L;   // never out of range for a forest's keys
}

__global__ void __launch_bounds__(256) k_level_count_cta(const uint8_t* __restrict__ land,
                                                         const long long* __restrict__ key, size_t N, int levels,
                                                         int* __restrict__ count) {
    __shared__ int hist[LVL_SMEM];
    for (int l = threadIdx.x; l < levels; l += blockDim.x) hist[l] = 0;
    __syncthreads();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        const int L = level_of(land, key, i, N, levels);
        if (L >= 0) atomicAdd(&hist[L], 1);
    }
    __syncthreads();
    for (int l = threadIdx.x; l < levels; l += blockDim.x)
        if (hist[l]) atomicAdd(&count[l], hist[l]);
}

__global__ void __launch_bounds__(256) k_level_scatter_cta(const uint8_t* __restrict__ land,
                                                           const long long* __restrict__ key, size_t N, int levels,
                                                           const int* __restrict__ start, int* __restrict__ cursor,
                                                           int* __restrict__ bucket) {
    __shared__ int hist[LVL_SMEM];
    const size_t chunk = (size_t)blockDim.x * LVL_PER;
    for (size_t cb = (size_t)blockIdx.x * chunk; cb < N; cb += (size_t)gridDim.x * chunk) {
        for (int l = threadIdx.x; l < levels; l += blockDim.x) hist[l] = 0;
        __syncthreads();
        int lv[LVL_PER], rank[LVL_PER];
#pragma unroll
        for (int k = 0; k < LVL_PER; ++k) {
            lv[k] = level_of(land, key, cb + (size_t)k * blockDim.x + threadIdx.x, N, levels);
            rank[k] = lv[k] >= 0 ? atomicAdd(&hist[lv[k]], 1) : 0;
        }
        __syncthreads();
        for (int l = threadIdx.x; l < levels; l += blockDim.x)
            if (hist[l]) hist[l] = start[l] + atomicAdd(&cursor[l], hist[l]);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < LVL_PER; ++k)
            if (lv[k] >= 0) bucket[hist[lv[k]] + rank[k]] = (int)(cb + (size_t)k * blockDim.x + threadIdx.x);
        __syncthreads();
    }
}

__global__ void k_level_count(const uint8_t* __restrict__ land, const long long* __restrict__ key, size_t N,
                              int levels, int* __restrict__ count) {
    const unsigned FULL = 0xFFFFFFFFu;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < N; base += stride) {
        const int L = level_of(land, key, base + threadIdx.x, N, levels);
        unsigned group = __match_any_sync(FULL, L);
        if (L >= 0 && (threadIdx.x & 31) == __ffs(group) - 1) atomicAdd(&count[L], __popc(group));
    }
}
__global__ void k_level_scatter(const uint8_t* __restrict__ land, const long long* __restrict__ key, size_t N,
                                int levels, const int* __restrict__ start, int* __restrict__ cursor,
                                int* __restrict__ bucket) {
    const unsigned FULL = 0xFFFFFFFFu;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < N; base += stride) {
        const size_t i = base + threadIdx.x;
        const int L = level_of(land, key, i, N, levels);
        unsigned group = __match_any_sync(FULL, L);
        int leader = __ffs(group) - 1;
        int slot = 0;
        if (L >= 0 && lane == leader) slot = atomicAdd(&cursor[L], __popc(group));
        slot = __shfl_sync(FULL, slot, leader);
        if (L >= 0) bucket[start[L] + slot + __popc(group & ((1u << lane) - 1u))] = (int)i;
    }
}

struct InciseDev {
    InciseArgs a;
    int W;
    const uint8_t* land;
    const int32_t* recv;
    const float* ground;
    const float* rel;
    const float* area;
    const float* erod;
    float* surface;
    float* water;
    double* incised_at; // or NULL
    const int* start;   // depth buckets, [levels + 1]
    const int* bucket;
    int4* fixed;        // per slot of the buckets: what no other cell changes (IncisedCell)
    float* courant;
    int levels;
    int* split;         // the highest level left to the whole grid
};

// A cell of HydraulicErosion.incise (HydraulicErosion.kt:2322-2359) is settled in two parts. What the
// rest of the sweep cannot change (its receiver, its fill, its Courant number, its own height, which only
// its own step lowers) is gathered for every cell at once before the levels run; the levels then read it in
// slot order and wait for nothing but the receiver's height and water.
constexpr int kUnder = 1 << 30, kLandBelow = (int)(1u << 31);

__device__ void gather_incise(const InciseDev& d, int slot) {
    const int cell = d.bucket[slot], r = d.recv[cell];
    const float ground = d.ground[cell];
    int flags = __fsub_rn(ground, d.rel[cell]) > d.a.pond_depth ? kUnder : 0;
    if (r >= 0 && d.land[r]) flags |= kLandBelow;
    // GroundSteps.between (MA/GroundSteps.kt:45-53).
    const bool same_row = pdiv(cell, d.W) == pdiv(r, d.W), same_col = pmod(cell, d.W) == pmod(r, d.W);
    const float step = (!same_row && !same_col) ? d.a.step_diag : (!same_row ? d.a.step_ns : 1.0f);
    d.courant[slot] = __fdiv_rn(__fmul_rn(__fmul_rn(d.a.courant_coefficient,
                                                    __fsqrt_rn(__fdiv_rn(d.area[cell], d.a.land_cells))),
                                          d.erod[cell]),
                                step);
    const float filled_level = __fadd_rn(d.a.shoreline, __fmul_rn(ground, d.a.land_range));
    d.fixed[slot] = make_int4(cell | flags, r, __float_as_int(filled_level), __float_as_int(d.surface[cell]));
}

__device__ __forceinline__ void incise_cell(const InciseDev& d, int4 fixed, float courant) {
    const int cell = fixed.x & (kUnder - 1), r = fixed.y;
    const bool under = (fixed.x & kUnder) != 0, land_below = fixed.x < 0;
    const float filled_level = __int_as_float(fixed.z), height = __int_as_float(fixed.w);
    if (r < 0) {
        if (under) __stcg(d.water + cell, filled_level);
        return;
    }
    // HydraulicErosion.baseLevel (HydraulicErosion.kt:2380-2390).
    float base_after = d.a.shoreline, wr = NAN;
    if (land_below) {
        base_after = __ldcg(d.surface + r);
        wr = __ldcg(d.water + r);
        if (!isnan(wr)) base_after = fmaxf(base_after, wr);
    }
    float water = NAN;
    if (under) {
        water = fminf(filled_level, !isnan(wr) ? wr : base_after);
        __stcg(d.water + cell, water);
    }
    const float grades_to = base_after;   // no unresolved relief in this profile
    const bool submerged = under && height <= water;
    float after;
    if (submerged || (height <= grades_to && d.a.only_above_base)) {
        after = height;
    } else {
        double g = (double)grades_to;
        after = (float)__dadd_rn(g, __ddiv_rn((double)__fsub_rn(height, grades_to), __dadd_rn(1.0, (double)courant)));
    }
    if (after != height) {
        __stcg(d.surface + cell, after);
        if (d.incised_at && after < height) d.incised_at[cell] = __dsub_rn((double)height, (double)after);
    }
}

// Levels from the top down. The highest levels are the main stems of the largest rivers, a few
// cells each: while a level fits two passes of a CTA, the first CTA takes it alone, with a CTA barrier
// between levels (its own writes are visible to it); the rest of the grid waits at one grid barrier
// and then sweeps the lower, larger levels with a grid barrier per level. A thread's first cell of the next
// level is loaded before the barrier, so a level costs a barrier, the receiver's loads and one division. With
// the whole cell read in its level a sweep took 240 us at 2048 x 1024 and 1.85 ms at 8192 x 4096; now 158 us
// and 1.37 ms.
__global__ void __launch_bounds__(kLevelThreads) k_incise_levels(InciseDev d) {
    cgr::grid_group grid = cgr::this_grid();
    const int t = blockIdx.x * kLevelThreads + threadIdx.x, stride = gridDim.x * kLevelThreads;
    for (int slot = t; slot < d.start[d.levels]; slot += stride) gather_incise(d, slot);
    grid.sync();
    const int4 none = make_int4(0, -1, 0, 0);
    if (blockIdx.x == 0) {
        int level = d.levels - 1;
        int lo = d.start[level], hi = d.start[level + 1];
        int4 fixed = none;
        float courant = 0.0f;
        auto load = [&](int slot, int end) {
            if (slot < end) {
                fixed = __ldcg(d.fixed + slot);
                courant = __ldcg(d.courant + slot);
            }
        };
        load(lo + (int)threadIdx.x, hi);
        for (; level >= 0 && hi - lo <= 2 * kLevelThreads; --level) {
            int slot = lo + (int)threadIdx.x;
            if (slot < hi) incise_cell(d, fixed, courant);
            slot += kLevelThreads;
            if (slot < hi) incise_cell(d, __ldcg(d.fixed + slot), __ldcg(d.courant + slot));
            hi = lo;
            lo = level > 0 ? d.start[level - 1] : 0;
            load(lo + (int)threadIdx.x, hi);
            __syncthreads();
        }
        if (threadIdx.x == 0) *d.split = level;
    }
    grid.sync();
    const int top = *(volatile int*)d.split;
    if (top < 0) return;
    int lo = d.start[top], hi = d.start[top + 1];
    int4 fixed = none;
    float courant = 0.0f;
    if (lo + t < hi) {
        fixed = __ldcg(d.fixed + lo + t);
        courant = __ldcg(d.courant + lo + t);
    }
    for (int level = top;; --level) {
        if (lo + t < hi) incise_cell(d, fixed, courant);
        for (int slot = lo + t + stride; slot < hi; slot += stride)
            incise_cell(d, __ldcg(d.fixed + slot), __ldcg(d.courant + slot));
        if (level == 0) break;
        hi = lo;
        lo = d.start[level - 1];
        if (lo + t < hi) {
            fixed = __ldcg(d.fixed + lo + t);
            courant = __ldcg(d.courant + lo + t);
        }
        grid.sync();
    }
}

__global__ void k_water_init(float* __restrict__ water, size_t N) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        water[i] = NAN;
}

// ---- spillways

__device__ __forceinline__ unsigned ordered_key(float f) {
    if (f == 0.0f) f = 0.0f;   // -0 and +0 compare equal in the reference
    unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ordered_key(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

__global__ void k_ponded(const uint8_t* __restrict__ land, const float* __restrict__ filled,
                         const float* __restrict__ rel, float pond, size_t N, uint8_t* __restrict__ ponded) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        ponded[i] = land[i] && __fsub_rn(filled[i], rel[i]) > pond;
}

struct BasinDev {
    int* cells;
    unsigned* floor_key;
    unsigned long long* spill_key;
};

__global__ void k_basin_init(BasinDev b, int count) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    b.cells[i] = 0;
    b.floor_key[i] = 0xFFFFFFFFu;
    b.spill_key[i] = 0xFFFFFFFFFFFFFFFFull;
}

__global__ void k_basin_gather(const int* __restrict__ label, const uint8_t* __restrict__ ponded,
                               const uint8_t* __restrict__ land, const float* __restrict__ rel,
                               const float* __restrict__ filled, const int32_t* __restrict__ recv, size_t N,
                               BasinDev b) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        int l = label[i];
        if (l < 0) continue;
        atomicAdd(&b.cells[l], 1);
        atomicMin(&b.floor_key[l], ordered_key(rel[i]));
        int r = recv[i];
        if (r >= 0 && land[r] && !ponded[r]) {
            unsigned long long k = ((unsigned long long)ordered_key(filled[r]) << 32) | (unsigned)r;
            atomicMin(&b.spill_key[l], k);
        }
    }
}

// Per basin: the pour point down the outflow's path, the level and the fill depth
// (FlowRouting.kt:637-671).
__global__ void k_basin_finish(BasinDev b, int count, const uint8_t* __restrict__ land,
                               const float* __restrict__ rel, const float* __restrict__ filled,
                               const int32_t* __restrict__ recv, long long N, int* __restrict__ entry,
                               int* __restrict__ spill, float* __restrict__ level, float* __restrict__ floor_out,
                               float* __restrict__ depth) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float basin_floor = from_ordered_key(b.floor_key[i]);
    unsigned long long sk = b.spill_key[i];
    int sp = -1;
    float spill_level = FLT_MAX;
    if (sk != 0xFFFFFFFFFFFFFFFFull) {
        sp = (int)(sk & 0xFFFFFFFFull);
        spill_level = filled[sp];
    }
    int pour = sp;
    if (sp >= 0) {
        int cell = sp;
        long long steps = 0;
        while (cell >= 0 && land[cell] && filled[cell] > rel[cell] && steps < N) {
            cell = recv[cell];
            ++steps;
        }
        if (cell >= 0 && land[cell]) pour = cell;
    }
    float pour_level = pour >= 0 ? filled[pour] : spill_level;
    entry[i] = sp;
    spill[i] = pour;
    level[i] = pour >= 0 ? pour_level : basin_floor;
    floor_out[i] = basin_floor;
    depth[i] = pour >= 0 ? __fsub_rn(pour_level, basin_floor) : 0.0f;
}

}  // namespace

// The links, down then mask, and behind them the largest key and the number of sources. The mask is written a
// word at a time, so it starts at one on grids of two cells too.
struct Links {
    uint8_t *down, *mask;
    unsigned long long* max_key;
    int* sources;
};
static size_t link_stride(size_t N) { return (N + 15) & ~(size_t)15; }
static size_t link_bytes(size_t N) { return 2 * link_stride(N) + 32; }
static Links links_at(uint8_t* d_links, size_t N) {
    Links l;
    l.down = d_links;
    l.mask = d_links + link_stride(N);
    l.max_key = reinterpret_cast<unsigned long long*>(l.mask + link_stride(N));
    l.sources = reinterpret_cast<int*>(l.max_key + 1);
    return l;
}

cg_status tree_walk_dev(cg_ctx* ctx, int W, int H, const uint8_t* d_land, const int32_t* d_recv,
                        const float* d_weights, long long* d_key, int32_t* d_donors, float* d_area, int* h_levels,
                        const double* d_inflow, double* d_flow, ReadBack also) {
    size_t N = (size_t)W * H;
    cudaStream_t sm = ctx->stream;
    int grid = ctx->num_sms * 8;
    CG_BUF(int32_t, d_pending, ctx, S_DEPTH, N);
    CG_BUF(uint8_t, d_links, ctx, S_LINKS, link_bytes(N));
    CG_BUF(int, d_sources, ctx, S_SOURCES, N);
    const Links links = links_at(d_links, N);
    uint8_t *d_down = links.down, *d_mask = links.mask;
    unsigned long long* d_max = links.max_key;
    int* d_nsrc = links.sources;   // zeroed with the mask and the largest key
    CG_CUDA(ctx, cudaMemsetAsync(d_mask, 0, (uint8_t*)(d_nsrc + 1) - d_mask, sm));
    CG_LAUNCH(ctx) k_links<<<grid, 256, 0, sm>>>(d_land, d_recv, W, H, d_down, d_mask);
    CG_LAUNCH(ctx) k_sources<<<grid, 256, 0, sm>>>(d_land, d_mask, N, d_donors, d_pending, d_sources, d_nsrc);
    if (d_area) CG_LAUNCH(ctx) k_area_sea<<<grid, 256, 0, sm>>>(d_land, N, d_area);
    CG_CHECK_LAUNCH(ctx);
    // A thread a source. Up to 2^21 cells the launch is sized for as many sources as cells, up to half a
    // million (its idle CTAs cost less than the 10 us of a host read); larger worlds read their number.
    int n_sources = (int)std::min(N, (size_t)1 << 19);
    if (N > (size_t)1 << 21) {
        CG_TRY_ST(read_back(ctx, {{&n_sources, d_nsrc, sizeof(int)}}));
    }
    WalkArgs a{W, H, d_down, d_mask, d_pending, d_key, d_weights, d_area, d_inflow, d_flow, d_sources, d_nsrc, d_max};
    const int ctas = (n_sources + 63) / 64;
    if (ctas > 0) {
        if (d_flow) CG_LAUNCH(ctx) k_walk<WALK_DISCHARGE><<<ctas, 64, 0, sm>>>(a);
        else if (d_weights) CG_LAUNCH(ctx) k_walk<WALK_AREA><<<ctas, 64, 0, sm>>>(a);
        else CG_LAUNCH(ctx) k_walk<WALK_KEYS><<<ctas, 64, 0, sm>>>(a);
    }
    CG_CHECK_LAUNCH(ctx);
    if (h_levels) {
        unsigned long long mk;
        CG_TRY_ST(read_back(ctx, {{&mk, d_max, sizeof(mk)}, also}));
        *h_levels = (int)(mk >> 32) + 1;
    }
    return CG_OK;
}

cg_status flow_walk_dev(cg_ctx* ctx, int W, int H, long long* d_key, double* d_flow) {
    const size_t N = (size_t)W * H;
    CG_BUF(int32_t, d_pending, ctx, S_DEPTH, N);
    CG_BUF(uint8_t, d_links, ctx, S_LINKS, link_bytes(N));
    CG_BUF(int, d_sources, ctx, S_SOURCES, N);
    const Links links = links_at(d_links, N);
    WalkArgs a{W, H, links.down, links.mask, d_pending, d_key, nullptr, nullptr, nullptr, d_flow, d_sources, links.sources,
               nullptr};
    const int ctas = ((int)std::min(N, (size_t)1 << 19) + 63) / 64;
    CG_LAUNCH(ctx) k_walk<WALK_FLOW><<<ctas, 64, 0, ctx->stream>>>(a);
    CG_CHECK_LAUNCH(ctx);
    return CG_OK;
}

cg_status order_from_keys_dev(cg_ctx* ctx, int W, int H, const uint8_t* d_land, const long long* d_key,
                              int land_cells, int32_t* d_order, int levels, const int* d_cells) {
    size_t N = (size_t)W * H;
    cudaStream_t sm = ctx->stream;
    int grid = ctx->num_sms * 8;
    if (land_cells <= 0) return CG_OK;
    const int n = land_cells;
    const int tile = std::min(kRsTile, std::max(1, n / (2 * ctx->num_sms * 256)) * 256);
    const int tiles = (n + tile - 1) / tile;
    CG_BUF(unsigned long long, d_keys, ctx, S_RS_KEYS, 2 * (size_t)n + 1);
    CG_BUF(int, d_vals, ctx, S_RS_VALS, 2 * (size_t)n);
    CG_BUF(int, d_hist, ctx, S_RS_HIST, 2 * (size_t)tiles * 256 + 256);
    unsigned long long* kmax = d_keys + 2 * (size_t)n;
    unsigned long long* ka = d_keys;
    unsigned long long* kb = d_keys + n;
    int* va = d_vals;
    int* vb = d_vals + n;
    int* d_off = d_hist + (size_t)tiles * 256;
    // The largest compact key: from the levels where the caller knows them (its bits, at any rate).
    unsigned long long hmax = levels > 0 ? (unsigned long long)levels * N - 1 : 0;
    if (d_cells && levels > 0) {
        CG_LAUNCH(ctx) k_list_ck<<<std::min(grid, (n + 255) / 256), 256, 0, sm>>>(d_cells, n, d_key, N, ka, va);
        CG_CHECK_LAUNCH(ctx);
    } else {
        CG_BUF(int, d_flag, ctx, S_SCRATCH0, N);
        CG_BUF(int, d_pos, ctx, S_SCRATCH1, N);
        CG_LAUNCH(ctx) k_land_flags<<<grid, 256, 0, sm>>>(d_land, N, d_flag);
        CG_CHECK_LAUNCH(ctx);
        cg_status st = exclusive_scan(ctx, d_flag, d_pos, (int)N, nullptr);
        if (st != CG_OK) return st;
        if (levels <= 0) CG_CUDA(ctx, cudaMemsetAsync(kmax, 0, sizeof(unsigned long long), sm));
        CG_LAUNCH(ctx) k_land_compact_ck<<<grid, 256, 0, sm>>>(d_land, d_pos, d_key, N, ka, va, levels > 0 ? nullptr : kmax);
        CG_CHECK_LAUNCH(ctx);
        if (levels <= 0) CG_TRY_ST(read_back(ctx, {{&hmax, kmax, sizeof(hmax)}}));
    }
    int bits = 0;
    while (bits < 64 && (hmax >> bits) != 0) ++bits;
    if (bits > 0 && n <= ctx->num_sms * kRsOneLaunch) {
        RsArgs a;
        a.keys[0] = ka;
        a.keys[1] = kb;
        a.vals[0] = va;
        a.vals[1] = vb;
        a.n = n;
        a.tile = std::max(1, (n + ctx->num_sms * 256 - 1) / (ctx->num_sms * 256)) * 256;
        a.tiles = (n + a.tile - 1) / a.tile;   // no more than the SMs, and than `tiles`
        a.bits = bits;
        a.hist = d_hist;
        a.before = d_off;
        a.total = d_off + (size_t)tiles * 256;
        a.out = d_order;
        int per_sm = 0;
        CG_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_rs_sort, 256, 0));
        if (per_sm < 1) return fail(ctx, CG_CUDA, "the order's sort cannot be resident");
        void* kargs[] = {&a};
        ctx->launches++;
        CG_CUDA(ctx, cudaLaunchCooperativeKernel((void*)k_rs_sort, a.tiles, 256, kargs, 0, sm));
        return CG_OK;
    }
    for (int shift = 0; shift < bits; shift += 8) {
        CG_LAUNCH(ctx) k_rs_hist<<<tiles, 256, 0, sm>>>(ka, n, shift, tile, tiles, d_hist);
        CG_CHECK_LAUNCH(ctx);
        cg_status st = exclusive_scan(ctx, d_hist, d_off, tiles * 256, nullptr);
        if (st != CG_OK) return st;
        CG_LAUNCH(ctx) k_rs_scatter<<<tiles, 256, 0, sm>>>(ka, va, n, shift, tile, tiles, d_off, kb, vb);
        CG_CHECK_LAUNCH(ctx);
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    CG_CUDA(ctx, cudaMemcpyAsync(d_order, va, sizeof(int) * (size_t)n, cudaMemcpyDeviceToDevice, sm));
    return CG_OK;
}

cg_status level_bounds_dev(cg_ctx* ctx, const int* d_order, const long long* d_key, int n, int levels, int* d_start) {
    CG_LAUNCH(ctx) k_level_bounds<<<std::min(ctx->num_sms * 8, (n + 255) / 256), 256, 0, ctx->stream>>>(d_order, d_key, n,
                                                                                                      levels, d_start);
    CG_CHECK_LAUNCH(ctx);
    return CG_OK;
}

cg_status level_buckets_dev(cg_ctx* ctx, int W, int H, const uint8_t* d_land, const long long* d_key, int levels,
                            int** out_bucket, int** out_start) {
    size_t N = (size_t)W * H;
    cudaStream_t sm = ctx->stream;
    int grid = ctx->num_sms * 8;
    CG_BUF(int, d_bucket, ctx, S_SCRATCH2, N);
    CG_BUF(int, d_cnt, ctx, S_DEPTH, (size_t)levels + 1);
    CG_BUF(int, d_start, ctx, S_CG2, 2 * (size_t)levels + 2);
    int* d_cursor = d_start + levels + 1;
    CG_CUDA(ctx, cudaMemsetAsync(d_cnt, 0, ((size_t)levels + 1) * sizeof(int), sm));
    CG_CUDA(ctx, cudaMemsetAsync(d_cursor, 0, ((size_t)levels + 1) * sizeof(int), sm));
    const bool cta_hist = levels <= LVL_SMEM;
    if (cta_hist) CG_LAUNCH(ctx) k_level_count_cta<<<grid, 256, 0, sm>>>(d_land, d_key, N, levels, d_cnt);
    else CG_LAUNCH(ctx) k_level_count<<<grid, 256, 0, sm>>>(d_land, d_key, N, levels, d_cnt);
    CG_CHECK_LAUNCH(ctx);
    cg_status st = exclusive_scan(ctx, d_cnt, d_start, levels + 1, nullptr);
    if (st != CG_OK) return st;
    if (cta_hist) CG_LAUNCH(ctx) k_level_scatter_cta<<<grid, 256, 0, sm>>>(d_land, d_key, N, levels, d_start, d_cursor, d_bucket);
    else CG_LAUNCH(ctx) k_level_scatter<<<grid, 256, 0, sm>>>(d_land, d_key, N, levels, d_start, d_cursor, d_bucket);
    CG_CHECK_LAUNCH(ctx);
    *out_bucket = d_bucket;
    *out_start = d_start;
    return CG_OK;
}

cg_status incise_dev(cg_ctx* ctx, int W, int H, const uint8_t* d_land, const int32_t* d_recv, const long long* d_key,
                     int levels, int land_cells, const float* d_ground, const float* d_rel, const float* d_area, const float* d_erod,
                     float* d_surface, const InciseArgs& args, double* d_incised_at) {
    size_t N = (size_t)W * H;
    cudaStream_t sm = ctx->stream;
    int grid = ctx->num_sms * 8;
    if (levels <= 0) return CG_OK;
    CG_BUF(int, d_bucket, ctx, S_SCRATCH2, N);
    CG_BUF(float, d_water, ctx, S_WATER, N);
    CG_BUF(int, d_cnt, ctx, S_DEPTH, (size_t)levels + 1);
    CG_BUF(int, d_start, ctx, S_CG2, 2 * (size_t)levels + 2);
    int* d_cursor = d_start + levels + 1;
    CG_CUDA(ctx, cudaMemsetAsync(d_cnt, 0, ((size_t)levels + 1) * sizeof(int), sm));
    CG_CUDA(ctx, cudaMemsetAsync(d_cursor, 0, ((size_t)levels + 1) * sizeof(int), sm));
    const bool cta_hist = levels <= LVL_SMEM;
    if (cta_hist) CG_LAUNCH(ctx) k_level_count_cta<<<grid, 256, 0, sm>>>(d_land, d_key, N, levels, d_cnt);
    else CG_LAUNCH(ctx) k_level_count<<<grid, 256, 0, sm>>>(d_land, d_key, N, levels, d_cnt);
    CG_CHECK_LAUNCH(ctx);
    // The exclusive scan of levels + 1 counts (the last is zero) ends with the total at start[levels].
    cg_status st = exclusive_scan(ctx, d_cnt, d_start, levels + 1, nullptr);
    if (st != CG_OK) return st;
    if (cta_hist) CG_LAUNCH(ctx) k_level_scatter_cta<<<grid, 256, 0, sm>>>(d_land, d_key, N, levels, d_start, d_cursor, d_bucket);
    else CG_LAUNCH(ctx) k_level_scatter<<<grid, 256, 0, sm>>>(d_land, d_key, N, levels, d_start, d_cursor, d_bucket);
    CG_LAUNCH(ctx) k_water_init<<<grid, 256, 0, sm>>>(d_water, N);
    CG_CHECK_LAUNCH(ctx);
    InciseDev d;
    d.a = args;
    d.W = W;
    d.land = d_land;
    d.recv = d_recv;
    d.ground = d_ground;
    d.rel = d_rel;
    d.area = d_area;
    d.erod = d_erod;
    d.surface = d_surface;
    d.water = d_water;
    d.incised_at = d_incised_at;
    d.start = d_start;
    d.bucket = d_bucket;
    CG_BUF(int4, d_fixed, ctx, S_INCFIXED, land_cells);
    CG_BUF(float, d_courant, ctx, S_INCCOURANT, land_cells);
    d.fixed = d_fixed;
    d.courant = d_courant;
    d.levels = levels;
    d.split = d_cursor;   // the scatter's cursors are free by now
    int per_sm = 0;
    CG_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_incise_levels, kLevelThreads, 0));
    if (per_sm < 1) return fail(ctx, CG_CUDA, "incise kernel cannot be resident");
    int cgrid = ctx->num_sms;
    void* kargs[] = {&d};
    ctx->launches++;
    CG_CUDA(ctx, cudaLaunchCooperativeKernel((void*)k_incise_levels, cgrid, kLevelThreads, kargs, 0, sm));
    return CG_OK;
}

cg_status basins_dev(cg_ctx* ctx, int W, int H, const uint8_t* d_land, const float* d_rel, const float* d_filled,
                     const int32_t* d_recv, float pond_depth, int32_t* d_label, BasinArrays* out, int* h_count) {
    size_t N = (size_t)W * H;
    cudaStream_t sm = ctx->stream;
    int grid = ctx->num_sms * 8;
    CG_BUF(uint8_t, d_ponded, ctx, S_FLATS, N);
    CG_BUF(int, d_root, ctx, S_LABEL, N);
    CG_LAUNCH(ctx) k_ponded<<<grid, 256, 0, sm>>>(d_land, d_filled, d_rel, pond_depth, N, d_ponded);
    CG_CHECK_LAUNCH(ctx);
    int count = 0;
    cg_status st = component_labels(ctx, W, H, d_ponded, d_root, d_label, &count);
    if (st != CG_OK) return st;
    *h_count = count;
    *out = BasinArrays{};
    if (count == 0) return CG_OK;
    // One block: spill keys (8 bytes each) first for alignment, then seven 4-byte arrays.
    CG_BUF(unsigned long long, d_b, ctx, S_BASIN, (size_t)count * 5 + 8);
    BasinDev b;
    b.spill_key = d_b;
    b.cells = (int*)(d_b + count);
    b.floor_key = (unsigned*)(b.cells + count);
    out->cells = b.cells;
    out->entry = (int*)(b.floor_key + count);
    out->spill = out->entry + count;
    out->level = (float*)(out->spill + count);
    out->floor_ = out->level + count;
    out->depth = out->floor_ + count;
    CG_LAUNCH(ctx) k_basin_init<<<(count + 255) / 256, 256, 0, sm>>>(b, count);
    CG_LAUNCH(ctx) k_basin_gather<<<grid, 256, 0, sm>>>(d_label, d_ponded, d_land, d_rel, d_filled, d_recv, N, b);
    CG_LAUNCH(ctx) k_basin_finish<<<(count + 255) / 256, 256, 0, sm>>>(b, count, d_land, d_rel, d_filled, d_recv, (long long)N,
                                                        out->entry, out->spill, out->level, out->floor_, out->depth);
    CG_CHECK_LAUNCH(ctx);
    return CG_OK;
}

cg_status spillways_dev(cg_ctx* ctx, int W, int H, const uint8_t* d_land, const float* d_rel, const float* d_filled,
                        const int32_t* d_recv, float pond_depth, int32_t* d_label, cg_basins* hb) {
    cudaStream_t sm = ctx->stream;
    int count = 0;
    BasinArrays d;
    cg_status st = basins_dev(ctx, W, H, d_land, d_rel, d_filled, d_recv, pond_depth, d_label, &d, &count);
    if (st != CG_OK) return st;
    if (hb) {
        hb->count = count;
        hb->largest = -1;
        hb->largest_cells = 0;
        hb->largest_depth = 0.0f;
        hb->deepest = 0.0f;
    }
    if (count == 0 || !hb) return sync(ctx);
    std::vector<int> cells(count), entry(count), spill(count);
    std::vector<float> level(count), flo(count), depth(count);
    CG_CUDA(ctx, cudaMemcpyAsync(cells.data(), d.cells, count * sizeof(int), cudaMemcpyDeviceToHost, sm));
    CG_CUDA(ctx, cudaMemcpyAsync(entry.data(), d.entry, count * sizeof(int), cudaMemcpyDeviceToHost, sm));
    CG_CUDA(ctx, cudaMemcpyAsync(spill.data(), d.spill, count * sizeof(int), cudaMemcpyDeviceToHost, sm));
    CG_CUDA(ctx, cudaMemcpyAsync(level.data(), d.level, count * sizeof(float), cudaMemcpyDeviceToHost, sm));
    CG_CUDA(ctx, cudaMemcpyAsync(flo.data(), d.floor_, count * sizeof(float), cudaMemcpyDeviceToHost, sm));
    CG_CUDA(ctx, cudaMemcpyAsync(depth.data(), d.depth, count * sizeof(float), cudaMemcpyDeviceToHost, sm));
    CG_CUDA(ctx, cudaStreamSynchronize(sm));
    // The running largest / deepest of FlowRouting.kt:664-670, in basin order.
    int largest = -1, largest_cells = 0;
    float largest_depth = 0.0f, deepest = 0.0f;
    for (int i = 0; i < count; ++i) {
        if (cells[i] > largest_cells) {
            largest = i;
            largest_cells = cells[i];
            largest_depth = depth[i];
        }
        if (depth[i] > deepest) deepest = depth[i];
    }
    hb->largest = largest;
    hb->largest_cells = largest_cells;
    hb->largest_depth = largest_depth;
    hb->deepest = deepest;
    int n = count < hb->capacity ? count : hb->capacity;
    for (int i = 0; i < n; ++i) {
        if (hb->spill) hb->spill[i] = spill[i];
        if (hb->entry) hb->entry[i] = entry[i];
        if (hb->level) hb->level[i] = level[i];
        if (hb->floor) hb->floor[i] = flo[i];
        if (hb->cells) hb->cells[i] = cells[i];
    }
    return CG_OK;
}

}  // namespace cg
