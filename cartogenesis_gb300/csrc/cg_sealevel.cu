// SeaLevelStage.apply's cut up to the drowned basins' outlets (SeaLevelStage.kt:243-270) on the
// device: the percentile cut, the enclosure rule (markUnreachableWaterAsLand, SeaLevelStage.kt:
// 371-437) and the post-cut outlet passes (drainDrownedBasins, SeaLevelStage.kt:478-560). This is
// the reference reusing the erosion stage's routing outside it (FlowRouting.kt:14-17): each pass is
// a fill, a routing, an accumulation and the spillways over the whole grid, then the outlet notch run
// again with belowSea on, over the basins whose floor lies below the shoreline.
//
// The enclosure rule labels the water's 8-connected bodies (the same union-find labels as the
// basins, numbered by their lowest cell, which is the order the reference's scan finds them in);
// the ocean is the largest body, the first found of that size. The belowSea notch takes the drowned
// basins in the order spillways found them, and the lake-bed walk that belowSea adds follows the ponded
// cells as the cutting leaves them, so its footprint is not known before the cut. What bounds it is the
// chain of dependent loads a walk is, so one CTA walks 32 basins at a time, a warp each, without
// cutting: each lists the cells it reads and its cuts and stamps the cells it would cut, then looks
// whether a basin before it stamped a cell it read. The basins before the first that finds one cut as
// they would have one after another, and the next 32 start there: 11 to 17 basins a wave at 1024 x 512.
// (One thread taking the basins in turn: 3.8 ms a pass there; one warp with the others loading ahead of
// it 1.9; each walking twice instead of listing what it reads 0.85.)
#include <algorithm>
#include <cmath>

#include "cg_common.cuh"
#include "cg_internal.h"
#include "cg_params.h"
#include "cg_util.h"

namespace cg {
namespace {

__global__ void k_water_mask(const uint8_t* __restrict__ land, size_t N, uint8_t* __restrict__ mask) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        mask[i] = land[i] ? 0 : 1;
}

// Cells per water body. Nearly every cell is the ocean's, one counter, so a warp takes a stretch of
// kBodyRun x 32 cells and keeps the count of the body it is in, adding it once when the body changes
// (an atomic a cell cost 230 us at 1024 x 512); cells of a mixed row of 32 go by groups of one body.
constexpr int kBodyRun = 16;

__global__ void k_body_sizes(const int* __restrict__ label, size_t N, int* __restrict__ size) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const size_t warps = (size_t)gridDim.x * blockDim.x / 32;
    for (size_t run = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) / 32; run * (kBodyRun * 32) < N; run += warps) {
        int body = -1, cells = 0;   // the same in every lane
        for (int k = 0; k < kBodyRun; ++k) {
            const size_t i = (run * kBodyRun + k) * 32 + lane;
            const int l = i < N ? label[i] : -1;
            const int l0 = __shfl_sync(FULL, l, 0);
            if (__all_sync(FULL, l == l0)) {
                if (l0 != body) {
                    if (lane == 0 && body >= 0) atomicAdd(&size[body], cells);
                    body = l0;
                    cells = 0;
                }
                cells += 32;
            } else {
                const unsigned peers = __match_any_sync(FULL, l);
                if (l >= 0 && lane == __ffs(peers) - 1) atomicAdd(&size[l], __popc(peers));
            }
        }
        if (lane == 0 && body >= 0) atomicAdd(&size[body], cells);
    }
}

// The ocean: the largest body, the lowest label (the first found) among equals.
__global__ void k_ocean(const int* __restrict__ size, int count, unsigned long long* __restrict__ best) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < count; b += gridDim.x * blockDim.x)
        atomicMax(best, ((unsigned long long)(unsigned)size[b] << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned)b));
}

// Every water body but the ocean, no larger than the largest lake, becomes land at its own height.
__global__ void k_enclose(uint8_t* __restrict__ land, float* __restrict__ rel, const int* __restrict__ label,
                          const int* __restrict__ size, const unsigned long long* __restrict__ best, int largest,
                          const float* __restrict__ h, float shoreline, float land_half, size_t N, int* __restrict__ added) {
    const int ocean = (int)(0xFFFFFFFFu - (unsigned)(*best & 0xFFFFFFFFull));
    int mine = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        const int b = label[i];
        if (b < 0 || b == ocean || size[b] > largest) continue;
        land[i] = 1;
        rel[i] = __fdiv_rn(__fsub_rn(h[i], shoreline), land_half);
        ++mine;
    }
    if (mine) atomicAdd(added, mine);
}

// SeaLevelStage.landAndWaterAt at a given shoreline.
__global__ void k_land_water_at(const float* __restrict__ h, size_t N, float shoreline, float land_half, float sea_half,
                                uint8_t* __restrict__ land, float* __restrict__ rel, int* __restrict__ count) {
    int mine = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        const float g = h[i];
        const bool on = g >= shoreline;
        land[i] = on ? 1 : 0;
        rel[i] = __fdiv_rn(__fsub_rn(g, shoreline), on ? land_half : sea_half);
        mine += on ? 1 : 0;
    }
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xFFFFFFFFu, mine, o);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(count, mine);
}

// The drowned basins, those whose floor stands below the shoreline and that have a spill, listed in
// basin order by one CTA (the others are the rounds' notch's). The notch's one thread stepping over
// every basin took 4.4 ms a pass at 1024 x 512.
struct Drowned {
    int spill, entry;
    float level, floor_;
};

__global__ void __launch_bounds__(1024) k_list_drowned(const int* __restrict__ spill, const int* __restrict__ entry,
                                                       const float* __restrict__ level, const float* __restrict__ floor_,
                                                       int count, Drowned* __restrict__ list, int* __restrict__ drowned) {
    __shared__ int warps[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int listed = 0;
    for (int base = 0; base < count; base += 1024) {
        const int b = base + (int)threadIdx.x;
        const int sp = b < count ? spill[b] : -1;
        const float fl = b < count ? floor_[b] : 0.0f;
        const bool in = sp >= 0 && !(fl >= 0.0f);
        const unsigned ballot = __ballot_sync(0xFFFFFFFFu, in);
        if (lane == 0) warps[warp] = __popc(ballot);
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            before += w < warp ? warps[w] : 0;
            all += warps[w];
        }
        if (in) list[listed + before + __popc(ballot & ((1u << lane) - 1u))] = Drowned{sp, entry[b], level[b], fl};
        listed += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *drowned = listed;
}

struct NotchArgs {
    int W, H, count;
    const Drowned* list;
    int cap;             // cells a walk can hold
    int* cut_cell;       // scratch, 3 cap a warp: the cells its basin cuts and the levels it cuts them to
    float* cut_level;
    int* chain;          // scratch, cap a warp: a margin's cells
    int* read_cell;      // scratch, 11 cap a warp: the cells whose heights a basin's walks read
    int* stamp;          // per cell: the wave and the first basin of it that cuts the cell
    int wave0;           // waves stamped so far
    const uint8_t* land;
    const int32_t* dirs;
    const float* area;
    float* rel;
    float* ground;
    float* surface;
    float land_cells, land_range, pond_depth, coefficient, gradient, reach, step_ns, step_diag;
    int* cells;
};

__device__ __forceinline__ float jvm_minf(float a, float b) {
    if (a != a) return a;
    if (b != b) return b;
    if (a == 0.0f && b == 0.0f) return __float_as_int(a) < 0 ? a : b;
    return a < b ? a : b;
}

__device__ __forceinline__ float step_between(const NotchArgs& a, int from, int to) {
    const bool same_row = pdiv(from, a.W) == pdiv(to, a.W), same_col = pmod(from, a.W) == pmod(to, a.W);
    return (!same_row && !same_col) ? a.step_diag : (!same_row ? a.step_ns : 1.0f);
}

// HydraulicErosion.raise with -take, and the relative fields it lowers; returns whether it cut.
__device__ bool take_down(const NotchArgs& a, int cell, float cut_level, bool lower_ground) {
    const double take = (double)(a.rel[cell] - cut_level) * (double)a.land_range;
    const bool ponded = a.ground[cell] - a.rel[cell] > a.pond_depth;
    const float prior = a.surface[cell];
    a.surface[cell] = (float)((double)prior + -take);
    const double removed = -((double)a.surface[cell] - (double)prior);
    if (removed > 0.0) {
        const float as_relative = (float)(removed / (double)a.land_range);
        a.rel[cell] -= as_relative;
        if (lower_ground && !ponded) a.ground[cell] -= as_relative;
        return true;
    }
    return false;
}

// A wave of the notch: up to `kNotchWarps` basins, `rank` this warp's among them. A stamp orders waves, then
// the basins of a wave, the first the greatest. A basin's lists hold kNotchWords words for every cell that a
// walk can reach, the whole map where the reach is wider than it: fewer basins a wave then, so that the lists
// stay within kNotchScratch (4.8 GB at 2048 x 1024 with 32, and at 2^27 cells more than the GPU holds).
constexpr int kNotchWarps = 32, kNotchWords = 18;
constexpr size_t kNotchScratch = 512ull << 20;
struct NotchTurn {
    int wave, rank;
    int* cut_cell;
    float* cut_level;
    int* chain;
    int* read_cell;
    int reads;
    __device__ int stamp() const { return wave * kNotchWarps + (kNotchWarps - 1 - rank); }
    __device__ void read(int cell) {   // a walk's read, the same cell in every lane
        if ((threadIdx.x & 31) == 0) read_cell[reads] = cell;
        ++reads;
    }
    __device__ void read_where(bool mine, int cell) {   // a cell of each lane that asks
        const unsigned lanes = __ballot_sync(0xFFFFFFFFu, mine);
        if (mine) read_cell[reads + __popc(lanes & ((1u << (threadIdx.x & 31)) - 1u))] = cell;
        reads += __popc(lanes);
    }
};

// HydraulicErosion.breach with belowSea on (HydraulicErosion.kt:1931-2171) for one basin, by a warp; the
// walks run the same in every lane. The cuts are listed, not made: every cell of a basin's three walks
// is a different one, and no walk reads a cell another of them cuts. Returns their number, and in
// *lowers_ground the first so many of them that take the filled surface down too.
__device__ int notch_basin(const NotchArgs& a, const Drowned& d, NotchTurn& t, int* lowers_ground) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const int spill = d.spill;
    const float level = d.level, floor_ = d.floor_;
    *lowers_ground = 0;
    if (level - floor_ <= 0.0f) return 0;
    float fall = 0.0f, length = 0.0f, last_step = 1.0f;
    int walked = 0, cell = spill;
    while (cell >= 0 && a.land[cell] && length < a.reach) {
        t.read(cell);
        fall = level - a.rel[cell];
        if (fall > level - floor_) break;
        const int next = a.dirs[cell];
        last_step = next >= 0 ? step_between(a, cell, next) : 1.0f;
        length += last_step;
        walked++;
        cell = next;
    }
    if (fall <= 1e-6f * (float)walked && cell >= 0 && !a.land[cell]) {   // outletFallToTheWater
        fall = level - a.rel[cell];
        length += last_step;
    }
    if (walked == 0) return 0;
    float slope = fall / length * (float)a.W;
    if (slope < 0.0f) slope = 0.0f;
    const float power = a.coefficient * sqrtf(a.area[spill] / a.land_cells) * slope;
    const float drop = jvm_minf(power, level - floor_);
    if (drop <= 0.0f) return 0;
    const float new_level = level - drop;
    float from_lip = 0.0f;
    int n = 0;
    cell = spill;
    while (cell >= 0 && a.land[cell] && from_lip < a.reach) {
        const float cut_level = new_level - from_lip * a.gradient;
        t.read(cell);
        if (a.rel[cell] <= cut_level) break;
        if (lane == 0) {
            t.cut_cell[n] = cell;
            t.cut_level[n] = cut_level;
        }
        ++n;
        const int next = a.dirs[cell];
        from_lip += next >= 0 ? step_between(a, cell, next) : 1.0f;
        cell = next;
    }
    const int entry = d.entry;
    float back = 0.0f;
    if (entry >= 0 && entry != spill) {
        int margin_cells = 0, walker = entry;
        float widths = 0.0f;
        while (walker >= 0 && walker != spill && a.land[walker] && widths <= a.reach) {
            const int next = a.dirs[walker];
            widths += next >= 0 ? step_between(a, walker, next) : 1.0f;
            if (lane == 0) t.chain[margin_cells] = walker;
            margin_cells++;
            walker = next;
        }
        __syncwarp();
        if (walker == spill) {
            // The margin from the lip back towards the entry: the chain entry -> ... -> spill, walked
            // backwards over its listed cells (distinct, as a forest's chain is).
            int downstream = spill;
            for (int i = margin_cells - 1; i >= 0; --i) {
                const int m = t.chain[i];
                back += step_between(a, m, downstream);
                const float cut_level = new_level + back * a.gradient;
                t.read(m);
                if (a.rel[m] <= cut_level) break;
                if (lane == 0) {
                    t.cut_cell[n] = m;
                    t.cut_level[n] = cut_level;
                }
                ++n;
                downstream = m;
            }
        }
        __syncwarp();   // the chain is read before the next walk writes it
    }
    // The sill on the basin's own side: up the inflow of the largest catchment across the bed. A step
    // reads only cells upstream of `from`, which no cut of this basin touched.
    int from = entry >= 0 ? entry : spill;
    *lowers_ground = n;
    while (back <= a.reach) {
        const int k = lane < 4 ? lane : lane + 1;   // lanes 0-7: the neighbours, rows then columns
        const int nr = pdiv(from, a.W) + k / 3 - 1;
        int best = -1;
        float best_area = -1.0f;
        const int nb = nr * a.W + ((pmod(from, a.W) + k % 3 - 1) & (a.W - 1));
        const bool donor = lane < 8 && nr >= 0 && nr < a.H && a.land[nb] && a.dirs[nb] == from;
        t.read_where(donor, nb);
        if (donor) {
            const float ar = a.area[nb];
            if (a.ground[nb] - a.rel[nb] > a.pond_depth && ar >= -1.0f) {
                best = nb;
                best_area = ar;
            }
        }
        for (int o = 4; o > 0; o >>= 1) {   // the largest catchment, ties on the lower index
            const int ob = __shfl_down_sync(FULL, best, o);
            const float oa = __shfl_down_sync(FULL, best_area, o);
            if (ob >= 0 && (best < 0 || oa > best_area || (oa == best_area && ob < best))) {
                best = ob;
                best_area = oa;
            }
        }
        best = __shfl_sync(FULL, best, 0);
        if (best < 0) break;
        back += step_between(a, best, from);
        if (back > a.reach) break;
        const float cut_level = new_level + back * a.gradient;
        if (a.rel[best] <= cut_level) break;
        if (lane == 0) {
            t.cut_cell[n] = best;
            t.cut_level[n] = cut_level;
        }
        ++n;
        from = best;
    }
    return n;
}

// The drowned basins in waves of up to a basin a warp, in order. The first basin of a wave never finds a clash,
// so every wave cuts at least one.
__global__ void __launch_bounds__(32 * kNotchWarps) k_notch_below_sea(NotchArgs a) {
    __shared__ int first_clash;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    NotchTurn t;
    t.wave = a.wave0;
    t.rank = warp;
    t.cut_cell = a.cut_cell + (size_t)warp * 3 * a.cap;
    t.cut_level = a.cut_level + (size_t)warp * 3 * a.cap;
    t.chain = a.chain + (size_t)warp * a.cap;
    t.read_cell = a.read_cell + (size_t)warp * 11 * a.cap;
    int cells = 0;
    for (int b0 = 0; b0 < a.count;) {
        ++t.wave;
        t.reads = 0;
        if (threadIdx.x == 0) first_clash = warps;
        const int b = b0 + warp;
        int n = 0, lowers = 0;
        Drowned d{};
        if (b < a.count) {
            d = a.list[b];
            n = notch_basin(a, d, t, &lowers);
            __syncwarp();
            for (int i = lane; i < n; i += 32) atomicMax(&a.stamp[t.cut_cell[i]], t.stamp());
        }
        __syncthreads();
        bool clash = false;
        for (int i = lane; i < t.reads; i += 32) {
            const int stamp = __ldcg(&a.stamp[t.read_cell[i]]);
            clash |= stamp > t.stamp() && stamp < (t.wave + 1) * kNotchWarps;
        }
        if (__any_sync(0xFFFFFFFFu, clash) && lane == 0) atomicMin(&first_clash, warp);
        __syncthreads();
        const int go = min(first_clash, a.count - b0);
        if (warp < go)
            for (int i = lane; i < n; i += 32)
                if (take_down(a, t.cut_cell[i], t.cut_level[i], i < lowers)) ++cells;
        __syncthreads();   // the cuts are made, and first_clash read, before the next wave
        b0 += go;
    }
    cells = __reduce_add_sync(0xFFFFFFFFu, cells);
    if (threadIdx.x == 0) *a.cells = 0;
    __syncthreads();
    if (lane == 0 && cells) atomicAdd(a.cells, cells);
}

cg_status enclose_dev(cg_ctx* ctx, int W, int H, uint8_t* d_land, float* d_rel, const float* d_h, float shoreline,
                      float land_half, int largest_lake, int* land_cells) {
    const size_t N = (size_t)W * H;
    cudaStream_t sm = ctx->stream;
    const int grid = ctx->num_sms * 8;
    CG_BUF(uint8_t, d_mask, ctx, S_SL_MASK, N);
    CG_BUF(int, d_root, ctx, S_LABEL, N);
    CG_BUF(int, d_label, ctx, S_SL_LABEL, N);
    CG_LAUNCH(ctx) k_water_mask<<<grid, 256, 0, sm>>>(d_land, N, d_mask);
    CG_CHECK_LAUNCH(ctx);
    int bodies = 0;
    CG_TRY_ST(component_labels(ctx, W, H, d_mask, d_root, d_label, &bodies));
    if (bodies <= 1) return CG_OK;
    CG_BUF(int, d_size, ctx, S_SL_SIZE, (size_t)bodies + 4);
    unsigned long long* d_best = (unsigned long long*)(d_size + bodies + (bodies & 1));
    int* d_added = (int*)(d_best + 1);
    CG_CUDA(ctx, cudaMemsetAsync(d_size, 0, ((size_t)bodies + 4) * sizeof(int), sm));
    CG_LAUNCH(ctx) k_body_sizes<<<grid, 256, 0, sm>>>(d_label, N, d_size);
    CG_LAUNCH(ctx) k_ocean<<<(bodies + 255) / 256, 256, 0, sm>>>(d_size, bodies, d_best);
    CG_LAUNCH(ctx) k_enclose<<<grid, 256, 0, sm>>>(d_land, d_rel, d_label, d_size, d_best, largest_lake, d_h, shoreline,
                                                 land_half, N, d_added);
    CG_CHECK_LAUNCH(ctx);
    int added = 0;
    CG_CUDA(ctx, cudaMemcpyAsync(&added, d_added, sizeof(int), cudaMemcpyDeviceToHost, sm));
    CG_CUDA(ctx, cudaStreamSynchronize(sm));
    *land_cells += added;
    return CG_OK;
}

}  // namespace
}  // namespace cg

using namespace cg;

extern "C" cg_status cg_sea_level_cut(cg_ctx* ctx, const cg_erosion_params* p, const float* height,
                                      double enclosed_sea_max_share, int32_t post_cut_outlet, float* shoreline,
                                      uint8_t* is_land, float* relative, int32_t* land_cells, int32_t* passes) {
    if (!ctx || !p || !height || !shoreline || !is_land || !relative || !land_cells) return CG_BAD_ARG;
    ctx->run.active = false;   // this call reuses the resident world's buffers
    const int W = p->width, H = p->height;
    if (W <= 0 || H <= 0 || (W & (W - 1)) || (H & (H - 1)) || (int64_t)W * H > ((int64_t)1 << 30))
        return fail(ctx, CG_BAD_ARG, "width/height must be powers of two (got %d x %d)", W, H);
    if (p->abi_version != CG_ABI_VERSION) return fail(ctx, CG_BAD_ARG, "params carry ABI version %u", p->abi_version);
    if (!(enclosed_sea_max_share >= 0.0)) return fail(ctx, CG_BAD_ARG, "negative enclosed-sea share");
    CG_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t N = (size_t)W * H;
    cudaStream_t sm = ctx->stream;
    const int grid = ctx->num_sms * 8;
    const ScaleF sc = scale_of(*p);
    const RatesF rates = rates_of(*p);
    const float land_half = std::fmax(sc.land_half(), 1e-6f);
    const float sea_half = std::fmax(sc.sea_half(), 1e-6f);
    const double km2_per_cell = sc.cell_width_km(W) * sc.cell_height_km(H);
    const int largest_lake = (int)(enclosed_sea_max_share * sc.world_area_km2() / km2_per_cell);
    CG_BUF(float, d_h, ctx, S_H0, N);
    CG_BUF(float, d_terrain, ctx, S_H1, N);
    CG_BUF(uint8_t, d_land, ctx, S_LAND, N);
    CG_BUF(float, d_rel, ctx, S_REL, N);
    CG_BUF(float, d_filled, ctx, S_FILLED, N);
    CG_BUF(double, d_surface, ctx, S_SURFACE, N);
    CG_BUF(int32_t, d_recv, ctx, S_RECV, N);
    CG_BUF(int32_t, d_donors, ctx, S_DONORS, N);
    CG_BUF(long long, d_key, ctx, S_KEY, N);
    CG_BUF(float, d_area, ctx, S_AREA, N);
    CG_BUF(float, d_ones, ctx, S_RUNOFF, N);
    CG_BUF(int32_t, d_bl, ctx, S_BASIN2, N);
    CG_BUF(int, d_words, ctx, S_SL_WORDS, 4);
    CG_CUDA(ctx, cudaMemcpyAsync(d_h, height, N * 4, cudaMemcpyHostToDevice, sm));
    float s = 0.0f;
    int n = 0;
    CG_TRY_ST(percentile_cut_dev(ctx, W, H, d_h, p->sea_level, land_half, sea_half, 0.0f, d_land, d_rel, &s, &n));
    CG_TRY_ST(enclose_dev(ctx, W, H, d_land, d_rel, d_h, s, land_half, largest_lake, &n));
    int run = 0;
    bool have_terrain = false;
    int waves = 0;
    for (int pass = 0; post_cut_outlet && pass < 16 && n > 0; ++pass) {   // MAX_POST_CUT_OUTLET_PASSES
        CG_TRY_ST(fill_depressions_dev(ctx, W, H, d_land, d_rel, d_filled, nullptr, nullptr));
        FlatCounts fc{0, 0, 0};
        CG_TRY_ST(flow_directions_dev(ctx, W, H, d_land, d_rel, d_filled, p->seed, rates.cell_height_in_cell_widths,
                                      smooth_field_lattice_columns(p->world_width_km), p->facet_routing != 0,
                                      p->flat_potential != 0, d_recv, d_surface, &fc));
        CG_TRY_ST(runoff_weights_dev(ctx, W, H, nullptr, d_land, n, d_ones));
        CG_TRY_ST(tree_walk_dev(ctx, W, H, d_land, d_recv, d_ones, d_key, d_donors, d_area, nullptr));
        BasinArrays bas;
        int count = 0;
        CG_TRY_ST(basins_dev(ctx, W, H, d_land, d_rel, d_filled, d_recv, rates.pond_depth, d_bl, &bas, &count));
        if (count == 0) break;
        CG_BUF(Drowned, d_list, ctx, S_SL_LIST, (size_t)count);
        // A walk's cells are distinct and their summed steps stay within the reach; twice that leaves room
        // for the rounding of the sums.
        const float least = std::fmin(1.0f, rates.step_ns);
        const size_t cap = (size_t)std::fmin((double)N, 2.0 * std::ceil((double)rates.outlet_reach_cells / least) + 64.0) + 4;
        const size_t warps = std::max<size_t>(1, std::min<size_t>(kNotchWarps, kNotchScratch / (kNotchWords * sizeof(int) * cap)));
        CG_BUF(int, d_chain, ctx, S_SL_CHAIN, kNotchWords * warps * cap);
        CG_BUF(int, d_stamp, ctx, S_SL_STAMP, N);
        if (pass == 0 || waves > (1 << 24)) {   // stamps stay within an int
            CG_CUDA(ctx, cudaMemsetAsync(d_stamp, 0, N * sizeof(int), sm));
            waves = 0;
        }
        CG_CUDA(ctx, cudaMemsetAsync(d_words, 0, 4 * sizeof(int), sm));
        CG_LAUNCH(ctx) k_list_drowned<<<1, 1024, 0, sm>>>(bas.spill, bas.entry, bas.level, bas.floor_, count, d_list, d_words);
        CG_CHECK_LAUNCH(ctx);
        int drowned = 0;
        CG_CUDA(ctx, cudaMemcpyAsync(&drowned, d_words, sizeof(int), cudaMemcpyDeviceToHost, sm));
        CG_CUDA(ctx, cudaStreamSynchronize(sm));
        if (drowned == 0) break;
        if (!have_terrain) {
            CG_CUDA(ctx, cudaMemcpyAsync(d_terrain, d_h, N * 4, cudaMemcpyDeviceToDevice, sm));
            have_terrain = true;
        }
        run = pass + 1;
        NotchArgs a;
        a.W = W;
        a.H = H;
        a.count = drowned;
        a.list = d_list;
        a.chain = d_chain;
        a.cut_cell = d_chain + warps * cap;
        a.cut_level = (float*)(d_chain + 4 * warps * cap);
        a.read_cell = d_chain + 7 * warps * cap;
        a.cap = (int)cap;
        a.stamp = d_stamp;
        a.wave0 = waves;
        waves += drowned;   // a wave cuts a basin at least
        a.land = d_land;
        a.dirs = d_recv;
        a.area = d_area;
        a.rel = d_rel;
        a.ground = d_filled;
        a.surface = d_terrain;
        a.land_cells = (float)n;
        a.land_range = land_half;
        a.pond_depth = rates.pond_depth;
        a.coefficient = rates.relative_incision_coefficient * 1.125f;   // ErosionConfig.outletIncisionRatio
        a.gradient = rates.notch_fall_per_cell;
        a.reach = (float)rates.outlet_reach_cells;
        a.step_ns = rates.step_ns;
        a.step_diag = rates.step_diag;
        a.cells = d_words + 1;
        CG_LAUNCH(ctx) k_notch_below_sea<<<1, 32 * (unsigned)warps, 0, sm>>>(a);
        CG_CHECK_LAUNCH(ctx);
        int cut = 0;
        CG_CUDA(ctx, cudaMemcpyAsync(&cut, d_words + 1, sizeof(int), cudaMemcpyDeviceToHost, sm));
        CG_CUDA(ctx, cudaStreamSynchronize(sm));
        if (cut == 0) break;
        // The re-cut at the same shoreline over the cut terrain, and the enclosure rule again.
        CG_CUDA(ctx, cudaMemsetAsync(d_words + 2, 0, sizeof(int), sm));
        CG_LAUNCH(ctx) k_land_water_at<<<grid, 256, 0, sm>>>(d_terrain, N, s, land_half, sea_half, d_land, d_rel,
                                                           d_words + 2);
        CG_CHECK_LAUNCH(ctx);
        CG_CUDA(ctx, cudaMemcpyAsync(&n, d_words + 2, sizeof(int), cudaMemcpyDeviceToHost, sm));
        CG_CUDA(ctx, cudaStreamSynchronize(sm));
        CG_TRY_ST(enclose_dev(ctx, W, H, d_land, d_rel, d_terrain, s, land_half, largest_lake, &n));
    }
    CG_CUDA(ctx, cudaMemcpyAsync(is_land, d_land, N, cudaMemcpyDeviceToHost, sm));
    CG_CUDA(ctx, cudaMemcpyAsync(relative, d_rel, N * 4, cudaMemcpyDeviceToHost, sm));
    CG_TRY_ST(sync(ctx));
    *shoreline = s;
    *land_cells = n;
    if (passes) *passes = run;
    return CG_OK;
}
