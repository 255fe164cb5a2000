// Musgrave thermal sweeps (ErosionStage.thermalSweep, ErosionStage.kt:235-403), fused for GB300.
//
// One sweep is two passes in the reference: every cell's give rate from its 8 neighbours, then
// every cell's new height from its neighbours' give rates. Here one CTA owns a tile (64 x 32, 32 x 16 on small grids) and
// loads it with a halo of 4 cells into shared memory; it runs two sweeps there (or one, for an odd
// remainder), each sweep's region shrinking by two cells a side (one for the give pass, one for
// the move pass), and writes the tile back once.
//
// The passes are bound by instruction issue, so they issue little for a cell at rest (most cells are, in
// most sweeps) and share work between the passes: a cell gives only if it stands above its lowest
// neighbour by more than the least limit, and that lowest is kept row by row as a 3 x 3 window slides
// down a thread's column; the give pass also takes what the cell itself gives off its height, with the
// falls it has at hand, so the move pass only adds what comes in and leaves a cell alone when no
// neighbour gives. A thread takes a column of 8 to 10 rows (4 to 6), so that four runs of rows times the
// region's columns are one step of the CTA's 288 threads (92% busy over the four passes) and the
// window's two extra rows cost a fifth of the loads. The 384 launches of an 8192 x 4096 stage take 89.5
// ms (113 with each pass running its whole rule on 4-row columns), 192 sweeps at 4096 x 2048 5.5 ms
// (6.5). Queueing the active cells and running the rules on 32 of them at a time was slower (10.4 ms):
// the queue's own instructions are as many as the rules'.
//
// The arithmetic per cell is the reference's, in the same neighbour order, in float, with no
// fused multiply-add, so the result is bit-identical to ErosionStage.thermalSweep. Rows off the grid
// hold NaN, which no comparison of the rules lets through. Limits below zero (no preset has them) take
// a plain per-cell form of the same rules.
#include <cuda.h>

#include <cmath>

#include "cg_common.cuh"
#include "cg_internal.h"

namespace cg {

namespace {

constexpr int KMAX = 2;
constexpr int HALO = 2 * KMAX;

// A CTA's tile, its region with the halo, and its threads: four runs of rows times up to RW - 2 columns, a
// thread each.
template <int X, int Y, int CTAS>
struct Shape {
    static constexpr int TX = X, TY = Y;
    static constexpr int RW = TX + 2 * HALO, RH = TY + 2 * HALO;
    static constexpr int THREADS = (4 * (RW - 2) + 31) / 32 * 32;
    static constexpr int MIN_CTAS = CTAS;
};
using Wide = Shape<64, 32, 5>;    // 288 threads
using Small = Shape<32, 16, 8>;   // 160 threads
// A grid of fewer Wide tiles than SMs is a matter of one CTA's time, and a Small tile's columns are 4 to 6
// rows long instead of 8 to 10: 24 sweeps at 512 x 256 took 128 us with 64 Wide tiles and take 108 with 256
// Small ones, though nearly half of their region is halo.
bool small_tiles(int W, int H) {
    return (long long)((W + Wide::TX - 1) / Wide::TX) * ((H + Wide::TY - 1) / Wide::TY) < kSMs;
}

struct ThermalArgs {
    float limit[8];
    float settled;
    float rate;
    float ew, ns, diag;   // the limits by neighbour kind
    float least;          // the least of them
    int plain;            // every limit >= 0 and settled >= 0: the forms below are exact
};

// Settled-tile skip (the reference's own skip, ErosionStage.kt:269-342, restated for fused launches).
// A launch carries any change at most 4 cells, less than a tile's side, so a tile can
// change only if a cell of it or of one of its 8 neighbouring tiles changed in the previous launch.
// `prev` holds those per-tile "changed" bits (null: compute every tile); each launch writes its own
// into `cur`. A skipped tile is not even copied: the launches ping-pong between two buffers, and a
// tile that did not change in the previous launch holds the same bits in both.
struct TileFlags {
    const uint8_t* prev;
    uint8_t* cur;
};

// The region load by the tensor memory accelerator: one cp.async.bulk.tensor.2d per CTA of the
// whole RW x RH region, rows off the grid filled with NaN by the copy itself. Used on tiles whose
// region does not wrap east-west (its first column, TX bx - 4, is 16-byte aligned as TMA requires); the
// two wrapping tile columns load by threads. `err` (device) is set when a copy's wait runs out, after
// which the CTA waits once more for its copy and leaves without computing; the host reports it.
struct RegionLoad {
    CUtensorMap map;   // the source field, box = the region
    int on;            // a map was made for this launch
    int* err;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Waits on the mbarrier's phase 0 for at most `tries` polls; true when the phase completed.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, int tries) {
    for (int i = 0; i < tries; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(0)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Neighbours in the reference's order: E, W, S, N, then SE, NE, SW, NW.
struct Around {
    float v[8];
};
__device__ __forceinline__ float limit_of(const ThermalArgs& a, int n) { return n >= 4 ? a.diag : n >= 2 ? a.ns : a.ew; }

// The give pass's rule on a cell of height c that stands above its lowest neighbour by more than the least
// limit (ErosionStage.kt:283-311 and the giving half of 313-340), limits >= 0: returns its give rate and
// takes what it gives off c. A fall counts when it is above its limit; a fall at or below it enters the
// sums as +0, which changes no bit of a sum that starts at +0 and gains only terms >= 0. The steepest
// fall is that to the lowest neighbour (float subtraction is monotone).
__device__ __forceinline__ float give(float& c, const Around& nb, float lowest, const ThermalArgs& a) {
    float over[8];
    float excess = 0.0f;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        over[n] = fmaxf(__fsub_rn(__fsub_rn(c, nb.v[n]), limit_of(a, n)), 0.0f);
        excess = __fadd_rn(excess, over[n]);
    }
    if (!(excess > a.settled)) return 0.0f;
    const float p = __fmul_rn(a.rate, excess), q = __fmul_rn(__fsub_rn(c, lowest), 0.5f);
    const float rate = __fdiv_rn(p <= q ? p : q, excess);
    float given = 0.0f;
#pragma unroll
    for (int n = 0; n < 8; ++n) given = __fadd_rn(given, __fmul_rn(rate, over[n]));
    c = __fsub_rn(c, given);
    return rate;
}

// The move pass's rule on a cell of height c: what the neighbours that stand above it by more than their
// limits give it (ErosionStage.kt:313-340).
__device__ __forceinline__ float received(float c, const Around& nb, const Around& g, const ThermalArgs& a) {
    float sum = 0.0f;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        const float over = __fsub_rn(__fsub_rn(nb.v[n], c), limit_of(a, n));
        const float p = __fmul_rn(g.v[n], over);
        if (over > 0.0f) sum = __fadd_rn(sum, p);
    }
    return sum;
}

// This thread's column and run of rows [row0, row1) of the region's rows and columns [M, R - M).
struct Run {
    int col, row0, row1;
};
template <class S, int M>
__device__ __forceinline__ bool run_of(Run& r) {
    constexpr int COLS = S::RW - 2 * M, PER = (S::RH - 2 * M + 3) / 4;
    static_assert(4 * COLS <= S::THREADS, "a thread takes one run");
    const int part = (int)threadIdx.x / COLS;
    r.col = M + (int)threadIdx.x - part * COLS;
    r.row0 = M + part * PER;
    r.row1 = min(r.row0 + PER, S::RH - M);
    return part < 4;
}
// A change at this row counts for the tile's flag where the column and row are the tile's own.
template <class S>
__device__ __forceinline__ bool own_col(int col) { return col >= HALO && col < HALO + S::TX; }
template <class S>
__device__ __forceinline__ bool own_row(int row) { return row >= HALO && row < HALO + S::TY; }

// The give pass from h: rates into g, what is left of the heights into left. The left height is
// (c - given) + 0, since the reference adds what a cell receives, if only +0. Returns whether any of the
// thread's cells gives.
template <class S, int M>
__device__ __forceinline__ bool give_pass(const float* __restrict__ h, float* __restrict__ left, float* __restrict__ g,
                                          const ThermalArgs& a, bool& changed) {
    constexpr int RW = S::RW;
    Run r;
    if (!run_of<S, M>(r)) return false;
    bool any = false;
    unsigned moved = 0;
    const bool own = own_col<S>(r.col);
    const float* p = h + (r.row0 - 1) * RW + r.col;
    float nw = p[-1], n = p[0], ne = p[1], w = p[RW - 1], c = p[RW], e = p[RW + 1];
    float top = fminf(fminf(nw, n), ne), mid = fminf(fminf(w, c), e);
#pragma unroll 3
    for (int row = r.row0; row < r.row1; ++row) {
        const int i = row * RW + r.col;
        const float sw = h[i + RW - 1], s = h[i + RW], se = h[i + RW + 1];
        const float bot = fminf(fminf(sw, s), se);
        const float lowest = fminf(fminf(top, mid), bot);
        float rate = 0.0f, v = c;
        if (__fsub_rn(c, lowest) > a.least) rate = give(v, Around{{e, w, s, n, se, ne, sw, nw}}, lowest, a);
        v = __fadd_rn(v, 0.0f);
        g[i] = rate;
        left[i] = v;
        any |= rate != 0.0f;
        if (own_row<S>(row)) moved |= __float_as_uint(v) ^ __float_as_uint(c);
        nw = w, n = c, ne = e;
        w = sw, c = s, e = se;
        top = mid, mid = bot;
    }
    if (own && moved) changed = true;
    return any;
}

// The move pass: what each cell receives, read from h and g, onto left.
template <class S, int M>
__device__ __forceinline__ void move_pass(const float* __restrict__ h, float* __restrict__ left, const float* __restrict__ g,
                                          const ThermalArgs& a, bool& changed) {
    constexpr int RW = S::RW;
    Run r;
    if (!run_of<S, M>(r)) return;
    unsigned moved = 0;
    const bool own = own_col<S>(r.col);
    const float* p = h + (r.row0 - 1) * RW + r.col;
    const float* q = g + (r.row0 - 1) * RW + r.col;
    float nw = p[-1], n = p[0], ne = p[1], w = p[RW - 1], c = p[RW], e = p[RW + 1];
    float gnw = q[-1], gn = q[0], gne = q[1], gw = q[RW - 1], gc = q[RW], ge = q[RW + 1];
    unsigned top = __float_as_uint(gnw) | __float_as_uint(gn) | __float_as_uint(gne);
#pragma unroll 3
    for (int row = r.row0; row < r.row1; ++row) {
        const int i = row * RW + r.col;
        const float sw = h[i + RW - 1], s = h[i + RW], se = h[i + RW + 1];
        const float gsw = g[i + RW - 1], gs = g[i + RW], gse = g[i + RW + 1];
        const unsigned sides = __float_as_uint(gw) | __float_as_uint(ge);
        const unsigned bot = __float_as_uint(gsw) | __float_as_uint(gs) | __float_as_uint(gse);
        if (top | sides | bot) {   // a neighbour gives
            const float v = __fadd_rn(left[i], received(c, Around{{e, w, s, n, se, ne, sw, nw}},
                                                        Around{{ge, gw, gs, gn, gse, gne, gsw, gnw}}, a));
            left[i] = v;
            if (own_row<S>(row)) moved |= __float_as_uint(v) ^ __float_as_uint(c);
        }
        top = sides | __float_as_uint(gc);
        nw = w, n = c, ne = e;
        w = sw, c = s, e = se;
        gnw = gw, gn = gc, gne = ge;
        gw = gsw, gc = gs, ge = gse;
    }
    if (own && moved) changed = true;
}

// The reference's rules on one cell of the region for any limits: rows off the grid are told apart by
// `has_s` / `has_n` (the rows below and above exist).
template <class S>
__device__ float give_rate(const float* h, int i, bool has_s, bool has_n, const ThermalArgs& a) {
    constexpr int RW = S::RW;
    const int off[8] = {1, -1, RW, -RW, RW + 1, -RW + 1, RW - 1, -RW - 1};
    const bool ok[8] = {true, true, has_s, has_n, has_s, has_n, has_s, has_n};
    float excess = 0.0f, steepest = 0.0f;
    for (int n = 0; n < 8; ++n) {
        if (!ok[n]) continue;
        const float drop = __fsub_rn(h[i], h[i + off[n]]);
        if (drop > steepest) steepest = drop;
        if (drop > 0.0f && drop > a.limit[n]) excess = __fadd_rn(excess, __fsub_rn(drop, a.limit[n]));
    }
    if (!(excess > a.settled)) return 0.0f;
    const float p = __fmul_rn(a.rate, excess), q = __fmul_rn(steepest, 0.5f);
    return __fdiv_rn(p <= q ? p : q, excess);
}

template <class S>
__device__ float moved(const float* h, const float* g, int i, bool has_s, bool has_n, const ThermalArgs& a) {
    constexpr int RW = S::RW;
    const int off[8] = {1, -1, RW, -RW, RW + 1, -RW + 1, RW - 1, -RW - 1};
    const bool ok[8] = {true, true, has_s, has_n, has_s, has_n, has_s, has_n};
    float received = 0.0f, given = 0.0f;
    for (int n = 0; n < 8; ++n) {
        if (!ok[n]) continue;
        const float incoming = __fsub_rn(h[i + off[n]], h[i]);
        if (incoming > a.limit[n])
            received = __fadd_rn(received, __fmul_rn(g[i + off[n]], __fsub_rn(incoming, a.limit[n])));
        else if (-incoming > a.limit[n])
            given = __fadd_rn(given, __fmul_rn(g[i], __fsub_rn(-incoming, a.limit[n])));
    }
    return __fadd_rn(__fsub_rn(h[i], given), received);
}

// One sweep by those rules over rows and columns [M + 1, R - M - 1) from h into to.
template <class S, int M>
__device__ void any_sweep(const float* h, float* to, float* g, int y0, int H, const ThermalArgs& a, bool& changed) {
    constexpr int RW = S::RW, RH = S::RH, TX = S::TX, TY = S::TY, THREADS = S::THREADS;
    for (int i = threadIdx.x; i < RW * RH; i += THREADS) {
        const int row = i / RW, col = i % RW, y = y0 + row;
        if (row < M || row >= RH - M || col < M || col >= RW - M || y < 0 || y >= H) continue;
        g[i] = give_rate<S>(h, i, y + 1 < H, y > 0, a);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < RW * RH; i += THREADS) {
        const int row = i / RW, col = i % RW, y = y0 + row;
        if (row <= M || row >= RH - M - 1 || col <= M || col >= RW - M - 1 || y < 0 || y >= H) continue;
        to[i] = moved<S>(h, g, i, y + 1 < H, y > 0, a);
        if (__float_as_uint(to[i]) != __float_as_uint(h[i]) && row >= HALO && row < HALO + TY && col >= HALO &&
            col < HALO + TX)
            changed = true;
    }
    __syncthreads();
}

// `k` sweeps (1 or 2) of the field `in` into `out`, a CTA a tile.
template <class S>
__global__ void __launch_bounds__(S::THREADS, S::MIN_CTAS) thermal_sweeps_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                                    int W, int H, int k, ThermalArgs a, TileFlags fl,
                                                                    const __grid_constant__ RegionLoad rl) {
    constexpr int RW = S::RW, RH = S::RH, TX = S::TX, TY = S::TY, THREADS = S::THREADS;
    __shared__ __align__(128) float sm_a[RW * RH];
    __shared__ __align__(16) float sm_b[RW * RH], sm_g[RW * RH];
    __shared__ __align__(8) unsigned long long bar;

    const int tile = blockIdx.y * gridDim.x + blockIdx.x;
    if (fl.prev) {
        bool near_change = false;
        for (int dy = -1; dy <= 1; ++dy) {
            int ty = (int)blockIdx.y + dy;
            if (ty < 0 || ty >= (int)gridDim.y) continue;
            for (int dx = -1; dx <= 1; ++dx) {
                int tx = ((int)blockIdx.x + dx + (int)gridDim.x) % (int)gridDim.x;
                if (fl.prev[ty * gridDim.x + tx]) near_change = true;
            }
        }
        if (!near_change) {
            if (threadIdx.x == 0) fl.cur[tile] = 0;
            return;
        }
    }

    const int x0 = blockIdx.x * TX - HALO;
    const int y0 = blockIdx.y * TY - HALO;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool tma = rl.on && x0 >= 0 && x0 + RW <= W;
    const uint32_t b = smem_addr(&bar);
    if (tma && threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(RW * RH * 4) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
            ::"r"(smem_addr(sm_a)), "l"(&rl.map), "r"(x0), "r"(y0), "r"(b)
            : "memory");
    }
    if (tma) {
        __syncthreads();
        if (!mbar_wait(b, 1 << 22)) {
            // The copy did not land: record it, give it one more bounded wait, and leave.
            if (threadIdx.x == 0) {
                atomicOr(rl.err, 1);
                mbar_wait(b, 1 << 22);
            }
            __syncthreads();
            return;
        }
    } else {
        for (int ry = warp; ry < RH; ry += THREADS / 32) {
            const int gy = y0 + ry;
            const bool valid = gy >= 0 && gy < H;
            const float* rowp = in + (size_t)(valid ? gy : 0) * W;
            for (int rx = lane; rx < RW; rx += 32)
                sm_a[ry * RW + rx] = valid ? rowp[wrap_col(x0 + rx, W)] : __int_as_float(0x7FFFFFFF);
        }
    }
    __syncthreads();

    bool moved_any = false;
    const float* res = sm_b;
    if (a.plain) {
        // A region in which no cell gives has nothing to move in the second sweep either.
        if (__syncthreads_or(give_pass<S, 1>(sm_a, sm_b, sm_g, a, moved_any))) {
            move_pass<S, 2>(sm_a, sm_b, sm_g, a, moved_any);
            __syncthreads();
            if (k == 2) {
                if (__syncthreads_or(give_pass<S, 3>(sm_b, sm_a, sm_g, a, moved_any)))
                    move_pass<S, 4>(sm_b, sm_a, sm_g, a, moved_any);
                res = sm_a;
            }
        }
    } else {
        any_sweep<S, 1>(sm_a, sm_b, sm_g, y0, H, a, moved_any);
        if (k == 2) {
            any_sweep<S, 3>(sm_b, sm_a, sm_g, y0, H, a, moved_any);
            res = sm_a;
        }
    }
    const int changed = __syncthreads_or(moved_any);   // the tile's result is in place, too
    if (fl.cur && threadIdx.x == 0) fl.cur[tile] = changed ? 1 : 0;

    if (W >= TX && (((uintptr_t)out) & 15) == 0) {
        for (int i = threadIdx.x; i < TY * TX / 4; i += THREADS) {
            const int yy = i / (TX / 4), xx = 4 * (i % (TX / 4)), gy = blockIdx.y * TY + yy;
            if (gy < H)
                *reinterpret_cast<float4*>(out + (size_t)gy * W + blockIdx.x * TX + xx) =
                    *reinterpret_cast<const float4*>(res + (yy + HALO) * RW + xx + HALO);
        }
    } else {
        for (int i = threadIdx.x; i < TY * TX; i += THREADS) {
            const int yy = i / TX, xx = i % TX, gy = blockIdx.y * TY + yy, gx = blockIdx.x * TX + xx;
            if (gy < H && gx < W) out[(size_t)gy * W + gx] = res[(yy + HALO) * RW + xx + HALO];
        }
    }
}

cudaError_t launch(const float* in, float* out, int W, int H, int k, const ThermalArgs& a, cudaStream_t st,
                   TileFlags fl = TileFlags{nullptr, nullptr}, const RegionLoad* rl = nullptr) {
    static const RegionLoad none{};
    auto run = [&](auto shape) {
        using S = decltype(shape);
        const dim3 grid((W + S::TX - 1) / S::TX, (H + S::TY - 1) / S::TY);
        thermal_sweeps_kernel<S><<<grid, S::THREADS, 0, st>>>(in, out, W, H, k, a, fl, rl ? *rl : none);
    };
    if (small_tiles(W, H)) run(Small{});
    else run(Wide{});
    return cudaGetLastError();
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's cuTensorMapEncodeTiled, fetched through the runtime (the library links no libcuda).
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// The region-load map of a field: the whole W x H field, a box of the region.
// Off (threads load every tile) where the driver has no encoder or the grid is too narrow.
RegionLoad region_load_of(const float* field, int W, int H, int* err) {
    RegionLoad rl{};
    rl.err = err;
    EncodeTiledFn enc = encode_tiled();
    const int rw = small_tiles(W, H) ? Small::RW : Wide::RW, rh = small_tiles(W, H) ? Small::RH : Wide::RH;
    if (!enc || !err || W < 2 * rw || (((uintptr_t)field) & 15) != 0) return rl;
    const cuuint64_t dims[2] = {(cuuint64_t)W, (cuuint64_t)H};
    const cuuint64_t strides[1] = {(cuuint64_t)W * sizeof(float)};
    const cuuint32_t box[2] = {(cuuint32_t)rw, (cuuint32_t)rh};
    const cuuint32_t estride[2] = {1, 1};
    if (enc(&rl.map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)field, dims, strides, box, estride,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NAN_REQUEST_ZERO_FMA) == CUDA_SUCCESS)
        rl.on = 1;
    return rl;
}

ThermalArgs args_of(const ThermalLaunch& t) {
    ThermalArgs a;
    a.plain = t.settled >= 0.0f;
    for (int n = 0; n < 8; ++n) {
        a.limit[n] = t.limit[n];
        if (!(t.limit[n] >= 0.0f)) a.plain = 0;
    }
    a.ew = t.limit[0];
    a.ns = t.limit[2];
    a.diag = t.limit[4];
    a.least = std::fmin(std::fmin(a.ew, a.ns), a.diag);
    a.settled = t.settled;
    a.rate = t.rate;
    return a;
}

}  // namespace

ThermalLaunch thermal_launch_args(cg_thermal_limits lim, float rate) {
    ThermalLaunch t;
    for (int n = 0; n < 8; ++n)
        t.limit[n] = n >= 4 ? lim.diagonal : (thermal_row_step(n) != 0 ? lim.north_south : lim.east_west);
    t.settled = lim.east_west * 1e-3f;   // SETTLED_SHARE_OF_CRITICAL_SLOPE (ErosionStage.kt:92)
    t.rate = rate;
    return t;
}

int thermal_step(int passes_left) { return passes_left >= KMAX ? KMAX : 1; }

int thermal_launches(int passes) {
    int n = 0;
    while (passes > 0) passes -= thermal_step(passes), ++n;
    return n;
}

// One fused launch of k sweeps (k = thermal_step(...)) from src into dst on `stream`.
cudaError_t thermal_launch(const float* src, float* dst, int W, int H, const ThermalLaunch& t, int k,
                           cudaStream_t stream) {
    return launch(src, dst, W, H, k, args_of(t), stream);
}

// `passes` sweeps from d_a; the result lands in *result (d_a or d_b). Deterministic ping-pong.
cg_status thermal_sweeps_dev(cg_ctx* ctx, int W, int H, float* d_a, float* d_b, cg_thermal_limits lim, int passes,
                             float rate, float** result) {
    const ThermalArgs a = args_of(thermal_launch_args(lim, rate));
    // Per-tile change bits of the previous and the current launch. The first launch computes every
    // tile (the destination holds nothing yet); after it, both buffers hold a tile's bits whenever
    // that tile did not change, so the skip needs no copy.
    const int tx = small_tiles(W, H) ? Small::TX : Wide::TX, ty = small_tiles(W, H) ? Small::TY : Wide::TY;
    const int tiles = ((W + tx - 1) / tx) * ((H + ty - 1) / ty);
    CG_BUF(uint8_t, d_flags, ctx, S_THERMFLAG, 2 * (size_t)tiles);
    CG_BUF(int, d_err, ctx, S_THERMERR, 1);
    uint8_t* prev = d_flags;
    uint8_t* cur = d_flags + tiles;
    float* src = d_a;
    float* dst = d_b;
    const RegionLoad maps[2] = {region_load_of(d_a, W, H, d_err), region_load_of(d_b, W, H, d_err)};
    bool first = true;
    while (passes > 0) {
        const int k = thermal_step(passes);
        TileFlags fl{first ? nullptr : prev, cur};
        const RegionLoad* rl = &maps[src == d_a ? 0 : 1];
        cudaError_t e = launch(src, dst, W, H, k, a, ctx->stream, fl, rl);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "thermal_sweeps_kernel", __FILE__, __LINE__);
        passes -= k;
        ctx->launches++;
        first = false;
        float* t = src;
        src = dst;
        dst = t;
        uint8_t* tf = prev;
        prev = cur;
        cur = tf;
    }
    *result = src;
    return CG_OK;
}

cg_status thermal_error_reset_dev(cg_ctx* ctx) {
    CG_BUF(int, d_err, ctx, S_THERMERR, 1);
    CG_CUDA(ctx, cudaMemsetAsync(d_err, 0, sizeof(int), ctx->stream));
    return CG_OK;
}

cg_status thermal_error_check(cg_ctx* ctx) {
    CG_BUF(int, d_err, ctx, S_THERMERR, 1);
    int err = 0;
    CG_TRY_ST(read_back(ctx, {{&err, d_err, sizeof(int)}}));
    if (err) return fail(ctx, CG_TIMEOUT, "thermal sweeps: a region copy did not arrive in its bounded wait");
    return CG_OK;
}

}  // namespace cg
