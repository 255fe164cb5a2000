// Device building blocks shared by the phases: an exclusive prefix sum, and connected-component
// labels over an 8-neighbour mask whose root is the component's smallest cell index (the order the
// reference's DFS walks number components in: ascending start cell).
#include <algorithm>
#include <cstring>

#include "cg_common.cuh"
#include "cg_util.h"

namespace cg {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanTile = 4096;         // elements a CTA scans: 16 a thread
constexpr int kScanDirect = kScanTile;  // tiles whose sums every CTA adds up itself

// The exclusive prefix of v over the CTA's threads, and the total; sh holds kScanThreads / 32 ints.
__device__ __forceinline__ int cta_prefix(int v, int* total, int* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
        before += w < warp ? sh[w] : 0;
        all += sh[w];
    }
    __syncthreads();
    *total = all;
    return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_sums(const int* __restrict__ in, int n, int* __restrict__ sums) {
    __shared__ int sh[kScanThreads / 32];
    const int base = blockIdx.x * kScanTile;
    int v = 0;
#pragma unroll
    for (int k = 0; k < kScanTile / kScanThreads; ++k) {
        const int i = base + k * kScanThreads + (int)threadIdx.x;
        v += i < n ? in[i] : 0;
    }
    int total;
    cta_prefix(v, &total, sh);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// A tile's exclusive scan, from the sum of the tiles before it: added up here from the tiles' sums, or
// read where they have been scanned. The last tile leaves the total.
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const int* __restrict__ in, int n,
                                                             const int* __restrict__ sums, const int* __restrict__ offs,
                                                             int* __restrict__ out, int* __restrict__ total) {
    __shared__ int sh[kScanThreads / 32];
    __shared__ int warp_sum[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kPer = kScanTile / kScanThreads;
    // A warp's kPer rows of 32 elements, a row a lane-wide scan.
    const int base = blockIdx.x * kScanTile + warp * 32 * kPer + lane;
    int v[kPer], run = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) v[k] = base + 32 * k < n ? in[base + 32 * k] : 0;
    int tile_offset = 0;
    if (offs) {
        tile_offset = offs[blockIdx.x];
    } else if (blockIdx.x > 0) {
        int part = 0;
        for (int b = threadIdx.x; b < (int)blockIdx.x; b += kScanThreads) part += sums[b];
        cta_prefix(part, &tile_offset, sh);
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        int x = v[k];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        v[k] = run + x - v[k];
        run += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
    if (lane == 0) warp_sum[warp] = run;
    __syncthreads();
    int before = tile_offset;
    for (int w = 0; w < warp; ++w) before += warp_sum[w];
#pragma unroll
    for (int k = 0; k < kPer; ++k)
        if (base + 32 * k < n) out[base + 32 * k] = before + v[k];
    if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) *total = before + run;
}

__device__ __forceinline__ int find_root(int* parent, int a) {
    int p = parent[a];
    while (p != a) {
        int gp = parent[p];
        if (gp != p) parent[a] = gp;   // path halving; a benign race, every write is an ancestor
        a = p;
        p = parent[a];
    }
    return a;
}

__device__ void unite(int* parent, int a, int b) {
    while (true) {
        a = find_root(parent, a);
        b = find_root(parent, b);
        if (a == b) return;
        if (a < b) {
            int t = a;
            a = b;
            b = t;
        }
        // Hook the larger root under the smaller; retry if another thread moved it first.
        int old = atomicCAS(&parent[a], a, b);
        if (old == a) return;
    }
}

__global__ void k_cc_init(const uint8_t* __restrict__ mask, int* __restrict__ parent, size_t N) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        parent[i] = mask[i] ? (int)i : -1;
}

// Each edge once: east, south-west, south, south-east (x wraps, y stops).
__global__ void k_cc_union(const uint8_t* __restrict__ mask, int* __restrict__ parent, int W, int H) {
    size_t N = (size_t)W * H;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        if (!mask[i]) continue;
        const int row = pdiv((int)i, W), col = pmod((int)i, W);
        int e = row * W + wrap_col(col + 1, W);
        if (mask[e]) unite(parent, (int)i, e);
        if (row + 1 < H) {
            for (int cs = -1; cs <= 1; ++cs) {
                int n = (row + 1) * W + wrap_col(col + cs, W);
                if (mask[n]) unite(parent, (int)i, n);
            }
        }
    }
}

// Point every cell straight at its root. Read-only walks: the only writes are true roots, so a
// concurrent walk through a cell sees either its old ancestor or its root, both on the way up.
// (Path halving here would race: a halving write could replace a root just written with an
// intermediate ancestor.)
__global__ void k_cc_flatten(int* __restrict__ parent, size_t N) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        int p = parent[i];
        if (p < 0) continue;
        int a = (int)i;
        while (p != a) {
            a = p;
            p = parent[a];
        }
        parent[i] = a;
    }
}

__global__ void k_root_flags(const int* __restrict__ parent, int* __restrict__ flag, size_t N) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        flag[i] = parent[i] == (int)i ? 1 : 0;
}

__global__ void k_label_from_root(const int* __restrict__ parent, const int* __restrict__ rank,
                                  int* __restrict__ label, size_t N) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        int p = parent[i];
        label[i] = p < 0 ? -1 : rank[p];
    }
}

}  // namespace

cg_status read_back(cg_ctx* ctx, std::initializer_list<ReadBack> parts) {
    size_t total = 0;
    for (const ReadBack& p : parts) total += (p.bytes + 15) & ~(size_t)15;
    cg_status st = CG_OK;
    char* staging = (char*)pinned(ctx, std::max<size_t>(total, 256), &st);
    if (st != CG_OK) return st;
    size_t at = 0;
    for (const ReadBack& p : parts) {
        if (p.bytes) CG_CUDA(ctx, cudaMemcpyAsync(staging + at, p.dev, p.bytes, cudaMemcpyDeviceToHost, ctx->stream));
        at += (p.bytes + 15) & ~(size_t)15;
    }
    CG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    at = 0;
    for (const ReadBack& p : parts) {
        if (p.bytes) std::memcpy(p.host, staging + at, p.bytes);
        at += (p.bytes + 15) & ~(size_t)15;
    }
    return CG_OK;
}

// Two launches, the tiles' sums and the tiles, each CTA adding up the sums before its own: a level of
// block scans and a pass adding their offsets took four to six. A read of up to kScanDirect sums a CTA
// stays below the tile's own; longer inputs scan the sums first (at 8192 tiles the last pass takes 49 us
// adding the sums up, and 42 after two launches of 3 and 4 that scan them).
static cg_status scan_dev(cg_ctx* ctx, const int* d_in, int* d_out, int n, int** total) {
    if (n > 1 << 30) return fail(ctx, CG_BAD_ARG, "scan of %d elements is too long", n);
    const int tiles = (n + kScanTile - 1) / kScanTile;
    const int tiles2 = tiles > kScanDirect ? (tiles + kScanTile - 1) / kScanTile : 0;
    CG_BUF(int, d_tmp, ctx, S_SCRATCH5, 2 * (size_t)tiles + tiles2 + 1);
    int* d_total = d_tmp;
    int* d_sums = d_tmp + 1;
    int* d_offs = tiles2 ? d_sums + tiles : nullptr;
    if (tiles > 1) CG_LAUNCH(ctx) k_scan_sums<<<tiles, kScanThreads, 0, ctx->stream>>>(d_in, n, d_sums);
    if (tiles2) {
        int* d_sums2 = d_offs + tiles;
        CG_LAUNCH(ctx) k_scan_sums<<<tiles2, kScanThreads, 0, ctx->stream>>>(d_sums, tiles, d_sums2);
        CG_LAUNCH(ctx) k_scan_tiles<<<tiles2, kScanThreads, 0, ctx->stream>>>(d_sums, tiles, d_sums2, nullptr, d_offs,
                                                                              nullptr);
    }
    CG_LAUNCH(ctx) k_scan_tiles<<<tiles, kScanThreads, 0, ctx->stream>>>(d_in, n, d_sums, d_offs, d_out, d_total);
    CG_CHECK_LAUNCH(ctx);
    *total = d_total;
    return CG_OK;
}

cg_status exclusive_scan(cg_ctx* ctx, const int* d_in, int* d_out, int n, int* h_total) {
    if (n <= 0) {
        if (h_total) *h_total = 0;
        return CG_OK;
    }
    int* d_total = nullptr;
    CG_TRY_ST(scan_dev(ctx, d_in, d_out, n, &d_total));
    return h_total ? read_back(ctx, {{h_total, d_total, sizeof(int)}}) : CG_OK;
}

cg_status component_labels(cg_ctx* ctx, int W, int H, const uint8_t* d_mask, int* d_root, int* d_label,
                           int* h_count, ReadBack also) {
    size_t N = (size_t)W * H;
    int grid = ctx->num_sms * 8;
    CG_LAUNCH(ctx) k_cc_init<<<grid, 256, 0, ctx->stream>>>(d_mask, d_root, N);
    CG_LAUNCH(ctx) k_cc_union<<<grid, 256, 0, ctx->stream>>>(d_mask, d_root, W, H);
    CG_LAUNCH(ctx) k_cc_flatten<<<grid, 256, 0, ctx->stream>>>(d_root, N);
    CG_CHECK_LAUNCH(ctx);
    if (d_label) {
        CG_BUF(int, d_flag, ctx, S_SCRATCH0, N);
        CG_BUF(int, d_rank, ctx, S_SCRATCH1, N);
        CG_LAUNCH(ctx) k_root_flags<<<grid, 256, 0, ctx->stream>>>(d_root, d_flag, N);
        CG_CHECK_LAUNCH(ctx);
        int* d_total = nullptr;
        CG_TRY_ST(scan_dev(ctx, d_flag, d_rank, (int)N, &d_total));
        if (h_count) CG_TRY_ST(read_back(ctx, {{h_count, d_total, sizeof(int)}, also}));
        CG_LAUNCH(ctx) k_label_from_root<<<grid, 256, 0, ctx->stream>>>(d_root, d_rank, d_label, N);
        CG_CHECK_LAUNCH(ctx);
    }
    return CG_OK;
}

}  // namespace cg
