// terrain.cu -- LavaCA::applyTerrain (engine/src/ca/LavaCA.hpp:185-211) on the device: ROCK columns and
// the spill levels (TerrainGenerator::fillDepressions, engine/src/terrain/TerrainGenerator.cpp:86-161).
//
// The spill level of a column is the lowest level at which water standing on it runs off to an outlet:
// the minimum over all paths to an outlet of the highest column on the path.  It is the largest W with
// W = h at the outlets and W = max(h, min of the four neighbours' W) elsewhere, so any order of
// relaxations from W = infinity ends at it, and the reference's priority flood gives the same levels.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <vector>

#include "vca.h"
#include "vca_internal.h"

namespace vca {

constexpr int kFloodTile = 32;                            // tile side: a warp per row, a lane per column
constexpr int kFloodThreads = kFloodTile * kFloodTile;
constexpr int kFloodInf = INT_MAX;

struct FloodCtrl {
    unsigned bar;          // arrivals at the grid barrier
    unsigned error;        // a bounded wait or the bounded number of rounds ran out
    unsigned woken[3];     // tiles woken in round r at [r % 3]
    unsigned pad[3];
};

struct FloodArgs {
    const int32_t* h;
    int32_t* w;
    int nx, ny, px, py;
    int tx, ty;            // tiles
    uint8_t* wake[2];      // per tile: to be relaxed in round r at [r & 1]
    FloodCtrl* ctrl;
};

// W before the first round: the outlets (the non-periodic edges; on a fully wrapped map the lowest
// columns) at their height, infinity elsewhere.
__global__ void flood_init_kernel(const FloodArgs f, int lowest) {
    const int64_t n = (int64_t)f.nx * f.ny, stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool edges = (!f.px && f.nx > 1) || (!f.py && f.ny > 1);
    for (int64_t i = i0; i < n; i += stride) {
        const int y = (int)(i / f.nx), x = (int)(i - (int64_t)y * f.nx);
        const int h = f.h[i];
        const bool out = edges ? (!f.px && f.nx > 1 && (x == 0 || x == f.nx - 1)) || (!f.py && f.ny > 1 && (y == 0 || y == f.ny - 1))
                               : h == lowest;
        f.w[i] = out ? h : kFloodInf;
    }
    for (int64_t i = i0; i < (int64_t)f.tx * f.ty; i += stride) {
        f.wake[0][i] = 1;
        f.wake[1][i] = 0;
    }
    if (i0 == 0) *f.ctrl = FloodCtrl{};
}

// One direction of relaxation along a warp: lane i holds f_i(w) = max(a, min(b, w)) (a = height, b = its
// W so far), the value that reaches the first lane is `in`.  Such functions compose to functions of the
// same form, so a prefix scan of five shuffles relaxes the whole row: W_i = f_i(f_i-1(..f_0(in))).
template <bool kUp>
__device__ __forceinline__ int flood_scan(int a, int b, int in, int lane) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int pa = kUp ? __shfl_up_sync(0xFFFFFFFFu, a, off) : __shfl_down_sync(0xFFFFFFFFu, a, off);
        const int pb = kUp ? __shfl_up_sync(0xFFFFFFFFu, b, off) : __shfl_down_sync(0xFFFFFFFFu, b, off);
        if (kUp ? lane >= off : lane + off < 32) {
            const int na = max(a, min(b, pa)), nb = max(a, min(b, pb));
            a = na;
            b = nb;
        }
    }
    return max(a, min(b, in));
}

// Rounds of tile relaxations in one cooperative launch, a grid barrier after each.  A block takes its
// woken tiles in turn: rows left and right, columns up and down until nothing changes, then wakes the
// tiles beside a changed edge.  Bounded by the rounds the levels need to cross the map tile by tile
// (some 3 us each: a tile's scans and the barrier).  vca_ca_apply_terrain of a 1024 x 1024 map with the
// host's priority flood (one thread, random accesses) 28.5 ms, with these rounds 0.93 ms; 256 x 256
// 0.92 -> 0.10 ms.
__global__ __launch_bounds__(kFloodThreads, 1) void flood_kernel(const FloodArgs f) {
    __shared__ int s_w[kFloodTile][kFloodTile + 1];
    __shared__ unsigned s_edges, s_go;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tiles = f.tx * f.ty;
    for (int round = 0;; ++round) {
        uint8_t* wake = f.wake[round & 1];
        uint8_t* next = f.wake[(round & 1) ^ 1];
        unsigned woken = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            if (!__ldcg(wake + tile)) continue;  // uniform over the block
            const int tcx = tile % f.tx, tcy = tile / f.tx;
            const int x0 = tcx * kFloodTile, y0 = tcy * kFloodTile;
            auto at = [&](int x, int y) -> int64_t { return x + (int64_t)f.nx * y; };
            // the W of a column just outside the tile: through the frame when the axis wraps
            auto outside = [&](int x, int y) -> int {
                if (x < 0 || x >= f.nx) {
                    if (!f.px) return kFloodInf;
                    x = x < 0 ? f.nx - 1 : 0;
                }
                if (y < 0 || y >= f.ny) {
                    if (!f.py) return kFloodInf;
                    y = y < 0 ? f.ny - 1 : 0;
                }
                return __ldcg(f.w + at(x, y));
            };
            // row-wise: (x0 + lane, y0 + warp); column-wise: (x0 + warp, y0 + lane).  Columns past the map
            // are identities (a = -inf, b = inf), so the far edge's value passes through them.
            const int x = x0 + lane, y = y0 + warp;
            const bool in = x < f.nx && y < f.ny, inT = x0 + warp < f.nx && y0 + lane < f.ny;
            const int h = in ? f.h[at(x, y)] : INT_MIN;
            const int hT = inT ? f.h[at(x0 + warp, y0 + lane)] : INT_MIN;
            const int w0 = in ? __ldcg(f.w + at(x, y)) : kFloodInf;
            const int xe = min(x0 + kFloodTile, f.nx), ye = min(y0 + kFloodTile, f.ny);
            int left = kFloodInf, right = kFloodInf, top = kFloodInf, bottom = kFloodInf;
            if (lane == 0 && y < f.ny) left = outside(x0 - 1, y), right = outside(xe, y);
            if (lane == 0 && x0 + warp < f.nx) top = outside(x0 + warp, y0 - 1), bottom = outside(x0 + warp, ye);
            left = __shfl_sync(0xFFFFFFFFu, left, 0);
            right = __shfl_sync(0xFFFFFFFFu, right, 0);
            top = __shfl_sync(0xFFFFFFFFu, top, 0);
            bottom = __shfl_sync(0xFFFFFFFFu, bottom, 0);
            int w = w0;
            if (threadIdx.x == 0) s_edges = 0;
            bool again = true;
            for (int pass = 0; again && pass < 4096; ++pass) {
                const int before = w;
                w = flood_scan<true>(h, w, left, lane);
                w = flood_scan<false>(h, w, right, lane);
                s_w[warp][lane] = in ? w : kFloodInf;
                __syncthreads();
                int v = s_w[lane][warp];
                v = flood_scan<true>(hT, v, top, lane);
                v = flood_scan<false>(hT, v, bottom, lane);
                s_w[lane][warp] = v;
                __syncthreads();
                w = in ? s_w[warp][lane] : kFloodInf;
                again = __syncthreads_or(w != before) != 0;
            }
            if (threadIdx.x == 0) wake[tile] = 0;  // every thread has read it
            unsigned edges = again ? 16u : 0u;     // stopped early: once more in the next round
            if (in && w != w0) {
                f.w[at(x, y)] = w;
                if (x == x0) edges |= 1u;
                if (x == xe - 1) edges |= 2u;
                if (y == y0) edges |= 4u;
                if (y == ye - 1) edges |= 8u;
            }
            edges = __reduce_or_sync(0xFFFFFFFFu, edges);
            if (lane == 0 && edges) atomicOr(&s_edges, edges);
            __syncthreads();
            if (threadIdx.x < 5 && ((s_edges >> threadIdx.x) & 1u)) {
                int cx = tcx, cy = tcy;
                if (threadIdx.x == 0) --cx;
                if (threadIdx.x == 1) ++cx;
                if (threadIdx.x == 2) --cy;
                if (threadIdx.x == 3) ++cy;
                bool ok = true;
                if (cx < 0 || cx >= f.tx) ok = ok && f.px, cx = cx < 0 ? f.tx - 1 : 0;
                if (cy < 0 || cy >= f.ty) ok = ok && f.py, cy = cy < 0 ? f.ty - 1 : 0;
                if (ok) {
                    next[cx + f.tx * cy] = 1;
                    ++woken;
                }
            }
            __syncthreads();  // s_edges is used again
        }
        if (woken) atomicAdd(&f.ctrl->woken[round % 3], woken);
        // grid barrier (bounded); block 0 clears the counter of the round after next
        __syncthreads();
        if (threadIdx.x == 0) {
            FloodCtrl* c = f.ctrl;
            const unsigned target = (unsigned)(round + 1) * gridDim.x;
            bool ok = true;
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(&c->bar) : "memory");
            for (int spins = 0;; ++spins) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(&c->bar) : "memory");
                if (v >= target) break;
                if (spins > (1 << 26) || ((spins & 1023) == 1023 && *(volatile unsigned*)&c->error)) {
                    ok = false;
                    break;
                }
            }
            if (round >= (1 << 20)) ok = false;
            if (!ok) atomicOr(&c->error, 1u);
            s_go = ok && __ldcg(&c->woken[round % 3]) != 0;
            if (blockIdx.x == 0) c->woken[(round + 2) % 3] = 0;
        }
        __syncthreads();
        if (!s_go) return;
    }
}

// ROCK for z < h(x, y) (LavaCA::applyTerrain, LavaCA.hpp:185-194) and, for a slab, both levels seen from
// its layer 0.  A thread takes four columns and writes their words bottom up; the warp's words of a
// level lie together.
__global__ void ca_terrain_kernel(uint8_t* type, int32_t* heights, int32_t* spill, int nx, int ny, int nz, int P, int shift) {
    const int quads = (nx + 3) / 4;
    const int64_t n = (int64_t)quads * ny;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int y = (int)(i / quads), x = 4 * (int)(i - (int64_t)y * quads);
        int h[4], most = 0, least = nz;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            h[j] = 0;
            if (x + j < nx) {
                const int64_t c = x + j + (int64_t)nx * y;
                h[j] = heights[c] - shift;
                if (shift) spill[c] -= shift;
            }
            most = max(most, min(h[j], nz));
            least = min(least, h[j]);
        }
        uint8_t* col = type + x + (int64_t)P * y;
        const int64_t zs = (int64_t)P * ny;
        int z = 0;
        for (; z < least; ++z) *reinterpret_cast<uint32_t*>(col + zs * z) = 0x01010101u * kRock;
        for (; z < most; ++z)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (z < h[j]) col[zs * z + j] = kRock;
    }
}

// Whether the device floods a map of `cols` columns and tx x ty tiles: its time grows with the rounds, so
// with the tiles of the longer side (about 3 us each on 40), the host's with the columns (13 ns each on
// 28 us).  Measured calls, host / device: 48 x 48 57 / 58 us, 64 x 64 87 / 51, 128 x 128 297 / 87,
// 256 x 256 918 / 97, 1024 x 1024 28500 / 929; sections 2048 x 1 49 / 210, 9000 x 1 133 / 886.
constexpr bool flood_on_device(size_t cols, size_t tx, size_t ty) { return cols >= 2048 + 256 * (tx > ty ? tx : ty); }

vca_status terrain_apply(vca_ca* h, const int32_t* heights, int32_t lowest) {
    const CaGeom& g = h->geom;
    const size_t cols = (size_t)g.nx * g.ny;
    VCA_CUDA(cudaMemcpyAsync(h->heights_dev, heights, sizeof(int32_t) * cols, cudaMemcpyHostToDevice, h->stream));
    std::vector<int32_t> spill;
    FloodArgs f{};
    const size_t tx = (size_t)((g.nx + kFloodTile - 1) / kFloodTile), ty = (size_t)((g.ny + kFloodTile - 1) / kFloodTile);
    const size_t tiles = tx * ty;
    if (!flood_on_device(cols, tx, ty) || sizeof(FloodCtrl) + 2 * tiles > sizeof(uint32_t) * (size_t)h->chg_cap) {
        spill = fill_depressions(std::vector<int32_t>(heights, heights + cols), g.nx, g.ny, g.per[0] != 0, g.per[1] != 0);
        VCA_CUDA(cudaMemcpyAsync(h->spill, spill.data(), sizeof(int32_t) * cols, cudaMemcpyHostToDevice, h->stream));
    } else {
        f.h = h->heights_dev;
        f.w = h->spill;
        f.nx = g.nx;
        f.ny = g.ny;
        f.px = g.per[0];
        f.py = g.per[1];
        f.tx = (int)tx;
        f.ty = (int)ty;
        // scratch: a change list (4 bytes per cell up to 16 MB), empty between set-ups
        f.ctrl = reinterpret_cast<FloodCtrl*>(h->chg_list[0]);
        f.wake[0] = reinterpret_cast<uint8_t*>(f.ctrl + 1);
        f.wake[1] = f.wake[0] + tiles;
        const int grid = (int)std::min<size_t>(tiles, (size_t)h->sms);
        flood_init_kernel<<<h->sms * 4, 256, 0, h->stream>>>(f, lowest);
        VCA_CUDA(cudaGetLastError());
        void* args[] = {&f};
        VCA_CUDA(cudaLaunchCooperativeKernel((const void*)flood_kernel, grid, kFloodThreads, args, 0, h->stream));
        h->launches += 2;
    }
    const int quads = (g.nx + 3) / 4;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)quads * g.ny + 255) / 256, 148 * 16));
    ca_terrain_kernel<<<blocks, 256, 0, h->stream>>>(h->type[h->cur()], h->heights_dev, h->spill, g.nx, g.ny, g.nz, g.P,
                                                     h->slab ? h->slab_z0 : 0);
    VCA_CUDA(cudaGetLastError());
    h->launches += 1;
    FloodCtrl c{};
    if (f.ctrl) VCA_CUDA(cudaMemcpyAsync(&c, f.ctrl, sizeof(c), cudaMemcpyDeviceToHost, h->stream));
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    if (c.error) {
        set_error("vca_ca_apply_terrain: a bounded grid-barrier wait ran out");
        return VCA_ERR_TIMEOUT;
    }
    return VCA_OK;
}

}  // namespace vca
