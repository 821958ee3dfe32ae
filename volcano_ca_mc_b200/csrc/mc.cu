// mc.cu -- Potts Monte Carlo crystallisation with the checkerboard update on sm_100a, and the
// vca_mc_* half of the C ABI.
//
// One MCS (PottsMC::sweep -> sweepColors, engine/src/mc/PottsMC.cpp:451-533) is one launch per
// colour.  The domain cells of a colour are a compact list of global indices (built once, in
// globalIndex order, by a device stream compaction), so a colour pass touches only domain cells:
// per trial it reads the list entry, the cell's mobility and spin, and its neighbours' spins
// (shared with the neighbouring trials through L1/L2), and writes the spin when accepted.
// Cells of one colour are never neighbours in any variant (PottsMC.cpp:160-165), so the trials
// of a colour are independent and the order inside the pass does not matter.
//
// Acceptance is decided in integers: the reference accepts an uphill move when
// toUniform(r) < exp(-dE/kT), i.e. (r >> 11) * 2^-53 < p.  Scaling by 2^53 is exact, so this is
// (r >> 11) < ceil(p * 2^53); the thresholds are built on the host with the host's exp(), once
// per (unlikeBefore, unlikeAfter) pair, and the device compares 64-bit integers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "vca.h"
#include "vca_device.cuh"
#include "vca_internal.h"

namespace vca {

constexpr int kMcThreads = 256;
constexpr int kTableSide = 27;  // unlike counts 0..26

// Exact 32-bit division by a runtime divisor (n < 2^32): q = (c * n) >> 64 with c = ceil(2^64 / d).
struct FastDiv {
    uint32_t d;
    uint64_t c;
};
inline FastDiv make_fastdiv(uint32_t d) { return FastDiv{d, d <= 1 ? 0 : ~0ULL / d + 1}; }
__device__ __forceinline__ uint32_t fdiv(uint32_t n, FastDiv f) { return f.d <= 1 ? n : (uint32_t)__umul64hi(f.c, (uint64_t)n); }

struct McCtrl {
    uint32_t sweeps;
    uint32_t ticket;
    unsigned long long attempts;
    unsigned long long accepted;
    unsigned long long uphill;
    unsigned long long energy_acc;
    unsigned long long sweep_accepted;  // accepted in the running sweep
    unsigned long long bar_arrived;     // grid barrier of the cooperative launches: arrivals so far
                                        // (zero between launches)
    unsigned int cooling[4];            // mc_cooling_kernel: largest step, largest time, largest ~time
    int error;                          // bit 0: a bounded barrier wait ran out
    int pad;
};

struct McArgs {
    int nx, ny, nz;
    int per[3];
    FastDiv div_nx, div_ny;
    int parity_colors;
    int classes[3];
    uint64_t seed;
    FastMod q_mod;       // % Q (initial orientation)
    FastMod qm1_mod;     // % (Q - 1) (proposal)
    FastMod var_mod;     // % variants
    int variants;
    int32_t* spin;
    const uint32_t* list;
    const float* list_mob;
    const unsigned long long* table;  // 27 x 27 acceptance thresholds
    const NbTable* nb;
    McCtrl* ctrl;
    McCtrl* mirror;      // host-mapped: where a launch's last block leaves the control block
    // z slab of a taller grid (vca_mc_set_slab): hashRand takes local index + gidx_base, colours
    // the global z = local z + zoff
    uint64_t gidx_base;
    int zoff;
};

__device__ __forceinline__ bool mc_wrap(int& v, int n, int periodic) {
    if (v >= 0 && v < n) return true;
    if (!periodic || n == 1) return false;
    v = v < 0 ? v + n : v - n;
    return true;
}
// Spin of a neighbour through the frame: periodic copy or 0 (PottsMC::fillFrame, PottsMC.cpp:226-277).
__device__ __forceinline__ int32_t spin_at(const McArgs& a, int x, int y, int z) {
    if (!mc_wrap(x, a.nx, a.per[0]) || !mc_wrap(y, a.ny, a.per[1]) || !mc_wrap(z, a.nz, a.per[2])) return 0;
    return a.spin[(uint64_t)x + (uint64_t)a.nx * ((uint64_t)y + (uint64_t)a.ny * z)];
}

// unlikeBeforeAfter's neighbour counts (PottsMC.cpp:394-430, PottsMC.hpp:191-204) for the cell
// (x, y, z) and variant var, one neighbour after another through the frame (the per-colour launches).
__device__ __forceinline__ void nb_counts_loop(const McArgs& a, const NbTable& nb, int var, int x, int y, int z,
                                               int32_t cur, int32_t prop, int& in_dom, int& same_a, int& same_b) {
    in_dom = same_a = same_b = 0;
    const int cnt = nb.count[var];
    for (int k = 0; k < cnt; ++k) {
        const int32_t sj = spin_at(a, x + nb.off[var][k][0], y + nb.off[var][k][1], z + nb.off[var][k][2]);
        in_dom += sj != 0;
        same_a += sj == cur;
        same_b += sj == prop;
    }
}
__device__ __forceinline__ void stage_nb(const McArgs& a, NbTable& s_nb) {
    const int* src = reinterpret_cast<const int*>(a.nb);
    int* dst = reinterpret_cast<int*>(&s_nb);
    for (int i = threadIdx.x; i < (int)(sizeof(NbTable) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
}
static_assert(sizeof(NbTable) % sizeof(int) == 0, "NbTable is copied as ints");

// PottsMC::axisClass / colorOf (PottsMC.cpp:145-158), colour numbering of buildColors (173-193).
__host__ __device__ inline int axis_class(int c, int n, int periodic) {
    if (periodic && (n % 2) == 1 && c == n - 1) return 2;
    return c & 1;
}
__host__ __device__ inline int color_of(const McArgs& a, int x, int y, int z) {
    z += a.zoff;  // a slab colours by global z (its z axis is never periodic)
    if (a.parity_colors) return (x + y + z) & 1;
    const int cx = axis_class(x, a.nx, a.per[0]), cy = axis_class(y, a.ny, a.per[1]), cz = axis_class(z, a.nz, a.per[2]);
    return cx + a.classes[0] * (cy + a.classes[1] * cz);
}

__device__ __forceinline__ void decode(const McArgs& a, uint32_t g, int& x, int& y, int& z) {
    const uint32_t r = fdiv(g, a.div_nx);
    x = (int)(g - r * (uint32_t)a.nx);
    const uint32_t zz = fdiv(r, a.div_ny);
    y = (int)(r - zz * (uint32_t)a.ny);
    z = (int)zz;
}

// PottsMC::initialize (PottsMC.cpp:104-143): 1 + hashRand(seed, 0, g, McInit) % Q in the domain.
__device__ __forceinline__ int32_t mc_first(const McArgs& a, uint64_t prefix, uint64_t g) {
    return 1 + (int32_t)fast_mod(hash_salt(hash_index(prefix, g + a.gidx_base), kSaltMcInit), a.q_mod);
}

// A whole-space domain: every cell an orientation, four per thread.
__global__ void mc_init_all_kernel(const __grid_constant__ McArgs a, uint64_t n) {
    const uint64_t prefix = hash_prefix(a.seed, 0);
    const uint64_t quads = (n + 3) / 4;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < quads; i += (uint64_t)gridDim.x * blockDim.x) {
        int32_t s[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = mc_first(a, prefix, 4 * i + j);
        if (4 * i + 4 <= n) *reinterpret_cast<int4*>(a.spin + 4 * i) = make_int4(s[0], s[1], s[2], s[3]);
        else
            for (int j = 0; 4 * i + j < n; ++j) a.spin[4 * i + j] = s[j];
    }
}

// The colour lists (buildColors, PottsMC.cpp:194-223) in three launches.  A block takes a contiguous run
// of the space, 16 domain bytes per thread at a time: the first pass writes the orientations (0 outside
// the domain) and counts the run's cells of each colour; the second, one block, turns the counts into
// places (colour by colour, run by run); the third puts the cells there.  Within a run the order is the
// atomics'; the trials of a colour do not depend on it.  Bounded by the bytes: 2 per cell read and 4
// written.  vca_mc_initialize of 512 x 512 x 256 cells on one B200 against a count and a stream selection
// per colour: 401 K in the domain 1.89 -> 0.24 ms, a whole space (now without lists) 2.7 -> 0.25 ms;
// 256 x 256 x 128, 81 K 0.35 -> 0.07 ms.
constexpr int kRunCells = 16 * kMcThreads;  // cells of one step of a block
struct McRuns {
    const uint8_t* domain;
    uint64_t n;
    uint64_t per_block;      // cells of a block's run, a multiple of kRunCells
    int colors;
    uint32_t* counts;        // [color][block]: counts, then places
};
template <class F>
__device__ __forceinline__ void mc_each_domain_cell(const McRuns& r, F&& f) {
    const uint64_t lo = blockIdx.x * r.per_block, hi = min(lo + r.per_block, r.n);
    for (uint64_t base = lo + 16 * threadIdx.x; base < hi; base += kRunCells) {
        uint32_t w[4] = {0, 0, 0, 0};
        if (base + 16 <= r.n) {
            const uint4 v = *reinterpret_cast<const uint4*>(r.domain + base);
            w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
        } else {
            for (int j = 0; base + j < r.n; ++j) w[j >> 2] |= (uint32_t)r.domain[base + j] << (8 * (j & 3));
        }
        f(base, w);
    }
}
__global__ __launch_bounds__(kMcThreads) void mc_runs_count_kernel(const __grid_constant__ McArgs a, const __grid_constant__ McRuns r,
                                                                   int first) {
    __shared__ uint32_t s_cnt[28];
    if (threadIdx.x < 28) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t prefix = hash_prefix(a.seed, 0);
    mc_each_domain_cell(r, [&](uint64_t base, const uint32_t w[4]) {
        int32_t s[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            s[j] = 0;
            if (((w[j >> 2] >> (8 * (j & 3))) & 0xFFu) == 0) continue;
            if (first) s[j] = mc_first(a, prefix, base + j);
            int x, y, z;
            decode(a, (uint32_t)(base + j), x, y, z);
            atomicAdd(&s_cnt[color_of(a, x, y, z)], 1u);
        }
        if (!first) return;
        if (base + 16 <= r.n) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<int4*>(a.spin + base + 4 * q) = make_int4(s[4 * q], s[4 * q + 1], s[4 * q + 2], s[4 * q + 3]);
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (base + j < r.n) a.spin[base + j] = s[j];
        }
    });
    __syncthreads();
    if (threadIdx.x < r.colors) r.counts[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x] = s_cnt[threadIdx.x];
}
// Exclusive places of every (colour, block), and the colours' totals for the host (host-mapped).
__global__ __launch_bounds__(1024) void mc_runs_place_kernel(uint32_t* counts, int colors, int blocks, volatile uint32_t* totals) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_base = 0;
    for (int c = 0; c < colors; ++c) {
        __syncthreads();
        const uint32_t first = s_base;
        for (int b0 = 0; b0 < blocks; b0 += 1024) {
            const int b = b0 + threadIdx.x;
            uint32_t* at = counts + (uint64_t)c * blocks + b;
            const uint32_t v = b < blocks ? *at : 0u;
            uint32_t incl = v;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, off);
                if (lane >= off) incl += u;
            }
            __syncthreads();  // s_base and s_warp of the round before have been read
            if (lane == 31) s_warp[warp] = incl;
            __syncthreads();
            uint32_t before = s_base;
            for (int w = 0; w < warp; ++w) before += s_warp[w];
            if (b < blocks) *at = before + incl - v;
            __syncthreads();
            if (threadIdx.x == 1023) s_base = before + incl;
            __syncthreads();
        }
        if (threadIdx.x == 0) totals[c] = s_base - first;
    }
}
__global__ __launch_bounds__(kMcThreads) void mc_runs_list_kernel(const __grid_constant__ McArgs a, const __grid_constant__ McRuns r,
                                                                  const float* mob, uint32_t* list, float* list_mob) {
    __shared__ uint32_t s_at[28];
    if (threadIdx.x < r.colors) s_at[threadIdx.x] = r.counts[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x];
    __syncthreads();
    mc_each_domain_cell(r, [&](uint64_t base, const uint32_t w[4]) {
        if (!(w[0] | w[1] | w[2] | w[3])) return;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if (((w[j >> 2] >> (8 * (j & 3))) & 0xFFu) == 0) continue;
            const uint32_t g = (uint32_t)(base + j);
            int x, y, z;
            decode(a, g, x, y, z);
            const uint32_t at = atomicAdd(&s_at[color_of(a, x, y, z)], 1u);
            list[at] = g;
            if (mob != nullptr) list_mob[at] = mob[g];
        }
    });
}

// One colour of one MCS: colorTrials (PottsMC.cpp:394-448) for the list entries [0, count).
template <bool kMobility, bool kRandomNb>
__global__ __launch_bounds__(kMcThreads) void mc_color_kernel(McArgs a, const uint32_t* list, const float* list_mob,
                                                              uint64_t count, int last_color) {
    __shared__ unsigned long long s_table[kTableSide * kTableSide];
    __shared__ unsigned long long s_red[3][kMcThreads / 32];
    __shared__ bool s_last;
    __shared__ NbTable s_nb;
    for (int i = threadIdx.x; i < kTableSide * kTableSide; i += kMcThreads) s_table[i] = a.table[i];
    stage_nb(a, s_nb);
    __syncthreads();
    McCtrl* ctrl = a.ctrl;
    const uint32_t t = ctrl->sweeps;
    const uint64_t prefix = hash_prefix(a.seed, t);
    const NbTable& nb = s_nb;
    unsigned my_att = 0, my_acc = 0, my_up = 0;
    for (uint64_t j = blockIdx.x * (uint64_t)kMcThreads + threadIdx.x; j < count; j += (uint64_t)gridDim.x * kMcThreads) {
        const uint32_t g = list[j];
        const uint64_t h = hash_index(prefix, g + a.gidx_base);
        if (kMobility) {
            const uint64_t r = hash_salt(h, kSaltMcMobility);
            if (__dmul_rn((double)(r >> 11), 1.0 / 9007199254740992.0) >= (double)list_mob[j]) continue;
        }
        ++my_att;
        int var = 0;
        if (kRandomNb) var = (int)fast_mod(hash_salt(h, kSaltNeighborhood), a.var_mod);
        int x, y, z;
        decode(a, g, x, y, z);
        const int32_t cur = a.spin[g];
        int32_t prop = 1 + (int32_t)fast_mod(hash_salt(h, kSaltMcOrient), a.qm1_mod);
        if (prop >= cur) ++prop;
        int in_dom, same_a, same_b;
        nb_counts_loop(a, nb, var, x, y, z, cur, prop, in_dom, same_a, same_b);
        const int before = in_dom - same_a, after = in_dom - same_b;
        const unsigned long long e = s_table[before * kTableSide + after];
        bool accept;
        if (e >> 63) {
            accept = true;
        } else {
            accept = e != 0 && (hash_salt(h, kSaltMcAccept) >> 11) < e;
            my_up += accept ? 1u : 0u;
        }
        if (accept) {
            a.spin[g] = prop;
            ++my_acc;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned ra = __reduce_add_sync(0xFFFFFFFFu, my_att);
    const unsigned rc = __reduce_add_sync(0xFFFFFFFFu, my_acc);
    const unsigned ru = __reduce_add_sync(0xFFFFFFFFu, my_up);
    if (lane == 0) {
        s_red[0][warp] = ra;
        s_red[1][warp] = rc;
        s_red[2][warp] = ru;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long sa = 0, sc = 0, su = 0;
        for (int w = 0; w < kMcThreads / 32; ++w) {
            sa += s_red[0][w];
            sc += s_red[1][w];
            su += s_red[2][w];
        }
        if (sa) atomicAdd(&ctrl->attempts, sa);
        if (sc) {
            atomicAdd(&ctrl->accepted, sc);
            atomicAdd(&ctrl->sweep_accepted, sc);
        }
        if (su) atomicAdd(&ctrl->uphill, su);
        s_last = false;
        if (last_color) {
            __threadfence();
            s_last = atomicAdd(&ctrl->ticket, 1u) == gridDim.x - 1;
        }
    }
    __syncthreads();
    if (s_last && threadIdx.x == 0) {
        __threadfence();
        ctrl->ticket = 0;
        ctrl->sweeps = t + 1;   // ++sweeps_ (PottsMC.cpp:531)
        __threadfence();
    }
}

// Offsets (index 0: coordinate - 1, 1: the cell, 2: coordinate + 1, times `stride`) and presence of
// the two neighbours of coordinate c on an axis of n cells: wrapped on a periodic axis (a 2-cell axis
// sees its other cell on both sides), absent at the frame otherwise (PottsMC::fillFrame,
// PottsMC.cpp:226-277).
__device__ __forceinline__ void mc_axis_nb(int c, int n, int per, int64_t stride, int64_t o[3], bool k[3]) {
    const bool wrap = per && n > 1;
    o[0] = c > 0 ? -stride : (int64_t)(n - 1) * stride;
    o[1] = 0;
    o[2] = c < n - 1 ? stride : -(int64_t)(n - 1) * stride;
    k[0] = c > 0 || wrap;
    k[1] = true;
    k[2] = c < n - 1 || wrap;
}

// unlikeBeforeAfter's counts (PottsMC.cpp:394-430) of the cell g = (x, y, z) over the neighbours
// whose bit (dx + 1) + 3 (dy + 1) + 9 (dz + 1) is set in `mask` (the variant's neighbourhood), on one
// path for every cell: nine row addresses and three x offsets, wrapped on periodic axes, a missing
// neighbour (frame) read as `none`.  All loads of the cell go out together.  A neighbour counts as in
// the domain when its value is not `none` (orientations: 0 outside the domain; the byte copy of a
// whole-space domain: every existing cell).
template <typename T>
__device__ __forceinline__ void mc_count_block(const McArgs& a, const T* base, uint32_t g, int x, int y, int z, uint32_t mask,
                                               uint32_t none, uint32_t cur, uint32_t prop, int& in_dom, int& same_a,
                                               int& same_b) {
    int64_t ox[3], oy[3], oz[3];
    bool kx[3], ky[3], kz[3];
    mc_axis_nb(x, a.nx, a.per[0], 1, ox, kx);
    mc_axis_nb(y, a.ny, a.per[1], a.nx, oy, ky);
    mc_axis_nb(z, a.nz, a.per[2], (int64_t)a.nx * a.ny, oz, kz);
    const T* p = base + g;
    uint32_t sv[27];
#pragma unroll
    for (int dz = 0; dz < 3; ++dz)
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
            const T* r = p + oz[dz] + oy[dy];
            const bool rk = kz[dz] && ky[dy];
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                const int bit = dx + 3 * dy + 9 * dz;
                const bool k = rk && kx[dx] && ((mask >> bit) & 1u);
                sv[bit] = k ? (uint32_t)r[ox[dx]] : none;
            }
        }
    in_dom = same_a = same_b = 0;
#pragma unroll
    for (int bit = 0; bit < 27; ++bit) {
        if (bit == 13) continue;  // the cell itself
        in_dom += sv[bit] != none;
        same_a += sv[bit] == cur;
        same_b += sv[bit] == prop;
    }
}

// Colour classes of the domain list: colour c is list[off[c] .. off[c + 1]).  Thread i of the sweep
// launch (T threads) takes the entries off[c] + i + k T, k < rounds[c], of colour c; with `cached`
// set, each block keeps its threads' entries (and their mobilities) in shared memory for the whole
// launch, round r of the launch at [round0[c] + k] x kMcThreads.
struct McColors {
    int colors;
    int cached;
    int pre;           // cached and at most kPreRounds rounds per colour: draws computed a pass ahead
    int total_rounds;
    int rounds[28];
    int round0[28];
    uint64_t off[28];
    uint32_t mask[6];  // per variant: bit (dx + 1) + 3 (dy + 1) + 9 (dz + 1) of each neighbour
};

// Sum over a warp, largest over a warp.
__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, off);
    return v;
}
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
    for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_down_sync(0xFFFFFFFFu, v, off));
    return v;
}

// Grid barrier of the cooperative sweep launches, in two halves so that a block can do work of its
// own between them.  Arrive: after __syncthreads (the block's writes of the pass are ordered before
// it), thread 0 adds one arrival with release semantics.  Wait: thread 0 polls the count with
// acquire loads until every block has arrived `epoch` times, then __syncthreads.  The count only
// grows during a launch and is zeroed before it.  The wait is bounded; a block that gives up, or
// sees that another gave up, returns false (ctrl->error is then set).
__device__ __forceinline__ void mc_barrier_arrive(McCtrl* ctrl) {
    __syncthreads();
    if (threadIdx.x == 0 && gridDim.x > 1)
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;\n" ::"l"(&ctrl->bar_arrived) : "memory");
}
// Polls the count until it has reached `target`; 0 when it gave up.
__device__ __forceinline__ int mc_barrier_poll(McCtrl* ctrl, unsigned long long target) {
    for (int spins = 0;; ++spins) {
        unsigned long long v;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(&ctrl->bar_arrived) : "memory");
        if (v >= target) return 1;
        // (a look at the error flag costs a round trip of its own: now and then)
        if (spins > (1 << 26) || ((spins & 1023) == 1023 && *(volatile int*)&ctrl->error)) {
            atomicOr(&ctrl->error, 1);
            return 0;
        }
    }
}
__device__ bool mc_barrier_wait(McCtrl* ctrl, unsigned nblocks, unsigned long long epoch) {
    __shared__ int s_ok;
    if (nblocks == 1) return true;  // the __syncthreads of the arrival has done it
    if (threadIdx.x == 0) s_ok = mc_barrier_poll(ctrl, epoch * nblocks);
    __syncthreads();
    return s_ok != 0;
}

// One thread per block, after the block's last access to the control block's sums: true for the last block.
__device__ __forceinline__ bool mc_last_block(unsigned* ticket) {
    unsigned left;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n" : "=r"(left) : "l"(ticket) : "memory");
    return left == gridDim.x - 1u;
}
// What the last block of a sweep or energy launch does: the control block into host-mapped memory (a copy
// would queue behind other handles' downloads, a launch for it costs another 5 us), then the counters of
// one launch back to zero.  With the memsets before the launch and the second wait gone, a call of 5 MCS
// on 50^3 takes 0.125 ms instead of 0.137, vca_mc_get_info 1 us instead of 15.
__device__ __forceinline__ void mc_hand_over(const McArgs& a) {
    static_assert(sizeof(McCtrl) % sizeof(uint4) == 0, "copied as 16-byte words");
    McCtrl* ctrl = a.ctrl;
    ctrl->ticket = 0;
    ctrl->bar_arrived = 0;
    uint4 w[sizeof(McCtrl) / sizeof(uint4)];
#pragma unroll
    for (int i = 0; i < (int)(sizeof(w) / sizeof(w[0])); ++i) w[i] = __ldcg(reinterpret_cast<const uint4*>(ctrl) + i);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(w) / sizeof(w[0])); ++i) reinterpret_cast<uint4*>(a.mirror)[i] = w[i];
    ctrl->sweep_accepted = 0;
    ctrl->energy_acc = 0;
}

// The random draws of one trial (hashRand of its sweep and cell: mobility test, neighbourhood
// variant, proposed orientation, acceptance number), which do not depend on any orientation.
struct McDraws {
    bool attempt;     // passed the mobility test
    int var;          // neighbourhood variant
    int32_t prop_raw; // 1 + r % (Q - 1), before the skip over the current orientation
    uint64_t acc;     // hashRand(..., McAccept)
};
template <bool kMobility, bool kRandomNb>
__device__ __forceinline__ McDraws mc_draws(const McArgs& a, uint64_t prefix, uint32_t g, float mob) {
    McDraws d;
    const uint64_t h = hash_index(prefix, g + a.gidx_base);
    d.attempt = true;
    if (kMobility) {
        const uint64_t r = hash_salt(h, kSaltMcMobility);
        d.attempt = __dmul_rn((double)(r >> 11), 1.0 / 9007199254740992.0) < (double)mob;
    }
    d.var = kRandomNb ? (int)fast_mod(hash_salt(h, kSaltNeighborhood), a.var_mod) : 0;
    d.prop_raw = 1 + (int32_t)fast_mod(hash_salt(h, kSaltMcOrient), a.qm1_mod);
    d.acc = hash_salt(h, kSaltMcAccept);
    return d;
}

// `sweeps` checkerboard MCS in one cooperative launch: the colour classes in ascending order
// (sweepColors, PottsMC.cpp:495-514), a grid barrier after each, the same trial as mc_color_kernel
// (colorTrials, PottsMC.cpp:394-493).  Replaces `sweeps` x `colors` launches.  A colour pass costs
// the latency of its rounds: the entry and mobility come from shared memory (staged once per
// launch); the draws of the trial were computed while the block waited at the previous barrier
// (col.pre: kept in shared memory, one slot per thread and round); the cell's spin and all its
// neighbours' spins are loaded together (one round trip to L2), then the decision and the store.
constexpr int kPreRounds = 4;  // rounds per colour whose draws are computed ahead
template <bool kMobility, bool kRandomNb>
__global__ __launch_bounds__(kMcThreads, 2) void mc_sweeps_kernel(const __grid_constant__ McArgs a,
                                                                  const __grid_constant__ McColors col, int sweeps) {
    // [total_rounds][kMcThreads] entries, then mobilities; then with col.pre the draws of the next
    // pass: [kPreRounds][kMcThreads] acceptance numbers, proposals, flags (bit 7 attempt, variant)
    extern __shared__ __align__(16) uint32_t s_ent[];
    __shared__ unsigned long long s_table[kTableSide * kTableSide];
    __shared__ unsigned long long s_red[3][kMcThreads / 32];
    for (int i = threadIdx.x; i < kTableSide * kTableSide; i += kMcThreads) s_table[i] = a.table[i];
    const uint64_t T = (uint64_t)gridDim.x * kMcThreads;
    const uint64_t me = (uint64_t)blockIdx.x * kMcThreads + threadIdx.x;
    const size_t cache_words = (size_t)col.total_rounds * kMcThreads * (kMobility ? 2 : 1);
    float* s_mob = reinterpret_cast<float*>(s_ent + (size_t)col.total_rounds * kMcThreads);
    uint64_t* s_pacc = reinterpret_cast<uint64_t*>(s_ent + cache_words);
    int32_t* s_pprop = reinterpret_cast<int32_t*>(s_pacc + kPreRounds * kMcThreads);
    uint8_t* s_pflag = reinterpret_cast<uint8_t*>(s_pprop + kPreRounds * kMcThreads);
    if (col.cached) {
        for (int c = 0; c < col.colors; ++c)
            for (int k = 0; k < col.rounds[c]; ++k) {
                const uint64_t j = col.off[c] + me + (uint64_t)k * T;
                const int slot = (col.round0[c] + k) * kMcThreads + threadIdx.x;
                const bool in = j < col.off[c + 1];
                s_ent[slot] = in ? a.list[j] : 0xFFFFFFFFu;
                if (kMobility) s_mob[slot] = in ? a.list_mob[j] : 0.f;
            }
    }
    __syncthreads();
    McCtrl* ctrl = a.ctrl;
    const uint32_t t0 = ctrl->sweeps;
    // this thread's draws of pass (sweep s, colour c) into its slots (col.pre only)
    auto precompute = [&](int s, int c) {
        const uint64_t prefix = hash_prefix(a.seed, t0 + (uint32_t)s);
        for (int k = 0; k < col.rounds[c]; ++k) {
            const int slot = (col.round0[c] + k) * kMcThreads + threadIdx.x;
            const uint32_t g = s_ent[slot];
            if (g == 0xFFFFFFFFu) continue;
            const McDraws d = mc_draws<kMobility, kRandomNb>(a, prefix, g, kMobility ? s_mob[slot] : 0.f);
            const int ps = k * kMcThreads + threadIdx.x;
            s_pacc[ps] = d.acc;
            s_pprop[ps] = d.prop_raw;
            s_pflag[ps] = (uint8_t)((d.attempt ? 0x80 : 0) | d.var);
        }
    };
    unsigned long long my_att = 0, my_acc = 0, my_up = 0;
    bool ok = true;
    unsigned long long epoch = 0;  // grid barriers passed in this launch
    if (col.pre && sweeps > 0) precompute(0, 0);
    for (int s = 0; s < sweeps && ok; ++s) {
        const uint64_t prefix = hash_prefix(a.seed, t0 + (uint32_t)s);
        for (int c = 0; c < col.colors && ok; ++c) {
            for (int k = 0; k < col.rounds[c]; ++k) {
                uint32_t g;
                float mob = 0.f;
                if (col.cached) {
                    const int slot = (col.round0[c] + k) * kMcThreads + threadIdx.x;
                    g = s_ent[slot];
                    if (kMobility && !col.pre) mob = s_mob[slot];
                } else {
                    const uint64_t j = col.off[c] + me + (uint64_t)k * T;
                    g = j < col.off[c + 1] ? a.list[j] : 0xFFFFFFFFu;
                    if (kMobility && g != 0xFFFFFFFFu) mob = a.list_mob[j];
                }
                if (g == 0xFFFFFFFFu) continue;
                McDraws d;
                if (col.pre) {
                    const int ps = k * kMcThreads + threadIdx.x;
                    const unsigned f = s_pflag[ps];
                    d.attempt = (f & 0x80u) != 0;
                    d.var = (int)(f & 0x7Fu);
                    d.prop_raw = s_pprop[ps];
                    d.acc = s_pacc[ps];
                } else {
                    d = mc_draws<kMobility, kRandomNb>(a, prefix, g, mob);
                }
                if (!d.attempt) continue;
                ++my_att;
                const int var = d.var;
                int x, y, z;
                decode(a, g, x, y, z);
                const int32_t cur = a.spin[g];
                int32_t prop = d.prop_raw;
                if (prop >= cur) ++prop;
                int in_dom, same_a, same_b;
                mc_count_block(a, a.spin, g, x, y, z, col.mask[var], 0u, (uint32_t)cur, (uint32_t)prop, in_dom,
                                     same_a, same_b);
                const unsigned long long th = s_table[(in_dom - same_a) * kTableSide + (in_dom - same_b)];
                bool accept;
                if (th >> 63) {
                    accept = true;
                } else {
                    accept = th != 0 && (d.acc >> 11) < th;
                    my_up += accept ? 1u : 0u;
                }
                if (accept) {
                    a.spin[g] = prop;
                    ++my_acc;
                }
            }
            mc_barrier_arrive(ctrl);
            if (col.pre) {  // the next pass's draws while the other blocks finish this one
                const bool last_c = c + 1 == col.colors;
                if (!last_c) precompute(s, c + 1);
                else if (s + 1 < sweeps) precompute(s + 1, 0);
            }
            ok = mc_barrier_wait(ctrl, gridDim.x, ++epoch);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long ra = my_att, rc = my_acc, ru = my_up;
    for (int off = 16; off > 0; off >>= 1) {
        ra += __shfl_down_sync(0xFFFFFFFFu, ra, off);
        rc += __shfl_down_sync(0xFFFFFFFFu, rc, off);
        ru += __shfl_down_sync(0xFFFFFFFFu, ru, off);
    }
    if (lane == 0) {
        s_red[0][warp] = ra;
        s_red[1][warp] = rc;
        s_red[2][warp] = ru;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long sa = 0, sc = 0, su = 0;
        for (int w = 0; w < kMcThreads / 32; ++w) {
            sa += s_red[0][w];
            sc += s_red[1][w];
            su += s_red[2][w];
        }
        if (sa) atomicAdd(&ctrl->attempts, sa);
        if (sc) {
            atomicAdd(&ctrl->accepted, sc);
            atomicAdd(&ctrl->sweep_accepted, sc);
        }
        if (su) atomicAdd(&ctrl->uphill, su);
        // every block passed the last barrier, so no block reads ctrl->sweeps any more
        if (blockIdx.x == 0 && ok) ctrl->sweeps = t0 + (uint32_t)sweeps;
        if (mc_last_block(&ctrl->ticket)) mc_hand_over(a);
    }
}

// ------------------------------------------------------------------------------------------
// Whole-space domain (mc.domain = full, every cell a trial each MCS) with Q <= 256: the sweeps run on
// a one-byte copy of the orientations (orientation - 1, so 67 M cells take 69 MB and stay in L2).
//
// A thread takes the four cells of a colour among eight neighbouring x (every colour steps by two in x)
// and counts their unlike neighbours four bytes at a time: per row of the 3 x 3 x 3 block one aligned
// 8-byte load and one byte beside it give the left, middle and right neighbours of the four cells as
// three words; a byte of x = word ^ orientations is zero where the neighbour is alike, and x + 0x7f..
// has bit 7 set where it is not (Q <= 128).  The 26 words are added as one-bit numbers with bitwise
// adders, about half the operations of shifting each into a byte counter.
//
// The copy has rows of P8 bytes: 8 in front (the last one holds the orientation at x = nx - 1, the left
// neighbour of x = 0 on a wrapped axis), nx cells, the orientation at x = 0, and room for the last load.
// What bounds it: the integer ALU (84 % busy), three 64-bit hashes of a trial (two at kT = 0) above all.
// Per MCS on one B200 against a thread per cell with 26 byte loads and compares (709 instructions per
// trial): 512 x 512 x 256 Moore, Q = 64, kT = 0.5 1.80 -> 0.73 ms, the same von Neumann 1.88 -> 0.54 ms,
// 256 x 256 x 128 pentagonal 0.30 -> 0.16 ms, 100^3 Moore 38 -> 31 us.  Three resident blocks per SM
// instead of two (80 registers, spills) 0.85 ms; moving adds and shifts to the FMA pipe 0.89 ms.
// ------------------------------------------------------------------------------------------
// Threads of a block (kThreads): one block of 512 per SM where a colour has a group for each of their threads
// (half the arrivals at the barriers: 512 x 512 x 256, 10 MCS 7.95 -> 7.39 ms, 200^3 pentagonal, 40 MCS 6.24 ->
// 6.01), else blocks of 128, which reach more SMs (80^3 1.21 -> 1.02 ms, 120^3 1.66 -> 1.43; by 512 1.67, 1.66).
constexpr int kSpaceThreads = 512, kSpaceSmall = 128;
constexpr int kSpaceResident = 512;  // threads of an SM the registers are limited to
struct McSpace {
    uint8_t* sp;             // P8-byte rows: orientation - 1
    const float* mob;        // mobility of every cell (kMobility)
    int P8;
    int gx[3], g0[3];        // groups of 8 x per row that hold cells of x class c, the first one
    int xlo[3], xhi[3];      // x range of class c (its parity: c & 1)
    int cnt[3][3];           // per axis and class: coordinates of the class (y and z)
    FastDiv32 div_gx[3], div_cy[3];
    uint32_t qm1, qm1_inv, qm1_2p32;  // Q - 1, floor((2^32 - 1) / (Q - 1)), 2^32 mod (Q - 1)
    uint32_t mask[6];        // per variant: bit (dx + 1) + 3 (dy + 1) + 9 (dz + 1) of each neighbour
    int uphill;              // kT > 0: some uphill moves are accepted
};

// Coordinate i of class c on an axis of n cells split into `classes` classes (axisClass,
// PottsMC.cpp:145-151): every coordinate (1 class), c + 2 i (classes 0 and 1), the last cell (class 2
// of a periodic odd axis).
__device__ __forceinline__ int class_coord(int i, int c, int classes, int n) {
    return classes == 1 ? i : (c == 2 ? n - 1 : 2 * i + c);
}

// The byte copy of the orientations with its frame columns, and back.  A thread moves the cells of one
// group of eight.
__global__ void mc_pack8_kernel(const int32_t* spin, uint8_t* sp, int nx, int P8, uint64_t rows) {
    const int groups = P8 / 8 - 2;
    const uint64_t n = (uint64_t)groups * rows;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t row = i / (uint64_t)groups;
        const int x0 = 8 * (int)(i - row * (uint64_t)groups);
        const int32_t* from = spin + row * (uint64_t)nx;
        uint8_t* to = sp + row * (uint64_t)P8 + 8;
        uint32_t w[2] = {0, 0};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int x = x0 + j;
            // past the row: x = nx is the frame column
            const int32_t v = x < nx ? from[x] : from[0];
            w[j >> 2] |= (uint32_t)(uint8_t)(v - 1) << (8 * (j & 3));
        }
        *reinterpret_cast<uint2*>(to + x0) = make_uint2(w[0], w[1]);
        if (x0 == 0) to[-1] = (uint8_t)(from[nx - 1] - 1);
        if (x0 + 8 == nx) to[nx] = (uint8_t)(from[0] - 1);
    }
}
__global__ void mc_unpack8_kernel(const uint8_t* sp, int32_t* spin, int nx, int P8, uint64_t rows) {
    const int groups = P8 / 8 - 2;
    const uint64_t n = (uint64_t)groups * rows;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t row = i / (uint64_t)groups;
        const int x0 = 8 * (int)(i - row * (uint64_t)groups);
        const uint2 v = *reinterpret_cast<const uint2*>(sp + row * (uint64_t)P8 + 8 + x0);
        int32_t* to = spin + row * (uint64_t)nx + x0;
        int32_t o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (int32_t)(((j < 4 ? v.x : v.y) >> (8 * (j & 3))) & 0xFFu) + 1;
        if ((nx & 3) == 0 && x0 + 8 <= nx) {
            *reinterpret_cast<int4*>(to) = make_int4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<int4*>(to + 4) = make_int4(o[4], o[5], o[6], o[7]);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (x0 + j < nx) to[j] = o[j];
        }
    }
}

// x mod d for d <= 255 from the 32-bit halves: hi (2^32 mod d) + lo, each remainder below 2 d (the
// quotient is exact or one too small), is below 2^18; the last remainder is finished by one subtraction.
__device__ __forceinline__ uint32_t mod_q(const McSpace& d, uint64_t x) {
    auto rem = [&](uint32_t v) { return v - __umulhi(v, d.qm1_inv) * d.qm1; };
    const uint32_t r = rem(rem((uint32_t)(x >> 32)) * d.qm1_2p32 + rem((uint32_t)x));
    return min(r, r - d.qm1);
}

// Bitwise adders over words of one-bit numbers: sum and carry of three, of two.
__device__ __forceinline__ void add3(uint32_t a, uint32_t b, uint32_t c, uint32_t& sum, uint32_t& carry) {
    sum = a ^ b ^ c;
    carry = (a & b) | (c & (a | b));
}
__device__ __forceinline__ void add2(uint32_t a, uint32_t b, uint32_t& sum, uint32_t& carry) {
    sum = a ^ b;
    carry = a & b;
}
// Numbers of up to four bits, one per byte: bit 7 of each byte of w[i] is bit i (the other bits are unused).
struct Planes {
    uint32_t w[4];
};
// The nine inputs of a plane of the 3 x 3 x 3 block, given as sum and carry of each row.
__device__ __forceinline__ Planes add_rows(const uint32_t s[3], const uint32_t c[3]) {
    Planes p;
    uint32_t k2, x2, k4, k4b;
    add3(s[0], s[1], s[2], p.w[0], k2);
    add3(c[0], c[1], c[2], x2, k4);
    add2(k2, x2, p.w[1], k4b);
    add2(k4, k4b, p.w[2], p.w[3]);
    return p;
}
// The sum of three planes (up to 27) as one byte per number.
__device__ __forceinline__ uint32_t add_planes(const Planes& a, const Planes& b, const Planes& c) {
    uint32_t p0, p1, p2, p3, p4, c2, x, c4, c4b, y, c8, c8b, z, c16, c16b;
    add3(a.w[0], b.w[0], c.w[0], p0, c2);
    add3(a.w[1], b.w[1], c.w[1], x, c4);
    add2(x, c2, p1, c4b);
    add3(a.w[2], b.w[2], c.w[2], y, c8);
    add3(y, c4, c4b, p2, c8b);
    add3(a.w[3], b.w[3], c.w[3], z, c16);
    add3(z, c8, c8b, p3, c16b);
    p4 = c16 | c16b;
    return ((p0 >> 7) & 0x01010101u) | ((p1 >> 6) & 0x02020202u) | ((p2 >> 5) & 0x04040404u) | ((p3 >> 4) & 0x08080808u) |
           ((p4 >> 3) & 0x10101010u);
}

// kNb: 0 the whole 3 x 3 x 3 block (Moore), 1 the six faces (von Neumann), 2 by the variants' masks.
// kWide: Q > 128, so an orientation - 1 takes all eight bits of its byte.
template <bool kMobility, int kNb, bool kParity, bool kWide, int kThreads>
__global__ __launch_bounds__(kThreads, kSpaceResident / kThreads) void mc_space_sweeps_kernel(const __grid_constant__ McArgs a,
                                                                        const __grid_constant__ McSpace d, int sweeps) {
    __shared__ unsigned long long s_table[kTableSide * kTableSide];
    __shared__ unsigned long long s_red[3][kThreads / 32];
    for (int i = threadIdx.x; i < kTableSide * kTableSide; i += kThreads) {
        // (r >> 11) < th is r < th << 11 as long as that fits
        const unsigned long long th = a.table[i];
        s_table[i] = th >> 63 ? 1ull : (th >> 53 ? 2ull : th << 11);
    }
    __syncthreads();
    McCtrl* ctrl = a.ctrl;
    const uint32_t t0 = ctrl->sweeps;
    const uint32_t T = gridDim.x * kThreads, me = blockIdx.x * kThreads + threadIdx.x;
    const int colors = kParity ? 2 : a.classes[0] * a.classes[1] * a.classes[2];
    unsigned long long sum_att = 0, sum_acc = 0, sum_up = 0;
    uint32_t my_att = 0, my_acc = 0, my_up = 0;  // of one sweep

    struct Cells {              // the four cells of a thread in one pass
        int cx, gi, y, z, par;
        unsigned on;            // cells that attempt a change
        uint32_t prop;          // proposals before the skip over the cell's own orientation
        uint32_t nb[4];         // kNb == 2: byte j of nb[k]: bits 8 k .. 8 k + 7 of cell j's variant mask
        uint64_t acc[4];        // acceptance numbers
    };
    struct Rows {               // what the trials read: the nine rows' eight bytes and the byte beside them
        uint2 v[9];
        uint8_t by[9];
    };
    // The cells of index i of colour c.
    auto locate = [&](int c, uint64_t i, Cells& q) {
        int cx = 0, cy = 0, cz = 0;
        if (!kParity) {
            cx = c % a.classes[0];
            const int r = c / a.classes[0];
            cy = r % a.classes[1];
            cz = r / a.classes[1];
        }
        uint32_t ig, iy;
        const uint32_t r = fast_divmod((uint32_t)i, d.div_gx[cx], ig);
        const uint32_t iz = fast_divmod(r, d.div_cy[cy], iy);
        q.cx = cx;
        q.gi = (int)ig + d.g0[cx];
        q.y = kParity ? (int)iy : class_coord((int)iy, cy, a.classes[1], a.ny);
        q.z = kParity ? (int)iz : class_coord((int)iz, cz, a.classes[2], a.nz);
        q.par = kParity ? (c + q.y + q.z + a.zoff) & 1 : cx & 1;
    };
    // Their draws (hashRand of the sweep and cell; they depend on no orientation).
    auto draw = [&](uint64_t prefix, Cells& q) {
        q.on = 0;
        q.prop = 0;
        uint32_t vm[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int x = 8 * q.gi + q.par + 2 * j;
            const bool in = x >= d.xlo[q.cx] && x < d.xhi[q.cx];
            const uint32_t g = (uint32_t)(in ? x : 0) + (uint32_t)a.nx * ((uint32_t)q.y + (uint32_t)a.ny * (uint32_t)q.z);
            const uint64_t h = hash_index(prefix, g + a.gidx_base);
            bool on = in;
            if (kMobility) {
                const uint64_t rr = hash_salt(h, kSaltMcMobility);
                on = on && __dmul_rn((double)(rr >> 11), 1.0 / 9007199254740992.0) < (double)d.mob[g];
            }
            if (kNb == 2) vm[j] = d.mask[a.variants == 1 ? 0 : (int)fast_mod(hash_salt(h, kSaltNeighborhood), a.var_mod)];
            q.on |= (unsigned)on << j;
            q.prop |= mod_q(d, hash_salt(h, kSaltMcOrient)) << (8 * j);
            q.acc[j] = d.uphill ? hash_salt(h, kSaltMcAccept) : 0;
        }
        if (kNb == 2) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                q.nb[k] = ((vm[0] >> 8 * k) & 0xFFu) | (((vm[1] >> 8 * k) & 0xFFu) << 8) | (((vm[2] >> 8 * k) & 0xFFu) << 16) |
                          (((vm[3] >> 8 * k) & 0xFFu) << 24);
        }
    };
    // All loads of the trials in one round, a missing row of the frame as the cells' own.
    auto load = [&](const Cells& q, Rows& w) {
        const uint8_t* row = d.sp + ((uint64_t)q.y + (uint64_t)a.ny * q.z) * (uint64_t)d.P8 + 8 + 8 * q.gi;
        const int side = q.par ? 8 : -1;
        int64_t oy[3], oz[3];
        bool ky[3], kz[3];
        mc_axis_nb(q.y, a.ny, a.per[1], d.P8, oy, ky);
        mc_axis_nb(q.z, a.nz, a.per[2], (int64_t)d.P8 * a.ny, oz, kz);
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const int dy = i % 3, dz = i / 3;
            if (kNb == 1 && dy != 1 && dz != 1) continue;
            const uint8_t* p = row + (ky[dy] && kz[dz] ? oy[dy] + oz[dz] : 0);
            w.v[i] = *reinterpret_cast<const uint2*>(p);
            if (kNb != 1 || i == 4) w.by[i] = p[side];
        }
    };
    // The trials (colorTrials, PottsMC.cpp:394-493).
    auto trials_of = [&](const Cells& q, const Rows& rows, auto parity) {
        const int par = decltype(parity)::value < 0 ? q.par : decltype(parity)::value;
        if (!q.on) return;
        my_att += __popc(q.on);
        uint8_t* row = d.sp + ((uint64_t)q.y + (uint64_t)a.ny * q.z) * (uint64_t)d.P8 + 8 + 8 * q.gi;
        // rows that exist: bytes of ones
        const uint32_t wy[3] = {q.y > 0 || (a.per[1] && a.ny > 1) ? ~0u : 0u, ~0u, q.y < a.ny - 1 || (a.per[1] && a.ny > 1) ? ~0u : 0u};
        const uint32_t wz[3] = {q.z > 0 || (a.per[2] && a.nz > 1) ? ~0u : 0u, ~0u, q.z < a.nz - 1 || (a.per[2] && a.nz > 1) ? ~0u : 0u};
        // a frame that does not wrap: no left neighbour at x = 0, no right one at x = nx - 1
        uint32_t ml = 0xFFFFFFFFu, mr = 0xFFFFFFFFu;
        if (!a.per[0]) {
            if (q.gi == 0 && par == 0) ml = 0xFFFFFF00u;
            const int jr = a.nx - 1 - 8 * q.gi - par;
            if ((jr & 1) == 0 && jr >= 0 && jr < 8) mr &= ~(0xFFu << (4 * jr));
        }
        // left, middle and right neighbours of the four cells in row i
        auto words = [&](int i, uint32_t& left, uint32_t& mid, uint32_t& right) {
            const uint32_t by = rows.by[i];
            const uint32_t even = __byte_perm(rows.v[i].x, rows.v[i].y, 0x6420), odd = __byte_perm(rows.v[i].x, rows.v[i].y, 0x7531);
            left = par ? even : __byte_perm(odd, by, 0x2104);   // bytes by, odd 0 .. 2
            mid = par ? odd : even;
            right = par ? __byte_perm(even, by, 0x4321) : odd;  // bytes even 1 .. 3, by
        };
        uint32_t lw, cur, rw;
        words(4, lw, cur, rw);
        // the proposals skip their cell's orientation: + 1 where proposal >= orientation, byte by byte
        // (bit 7 of a - b with the borrow kept inside the byte, corrected where the top bits differ)
        uint32_t prop;
        {
            const uint32_t pr = q.prop, dif = (pr | 0x80808080u) - (cur & 0x7F7F7F7Fu);
            const uint32_t ge = (pr & ~cur) | (~(pr ^ cur) & dif);
            prop = pr + ((ge >> 7) & 0x01010101u);
        }
        // bit 7 of each byte: the neighbour of that cell is unlike `v` (m: 0 bytes for missing neighbours)
        auto unlike = [&](uint32_t w, uint32_t v, uint32_t m) -> uint32_t {
            const uint32_t x = (w ^ v) & m;
            return kWide ? ((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x : x + 0x7F7F7F7Fu;
        };
        Planes pa[3], pb[3];
#pragma unroll
        for (int dz = 0; dz < 3; ++dz) {
            uint32_t sa[3], ca[3], sb[3], cb[3];
#pragma unroll
            for (int dy = 0; dy < 3; ++dy) {
                sa[dy] = ca[dy] = sb[dy] = cb[dy] = 0;
                if (kNb == 1 && dy != 1 && dz != 1) continue;
                const int i = dy + 3 * dz;
                const bool self = i == 4;
                const uint32_t here = wy[dy] & wz[dz];
                uint32_t w[3] = {lw, 0, rw}, ua[3] = {0, 0, 0}, ub[3] = {0, 0, 0};
                if (!self && kNb == 1) w[1] = __byte_perm(rows.v[i].x, rows.v[i].y, par ? 0x7531 : 0x6420);
                if (!self && kNb != 1) words(i, w[0], w[1], w[2]);
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) {
                    if (self ? dx == 1 : kNb == 1 && dx != 1) continue;
                    const uint32_t m = dx == 0 ? ml & here : dx == 2 ? mr & here : here;
                    ua[dx] = unlike(w[dx], cur, m);
                    ub[dx] = unlike(w[dx], prop, m);
                    if (kNb == 2) {  // only the neighbours of the cell's variant
                        const int bit = dx + 3 * dy + 9 * dz;
                        const uint32_t of = q.nb[bit >> 3] << (7 - (bit & 7));
                        ua[dx] &= of;
                        ub[dx] &= of;
                    }
                }
                add3(ua[0], ua[1], ua[2], sa[dy], ca[dy]);
                add3(ub[0], ub[1], ub[2], sb[dy], cb[dy]);
            }
            pa[dz] = add_rows(sa, ca);
            pb[dz] = add_rows(sb, cb);
        }
        // unlike neighbours of the orientations and of the proposals, a byte per cell
        const uint32_t ua = add_planes(pa[0], pa[1], pa[2]), ub = add_planes(pb[0], pb[1], pb[2]);
        unsigned took = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!((q.on >> j) & 1u)) continue;
            // threshold << 11 (0: never), bit 0: not uphill, bit 1: uphill and always
            const unsigned long long th = s_table[((ua >> (8 * j)) & 0xFFu) * kTableSide + ((ub >> (8 * j)) & 0xFFu)];
            const bool free = ((uint32_t)th & 1u) != 0, accept = ((uint32_t)th & 3u) != 0 || q.acc[j] < th;
            my_up += accept && !free ? 1u : 0u;
            took |= (unsigned)accept << j;
        }
        if (!took) return;
        my_acc += __popc(took);
        if (8 * q.gi + 8 <= a.nx) {
            // the eight bytes are this thread's alone in this pass: one store
            const uint32_t m = ((took & 1u) | ((took & 2u) << 7) | ((took & 4u) << 14) | ((took & 8u) << 21)) * 0xFFu;
            const uint32_t now = (prop & m) | (cur & ~m), even = par ? lw : now, odd = par ? now : rw;
            *reinterpret_cast<uint2*>(row) = make_uint2(__byte_perm(even, odd, 0x5140), __byte_perm(even, odd, 0x7362));
        } else {  // the last group of a row: the byte behind the cells is a frame column
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if ((took >> j) & 1u) row[par + 2 * j] = (uint8_t)(prop >> (8 * j));
        }
        if (a.per[0]) {  // the frame columns
            if (q.gi == 0 && par == 0 && (took & 1u)) row[a.nx] = (uint8_t)prop;
            const int jr = a.nx - 1 - 8 * q.gi - par;
            if ((jr & 1) == 0 && jr >= 0 && jr < 8 && ((took >> (jr / 2)) & 1u)) row[-1 - 8 * q.gi] = (uint8_t)(prop >> (4 * jr));
        }
    };
    // (the parity of x is the pass's own unless the colours are checkerboard parities)
    auto trials = [&](const Cells& q, const Rows& rows) {
        if constexpr (kParity) trials_of(q, rows, std::integral_constant<int, -1>{});
        else if (q.par) trials_of(q, rows, std::integral_constant<int, 1>{});
        else trials_of(q, rows, std::integral_constant<int, 0>{});
    };
    auto total_of = [&](int c) -> uint64_t {
        int cx = 0, cy = 0, cz = 0;
        if (!kParity) {
            cx = c % a.classes[0];
            const int r = c / a.classes[0];
            cy = r % a.classes[1];
            cz = r / a.classes[1];
        }
        return (uint64_t)d.gx[cx] * (uint32_t)d.cnt[1][cy] * (uint32_t)d.cnt[2][cz];
    };

    bool ok = true;
    unsigned long long epoch = 0;
    // the first cells of the next pass are drawn while the other blocks finish this one
    Cells q;
    if (sweeps > 0 && me < total_of(0)) {
        locate(0, me, q);
        draw(hash_prefix(a.seed, t0), q);
    }
    for (int s = 0; s < sweeps && ok; ++s) {
        const uint64_t prefix = hash_prefix(a.seed, t0 + (uint32_t)s);
        for (int c = 0; c < colors && ok; ++c) {
            const uint64_t total = total_of(c);
            Rows rows;
            if (me < total) {
                load(q, rows);
                trials(q, rows);
            }
            for (uint64_t i = (uint64_t)me + T; i < total; i += T) {
                locate(c, i, q);
                load(q, rows);
                draw(prefix, q);  // while the rows arrive
                trials(q, rows);
            }
            mc_barrier_arrive(ctrl);
            const bool last = c + 1 == colors;
            const int nc = last ? 0 : c + 1;
            if ((!last || s + 1 < sweeps) && me < total_of(nc)) {
                locate(nc, me, q);
                draw(last ? hash_prefix(a.seed, t0 + (uint32_t)s + 1u) : prefix, q);
            }
            ok = mc_barrier_wait(ctrl, gridDim.x, ++epoch);
        }
        sum_att += my_att, sum_acc += my_acc, sum_up += my_up;
        my_att = my_acc = my_up = 0;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long ra = sum_att, rc = sum_acc, ru = sum_up;
    for (int off = 16; off > 0; off >>= 1) {
        ra += __shfl_down_sync(0xFFFFFFFFu, ra, off);
        rc += __shfl_down_sync(0xFFFFFFFFu, rc, off);
        ru += __shfl_down_sync(0xFFFFFFFFu, ru, off);
    }
    if (lane == 0) {
        s_red[0][warp] = ra;
        s_red[1][warp] = rc;
        s_red[2][warp] = ru;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long sa = 0, sc = 0, su = 0;
        for (int w = 0; w < kThreads / 32; ++w) {
            sa += s_red[0][w];
            sc += s_red[1][w];
            su += s_red[2][w];
        }
        if (sa) atomicAdd(&ctrl->attempts, sa);
        if (sc) {
            atomicAdd(&ctrl->accepted, sc);
            atomicAdd(&ctrl->sweep_accepted, sc);
        }
        if (su) atomicAdd(&ctrl->uphill, su);
        if (blockIdx.x == 0 && ok) ctrl->sweeps = t0 + (uint32_t)sweeps;
        if (mc_last_block(&ctrl->ticket)) mc_hand_over(a);
    }
}

// ------------------------------------------------------------------------------------------
// Listed domains (basalt) with Q <= 256 whose entries fit in shared memory: the same byte copy, written
// for the domain's cells alone when the launch starts.  A colour pass is a chain of latencies (the wait
// at the barrier, one round of loads, the decision, the store, the barrier's release), so everything
// that does not depend on an orientation is done while the block waits: the cell's address, its edges and
// its draws.  Which neighbours are in the domain never changes: 27 bits per entry, taken once per
// launch.  A row of three neighbours is an aligned word of eight (and a second for one cell in four) and a
// funnel shift; the unlike bits of the nine rows are added with bitwise adders and counted.
// Measured on one B200 against 27 loads of 32-bit orientations per trial: 401 K cells, 200 MCS of 8
// colours 7.04 -> 5.03 ms (3.1 us a pass, of which the release about 0.6 and the loads 1.0), 81 K cells,
// 100 MCS in four calls 2.73 -> 1.92 ms.
// ------------------------------------------------------------------------------------------
constexpr int kListThreads = 1024;                 // most threads of a block; one block per SM
constexpr size_t kListSmemMax = 200 * 1024;        // shared memory a block may spend on its entries
struct McBytes {
    uint8_t* sp;             // P8-byte rows: orientation - 1 of the domain's cells, frame columns as in McSpace
    uint32_t P8;
    uint32_t qm1, qm1_inv, qm1_2p32;  // as in McSpace
    int uphill;
};

template <bool kMobility, bool kRandomNb>
__global__ __launch_bounds__(kListThreads, 1) void mc_list_sweeps_kernel(const __grid_constant__ McArgs a,
                                                                         const __grid_constant__ McColors col,
                                                                         const __grid_constant__ McBytes b, int sweeps) {
    extern __shared__ __align__(16) uint32_t s_ent[];  // [total_rounds][threads]: cells, neighbour bits, mobilities
    __shared__ unsigned long long s_table[kTableSide * kTableSide];
    __shared__ unsigned long long s_sum[3];
    __shared__ int s_ok;
    // the last warp holds no entries: it arrives at the barriers and polls them while the others prepare
    const uint32_t B = blockDim.x - 32, tid = threadIdx.x;
    const bool poller = tid >= B;
    uint32_t* s_dom = s_ent + (size_t)col.total_rounds * B;
    float* s_mob = reinterpret_cast<float*>(s_dom + (size_t)col.total_rounds * B);
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    enum : uint32_t { X0 = 1, X1 = 2, Y0 = 4, Y1 = 8, Z0 = 16, Z1 = 32 };  // faces a cell lies on
    for (int i = tid; i < kTableSide * kTableSide; i += blockDim.x) {
        // (r >> 11) < th is r < th << 11 as long as that fits; 1: not uphill, 2: uphill and always
        const unsigned long long th = a.table[i];
        s_table[i] = th >> 63 ? 1ull : (th >> 53 ? 2ull : th << 11);
    }
    if (tid < 3) s_sum[tid] = 0;
    if (tid == 0) s_ok = 1;
    auto place = [&](uint32_t g, uint32_t& off, uint32_t& faces) {
        int x, y, z;
        decode(a, g, x, y, z);
        off = b.P8 * ((uint32_t)y + (uint32_t)a.ny * (uint32_t)z) + 8u + (uint32_t)x;
        faces = (x == 0 ? X0 : 0) | (x == a.nx - 1 ? X1 : 0) | (y == 0 ? Y0 : 0) | (y == a.ny - 1 ? Y1 : 0) |
                (z == 0 ? Z0 : 0) | (z == a.nz - 1 ? Z1 : 0);
    };
    auto put = [&](uint32_t off, uint32_t faces, uint8_t v) {
        b.sp[off] = v;
        if (a.per[0]) {  // the frame columns
            if (faces & X0) b.sp[off + (uint32_t)a.nx] = v;
            if (faces & X1) b.sp[off - (uint32_t)a.nx] = v;
        }
    };
    // this thread's entries: cell, neighbours in the domain, mobility; their bytes into the copy
    const uint64_t T = (uint64_t)gridDim.x * B, me = (uint64_t)blockIdx.x * B + tid;
    for (int c = 0; c < col.colors && !poller; ++c)
        for (int k = 0; k < col.rounds[c]; ++k) {
            const uint64_t j = col.off[c] + me + (uint64_t)k * T;
            const uint32_t slot = (uint32_t)(col.round0[c] + k) * B + tid;
            const uint32_t g = j < col.off[c + 1] ? a.list[j] : kNone;
            s_ent[slot] = g;
            if (g == kNone) continue;
            if (kMobility) s_mob[slot] = a.list_mob[j];
            int x, y, z;
            decode(a, g, x, y, z);
            int64_t ox[3], oy[3], oz[3];
            bool kx[3], ky[3], kz[3];
            mc_axis_nb(x, a.nx, a.per[0], 1, ox, kx);
            mc_axis_nb(y, a.ny, a.per[1], a.nx, oy, ky);
            mc_axis_nb(z, a.nz, a.per[2], (int64_t)a.nx * a.ny, oz, kz);
            uint32_t dom = 0;
#pragma unroll
            for (int i = 0; i < 27; ++i) {
                const bool in = kx[i % 3] && ky[i / 3 % 3] && kz[i / 9] && i != 13;
                const int32_t v = a.spin[in ? g + ox[i % 3] + oy[i / 3 % 3] + oz[i / 9] : (int64_t)g];
                dom |= (uint32_t)(in && v != 0) << i;
            }
            s_dom[slot] = dom;
            uint32_t off, faces;
            place(g, off, faces);
            put(off, faces, (uint8_t)(a.spin[g] - 1));
        }
    McCtrl* ctrl = a.ctrl;
    const uint32_t t0 = ctrl->sweeps;
    unsigned long long epoch = 0;
    bool ok = true;
    // mc_barrier_arrive and mc_barrier_wait with the thread of the last warp; `work` is done by the others
    auto barrier = [&](auto&& work) {
        __syncthreads();
        ++epoch;
        if (!poller) {
            work();
        } else if (tid == B && gridDim.x > 1) {
            asm volatile("red.release.gpu.global.add.u64 [%0], 1;\n" ::"l"(&ctrl->bar_arrived) : "memory");
            s_ok = mc_barrier_poll(ctrl, epoch * gridDim.x);
        }
        __syncthreads();
        ok = s_ok != 0;
    };
    barrier([] {});

    struct Trial {
        uint32_t off, faces, nb, prop;  // nb: the neighbours that count
        uint64_t acc;
        bool on;
    };
    auto prepare = [&](int s, int c, int k, Trial& q) {
        q.on = false;
        if (k >= col.rounds[c]) return;
        const uint32_t slot = (uint32_t)(col.round0[c] + k) * B + tid;
        const uint32_t g = s_ent[slot];
        if (g == kNone) return;
        const uint64_t h = hash_index(hash_prefix(a.seed, t0 + (uint32_t)s), g);
        if (kMobility) {
            const uint64_t r = hash_salt(h, kSaltMcMobility);
            if (__dmul_rn((double)(r >> 11), 1.0 / 9007199254740992.0) >= (double)s_mob[slot]) return;
        }
        q.on = true;
        const int var = kRandomNb ? (int)fast_mod(hash_salt(h, kSaltNeighborhood), a.var_mod) : 0;
        q.nb = s_dom[slot] & col.mask[var];
        const uint64_t o = hash_salt(h, kSaltMcOrient);
        auto rem = [&](uint32_t v) { return v - __umulhi(v, b.qm1_inv) * b.qm1; };  // below 2 (Q - 1), as in mod_q
        const uint32_t r = rem(rem((uint32_t)(o >> 32)) * b.qm1_2p32 + rem((uint32_t)o));
        q.prop = min(r, r - b.qm1);
        q.acc = b.uphill ? hash_salt(h, kSaltMcAccept) : 0;
        place(g, q.off, q.faces);
    };
    uint32_t my_att = 0, my_acc = 0, my_up = 0;  // of one sweep
    unsigned long long sum_att = 0, sum_acc = 0, sum_up = 0;
    const uint32_t zs = b.P8 * (uint32_t)a.ny;
    auto trial = [&](const Trial& q) {
        if (!q.on) return;
        ++my_att;
        // offsets of the rows at y - 1, y + 1, z - 1, z + 1 through the frame (a missing row: the cell's own,
        // whose bits are not in q.nb)
        const uint32_t ym = q.faces & Y0 ? (a.per[1] ? b.P8 * (uint32_t)(a.ny - 1) : 0u) : 0u - b.P8;
        const uint32_t yp = q.faces & Y1 ? (a.per[1] ? 0u - b.P8 * (uint32_t)(a.ny - 1) : 0u) : b.P8;
        const uint32_t zm = q.faces & Z0 ? (a.per[2] ? zs * (uint32_t)(a.nz - 1) : 0u) : 0u - zs;
        const uint32_t zp = q.faces & Z1 ? (a.per[2] ? 0u - zs * (uint32_t)(a.nz - 1) : 0u) : zs;
        // a row's three bytes lie in one aligned word of eight for three cells in four
        const uint32_t at = (q.off - 1u) & ~7u, sh = 8u * ((q.off - 1u) & 7u);
        const bool over = sh >= 48u;
        uint2 w[9];
        uint32_t v[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const uint32_t dy = i % 3 == 0 ? ym : i % 3 == 2 ? yp : 0u, dz = i / 3 == 0 ? zm : i / 3 == 2 ? zp : 0u;
            const uint8_t* p = b.sp + (at + dy + dz);
            w[i] = *reinterpret_cast<const uint2*>(p);
            v[i] = over ? *reinterpret_cast<const uint32_t*>(p + 8) : 0u;
        }
#pragma unroll
        for (int i = 0; i < 9; ++i)  // bytes: x - 1, x, x + 1
            v[i] = sh >= 32u ? __funnelshift_r(w[i].y, v[i], sh) : __funnelshift_r(w[i].x, w[i].y, sh);
        const uint32_t cur = (v[4] >> 8) & 0xFFu, prop = q.prop + (q.prop >= cur ? 1u : 0u);
        const uint32_t cur3 = cur * 0x010101u, prop3 = prop * 0x010101u;
        uint32_t ua[9], ub[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const uint32_t m = ((((q.nb >> (3 * i)) & 7u) * 0x4081u) & 0x10101u) << 7;  // bit 7 of the counted bytes
            const uint32_t xa = v[i] ^ cur3, xb = v[i] ^ prop3;
            ua[i] = (((xa & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | xa) & m;
            ub[i] = (((xb & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | xb) & m;
        }
        auto total = [](const uint32_t u[9]) -> uint32_t {
            uint32_t sm[3], cy[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) add3(u[3 * i], u[3 * i + 1], u[3 * i + 2], sm[i], cy[i]);
            const Planes p = add_rows(sm, cy);
            return __popc(p.w[0]) + 2 * __popc(p.w[1]) + 4 * __popc(p.w[2]) + 8 * __popc(p.w[3]);
        };
        const unsigned long long th = s_table[total(ua) * kTableSide + total(ub)];
        const bool accept = ((uint32_t)th & 3u) != 0 || q.acc < th;
        if (accept) {
            put(q.off, q.faces, (uint8_t)prop);
            ++my_acc;
            my_up += ((uint32_t)th & 1u) ? 0u : 1u;
        }
    };
    Trial q;
    q.on = false;
    if (!poller) prepare(0, 0, 0, q);
    for (int s = 0; s < sweeps && ok; ++s) {
        for (int c = 0; c < col.colors && ok; ++c) {
            trial(q);
            for (int k = 1; k < col.rounds[c] && !poller; ++k) {
                prepare(s, c, k, q);
                trial(q);
            }
            const bool last = c + 1 == col.colors;
            barrier([&] {
                q.on = false;
                if (!last || s + 1 < sweeps) prepare(last ? s + 1 : s, last ? 0 : c + 1, 0, q);
            });
        }
        sum_att += my_att, sum_acc += my_acc, sum_up += my_up;
        my_att = my_acc = my_up = 0;
    }
    // the entries' orientations back
    for (int r = 0; r < col.total_rounds && !poller; ++r) {
        const uint32_t g = s_ent[(uint32_t)r * B + tid];
        if (g == kNone) continue;
        uint32_t off, faces;
        place(g, off, faces);
        a.spin[g] = (int32_t)b.sp[off] + 1;
    }
    const unsigned long long ra = warp_sum(sum_att), rc = warp_sum(sum_acc), ru = warp_sum(sum_up);
    if ((tid & 31) == 0) {
        if (ra) atomicAdd(&s_sum[0], ra);
        if (rc) atomicAdd(&s_sum[1], rc);
        if (ru) atomicAdd(&s_sum[2], ru);
    }
    __syncthreads();
    if (tid == 0) {
        if (s_sum[0]) atomicAdd(&ctrl->attempts, s_sum[0]);
        if (s_sum[1]) {
            atomicAdd(&ctrl->accepted, s_sum[1]);
            atomicAdd(&ctrl->sweep_accepted, s_sum[1]);
        }
        if (s_sum[2]) atomicAdd(&ctrl->uphill, s_sum[2]);
        // every block passed the last barrier, so no block reads ctrl->sweeps any more
        if (blockIdx.x == 0 && ok) ctrl->sweeps = t0 + (uint32_t)sweeps;
        if (mc_last_block(&ctrl->ticket)) mc_hand_over(a);
    }
}

// PottsMC::totalEnergy (PottsMC.cpp:590-664): unlike pairs.  Deterministic neighbourhoods count
// each pair once through the forward offsets; random ones sum E_i over the cells with the
// variant of MCS t (the caller halves it).  Bounded by the launch and the wait for it: the neighbours of a
// cell are loaded together.  One after another through the neighbourhood's table a call for 50^3 Moore took
// 24 us, for 401 K listed pentagonal cells 47; now 18 and 31.
struct McMasks {
    uint32_t of[6];  // per variant: bit (dx + 1) + 3 (dy + 1) + 9 (dz + 1) of each neighbour
};
template <bool kForward>
__global__ __launch_bounds__(kMcThreads) void mc_energy_kernel(const __grid_constant__ McArgs a, const __grid_constant__ McMasks m,
                                                               const uint32_t* list, uint64_t count) {
    __shared__ unsigned long long s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    const uint64_t prefix = hash_prefix(a.seed, a.ctrl->sweeps);
    unsigned long long mine = 0;
    for (uint64_t j = blockIdx.x * (uint64_t)kMcThreads + threadIdx.x; j < count; j += (uint64_t)gridDim.x * kMcThreads) {
        const uint32_t g = list ? list[j] : (uint32_t)j;  // no list: the whole space in order
        int x, y, z;
        decode(a, g, x, y, z);
        const int32_t s = a.spin[g];
        int var = 0;
        if (!kForward && a.variants > 1)
            var = (int)fast_mod(hash_salt(hash_index(prefix, g + a.gidx_base), kSaltNeighborhood), a.var_mod);
        const uint32_t mask = m.of[var];
        int64_t ox[3], oy[3], oz[3];
        bool kx[3], ky[3], kz[3];
        mc_axis_nb(x, a.nx, a.per[0], 1, ox, kx);
        mc_axis_nb(y, a.ny, a.per[1], a.nx, oy, ky);
        mc_axis_nb(z, a.nz, a.per[2], (int64_t)a.nx * a.ny, oz, kz);
        const uint32_t dx[3] = {(uint32_t)ox[0], 0u, (uint32_t)ox[2]}, dy[3] = {(uint32_t)oy[0], 0u, (uint32_t)oy[2]},
                       dz[3] = {(uint32_t)oz[0], 0u, (uint32_t)oz[2]};  // (below 2^32 cells)
        int32_t v[27];
#pragma unroll
        for (int i = kForward ? 14 : 0; i < 27; ++i) {
            v[i] = 0;
            if (i != 13 && ((mask >> i) & 1u) && kx[i % 3] && ky[i / 3 % 3] && kz[i / 9])
                v[i] = a.spin[g + dx[i % 3] + dy[i / 3 % 3] + dz[i / 9]];
        }
        int unlike = 0;
#pragma unroll
        for (int i = kForward ? 14 : 0; i < 27; ++i)
            if (i != 13 && ((mask >> i) & 1u)) unlike += (int)(v[i] != 0) - (int)(v[i] == s);
        mine += (unsigned long long)unlike;
    }
    for (int off = 16; off > 0; off >>= 1) mine += __shfl_down_sync(0xFFFFFFFFu, mine, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, mine);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_sum) atomicAdd(&a.ctrl->energy_acc, s_sum);
        if (mc_last_block(&a.ctrl->ticket)) mc_hand_over(a);
    }
}

// ------------------------------------------------------------------------------------------
// Grain statistics on the device (labelGrains, engine/src/mc/Grains.cpp:33-150; the majority
// classes by mobility of McStage, engine/src/app/McStage.cpp:38-66).  A grain is a connected set
// of domain cells of one orientation (von Neumann or Moore connectivity, periodic axes joined).
// Lock-free union-find over the domain list: a root is only ever linked to a smaller root by
// compare-and-swap, so parents only decrease and every loop ends; the components do not depend on
// the order of the unions.  Loops are bounded anyway; running out sets an error flag.
// ------------------------------------------------------------------------------------------
struct GrainAcc {
    unsigned long long grains, cells, largest, high_cells;
    unsigned long long high_grains, high_in, high_largest, low_grains, low_in, low_largest;
    unsigned int error;
    unsigned int left;     // blocks that have added their sums
};

__device__ __forceinline__ uint32_t gr_find(uint32_t* parent, uint32_t x, unsigned* err) {
    for (int i = 0; i < (1 << 24); ++i) {
        const uint32_t p = parent[x];
        if (p == x) return x;
        const uint32_t gp = parent[p];
        if (gp != p) parent[x] = gp;  // path halving: gp is an ancestor of x, so the write is benign
        x = gp;
    }
    atomicOr(err, 1u);
    return x;
}

__device__ __forceinline__ void gr_union(uint32_t* parent, uint32_t a, uint32_t b, unsigned* err) {
    for (int i = 0; i < (1 << 20); ++i) {
        uint32_t ra = gr_find(parent, a, err), rb = gr_find(parent, b, err);
        if (ra == rb) return;
        if (ra > rb) {
            const uint32_t t = ra;
            ra = rb;
            rb = t;
        }
        if (atomicCAS(&parent[rb], rb, ra) == rb) return;  // rb was still a root: linked under ra
        a = ra;
        b = rb;
    }
    atomicOr(err, 1u);
}

// Threads of a block of the grain pass: its grid barriers cost an arrival per block, so fewer and larger blocks
// are faster until they leave SMs without one.  50^3 after 90 MCS, by 256 / 512 / 1024 threads: 64 / 52 / 52 us
// a call; 128^3 456 / 390 / 356; 30^3 40 / 42 / 43; 81 K listed cells 45 / 46 / 55.
constexpr int kGrainThreads = 512;

// All passes in one cooperative launch (a grid barrier after each): every cell under its run in x; unions
// over the forward offsets of the connectivity (dz, dy, dx order) on the axes of size > 1; sizes and high
// cells per root; the statistics, summed per block before they reach the counters.  The last block hands
// them to the host (out: host-mapped).  With a few 10^5 cells the four passes are latencies; separate
// launches with an atomic per thread and counter took 2.05 ms a call for 401 K cells and 0.18 ms for 50^3,
// this one 0.088 and 0.052 ms (0.035 before the first sweep: what is left grows with the unions).
__global__ __launch_bounds__(kGrainThreads) void mc_grains_kernel(const __grid_constant__ McArgs a, const uint32_t* list,
                                                               uint64_t count, int moore, const float* mob, double threshold,
                                                               uint32_t* parent, uint32_t* gsize, uint32_t* ghigh, GrainAcc* acc,
                                                               GrainAcc* out) {
    const uint64_t i0 = blockIdx.x * (uint64_t)kGrainThreads + threadIdx.x, T = (uint64_t)gridDim.x * kGrainThreads;
    const int lane = threadIdx.x & 31;
    // a cell starts under the first cell of its run of one orientation in x, as far as the warp (in cell
    // order) or four cells (a list) show it; rows that wrap are united below
    for (uint64_t base = i0 - lane; base < count; base += T) {  // uniform over the warp
        const uint64_t j = base + lane;
        const uint32_t g = j < count ? (list ? list[j] : (uint32_t)j) : 0u;
        const uint32_t x = g % (uint32_t)a.nx;
        const int32_t sg = a.spin[g];
        uint32_t back = 0;
        if (list) {
            uint32_t same = 0;
#pragma unroll
            for (uint32_t i = 1; i <= 4; ++i) same |= (uint32_t)(x >= i && a.spin[x >= i ? g - i : g] == sg) << i;
            while ((same >> (back + 1)) & 1u) ++back;
        } else {
            const bool on = x != 0 && a.spin[x != 0 ? g - 1u : g] == sg;
            const unsigned heads = ~__ballot_sync(0xFFFFFFFFu, on) & (0xFFFFFFFFu >> (31 - lane));
            back = heads ? lane - (31 - __clz(heads)) : lane + 1;
        }
        if (j < count) {
            parent[g] = g - back;
            gsize[g] = 0;
            ghigh[g] = 0;
        }
    }
    mc_barrier_arrive(a.ctrl);
    if (!mc_barrier_wait(a.ctrl, gridDim.x, 1)) return;
    for (uint64_t j = i0; j < count; j += T) {
        const uint32_t g = list ? list[j] : (uint32_t)j;
        const int32_t sg = a.spin[g];
        if (sg <= 0) continue;
        int x, y, z;
        decode(a, g, x, y, z);
        // the forward neighbours and the left one, all loads together: bit i alike
        int64_t ox[3], oy[3], oz[3];
        bool kx[3], ky[3], kz[3];
        mc_axis_nb(x, a.nx, a.per[0], 1, ox, kx);
        mc_axis_nb(y, a.ny, a.per[1], a.nx, oy, ky);
        mc_axis_nb(z, a.nz, a.per[2], (int64_t)a.nx * a.ny, oz, kz);
        auto at = [&](int i) -> int64_t { return (int64_t)g + ox[i % 3] + oy[i / 3 % 3] + oz[i / 9]; };
        uint32_t alike = 0;
#pragma unroll
        for (int i = 12; i < 27; ++i) {
            if (i == 13) continue;
            const bool in = kx[i % 3] && ky[i / 3 % 3] && kz[i / 9];
            const int32_t v = a.spin[in ? at(i) : (int64_t)g];
            alike |= (uint32_t)(in && v == sg) << i;
        }
        // of a row's three only the unions that no other cell's give: the row's cells hang together, and
        // what the left (right) neighbour shares with the row it unites itself
        // (the first cell of a row that wraps unites for itself, or a ring would leave it to nobody)
        const bool left = ((alike >> 12) & 1u) && x > 0, right = (alike >> 14) & 1u;
        uint32_t todo = right && x == a.nx - 1 ? 1u << 14 : 0u;
#pragma unroll
        for (int row = 5; row < 9; ++row) {
            if (!moore && row != 5 && row != 7) continue;  // (y + 1, z) or (y, z + 1)
            const uint32_t r = alike >> (3 * row);
            const bool l = r & 1u, m = r & 2u, n = r & 4u;
            if (m && !(left && l)) todo |= 2u << (3 * row);
            if (moore && l && !m && !left) todo |= 1u << (3 * row);
            if (moore && n && !m && !right) todo |= 4u << (3 * row);
        }
        for (; todo; todo &= todo - 1) {
            const int i = __ffs(todo) - 1;
            const int dx = i % 3, dy = i / 3 % 3, dz = i / 9;
            const int64_t q = (int64_t)g + (dx == 0 ? ox[0] : dx == 2 ? ox[2] : 0) + (dy == 0 ? oy[0] : dy == 2 ? oy[2] : 0) +
                              (dz == 2 ? oz[2] : 0);
            gr_union(parent, g, (uint32_t)q, &acc->error);
        }
    }
    mc_barrier_arrive(a.ctrl);
    if (!mc_barrier_wait(a.ctrl, gridDim.x, 2)) return;
    unsigned long long cells = 0, high = 0;
    for (uint64_t base = i0 - lane; base < count; base += T) {  // uniform over the warp
        const uint64_t j = base + lane;
        const uint32_t g = j < count ? (list ? list[j] : (uint32_t)j) : 0u;
        const bool on = j < count && a.spin[g] > 0;
        uint32_t r = 0xFFFFFFFFu;
        bool up = false;
        if (on) {
            r = gr_find(parent, g, &acc->error);
            parent[g] = r;
            up = mob != nullptr && (double)mob[g] >= threshold;
            ++cells;
            high += up;
        }
        // one addition per root among the warp's cells (the cells of a large grain lie together)
        const unsigned same = __match_any_sync(0xFFFFFFFFu, r), ups = __ballot_sync(0xFFFFFFFFu, up);
        if (on && lane == __ffs(same) - 1) {
            atomicAdd(&gsize[r], (unsigned)__popc(same));
            if (same & ups) atomicAdd(&ghigh[r], (unsigned)__popc(same & ups));
        }
    }
    mc_barrier_arrive(a.ctrl);
    if (!mc_barrier_wait(a.ctrl, gridDim.x, 3)) return;
    unsigned long long v[5] = {0, 0, 0, 0, 0};  // grains; high ones, their cells; low ones, their cells
    unsigned long long largest = 0, hl = 0, ll = 0;
    for (uint64_t j = i0; j < count; j += T) {
        const uint32_t g = list ? list[j] : (uint32_t)j;
        if (a.spin[g] <= 0 || parent[g] != g) continue;
        const unsigned long long sz = __ldcg(&gsize[g]);
        ++v[0];
        largest = max(largest, sz);
        if (2ull * __ldcg(&ghigh[g]) >= sz) {  // the class of the majority of its cells (ties: high)
            ++v[1];
            v[2] += sz;
            hl = max(hl, sz);
        } else {
            ++v[3];
            v[4] += sz;
            ll = max(ll, sz);
        }
    }
    __shared__ unsigned long long s_sum[10];
    if (threadIdx.x < 10) s_sum[threadIdx.x] = 0;
    __syncthreads();
    const unsigned long long sums[7] = {warp_sum(v[0]), warp_sum(v[1]), warp_sum(v[2]), warp_sum(v[3]),
                                        warp_sum(v[4]), warp_sum(cells), warp_sum(high)};
    const unsigned long long most[3] = {warp_max(largest), warp_max(hl), warp_max(ll)};
    if (lane == 0) {
        for (int i = 0; i < 7; ++i)
            if (sums[i]) atomicAdd(&s_sum[i], sums[i]);
        for (int i = 0; i < 3; ++i)
            if (most[i]) atomicMax(&s_sum[7 + i], most[i]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long* to[10] = {&acc->grains, &acc->high_grains, &acc->high_in, &acc->low_grains, &acc->low_in,
                                      &acc->cells,  &acc->high_cells,  &acc->largest, &acc->high_largest, &acc->low_largest};
        for (int i = 0; i < 7; ++i)
            if (s_sum[i]) atomicAdd(to[i], s_sum[i]);
        for (int i = 7; i < 10; ++i)
            if (s_sum[i]) atomicMax(to[i], s_sum[i]);
        if (mc_last_block(&acc->left)) {  // hands them over and leaves zeroes for the next call
            static_assert(sizeof(GrainAcc) % sizeof(uint2) == 0, "copied as 8-byte words");
            uint2 w[sizeof(GrainAcc) / sizeof(uint2)];
#pragma unroll
            for (int i = 0; i < (int)(sizeof(w) / sizeof(w[0])); ++i) w[i] = __ldcg(reinterpret_cast<const uint2*>(acc) + i);
#pragma unroll
            for (int i = 0; i < (int)(sizeof(w) / sizeof(w[0])); ++i) {
                reinterpret_cast<uint2*>(out)[i] = w[i];
                reinterpret_cast<uint2*>(acc)[i] = make_uint2(0, 0);
            }
            a.ctrl->bar_arrived = 0;
        }
    }
}

// CoolingMobility (engine/src/mc/CoolingMobility.cpp) on the device.  W cells of a row per thread (W
// divides nx, so that a group is aligned in the pitched planes and in the unpitched domain).
template <int W>
struct Cells8 {  // W bytes
    uint8_t v[W];
};
template <int W>
__device__ __forceinline__ Cells8<W> load_bytes(const uint8_t* p) {
    Cells8<W> c;
    if constexpr (W == 16) *reinterpret_cast<uint4*>(c.v) = *reinterpret_cast<const uint4*>(p);
    else if constexpr (W == 4) *reinterpret_cast<uint32_t*>(c.v) = *reinterpret_cast<const uint32_t*>(p);
    else c.v[0] = *p;
    return c;
}
template <int W>
__global__ void mc_domain_from_ca_kernel(const uint8_t* type, int nx, int P, uint64_t rows, uint8_t* domain) {
    const uint32_t per_row = (uint32_t)nx / W;
    const uint64_t n = per_row * rows;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = i / per_row;
        const uint32_t x = W * (uint32_t)(i - r * per_row);
        __align__(16) Cells8<W> c = load_bytes<W>(type + r * (uint64_t)P + x);
#pragma unroll
        for (int j = 0; j < W; ++j) c.v[j] = (c.v[j] == kBasalt || c.v[j] == kLava) ? 1 : 0;  // basaltDomain (CoolingMobility.cpp:8-14)
        uint8_t* to = domain + r * (uint64_t)nx + x;
        if constexpr (W == 16) *reinterpret_cast<uint4*>(to) = *reinterpret_cast<const uint4*>(c.v);
        else if constexpr (W == 4) *reinterpret_cast<uint32_t*>(to) = *reinterpret_cast<const uint32_t*>(c.v);
        else *to = c.v[0];
    }
}

struct McCooling {
    const uint8_t* type;
    const uint16_t* solid;
    const uint16_t* arrival;
    const uint8_t* domain;
    int nx, P;
    uint64_t rows;
    double mobility_min;
    unsigned int* sums;      // largest step, largest time, largest ~time (all zero before the launch)
    float* mobility;
    McCtrl* ctrl;
};
// fromCooling in one cooperative launch: endStep, the largest solidStep / arrivalStep in the domain
// (CoolingMobility.cpp:16-25); liquidTime (32-45) and its range (timeRange, 47-56); normalize (58-74):
// mobilityMin + (1 - mobilityMin) * (t - tMin) / (tMax - tMin) in double, each operation rounded once (no
// contraction), then to float.  Bounded by the 4 bytes per cell it writes; a call for 512 x 512 x 256
// cells took 0.52 ms with three launches over a plane of times, 0.20 ms with this one.
template <int W>
__global__ __launch_bounds__(kMcThreads) void mc_cooling_kernel(const __grid_constant__ McCooling m) {
    const uint32_t per_row = (uint32_t)m.nx / W;
    const uint64_t n = per_row * m.rows, T = (uint64_t)gridDim.x * blockDim.x, i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    auto any = [](const Cells8<W>& d) {
        unsigned v = 0;
#pragma unroll
        for (int j = 0; j < W; ++j) v |= d.v[j];
        return v != 0;
    };
    unsigned last = 0;
    for (uint64_t i = i0; i < n; i += T) {
        __align__(16) const Cells8<W> d = load_bytes<W>(m.domain + i * W);
        if (!any(d)) continue;
        const uint64_t r = i / per_row, p = r * (uint64_t)m.P + W * (i - r * per_row);
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (d.v[j]) last = max(last, (unsigned)max(m.solid[p + j], m.arrival[p + j]));
    }
    last = __reduce_max_sync(0xFFFFFFFFu, last);
    if ((threadIdx.x & 31) == 0 && last) atomicMax(&m.sums[0], last);
    mc_barrier_arrive(m.ctrl);
    if (!mc_barrier_wait(m.ctrl, gridDim.x, 1)) return;
    const unsigned end = __ldcg(&m.sums[0]);
    auto time_of = [&](uint64_t p) -> unsigned {
        const unsigned s = m.type[p] == kBasalt ? m.solid[p] : end, ar = m.arrival[p];
        return s > ar ? s - ar : 0;
    };
    unsigned hi = 0, nlo = 0;
    for (uint64_t i = i0; i < n; i += T) {
        __align__(16) const Cells8<W> d = load_bytes<W>(m.domain + i * W);
        if (!any(d)) continue;
        const uint64_t r = i / per_row, p = r * (uint64_t)m.P + W * (i - r * per_row);
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (d.v[j]) {
                const unsigned t = time_of(p + j);
                hi = max(hi, t);
                nlo = max(nlo, ~t);
            }
    }
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    nlo = __reduce_max_sync(0xFFFFFFFFu, nlo);
    if ((threadIdx.x & 31) == 0) {
        if (hi) atomicMax(&m.sums[1], hi);
        if (nlo) atomicMax(&m.sums[2], nlo);
    }
    mc_barrier_arrive(m.ctrl);
    if (!mc_barrier_wait(m.ctrl, gridDim.x, 2)) return;
    hi = __ldcg(&m.sums[1]);
    const unsigned lo = ~__ldcg(&m.sums[2]);
    for (uint64_t i = i0; i < n; i += T) {
        __align__(16) const Cells8<W> d = load_bytes<W>(m.domain + i * W);
        __align__(16) float v[W];
#pragma unroll
        for (int j = 0; j < W; ++j) v[j] = 0.0f;
        if (any(d)) {
            const uint64_t r = i / per_row, p = r * (uint64_t)m.P + W * (i - r * per_row);
#pragma unroll
            for (int j = 0; j < W; ++j) {
                if (!d.v[j]) continue;
                if (hi == lo) {
                    v[j] = 1.0f;
                } else {
                    const double norm = __ddiv_rn((double)(time_of(p + j) - lo), (double)(hi - lo));
                    v[j] = __double2float_rn(__dadd_rn(m.mobility_min, __dmul_rn(__dsub_rn(1.0, m.mobility_min), norm)));
                }
            }
        }
        float* to = m.mobility + i * W;
        if constexpr (W >= 4) {
#pragma unroll
            for (int q = 0; q < W / 4; ++q) reinterpret_cast<float4*>(to)[q] = reinterpret_cast<const float4*>(v)[q];
        } else {
            *to = v[0];
        }
    }
}

}  // namespace vca

using namespace vca;

struct vca_mc {
    vca_mc_desc desc;
    int device = 0;
    cudaStream_t stream = nullptr;
    NbTable nb_host;
    NbTable* nb = nullptr;
    int per[3] = {0, 0, 0};
    int colors = 0;
    int parity_colors = 0;
    int classes[3] = {1, 1, 1};
    uint64_t n = 0;
    uint64_t cap_n = 0;                  // cells the per-cell buffers hold (a resident handle runs smaller spaces)
    int32_t* spin = nullptr;
    uint8_t* domain = nullptr;
    float* mobility = nullptr;     // N floats when set
    bool mobility_set = false;
    bool mobility_on = false;
    uint32_t* list = nullptr;      // domain cells by colour
    float* list_mob = nullptr;
    std::vector<uint64_t> color_off;
    unsigned long long* table = nullptr;
    McCtrl* ctrl = nullptr;
    McCtrl* ctrl_host = nullptr;      // pinned, host-mapped mirror
    bool mirrored = false;            // it holds what the last call left, and the counters of one launch are zero
    McCtrl* ctrl_host_dev = nullptr;  // its device address
    bool domain_set = false;
    bool initialized = false;
    int sms = 148;
    // set-up buffers, allocated on first use and kept (no cudaMalloc / cudaFree per call)
    uint32_t* run_counts = nullptr;      // [color][block] of the list build
    uint32_t* totals_host = nullptr;     // pinned, host-mapped: cells per colour (behind gacc_host)
    uint32_t* totals_host_dev = nullptr; // its device address
    bool domain_all = false;             // every cell is in the domain
    bool listed = false;                 // the colour lists are built (a whole space needs them rarely)
    uint32_t* gparent = nullptr;         // grain statistics: parent, size, high count per cell (n each)
    uint32_t* gsize = nullptr;
    uint32_t* ghigh = nullptr;
    void* gacc = nullptr;                // GrainAcc
    GrainAcc* gacc_host = nullptr;       // pinned, host-mapped copy of it (behind ctrl_host)
    GrainAcc* gacc_host_dev = nullptr;   // its device address
    int grain_per_sm = 0;                // resident blocks of the grain kernel
    cudaEvent_t ev_a = nullptr, ev_b = nullptr;
    double total_ms = 0.0;
    double color_ms = 0.0;
    uint64_t color_launches = 0;
    uint64_t launches = 0;
    int profile_kernels = 0;
    std::vector<cudaEvent_t> prof_events;
    int slab_zoff = -1;                  // z slab of a taller grid (vca_mc_set_slab), -1: none
    uint8_t* sp8 = nullptr;              // orientation - 1 per cell, for the whole-space sweeps (grows only)
    size_t sp8_cap = 0;
    bool user_spins = false;             // orientations were written from outside since vca_mc_initialize
};

namespace {

vca_status mc_check(const vca_mc* h) {
    if (!h) {
        set_error("null vca_mc handle");
        return VCA_ERR_ARG;
    }
    return VCA_OK;
}

McArgs mc_args(const vca_mc* h) {
    McArgs a;
    std::memset(&a, 0, sizeof(a));
    a.nx = h->desc.nx;
    a.ny = h->desc.ny;
    a.nz = h->desc.nz;
    for (int i = 0; i < 3; ++i) {
        a.per[i] = h->per[i];
        a.classes[i] = h->classes[i];
    }
    a.div_nx = make_fastdiv((uint32_t)a.nx);
    a.div_ny = make_fastdiv((uint32_t)a.ny);
    a.parity_colors = h->parity_colors;
    a.seed = h->desc.seed;
    a.q_mod = make_fastmod((uint64_t)h->desc.Q);
    a.qm1_mod = make_fastmod((uint64_t)(h->desc.Q - 1));
    a.var_mod = make_fastmod((uint64_t)h->nb_host.variants);
    a.variants = h->nb_host.variants;
    a.spin = h->spin;
    a.list = h->list;
    a.list_mob = h->list_mob;
    a.table = h->table;
    a.nb = h->nb;
    a.ctrl = h->ctrl;
    a.mirror = h->ctrl_host_dev;
    a.zoff = h->slab_zoff > 0 ? h->slab_zoff : 0;
    a.gidx_base = (uint64_t)h->desc.nx * h->desc.ny * (uint64_t)a.zoff;
    return a;
}

// The control block copied by one warp into host-mapped pinned memory (not a device-to-host copy,
// which would queue behind another handle's large download on the copy engines).
__global__ void mc_ctrl_snapshot_kernel(const McCtrl* src, McCtrl* dst) {
    static_assert(sizeof(McCtrl) % sizeof(uint32_t) == 0, "McCtrl is copied as words");
    const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
    volatile uint32_t* d = reinterpret_cast<volatile uint32_t*>(dst);
    for (int i = threadIdx.x; i < (int)(sizeof(McCtrl) / sizeof(uint32_t)); i += 32) d[i] = s[i];
}

vca_status mc_sync(vca_mc* h) {
    mc_ctrl_snapshot_kernel<<<1, 32, 0, h->stream>>>(h->ctrl, h->ctrl_host_dev);
    VCA_CUDA(cudaGetLastError());
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    return VCA_OK;
}

int grid_for(uint64_t work, int sms) {
    const uint64_t b = (work + kMcThreads - 1) / kMcThreads;
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(b, (uint64_t)sms * 16));
}

void mc_free(vca_mc* h) {
    cudaSetDevice(h->device);
    cudaFree(h->nb);
    cudaFree(h->spin);
    cudaFree(h->domain);
    cudaFree(h->mobility);
    cudaFree(h->list);
    cudaFree(h->list_mob);
    cudaFree(h->table);
    cudaFree(h->ctrl);
    cudaFree(h->run_counts);
    cudaFree(h->gparent);
    cudaFree(h->gsize);
    cudaFree(h->ghigh);
    cudaFree(h->gacc);
    cudaFree(h->sp8);
    if (h->ctrl_host) cudaFreeHost(h->ctrl_host);
    if (h->ev_a) cudaEventDestroy(h->ev_a);
    if (h->ev_b) cudaEventDestroy(h->ev_b);
    for (cudaEvent_t e : h->prof_events) cudaEventDestroy(e);
    if (h->stream) cudaStreamDestroy(h->stream);
}

// A variant's neighbours as bits (dx + 1) + 3 (dy + 1) + 9 (dz + 1) of the 3 x 3 x 3 block.
uint32_t nb_mask(const NbTable& nb, int v) {
    uint32_t m = 0;
    if (v < nb.variants)
        for (int k = 0; k < nb.count[v]; ++k)
            m |= 1u << ((nb.off[v][k][0] + 1) + 3 * (nb.off[v][k][1] + 1) + 9 * (nb.off[v][k][2] + 1));
    return m;
}

using SweepsKernel = void (*)(McArgs, McColors, int);

SweepsKernel sweeps_kernel_of(const vca_mc* h) {
    const bool random_nb = h->nb_host.variants > 1;
    if (h->mobility_on) return random_nb ? mc_sweeps_kernel<true, true> : mc_sweeps_kernel<true, false>;
    return random_nb ? mc_sweeps_kernel<false, true> : mc_sweeps_kernel<false, false>;
}

constexpr size_t kMcEntryCacheMax = 160 * 1024;  // shared memory a block may spend on its entries

// The sweep kernel's cooperative grid (all blocks resident at once, no more blocks than the widest
// colour needs), its rounds per colour, and whether the blocks' entries fit in shared memory at
// that occupancy (then the dynamic shared memory size in *smem).
vca_status sweeps_launch_shape(vca_mc* h, SweepsKernel kernel, McColors* col, int* grid, size_t* smem) {
    uint64_t widest = 0;
    for (int c = 0; c < h->colors; ++c) widest = std::max<uint64_t>(widest, h->color_off[c + 1] - h->color_off[c]);
    const uint64_t need = std::max<uint64_t>(1, (widest + kMcThreads - 1) / kMcThreads);
    const size_t per_entry = h->mobility_on ? 8 : 4;
    VCA_CUDA(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMcEntryCacheMax));
    int per_sm_max = 0;
    VCA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_max, kernel, kMcThreads, 0));
    per_sm_max = std::max(1, per_sm_max);
    auto rounds_for = [&](uint64_t threads) {
        int total = 0;
        for (int c = 0; c < h->colors; ++c) {
            const uint64_t n = h->color_off[c + 1] - h->color_off[c];
            col->rounds[c] = (int)((n + threads - 1) / threads);
            col->round0[c] = total;
            total += col->rounds[c];
        }
        col->total_rounds = total;
    };
    for (int per_sm = per_sm_max; per_sm >= 1; --per_sm) {
        const int g = (int)std::max<uint64_t>(1, std::min<uint64_t>(need, (uint64_t)h->sms * per_sm));
        rounds_for((uint64_t)g * kMcThreads);
        int most = 0;
        for (int c = 0; c < h->colors; ++c) most = std::max(most, col->rounds[c]);
        const bool pre = most <= kPreRounds;
        const size_t bytes = (size_t)col->total_rounds * kMcThreads * per_entry +
                             (pre ? (size_t)kPreRounds * kMcThreads * (8 + 4 + 1) : 0);
        if (bytes > kMcEntryCacheMax) continue;
        int fit = 0;
        VCA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, kMcThreads, bytes));
        if ((uint64_t)fit * h->sms < (uint64_t)g) continue;
        col->cached = 1;
        col->pre = pre;
        *grid = g;
        *smem = bytes;
        return VCA_OK;
    }
    // entries from global memory at full occupancy
    const int g = (int)std::max<uint64_t>(1, std::min<uint64_t>(need, (uint64_t)h->sms * per_sm_max));
    rounds_for((uint64_t)g * kMcThreads);
    col->cached = 0;
    col->pre = 0;
    *grid = g;
    *smem = 0;
    return VCA_OK;
}

using SpaceKernel = void (*)(McArgs, McSpace, int);

template <bool kMobility, bool kWide, int kThreads>
SpaceKernel space_kernel_of(const vca_mc* h) {
    if (h->parity_colors) return mc_space_sweeps_kernel<kMobility, 1, true, kWide, kThreads>;
    switch (h->desc.neighborhood) {
        case VCA_NB_MOORE: return mc_space_sweeps_kernel<kMobility, 0, false, kWide, kThreads>;
        case VCA_NB_VON_NEUMANN: return mc_space_sweeps_kernel<kMobility, 1, false, kWide, kThreads>;
        default: return mc_space_sweeps_kernel<kMobility, 2, false, kWide, kThreads>;
    }
}
template <int kThreads>
SpaceKernel space_kernel_of(const vca_mc* h) {
    if (h->desc.Q > 128) return h->mobility_on ? space_kernel_of<true, true, kThreads>(h) : space_kernel_of<false, true, kThreads>(h);
    return h->mobility_on ? space_kernel_of<true, false, kThreads>(h) : space_kernel_of<false, false, kThreads>(h);
}

// Bytes of a row of the byte copy: 8 in front, the cells, 8 behind.
int space_pitch(int nx) { return 8 + (nx + 7) / 8 * 8 + 8; }

// A space that is one cell wide in x has the same order of cells as a plane of ny x nz: the sweeps see it
// as that (the neighbourhood's offsets move down an axis).
bool space_turned(const vca_mc* h) { return h->desc.nx == 1; }

// Cells of colour c when every cell is in the domain.
uint64_t whole_color_size(const vca_mc* h, int c) {
    if (h->parity_colors) return c == 0 ? (h->n + 1) / 2 : h->n / 2;  // (x + y + z) & 1
    const int dims[3] = {h->desc.nx, h->desc.ny, h->desc.nz};
    uint64_t size = 1;
    for (int a = 0; a < 3; ++a) {
        const int k = c % h->classes[a], n = dims[a];
        c /= h->classes[a];
        size *= (uint64_t)(h->classes[a] == 1 ? n : h->classes[a] == 2 ? (n + 1 - k) / 2 : k == 2 ? 1 : (n - 1) / 2);
    }
    return size;
}

// The colour lists of the domain; with `first` also the first orientations (vca_mc_initialize), else the
// orientations stay (a whole space whose lists are wanted after all).
vca_status build_lists(vca_mc* h, bool first) {
    const uint64_t steps = (h->n + kRunCells - 1) / kRunCells;
    const uint64_t cap_steps = (h->cap_n + kRunCells - 1) / kRunCells, most = (uint64_t)h->sms * 16;
    // sized for the capacity, so that later, larger spaces on a resident handle allocate nothing
    if (!h->run_counts) VCA_CUDA(cudaMalloc(&h->run_counts, sizeof(uint32_t) * 28 * std::max<uint64_t>(1, std::min(cap_steps, most))));
    if (!h->list || (h->mobility_on && !h->list_mob)) {
        cudaFree(h->list);
        cudaFree(h->list_mob);
        h->list = nullptr;
        h->list_mob = nullptr;
        VCA_CUDA(cudaMalloc(&h->list, 4 * std::max<uint64_t>(h->cap_n, 1)));
        VCA_CUDA(cudaMalloc(&h->list_mob, 4 * std::max<uint64_t>(h->cap_n, 1)));
    }
    const McArgs a = mc_args(h);
    McRuns r;
    std::memset(&r, 0, sizeof(r));
    r.domain = h->domain;
    r.n = h->n;
    r.per_block = (steps + most - 1) / most * kRunCells;
    r.colors = h->colors;
    r.counts = h->run_counts;
    const int blocks = (int)((h->n + r.per_block - 1) / r.per_block);
    mc_runs_count_kernel<<<blocks, kMcThreads, 0, h->stream>>>(a, r, first ? 1 : 0);
    mc_runs_place_kernel<<<1, 1024, 0, h->stream>>>(h->run_counts, h->colors, blocks, h->totals_host_dev);
    mc_runs_list_kernel<<<blocks, kMcThreads, 0, h->stream>>>(a, r, h->mobility_on ? h->mobility : nullptr, h->list, h->list_mob);
    VCA_CUDA(cudaGetLastError());
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    h->color_off.assign((size_t)h->colors + 1, 0);
    for (int c = 0; c < h->colors; ++c) h->color_off[(size_t)c + 1] = h->color_off[(size_t)c] + h->totals_host[c];
    h->listed = true;
    return VCA_OK;
}
vca_status want_lists(vca_mc* h) { return h->listed ? VCA_OK : build_lists(h, false); }

// The whole-space sweeps apply when every cell is in the domain, an orientation fits a byte, and the
// rows are not so short that their frame columns outweigh them (below 6 cells).
bool space_applies(const vca_mc* h) {
    const int nx = space_turned(h) ? h->desc.ny : h->desc.nx;
    return !h->profile_kernels && h->slab_zoff < 0 && h->desc.Q <= 256 && !h->color_off.empty() &&
           h->color_off.back() == h->n && h->n > 0 && nx >= 6;
}

// A whole space whose colours leave a thread of the grid about one cell: the listed kernel's pass, a cell
// per thread and its draws done while the block waits, is then shorter than four cells per thread.  Per MCS
// of 8 colours, listed against four cells: 50^3 18 / 31 us, 64^3 21 / 30, 80^3 (64 000 cells a colour)
// 26 / 30 and level with the lists' set-up in calls of 5 MCS, 100^3 32 / 31; 512 x 512 in 4 colours of
// 65 536 12.5 / 15.4.  The lists cost what four MCS save; a handle made for a much larger space would
// allocate them for it.
constexpr uint64_t kListWhole = 48000;   // cells of the widest colour
constexpr int kListWholeSweeps = 4;
bool small_space_listed(const vca_mc* h, int count) {
    if (h->user_spins || h->desc.Q > 256 || h->desc.nx < 6 || h->slab_zoff >= 0) return false;
    if (!h->listed && (count < kListWholeSweeps || (!h->list && h->cap_n > 64 * kListWhole))) return false;
    uint64_t widest = 0;
    for (int c = 0; c < h->colors; ++c) widest = std::max<uint64_t>(widest, h->color_off[c + 1] - h->color_off[c]);
    return widest <= kListWhole;
}

// The byte copy's shape and the colour classes; `a` becomes the sweep's view of a turned space.
McSpace space_args(const vca_mc* h, McArgs& a) {
    McSpace d;
    std::memset(&d, 0, sizeof(d));
    for (int v = 0; v < 6; ++v) d.mask[v] = nb_mask(h->nb_host, v);
    if (space_turned(h)) {
        a.nx = h->desc.ny, a.ny = h->desc.nz, a.nz = 1;
        for (int i = 0; i < 3; ++i) {
            a.per[i] = i < 2 ? h->per[i + 1] : 0;
            a.classes[i] = i < 2 ? h->classes[i + 1] : 1;
        }
        for (uint32_t& m : d.mask) {  // (0, dy, dz) -> (dy, dz, 0)
            uint32_t to = 0;
            for (int i = 0; i < 9; ++i)
                if ((m >> (3 * i + 1)) & 1u) to |= 1u << (9 + i);
            m = to;
        }
    }
    d.sp = h->sp8;
    d.mob = h->mobility_on ? h->mobility : nullptr;
    d.P8 = space_pitch(a.nx);
    const int dims[3] = {a.nx, a.ny, a.nz};
    for (int ax = 0; ax < 3; ++ax) {
        const int n = dims[ax], classes = h->parity_colors ? 1 : a.classes[ax];
        int* c = d.cnt[ax];
        c[0] = classes == 1 ? n : classes == 2 ? (n + 1) / 2 : (n - 1) / 2;
        c[1] = classes == 1 ? 1 : n / 2;
        c[2] = 1;
    }
    const int cx = h->parity_colors ? 1 : a.classes[0];
    for (int c = 0; c < 3; ++c) {
        d.xlo[c] = c == 2 ? a.nx - 1 : 0;
        d.xhi[c] = cx == 3 && c < 2 ? a.nx - 1 : a.nx;
        d.g0[c] = d.xlo[c] / 8;
        d.gx[c] = (d.xhi[c] + 7) / 8 - d.g0[c];
        d.div_gx[c] = make_fastdiv32((uint32_t)d.gx[c]);
        d.div_cy[c] = make_fastdiv32((uint32_t)std::max(1, d.cnt[1][c]));
    }
    d.qm1 = (uint32_t)h->desc.Q - 1u;
    d.qm1_inv = 0xFFFFFFFFu / d.qm1;
    d.qm1_2p32 = (uint32_t)((1ULL << 32) % d.qm1);
    d.uphill = h->desc.kT > 0.0;
    return d;
}

using ListKernel = void (*)(McArgs, McColors, McBytes, int);

ListKernel list_kernel_of(const vca_mc* h) {
    const bool random_nb = h->nb_host.variants > 1;
    if (h->mobility_on) return random_nb ? mc_list_sweeps_kernel<true, true> : mc_list_sweeps_kernel<true, false>;
    return random_nb ? mc_list_sweeps_kernel<false, true> : mc_list_sweeps_kernel<false, false>;
}

uint64_t list_bytes(const vca_mc* h) { return (uint64_t)space_pitch(h->desc.nx) * (uint64_t)h->desc.ny * (uint64_t)h->desc.nz; }

// The byte copy grows only (a resident handle allocates nothing per job).
vca_status sp8_reserve(vca_mc* h, uint64_t bytes) {
    if (bytes <= h->sp8_cap) return VCA_OK;
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    cudaFree(h->sp8);
    h->sp8 = nullptr;
    h->sp8_cap = 0;
    VCA_CUDA(cudaMalloc(&h->sp8, bytes));
    h->sp8_cap = bytes;
    return VCA_OK;
}

// Whether the byte form of the list sweeps applies, and its launch: Q <= 256, orientations as
// vca_mc_initialize and the sweeps left them (only the domain's cells are copied, so a value set outside
// of it would be missed), 32-bit offsets, rows not too short for their frame columns, and every block's
// entries in shared memory.  At least 96 threads per block, then one block per SM
// (81 K cells, 400 passes: 1.92 ms; by 128 threads 1.96, 192 2.14, 256 2.24).
bool list_bytes_shape(const vca_mc* h, McColors* col, int* grid, int* threads, size_t* smem) {
    if (h->desc.Q > 256 || h->slab_zoff >= 0 || h->user_spins || h->desc.nx < 6 || list_bytes(h) > 0xFFFFFFF0ull) return false;
    uint64_t widest = 1;
    for (int c = 0; c < h->colors; ++c) widest = std::max<uint64_t>(widest, h->color_off[c + 1] - h->color_off[c]);
    const uint64_t g = std::min<uint64_t>((widest + 95) / 96, (uint64_t)h->sms);
    const uint64_t t = std::min<uint64_t>(((widest + g - 1) / g + 31) / 32 * 32, (uint64_t)kListThreads - 32);
    int total = 0;
    for (int c = 0; c < h->colors; ++c) {
        const uint64_t n = h->color_off[c + 1] - h->color_off[c];
        col->rounds[c] = (int)((n + g * t - 1) / (g * t));
        col->round0[c] = total;
        total += col->rounds[c];
    }
    col->total_rounds = total;
    *grid = (int)g;
    *threads = (int)t + 32;  // and the polling warp
    *smem = (size_t)total * t * (h->mobility_on ? 12 : 8);
    return *smem <= kListSmemMax;
}

}  // namespace

namespace {

vca_status mc_validate(const vca_mc_desc* d, const char* who) {
    auto bad = [&](const std::string& m) {
        set_error(std::string(who) + ": " + m);
        return VCA_ERR_ARG;
    };
    if (d->nx < 1 || d->ny < 1 || d->nz < 1 || (d->nx > 1) + (d->ny > 1) + (d->nz > 1) < 2)
        return bad("the space must be 2D or 3D");
    if ((uint64_t)d->nx * d->ny * d->nz > 2000000000ULL) return bad("more than 2 000 000 000 cells");
    if (d->Q < 2) return bad("Q must be at least 2 (PottsMC needs two orientations)");
    if (!(d->J > 0.0) || !(d->kT >= 0.0)) return bad("J must be > 0 and kT >= 0");
    NbTable nb;
    if (!build_nb(d->neighborhood, d->nx, d->ny, d->nz, nb)) return bad("the hexagonal neighbourhood is defined in 2D only");
    return VCA_OK;
}

// The space and parameters of an MC handle: neighbourhood, periodic axes, colours, acceptance
// table; orientations and domain cleared.  Allocates nothing.
vca_status mc_configure(vca_mc* h, const vca_mc_desc* d) {
    h->desc = *d;
    h->n = (uint64_t)d->nx * d->ny * d->nz;
    build_nb(d->neighborhood, d->nx, d->ny, d->nz, h->nb_host);
    h->slab_zoff = -1;
    // Periodic axes: PottsMC ctor (PottsMC.cpp:18) with the Boundary of McStage::run (McStage.cpp:106).
    const bool periodic = d->boundary == VCA_BC_PERIODIC;
    h->per[0] = periodic && d->nx > 1;
    h->per[1] = periodic && d->ny > 1;
    h->per[2] = periodic && d->domain_full && d->nz > 1;
    // Colours (PottsMC::buildColors, PottsMC.cpp:160-193).
    const int dims[3] = {d->nx, d->ny, d->nz};
    bool odd = false;
    for (int a = 0; a < 3; ++a) odd = odd || (h->per[a] && dims[a] % 2 == 1);
    h->parity_colors = d->neighborhood == VCA_NB_VON_NEUMANN && !odd;
    for (int a = 0; a < 3; ++a) h->classes[a] = 1;
    if (h->parity_colors) {
        h->colors = 2;
    } else {
        h->colors = 1;
        for (int a = 0; a < 3; ++a) {
            h->classes[a] = dims[a] == 1 ? 1 : (h->per[a] && dims[a] % 2 == 1 ? 3 : 2);
            h->colors *= h->classes[a];
        }
    }
    // Acceptance thresholds for every (unlikeBefore, unlikeAfter): dE = J*after - J*before
    // (PottsMC.cpp:431); dE <= 0 always (bit 63), else ceil(exp(-dE/kT) * 2^53), or 0 when kT = 0.
    std::vector<unsigned long long> table(kTableSide * kTableSide, 0);
    for (int b = 0; b < kTableSide; ++b)
        for (int a = 0; a < kTableSide; ++a) {
            const double dE = d->J * a - d->J * b;
            unsigned long long v = 0;
            if (dE <= 0.0) {
                v = 1ULL << 63;
            } else if (d->kT > 0.0) {
                const double p = std::exp(-dE / d->kT);
                v = (unsigned long long)std::ceil(p * 9007199254740992.0);
            }
            table[b * kTableSide + a] = v;
        }
    VCA_CUDA(cudaMemcpyAsync(h->nb, &h->nb_host, sizeof(NbTable), cudaMemcpyHostToDevice, h->stream));
    VCA_CUDA(cudaMemcpyAsync(h->table, table.data(), 8 * table.size(), cudaMemcpyHostToDevice, h->stream));
    VCA_CUDA(cudaMemsetAsync(h->spin, 0, 4 * h->n, h->stream));
    VCA_CUDA(cudaMemsetAsync(h->domain, 0, h->n, h->stream));
    VCA_CUDA(cudaMemsetAsync(h->ctrl, 0, sizeof(McCtrl), h->stream));
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    h->domain_set = false;
    h->mobility_set = false;
    h->mobility_on = false;
    h->initialized = false;
    h->color_off.assign(1, 0);
    return VCA_OK;
}

}  // namespace

extern "C" {

vca_status vca_mc_create(const vca_mc_desc* d, vca_mc** out) {
    if (!d || !out) {
        set_error("vca_mc_create: null argument");
        return VCA_ERR_ARG;
    }
    *out = nullptr;
    if (vca_status s = mc_validate(d, "vca_mc_create")) return s;
    const uint64_t n = (uint64_t)d->nx * d->ny * d->nz;
    vca_mc* h = new vca_mc();
    h->device = d->device;
    h->cap_n = n;
    auto fail = [&](vca_status s) {
        mc_free(h);
        delete h;
        return s;
    };
    cudaError_t e = cudaSetDevice(d->device);
    if (e != cudaSuccess) return fail(cuda_fail(e, "cudaSetDevice"));
    cudaDeviceProp prop;
    if ((e = cudaGetDeviceProperties(&prop, d->device)) != cudaSuccess) return fail(cuda_fail(e, "cudaGetDeviceProperties"));
    if (prop.major < 10) {
        set_error("vca_mc_create: needs an sm_100 (Blackwell) device");
        return fail(VCA_ERR_CUDA);
    }
    h->sms = prop.multiProcessorCount;
    e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) return fail(cuda_fail(e, "cudaStreamCreate"));
    if ((e = cudaMalloc(&h->nb, sizeof(NbTable))) != cudaSuccess || (e = cudaMalloc(&h->spin, 4 * n)) != cudaSuccess ||
        (e = cudaMalloc(&h->domain, n)) != cudaSuccess ||
        (e = cudaMalloc(&h->table, 8 * kTableSide * kTableSide)) != cudaSuccess ||
        (e = cudaMalloc(&h->ctrl, sizeof(McCtrl))) != cudaSuccess)
        return fail(cuda_fail(e, "cudaMalloc"));
    // one pinned block: the mirror of the control block, that of the grain statistics, colour totals
    static_assert(sizeof(McCtrl) % alignof(GrainAcc) == 0, "GrainAcc follows McCtrl");
    if ((e = cudaHostAlloc(&h->ctrl_host, sizeof(McCtrl) + sizeof(GrainAcc) + 28 * sizeof(uint32_t), cudaHostAllocMapped)) !=
            cudaSuccess ||
        (e = cudaHostGetDevicePointer(&h->ctrl_host_dev, h->ctrl_host, 0)) != cudaSuccess)
        return fail(cuda_fail(e, "cudaHostAlloc (mapped)"));
    h->gacc_host = reinterpret_cast<GrainAcc*>(h->ctrl_host + 1);
    h->gacc_host_dev = reinterpret_cast<GrainAcc*>(h->ctrl_host_dev + 1);
    h->totals_host = reinterpret_cast<uint32_t*>(h->gacc_host + 1);
    h->totals_host_dev = reinterpret_cast<uint32_t*>(h->gacc_host_dev + 1);
    if ((e = cudaEventCreate(&h->ev_a)) != cudaSuccess || (e = cudaEventCreate(&h->ev_b)) != cudaSuccess)
        return fail(cuda_fail(e, "cudaEventCreate"));
    const char* prof = std::getenv("VCA_PROFILE_KERNELS");
    h->profile_kernels = prof != nullptr && prof[0] == '1';
    if (vca_status s = mc_configure(h, d)) return fail(s);
    *out = h;
    return VCA_OK;
}

vca_status vca_mc_reconfigure(vca_mc* h, const vca_mc_desc* d) {
    if (vca_status s = mc_check(h)) return s;
    if (!d) {
        set_error("vca_mc_reconfigure: null desc");
        return VCA_ERR_ARG;
    }
    if (vca_status s = mc_validate(d, "vca_mc_reconfigure")) return s;
    if (d->device != h->device || (uint64_t)d->nx * d->ny * d->nz > h->cap_n) {
        set_error("vca_mc_reconfigure: the space does not fit the handle (more cells, or another device)");
        return VCA_ERR_ARG;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    return mc_configure(h, d);
}

vca_status vca_mc_footprint(const vca_mc_desc* d, uint64_t* bytes) {
    if (!d || !bytes) {
        set_error("vca_mc_footprint: null argument");
        return VCA_ERR_ARG;
    }
    if (vca_status s = mc_validate(d, "vca_mc_footprint")) return s;
    const uint64_t n = (uint64_t)d->nx * d->ny * d->nz;
    // spin 4 + domain 1 + mobility 4 + colour lists 8 + grain labels 12 bytes per cell, the byte copy of the
    // orientations (at most 4 bytes per cell), the list build's counts, tables and counters
    *bytes = 37 * n + 8 * kTableSide * kTableSide + sizeof(McCtrl) + 8 * 28 + sizeof(NbTable) + 4096;
    return VCA_OK;
}

vca_status vca_mc_set_domain(vca_mc* h, const uint8_t* in_domain) {
    if (vca_status s = mc_check(h)) return s;
    VCA_CUDA(cudaSetDevice(h->device));
    if (in_domain) {
        std::vector<uint8_t> d(in_domain, in_domain + h->n);
        for (auto& v : d) v = v ? 1 : 0;
        VCA_CUDA(cudaMemcpyAsync(h->domain, d.data(), h->n, cudaMemcpyHostToDevice, h->stream));
        VCA_CUDA(cudaStreamSynchronize(h->stream));
    } else {
        VCA_CUDA(cudaMemsetAsync(h->domain, 1, h->n, h->stream));
    }
    h->domain_all = in_domain == nullptr;
    h->domain_set = true;
    h->initialized = false;
    return VCA_OK;
}

vca_status vca_mc_set_mobility(vca_mc* h, const float* mobility) {
    if (vca_status s = mc_check(h)) return s;
    VCA_CUDA(cudaSetDevice(h->device));
    if (!mobility) {
        h->mobility_on = false;
        return VCA_OK;
    }
    if (!h->mobility) VCA_CUDA(cudaMalloc(&h->mobility, 4 * h->cap_n));
    VCA_CUDA(cudaMemcpyAsync(h->mobility, mobility, 4 * h->n, cudaMemcpyHostToDevice, h->stream));
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    h->mobility_set = true;
    h->mobility_on = true;
    h->initialized = false;
    return VCA_OK;
}

vca_status vca_mc_set_domain_from_ca(vca_mc* h, vca_ca* ca) {
    if (vca_status s = mc_check(h)) return s;
    CaView v;
    if (vca_status s = ca_view(ca, &v)) return s;
    if (v.nx != h->desc.nx || v.ny != h->desc.ny || v.nz != h->desc.nz) {
        set_error("vca_mc_set_domain_from_ca: CA and MC dimensions differ");
        return VCA_ERR_ARG;
    }
    if (v.device != h->device) {
        set_error("vca_mc_set_domain_from_ca: CA and MC handles live on different devices");
        return VCA_ERR_ARG;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    VCA_CUDA(cudaStreamSynchronize(v.stream));
    const uint64_t rows = (uint64_t)v.ny * v.nz;
    if (v.nx % 16 == 0) mc_domain_from_ca_kernel<16><<<h->sms * 8, 256, 0, h->stream>>>(v.type, v.nx, v.P, rows, h->domain);
    else if (v.nx % 4 == 0) mc_domain_from_ca_kernel<4><<<h->sms * 8, 256, 0, h->stream>>>(v.type, v.nx, v.P, rows, h->domain);
    else mc_domain_from_ca_kernel<1><<<h->sms * 8, 256, 0, h->stream>>>(v.type, v.nx, v.P, rows, h->domain);
    VCA_CUDA(cudaGetLastError());
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    h->domain_all = false;
    h->domain_set = true;
    h->initialized = false;
    return VCA_OK;
}

vca_status vca_mc_set_mobility_from_ca(vca_mc* h, vca_ca* ca, double mobility_min, int use_in_dynamics) {
    if (vca_status s = mc_check(h)) return s;
    if (!h->domain_set) {
        set_error("vca_mc_set_mobility_from_ca: set the domain first");
        return VCA_ERR_STATE;
    }
    CaView v;
    if (vca_status s = ca_view(ca, &v)) return s;
    if (v.nx != h->desc.nx || v.ny != h->desc.ny || v.nz != h->desc.nz || v.device != h->device) {
        set_error("vca_mc_set_mobility_from_ca: CA and MC handles do not match");
        return VCA_ERR_ARG;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    VCA_CUDA(cudaStreamSynchronize(v.stream));
    if (!h->mobility) VCA_CUDA(cudaMalloc(&h->mobility, 4 * h->cap_n));
    McCooling m;
    std::memset(&m, 0, sizeof(m));
    m.type = v.type;
    m.solid = v.solid;
    m.arrival = v.arrival;
    m.domain = h->domain;
    m.nx = v.nx;
    m.P = v.P;
    m.rows = (uint64_t)v.ny * v.nz;
    m.mobility_min = mobility_min;
    m.sums = h->ctrl->cooling;
    m.mobility = h->mobility;
    m.ctrl = h->ctrl;
    const int w = v.nx % 16 == 0 ? 16 : v.nx % 4 == 0 ? 4 : 1;
    const void* kernel = w == 16 ? (const void*)mc_cooling_kernel<16> : w == 4 ? (const void*)mc_cooling_kernel<4>
                                                                              : (const void*)mc_cooling_kernel<1>;
    int per_sm = 0;
    VCA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kMcThreads, 0));
    const int grid = (int)std::min<uint64_t>((h->n / w + kMcThreads - 1) / kMcThreads, (uint64_t)h->sms * std::max(1, std::min(per_sm, 4)));
    static_assert(offsetof(McCtrl, cooling) == offsetof(McCtrl, bar_arrived) + 8, "one memset clears both");
    VCA_CUDA(cudaMemsetAsync(&h->ctrl->bar_arrived, 0, 8 + sizeof(h->ctrl->cooling), h->stream));
    void* args[] = {&m};
    VCA_CUDA(cudaLaunchCooperativeKernel(kernel, grid, kMcThreads, args, 0, h->stream));
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    h->mobility_set = true;
    h->mobility_on = use_in_dynamics != 0;
    h->initialized = false;
    return VCA_OK;
}

vca_status vca_mc_mobility(vca_mc* h, float* out) {
    if (vca_status s = mc_check(h)) return s;
    if (!h->mobility_set) {
        set_error("vca_mc_mobility: no mobility was set");
        return VCA_ERR_STATE;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    VCA_CUDA(cudaMemcpyAsync(out, h->mobility, 4 * h->n, cudaMemcpyDeviceToHost, h->stream));
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    return VCA_OK;
}

vca_status vca_mc_initialize(vca_mc* h) {
    if (vca_status s = mc_check(h)) return s;
    if (!h->domain_set) {
        set_error("vca_mc_initialize: set the domain first");
        return VCA_ERR_STATE;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    h->listed = false;
    if (h->domain_all && h->slab_zoff < 0) {
        // a whole space: the colours' sizes are known, and its sweeps, energy and grains need no lists
        mc_init_all_kernel<<<h->sms * 8, 256, 0, h->stream>>>(mc_args(h), h->n);
        VCA_CUDA(cudaGetLastError());
        h->color_off.assign((size_t)h->colors + 1, 0);
        for (int c = 0; c < h->colors; ++c) h->color_off[(size_t)c + 1] = h->color_off[(size_t)c] + whole_color_size(h, c);
    } else if (vca_status s = build_lists(h, true)) {
        return s;
    }
    VCA_CUDA(cudaMemsetAsync(h->ctrl, 0, sizeof(McCtrl), h->stream));
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    std::memset(h->ctrl_host, 0, sizeof(McCtrl));
    h->mirrored = true;
    h->user_spins = false;
    h->initialized = true;
    return VCA_OK;
}

vca_status vca_mc_sweep(vca_mc* h, int count, uint64_t* accepted) {
    if (vca_status s = mc_check(h)) return s;
    if (!h->initialized) {
        set_error("vca_mc_sweep: initialize first");
        return VCA_ERR_STATE;
    }
    if (count < 0) {
        set_error("vca_mc_sweep: negative count");
        return VCA_ERR_ARG;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    McArgs a = mc_args(h);
    // (a sweep launch leaves the counters of one launch at zero; single colour passes do not)
    if (!h->mirrored) VCA_CUDA(cudaMemsetAsync(&h->ctrl->sweep_accepted, 0, 8, h->stream));
    h->mirrored = false;
    if (!h->profile_kernels) {
        // all sweeps in one cooperative launch (colour passes separated by grid barriers)
        const bool space = space_applies(h) && !small_space_listed(h, count);
        VCA_CUDA(cudaEventRecord(h->ev_a, h->stream));
        if (count > 0 && space) {
            // whole space: sweeps on the byte copy of the orientations, copied back after
            McArgs va = a;
            McSpace d = space_args(h, va);
            const uint64_t rows = (uint64_t)va.ny * va.nz, bytes = (uint64_t)d.P8 * rows;
            if (vca_status s = sp8_reserve(h, bytes)) return s;
            d.sp = h->sp8;
            // groups of the largest colour: no more blocks than they fill
            const uint64_t most = (uint64_t)d.gx[0] * (uint64_t)d.cnt[1][0] * (uint64_t)d.cnt[2][0];
            const int threads = most >= (uint64_t)h->sms * kSpaceThreads ? kSpaceThreads : kSpaceSmall;
            SpaceKernel sk = threads == kSpaceThreads ? space_kernel_of<kSpaceThreads>(h) : space_kernel_of<kSpaceSmall>(h);
            int per_sm = 0;
            VCA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sk, threads, 0));
            const int sgrid = (int)std::max<uint64_t>(1, std::min<uint64_t>((most + threads - 1) / threads, (uint64_t)h->sms * std::max(1, per_sm)));
            const int blocks = grid_for(bytes / 8, h->sms);
            mc_pack8_kernel<<<blocks, 256, 0, h->stream>>>(h->spin, h->sp8, va.nx, d.P8, rows);
            VCA_CUDA(cudaGetLastError());
            int n = count;
            void* args[] = {&va, &d, &n};
            VCA_CUDA(cudaLaunchCooperativeKernel((const void*)sk, sgrid, threads, args, 0, h->stream));
            mc_unpack8_kernel<<<blocks, 256, 0, h->stream>>>(h->sp8, h->spin, va.nx, d.P8, rows);
            VCA_CUDA(cudaGetLastError());
            h->launches += 3;
        } else if (count > 0 && h->color_off.back() > 0) {
            if (vca_status s = want_lists(h)) return s;
            a = mc_args(h);
            McColors col;
            std::memset(&col, 0, sizeof(col));
            col.colors = h->colors;
            for (int c = 0; c <= h->colors; ++c) col.off[c] = h->color_off[c];
            for (int v = 0; v < 6; ++v) col.mask[v] = nb_mask(h->nb_host, v);
            int list_grid = 0, list_threads = 0;
            size_t list_smem = 0;
            if (list_bytes_shape(h, &col, &list_grid, &list_threads, &list_smem)) {
                if (vca_status s = sp8_reserve(h, list_bytes(h))) return s;
                McBytes b;
                std::memset(&b, 0, sizeof(b));
                b.sp = h->sp8;
                b.P8 = (uint32_t)space_pitch(h->desc.nx);
                b.qm1 = (uint32_t)h->desc.Q - 1u;
                b.qm1_inv = 0xFFFFFFFFu / b.qm1;
                b.qm1_2p32 = (uint32_t)((1ULL << 32) % b.qm1);
                b.uphill = h->desc.kT > 0.0;
                ListKernel kernel = list_kernel_of(h);
                VCA_CUDA(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kListSmemMax));
                int n = count;
                void* args[] = {&a, &col, &b, &n};
                    VCA_CUDA(cudaLaunchCooperativeKernel((const void*)kernel, list_grid, list_threads, args, list_smem, h->stream));
                h->launches += 1;
            } else {
            int grid = 1;
            size_t smem = 0;
            SweepsKernel kernel = sweeps_kernel_of(h);
            if (vca_status s = sweeps_launch_shape(h, kernel, &col, &grid, &smem)) return s;
            int n = count;
            void* args[] = {&a, &col, &n};
            VCA_CUDA(cudaLaunchCooperativeKernel((const void*)kernel, grid, kMcThreads, args, smem, h->stream));
            h->launches += 1;
            }
        } else if (count > 0) {
            // empty domain: the sweeps still count (sweepsDone)
            McCtrl* c = h->ctrl_host;
            VCA_CUDA(cudaMemcpyAsync(c, h->ctrl, sizeof(McCtrl), cudaMemcpyDeviceToHost, h->stream));
            VCA_CUDA(cudaStreamSynchronize(h->stream));
            c->sweeps += (uint32_t)count;
            VCA_CUDA(cudaMemcpyAsync(h->ctrl, c, sizeof(McCtrl), cudaMemcpyHostToDevice, h->stream));
        }
        VCA_CUDA(cudaEventRecord(h->ev_b, h->stream));
        VCA_CUDA(cudaEventSynchronize(h->ev_b));
        float ms = 0.f;
        VCA_CUDA(cudaEventElapsedTime(&ms, h->ev_a, h->ev_b));
        h->total_ms += ms;
        if (count > 0 && h->color_off.back() > 0) h->mirrored = true;  // handed over by the launch
        else if (vca_status s_ = mc_sync(h)) return s_;
        if (h->ctrl_host->error) {
            set_error("vca_mc_sweep: a bounded grid-barrier wait ran out");
            return VCA_ERR_TIMEOUT;
        }
        if (accepted) *accepted = h->ctrl_host->sweep_accepted;
        return VCA_OK;
    }
    if (vca_status s = want_lists(h)) return s;
    a = mc_args(h);
    VCA_CUDA(cudaEventRecord(h->ev_a, h->stream));
    const bool random_nb = h->nb_host.variants > 1;
    size_t ev_used = 0;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> prof;
    for (int s = 0; s < count; ++s) {
        for (int c = 0; c < h->colors; ++c) {
            const uint64_t b = h->color_off[c], e = h->color_off[c + 1];
            const uint64_t cnt = e - b;
            const int grid = grid_for(cnt, h->sms);
            const uint32_t* list = h->list + b;
            const float* mob = h->mobility_on ? h->list_mob + b : nullptr;
            const int last = c == h->colors - 1;
            cudaEvent_t e0 = nullptr, e1 = nullptr;
            if (h->profile_kernels) {
                while (h->prof_events.size() < ev_used + 2) {
                    cudaEvent_t ev;
                    VCA_CUDA(cudaEventCreate(&ev));
                    h->prof_events.push_back(ev);
                }
                e0 = h->prof_events[ev_used];
                e1 = h->prof_events[ev_used + 1];
                ev_used += 2;
                VCA_CUDA(cudaEventRecord(e0, h->stream));
            }
            if (h->mobility_on) {
                if (random_nb) mc_color_kernel<true, true><<<grid, kMcThreads, 0, h->stream>>>(a, list, mob, cnt, last);
                else mc_color_kernel<true, false><<<grid, kMcThreads, 0, h->stream>>>(a, list, mob, cnt, last);
            } else {
                if (random_nb) mc_color_kernel<false, true><<<grid, kMcThreads, 0, h->stream>>>(a, list, mob, cnt, last);
                else mc_color_kernel<false, false><<<grid, kMcThreads, 0, h->stream>>>(a, list, mob, cnt, last);
            }
            if (h->profile_kernels) {
                VCA_CUDA(cudaEventRecord(e1, h->stream));
                prof.push_back({e0, e1});
            }
        }
        h->launches += (uint64_t)h->colors;
        if (h->profile_kernels && prof.size() > 2048) break;  // bounded event pool per call
    }
    VCA_CUDA(cudaGetLastError());
    VCA_CUDA(cudaEventRecord(h->ev_b, h->stream));
    VCA_CUDA(cudaEventSynchronize(h->ev_b));
    float ms = 0.f;
    VCA_CUDA(cudaEventElapsedTime(&ms, h->ev_a, h->ev_b));
    h->total_ms += ms;
    for (auto& pr : prof) {
        float m = 0.f;
        VCA_CUDA(cudaEventElapsedTime(&m, pr.first, pr.second));
        h->color_ms += m;
        ++h->color_launches;
    }
    if (vca_status s_ = mc_sync(h)) return s_;
    if (accepted) *accepted = h->ctrl_host->sweep_accepted;
    return VCA_OK;
}

vca_status vca_mc_get_info(vca_mc* h, vca_mc_info* out) {
    if (vca_status s = mc_check(h)) return s;
    VCA_CUDA(cudaSetDevice(h->device));
    if (!h->mirrored)
        if (vca_status s_ = mc_sync(h)) return s_;
    out->sweeps = (int)h->ctrl_host->sweeps;
    out->colors = h->colors;
    out->domain_cells = h->initialized ? h->color_off.back() : 0;
    out->attempts = h->ctrl_host->attempts;
    out->accepted = h->ctrl_host->accepted;
    out->uphill = h->ctrl_host->uphill;
    out->kernel_launches = h->launches;
    return VCA_OK;
}

vca_status vca_mc_grains(vca_mc* h, int moore, double mobility_threshold, vca_mc_grain_stats* out) {
    if (vca_status s = mc_check(h)) return s;
    if (!out) {
        set_error("vca_mc_grains: null output");
        return VCA_ERR_ARG;
    }
    if (!h->initialized) {
        set_error("vca_mc_grains: initialize first");
        return VCA_ERR_STATE;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    if (!h->gparent) {
        VCA_CUDA(cudaMalloc(&h->gparent, 4 * h->cap_n));
        VCA_CUDA(cudaMalloc(&h->gsize, 4 * h->cap_n));
        VCA_CUDA(cudaMalloc(&h->ghigh, 4 * h->cap_n));
        VCA_CUDA(cudaMalloc(&h->gacc, sizeof(GrainAcc)));
        VCA_CUDA(cudaMemsetAsync(h->gacc, 0, sizeof(GrainAcc), h->stream));
        VCA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&h->grain_per_sm, mc_grains_kernel, kGrainThreads, 0));
        h->grain_per_sm = std::max(1, std::min(h->grain_per_sm, 4 * 256 / kGrainThreads));  // more blocks lengthen its barriers
    }
    GrainAcc* acc = static_cast<GrainAcc*>(h->gacc);
    uint64_t total = h->color_off.back();
    McArgs a = mc_args(h);
    const float* mob = h->mobility_set ? h->mobility : nullptr;
    *h->gacc_host = GrainAcc{};
    if (total) {
        const int grid = (int)std::min<uint64_t>((total + kGrainThreads - 1) / kGrainThreads, (uint64_t)h->sms * h->grain_per_sm);
        const uint32_t* list = total < h->n ? h->list : nullptr;  // none: every cell in order (also where there is a list)
        GrainAcc* out = h->gacc_host_dev;
        void* args[] = {&a, &list, &total, &moore, &mob, &mobility_threshold, &h->gparent, &h->gsize, &h->ghigh, &acc, &out};
        VCA_CUDA(cudaLaunchCooperativeKernel((const void*)mc_grains_kernel, grid, kGrainThreads, args, 0, h->stream));
        h->launches += 1;
    }
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    const GrainAcc r = *h->gacc_host;
    if (total && r.left == 0) {  // some blocks left early: nobody zeroed the counters
        VCA_CUDA(cudaMemsetAsync(acc, 0, sizeof(GrainAcc), h->stream));
        VCA_CUDA(cudaMemsetAsync(&h->ctrl->bar_arrived, 0, sizeof(unsigned long long), h->stream));
        set_error("vca_mc_grains: a bounded grid-barrier wait ran out");
        return VCA_ERR_TIMEOUT;
    }
    if (r.error) {
        set_error("vca_mc_grains: a bounded union-find loop ran out");
        return VCA_ERR_TIMEOUT;
    }
    out->grains = r.grains;
    out->cells = r.cells;
    out->largest = r.largest;
    out->high_cells = r.high_cells;
    out->high_grains = r.high_grains;
    out->high_grain_cells = r.high_in;
    out->high_largest = r.high_largest;
    out->low_grains = r.low_grains;
    out->low_grain_cells = r.low_in;
    out->low_largest = r.low_largest;
    return VCA_OK;
}

vca_status vca_mc_set_mobility_values(vca_mc* h, const float* mobility, int use_in_dynamics) {
    if (vca_status s = vca_mc_set_mobility(h, mobility)) return s;
    if (mobility) h->mobility_on = use_in_dynamics != 0;
    return VCA_OK;
}

vca_status vca_mc_energy(vca_mc* h, double* energy) {
    if (vca_status s = mc_check(h)) return s;
    if (!h->initialized) {
        set_error("vca_mc_energy: initialize first");
        return VCA_ERR_STATE;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    const uint64_t total = h->color_off.back();
    const bool forward = h->nb_host.variants == 1;
    if (total) {
        McMasks m;
        for (int v = 0; v < 6; ++v) m.of[v] = nb_mask(h->nb_host, v);
        const uint32_t* list = total < h->n ? h->list : nullptr;  // none: every cell in order
        const int grid = std::min(grid_for(total, h->sms), h->sms * 4);  // more blocks queue at its atomics
        if (forward) mc_energy_kernel<true><<<grid, kMcThreads, 0, h->stream>>>(mc_args(h), m, list, total);
        else mc_energy_kernel<false><<<grid, kMcThreads, 0, h->stream>>>(mc_args(h), m, list, total);
    }
    h->launches += total ? 1 : 0;
    VCA_CUDA(cudaGetLastError());
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    if (total) h->mirrored = true;
    const double unlike = total ? (double)h->ctrl_host->energy_acc : 0.0;
    *energy = forward ? h->desc.J * unlike : 0.5 * h->desc.J * unlike;
    return VCA_OK;
}

vca_status vca_mc_crystals(vca_mc* h, int32_t* out) {
    if (vca_status s = mc_check(h)) return s;
    VCA_CUDA(cudaSetDevice(h->device));
    VCA_CUDA(cudaMemcpyAsync(out, h->spin, 4 * h->n, cudaMemcpyDeviceToHost, h->stream));
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    return VCA_OK;
}

vca_status vca_mc_set_spins(vca_mc* h, const int32_t* spins) {
    if (vca_status s = mc_check(h)) return s;
    if (!spins) {
        set_error("vca_mc_set_spins: null spins");
        return VCA_ERR_ARG;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    VCA_CUDA(cudaMemcpyAsync(h->spin, spins, 4 * h->n, cudaMemcpyHostToDevice, h->stream));
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    h->user_spins = true;
    return VCA_OK;
}

vca_status vca_mc_set_slab(vca_mc* h, int z_offset) {
    if (vca_status s = mc_check(h)) return s;
    if (z_offset < 0 || h->per[2] || h->desc.nz < 2) {
        set_error("vca_mc_set_slab: a slab needs z_offset >= 0, nz > 1 and no periodic z axis");
        return VCA_ERR_ARG;
    }
    if (h->initialized) {
        set_error("vca_mc_set_slab: set the slab before vca_mc_initialize");
        return VCA_ERR_STATE;
    }
    h->slab_zoff = z_offset;
    return VCA_OK;
}

vca_status vca_mc_color_pass(vca_mc* h, int color) {
    if (vca_status s = mc_check(h)) return s;
    if (!h->initialized) {
        set_error("vca_mc_color_pass: initialize first");
        return VCA_ERR_STATE;
    }
    if (color < 0 || color >= h->colors) {
        set_error("vca_mc_color_pass: colour out of range");
        return VCA_ERR_ARG;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    h->mirrored = false;
    if (vca_status s = want_lists(h)) return s;
    const McArgs a = mc_args(h);
    const uint64_t b = h->color_off[color], cnt = h->color_off[color + 1] - b;
    const int grid = grid_for(cnt, h->sms);
    const uint32_t* list = h->list + b;
    const float* mob = h->mobility_on ? h->list_mob + b : nullptr;
    const int last = color == h->colors - 1;
    const bool random_nb = h->nb_host.variants > 1;
    if (h->mobility_on) {
        if (random_nb) mc_color_kernel<true, true><<<grid, kMcThreads, 0, h->stream>>>(a, list, mob, cnt, last);
        else mc_color_kernel<true, false><<<grid, kMcThreads, 0, h->stream>>>(a, list, mob, cnt, last);
    } else {
        if (random_nb) mc_color_kernel<false, true><<<grid, kMcThreads, 0, h->stream>>>(a, list, mob, cnt, last);
        else mc_color_kernel<false, false><<<grid, kMcThreads, 0, h->stream>>>(a, list, mob, cnt, last);
    }
    VCA_CUDA(cudaGetLastError());
    h->launches += 1;
    return VCA_OK;
}

static vca_status spin_layers(vca_mc* h, int z0, int layers, void* buf, bool to_buf, const char* who) {
    if (vca_status s = mc_check(h)) return s;
    if (buf == nullptr || z0 < 0 || layers < 0 || z0 + layers > h->desc.nz) {
        set_error(std::string(who) + ": layers outside the grid or null buffer");
        return VCA_ERR_ARG;
    }
    VCA_CUDA(cudaSetDevice(h->device));
    const size_t L = (size_t)h->desc.nx * h->desc.ny;
    int32_t* dev = h->spin + (size_t)z0 * L;
    const size_t bytes = (size_t)layers * L * sizeof(int32_t);
    if (to_buf)
        VCA_CUDA(cudaMemcpyAsync(buf, dev, bytes, cudaMemcpyDefault, h->stream));
    else {
        VCA_CUDA(cudaMemcpyAsync(dev, buf, bytes, cudaMemcpyDefault, h->stream));
        h->user_spins = true;
    }
    VCA_CUDA(cudaStreamSynchronize(h->stream));
    return VCA_OK;
}

vca_status vca_mc_pack_spins(vca_mc* h, int z0, int layers, void* buf) {
    return spin_layers(h, z0, layers, buf, true, "vca_mc_pack_spins");
}

vca_status vca_mc_unpack_spins(vca_mc* h, int z0, int layers, const void* buf) {
    return spin_layers(h, z0, layers, const_cast<void*>(buf), false, "vca_mc_unpack_spins");
}

vca_status vca_mc_timing(vca_mc* h, double* total_ms, double* color_kernel_ms, uint64_t* color_launches) {
    if (vca_status s = mc_check(h)) return s;
    if (total_ms) *total_ms = h->total_ms;
    if (color_kernel_ms) *color_kernel_ms = h->color_launches ? h->color_ms / (double)h->color_launches : 0.0;
    if (color_launches) *color_launches = h->color_launches;
    return VCA_OK;
}

void vca_mc_destroy(vca_mc* h) {
    if (!h) return;
    mc_free(h);
    delete h;
}

}  // extern "C"
