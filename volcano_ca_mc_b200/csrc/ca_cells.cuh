// ca_cells.cuh -- cell addressing, frame semantics and the candidate vote, shared by the tile kernels
// (ca.cu) and the front kernels (front.cu) of the lava CA.
#pragma once

#include <cuda_runtime.h>

#include "vca_device.cuh"
#include "vca_internal.h"

namespace vca {

constexpr int kMaxDrop = 16;        // LavaCA::kMaxDrop (LavaCA.hpp:1293)

// ------------------------------------------------------------------------------------------
// Addressing with the reference's frame semantics: a coordinate one step outside the interior is
// the opposite layer on a periodic axis, else the VOID frame (Boundary::applyWith,
// engine/src/core/Boundary.hpp:75-131).
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ int64_t pidx(const CaGeom& g, int x, int y, int z) {
    return (int64_t)x + (int64_t)g.P * ((int64_t)y + (int64_t)g.ny * z);
}
__device__ __forceinline__ bool wrap_axis(int& v, int n, int periodic) {
    if (v >= 0 && v < n) return true;
    if (!periodic || n == 1) return false;
    v = v < 0 ? v + n : v - n;
    return true;
}
__device__ __forceinline__ bool resolve(const CaGeom& g, int& x, int& y, int& z) {
    return wrap_axis(x, g.nx, g.per[0]) && wrap_axis(y, g.ny, g.per[1]) && wrap_axis(z, g.nz, g.per[2]);
}
// A halo coordinate of a tile: up to one cell outside [0, n) maps through the frame; further out
// (past a partial last tile) is outside the grid.
__device__ __forceinline__ bool halo_axis(int& v, int n, int periodic) {
    if (v > n) return false;
    return wrap_axis(v, n, periodic);
}
__device__ __forceinline__ bool solid_ground(int t) { return t == kRock || t == kBasalt; }
// resolve() for a neighbour one cell away, as selects instead of branches, so that the loads of
// all neighbours of a cell can be issued together.  v is only meaningful when the result is true.
__device__ __forceinline__ bool wrap1_sel(int& v, int n, int periodic) {
    const bool in = (unsigned)v < (unsigned)n;
    const int w = v < 0 ? v + n : v - n;
    v = in ? v : w;
    return in | ((periodic != 0) & (n > 1));
}
__device__ __forceinline__ bool resolve1_sel(const CaGeom& g, int& x, int& y, int& z) {
    const bool a = wrap1_sel(x, g.nx, g.per[0]), b = wrap1_sel(y, g.ny, g.per[1]), c = wrap1_sel(z, g.nz, g.per[2]);
    return a & b & c;
}

// CandidateVote (engine/src/ca/CaRules.hpp:127-183).
struct Vote {
    int n;
    int32_t ids[26];
    int counts[26];
    float max_temp[26];
    __device__ void add(int32_t id, float t) {
        for (int i = 0; i < n; ++i)
            if (ids[i] == id) {
                ++counts[i];
                max_temp[i] = fmaxf(max_temp[i], t);
                return;
            }
        ids[n] = id;
        counts[n] = 1;
        max_temp[n] = t;
        ++n;
    }
    // Most votes; ties: tied ids ascending, pick hashRand(seed, t, idx, TieBreak) % k.
    __device__ int winner(uint64_t prefix, uint64_t gidx) const {
        if (n == 1) return 0;
        int best = 0;
        for (int i = 0; i < n; ++i) best = max(best, counts[i]);
        int tied[26];
        int k = 0;
        for (int i = 0; i < n; ++i)
            if (counts[i] == best) tied[k++] = i;
        if (k == 1) return tied[0];
        for (int i = 1; i < k; ++i) {
            const int t = tied[i];
            int j = i;
            while (j > 0 && ids[tied[j - 1]] > ids[t]) {
                tied[j] = tied[j - 1];
                --j;
            }
            tied[j] = t;
        }
        const uint64_t r = hash_salt(hash_index(prefix, gidx), kSaltTieBreak);
        return tied[(int)(r % (uint64_t)k)];
    }
    __device__ bool overflow() const { return false; }
    __device__ void pick(uint64_t prefix, uint64_t gidx, int32_t* id, float* t) const {
        const int w = winner(prefix, gidx);
        *id = ids[w];
        *t = max_temp[w];
    }
};

// The same vote for up to 4 distinct flowIds, held in registers (every index is a compile-time
// constant after unrolling).  A fifth distinct id sets overflow; the caller then recounts with Vote.
struct SmallVote {
    int n;
    bool over;
    int32_t ids[4];
    int counts[4];
    float max_temp[4];
    __device__ void add(int32_t id, float t) {
        bool hit = false;
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (s < n && ids[s] == id) {
                ++counts[s];
                max_temp[s] = fmaxf(max_temp[s], t);
                hit = true;
            }
        if (hit) return;
        if (n == 4) {
            over = true;
            return;
        }
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (s == n) {
                ids[s] = id;
                counts[s] = 1;
                max_temp[s] = t;
            }
        ++n;
    }
    __device__ bool overflow() const { return over; }
    // Most votes; ties: the (r % k)-th smallest tied id, r = hashRand(seed, t, idx, TieBreak).
    __device__ void pick(uint64_t prefix, uint64_t gidx, int32_t* id, float* t) const {
        int best = 0;
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (s < n) best = max(best, counts[s]);
        int k = 0;
#pragma unroll
        for (int s = 0; s < 4; ++s) k += (s < n && counts[s] == best) ? 1 : 0;
        int want = 0;
        if (k > 1) want = (int)(hash_salt(hash_index(prefix, gidx), kSaltTieBreak) % (uint64_t)k);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (!(s < n && counts[s] == best)) continue;
            int rank = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) rank += (u < n && counts[u] == best && ids[u] < ids[s]) ? 1 : 0;
            if (rank == want) {
                *id = ids[s];
                *t = max_temp[s];
            }
        }
    }
};

// Warp-aggregated append of n entries (values v[0..n-1], n <= 4) per lane to list/count.
__device__ __forceinline__ void warp_append(uint32_t* list, unsigned int* count, uint32_t cap, int lane, unsigned n,
                                            const uint32_t* v) {
    unsigned incl = n;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned u = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if (lane >= off) incl += u;
    }
    unsigned base = 0;
    if (lane == 31 && incl) base = atomicAdd(count, incl);
    base = __shfl_sync(0xFFFFFFFFu, base, 31) + incl - n;
    for (unsigned j = 0; j < n; ++j)
        if (base + j < cap) list[base + j] = v[j];
}

}  // namespace vca
