// front.cu -- the ACTIVE schedule of the lava CA as a list of LAVA cells, stepped by one persistent
// cooperative launch.
//
// Only LAVA cells and AIR cells that a LAVA cell reaches can change in a step (the front set of
// LavaCA::frontCandidatesLayer, engine/src/ca/LavaCA.hpp:907-940).  A tile schedule still streams every
// cell of a tile that holds one of them, twice buffered; here a step touches the LAVA cells and the
// cells they reach, in place:
//   phase A (per LAVA cell)  its temperature of this step; whether it solidifies in it (updateLava's
//                            LAVA branch, LavaCA.hpp:1135-1151); for every AIR cell it reaches
//                            (gatherLavaCandidates / tryPonding seen from the source, LavaCA.hpp:443-519)
//                            its bit in that cell's mark, and an entry in the block's candidate list;
//   phase B (per candidate)  the vote among the marked sources of the cell's variant, the solidus test,
//                            the new LAVA cell (updateLava's AIR branch, LavaCA.hpp:1121-1134); of a cell
//                            listed more than once the entry that takes its mark decides it; the cells
//                            that solidify become BASALT.
// A grid barrier follows each phase.  Types are read only in phase A and written only in phase B; the
// temperatures that phase B reads are written only in phase A, so no plane needs a second buffer.  The
// drop depths of the AIR cells beside a LAVA cell are found by looking down their columns (dropDepth,
// LavaCA.hpp:404-414), so there is no plane of them to keep current.
//
// Most LAVA cells only cool:
//   quiet  no AIR below, beside or (where it could pond) above.  AIR never comes back, so for good;
//   idle   the last look found no cell to reach.  What it saw lies in its column and the eight beside
//          it, so it looks again only after a step that changed a type there (the column stamps).
// The others are gathered in shared memory and looked at by half a warp each, one lane per column.
//
// What bounds a step: with few cells (up to some 10^5) the latency of its chains -- list entry, types,
// the barrier's release and poll, mark, source temperatures, slot of the new cell, the second barrier --
// some 7 us with all SMs and 5 us in one block, whose barriers are __syncthreads; above that the list
// stream (9 bytes per LAVA cell from L2).  Against the tile schedule on one B200: 1024 x 1024 x 256,
// 800 steps, up to 1.0 M LAVA cells 208 -> 13.8 ms; 256 x 256 x 128, 400 steps 14.9 -> 2.8 ms;
// 512 x 1 x 256, 300 steps 8.1 -> 1.45 ms; classic 100^3, 70 steps 2.4 -> 1.2 ms; ten mixed jobs in a
// batch 19.8 -> 4.1 ms.  Three forms brought the last part of it (mid: 256 x 256 x 128, 3.3 -> 2.8 ms):
// slots held in registers while each thread has at most one; a block's births counted in shared memory, so
// that each block takes its slots of the list with one atomic; and votes among five and more sources of
// several flows by a warp, one lane per source (one thread counting them in local arrays held up the second
// barrier of every step with such a cell).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>

#include "ca_cells.cuh"
#include "vca.h"
#include "vca_device.cuh"
#include "vca_internal.h"

namespace vca {

constexpr int kFrontThreads = 1024;   // a single grid: one block per SM
// quiet and idle: above; vent: reheated while erupting; dead: solidified (its last temperature stays in
// the list until it is stored)
constexpr uint8_t kFrontQuiet = 1, kFrontVent = 2, kFrontDead = 4, kFrontIdle = 8, kFrontStored = 16;
constexpr int kWordBits = 10;         // barrier words count blocks in 10-bit fields
constexpr unsigned kWordMask = (1u << kWordBits) - 1u;

// Shared lists of a block of kThreads threads.  The queue is emptied when it is full; candidates and
// solidifying slots that do not fit are listed in global memory, births that do not fit one by one.
template <int kThreads>
struct FrontShared {
    static constexpr int kQueue = 2 * kThreads, kCand = 4 * kThreads, kSolid = kThreads;
    unsigned nqueue, ncand, nsolid, active, changed, born, base;
    unsigned long long word;    // the barrier word all blocks have arrived at, 0: gave up
    // phase A: the slots that look around (bit 31: vent), or with resident slots their threads; their cells
    // and temperatures.  Phase B: the cells born in this step
    uint32_t q_slot[kQueue];
    uint32_t q_cell[kQueue];
    float q_temp[kQueue];
    uint32_t cand[kCand], solid[kSolid];
    uint8_t flags[kThreads];    // resident slots: the flags of each thread's slot
};
constexpr uint32_t kVentBit = 1u << 31;
constexpr uint32_t kRun = 8;          // consecutive slots of a block

__device__ __forceinline__ void front_decode(const CaFrontArgs& k, uint32_t c, int& x, int& y, int& z) {
    uint32_t ux, uy;
    const uint32_t r = fast_divmod(c, k.div_nx, ux);
    z = (int)fast_divmod(r, k.div_ny, uy);
    x = (int)ux;
    y = (int)uy;
}

// The temperature of a LAVA cell after step t.
__device__ __forceinline__ float front_cool(const CaFrontArgs& k, float temp, bool vent, int64_t t) {
    return vent && t < (int64_t)k.eruption_steps ? k.erupt_temp : __fsub_rn(temp, k.cool_ambient);
}

__device__ __forceinline__ bool front_is_vent(const CaFrontArgs& k, int32_t flow, int x, int y, int z) {
    if (k.classic || flow <= 0 || flow >= k.vent_slots) return false;
    const int4 v = __ldg(k.vents + flow);
    return v.x == x && v.y == y && v.z == z;
}

__device__ __forceinline__ int axis_at(int c, int d, int n) {
    const int v = c + d;
    return v < 0 ? v + n : (v >= n ? v - n : v);
}

// dropDepth of an AIR cell at plane index p, level z, with two AIR cells below it: the run of AIR below
// it, at most 16 deep, and the support of the run's bottom cell.
__device__ __noinline__ int front_fall_depth(const uint8_t* type, int64_t p, int64_t zs, int z, int spill_level) {
    for (int i = 3; i <= kMaxDrop; i += 7) {
        uint8_t t[7];
#pragma unroll
        for (int j = 0; j < 7; ++j) t[j] = z - i - j >= 0 ? type[p - zs * (i + j)] : kRock;  // the floor supports
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            if (t[j] == kAir) continue;
            const bool sup = solid_ground(t[j]) || (t[j] == kLava && z - i - j < spill_level);
            return sup ? i + j - 1 : -1;
        }
    }
    return kMaxDrop;
}

// Lists the cell (cx, cy, cz) for phase B with this source's bit, for the lanes with `emit`: bit i means
// that the source is the neighbour at offset (i % 3 - 1, i / 3 % 3 - 1, i / 9 - 1) of the listed cell.
template <class S>
__device__ __forceinline__ void front_emit(const CaFrontArgs& k, S& s, uint32_t* over, bool emit, int lane, int cx, int cy, int cz,
                                           int bit) {
    const unsigned who = __ballot_sync(0xFFFFFFFFu, emit);
    if (!who) return;
    unsigned at = 0;
    if (lane == 0) at = atomicAdd(&s.ncand, (unsigned)__popc(who));
    at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(who & ((1u << lane) - 1u));
    if (!emit) return;
    uint32_t* mark = k.mark + pidx(k.g, cx, cy, cz);
    const uint32_t c = (uint32_t)(cx + k.g.nx * (cy + k.g.ny * cz));
    if (at < (unsigned)S::kCand) {
        atomicOr(mark, 1u << bit);  // no answer is waited for
        s.cand[at] = c;
    } else if (atomicOr(mark, 1u << bit) == 0u) {  // each cell at most once: the list cannot overflow
        k.work[atomicAdd(over, 1u)] = c;
    }
}

// Phase A for the queued LAVA cells of a lava grid: half a warp per cell, lane l < 9 in the column at
// (l % 3 - 1, l / 3 - 1) of it; lane 4 is the cell's own column.  Everything a lane needs short of a
// fall of more than two cells comes in one round of loads.
template <int kThreads>
__device__ __forceinline__ void front_look_lava(const CaFrontArgs& k, FrontShared<kThreads>& s, uint32_t* over, unsigned nq, bool resident) {
    const CaGeom& g = k.g;
    const int lane = threadIdx.x & 31, l = lane & 15, sh = lane & 16;
    const int i = l < 9 ? l : 4;
    const bool own = l == 4;
    const bool is_side = l < 9 && ((k.side_mask >> i) & 1u), is_diag = l < 9 && !own && ((k.umask >> (26 - i)) & 1u);
    const bool has_spill = k.spill != nullptr;
    const int64_t zs = (int64_t)g.P * g.ny;
    for (unsigned base = 2 * (threadIdx.x >> 5); base < nq; base += 2 * (kThreads / 32)) {  // uniform over the warp
        const unsigned j = base + (sh >> 4);
        const bool on = j < nq;
        int x, y, z;
        front_decode(k, s.q_cell[on ? j : base], x, y, z);
        int cx = x + i % 3 - 1, cy = y + i / 3 - 1;
        const bool in = (wrap1_sel(cx, g.nx, g.per[0]) & wrap1_sel(cy, g.ny, g.per[1])) && on && (is_side || is_diag || own);
        const int64_t q = pidx(g, cx, cy, z);
        // the cell beside (own column: the cell above), the two below it, its column's spill level
        int st = kVoid, under = kRock, under2 = kRock, csp = INT_MIN;
        if (in) {
            if (own ? z + 1 < g.nz : is_side) st = k.type[own ? q + zs : q];
            if (z > 0) under = k.type[q - zs];  // the floor supports
            if (z > 1) under2 = k.type[q - 2 * zs];
            if (has_spill) csp = __ldg(k.spill + cx + (int64_t)g.nx * cy);
        }
        // hasSupport of the cell over `under` and of the one over `under2` (LavaCA.hpp:390-399)
        const bool sup1 = solid_ground(under) || (under == kLava && z - 1 < csp);
        const bool sup2 = solid_ground(under2) || (under2 == kLava && z - 2 < csp);
        // the drop depth of an AIR cell beside; D(n) is the largest, at least 0 (computeDescent, LavaCA.hpp:551-566)
        const bool air = in && !own && st == kAir;
        int v = -1;
        if (air) {
            if (sup1) v = 0;
            else if (under == kAir) v = under2 == kAir ? front_fall_depth(k.type, q, zs, z, csp) : (sup2 ? 1 : -1);
        }
        int d = max(v, 0);
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) d = max(d, __shfl_xor_sync(0xFFFFFFFFu, d, off));
        auto half = [&](bool b) { return (__ballot_sync(0xFFFFFFFFu, b) >> sh) & 0xFFFFu; };
        const unsigned airs = half(air);
        const bool supported = half(in && own && sup1) != 0;
        const bool below_air = half(in && own && under == kAir) != 0;
        // ponding (tryPonding, LavaCA.hpp:443-461): up to the spill level, supported, closed on every face
        // (AIR and the frame are open)
        const bool can_pond = half(in && own && k.ponding && st == kAir && z + 1 <= csp) != 0;
        const unsigned closed = half(in && st != kAir && st != kVoid);
        const unsigned faces = g.ny > 1 ? 0xAAu : 0x28u;
        const bool pond = can_pond && supported && (closed & faces) == faces;
        const bool falls = d == 1 && k.diag_falls;
        // each lane reaches at most one cell: own column: the one below (a fall, always) or above (a pond);
        // beside: the cells with drop depth D(n), or with D(n) = 1 and diagonal falls the cells diagonally
        // below that stand on something
        const bool e_side = air && supported && v == d && !falls;
        const bool e_down = own ? in && under == kAir : in && is_diag && supported && falls && under == kAir && sup2;
        const bool e_up = in && own && pond;
        const int dz = e_down ? -1 : (e_up ? 1 : 0);
        const bool emit = e_side || e_down || e_up;
        const bool any = half(emit) != 0;
        front_emit(k, s, over, emit, lane, cx, cy, z + dz, 17 - i - 9 * dz);
        if (on && own) {
            const uint32_t qs = s.q_slot[j];
            if (any) k.temp[q] = s.q_temp[j];  // what the votes read
            const uint8_t fl = (qs & kVentBit ? kFrontVent : 0) | (any ? 0 : kFrontIdle) |
                               (!below_air && airs == 0 && !can_pond ? kFrontQuiet : 0);
            *(resident ? s.flags + (qs & ~kVentBit) : k.flags + (qs & ~kVentBit)) = fl;
        }
    }
}

// Phase A for the queued grain cells of a classic grid: every AIR cell of the neighbourhood, lane l at
// the offsets l and l + 16.
template <int kThreads>
__device__ __forceinline__ void front_look_classic(const CaFrontArgs& k, FrontShared<kThreads>& s, uint32_t* over, unsigned nq, bool resident) {
    const CaGeom& g = k.g;
    const int lane = threadIdx.x & 31, l = lane & 15, sh = lane & 16;
    for (unsigned base = 2 * (threadIdx.x >> 5); base < nq; base += 2 * (kThreads / 32)) {
        const unsigned j = base + (sh >> 4);
        const bool on = j < nq;
        int x, y, z;
        front_decode(k, s.q_cell[on ? j : base], x, y, z);
        bool emit[2];
        int cx[2], cy[2], cz[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int i = l + 16 * r;  // the cell at offset d has this one at offset -d: bit 26 - i
            cx[r] = x + i % 3 - 1;
            cy[r] = y + i / 3 % 3 - 1;
            cz[r] = z + i / 9 - 1;
            const bool in = on && i < 27 && i != 13 && ((k.umask >> ((26 - i) & 31)) & 1u) && resolve1_sel(g, cx[r], cy[r], cz[r]);
            emit[r] = in && k.type[pidx(g, cx[r], cy[r], cz[r])] == kAir;
        }
        const bool any = ((__ballot_sync(0xFFFFFFFFu, emit[0] || emit[1]) >> sh) & 0xFFFFu) != 0;
#pragma unroll
        for (int r = 0; r < 2; ++r) front_emit(k, s, over, emit[r], lane, cx[r], cy[r], cz[r], 26 - (l + 16 * r));
        if (on && l == 0) *(resident ? s.flags + s.q_slot[j] : k.flags + s.q_slot[j]) = any ? 0 : kFrontQuiet;  // no AIR around: for good
    }
}

// r % n for 1 <= n <= 26, r = hashRand(seed, t, idx, TieBreak), by the halves of r: 2^32 is (2^32 - 1) % n + 1
// modulo n.
__device__ __forceinline__ unsigned front_tie(uint64_t prefix, uint64_t cell, unsigned n) {
    const uint64_t h = hash_salt(hash_index(prefix, cell), kSaltTieBreak);
    return (((uint32_t)(h >> 32) % n) * (0xFFFFFFFFu % n + 1u) + (uint32_t)h % n) % n;
}

// One source of a candidate at (x, y, z): bit i of its mark.
template <bool kClassic>
__device__ __forceinline__ void front_source(const CaFrontArgs& k, int x, int y, int z, int i, int32_t& flow, float& temp) {
    const CaGeom& g = k.g;
    const int64_t q = pidx(g, axis_at(x, i % 3 - 1, g.nx), axis_at(y, i / 3 % 3 - 1, g.ny), axis_at(z, i / 9 - 1, g.nz));
    flow = k.flow[q];
    // the source wrote its temperature of this step there; one above falls, the others spread
    temp = kClassic ? 0.0f : __fsub_rn(k.temp[q], i >= 18 ? k.cool_fall : k.cool_lateral);
}

// The vote among five and more sources `m` of several flows (CandidateVote, CaRules.hpp:127-183), a warp
// for the candidate, lane i for source i; the winner in every lane.
template <bool kClassic>
__device__ __forceinline__ void front_vote(const CaFrontArgs& k, uint32_t c, uint32_t m, uint32_t t, int lane, int32_t& flow,
                                           float& temp) {
    int x, y, z;
    front_decode(k, c, x, y, z);
    const bool have = (m >> lane) & 1u;
    int32_t fl = 0;
    float te = 0.0f;
    if (have) front_source<kClassic>(k, x, y, z, lane, fl, te);
    const unsigned alike = __match_any_sync(0xFFFFFFFFu, fl) & m;
    const bool lead = have && lane == __ffs(alike) - 1;
    const int votes = lead ? __popc(alike) : 0, best = __reduce_max_sync(0xFFFFFFFFu, votes);
    const unsigned tied = __ballot_sync(0xFFFFFFFFu, lead && votes == best), ties = __popc(tied);
    // ties: the (r % ties)-th smallest tied id
    const unsigned want = ties > 1 ? front_tie(hash_prefix(k.seed, t), c, ties) : 0u;
    unsigned rank = 0;
    for (unsigned r = tied; r; r &= r - 1) rank += __shfl_sync(0xFFFFFFFFu, fl, __ffs(r) - 1) < fl;
    const unsigned won = __ballot_sync(0xFFFFFFFFu, lead && votes == best && rank == want);
    const int src = __ffs(won) - 1;
    flow = __shfl_sync(0xFFFFFFFFu, fl, src);
    const unsigned of = __shfl_sync(0xFFFFFFFFu, alike, src);
    temp = __shfl_sync(0xFFFFFFFFu, te, src);
    for (unsigned r = of; r; r &= r - 1) temp = fmaxf(temp, __shfl_sync(0xFFFFFFFFu, te, __ffs(r) - 1));
}

// Phase B for one candidate: returns true when it becomes LAVA with (nf, nt); `hard` gets its sources when
// five or more of several flows have to be counted (front_vote; the result is then false).
template <bool kClassic>
__device__ __forceinline__ bool front_decide(const CaFrontArgs& k, uint32_t c, int x, int y, int z, int64_t p, uint32_t t,
                                             int32_t& nf, float& nt, uint32_t& hard) {
    const uint32_t m = atomicExch(k.mark + p, 0u);
    const int var =
        k.variants == 1 ? 0 : (int)fast_mod(hash_salt(hash_index(hash_prefix(k.seed, t), c), kSaltNeighborhood), k.var_mod);
    const uint32_t use = m & k.vmask[var];
    if (!use) return false;
    // four sources a round; the slots past the last one hold the first again
    const int n = __popc(use);
    int32_t fl[4];
    float te[4];
    uint32_t r = use;
    bool same = true;
    auto fetch = [&]() {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            fl[q] = q ? fl[0] : nf;
            te[q] = q ? te[0] : nt;
            if (!r) continue;
            front_source<kClassic>(k, x, y, z, __ffs(r) - 1, fl[q], te[q]);
            r &= r - 1;
        }
    };
    auto fold = [&]() {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            same = same && fl[q] == nf;
            nt = fmaxf(nt, te[q]);
        }
    };
    fetch();
    nf = fl[0];
    nt = te[0];
    fold();
    // sources of one flow need no vote: its highest temperature decides
    if (n > 4) {
        while (r) {
            fetch();
            fold();
        }
        if (!same) {
            hard = use;
            return false;
        }
    } else if (!same) {
        // the vote among two to four: most votes; ties: the (r % ties)-th smallest tied id
        int votes[4], best = 0;
        float most[4];
        bool lead[4];  // the first source of its flow
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            votes[i] = 0;
            most[i] = te[i];
            lead[i] = i < n;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool alike = j < n && fl[j] == fl[i];
                votes[i] += alike;
                if (alike) most[i] = fmaxf(most[i], te[j]);
                if (alike && j < i) lead[i] = false;
            }
            if (lead[i]) best = max(best, votes[i]);
        }
        unsigned ties = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            lead[i] = lead[i] && votes[i] == best;
            ties += lead[i];
        }
        const unsigned want = ties > 1 ? front_tie(hash_prefix(k.seed, t), c, ties) : 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            unsigned rank = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) rank += lead[j] && fl[j] < fl[i];
            if (lead[i] && rank == want) {
                nf = fl[i];
                nt = most[i];
            }
        }
    }
    return kClassic || nt >= k.solidus;
}

// Thread 0's half of the barrier of a grid's `nblk` blocks: adds `add` (one arrival in the low field) to
// the word with release semantics and polls it with acquire loads until every block has arrived; the
// word then holds the sums of all blocks' fields.  __syncthreads on both sides.  The wait is bounded; a
// block that gives up, or sees that another gave up, gets 0 with ctrl->error set.
__device__ __forceinline__ unsigned long long front_arrive(CaCtrl* ctrl, unsigned long long* word, unsigned long long add,
                                                           uint32_t nblk) {
    if (nblk == 1) return add;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;\n" ::"l"(word), "l"(add) : "memory");
    for (int spins = 0;; ++spins) {
        unsigned long long v;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(word) : "memory");
        if (((unsigned)v & kWordMask) == nblk) return v;
        if (spins > (1 << 26) || ((spins & 1023) == 1023 && *(volatile int*)&ctrl->error)) {
            atomicOr(&ctrl->error, 1);
            return 0ull;
        }
    }
}

// The cells of the column at (i % 3 - 1, i / 3 - 1) of cell c's look again in step t + 1: a type changed
// at c in step t.
__device__ __forceinline__ void front_stamp(const CaFrontArgs& k, uint32_t c, int i, uint32_t t) {
    int x, y, z;
    front_decode(k, c, x, y, z);
    x += i % 3 - 1;
    y += i / 3 - 1;
    if (wrap1_sel(x, k.g.nx, k.g.per[0]) & wrap1_sel(y, k.g.ny, k.g.per[1])) k.stamp[x + (int64_t)k.g.nx * y] = t;
}

// Up to `steps` steps of one grid by its `nblk` blocks (block `bid`), until its stop rule holds or its
// list has grown beyond `most` slots.
//
// The list goes round the blocks in runs of 8 slots, a sector of each array: the cells that look around
// lie together (the last ones born first of all) and are shared out.  While the list is no longer than the
// launch has threads, a slot is resident in its thread: its cell and temperature stay in registers, its flags in shared memory, so that a step starts with one load (an idle cell's stamp)
// instead of three dependent ones.  A longer list is streamed, four slots per thread.
template <int kThreads, bool kClassic>
__device__ __forceinline__ void front_body(const CaFrontArgs& k, FrontShared<kThreads>& s, uint32_t bid, uint32_t nblk, int steps,
                                           uint32_t most, CaCtrl* snap) {
    using S = FrontShared<kThreads>;
    CaCtrl* ctrl = k.ctrl;
    if (ctrl->stop || ctrl->error) return;  // neither changes before every block has passed the first barrier
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t T = nblk * kThreads;
    const uint32_t t_first = ctrl->steps;
    uint32_t t = t_first, n = ctrl->front_n, prev = ctrl->front_prev;
    uint64_t air = ctrl->air, visited = 0;
    int stop = VCA_STOP_RUNNING;
    bool ok = true;
    // the resident slot of this thread, once the list reaches it
    bool resident = n <= T, have = false, dying = false;
    const uint32_t my_slot = ((uint32_t)(tid / kRun) * nblk + bid) * kRun + tid % kRun;
    uint32_t my_cell = 0, my_col = 0;
    float my_temp = 0.0f;
    if (tid == 0) s.nqueue = s.ncand = s.nsolid = s.active = s.changed = s.born = 0;
    __syncthreads();
    auto column = [&](uint32_t cell) -> uint32_t {
        uint32_t x, y;
        const uint32_t r = fast_divmod(cell, k.div_nx, x);
        fast_divmod(r, k.div_ny, y);
        return x + (uint32_t)k.g.nx * y;
    };
    auto stamp_type = [&](uint32_t c) {
        for (int i = 0; i < 9; ++i) front_stamp(k, c, i, t);
    };
    // the resident slots back into the list
    auto write_back = [&]() {
        if (!have) return;
        k.flags[my_slot] = s.flags[tid];
        if (!kClassic) k.ltemp[my_slot] = my_temp;
    };
    while (t - t_first < (uint32_t)steps && stop == VCA_STOP_RUNNING && n <= most) {
        uint32_t* over = ctrl->front_over[t % 3u];
        unsigned my_active = 0, my_changed = 0;
        if (resident && n > T) {  // outgrown: the same blocks go on with the same runs from memory
            write_back();
            resident = have = false;
            __syncthreads();
        }
        auto look = [&]() {
            __syncthreads();
            const unsigned nq = min(s.nqueue, (unsigned)S::kQueue);
            if (kClassic) front_look_classic(k, s, over, nq, resident);
            else front_look_lava(k, s, over, nq, resident);
        };
        // ---- phase A
        if (resident) {
            unsigned fl = 0;
            uint32_t seen = t - 1u;
            if (have) {
                fl = s.flags[tid];
                if ((fl & (kFrontIdle | kFrontQuiet | kFrontDead)) == kFrontIdle) seen = k.stamp[my_col];
            } else if (my_slot < n) {
                have = true;
                fl = k.flags[my_slot];
                my_cell = k.idx[my_slot];
                if (!kClassic) my_temp = k.ltemp[my_slot];
                my_col = column(my_cell);
                s.flags[tid] = (uint8_t)fl;
                if ((fl & (kFrontIdle | kFrontQuiet | kFrontDead)) == kFrontIdle) seen = k.stamp[my_col];
            }
            if (have) {
                const bool vent = (fl & kFrontVent) != 0;
                if (fl & kFrontDead) {
                    if (!kClassic && !(fl & kFrontStored)) {  // its last temperature, now that no vote reads it
                        int x, y, z;
                        front_decode(k, my_cell, x, y, z);
                        k.temp[pidx(k.g, x, y, z)] = my_temp;
                        s.flags[tid] = (uint8_t)(fl | kFrontStored);
                    }
                } else {
                    if (kClassic) {
                        ++my_active;
                    } else {
                        if (my_slot < prev) my_temp = front_cool(k, my_temp, vent, (int64_t)t - 1);  // the update of the last step
                        const float next = front_cool(k, my_temp, vent, t);
                        dying = next < k.solidus;
                        if (dying) {
                            ++my_changed;
                            s.nsolid = 1;  // there is work for phase B
                        } else {
                            ++my_active;
                            my_changed += next != my_temp;
                        }
                    }
                    if (!(fl & kFrontQuiet) && seen == t - 1u) {  // an idle cell: the last step changed a type around its column
                        const unsigned at = atomicAdd(&s.nqueue, 1u);  // kQueue >= kThreads
                        s.q_slot[at] = (uint32_t)tid | (vent ? kVentBit : 0u);
                        s.q_cell[at] = my_cell;
                        s.q_temp[at] = my_temp;
                    }
                }
            }
            look();
        } else {
            // four slots per thread, two threads per run; a full queue is emptied in between
            for (uint32_t run0 = 0; run0 * nblk * kRun < n; run0 += 4 * kThreads / kRun) {  // uniform over the block
                const uint32_t base = ((run0 + tid / 2) * nblk + bid) * kRun + 4 * (tid % 2);
                unsigned want = 0;
                uint32_t f4 = 0;
                float te[4] = {0.f, 0.f, 0.f, 0.f};
                uint32_t cell[4] = {0, 0, 0, 0};
                if (base < n) {
                    f4 = *reinterpret_cast<const uint32_t*>(k.flags + base);
                    if (!kClassic) {
                        const float4 t4 = *reinterpret_cast<const float4*>(k.ltemp + base);
                        te[0] = t4.x, te[1] = t4.y, te[2] = t4.z, te[3] = t4.w;
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t slot = base + j;
                        const unsigned fl = (f4 >> (8 * j)) & 0xFFu;
                        if (slot >= n || (fl & kFrontDead)) continue;
                        if (kClassic) {
                            ++my_active;
                        } else {
                            const bool vent = (fl & kFrontVent) != 0;
                            if (slot < prev) te[j] = front_cool(k, te[j], vent, (int64_t)t - 1);
                            const float next = front_cool(k, te[j], vent, t);
                            if (next < k.solidus) {
                                ++my_changed;
                                const unsigned at = atomicAdd(&s.nsolid, 1u);
                                if (at < (unsigned)S::kSolid) s.solid[at] = slot;
                                else k.work[k.work_cap - 1u - atomicAdd(&over[1], 1u)] = slot;
                            } else {
                                ++my_active;
                                my_changed += next != te[j];
                            }
                        }
                        if (!(fl & kFrontQuiet)) want |= 1u << j;
                    }
                    if (!kClassic) *reinterpret_cast<float4*>(k.ltemp + base) = make_float4(te[0], te[1], te[2], te[3]);
                    if (want) {
                        const uint4 c4 = *reinterpret_cast<const uint4*>(k.idx + base);
                        cell[0] = c4.x, cell[1] = c4.y, cell[2] = c4.z, cell[3] = c4.w;
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (((want >> j) & 1u) && ((f4 >> (8 * j)) & kFrontIdle) && k.stamp[column(cell[j])] != t - 1u)
                                want &= ~(1u << j);
                    }
                }
                for (;;) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (!((want >> j) & 1u)) continue;
                        const unsigned at = atomicAdd(&s.nqueue, 1u);
                        if (at >= (unsigned)S::kQueue) continue;
                        s.q_slot[at] = (base + j) | ((f4 >> (8 * j)) & kFrontVent ? kVentBit : 0u);
                        s.q_cell[at] = cell[j];
                        s.q_temp[at] = te[j];
                        want &= ~(1u << j);
                    }
                    if (!__syncthreads_or(want != 0)) break;
                    look();
                    __syncthreads();
                    if (tid == 0) s.nqueue = 0;
                    __syncthreads();
                }
            }
            look();
        }
        const unsigned wa = __reduce_add_sync(0xFFFFFFFFu, my_active), wc = __reduce_add_sync(0xFFFFFFFFu, my_changed);
        if (lane == 0) {
            if (wa) atomicAdd(&s.active, wa);
            if (wc) atomicAdd(&s.changed, wc);
        }
        __syncthreads();
        // ---- barrier: blocks with work for phase B, with active and with changed cells, with overflow lists
        unsigned long long wordA = 0;
        if (nblk == 1 || tid == 0) {
            const bool work = (s.ncand | s.nsolid) != 0, more = s.ncand > (unsigned)S::kCand || s.nsolid > (unsigned)S::kSolid;
            wordA = 1ull | ((unsigned long long)work << kWordBits) | ((unsigned long long)(s.active != 0) << 2 * kWordBits) |
                    ((unsigned long long)(s.changed != 0) << 3 * kWordBits) | ((unsigned long long)more << 4 * kWordBits);
            if (nblk > 1) s.word = front_arrive(ctrl, &ctrl->front_word[t % 3u][0], wordA, nblk);
        }
        if (tid == 32) {
            if (s.active) atomicAdd(&k.hist_active[t], (unsigned long long)s.active);
            if (s.changed) atomicAdd(&k.hist_changed[t], (unsigned long long)s.changed);
        }
        __syncthreads();
        if (nblk > 1) wordA = s.word;
        if (wordA == 0ull) {
            ok = false;
            break;
        }
        if (tid == 0) s.nqueue = s.active = s.changed = 0;  // used again after another __syncthreads
        if (bid == 0 && tid == 64) {  // step t + 2 starts at zero (its words' last readers passed the barrier above)
            const uint32_t r = (t + 2u) % 3u;
            ctrl->front_word[r][0] = ctrl->front_word[r][1] = 0ull;
            ctrl->front_over[r][0] = ctrl->front_over[r][1] = 0u;
        }
        auto field = [&](int i) { return (unsigned)(wordA >> (i * kWordBits)) & kWordMask; };
        uint32_t born = 0;
        if (field(1)) {
            // ---- phase B
            const uint16_t stamp = (uint16_t)min(t, 65535u);
            // births in the lower half of the queue's arrays, hard votes in the upper one
            auto birth = [&](uint32_t c, int x, int y, int z, int64_t p, int32_t nf, float nt) {
                k.type[p] = kLava;
                k.flow[p] = nf;
                k.temp[p] = nt;
                k.solid[p] = 0;
                k.arrival[p] = stamp;
                const bool vent = !kClassic && front_is_vent(k, nf, x, y, z);
                const unsigned at = atomicAdd(&s.born, 1u);
                if (at < (unsigned)kThreads) {
                    s.q_slot[at] = vent ? kVentBit : 0u;
                    s.q_cell[at] = c;
                    s.q_temp[at] = nt;
                } else {
                    const unsigned slot = atomicAdd(&ctrl->front_n, 1u);
                    k.idx[slot] = c;
                    k.ltemp[slot] = nt;
                    k.flags[slot] = vent ? kFrontVent : 0;
                    stamp_type(c);
                }
            };
            auto candidates = [&](uint32_t first, uint32_t count, uint32_t stride, const uint32_t* list) {
                for (uint32_t base = first; base < count; base += stride) {  // uniform over the block
                    uint32_t hard = 0;
                    if (base + tid < count) {
                        const uint32_t c = list[base + tid];
                        int x, y, z;
                        front_decode(k, c, x, y, z);
                        const int64_t p = pidx(k.g, x, y, z);
                        int32_t nf = 0;
                        float nt = 0.f;
                        if (front_decide<kClassic>(k, c, x, y, z, p, t, nf, nt, hard)) birth(c, x, y, z, p, nf, nt);
                        if (hard) {
                            const unsigned at = kThreads + atomicAdd(&s.nqueue, 1u);
                            s.q_slot[at] = hard;
                            s.q_cell[at] = c;
                        }
                    }
                    if (!__syncthreads_or(hard != 0)) continue;
                    const unsigned nh = s.nqueue;
                    for (unsigned j = warp; j < nh; j += kThreads / 32) {
                        const uint32_t c = s.q_cell[kThreads + j];
                        int32_t nf;
                        float nt;
                        front_vote<kClassic>(k, c, s.q_slot[kThreads + j], t, lane, nf, nt);
                        if (lane == 0 && (kClassic || nt >= k.solidus)) {
                            int x, y, z;
                            front_decode(k, c, x, y, z);
                            birth(c, x, y, z, pidx(k.g, x, y, z), nf, nt);
                        }
                    }
                    __syncthreads();
                    if (tid == 0) s.nqueue = 0;
                    __syncthreads();
                }
            };
            // A dead cell's temperature does not go into the plane yet: as a source of this step's votes the
            // cell still has the one before.
            auto solidify = [&](uint32_t c) {
                int x, y, z;
                front_decode(k, c, x, y, z);
                const int64_t p = pidx(k.g, x, y, z);
                k.type[p] = kBasalt;
                k.solid[p] = stamp;
                stamp_type(c);
            };
            auto solidify_slot = [&](uint32_t slot) {
                k.ltemp[slot] = front_cool(k, k.ltemp[slot], (k.flags[slot] & kFrontVent) != 0, t);
                k.flags[slot] = kFrontDead;
                solidify(k.idx[slot]);
            };
            __syncthreads();  // the queue counters are clear
            candidates(0, min(s.ncand, (unsigned)S::kCand), kThreads, s.cand);
            if (resident) {
                if (dying) {
                    my_temp = front_cool(k, my_temp, (s.flags[tid] & kFrontVent) != 0, t);
                    s.flags[tid] = kFrontDead;
                    dying = false;
                    solidify(my_cell);
                }
            } else {
                const uint32_t ns = min(s.nsolid, (unsigned)S::kSolid);
                for (uint32_t j = tid; j < ns; j += kThreads) solidify_slot(s.solid[j]);
            }
            if (field(4)) {  // overflow lists, shared by all blocks
                const uint32_t oc = __ldcg(&over[0]), os = __ldcg(&over[1]);
                candidates(bid * kThreads, oc, T, k.work);
                for (uint32_t j = bid * kThreads + tid; j < os; j += T) solidify_slot(__ldcg(k.work + (k.work_cap - 1u - j)));
            }
            __syncthreads();
            // the block's births: their place in the list, meanwhile the stamps around them
            const unsigned nb = s.born, listed = min(nb, (unsigned)kThreads);
            if (listed) {
                if (tid == 0) s.base = atomicAdd(&ctrl->front_n, listed);
                for (unsigned j = tid; j < 9u * listed; j += kThreads) front_stamp(k, s.q_cell[j / 9u], j % 9u, t);
                __syncthreads();
                for (unsigned j = tid; j < listed; j += kThreads) {
                    const unsigned slot = s.base + j;
                    k.idx[slot] = s.q_cell[j];
                    k.ltemp[slot] = s.q_temp[j];
                    k.flags[slot] = s.q_slot[j] ? kFrontVent : 0;
                }
                __syncthreads();
            }
            unsigned long long wordB = 1ull | ((unsigned long long)nb << kWordBits);
            if (tid == 0) {
                if (nblk > 1) s.word = front_arrive(ctrl, &ctrl->front_word[t % 3u][1], wordB, nblk);
                s.ncand = s.nsolid = 0;
            } else if (tid == 32 && nb) {
                atomicAdd(&k.hist_active[t], (unsigned long long)nb);
                atomicAdd(&k.hist_changed[t], (unsigned long long)nb);
            }
            __syncthreads();
            if (nblk > 1) wordB = s.word;
            if (wordB == 0ull) {
                ok = false;
                break;
            }
            if (tid == 0) s.born = 0;
            born = (uint32_t)(wordB >> kWordBits);
        }
        // ---- finishStep (LavaCA.hpp:1206-1229), the same in every block
        air -= born;
        visited += n;
        prev = n;
        n += born;
        ++t;
        if (!kClassic && !field(2) && !born) stop = VCA_STOP_NO_LAVA;
        else if (kClassic && air == 0) stop = VCA_STOP_NO_AIR;
        else if (!field(3) && !born && !k.random_nb) stop = VCA_STOP_NO_CHANGE;
        else if ((int)t >= k.max_steps) stop = VCA_STOP_MAX_STEPS;
        if (!field(1)) __syncthreads();  // the counters are clear before the next phase A
    }
    if (ok && resident) write_back();
    if (ok && !kClassic) {
        // the temperatures of the LAVA cells back into their plane, and once those of the dead ones
        auto store = [&](uint32_t slot, unsigned fl, uint32_t cell, float te) {
            if (fl & kFrontStored) return;
            if (fl & kFrontDead) k.flags[slot] = (uint8_t)(fl | kFrontStored);
            else if (slot < prev) te = front_cool(k, te, (fl & kFrontVent) != 0, (int64_t)t - 1);
            int x, y, z;
            front_decode(k, cell, x, y, z);
            k.temp[pidx(k.g, x, y, z)] = te;
        };
        if (resident) {
            // (a slot born in the last step is not resident yet; its plane has its temperature)
            if (have) store(my_slot, s.flags[tid], my_cell, my_temp);
        } else {
            for (uint32_t slot = bid * kThreads + tid; slot < n; slot += T) store(slot, k.flags[slot], k.idx[slot], k.ltemp[slot]);
        }
    }
    __syncthreads();
    if (warp != 0) return;
    bool last = false;
    if (lane == 0) {
        if (bid == 0 && ok && t != t_first) {
            ctrl->steps = t;
            ctrl->stop = stop;
            ctrl->air = air;
            ctrl->front_prev = prev;
            ctrl->tiles_processed += visited;  // cells here: vca_ca_get_info gives them in tiles
        }
        unsigned left;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n" : "=r"(left) : "l"(&ctrl->front_exit) : "memory");
        last = left == nblk - 1u;
        if (last) {  // the last block out: every block's totals are in
            ctrl->front_exit = 0;
            if (ok && t != t_first) ctrl->lava = __ldcg(&k.hist_active[t - 1u]);
        }
    }
    if (!__shfl_sync(0xFFFFFFFFu, (int)last, 0) || snap == nullptr) return;
    __syncwarp();
    const uint32_t* from = reinterpret_cast<const uint32_t*>(ctrl);
    volatile uint32_t* to = reinterpret_cast<volatile uint32_t*>(snap);
    for (int i = lane; i < (int)(sizeof(CaCtrl) / sizeof(uint32_t)); i += 32) to[i] = __ldcg(from + i);
}

template <int kThreads, bool kClassic>
__global__ __launch_bounds__(kThreads, 1) void ca_front_kernel(const __grid_constant__ CaFrontArgs k, int steps, uint32_t most,
                                                               CaCtrl* snap) {
    __shared__ FrontShared<kThreads> s;
    front_body<kThreads, kClassic>(k, s, blockIdx.x, gridDim.x, steps, most, snap);
}

// Many grids in one launch: a block serves one member, `n[slot]` blocks share a member's steps and its
// barrier (CaFrontBatch).
__global__ __launch_bounds__(kFrontBatchThreads, 4) void ca_front_batch_kernel(const __grid_constant__ CaFrontBatch b, int steps) {
    const int2 m = b.map[blockIdx.x];
    if (m.x < 0) return;
    __shared__ __align__(16) CaFrontArgs s_k;
    __shared__ FrontShared<kFrontBatchThreads> s;
    static_assert(sizeof(CaFrontArgs) % sizeof(uint2) == 0, "copied as 8-byte words");
    const uint2* from = reinterpret_cast<const uint2*>(b.args + m.x);
    for (int i = threadIdx.x; i < (int)(sizeof(CaFrontArgs) / sizeof(uint2)); i += blockDim.x)
        reinterpret_cast<uint2*>(&s_k)[i] = from[i];
    __syncthreads();
    if (s_k.classic) front_body<kFrontBatchThreads, true>(s_k, s, (uint32_t)m.y, (uint32_t)b.n[m.x], steps, 0xFFFFFFFFu, nullptr);
    else front_body<kFrontBatchThreads, false>(s_k, s, (uint32_t)m.y, (uint32_t)b.n[m.x], steps, 0xFFFFFFFFu, nullptr);
}

// The front list of the current planes: every LAVA cell, 16 cells of a row per thread (a row is a
// multiple of 64 cells); the scratch of the steps cleared on the way.  With `snap` also the LAVA and AIR
// cells of the grid and the stop state they give (countInitialState, LavaCA.hpp:1252-1280), which the last
// block leaves in the control block and in host-mapped memory.  Reads one byte per cell and writes four.
__global__ __launch_bounds__(256) void ca_front_list_kernel(const __grid_constant__ CaFrontArgs k, uint64_t cells, int t0, CaCtrl* snap) {
    const int lane = threadIdx.x & 31;
    const uint64_t chunks = cells / 16, stride = (uint64_t)gridDim.x * blockDim.x, me = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    unsigned long long air = 0;
    for (uint64_t i = me; i < cells / 4; i += stride) reinterpret_cast<uint4*>(k.mark)[i] = make_uint4(0, 0, 0, 0);
    for (uint64_t i = me; i < (uint64_t)k.g.nx * k.g.ny; i += stride) k.stamp[i] = 0xFFFFFFFFu;  // no step
    if (snap)  // the steps to come add their totals up in the histories
        for (int64_t t = t0 + (int64_t)me; t < k.max_steps; t += stride) k.hist_active[t] = k.hist_changed[t] = 0;
    for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x; base < chunks; base += stride) {  // uniform over the block
        const uint64_t ch = base + threadIdx.x;
        uint32_t w[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
        if (ch < chunks) {
            const uint4 v = *reinterpret_cast<const uint4*>(k.type + 16 * ch);
            w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
        }
        unsigned count = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            count += __popc(__vcmpeq4(w[i], 0x02020202u)) >> 3;
            air += __popc(__vcmpeq4(w[i], 0u)) >> 3;  // padding cells are VOID
        }
        if (!__any_sync(0xFFFFFFFFu, count != 0)) continue;
        unsigned incl = count;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned u = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= off) incl += u;
        }
        unsigned at = 0;
        if (lane == 31) at = atomicAdd(&k.ctrl->front_n, incl);
        at = __shfl_sync(0xFFFFFFFFu, at, 31) + incl - count;
        if (count == 0) continue;
        const uint64_t p0 = 16 * ch, row = p0 / (uint64_t)k.g.P;
        const int x0 = (int)(p0 - row * (uint64_t)k.g.P);
        const int y = (int)(row % (uint64_t)k.g.ny), z = (int)(row / (uint64_t)k.g.ny);
        for (int i = 0; i < 16; ++i) {
            if (((w[i >> 2] >> (8 * (i & 3))) & 0xFFu) != kLava) continue;
            k.idx[at] = (uint32_t)(x0 + i + k.g.nx * (y + k.g.ny * z));
            k.ltemp[at] = k.temp[p0 + i];
            k.flags[at] = front_is_vent(k, k.flow[p0 + i], x0 + i, y, z) ? kFrontVent : 0;
            ++at;
        }
    }
    if (!snap) return;
    const unsigned a = __reduce_add_sync(0xFFFFFFFFu, (unsigned)air);
    CaCtrl* ctrl = k.ctrl;
    if (lane == 0 && a) atomicAdd(&ctrl->acc_born, (unsigned long long)a);
    __syncthreads();
    if (threadIdx.x >= 32) return;
    unsigned left = 0;
    if (lane == 0) asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n" : "=r"(left) : "l"(&ctrl->front_exit) : "memory");
    if (__shfl_sync(0xFFFFFFFFu, left, 0) != gridDim.x - 1u) return;
    if (lane == 0) {  // the last block: LavaCA::countInitialState (LavaCA.hpp:1272-1279)
        const uint64_t lava = __ldcg(&ctrl->front_n), none = __ldcg(&ctrl->acc_born);
        int stop = VCA_STOP_RUNNING;
        if (!k.classic && lava == 0) stop = VCA_STOP_NO_LAVA;
        else if (k.classic && none == 0) stop = VCA_STOP_NO_AIR;
        else if (k.max_steps <= t0) stop = VCA_STOP_MAX_STEPS;
        ctrl->front_exit = 0;
        ctrl->acc_born = 0;
        ctrl->lava = lava;
        ctrl->air = none;
        ctrl->stop = stop;
        __threadfence();
    }
    __syncwarp();
    const uint32_t* from = reinterpret_cast<const uint32_t*>(ctrl);
    volatile uint32_t* to = reinterpret_cast<volatile uint32_t*>(snap);
    for (int i = lane; i < (int)(sizeof(CaCtrl) / sizeof(uint32_t)); i += 32) to[i] = __ldcg(from + i);
}

// ============================================================================================
// Host side
// ============================================================================================
CaFrontArgs front_args(const vca_ca* h) {
    CaFrontArgs k;
    std::memset(&k, 0, sizeof(k));
    const NbTable& nb = h->tables_host.nb;
    const int b = h->front_buf, o = b ^ 1;
    k.g = h->geom;
    k.div_nx = make_fastdiv32((uint32_t)h->geom.nx);
    k.div_ny = make_fastdiv32((uint32_t)h->geom.ny);
    k.classic = h->desc.mode == VCA_MODE_CLASSIC;
    k.ponding = h->desc.ponding != 0;
    k.variants = nb.variants;
    k.random_nb = nb.variants > 1;
    for (int v = 0; v < nb.variants; ++v)
        for (int i = 0; i < nb.count[v]; ++i) {
            const int8_t* d = nb.off[v][i];
            k.vmask[v] |= 1u << ((d[0] + 1) + 3 * (d[1] + 1) + 9 * (d[2] + 1));
            if (d[2] == -1 && (d[0] != 0 || d[1] != 0)) k.diag_falls = 1;
        }
    for (uint32_t m : k.vmask) k.umask |= m;
    for (int i = 0; i < h->tables_host.nside; ++i)
        k.side_mask |= 1u << (3 * (h->tables_host.side[i][1] + 1) + (h->tables_host.side[i][0] + 1));
    k.max_steps = h->desc.max_steps;
    k.eruption_steps = h->desc.eruption_steps;
    k.erupt_temp = h->desc.erupt_temp;
    k.solidus = h->desc.solidus_temp;
    k.cool_ambient = h->desc.cooling_ambient;
    k.cool_lateral = h->desc.cooling_lateral;
    k.cool_fall = h->desc.cooling_fall;
    k.seed = h->desc.seed;
    k.var_mod = make_fastmod((uint64_t)nb.variants);
    k.type = h->type[b];
    k.flow = h->flow[b];
    k.temp = h->temp[b];
    k.solid = h->solid[b];
    k.arrival = h->arrival[b];
    k.spill = h->has_terrain ? h->spill : nullptr;
    k.vents = h->vents;
    k.vent_slots = h->vent_slots;
    // scratch: the other buffer's planes (4 bytes per cell each), the drop plane, the candidate list, and
    // the heights of the last apply_terrain, which only its own kernel reads
    k.mark = reinterpret_cast<uint32_t*>(h->flow[o]);
    k.stamp = reinterpret_cast<uint32_t*>(h->heights_dev);
    k.ltemp = h->temp[o];
    k.work = reinterpret_cast<uint32_t*>(h->solid[o]);
    k.work_cap = (uint32_t)std::min<uint64_t>((uint64_t)h->cap.plane_cells, 0xFFFFFFFFu);
    k.idx = h->cand_list;
    k.flags = reinterpret_cast<uint8_t*>(h->drop_plane);
    k.ctrl = h->ctrl;
    k.hist_active = h->hist_active;
    k.hist_changed = h->hist_changed;
    return k;
}

static vca_status front_list_launch(vca_ca* h, int t0, CaCtrl* snap) {
    const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>((h->plane_cells / 16 + 255) / 256, (uint64_t)h->sms * 8));
    ca_front_list_kernel<<<blocks, 256, 0, h->stream>>>(front_args(h), h->plane_cells, t0, snap);
    VCA_CUDA(cudaGetLastError());
    h->launches += 1;
    h->front_listed = true;
    return VCA_OK;
}

// The list, the totals and the stop state of the current buffer, for a control block that is zero but for
// its step and its rules; left in the host's mirror.
vca_status front_init(vca_ca* h, int steps_done) { return front_list_launch(h, steps_done, h->ctrl_host_dev); }
// The list alone.
vca_status front_list(vca_ca* h) {
    VCA_CUDA(cudaMemsetAsync(&h->ctrl->front_n, 0, 2 * sizeof(uint32_t), h->stream));  // and front_prev
    return front_list_launch(h, 0, nullptr);
}

int front_batch_grid(int sms) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ca_front_batch_kernel, kFrontBatchThreads, 0) != cudaSuccess) return 0;
    return sms * std::min(per_sm, 4);
}
cudaError_t front_batch_launch(const CaFrontBatch& view, int grid, int steps, cudaStream_t stream) {
    CaFrontBatch b = view;
    void* args[] = {&b, &steps};
    return cudaLaunchCooperativeKernel((const void*)ca_front_batch_kernel, grid, kFrontBatchThreads, args, 0, stream);
}

constexpr int kFrontChunk = 256;       // most steps per launch of a run (64: 1 % slower)

// The launch for a list of n slots.  Up to kFrontSolo one block with a thread per slot, which keeps it in
// registers: its step has no grid barrier, and its barriers wait for no more warps than needed (512 x 1 x 256,
// 300 steps, up to 513 slots: 1.45 ms; 256 threads that stream the list beyond 256 slots 1.60 ms; all SMs
// beyond 256 slots 1.84 ms; one block of 1024 threads 1.9 ms).  Up to kFrontSmall blocks of 256 threads on all
// SMs, which hold a slot per thread up to 37 888 slots; beyond, the list is streamed and 1024 threads stream it
// faster (256 x 256 x 128, 400 steps: 2.80 ms with the line at 40 000, 2.98 ms without the small blocks;
// classic 100^3: 1.21 ms, with the line at 160 000 1.34 ms).  A launch ends early when its list has
// outgrown `most`.
constexpr uint32_t kFrontSolo = 512, kFrontSmall = 40000;
struct FrontShape {
    int threads, blocks;
    uint32_t most;
};
static FrontShape front_shape(const vca_ca* h, uint64_t n) {
    if (n <= kFrontSolo / 2) return {256, 1, kFrontSolo / 2};
    if (n <= kFrontSolo) return {512, 1, kFrontSolo};
    if (n <= kFrontSmall) return {256, h->sms, 2 * kFrontSmall};
    return {kFrontThreads, h->sms, 0xFFFFFFFFu};
}

vca_status front_run(vca_ca* h, int max_new_steps, bool until_stop) {
    if (!h->front_listed)
        if (vca_status s = front_list(h)) return s;
    CaFrontArgs k = front_args(h);
    VCA_CUDA(cudaEventRecord(h->ev_a, h->stream));
    CaCtrl last = *h->ctrl_host;
    auto launch = [&](int steps, uint32_t n, int slot) -> vca_status {
        const FrontShape f = front_shape(h, n);
        uint32_t most = until_stop ? f.most : 0xFFFFFFFFu;
        CaCtrl* snap = h->ctrl_ring_dev + slot;
        const auto kernel = f.threads == 256   ? (k.classic ? ca_front_kernel<256, true> : ca_front_kernel<256, false>)
                            : f.threads == 512 ? (k.classic ? ca_front_kernel<512, true> : ca_front_kernel<512, false>)
                                               : (k.classic ? ca_front_kernel<kFrontThreads, true> : ca_front_kernel<kFrontThreads, false>);
        if (f.blocks == 1) {
            kernel<<<1, f.threads, 0, h->stream>>>(k, steps, most, snap);
            VCA_CUDA(cudaGetLastError());
        } else {
            void* args[] = {&k, &steps, &most, &snap};
            VCA_CUDA(cudaLaunchCooperativeKernel((const void*)kernel, f.blocks, f.threads, args, 0, h->stream));
        }
        h->launches += 1;
        return VCA_OK;
    };
    if (!until_stop) {
        if (vca_status s = launch(max_new_steps, last.front_n, 0)) return s;
    } else {
        // the state after launch i is read while launch i + 1 runs
        int pending = -1, slot = 0;
        for (;;) {
            if (vca_status s = launch(kFrontChunk, last.front_n, slot)) return s;
            VCA_CUDA(cudaEventRecord(h->ring_ev[slot], h->stream));
            if (pending >= 0) {
                VCA_CUDA(cudaEventSynchronize(h->ring_ev[pending]));
                last = h->ctrl_ring[pending];
                if (last.stop != VCA_STOP_RUNNING || last.error) break;
            }
            pending = slot;
            slot ^= 1;
        }
    }
    VCA_CUDA(cudaEventRecord(h->ev_b, h->stream));
    VCA_CUDA(cudaEventSynchronize(h->ev_b));
    float ms = 0.f;
    VCA_CUDA(cudaEventElapsedTime(&ms, h->ev_a, h->ev_b));
    h->total_ms += ms;
    if (!until_stop) last = h->ctrl_ring[0];
    return sync_ctrl(h, last);
}

}  // namespace vca
