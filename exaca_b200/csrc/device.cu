// B200 kernels and pool runtime for ExaCA's per-cycle cellular-automaton update.
//
// One CA cycle (src/runCA.cpp:290-341; src/CAupdate.cpp:67-728) is a start and two passes over a
// pool of domains:
//   begin_cycle: per domain, the device-side termination check, cycle/epoch advance and nucleation
//          of the sites whose time has come (nuclei are pre-sorted by time, one cursor each).
//   grow/claim: streams the 16-byte records of the active cells (shared compacted list): diagonal
//          growth from the host-built increment table, solidification of cells with no liquid
//          neighbour, and a 64-bit atomicMin claim (epoch, capturer index) on every liquid neighbour
//          the octahedron reaches. Liquid neighbours come from a per-cell mask kept up to date by
//          captures and nucleations; the 26 critical lengths are read only when the diagonal has
//          reached the cached minimum over the liquid neighbours.
//   capture: per claimed cell: capture by the lowest-index claimant (new decentred octahedron, 26
//          critical lengths), mask updates of its active neighbours, and for those the
//          solidification re-check.
// Stretches of cycles run in one persistent cooperative kernel (k_cycles) whose blocks meet at
// bounded grid-wide barriers, two per cycle: after the claims and after the captures. Each block runs
// the claim steps of the records it flagged right after its own growth (a shared-memory queue; a
// grid-wide claim pass runs only in a cycle where some block's queue overflowed), and captures the
// winners among its own claims. The start of the next cycle runs under the capture pass, in a few
// warps of their own. The same passes also run as separate kernels (per-pass timing).
// The claim rule reproduces the Kokkos-Serial loop order exactly: serial visits active cells in
// ascending index and captures flip Liquid to Active in place, so the capturer of a cell is the
// lowest-index claimant, and an active cell sees a neighbour as liquid iff it was liquid at the
// start of the cycle and no lower-index cell claimed it. Only cells next to a claimed cell can lose
// their last such neighbour, so only they are re-checked.
//
// Arithmetic follows the reference's types and operation order; this file is compiled with
// -fmad=false so no multiply-add is contracted, and sqrt/division are IEEE round-to-nearest.
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <sstream>
#include <stdexcept>
#include <thread>

#include "pool.hpp"

namespace exaca {

#define CUDA_OK(x)                                                                                                     \
    do {                                                                                                               \
        cudaError_t e__ = (x);                                                                                         \
        if (e__ != cudaSuccess)                                                                                        \
            throw DeviceError(std::string("CUDA error ") + cudaGetErrorString(e__) + " at " #x);                     \
    } while (0)

// A direction's components, its opposite and the capture pass's slot order (directions.hpp), read
// from immediates: lanes asking for different directions read no table.
__device__ __forceinline__ int nb_dx(int l) { return (int)((kDirXP >> l) & 1u) - (int)((kDirXM >> l) & 1u); }
__device__ __forceinline__ int nb_dy(int l) { return (int)((kDirYP >> l) & 1u) - (int)((kDirYM >> l) & 1u); }
__device__ __forceinline__ int nb_dz(int l) { return (int)((kDirZP >> l) & 1u) - (int)((kDirZM >> l) & 1u); }
__device__ __forceinline__ unsigned int field5(unsigned long long a, unsigned long long b, unsigned long long c,
                                               int i) {
    const unsigned long long v = i < 12 ? a : (i < 24 ? b : c);
    const int f = i < 12 ? i : (i < 24 ? i - 12 : i - 24);
    return (unsigned int)(v >> (5 * f)) & 31u;
}
__device__ __forceinline__ int nb_opp(int l) { return (int)field5(kOppA, kOppB, kOppC, l); }
// direction of capture slot s (slots by z, then x, then y); 31 for s >= 26
__device__ __forceinline__ int slot_dir(int s) { return s < 26 ? (int)field5(kSlotA, kSlotB, kSlotC, s) : 31; }

constexpr unsigned int kMaskFresh = 1u << 31; // liquid-neighbour mask not built yet
constexpr unsigned int kMaskDead = 1u << 30;  // solidified by a re-check: leaves the list next cycle
constexpr unsigned int kMaskKeep = 1u << 29;  // this cycle, a neighbour was captured by an index >= this cell's
// the record has been grown (cycle > its CritTimeStep): set by the first growth step, so that the
// capture pass's re-check needs no CritTimeStep (a record's eligibility only changes at a layer
// change, which rebuilds the list)
constexpr unsigned int kMaskGrown = 1u << 28;
// a neighbour nucleated at the start of this cycle: the growth pass drops the directions that are no
// longer liquid from the mask (set only inside the persistent kernel, between two of its cycles)
constexpr unsigned int kMaskNuc = 1u << 27;
constexpr unsigned int kMaskTomb = 1u << 26; // a dropped record (the whole status word)
constexpr unsigned int kDirBits = (1u << 26) - 1;
// CellType of a liquid cell that nucleates at the start of the next cycle unless it is claimed in
// this one; two codes, alternating by cycle, so that the captures of a cycle tell the sites that fire
// after it (no longer liquid for a captured cell's mask) from those marked for the cycle after that
// (still liquid). Only inside the persistent kernel: no mark is left when it ends.
constexpr int8_t kMark0 = 8;
__device__ __forceinline__ int8_t mark_code(int cycle_index) { return (int8_t)(kMark0 + (cycle_index & 1)); }
// liquid at the start of the current cycle, for a pass in which claims are being made
__device__ __forceinline__ bool liquid_type(int8_t t) { return t == kLiquid || t == kTemporaryUpdate || t >= kMark0; }
constexpr int kErrGrowthTable = 1;
constexpr int kErrListOverflow = 2;
constexpr int kErrBounds = 4;
// One 512-thread block per SM for the persistent kernel (16 warps per SM, 128 registers each): half
// the blocks of two 256-thread ones, so half the arrivals at every grid-wide meeting, and a claim
// step of up to 512 flagged records per block in one round.
constexpr int kBlock = 512;
// A record's domain word: its domain, and in the upper half the direction of the cached minimum critical
// length (kNoDir: not known, or there is none; the cached minimum alone applies).
constexpr unsigned int kNoDir = 31u;
__device__ __forceinline__ unsigned int dom_word(unsigned int dom, unsigned int dir) { return dom | (min(dir, kNoDir) << 16); }
__device__ __forceinline__ unsigned int word_dom(unsigned int w) { return w & 0xffffu; }
// The cached minimum, or the second-smallest length once the minimum's neighbour is no longer liquid (both
// are lower bounds of the current liquid neighbours' lengths).
__device__ __forceinline__ float effective_min(float cdl_min, float min2, unsigned int m, unsigned int w) {
    const unsigned int d1 = w >> 16;
    return d1 < 26u && !((m >> d1) & 1u) ? min2 : cdl_min;
}

__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; } // std::min
__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; } // std::max

// Number of executed cycles in [1, x]: cycles skipped by the type-S/R jump
// (src/CAupdate.cpp:812-817) are not executed and add no undercooling.
__device__ __forceinline__ long long executed_upto(const DomainDesc &D, long long x) {
    if (x <= 0)
        return 0;
    long long e = x;
    for (int j = 0; j < D.n_jumps; j++) {
        long long lo = D.jump_lo[j], hi = D.jump_hi[j];
        if (x > lo)
            e -= (x < hi ? x : hi) - lo;
    }
    return e;
}

// What a reservation of [first, first + total) takes past `cap` is given back and flagged. A counter that
// has reached its limit never falls below it, so every slot below `cap` belongs to one reservation, whose
// owner writes it, and no counter stays past the array that it counts.
__device__ __forceinline__ void reserved_past(unsigned long long *counter, unsigned long long cap, int *error,
                                              unsigned long long first, unsigned long long total) {
    if (first + total <= cap)
        return;
    atomicOr(error, kErrListOverflow);
    atomicAdd(counter, (first > cap ? first : cap) - (first + total));
}

// Block-aggregated reservation of `n` (0 or 1) slots per thread on `counter`: one atomicAdd per block.
// Must be called by every thread of the block. Returns this thread's slot, or ULLONG_MAX past `cap` (the
// pool error flag is set).
__device__ __forceinline__ unsigned long long block_reserve_on(unsigned long long *counter, unsigned long long cap,
                                                              int *error, unsigned int n) {
    __shared__ unsigned int s_warp[32];
    __shared__ unsigned long long s_base;
    // the launch's own warp count (callers launch with different block sizes)
    const unsigned int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    unsigned int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (unsigned)o)
            incl += v;
    }
    if (lane == 31)
        s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        unsigned int v = lane < n_warps ? s_warp[lane] : 0;
        unsigned int inc2 = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned int u = __shfl_up_sync(0xffffffffu, inc2, o);
            if (lane >= (unsigned)o)
                inc2 += u;
        }
        if (lane < n_warps)
            s_warp[lane] = inc2 - v;
        unsigned int total = __shfl_sync(0xffffffffu, inc2, n_warps - 1);
        if (lane == 0) {
            unsigned long long b = total ? atomicAdd(counter, (unsigned long long)total) : 0ull;
            reserved_past(counter, cap, error, b, total);
            s_base = b;
        }
    }
    __syncthreads();
    const unsigned long long r = s_base + s_warp[warp] + (incl - n);
    __syncthreads(); // s_warp / s_base are reused by the next call
    return r < cap ? r : ULLONG_MAX;
}

__device__ __forceinline__ unsigned long long block_reserve(PoolState *P, int slot, unsigned int n) {
    return block_reserve_on(&P->cnt[slot], P->capacity, &P->error, n);
}

// Warp-aggregated reservation (any subset of lanes may call, all with the same counter).
__device__ __forceinline__ unsigned long long warp_reserve(unsigned long long *counter, unsigned long long cap,
                                                           int *error) {
    unsigned int act = __activemask();
    int lane = threadIdx.x & 31;
    int leader = __ffs(act) - 1;
    unsigned long long base = 0;
    if (lane == leader) {
        base = atomicAdd(counter, (unsigned long long)__popc(act));
        reserved_past(counter, cap, error, base, (unsigned long long)__popc(act));
    }
    base = __shfl_sync(act, base, leader);
    const unsigned long long r = base + __popc(act & ((1u << lane) - 1));
    return r < cap ? r : ULLONG_MAX;
}

// Block-level sum of per-thread statistics into one shard of the pool counters.
__device__ __forceinline__ void block_stats(PoolState *P, unsigned long long a, unsigned long long b, int ia, int ib) {
    __shared__ unsigned long long s_a[32], s_b[32];
    for (int o = 16; o; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        s_a[threadIdx.x >> 5] = a;
        s_b[threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long ta = 0, tb = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            ta += s_a[w];
            tb += s_b[w];
        }
        int shard = blockIdx.x & (kStatShards - 1);
        if (ta)
            atomicAdd(&P->stat[shard][ia], ta);
        if (tb)
            atomicAdd(&P->stat[shard][ib], tb);
    }
}

__device__ __forceinline__ void cell_coords(const DomainDesc &D, unsigned int c, int &rx, int &ry, int &rz) {
    unsigned int plane = (unsigned int)(D.mx * D.my);
    unsigned int z = c / plane;
    unsigned int rem = c - z * plane;
    unsigned int x = rem / (unsigned int)D.my;
    rz = (int)z;
    rx = (int)x;
    ry = (int)(rem - x * (unsigned int)D.my);
}

// Edge case of src/CAfunctions.cpp:169-213 as a direction mask (ItList, src/CAinitialize.cpp:676-745:
// the edge cases drop the directions leaving the x / y extent, x = 0 before x = mx - 1 and y = 0
// before y = my - 1), restricted to the top of the active window in z (src/CAupdate.cpp:328 checks
// MyNeighborZ < nzActive, window-relative; there is no lower check in the reference, which reads
// one plane below the window; here z >= 0 is kept as a guard).
__device__ __forceinline__ unsigned int edge_mask(int rx, int ry, int rz, int mx, int my, int z_end) {
    unsigned int m = (1u << 26) - 1u;
    m &= ~(ry == 0 ? kDirYM : (ry == my - 1 ? kDirYP : 0u));
    m &= ~(rx == 0 ? kDirXM : (rx == mx - 1 ? kDirXP : 0u));
    if (rz + 1 >= z_end)
        m &= ~kDirZP;
    if (rz - 1 < 0)
        m &= ~kDirZM;
    return m;
}
__device__ __forceinline__ unsigned int neighbour_mask(const DomainDesc &D, int rx, int ry, int rz) {
    return edge_mask(rx, ry, rz, D.mx, D.my, D.z_end);
}

__device__ __forceinline__ int nb_offset(int l, int plane, int my) { return nb_dz(l) * plane + nb_dx(l) * my + nb_dy(l); }

// Fresh octahedron of a newly active cell at its own centre (src/CAupdate.cpp:100-194,
// src/CAinitialize.cpp:1942-2042): DL = 0.01, centre = cell centre, CDL from the orientation table.
__device__ void make_fresh_octahedron(const DomainDesc &D, unsigned int c) {
    int rx, ry, rz;
    cell_coords(D, c, rx, ry, rz);
    int h = D.gid[c];
    int ori = (abs(h) - 1) % 10000;
    if (ori < 0)
        ori += 10000;
    D.dl[c] = 0.01f;
    D.doc[3ull * c + 0] = (float)((double)(rx + D.xoff) + 0.5);
    D.doc[3ull * c + 1] = (float)((double)(ry + D.yoff) + 0.5);
    D.doc[3ull * c + 2] = (float)((double)rz + 0.5);
    const float2 *t = reinterpret_cast<const float2 *>(D.cdl_table + 26 * ori);
    float2 *o = reinterpret_cast<float2 *>(D.cdl + 26ull * c);
#pragma unroll
    for (int n = 0; n < 13; n++)
        o[n] = t[n];
}


__device__ __forceinline__ long long domain_liquid(const DomainDesc &D) {
    long long v = D.liquid;
#pragma unroll
    for (int q = 0; q < kLiquidShards; q++)
        v += __ldcg(&D.liquid_shard[q]);
    return v;
}

// One list of active-cell records (PoolState).
struct RecordList {
    ActiveRec *rec;
    unsigned int *cell, *dom;
    float *min2;
    RecordBody *body;
    unsigned int body_cap; // records below it have a body
};
__device__ __forceinline__ RecordList list_of(const PoolState *P, int q) {
    return RecordList{P->rec[q], P->rcell[q], P->rdom[q], P->rmin2[q], P->body[q], P->body_cap};
}
// GrainID (bits) and DOCenter of a body as one vector
__device__ __forceinline__ float4 &body_head(RecordBody &b) { return *reinterpret_cast<float4 *>(&b); }

// ---------------------------------------------------------------------------------------------
// Start of a CA cycle (src/runCA.cpp:290-298, src/CAupdate.cpp:67-200): list swap, device-side
// termination check, cycle advance, nucleation. In the persistent kernel the start of a few domains
// runs in one block while the rest of the grid waits, so its cost is its chain of dependent round
// trips to L2 / HBM. Every load that does not depend on an earlier one goes out in the same round:
//   1. the pool's list counters, and each domain's descriptor fields;
//   2. the next 32 nucleation sites by time, with the rest of the descriptor;
//   3. per due site: its CellType, LayerID, GrainID and CritTimeStep;
//   4. per firing site, with the whole warp: its critical-length row and its neighbours' CellTypes and
//      list positions (the list slots of all firing sites are reserved under the first such round).
// Reads that may see data other blocks of the same kernel wrote go through L2 (__ldcg).

// Entries of a queue's shard: none where its counter went past the shard's slots, since the warps that crossed
// the limit wrote none of theirs (the pool's overflow flag is set; what the shard held is not acted on).
__device__ __forceinline__ unsigned long long shard_count(const ShardCounter &c, unsigned long long cap) {
    const unsigned long long n = __ldcg(&c.v);
    return n <= cap ? n : 0ull;
}

// Pool part (warp 0): when `close`, the records the last capture pass appended join the list the
// next cycle reads, which ends the previous cycle; then the list swap, the compaction decision and
// the per-cycle counters. One round of loads. The list this cycle reads goes to *cur_out if given.
__device__ __forceinline__ void lists_start(PoolState *P, bool close, int *cur_out) {
    if (threadIdx.x < 32) {
        static_assert(kShards == 32, "one lane per shard");
        const int lane = threadIdx.x;
        unsigned long long added = __ldcg(&P->tomb_s[lane].v);
        unsigned long long appended = close ? shard_count(P->tcnt_s[lane], P->shard_cap) : 0ull;
        int prev = 0, cur = 0;
        unsigned long long cnt0 = 0, cnt1 = 0, tombs = 0, cap = 0;
        if (lane == 0) {
            prev = __ldcg(&P->cur);
            cur = __ldcg(&P->pending);
            cnt0 = __ldcg(&P->cnt[0]);
            cnt1 = __ldcg(&P->cnt[1]);
            tombs = __ldcg(&P->tombs);
            cap = P->capacity;
        }
        P->tomb_s[lane].v = 0;
        P->qcnt_s[lane].v = 0;
        P->tcnt_s[lane].v = 0;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            added += __shfl_down_sync(0xffffffffu, added, o);
            appended += __shfl_down_sync(0xffffffffu, appended, o);
        }
        if (lane == 0) {
            if (close) {
                // the capture pass reserved its new records' slots past the count of list `cur`
                const unsigned long long grown = (cur ? cnt1 : cnt0) + appended;
                if (grown <= cap) {
                    if (cur)
                        cnt1 = grown;
                    else
                        cnt0 = grown;
                    P->cnt[cur] = grown;
                }
            }
            // the list the previous cycle left becomes current; when it was a compacted copy, the old
            // one is emptied and carries no dropped records any more
            const unsigned long long cnt_cur = cur ? cnt1 : cnt0;
            // the sum of what blocks of the persistent kernel had not told may be negative
            tombs = (unsigned long long)max((long long)(tombs + added), 0ll);
            if (cur != prev) {
                P->cnt[prev] = 0;
                tombs = 0;
            }
            P->tombs = tombs;
            P->cur = cur;
            // compact when dropped records exceed a quarter of the list (an eighth, and a sixteenth,
            // measured slower: the compaction pass costs more per record than the tombstones it
            // removes)
            const int compact = tombs * 4 > cnt_cur ? 1 : 0;
            P->compact = compact;
            P->pending = compact ? cur ^ 1 : cur;
            if (compact)
                P->cnt[cur ^ 1] = 0;
            if (cur_out)
                *cur_out = cur;
        }
    }
}

__device__ __noinline__ void begin_lists(PoolState *P, bool close) { lists_start(P, close, nullptr); }

constexpr int kSerialDomains = 8; // up to this many domains one block starts each cycle alone

// The domains that had not ended at the last state read, when there are at most kSerialDomains of
// them (a kernel argument, so the cycle start reads their indices without a global round trip;
// the first has the most cells). n < 0: start every domain of the pool.
struct AliveSet {
    int n;
    int idx[kSerialDomains];
};

// Descriptor fields of the first round (the cursor into the nucleation sites and what decides
// whether the domain runs this cycle).
struct DomainStart {
    const int32_t *nuc_time, *nuc_loc;
    int8_t *ctype;
    int done, check_mode, cycle0, cursor0, n_nuclei;
};

__device__ __forceinline__ DomainStart load_start(const DomainDesc &D) {
    DomainStart s;
    s.nuc_time = D.nuc_time;
    s.nuc_loc = D.nuc_loc;
    s.ctype = D.ctype;
    s.n_nuclei = D.n_nuclei;
    s.check_mode = D.check_mode;
    s.done = __ldcg(&D.done);
    s.cycle0 = __ldcg(&D.cycle);
    s.cursor0 = __ldcg(&D.nuc_cursor);
    return s;
}

// The descriptor fields that a nucleation needs.
struct NucleationView {
    int32_t *gid;
    const int32_t *cts_run;
    float *dl, *doc, *cdl;
    const float *cdl_table;
    unsigned int *pos;
    int mx, my, z_end, xoff, yoff;
};
__device__ __forceinline__ NucleationView nucleation_view(const DomainDesc &D) {
    return NucleationView{D.gid, D.cts_run, D.dl, D.doc, D.cdl, D.cdl_table, D.pos, D.mx, D.my, D.z_end, D.xoff, D.yoff};
}

// Nucleation of one site by a warp (src/CAupdate.cpp:100-194), one round of loads: lanes 0-12 copy the
// fresh octahedron's critical lengths, lane n < 26 reads neighbour n's type and list position; an
// active neighbour's record goes to on_neighbour(position, direction from the site). The record goes
// to `slot` (ULLONG_MAX: none) of list L.
template <class OnNeighbour>
__device__ __forceinline__ void nucleate_site(const NucleationView &V, int8_t *ctype, const RecordList &L, unsigned int dom,
                                              unsigned int site, int site_gid, int cts, unsigned long long slot,
                                              OnNeighbour &&on_neighbour) {
    const unsigned int lane = threadIdx.x & 31;
    const int plane = V.mx * V.my;
    const unsigned int z = site / (unsigned int)plane;
    const unsigned int rem = site - z * (unsigned int)plane;
    const int rx = (int)(rem / (unsigned int)V.my), ry = (int)(rem - (unsigned int)rx * (unsigned int)V.my), rz = (int)z;
    const unsigned int valid = edge_mask(rx, ry, rz, V.mx, V.my, V.z_end);
    int ori = (abs(site_gid) - 1) % 10000;
    if (ori < 0)
        ori += 10000;
    float2 row = make_float2(0.0f, 0.0f);
    if (lane < 13)
        row = reinterpret_cast<const float2 *>(V.cdl_table + 26 * ori)[lane];
    const bool nb = lane < 26 && ((valid >> lane) & 1u);
    int8_t nb_type = kLiquid;
    unsigned int nb_pos = 0;
    if (nb) {
        const long long a = (long long)site + nb_offset((int)lane, plane, V.my);
        nb_type = __ldcg(ctype + a);
        nb_pos = __ldcg(V.pos + a);
    }
    const bool has_body = slot < L.body_cap;
    if (lane < 13) {
        reinterpret_cast<float2 *>(V.cdl + 26ull * site)[lane] = row;
        if (has_body)
            reinterpret_cast<float2 *>(L.body[slot].cdl)[lane] = row;
    }
    if (lane == 0) {
        const float cx = (float)((double)(rx + V.xoff) + 0.5), cy = (float)((double)(ry + V.yoff) + 0.5),
                    cz = (float)((double)rz + 0.5);
        V.dl[site] = 0.01f;
        V.doc[3ull * site + 0] = cx;
        V.doc[3ull * site + 1] = cy;
        V.doc[3ull * site + 2] = cz;
        if (slot != ULLONG_MAX) {
            L.rec[slot] = ActiveRec{0.01f, 0.0f, cts, kMaskFresh};
            L.cell[slot] = site;
            L.dom[slot] = dom_word(dom, kNoDir);
            L.min2[slot] = 0.0f;
            V.pos[site] = (unsigned int)slot;
        }
        if (has_body)
            body_head(L.body[slot]) = make_float4(__int_as_float(site_gid), cx, cy, cz);
        ctype[site] = kActive;
    }
    if (nb && nb_type == kActive)
        on_neighbour(nb_pos, (int)lane);
    __syncwarp();
}

// Marks the liquid sites from `mark` on that are due by `cycle` (one warp); returns the first site not
// due. Sites are sorted by time, so the due ones form a prefix.
__device__ __forceinline__ int mark_sites(DomainDesc &D, const DomainStart &s, int mark, int cycle, int8_t code,
                                          int layer_no, long long active_size) {
    const unsigned int lane = threadIdx.x & 31;
    while (mark < s.n_nuclei) {
        const int idx = mark + (int)lane;
        const int t = idx < s.n_nuclei ? __ldg(s.nuc_time + idx) : INT_MAX;
        const int l = idx < s.n_nuclei ? __ldg(s.nuc_loc + idx) : -1;
        const bool due = t <= cycle;
        const int n_due = __popc(__ballot_sync(0xffffffffu, due));
        if (n_due == 0)
            break;
        if (due) {
            if (l < 0 || l >= active_size)
                atomicOr(&D.error, kErrBounds);
            else if (__ldcg(s.ctype + l) == kLiquid && D.layer[l] <= layer_no)
                s.ctype[l] = code;
        }
        mark += n_due;
        if (n_due < 32)
            break;
    }
    return mark;
}

// The first cycle after `cycle` whose start has to be run, when no claim is made before it: the next
// one when sites are marked for it, the one that marks the next site (a site is marked at the start
// of the cycle before its own), or the one of a device-terminated domain's next check (start_domain).
__device__ __forceinline__ int next_start_of(const DomainStart &s, int cycle, int cursor, int mark) {
    if (mark > cursor)
        return cycle + 1;
    int next = mark < s.n_nuclei ? max(cycle + 1, __ldg(s.nuc_time + mark) - 1) : INT_MAX;
    if (s.check_mode) // cycle starts after a multiple of 64 or of 1000
        next = min(next, min((cycle + 63) / 64 * 64, (cycle + 999) / 1000 * 1000) + 1);
    return next;
}

// Cycle start of domain d by one warp (all lanes call with the same arguments). With `mark` the sites
// due at the next cycle's start are marked for start_next.
__device__ __forceinline__ void start_domain(PoolState *P, DomainDesc &D, const DomainStart &s, unsigned int d,
                                             int cur, bool mark, unsigned long long &nucleated) {
    const unsigned int lane = threadIdx.x & 31;
    if (s.ctype == nullptr || s.done)
        return;
    if (s.check_mode && s.cycle0 > 0 && s.cycle0 % 1000 == 0 && domain_liquid(D) == 0) {
        // src/CAupdate.cpp:782-783: no superheated or undercooled liquid left
        if (lane == 0)
            D.done = 1;
        return;
    }
    const int cycle = s.cycle0 + 1;
    int cursor = s.cursor0, fired_total = 0;
    // round 2: the rest of the descriptor goes out with the first batch of sites
    const int8_t *const layer = D.layer;
    const NucleationView V = nucleation_view(D);
    const int layer_no = D.layer_no;
    const long long active_size = D.active_size;
    const unsigned int epoch0 = __ldcg(&D.epoch);
    const int nn0 = __ldcg(&D.nn);
    const long long liquid0 = __ldcg(&D.liquid);
    // every 64th cycle of a device-terminated domain, in its last phase (every cell past its
    // CritTimeStep), whether any liquid is left: these loads go with this round, and the answer is
    // used after the sites, none of which can fire without liquid
    const bool probe = s.check_mode && (s.cycle0 & 63) == 0;
    const int dry_since = probe ? __ldcg(&D.dry_since) : 0;
    const int cts_max = probe ? D.cts_max : INT_MAX;
    long long dry = probe && lane < kLiquidShards ? __ldcg(&D.liquid_shard[lane]) : 0;
    const unsigned long long cap = P->capacity;
    const RecordList L = list_of(P, cur);
    // src/CAupdate.cpp:76-198: sites with cycle >= NucleationTimes that are still liquid
    while (cursor < s.n_nuclei) {
        const int idx = cursor + (int)lane;
        const int t = idx < s.n_nuclei ? __ldg(s.nuc_time + idx) : INT_MAX;
        const int l = idx < s.n_nuclei ? __ldg(s.nuc_loc + idx) : -1;
        const bool due = t <= cycle;
        // sites are sorted by time, so the due ones form a prefix
        const int n_due = __popc(__ballot_sync(0xffffffffu, due));
        if (n_due == 0)
            break;
        // round 3
        bool fire = false;
        unsigned int loc = 0;
        int h = 0, cts = 0;
        if (due) {
            if (l < 0 || l >= active_size) {
                atomicOr(&D.error, kErrBounds);
            }
            else {
                loc = (unsigned int)l;
                const int8_t site_type = __ldcg(s.ctype + loc);
                const int site_layer = layer[loc];
                h = __ldcg(V.gid + loc);
                cts = V.cts_run[loc];
                fire = site_type == kLiquid && site_layer <= layer_no;
            }
        }
        // list slots of the firing sites (one atomic; it completes under round 4)
        const unsigned long long my_slot = fire ? warp_reserve(&P->cnt[cur], cap, &P->error) : ULLONG_MAX;
        // round 4, one firing site at a time with the whole warp; an active neighbour drops the site
        // from its liquid mask
        for (unsigned int todo = __ballot_sync(0xffffffffu, fire); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            nucleate_site(V, s.ctype, L, d,
                          __shfl_sync(0xffffffffu, loc, src), __shfl_sync(0xffffffffu, h, src),
                          __shfl_sync(0xffffffffu, cts, src), __shfl_sync(0xffffffffu, my_slot, src),
                          [&](unsigned int nb_pos, int l) {
                              if (nb_pos < cap)
                                  atomicAnd(&L.rec[nb_pos].stat, ~(1u << nb_opp(l)));
                          });
        }
        fired_total += __popc(__ballot_sync(0xffffffffu, fire));
        cursor += n_due;
        if (n_due < 32)
            break;
    }
    bool ended = false;
    if (probe && s.cycle0 - 2 >= cts_max) {
#pragma unroll
        for (int o = 16; o; o >>= 1)
            dry += __shfl_xor_sync(0xffffffffu, dry, o);
        if (dry + liquid0 == 0 && fired_total == 0) {
            if (dry_since == 0) {
                if (lane == 0)
                    D.dry_since = s.cycle0;
            }
            else {
                // At least a whole cycle has run with no liquid and every cell past its CritTimeStep,
                // so every active cell has found no liquid neighbour and solidified
                // (src/CAupdate.cpp:722-725); nothing changes until the next 1000-cycle check, which
                // ends the domain (src/CAupdate.cpp:782-783). It ends here with that check's cycle.
                ended = true;
            }
        }
    }
    const int marked = mark && !ended ? mark_sites(D, s, cursor, cycle + 1, mark_code(1), layer_no, active_size) : cursor;
    if (lane == 0 && ended) {
        D.cycle = (s.cycle0 + 999) / 1000 * 1000;
        D.done = 1;
    }
    else if (lane == 0) {
        D.cycle = cycle;
        D.epoch = epoch0 + 1;
        D.next_start = next_start_of(s, cycle, cursor, marked);
        D.nuc_cursor = cursor;
        D.nuc_mark = marked;
        D.nn = nn0 + fired_total;
        D.liquid = liquid0 - fired_total;
        nucleated += fired_total;
    }
}

// Cycle start, per-domain part, across the grid: warps first_warp, first_warp + warp_stride, ...
// take one domain each (the current list was settled by begin_lists before a grid-wide meeting).
__device__ __noinline__ void begin_domains(PoolState *P, DomainDesc *desc, int n_domains, int first_warp, int warp_stride,
                                           bool mark) {
    const int cur = __ldcg(&P->cur);
    unsigned long long nucleated = 0;
    for (int d = first_warp; d < n_domains; d += warp_stride) {
        const DomainStart s = load_start(desc[d]);
        start_domain(P, desc[d], s, (unsigned int)d, cur, mark, nucleated);
    }
    if ((threadIdx.x & 31) == 0 && nucleated)
        atomicAdd(&P->stat[0][kStatNucleated], nucleated);
}

// Cycle start by one block: the pool part in warp 0 while every warp loads its first domain's
// descriptor, then the domains with the block's warps. With `close` it first ends the previous
// cycle (finish_capture); `mark` as start_domain.
__device__ __noinline__ void begin_cycle(PoolState *P, bool close, DomainDesc *desc, int n_domains, AliveSet alive,
                                         bool mark) {
    __shared__ int s_cur;
    const int w = (int)(threadIdx.x >> 5), nw = (int)(blockDim.x >> 5);
    const int n = alive.n < 0 ? n_domains : alive.n;
    DomainStart s{};
    if (w < n)
        s = load_start(desc[alive.n < 0 ? w : alive.idx[w]]);
    lists_start(P, close, &s_cur);
    __syncthreads();
    const int cur = s_cur;
    unsigned long long nucleated = 0;
    for (int i = w; i < n; i += nw) {
        const int d = alive.n < 0 ? i : alive.idx[i];
        if (i != w)
            s = load_start(desc[d]);
        start_domain(P, desc[d], s, (unsigned int)d, cur, mark, nucleated);
    }
    if ((threadIdx.x & 31) == 0 && nucleated)
        atomicAdd(&P->stat[0][kStatNucleated], nucleated);
}

__global__ void k_step_begin(PoolState *P) { begin_cycle(P, false, P->desc, P->n_domains, AliveSet{-1, {}}, false); }

// ---------------------------------------------------------------------------------------------
// One CA cycle after its start is three passes over the pool:
//   grow        every record of the current list (kBatch per lane, loads issued first): eligibility
//               and diagonal growth (src/CAupdate.cpp:257-261), drop of finished or
//               re-check-solidified cells, solidification of cells whose liquid mask is empty. A
//               record whose mask must still be built, or whose diagonal reached the cached minimum
//               critical length, is flagged for the claim pass.
//   claim       per flagged record: the liquid mask from the 26 neighbour types when it is not built
//               yet (nucleated and new-layer cells), the critical-length row (from the record's body)
//               and the claims (src/CAupdate.cpp:320-352); every claim is listed.
//   capture     per listed claim: the winner captures the cell (src/CAupdate.cpp:353-563), builds the
//               new record's liquid mask and cached minimum critical length, and re-checks the
//               captured cell's active neighbours.
// They run as three kernels per cycle (k_grow, k_claim, k_capture_pass) or, for stretches of cycles,
// inside the persistent cooperative kernel k_cycles: there a block claims for the records that it
// flagged and captures for the claims that it listed, the grid meets after the claims and after the
// captures, and the next cycle's start is spread over warps that have no capture left.
// Records per lane in flight in the growth pass (template argument).
constexpr int kBatchChoices[2] = {2, 4};
// The persistent kernel has a family of code for each range of list lengths (a kernel that held it all
// would be short of registers and of instruction cache: each pass runs once per cycle, and what a warp
// waits for is mostly the next instruction, not memory):
//   kLongList   hundreds of flagged records and captures per block and cycle: a lane per flagged record,
//               six captures' neighbours in flight per warp, two or four records per lane in the growth.
//   kMidList    tens of them: eight lanes per flagged record.
//   kShortList  as kMidList, and for blocks with no more claims than warps a warp per claim.
// Pool::shape_for chooses by the list's length.
enum { kLongList, kMidList, kShortList };
constexpr int kErrBarrier = 8;

// Work counts of one thread, added to the pool's at the end of a kernel and, in the persistent one,
// every kStatCycles cycles (32 bits hold a thread's records of that many cycles).
constexpr int kStatCycles = 512;
struct CycleStats {
    unsigned int listed = 0, grown = 0, dropped = 0, flagged = 0, claims = 0, rows = 0, fresh = 0, captured = 0,
                 rechecks = 0;
};

__device__ void flush_stats(PoolState *P, const CycleStats &st) {
    block_stats(P, st.listed, st.grown, kStatListed, kStatGrown);
    block_stats(P, st.dropped, st.flagged, kStatDropped, kStatFlagged);
    block_stats(P, st.claims, st.rows, kStatClaims, kStatRowReads);
    block_stats(P, st.fresh, st.captured, kStatFresh, kStatCaptured);
    block_stats(P, st.rechecks, 0, kStatRechecks, kStatRechecks);
}

// What a kernel reads again and again, in shared memory: the pool's pointers and the descriptor of
// one domain (the one with the most cells among few). A grid-wide meeting leaves L1 empty, so a
// pointer read from global memory costs a round trip to L2 before the load that needs it goes out.
// The copy's dynamic fields are those of the kernel's start; the persistent kernel refreshes cycle
// and epoch every cycle.
struct PassCtx {
    RecordList list[2];
    DomainDesc *desc;
    unsigned long long *tgt;
    unsigned long long capacity, segment, shard_cap; // segment: entries of tgt a block may fill
    long long hot_skipped;                           // cycles the hot domain's jumps skipped
    int extras;
    unsigned int hot;
    DomainDesc hot_desc;
};

// Fills X (all threads of the block call; a block barrier follows before X is read).
__device__ __forceinline__ void load_ctx(const PoolState *P, PassCtx &X, unsigned int hot) {
    static_assert(sizeof(DomainDesc) % 8 == 0, "copied in 8-byte words");
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(P->desc + hot);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(&X.hot_desc);
    for (unsigned int w = threadIdx.x; w < sizeof(DomainDesc) / 8; w += blockDim.x)
        dst[w] = __ldcg(src + w);
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; q++)
            X.list[q] = list_of(P, q);
        X.desc = P->desc;
        X.tgt = P->tgt;
        X.capacity = P->capacity;
        X.segment = P->tgt_len / gridDim.x;
        X.shard_cap = P->shard_cap;
        X.extras = P->extras;
        X.hot = hot;
        const DomainDesc &D = P->desc[hot];
        long long skipped = 0;
        for (int j = 0; j < D.n_jumps; j++)
            skipped += (long long)D.jump_hi[j] - D.jump_lo[j];
        X.hot_skipped = skipped;
    }
}

// Domain dom's descriptor: the shared copy for the hot domain. Static fields, and cycle / epoch.
__device__ __forceinline__ const DomainDesc &desc_of(const PassCtx &X, unsigned int dom) {
    return dom == X.hot ? X.hot_desc : X.desc[dom];
}

// The 26 critical lengths of record `pos` (cell `cell` of domain D): of its body, else the cell's own.
// Both hold the same values; the bodies of a long front lie in a few dozen MB, the rows of its cells
// all over an array of 104 bytes per cell.
__device__ __forceinline__ const float *row_of(const RecordList &L, const DomainDesc &D, unsigned int pos, unsigned int cell) {
    return pos < L.body_cap ? L.body[pos].cdl : D.cdl + 26ull * cell;
}

// A domain's dynamic fields in one load, past L1.
struct DomainDyn {
    int cycle;
    unsigned int epoch;
    int next_start, done;
};
__device__ __forceinline__ DomainDyn load_dyn(const DomainDesc &D) {
    static_assert(offsetof(DomainDesc, cycle) % 16 == 0 && offsetof(DomainDesc, epoch) == offsetof(DomainDesc, cycle) + 4 &&
                      offsetof(DomainDesc, next_start) == offsetof(DomainDesc, cycle) + 8 &&
                      offsetof(DomainDesc, done) == offsetof(DomainDesc, cycle) + 12,
                  "cycle, epoch, next_start and done are one 16-byte vector");
    const int4 v = __ldcg(reinterpret_cast<const int4 *>(&D.cycle));
    return DomainDyn{v.x, (unsigned int)v.y, v.z, v.w};
}

// What the growth of a domain's records needs of its descriptor: for the hot domain loaded once per
// growth pass, for the others per record (two 16-byte vectors of one 32-byte sector).
struct GrowView {
    const double *growth;
    int e_cycle; // executed cycles up to the current one
    int cycle;   // kDoneCycle: the domain has ended
    int growth_len;
    bool zero_du, jumps;
};
constexpr int kDoneCycle = INT_MIN;
__device__ __forceinline__ GrowView grow_view(const DomainDesc &D) {
    static_assert(offsetof(DomainDesc, growth) % 32 == 0 && offsetof(DomainDesc, growth_len) == offsetof(DomainDesc, growth) + 8 &&
                      offsetof(DomainDesc, zero_du) == offsetof(DomainDesc, growth) + 12 &&
                      offsetof(DomainDesc, n_jumps) == offsetof(DomainDesc, growth) + 14 &&
                      offsetof(DomainDesc, cycle) == offsetof(DomainDesc, growth) + 16,
                  "growth, growth_len, zero_du, n_jumps and the dynamic fields are one 32-byte sector");
    const int4 v = __ldcg(reinterpret_cast<const int4 *>(&D.growth));
    const DomainDyn dyn = load_dyn(D);
    GrowView g;
    g.growth = reinterpret_cast<const double *>((unsigned long long)(unsigned int)v.x | ((unsigned long long)(unsigned int)v.y << 32));
    g.growth_len = v.z;
    g.zero_du = (v.w & 0xffff) != 0;
    g.jumps = ((unsigned int)v.w >> 16) != 0;
    g.cycle = dyn.done ? kDoneCycle : dyn.cycle;
    g.e_cycle = g.jumps ? (int)executed_upto(D, dyn.cycle) : dyn.cycle;
    return g;
}
// What the short growth path needs of a domain without jumps, zero UndercoolingChange or growth extras;
// cycle kDoneCycle: its records take the general path. A block of the many-domain kernels holds those of
// the first kViews domains in shared memory, filled at each growth pass (one round of loads). Freed list
// positions are taken by whichever domain captures next in the block, so the records of a group of 32 come
// from many domains, and reading their descriptors' sectors per record put every warp's loads on the few
// L2 sectors that hold them. 256 domains: growth was 76 us per cycle at 2.2e6 records, three times a lone
// domain's per record; whole maps 1422 -> 1056 ms (96 domains 549 -> 516, 24 domains 418 -> 397). The
// short path with the fields still read from L2 gained nothing (574 against 547 ms at 96 domains).
struct alignas(16) ShortView {
    const double *table; // the growth table from the current cycle's entry, indexed by -CritTimeStep
    int cycle, len;
};
constexpr unsigned int kViews = 320; // what is left of 48 KB
__device__ __forceinline__ ShortView short_view(const DomainDesc &D, bool extras) {
    const GrowView g = grow_view(D);
    const bool plain = !extras && !g.jumps && !g.zero_du && g.cycle != kDoneCycle;
    return ShortView{g.growth + (plain ? g.cycle : 0), plain ? g.cycle : kDoneCycle, g.growth_len};
}
__device__ __forceinline__ GrowView hot_view(const PassCtx &X, const DomainDyn &dyn) {
    GrowView g;
    g.growth = X.hot_desc.growth;
    g.growth_len = X.hot_desc.growth_len;
    g.zero_du = X.hot_desc.zero_du != 0;
    g.jumps = X.hot_desc.n_jumps != 0;
    g.cycle = dyn.done ? kDoneCycle : dyn.cycle;
    g.e_cycle = dyn.cycle - (int)X.hot_skipped; // every jump ends below the current cycle
    return g;
}

// The diagonal's growth this cycle of a record of domain D: the table entry of the undercooling after
// the executed updates since the liquidus (src/CAupdate.cpp:236-237), plus those of earlier layers;
// the table of the cell's UndercoolingChange value. kNoGrowth beyond the table; 0 if not eligible.
constexpr double kNoGrowth = -1.0;
__device__ __forceinline__ double load_growth(const GrowView &g, const DomainDesc &D, unsigned int cell, int cts,
                                              bool extras) {
    if (!(g.cycle > cts))
        return 0.0;
    int nu = g.e_cycle - (g.jumps ? (int)executed_upto(D, cts) : max(cts, 0));
    const double *table = g.growth;
    if (extras) {
        if (D.nu_base)
            nu += __ldg(D.nu_base + cell);
        if (D.du_class)
            table += (size_t)__ldg(D.du_class + cell) * (size_t)g.growth_len;
    }
    if (g.zero_du && D.du[cell] == 0.0f)
        nu = 0;
    return (unsigned int)nu < (unsigned int)g.growth_len ? __ldg(table + nu) : kNoGrowth;
}

// Growth step of one record (status m, growth increment inc, its domain's cycle).
enum GrowAction {
    kDrop,  // dropped: finished domain, solidified by last cycle's re-check, or no liquid neighbour
    kWait,  // not eligible yet: unchanged
    kGrown, // r.dl grown
    kFlag   // grown, and its claim step is due: the mask must be built or the diagonal reached the
            // applicable lower bound of the liquid neighbours' critical lengths
};
__device__ __forceinline__ GrowAction grow_record(const PassCtx &X, int cycle, unsigned int cell, unsigned int dom, ActiveRec &r,
                                                  unsigned int m, double inc, float bound, CycleStats &st) {
    st.listed++;
    if (cycle == kDoneCycle || (m & kMaskDead)) {
        // a retired domain's records point at the placeholder descriptor, which has no fields
        float *dl = desc_of(X, dom).dl;
        if (dl)
            dl[cell] = r.dl;
        return kDrop;
    }
    if (!(cycle > r.cts))
        return kWait; // cts is INT_MAX outside the window and for LayerID > layer
    st.grown++;
    if (inc < 0.0) {
        atomicOr(&X.desc[dom].error, kErrGrowthTable);
        inc = 0.0;
    }
    r.dl = (float)((double)r.dl + inc);
    if ((m & kMaskFresh) || r.dl >= bound) {
        st.flagged++;
        return kFlag;
    }
    if ((m & kDirBits) == 0) {
        // no liquid neighbour: LCount stays 0 (src/CAupdate.cpp:722-725)
        const DomainDesc &D = desc_of(X, dom);
        D.ctype[cell] = kSolid;
        D.dl[cell] = r.dl;
        return kDrop;
    }
    return kGrown;
}

// The mask of a record next to cells that nucleated at the start of this cycle: without the
// directions that are no longer liquid (the nucleated cells; every other change cleared its bit).
__device__ __noinline__ unsigned int drop_nucleated(const DomainDesc &D, unsigned int c, unsigned int m) {
    const int plane = D.mx * D.my, my = D.my;
    const int8_t *ct = D.ctype + c;
    unsigned int gone = 0;
    for (unsigned int bits = m & kDirBits; bits; bits &= bits - 1) {
        const int l = __ffs(bits) - 1;
        if (!liquid_type(__ldcg(ct + nb_offset(l, plane, my))))
            gone |= 1u << l;
    }
    return m & ~(gone | kMaskNuc);
}

// Records the growth pass hands to the claim pass go to a global queue together with the state the
// claim pass needs (list position, cell, domain, liquid-neighbour mask, grown DiagonalLength), so the
// claim pass needs no dependent load before its own round of loads.
// Warp-aggregated reservation of n slots per lane on a global counter (every lane of the warp
// calls). Returns this lane's first slot, or ULLONG_MAX past `cap` (the pool error flag is set, and the
// counter stays past cap: shard_count).
__device__ __forceinline__ unsigned long long warp_reserve_n(unsigned long long *counter, unsigned long long cap,
                                                             int *error, unsigned int n) {
    const unsigned int lane = threadIdx.x & 31;
    unsigned int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (unsigned)o)
            incl += v;
    }
    const unsigned int total = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long base = 0;
    if (lane == 31 && total)
        base = atomicAdd(counter, (unsigned long long)total);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (base + total > cap) {
        if (lane == 31 && total)
            atomicOr(error, kErrListOverflow);
        return ULLONG_MAX;
    }
    return base + incl - n;
}

// A claim of cell c in the current cycle: later epochs and lower cells compare lower.
__device__ __forceinline__ unsigned long long claim_key(const DomainDesc &D, unsigned int c) {
    return ((unsigned long long)(0xffffffffu - D.epoch) << 32) | (unsigned long long)c;
}
// A listed claim: domain (13 bits), direction from the claimant and claimed cell; in a block's own list
// also 1 + the entry of BlockShared::claimants that holds the claimant's state (0: none).
constexpr int kClaimantShift = 50;
__device__ __forceinline__ unsigned long long claim_entry_of(unsigned int dom, int l, unsigned int t) {
    return ((unsigned long long)dom << 37) | ((unsigned long long)l << 32) | t;
}
__device__ __forceinline__ unsigned int claim_domain(unsigned long long e) { return (unsigned int)(e >> 37) & 0x1fffu; }

// A record the growth pass flagged for a claim step: its list position, domain, liquid mask and grown
// DiagonalLength.
struct ClaimItem {
    unsigned int pos, dom, mask;
    float dl;
};

// What a claim step leaves in one lane: the directions of its four that the record reaches, the claimant.
struct ClaimLane {
    unsigned int reach;       // bit j: direction dir0 + j
    int dir0;
    unsigned int cell, dom;
};

// The claim step of one flagged record by eight lanes (on: the group has one; every lane of the warp calls,
// src/CAupdate.cpp:320-352): lanes 1-7 read four critical lengths each (lane 0 the rest
// of the body), so a record is one 128-byte line in one load instruction of its group, and each lane compares four
// lengths. A record per lane, 26 lengths compared in turn from seven uncoalesced 16-byte loads, is the longer
// chain where a block has few of them (block_claims).
__device__ __forceinline__ ClaimLane claim_group(const PassCtx &X, int app, const ClaimItem &it, bool on, CycleStats &st,
                                                 unsigned int &tombs) {
    const unsigned int lane = threadIdx.x & 31, sub = lane & 7u, group = 0xffu << (lane & 24u);
    const RecordList &L = X.list[app];
    ClaimLane out{0u, 4 * (int)sub - 4, 0u, it.dom};
    if (!on)
        return out;
    const DomainDesc &D = desc_of(X, it.dom);
    ActiveRec *const rec = L.rec + it.pos;
    const unsigned int c = __ldcg(L.cell + it.pos); // a body does not wait for it
    out.cell = c;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (it.pos < L.body_cap) {
        static_assert(offsetof(RecordBody, cdl) == 16, "GrainID and DOCenter, then the lengths");
        v = __ldcg(reinterpret_cast<const float4 *>(L.body + it.pos) + sub);
    }
    else if (sub) {
        const float *row = D.cdl + 26ull * c + out.dir0;
        v.x = __ldcg(row);
        v.y = __ldcg(row + 1);
        if (sub < 7) {
            v.z = __ldcg(row + 2);
            v.w = __ldcg(row + 3);
        }
    }
    unsigned int m = it.mask;
    if (m & kMaskFresh) {
        // liquid neighbours from the 26 neighbour types (src/CAupdate.cpp:320-334); no other thread
        // writes this cell's mask now, captures and nucleations clear bits later. A cell claimed in
        // this same step (TemporaryUpdate) is still liquid.
        int rx, ry, rz;
        cell_coords(D, c, rx, ry, rz);
        const unsigned int valid = neighbour_mask(D, rx, ry, rz);
        const int plane = D.mx * D.my;
        m = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int l = out.dir0 + j;
            if (l >= 0 && l < 26 && ((valid >> l) & 1u) && liquid_type(__ldcg(D.ctype + c + nb_offset(l, plane, D.my))))
                m |= 1u << l;
        }
#pragma unroll
        for (int o = 4; o; o >>= 1)
            m |= __shfl_xor_sync(group, m, o);
        if (sub == 0) {
            st.fresh++;
            rec->stat = m | kMaskGrown; // a flagged record was grown this cycle
        }
    }
    m &= kDirBits;
    if (m == 0) {
        // no liquid neighbour: LCount stays 0 (src/CAupdate.cpp:722-725)
        if (sub == 0) {
            D.ctype[c] = kSolid;
            D.dl[c] = it.dl;
            rec->stat = kMaskTomb;
            st.dropped++;
            tombs++;
        }
        return out;
    }
    // Every reached cell is claimed and captured within this cycle, so the cached minimum only
    // covers the liquid neighbours not reached (+inf when none is left).
    const unsigned int mine = sub ? m >> out.dir0 : 0u;
    const float f[4] = {v.x, v.y, v.z, v.w};
    float mn = __int_as_float(0x7f800000), mn2 = mn;
    unsigned int d1 = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if ((mine >> j) & 1u) {
            if (it.dl >= f[j]) {
                out.reach |= 1u << j;
            }
            else if (f[j] < mn) {
                mn2 = mn;
                mn = f[j];
                d1 = (unsigned int)(out.dir0 + j);
            }
            else if (f[j] < mn2) {
                mn2 = f[j];
            }
        }
    }
#pragma unroll
    for (int o = 4; o; o >>= 1) {
        const float omn = __shfl_xor_sync(group, mn, o), omn2 = __shfl_xor_sync(group, mn2, o);
        const unsigned int od1 = __shfl_xor_sync(group, d1, o);
        if (omn < mn || (omn == mn && od1 < d1)) {
            mn2 = fminf(omn2, mn);
            mn = omn;
            d1 = od1;
        }
        else {
            mn2 = fminf(mn2, omn);
        }
    }
    if (sub == 0) {
        st.rows++;
        rec->cdl_min = mn;
        L.min2[it.pos] = mn2;
        L.dom[it.pos] = dom_word(it.dom, d1);
    }
    return out;
}

// The claim step of one flagged record by one lane: the form for blocks with hundreds of flagged
// records, whose loads are all in flight in one round. Returns the directions of the cells it reaches,
// which the caller claims (push_claims, issue_claims).
__device__ __forceinline__ unsigned int claim_record(const PassCtx &X, int app, const ClaimItem &it, unsigned int &c,
                                                     CycleStats &st, unsigned int &tombs) {
    const unsigned int i = it.pos, dom = it.dom;
    unsigned int m = it.mask;
    const float dl = it.dl;
    const DomainDesc &D = desc_of(X, dom);
    const RecordList &L = X.list[app];
    c = __ldcg(L.cell + i); // a body's row does not wait for it
    ActiveRec *recs = L.rec;
    const int plane = D.mx * D.my, my = D.my;
    // the 26 critical lengths as 7 aligned 16-byte loads: a cell's own row (26 * 4 * c bytes in) starts
    // on a 16-byte boundary for even c and 8 bytes past one for odd c, which read from 8 bytes before it
    // (the previous row's end). The 8 bytes read past an even row lie in the array, or for the last
    // row in the slot's next field array (sub-arrays start on 256-byte boundaries). A body's row is
    // even, with 8 bytes of its own after it.
    const float *const lengths = row_of(L, D, i, c);
    const bool odd = (reinterpret_cast<unsigned long long>(lengths) & 8u) != 0;
    const float4 *row = reinterpret_cast<const float4 *>(lengths - (odd ? 2 : 0));
    float f[28];
#pragma unroll
    for (int q = 0; q < 7; q++) {
        const float4 v = __ldcg(row + q);
        f[4 * q] = v.x;
        f[4 * q + 1] = v.y;
        f[4 * q + 2] = v.z;
        f[4 * q + 3] = v.w;
    }
    float cdl[26];
#pragma unroll
    for (int l = 0; l < 26; l++)
        cdl[l] = odd ? f[l + 2] : f[l];
    if (m & kMaskFresh) {
        // liquid neighbours from the 26 neighbour types (src/CAupdate.cpp:320-334); no other thread
        // writes this cell's mask now, captures and nucleations clear bits later. Invalid directions
        // read the cell itself. A cell claimed in this same step (TemporaryUpdate) is still liquid.
        st.fresh++;
        int rx, ry, rz;
        cell_coords(D, c, rx, ry, rz);
        const unsigned int valid = neighbour_mask(D, rx, ry, rz);
        const int8_t *ct = D.ctype + c;
        m = 0;
#pragma unroll
        for (int l = 0; l < 26; l++) {
            const bool v = (valid >> l) & 1u;
            const int8_t nt = __ldcg(ct + (v ? nb_offset(l, plane, my) : 0));
            m |= (v && liquid_type(nt)) ? (1u << l) : 0u;
        }
        recs[i].stat = m | kMaskGrown; // a flagged record was grown this cycle
    }
    if ((m & kDirBits) == 0) {
        // no liquid neighbour: LCount stays 0 (src/CAupdate.cpp:722-725)
        D.ctype[c] = kSolid;
        D.dl[c] = dl;
        recs[i].stat = kMaskTomb;
        st.dropped++;
        tombs++;
        return 0;
    }
    st.rows++;
    // Every reached cell is claimed and captured within this cycle, so the cached minimum only
    // covers the liquid neighbours not reached (+inf when none is left).
    float nm = __int_as_float(0x7f800000), nm2 = nm;
    unsigned int d1 = 0xffffffffu;
    unsigned int reach = 0;
#pragma unroll
    for (int l = 0; l < 26; l++) {
        if (m & (1u << l)) {
            if (dl >= cdl[l]) {
                reach |= 1u << l;
            }
            else if (cdl[l] < nm) {
                nm2 = nm;
                nm = cdl[l];
                d1 = l;
            }
            else if (cdl[l] < nm2) {
                nm2 = cdl[l];
            }
        }
    }
    recs[i].cdl_min = nm;
    L.min2[i] = nm2;
    L.dom[i] = dom_word(dom, d1);
    if (reach) {
        st.claims += __popc(reach);
    }
    return reach;
}

// The persistent kernel's working set of one block in shared memory. The records a block flags wait
// in its queue for its own claim step, which starts as soon as the block has grown its records (no
// grid-wide wait between growth and claims); records beyond kBlockQueue go to the global queue,
// whose claim pass then runs after a grid-wide barrier (a flag tells every block). The claims a block
// makes stay in its own list up to the capture pass, where the same block keeps the winners and
// captures them: nothing about a claim goes through global memory but the claim word itself. Claims
// beyond kBlockClaims go to the block's segment of PoolState::tgt.
constexpr int kBlockQueue = 1280;
constexpr int kBlockClaims = 1024;
constexpr int kFreeSlots = 1024;
// A winning claim, with the state of its claimant that the capture starts from.
struct WinItem {
    unsigned int t, c;    // captured cell, claimant
    unsigned int dom_dir; // (domain << 5) | direction from the claimant
    int h, cts;           // claimant's GrainID, CritTimeStep of t
    float docx, docy, docz;
    unsigned int slot; // of the new record (kNoRecord: none)
};
// What the geometry and the neighbours of a capture leave for its last stage.
struct CaptureItem {
    double cx, cy, cz; // centre of the new octahedron
    float dl;          // and its DiagonalLength
    unsigned int liq;  // the captured cell's liquid neighbours
};
constexpr int kCaptureItems = 128; // captures a block has in hand at a time

struct BlockShared {
    union {
        ClaimItem items[kBlockQueue]; // growth and claims
        WinItem wins[kBlock];         // capture
    };
    unsigned long long claims[kBlockClaims];
    unsigned int claim_pos[kBlockClaims]; // the claimant's record
    CaptureItem captures[kCaptureItems];
    float4 claimants[kBlock / 32]; // GrainID (bits) and DOCenter, kept by claim_warp for capture_claim
    unsigned int n_items;  // may exceed kBlockQueue (the excess went global)
    unsigned int n_claims; // may exceed kBlockClaims (the excess is in the block's segment)
    unsigned int n_wins;
    unsigned int n_first;    // cells of the hot domain this block was the first to claim this cycle
    unsigned int n_appended; // records appended this cycle (captures and nucleations)
    // Positions of dropped records that this block's captures may use again: those that it dropped
    // itself in this launch, and those that its growth met on the launch's first pass. n_free may
    // exceed kFreeSlots (the excess waits for a compaction); the captures of a cycle take the last
    // n_taken of them.
    unsigned int n_free, n_taken;
    int tombs; // change of the list's number of dropped records, not yet told to the grid
    unsigned int free_slots[kFreeSlots];
    unsigned int busy;       // 1: a record of the block was grown or dropped this cycle; kTellFlag beside it
    int min_cts;             // smallest CritTimeStep of the block's other records, while it is not busy
    PassCtx X;
};

// Puts the flagged records of one growth step into the claim queue (all lanes of the warp call).
template <int kBatch>
__device__ __forceinline__ void queue_flagged(PoolState *P, unsigned int shard, unsigned int nf, unsigned int flagged,
                                              const unsigned int *idx, const ActiveRec *r, const unsigned int *dom) {
    unsigned long long k = warp_reserve_n(&P->qcnt_s[shard].v, P->shard_cap, &P->error, nf);
    if (nf && k != ULLONG_MAX) {
        k += (unsigned long long)shard * P->shard_cap;
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
            if (flagged & (1u << q)) {
                P->qpos[k] = idx[q];
                P->qdom[k] = word_dom(dom[q]);
                P->qmask[k] = r[q].stat;
                P->qdl[k] = r[q].dl;
                k++;
            }
        }
    }
}

// Puts the flagged records of one growth step into the block's queue; those that do not fit go to
// the global queue (all lanes of the warp call). Every slot below kBlockQueue that a warp reserves
// is written in the same step, so the block's claim step reads only this cycle's records.
template <int kBatch>
__device__ __forceinline__ void block_queue_flagged(PoolState *P, BlockShared &B, unsigned int shard, unsigned int flagged,
                                                    const unsigned int *idx, const ActiveRec *r, const unsigned int *dom) {
    const unsigned int lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    unsigned int who[kBatch], total = 0;
#pragma unroll
    for (int q = 0; q < kBatch; q++) {
        who[q] = __ballot_sync(0xffffffffu, (flagged >> q) & 1u);
        total += __popc(who[q]);
    }
    if (total == 0)
        return;
    unsigned int base = 0;
    if (lane == 0)
        base = atomicAdd(&B.n_items, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    unsigned int first = base;
#pragma unroll
    for (int q = 0; q < kBatch; q++) {
        const unsigned int e = first + __popc(who[q] & below);
        if (((flagged >> q) & 1u) && e < (unsigned int)kBlockQueue)
            B.items[e] = ClaimItem{idx[q], word_dom(dom[q]), r[q].stat, r[q].dl};
        first += __popc(who[q]);
    }
    if (base + total > (unsigned int)kBlockQueue) {
        unsigned int beyond = 0;
        first = base;
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
            if (((flagged >> q) & 1u) && first + __popc(who[q] & below) >= (unsigned int)kBlockQueue)
                beyond |= 1u << q;
            first += __popc(who[q]);
        }
        queue_flagged<kBatch>(P, shard, __popc(beyond), beyond, idx, r, dom);
    }
}

// Claims of the block's list, and claim i of them (all threads agree after a block barrier).
__device__ __forceinline__ unsigned int claim_count(const BlockShared &B) {
    const unsigned long long most = kBlockClaims + B.X.segment;
    return B.n_claims < most ? B.n_claims : (unsigned int)most;
}
__device__ __forceinline__ unsigned long long claim_at(const BlockShared &B, unsigned int i) {
    return i < (unsigned int)kBlockClaims ? B.claims[i] : __ldcg(B.X.tgt + blockIdx.x * B.X.segment + (i - kBlockClaims));
}

// Puts the claims of one record per lane (all lanes of the warp call; reach 0: none) into the block's list.
__device__ __forceinline__ void push_claims(PoolState *P, BlockShared &B, unsigned int reach, unsigned int dom,
                                            unsigned int cell, unsigned int pos) {
    const unsigned int lane = threadIdx.x & 31, n = __popc(reach);
    unsigned int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (unsigned)o)
            incl += v;
    }
    unsigned int base = 0;
    if (lane == 31 && incl)
        base = atomicAdd(&B.n_claims, incl);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (reach) {
        const DomainDesc &D = desc_of(B.X, dom);
        const int plane = D.mx * D.my, my = D.my;
        unsigned int e = base + incl - n;
        for (unsigned int bits = reach; bits; bits &= bits - 1, e++) {
            const int l = __ffs(bits) - 1;
            const unsigned long long v = claim_entry_of(dom, l, (unsigned int)((long long)cell + nb_offset(l, plane, my)));
            if (e < (unsigned int)kBlockClaims) {
                B.claims[e] = v;
                B.claim_pos[e] = pos;
            }
            else {
                const unsigned long long k = e - kBlockClaims;
                if (k < B.X.segment)
                    B.X.tgt[blockIdx.x * B.X.segment + k] = v;
                else
                    atomicOr(&P->error, kErrListOverflow);
            }
        }
    }
}

// Issues the claims [first, claim_count) of the block's list, one per thread (src/CAupdate.cpp:336-352;
// all threads of the block call, after a block barrier). A claim that finds an older epoch in the
// claim word is the first on its cell, which is captured in this cycle: one liquid cell less, known
// before the capture pass. The hot domain's are counted in shared memory.
__device__ __forceinline__ void issue_claims(BlockShared &B, unsigned int first) {
    const unsigned int n = claim_count(B);
    unsigned int firsts = 0;
    for (unsigned int i = first + threadIdx.x; i < n; i += kBlock) {
        const unsigned long long e = claim_at(B, i);
        const unsigned int dom = claim_domain(e), t = (unsigned int)e;
        const DomainDesc &D = desc_of(B.X, dom);
        const unsigned int c = (unsigned int)((long long)t - nb_offset((int)((e >> 32) & 31u), D.mx * D.my, D.my));
        const unsigned long long key = claim_key(D, c);
        const unsigned long long old = atomicMin(D.claim + t, key);
        D.ctype[t] = kTemporaryUpdate;
        if ((old >> 32) != (key >> 32)) {
            if (dom == B.X.hot)
                firsts++;
            else
                atomicAdd((unsigned long long *)&B.X.desc[dom].liquid_shard[i & (kLiquidShards - 1)],
                          (unsigned long long)(-1ll));
        }
    }
    firsts = __reduce_add_sync(0xffffffffu, firsts);
    if ((threadIdx.x & 31) == 0 && firsts)
        atomicAdd(&B.n_first, firsts);
}

// The claim step of the block's item `i` by a whole warp: one direction per lane (claim_group and make_claims
// in one), the shortest chain for a block with no more flagged records than warps.
__device__ __forceinline__ void claim_warp(BlockShared &B, int app, unsigned int i, CycleStats &st, unsigned int &tombs) {
    const unsigned int lane = threadIdx.x & 31;
    const ClaimItem it = B.items[i];
    const unsigned int dom = it.dom;
    unsigned int m = it.mask;
    const DomainDesc &D = desc_of(B.X, dom);
    const int plane = D.mx * D.my, my = D.my;
    constexpr unsigned int kInf = 0x7f800000u;
    const RecordList &L = B.X.list[app];
    const unsigned int c = __ldcg(L.cell + it.pos); // a body does not wait for it
    // lanes 0-25: the critical lengths; 26: GrainID; 27-29: DOCenter
    unsigned int v = kInf;
    if (it.pos < L.body_cap) {
        if (lane < 30)
            v = __float_as_uint(__ldcg(reinterpret_cast<const float *>(L.body + it.pos) + (lane < 26 ? 4 + lane : lane - 26)));
    }
    else if (lane < 26)
        v = __float_as_uint(__ldcg(D.cdl + 26ull * c + lane));
    else if (lane == 26)
        v = (unsigned int)__ldcg(D.gid + c);
    else if (lane < 30)
        v = __float_as_uint(__ldcg(D.doc + 3ull * c + (lane - 27)));
    if (m & kMaskFresh) {
        // as claim_record
        int rx, ry, rz;
        cell_coords(D, c, rx, ry, rz);
        const bool nb = (neighbour_mask(D, rx, ry, rz) >> lane) & 1u;
        m = __ballot_sync(0xffffffffu, nb && liquid_type(__ldcg(D.ctype + c + (nb ? nb_offset((int)lane, plane, my) : 0))));
        if (lane == 0) {
            st.fresh++;
            L.rec[it.pos].stat = m | kMaskGrown;
        }
    }
    ActiveRec *rec = L.rec + it.pos;
    if ((m & kDirBits) == 0) {
        // no liquid neighbour: LCount stays 0 (src/CAupdate.cpp:722-725)
        if (lane == 0) {
            D.ctype[c] = kSolid;
            D.dl[c] = it.dl;
            rec->stat = kMaskTomb;
            st.dropped++;
            tombs++;
        }
        return;
    }
    const bool liquid = lane < 26 && ((m >> lane) & 1u), reached = liquid && it.dl >= __uint_as_float(v);
    const unsigned int reach = __ballot_sync(0xffffffffu, reached);
    if (reach) {
        unsigned int e = 0;
        if (lane == 0)
            e = atomicAdd(&B.n_claims, __popc(reach)); // at most 26 per warp: within kBlockClaims
        e = __shfl_sync(0xffffffffu, e, 0) + __popc(reach & ((1u << lane) - 1u));
        bool first = false;
        if (reached) {
            const unsigned int t = (unsigned int)((long long)c + nb_offset((int)lane, plane, my));
            const unsigned long long key = claim_key(D, c);
            const unsigned long long old = atomicMin(D.claim + t, key);
            D.ctype[t] = kTemporaryUpdate;
            B.claims[e] = claim_entry_of(dom, (int)lane, t) | ((unsigned long long)(i + 1) << kClaimantShift);
            B.claim_pos[e] = it.pos;
            first = (old >> 32) != (key >> 32);
            if (first && dom != B.X.hot)
                atomicAdd((unsigned long long *)&B.X.desc[dom].liquid_shard[lane & (kLiquidShards - 1)],
                          (unsigned long long)(-1ll));
        }
        if (lane >= 26 && lane < 30)
            reinterpret_cast<unsigned int *>(&B.claimants[i])[lane - 26] = v;
        const unsigned int firsts = __popc(__ballot_sync(0xffffffffu, first && dom == B.X.hot));
        if (lane == 0) {
            st.claims += __popc(reach);
            if (firsts)
                atomicAdd(&B.n_first, firsts);
        }
    }
    // the cached minimum over the liquid neighbours not reached, its lowest direction and the
    // second-smallest: lengths are not negative, so their bits order as the values do (a NaN counts
    // as +inf, which the comparisons of claim_record skip as well)
    const unsigned int b = liquid && !reached ? min(v, kInf) : kInf;
    const unsigned int nm = __reduce_min_sync(0xffffffffu, b);
    const unsigned int d1 = nm == kInf ? 0xffffffffu : (unsigned int)__ffs(__ballot_sync(0xffffffffu, b == nm)) - 1u;
    const unsigned int nm2 = __reduce_min_sync(0xffffffffu, lane == d1 ? kInf : b);
    if (lane == 0) {
        st.rows++;
        rec->cdl_min = __uint_as_float(nm);
        L.min2[it.pos] = __uint_as_float(nm2);
        L.dom[it.pos] = dom_word(dom, d1);
    }
}

// Makes a warp's claims (src/CAupdate.cpp:336-352): the lowest index wins. Nothing waits for the outcome:
// every claim is listed, in the block's own list, and the capture pass keeps the winner's. A claimed cell
// reads TemporaryUpdate until its capture makes it active, as in the reference's capture
// (src/CAupdate.cpp:343-352). A claim that finds an older epoch in the claim word is the first on its
// cell, which is captured in this cycle: one liquid cell less, known before the capture pass. The hot
// domain's are counted in shared memory.
__device__ __forceinline__ void make_claims(PoolState *P, BlockShared &B, const ClaimLane &cl, unsigned int pos,
                                            CycleStats &st) {
    const unsigned int lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    unsigned int who[4], total = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        who[j] = __ballot_sync(0xffffffffu, (cl.reach >> j) & 1u);
        total += __popc(who[j]);
    }
    if (total == 0)
        return;
    unsigned int base = 0;
    if (lane == 0)
        base = atomicAdd(&B.n_claims, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    unsigned int firsts = 0;
    if (cl.reach) {
        const DomainDesc &D = desc_of(B.X, cl.dom);
        const int plane = D.mx * D.my, my = D.my;
        const unsigned long long key = claim_key(D, cl.cell);
        unsigned long long old[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            old[j] = key;
            if ((cl.reach >> j) & 1u) {
                const unsigned int t = (unsigned int)((long long)cl.cell + nb_offset(cl.dir0 + j, plane, my));
                old[j] = atomicMin(D.claim + t, key);
                D.ctype[t] = kTemporaryUpdate;
                const unsigned int e = base + __popc(who[j] & below);
                const unsigned long long v = claim_entry_of(cl.dom, cl.dir0 + j, t);
                if (e < (unsigned int)kBlockClaims) {
                    B.claims[e] = v;
                    B.claim_pos[e] = pos;
                }
                else if (e - kBlockClaims < B.X.segment) {
                    B.X.tgt[blockIdx.x * B.X.segment + (e - kBlockClaims)] = v;
                }
                else {
                    atomicOr(&P->error, kErrListOverflow);
                }
            }
            base += __popc(who[j]);
        }
        st.claims += __popc(cl.reach);
#pragma unroll
        for (int j = 0; j < 4; j++)
            firsts += (old[j] >> 32) != (key >> 32) ? 1u : 0u;
        if (firsts && cl.dom != B.X.hot) {
            atomicAdd((unsigned long long *)&B.X.desc[cl.dom].liquid_shard[lane & (kLiquidShards - 1)],
                      (unsigned long long)(-(long long)firsts));
            firsts = 0;
        }
    }
    firsts = __reduce_add_sync(0xffffffffu, firsts);
    if (lane == 0 && firsts)
        atomicAdd(&B.n_first, firsts);
}

// The block's claim step over its queue (all threads of the block call, after the block's growth). In the
// families for shorter lists a warp per record where there are no more of them than warps, else eight lanes per
// record, consecutive records on different warps. In the one for long lists a record per lane: at 512^3 (270
// flagged records per block and cycle) 36.3 us per cycle against 40.1 with eight lanes, whose four rounds wait
// for memory in turn; at 256^3 (67) eight lanes take 16.9 against 17.9 with one.
template <int kFamily>
__device__ __forceinline__ void block_claims(PoolState *P, BlockShared &B, int app, CycleStats &st, unsigned int &tombs) {
    __syncthreads();
    const unsigned int n = min(B.n_items, (unsigned int)kBlockQueue);
    if (n == 0)
        return;
    constexpr unsigned int kWarps = kBlock / 32;
    const unsigned int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    if (kFamily != kLongList && n <= kWarps) {
        if (warp < n)
            claim_warp(B, app, warp, st, tombs);
    }
    else if (kFamily != kLongList) {
        for (unsigned int k0 = warp; k0 < n; k0 += 4 * kWarps) {
            const unsigned int k = k0 + lane / 8 * kWarps;
            const bool on = k < n;
            ClaimItem it{};
            if (on)
                it = B.items[k];
            const ClaimLane cl = claim_group(B.X, app, it, on, st, tombs);
            make_claims(P, B, cl, it.pos, st);
        }
    }
    else {
        for (unsigned int k0 = warp * 32; k0 < n; k0 += kBlock) {
            const unsigned int k = k0 + lane;
            unsigned int reach = 0, cell = 0;
            ClaimItem it{};
            if (k < n) {
                it = B.items[k];
                reach = claim_record(B.X, app, it, cell, st, tombs);
            }
            push_claims(P, B, reach, it.dom, cell, it.pos);
        }
        __syncthreads();
        issue_claims(B, 0);
    }
}

// The bodies of a warp's surviving records (one per lane, `moves`) to their new positions: a body at a
// time by eight lanes, four in flight; from the cell's own fields where the record had none.
__device__ __forceinline__ void move_bodies(const RecordList &from, const RecordList &to, const PassCtx &X, bool moves,
                                            unsigned int i, unsigned int pos, unsigned int cell, unsigned int dom) {
    const unsigned int lane = threadIdx.x & 31;
    unsigned int todo = __ballot_sync(0xffffffffu, moves && i < from.body_cap);
    const unsigned int gather = __ballot_sync(0xffffffffu, moves && i >= from.body_cap);
    while (todo) {
        // the lane's own body: the (lane / 8)-th of the next four
        unsigned int pick = todo;
        for (unsigned int k = 0; k < lane / 8 && pick; k++)
            pick &= pick - 1;
        const int src = pick ? __ffs(pick) - 1 : 0;
        const unsigned int si = __shfl_sync(0xffffffffu, i, src), sp = __shfl_sync(0xffffffffu, pos, src);
        if (pick)
            reinterpret_cast<float4 *>(to.body + sp)[lane & 7] = __ldcg(reinterpret_cast<const float4 *>(from.body + si) + (lane & 7));
        for (int k = 0; k < 4 && todo; k++)
            todo &= todo - 1;
    }
    if (gather && moves && i >= from.body_cap) {
        const DomainDesc &D = desc_of(X, dom);
        RecordBody &b = to.body[pos];
        body_head(b) = make_float4(__int_as_float(__ldcg(D.gid + cell)), __ldcg(D.doc + 3ull * cell), __ldcg(D.doc + 3ull * cell + 1),
                             __ldcg(D.doc + 3ull * cell + 2));
        for (int l = 0; l < 26; l++)
            b.cdl[l] = __ldcg(D.cdl + 26ull * cell + l);
    }
}

// Growth step of a compaction cycle: the survivors are written to the other list (rare; kept out of
// line).
__device__ __noinline__ void compact_pass(PoolState *P, const PassCtx &X, int cur, unsigned long long gw,
                                         unsigned long long nw, unsigned long long n, const DomainDyn &dyn,
                                         CycleStats &st, BlockShared *B) {
    const unsigned int lane = threadIdx.x & 31;
    const int nxt = cur ^ 1;
    const RecordList &from = X.list[cur], &to = X.list[nxt];
    const unsigned long long groups = (n + 31) / 32;
    for (unsigned long long g = gw; g < groups; g += nw) {
        const unsigned long long i = g * 32 + lane;
        bool keep = false, flag = false;
        ActiveRec r{};
        unsigned int cell = 0, word = 0, dom = 0;
        float mn2 = 0.0f;
        if (i < n) {
            const int4 v = __ldcg(reinterpret_cast<const int4 *>(from.rec + i));
            r = *reinterpret_cast<const ActiveRec *>(&v);
            cell = __ldcg(from.cell + i);
            word = __ldcg(from.dom + i);
            dom = word_dom(word);
            mn2 = __ldcg(from.min2 + i);
            if (!(r.stat & kMaskTomb)) {
                r.stat &= ~kMaskKeep;
                if (r.stat & kMaskNuc)
                    r.stat = drop_nucleated(desc_of(X, dom), cell, r.stat);
                const GrowView view = dom == X.hot ? hot_view(X, dyn) : grow_view(X.desc[dom]);
                const double inc = load_growth(view, desc_of(X, dom), cell, r.cts, X.extras);
                const GrowAction a = grow_record(X, view.cycle, cell, dom, r, r.stat, inc,
                                                 effective_min(r.cdl_min, mn2, r.stat, word), st);
                keep = a != kDrop;
                flag = a == kFlag;
                if (a >= kGrown)
                    r.stat |= kMaskGrown;
                if (!keep)
                    st.dropped++;
            }
        }
        const unsigned long long pos = warp_reserve_n(&P->cnt[nxt], X.capacity, &P->error, keep ? 1u : 0u);
        if (!(keep && pos != ULLONG_MAX))
            flag = false;
        else {
            to.rec[pos] = r;
            to.cell[pos] = cell;
            to.dom[pos] = word;
            to.min2[pos] = mn2;
            desc_of(X, dom).pos[cell] = (unsigned int)pos;
        }
        move_bodies(from, to, X, keep && pos < to.body_cap, (unsigned int)i, (unsigned int)pos, cell, dom);
        const unsigned int idx = (unsigned int)pos;
        if (B)
            block_queue_flagged<1>(P, *B, (unsigned int)(gw % kShards), flag ? 1u : 0u, &idx, &r, &word);
        else
            queue_flagged<1>(P, (unsigned int)(gw % kShards), flag ? 1u : 0u, flag ? 1u : 0u, &idx, &r, &word);
    }
}

// The position of a dropped record, for one of the block's later captures.
__device__ __forceinline__ void push_free(BlockShared &B, unsigned int pos) {
    const unsigned int e = atomicAdd(&B.n_free, 1u);
    if (e < (unsigned int)kFreeSlots)
        B.free_slots[e] = pos;
}

// Growth step of one record by one lane, every case of it: other domains, per-cell growth extras, cycle
// jumps, records that leave the list, masks to clear. Returns what became of it, its list entry updated.
struct GrowResult {
    GrowAction action;
    unsigned int stat;
    float dl;
};
template <bool kOwnClaims>
__device__ __forceinline__ GrowResult grow_any(const PassCtx &X, BlockShared *B, const DomainDyn &dyn, int cur, unsigned int idx,
                                             ActiveRec r, unsigned int cell, unsigned int word, float min2, CycleStats &st) {
    const RecordList &L = X.list[cur];
    const unsigned int dom = word_dom(word), before = r.stat;
    // the neighbour verdict of the previous cycle does not carry over
    r.stat &= ~kMaskKeep;
    if (r.stat & kMaskNuc)
        r.stat = drop_nucleated(desc_of(X, dom), cell, r.stat);
    const GrowView v = dom == X.hot ? hot_view(X, dyn) : grow_view(X.desc[dom]);
    const double inc = load_growth(v, desc_of(X, dom), cell, r.cts, X.extras);
    const GrowAction a =
        grow_record(X, v.cycle, cell, dom, r, r.stat, inc, effective_min(r.cdl_min, min2, r.stat, word), st);
    if (a == kDrop) {
        L.rec[idx].stat = kMaskTomb;
        if (kOwnClaims)
            push_free(*B, idx);
        st.dropped++;
        return GrowResult{a, kMaskTomb, r.dl};
    }
    if (a >= kGrown) {
        r.stat |= kMaskGrown;
        L.rec[idx].dl = r.dl;
    }
    if (r.stat != before)
        L.rec[idx].stat = r.stat;
    return GrowResult{a, r.stat, r.dl};
}
// The same out of line: one copy for the groups of a batch, which reach it rarely.
template <bool kOwnClaims>
__device__ __noinline__ GrowResult grow_slow(const PassCtx &X, BlockShared *B, DomainDyn dyn, int cur, unsigned int idx,
                                             ActiveRec r, unsigned int cell, unsigned int word, float min2, CycleStats &st) {
    return grow_any<kOwnClaims>(X, B, dyn, cur, idx, r, cell, word, min2, st);
}

// Growth of the list's groups of 32 consecutive records (one coalesced load), group g by warp g % (number of
// warps of the grid), consecutive warps on different blocks, so that records appended together spread over
// every SM; kBatch groups per warp in flight. No block-wide synchronisation. A record
// costs 24 bytes read (its 16-byte vector with the status word, its domain word and the second bound)
// and 4 written. Nearly every record of the hot domain takes the short path below (about 70 instead of
// 250 instructions per group of 32): eligible or waiting, with liquid neighbours. The others go through
// grow_slow, lane by lane. kCells (the shapes for short lists, where a round of loads more shows): the
// cell comes with the record, for 4 bytes more, so that the slow path does not wait for it and the short
// one takes domains with per-cell growth extras, jumps and zero UndercoolingChange too; without it the
// increment of a short-path record is one entry of the domain's table.
// kMany (pools of many domains): every domain's records take the short path, if it has no growth extras,
// jumps or zero UndercoolingChange; its growth fields come from the block's table of views.
template <int kBatch, bool kOwnClaims, bool kCells, bool kMany>
__device__ __forceinline__ void grow_groups(PoolState *P, const PassCtx &X, BlockShared *B, const DomainDyn &dyn, int cur,
                                            unsigned int n, unsigned int gw, unsigned int nw, bool first_pass,
                                            CycleStats &st, unsigned int &tombs, bool &busy, int &min_cts,
                                            const ShortView *views) {
    const unsigned int lane = threadIdx.x & 31, shard = gw % kShards;
    const RecordList &L = X.list[cur];
    ActiveRec *const in = L.rec;
    const unsigned int *const in_dom = L.dom, *const in_cell = L.cell;
    const float *const in_min2 = L.min2;
    const unsigned int groups = (n + 31) / 32;
    // the growth fields of the hot domain in registers; without the short path no record matches `hot`
    const GrowView v0 = hot_view(X, dyn);
    const bool extras = X.extras, plain = !extras && !v0.jumps && !v0.zero_du;
    const unsigned int hot = v0.cycle != kDoneCycle && (kCells || plain) ? X.hot : 0xffffffffu;
    const int cycle = v0.cycle;
    const double *const table = v0.growth + v0.e_cycle;
    // records are updated in place; dropped ones become tombstones
    for (unsigned int g0 = gw; g0 < groups; g0 += kBatch * nw) {
        ActiveRec r[kBatch];
        unsigned int word[kBatch], cell[kBatch], idx[kBatch];
        float min2[kBatch];
        double inc[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
            idx[q] = (g0 + q * nw) * 32 + lane;
            r[q].stat = kMaskTomb;
            if (g0 + q * nw < groups && idx[q] < n) {
                // streamed once per cycle: through L2 only
                const int4 v = __ldcg(reinterpret_cast<const int4 *>(in + idx[q]));
                r[q] = *reinterpret_cast<const ActiveRec *>(&v);
                word[q] = __ldcg(in_dom + idx[q]);
                min2[q] = __ldcg(in_min2 + idx[q]);
                if (kCells)
                    cell[q] = __ldcg(in_cell + idx[q]);
            }
        }
        // the short path: grows, or waits for its CritTimeStep
        unsigned int grows = 0, waits = 0;
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
            const unsigned int m = r[q].stat;
            inc[q] = 0.0;
            ShortView view{nullptr, kDoneCycle, 0};
            if (kMany && !(m & kMaskTomb) && word_dom(word[q]) < kViews)
                view = views[word_dom(word[q])];
            if (!(m & (kMaskTomb | kMaskDead | kMaskNuc | kMaskFresh)) && (m & kDirBits) &&
                (kMany ? view.cycle != kDoneCycle : word_dom(word[q]) == hot)) {
                if ((kMany ? view.cycle : cycle) > r[q].cts) {
                    if (kMany) {
                        const int from = max(r[q].cts, 0);
                        if ((unsigned int)(view.cycle - from) < (unsigned int)view.len) {
                            grows |= 1u << q;
                            inc[q] = __ldg(view.table - from);
                        }
                    }
                    else if (kCells && !plain) {
                        inc[q] = load_growth(v0, X.hot_desc, cell[q], r[q].cts, extras);
                        if (inc[q] >= 0.0)
                            grows |= 1u << q;
                    }
                    else {
                        const int from = max(r[q].cts, 0);
                        if ((unsigned int)(v0.e_cycle - from) < (unsigned int)v0.growth_len) {
                            grows |= 1u << q;
                            inc[q] = __ldg(table - from);
                        }
                    }
                }
                else if (!(m & kMaskKeep)) {
                    waits |= 1u << q;
                    min_cts = min(min_cts, r[q].cts);
                }
            }
        }
        unsigned int flagged = 0;
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
            if ((grows >> q) & 1u) {
                const unsigned int m = (r[q].stat & ~kMaskKeep) | kMaskGrown;
                r[q].dl = (float)((double)r[q].dl + inc[q]);
                in[idx[q]].dl = r[q].dl;
                if (m != r[q].stat)
                    in[idx[q]].stat = m;
                r[q].stat = m;
                if (r[q].dl >= effective_min(r[q].cdl_min, min2[q], m, word[q])) {
                    flagged |= 1u << q;
                    if (!kCells && idx[q] < L.body_cap) // the claim step's line, on its way to L2 meanwhile
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(L.body + idx[q]));
                }
            }
        }
        st.listed += __popc(grows | waits);
        st.grown += __popc(grows);
        st.flagged += __popc(flagged);
        busy = busy || grows != 0;
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
            if (((grows | waits) >> q) & 1u)
                continue;
            if (r[q].stat & kMaskTomb) {
                if (kOwnClaims && first_pass && g0 + q * nw < groups && idx[q] < n)
                    push_free(*B, idx[q]);
                continue;
            }
            const unsigned int c = kCells ? cell[q] : __ldcg(in_cell + idx[q]);
            const GrowResult a = kBatch == 1 ? grow_any<kOwnClaims>(X, B, dyn, cur, idx[q], r[q], c, word[q], min2[q], st)
                                             : grow_slow<kOwnClaims>(X, B, dyn, cur, idx[q], r[q], c, word[q], min2[q], st);
            r[q].stat = a.stat;
            r[q].dl = a.dl;
            if (a.action == kWait) {
                min_cts = min(min_cts, r[q].cts);
                continue;
            }
            busy = true;
            if (a.action == kDrop)
                tombs++;
            else if (a.action == kFlag)
                flagged |= 1u << q;
        }
        if (kOwnClaims)
            block_queue_flagged<kBatch>(P, *B, shard, flagged, idx, r, word);
        else
            queue_flagged<kBatch>(P, shard, __popc(flagged), flagged, idx, r, word);
    }
}

// With kOwnClaims (B given) the block's flagged records go to its queue and their claim steps follow
// here. cur is the list to read, n its length; with `compact` the survivors go to the other list.
template <int kBatch, bool kOwnClaims, int kFamily, bool kMany>
__device__ void grow_pass(PoolState *P, PassCtx &X, BlockShared *B, const DomainDyn &dyn, int cur, unsigned long long n,
                          bool compact, bool first_pass, CycleStats &st, unsigned int &tombs,
                          const ShortView *views = nullptr) {
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned long long nw = (unsigned long long)gridDim.x * (kBlock / 32);
    const unsigned long long gw = (unsigned long long)warp * gridDim.x + blockIdx.x;
    if (kOwnClaims && threadIdx.x == 0) {
        // read by the block's claim step, after its first barrier
        X.hot_desc.cycle = dyn.cycle;
        X.hot_desc.epoch = dyn.epoch;
    }
    if (compact) {
        compact_pass(P, X, cur, gw, nw, n, dyn, st, kOwnClaims ? B : nullptr);
        if (kOwnClaims) {
            B->busy = 1;
            block_claims<kFamily>(P, *B, cur ^ 1, st, tombs);
        }
        return;
    }
    // whether a record was grown or dropped, and the smallest CritTimeStep of the others
    bool busy = false;
    int min_cts = INT_MAX;
    // one group per warp at most: the shorter code for one group is the shorter chain
    if (kFamily != kLongList && (n + 31) / 32 <= nw)
        grow_groups<1, kOwnClaims, true, kMany>(P, X, B, dyn, cur, (unsigned int)n, (unsigned int)gw, (unsigned int)nw, first_pass, st,
                                   tombs, busy, min_cts, views);
    else
        grow_groups<kBatch, kOwnClaims, kFamily != kLongList, kMany>(P, X, B, dyn, cur, (unsigned int)n, (unsigned int)gw, (unsigned int)nw, first_pass,
                                        st, tombs, busy, min_cts, views);
    if (kOwnClaims) {
        busy = __any_sync(0xffffffffu, busy);
        min_cts = __reduce_min_sync(0xffffffffu, min_cts);
        if (lane == 0) {
            if (busy)
                B->busy = 1; // the same value from every warp
            else if (min_cts != INT_MAX)
                atomicMin(&B->min_cts, min_cts);
        }
        block_claims<kFamily>(P, *B, cur, st, tombs);
    }
}

// Dropped records stay as tombstones of the in-place list until the next compaction; the separate
// kernels count them in shards.
__device__ __forceinline__ void add_tombs(PoolState *P, unsigned int tombs) {
    tombs = __reduce_add_sync(0xffffffffu, tombs);
    if ((threadIdx.x & 31) == 0 && tombs)
        atomicAdd(&P->tomb_s[(blockIdx.x + (threadIdx.x >> 5)) % kShards].v, (unsigned long long)tombs);
}

// Exclusive prefix of the shard counts in shared memory (all threads of the block call).
__device__ __forceinline__ void shard_prefix(const ShardCounter *cnt, unsigned long long cap, unsigned long long *pre) {
    if (threadIdx.x < 32) {
        const unsigned int lane = threadIdx.x;
        const unsigned long long c = shard_count(cnt[lane], cap);
        unsigned long long incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (unsigned)o)
                incl += v;
        }
        pre[lane + 1] = incl;
        if (lane == 0)
            pre[0] = 0;
    }
    __syncthreads();
}

// Position in the sharded array of the k-th entry of the shards' concatenation.
__device__ __forceinline__ unsigned long long shard_entry(const unsigned long long *pre, unsigned long long cap,
                                                          unsigned long long k) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step; step >>= 1)
        if (pre[lo + step] <= k)
            lo += step;
    return (unsigned long long)lo * cap + (k - pre[lo]);
}

// The claim steps of the global queue, eight lanes per entry, consecutive warps on different blocks;
// every claim is listed, in the block's own list (B, persistent kernel) or, as (domain << 37) |
// (direction << 32) | claimed cell, in the sharded global one.
template <bool kOwnClaims>
__device__ void claim_pass(PoolState *P, PassCtx &X, BlockShared *B, int app, CycleStats &st, unsigned int &tombs) {
    __shared__ unsigned long long s_pre[kShards + 1];
    const unsigned long long cap = X.shard_cap;
    shard_prefix(P->qcnt_s, cap, s_pre);
    const unsigned long long nq = s_pre[kShards];
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned long long nw = (unsigned long long)gridDim.x * (kBlock / 32);
    const unsigned long long gw = (unsigned long long)warp * gridDim.x + blockIdx.x;
    for (unsigned long long k0 = gw * 4; k0 < nq; k0 += nw * 4) {
        const unsigned long long k = k0 + lane / 8;
        const bool on = k < nq;
        ClaimItem it{};
        if (on) {
            const unsigned long long e = shard_entry(s_pre, cap, k);
            it = ClaimItem{__ldcg(P->qpos + e), __ldcg(P->qdom + e), __ldcg(P->qmask + e), __ldcg(P->qdl + e)};
        }
        const ClaimLane cl = claim_group(X, app, it, on, st, tombs);
        if (kOwnClaims) {
            make_claims(P, *B, cl, it.pos, st);
        }
        else {
            const unsigned int shard = (unsigned int)(gw % kShards);
            unsigned long long pos = warp_reserve_n(&P->tcnt_s[shard].v, cap, &P->error, __popc(cl.reach));
            if (cl.reach) {
                const DomainDesc &D = desc_of(X, cl.dom);
                const unsigned long long key = claim_key(D, cl.cell);
                for (unsigned int bits = cl.reach; bits; bits &= bits - 1) {
                    const int l = cl.dir0 + __ffs(bits) - 1;
                    const unsigned int t = (unsigned int)((long long)cl.cell + nb_offset(l, D.mx * D.my, D.my));
                    atomicMin(D.claim + t, key);
                    D.ctype[t] = kTemporaryUpdate;
                    if (pos != ULLONG_MAX)
                        P->tgt[shard * cap + pos++] = claim_entry_of(cl.dom, l, t);
                }
                st.claims += __popc(cl.reach);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Capture of liquid cell t by active cell c (src/CAupdate.cpp:353-563, 713-717), in three parts: the
// geometry (one thread per capture), the neighbours of the captured cell, and the critical lengths.

// The new octahedron, from the claimant's GrainID and centre, with the reference's expressions.
__device__ __forceinline__ void capture_geometry(const DomainDesc &D, unsigned int t, int h, float docx, float docy,
                                                 float docz, CaptureItem &out) {
    int rx, ry, rz;
    cell_coords(D, t, rx, ry, rz);
    int ori = (abs(h) - 1) % 10000;
    if (ori < 0)
        ori += 10000;
    const float *g = D.guv + 9 * ori;
    const float g0 = g[0], g1 = g[1], g2 = g[2], g3 = g[3], g4 = g[4], g5 = g[5], g6 = g[6], g7 = g[7], g8 = g[8];
    const double cxold = docx, cyold = docy, czold = docz;
    const double xp = (rx + D.xoff) + 0.5, yp = (ry + D.yoff) + 0.5, zp = rz + 0.5;
    const double x0 = xp - cxold, y0 = yp - cyold, z0 = zp - czold;
    const double mag0 = sqrtf((float)(x0 * x0 + y0 * y0 + z0 * z0));
    // Angle1..3 (src/CAupdate.cpp:382-393) matter by their signs alone: that of the dot product, without
    // the division by the distance, unless the quotient could vanish
    const auto negative = [&](float a, float b, float c) {
        const double dot = a * x0 + b * y0 + c * z0;
        return (dot < -1e-200 && mag0 < 1e30) || dot / mag0 < 0;
    };
    const float s1 = negative(g0, g1, g2) ? 1.0f : -1.0f, s2 = negative(g3, g4, g5) ? 1.0f : -1.0f,
                s3 = negative(g6, g7, g8) ? 1.0f : -1.0f;
    double Diag1X = g0 * s1, Diag1Y = g1 * s1, Diag1Z = g2 * s1;
    double Diag2X = g3 * s2, Diag2Y = g4 * s2, Diag2Z = g5 * s2;
    double Diag3X = g6 * s3, Diag3Y = g7 * s3, Diag3Z = g8 * s3;
    double U1x = Diag2X - Diag1X, U1y = Diag2Y - Diag1Y, U1z = Diag2Z - Diag1Z;
    double U2x = Diag3X - Diag1X, U2y = Diag3Y - Diag1Y, U2z = Diag3Z - Diag1Z;
    double UUx = U1y * U2z - U1z * U2y;
    double UUy = U1z * U2x - U1x * U2z;
    double UUz = U1x * U2y - U1y * U2x;
    double NDem = sqrtf((float)(UUx * UUx + UUy * UUy + UUz * UUz));
    double n0 = UUx / NDem, n1 = UUy / NDem, n2 = UUz / NDem;
    double ParaT = (n0 * x0 + n1 * y0 + n2 * z0) / (n0 * Diag1X + n1 * Diag1Y + n2 * Diag1Z);
    const double TX0 = cxold + ParaT * Diag1X, TY0 = cyold + ParaT * Diag1Y, TZ0 = czold + ParaT * Diag1Z;
    const double TX1 = cxold + ParaT * Diag2X, TY1 = cyold + ParaT * Diag2Y, TZ1 = czold + ParaT * Diag2Z;
    const double TX2 = cxold + ParaT * Diag3X, TY2 = cyold + ParaT * Diag3Y, TZ2 = czold + ParaT * Diag3Z;
    const auto distance = [](double ax, double ay, double az, double bx, double by, double bz) -> double {
        return sqrtf((float)(((ax - bx) * (ax - bx)) + ((ay - by) * (ay - by)) + ((az - bz) * (az - bz))));
    };
    const double Dist0 = distance(TX0, TY0, TZ0, xp, yp, zp), Dist1 = distance(TX1, TY1, TZ1, xp, yp, zp),
                 Dist2 = distance(TX2, TY2, TZ2, xp, yp, zp);
    int x = (Dist0 < Dist1);
    int y = (Dist1 < Dist2);
    int z = (Dist2 < Dist0);
    // 0, 1 or 2; the points idx, idx + 1 and idx + 2 (mod 3) by selects, without a local array
    int idx = 2 * (z - y) * z + (y - x) * y;
    const bool p0 = idx == 0, p1 = idx == 1;
    double mindist = p0 ? Dist0 : (p1 ? Dist1 : Dist2);
    double xc = p0 ? TX0 : (p1 ? TX1 : TX2), yc = p0 ? TY0 : (p1 ? TY1 : TY2), zc = p0 ? TZ0 : (p1 ? TZ1 : TZ2);
    double x1 = p0 ? TX1 : (p1 ? TX2 : TX0), y1 = p0 ? TY1 : (p1 ? TY2 : TY0), z1 = p0 ? TZ1 : (p1 ? TZ2 : TZ0);
    double x2 = p0 ? TX2 : (p1 ? TX0 : TX1), y2 = p0 ? TY2 : (p1 ? TY0 : TY1), z2 = p0 ? TZ2 : (p1 ? TZ0 : TZ1);
    double D1 = distance(xp, yp, zp, x2, y2, z2), D2 = distance(xc, yc, zc, x2, y2, z2);
    double D3 = distance(xp, yp, zp, x1, y1, z1), D4 = distance(xc, yc, zc, x1, y1, z1);
    double I1 = 0, I2 = D2, J1 = 0, J2 = D4;
    if (mindist != 0) {
        I1 = D1 * ((xp - x2) * (xc - x2) + (yp - y2) * (yc - y2) + (zp - z2) * (zc - z2)) / (D1 * D2);
        I2 = D2 - I1;
        J1 = D3 * ((xp - x1) * (xc - x1) + (yp - y1) * (yc - y1) + (zp - z1) * (zc - z1)) / (D3 * D4);
        J2 = D4 - J1;
    }
    const double sqrt3 = sqrt(3.0);
    double L12 = 0.5 * (dmin(I1, sqrt3) + dmin(I2, sqrt3));
    double L13 = 0.5 * (dmin(J1, sqrt3) + dmin(J2, sqrt3));
    double NewODiagL = sqrt(2.0) * dmax(L12, L13);
    double cd0 = xc - cxold, cd1 = yc - cyold, cd2 = zc - czold;
    double nd = sqrt(cd0 * cd0 + cd1 * cd1 + cd2 * cd2);
    double uv0 = cd0 / nd, uv1 = cd1 / nd, uv2 = cd2 / nd;
    out.cx = xc - NewODiagL * uv0;
    out.cy = yc - NewODiagL * uv1;
    out.cz = zc - NewODiagL * uv2;
    out.dl = (float)NewODiagL;
}

// The critical lengths of capture w by a group of `per` lanes (a power of two; group: their mask), and with
// them the new record, in slot w.slot of list L.
__device__ __forceinline__ void capture_lengths(const DomainDesc &D, const RecordList &L, const WinItem &w,
                                                const CaptureItem &o, int per, int sub, unsigned int group,
                                                CycleStats &st) {
    const unsigned int t = w.t, dom = w.dom_dir >> 5;
    int rx, ry, rz;
    cell_coords(D, t, rx, ry, rz);
    const double xp = (rx + D.xoff) + 0.5, yp = (ry + D.yoff) + 0.5, zp = rz + 0.5;
    int ori = (abs(w.h) - 1) % 10000;
    if (ori < 0)
        ori += 10000;
    const float *g = D.guv + 9 * ori;
    const float g0 = g[0], g1 = g[1], g2 = g[2], g3 = g[3], g4 = g[4], g5 = g[5], g6 = g[6], g7 = g[7], g8 = g[8];
    const double cx = o.cx, cy = o.cy, cz = o.cz;
    const bool has_body = w.slot < L.body_cap;
    float *const row = D.cdl + 26ull * t, *const body_row = L.body[has_body ? w.slot : 0].cdl;
    // face normals: float sums of the unit-vector components (src/CAupdate.cpp:526-551)
    double Fx[4], Fy[4], Fz[4];
    Fx[0] = g0 + g3 + g6;
    Fx[1] = g0 - g3 + g6;
    Fx[2] = g0 + g3 - g6;
    Fx[3] = g0 - g3 - g6;
    Fy[0] = g1 + g4 + g7;
    Fy[1] = g1 - g4 + g7;
    Fy[2] = g1 + g4 - g7;
    Fy[3] = g1 - g4 - g7;
    Fz[0] = g2 + g5 + g8;
    Fz[1] = g2 - g5 + g8;
    Fz[2] = g2 + g5 - g8;
    Fz[3] = g2 - g5 - g8;
    // the new record's cached minimum over its liquid neighbours, with its direction and the
    // second-smallest (the state a claim step leaves), so that its first claim step runs only once
    // its DiagonalLength reaches a liquid neighbour
    float mn = __int_as_float(0x7f800000), mn2 = mn;
    unsigned int d1 = 0xffffffffu;
#pragma unroll 1
    for (int n = sub; n < 26; n += per) {
        double a0 = xp + nb_dx(n) - cx;
        double b0 = yp + nb_dy(n) - cy;
        double d0 = zp + nb_dz(n) - cz;
        double q0 = a0 * Fx[0] + b0 * Fy[0] + d0 * Fz[0];
        double q1 = a0 * Fx[1] + b0 * Fy[1] + d0 * Fz[1];
        double q2 = a0 * Fx[2] + b0 * Fy[2] + d0 * Fz[2];
        double q3 = a0 * Fx[3] + b0 * Fy[3] + d0 * Fz[3];
        double m = dmax(dmax(fabs(q0), fabs(q1)), dmax(fabs(q2), fabs(q3)));
        const float v = (float)m;
        row[n] = v;
        if (has_body)
            body_row[n] = v;
        if ((o.liq >> n) & 1u) {
            if (v < mn) {
                mn2 = mn;
                mn = v;
                d1 = (unsigned int)n;
            }
            else if (v < mn2) {
                mn2 = v;
            }
        }
    }
#pragma unroll 1
    for (int k = per / 2; k; k >>= 1) {
        const float omn = __shfl_xor_sync(group, mn, k), omn2 = __shfl_xor_sync(group, mn2, k);
        const unsigned int od1 = __shfl_xor_sync(group, d1, k);
        if (omn < mn || (omn == mn && od1 < d1)) {
            mn2 = fminf(omn2, mn);
            mn = omn;
            d1 = od1;
        }
        else {
            mn2 = fminf(mn2, omn);
        }
    }
    if (sub != 0)
        return;
    D.gid[t] = w.h;
    D.dl[t] = o.dl;
    D.doc[3ull * t + 0] = (float)cx;
    D.doc[3ull * t + 1] = (float)cy;
    D.doc[3ull * t + 2] = (float)cz;
    if (has_body)
        body_head(L.body[w.slot]) = make_float4(__int_as_float(w.h), (float)cx, (float)cy, (float)cz);
    if (w.slot != kNoRecord) {
        L.rec[w.slot] = ActiveRec{o.dl, mn, w.cts, o.liq};
        L.cell[w.slot] = t;
        L.dom[w.slot] = dom_word(dom, d1);
        L.min2[w.slot] = mn2;
        D.pos[t] = w.slot;
    }
    // read as active by the growth pass of the next cycle, after the octahedron is written
    D.ctype[t] = kActive;
    st.captured++;
}

// The neighbours of captured cell w.t by a warp, lane s < 26 the neighbour of slot s (slot_dir: a load
// instruction's lanes read neighbours in few rows of three consecutive cells): the cell's liquid mask,
// and the masks and solidification re-checks of its active neighbours. kN captures at a time, their
// loads in flight together. Records of the cells active at the start of the cycle lie below base; a cell
// of type also_liquid (a mark of the cycle after next, or kLiquid) is liquid in the next cycle.
template <int kN>
__device__ __forceinline__ void capture_neighbours(const PassCtx &X, int app, unsigned long long base, const WinItem *wins,
                                                   CaptureItem *items, unsigned int first, unsigned int stride,
                                                   unsigned int n, int8_t also_liquid, CycleStats &st) {
    const unsigned int lane = threadIdx.x & 31;
    const int dir = slot_dir((int)lane);
    const bool has = dir < 26;
    const int dx = has ? nb_dx(dir) : 0, dy = has ? nb_dy(dir) : 0, dz = has ? nb_dz(dir) : 0;
    const unsigned int dir_bit = has ? 1u << dir : 0u, opp_bit = has ? 1u << nb_opp(dir) : 0u;
    ActiveRec *const rec = X.list[app].rec;
    for (unsigned int i0 = first; i0 < n; i0 += kN * stride) {
        int8_t ct[kN];
        unsigned int p[kN], a[kN], c[kN], old[kN];
        bool in[kN];
#pragma unroll
        for (int k = 0; k < kN; k++) {
            const unsigned int i = i0 + k * stride;
            in[k] = false;
            ct[k] = kWall;
            p[k] = kNoRecord;
            a[k] = c[k] = 0;
            if (i < n) {
                const DomainDesc &D = desc_of(X, wins[i].dom_dir >> 5);
                const unsigned int t = wins[i].t;
                c[k] = wins[i].c;
                int tx, ty, tz;
                cell_coords(D, t, tx, ty, tz);
                in[k] = (neighbour_mask(D, tx, ty, tz) & dir_bit) != 0;
                a[k] = (unsigned int)((long long)t + (in[k] ? (dz * D.mx + dx) * D.my + dy : 0));
                if (in[k]) {
                    ct[k] = __ldcg(D.ctype + a[k]);
                    p[k] = __ldcg(D.pos + a[k]);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kN; k++) {
            const unsigned int i = i0 + k * stride;
            if (i >= n) // the whole warp agrees
                break;
            // The captured cell's liquid-neighbour mask, as its first claim step would build it from the
            // neighbour types at the start of a later cycle: the neighbours still liquid (a neighbour
            // claimed in this cycle reads TemporaryUpdate, or active once captured). Later captures and
            // nucleations clear bits of it as of every other record's.
            const unsigned int liq =
                __reduce_or_sync(0xffffffffu, in[k] && (ct[k] == kLiquid || ct[k] == also_liquid) ? dir_bit : 0u);
            if (lane == 0)
                items[i].liq = liq;
            // Serial order (src/CAupdate.cpp:333-334, 722-725): active cell a saw the captured cell t
            // as liquid iff t's capturer c does not precede a. a keeps a liquid neighbour iff it has an
            // unclaimed one (a set mask bit that nobody clears) or a claimed one with c >= a. Every
            // claimed liquid neighbour clears its own bit exactly once, so the update that clears the
            // last direction bit sees the final verdict: KEEP is always set before the clear of the
            // same update, and an update's two atomics reach the word in program order. Only records of
            // cells active at the start of the cycle (positions below base) need to take part. A neighbour
            // captured in this same cycle may show up too, as active with a position used again: its mask
            // has no bit for t (claimed when it was built), so the clear finds none and no re-check
            // follows, and a KEEP set after its record was written goes with the next growth step.
            in[k] = in[k] && ct[k] == kActive && p[k] < base;
            if (in[k] && c[k] >= a[k])
                atomicOr(&rec[p[k]].stat, kMaskKeep);
            old[k] = in[k] ? atomicAnd(&rec[p[k]].stat, ~opp_bit) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kN; k++) {
            if (!in[k] || (old[k] & (kMaskFresh | kMaskDead | kMaskKeep)) || (old[k] & kDirBits) != opp_bit ||
                !(old[k] & kMaskGrown))
                continue;
            // a lost its last liquid neighbour; it solidifies if it was grown this cycle (cycle >
            // its CritTimeStep, src/CAupdate.cpp:257-261)
            st.rechecks++;
            desc_of(X, wins[i0 + k * stride].dom_dir >> 5).ctype[a[k]] = kSolid;
            atomicOr(&rec[p[k]].stat, kMaskDead);
        }
    }
}

// Listed claim e: whether it won (the lowest claimant index holds the claim word) and its capture's
// starting state, in one round of loads. pos: the claimant's record in list L (kNoRecord: not known).
__device__ __forceinline__ bool load_win(const PassCtx &X, const RecordList &L, unsigned long long e, unsigned int pos,
                                         WinItem &w) {
    const unsigned int dom = claim_domain(e);
    const int l = (int)((e >> 32) & 31u);
    const DomainDesc &D = desc_of(X, dom);
    w.t = (unsigned int)e;
    w.c = (unsigned int)((long long)w.t - nb_offset(l, D.mx * D.my, D.my));
    w.dom_dir = (dom << 5) | (unsigned int)l;
    w.slot = kNoRecord;
    const unsigned long long key = __ldcg(D.claim + w.t);
    w.cts = __ldg(D.cts_run + w.t);
    if (pos < L.body_cap) {
        const float4 head = __ldcg(&body_head(L.body[pos]));
        w.h = __float_as_int(head.x);
        w.docx = head.y;
        w.docy = head.z;
        w.docz = head.w;
    }
    else {
        w.h = __ldcg(D.gid + w.c);
        w.docx = __ldcg(D.doc + 3ull * w.c + 0);
        w.docy = __ldcg(D.doc + 3ull * w.c + 1);
        w.docz = __ldcg(D.doc + 3ull * w.c + 2);
    }
    return (unsigned int)key == w.c;
}

// A barrier of the block's first `threads` threads (a multiple of 32).
__device__ __forceinline__ void capture_sync(unsigned int threads) {
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// The critical lengths of captures 0 .. n - 1 by the block's first `threads` threads.
__device__ __forceinline__ void capture_lengths_of(const PassCtx &X, const WinItem *w, const CaptureItem *items, unsigned int n,
                                                   unsigned int threads, int app, CycleStats &st) {
    unsigned int per = 32;
    while (per > 4 && n * per > threads)
        per >>= 1;
    const unsigned int lane = threadIdx.x & 31, in_group = lane & (per - 1u);
    const unsigned int group = (per == 32 ? 0xffffffffu : ((1u << per) - 1u)) << (lane - in_group);
    for (unsigned int i = threadIdx.x / per; i < n; i += threads / per)
        capture_lengths(desc_of(X, w[i].dom_dir >> 5), X.list[app], w[i], items[i], (int)per, (int)in_group, group, st);
}

// Captures of n winners by the block's first `threads` threads (at least 256), at most kCaptureItems at a
// time, in two stages with a barrier between them. First the geometry, one thread per capture in the
// first warps, while the other warps do the neighbours, a warp per capture: neither needs the other, and
// the geometry of a whole block is one chain (its nine divisions and nine roots of a capture overlap)
// instead of one per group of lanes. Then the critical lengths, as many lanes per capture (4-32) as the
// block has threads. alloc(wins, m), called by one warp in the first stage, sets the slots of m winners.
// kN: captures whose neighbours a warp has in flight.
template <int kN, class Alloc>
__device__ __forceinline__ void capture_winners(const PassCtx &X, WinItem *wins, CaptureItem *items, unsigned int threads,
                                                unsigned int n, int app, unsigned long long base, int8_t also_liquid,
                                                Alloc &&alloc, CycleStats &st) {
    const unsigned int warp = threadIdx.x / 32, n_warps = threads / 32;
    for (unsigned int first = 0; first < n; first += kCaptureItems) {
        const unsigned int m = min(n - first, (unsigned int)kCaptureItems), geometry_warps = (m + 31) / 32;
        WinItem *const w = wins + first;
        if (warp < geometry_warps) {
            if (threadIdx.x < m) {
                const WinItem &q = w[threadIdx.x];
                capture_geometry(desc_of(X, q.dom_dir >> 5), q.t, q.h, q.docx, q.docy, q.docz, items[threadIdx.x]);
            }
        }
        else {
            if (warp == n_warps - 1)
                alloc(w, m);
            capture_neighbours<kN>(X, app, base, w, items, warp - geometry_warps, n_warps - geometry_warps, m, also_liquid,
                                   st);
        }
        capture_sync(threads);
        capture_lengths_of(X, w, items, m, threads, app, st);
        if (first + kCaptureItems < n)
            capture_sync(threads);
    }
}

// Record slots for m captures of the block (one warp calls): the block's free slots first, the others
// appended to the list (one atomic on the grid's counter, which completes under the captures' first stage).
__device__ __forceinline__ void take_slots(PoolState *P, BlockShared &B, WinItem *w, unsigned int m, unsigned long long base,
                                           unsigned long long *appended) {
    const unsigned int lane = threadIdx.x & 31;
    const unsigned int free = min(B.n_free, (unsigned int)kFreeSlots), taken = min(B.n_taken, free);
    const unsigned int reused = min(m, free - taken);
    __syncwarp();
    unsigned long long s0 = 0;
    if (lane == 0) {
        B.n_taken += m;
        if (reused < m) {
            s0 = base + atomicAdd(appended, (unsigned long long)(m - reused));
            atomicAdd(&B.n_appended, m - reused);
        }
    }
    s0 = __shfl_sync(0xffffffffu, s0, 0);
    for (unsigned int k = lane; k < m; k += 32) {
        unsigned int slot = kNoRecord;
        if (k < reused)
            slot = B.free_slots[free - taken - 1u - k];
        else if (s0 + (k - reused) < B.X.capacity)
            slot = (unsigned int)(s0 + (k - reused));
        else
            atomicOr(&P->error, kErrListOverflow);
        w[k].slot = slot;
    }
}

// Claim i of the block's list by a whole warp, lane n < 26 direction n: the shortest chain for a block that
// has no more claims than warps. The winner test and every load go out in one round (held: the claimant's
// state was kept by its claim step, so the orientation does not wait for it either), the independent
// divisions and roots of the geometry run on lanes of their own, with capture_geometry's expressions on
// the same operands.
__device__ __forceinline__ void capture_claim(PoolState *P, BlockShared &B, unsigned int i, int app, unsigned long long base,
                                              unsigned long long *appended, int8_t also_liquid, CycleStats &st) {
    constexpr unsigned int kAll = 0xffffffffu;
    const unsigned int lane = threadIdx.x & 31;
    const unsigned long long e = claim_at(B, i);
    const unsigned int dom = claim_domain(e), held = (unsigned int)(e >> kClaimantShift), t = (unsigned int)e;
    const DomainDesc &D = desc_of(B.X, dom);
    const RecordList &L = B.X.list[app];
    const int plane = D.mx * D.my, my = D.my;
    const unsigned int c = (unsigned int)((long long)t - nb_offset((int)((e >> 32) & 31u), plane, my));
    const unsigned long long key = __ldcg(D.claim + t);
    const int cts = __ldg(D.cts_run + t);
    float4 head;
    if (held) {
        head = B.claimants[held - 1];
    }
    else {
        const unsigned int pos = B.claim_pos[i];
        const bool body = pos < L.body_cap;
        const float *doc = body ? L.body[pos].doc : D.doc + 3ull * c;
        head = make_float4(__int_as_float(__ldcg(body ? &L.body[pos].h : D.gid + c)), __ldcg(doc), __ldcg(doc + 1),
                           __ldcg(doc + 2));
    }
    const int h = __float_as_int(head.x);
    int rx, ry, rz;
    cell_coords(D, t, rx, ry, rz);
    const bool nb = (neighbour_mask(D, rx, ry, rz) >> lane) & 1u;
    const unsigned int a = (unsigned int)((long long)t + (nb ? nb_offset((int)lane, plane, my) : 0));
    const int8_t ct = __ldcg(D.ctype + a);
    const unsigned int p = __ldcg(D.pos + a);
    int ori = (abs(h) - 1) % 10000;
    if (ori < 0)
        ori += 10000;
    const float *g = D.guv + 9 * ori;
    const float g0 = g[0], g1 = g[1], g2 = g[2], g3 = g[3], g4 = g[4], g5 = g[5], g6 = g[6], g7 = g[7], g8 = g[8];
    if ((unsigned int)key != c)
        return; // a lower-index claimant captures t
    // the record's slot; the atomic completes under the capture
    unsigned int taken = 0, n_free = 0;
    unsigned long long appended_at = 0;
    if (lane == 0) {
        n_free = min(B.n_free, (unsigned int)kFreeSlots);
        taken = atomicAdd(&B.n_taken, 1u);
        if (taken >= n_free) {
            appended_at = base + atomicAdd(appended, 1ull);
            atomicAdd(&B.n_appended, 1u);
        }
    }
    // liquid mask, the neighbours' masks (see capture_neighbours)
    const unsigned int liq = __reduce_or_sync(kAll, nb && (ct == kLiquid || ct == also_liquid) ? 1u << lane : 0u);
    const bool act = nb && ct == kActive && p < base;
    const unsigned int opp = act ? 1u << nb_opp((int)lane) : 0u;
    if (act && c >= a)
        atomicOr(&L.rec[p].stat, kMaskKeep);
    const unsigned int old = act ? atomicAnd(&L.rec[p].stat, ~opp) : 0u;
    // geometry (capture_geometry)
    const int q3 = lane < 3 ? (int)lane : 0;
    const double cxold = head.y, cyold = head.z, czold = head.w;
    const double xp = (rx + D.xoff) + 0.5, yp = (ry + D.yoff) + 0.5, zp = rz + 0.5;
    const double x0 = xp - cxold, y0 = yp - cyold, z0 = zp - czold;
    const double mag0 = sqrtf((float)(x0 * x0 + y0 * y0 + z0 * z0));
    const float ga = q3 == 0 ? g0 : (q3 == 1 ? g3 : g6), gb = q3 == 0 ? g1 : (q3 == 1 ? g4 : g7),
                gc = q3 == 0 ? g2 : (q3 == 1 ? g5 : g8);
    const double dot = ga * x0 + gb * y0 + gc * z0;
    const unsigned int neg = __ballot_sync(kAll, (dot < -1e-200 && mag0 < 1e30) || dot / mag0 < 0);
    const float s1 = (neg & 1u) ? 1.0f : -1.0f, s2 = (neg & 2u) ? 1.0f : -1.0f, s3 = (neg & 4u) ? 1.0f : -1.0f;
    double Diag1X = g0 * s1, Diag1Y = g1 * s1, Diag1Z = g2 * s1;
    double Diag2X = g3 * s2, Diag2Y = g4 * s2, Diag2Z = g5 * s2;
    double Diag3X = g6 * s3, Diag3Y = g7 * s3, Diag3Z = g8 * s3;
    double U1x = Diag2X - Diag1X, U1y = Diag2Y - Diag1Y, U1z = Diag2Z - Diag1Z;
    double U2x = Diag3X - Diag1X, U2y = Diag3Y - Diag1Y, U2z = Diag3Z - Diag1Z;
    double UUx = U1y * U2z - U1z * U2y;
    double UUy = U1z * U2x - U1x * U2z;
    double UUz = U1x * U2y - U1y * U2x;
    double NDem = sqrtf((float)(UUx * UUx + UUy * UUy + UUz * UUz));
    const double nq = (q3 == 0 ? UUx : (q3 == 1 ? UUy : UUz)) / NDem;
    double n0 = __shfl_sync(kAll, nq, 0), n1 = __shfl_sync(kAll, nq, 1), n2 = __shfl_sync(kAll, nq, 2);
    double ParaT = (n0 * x0 + n1 * y0 + n2 * z0) / (n0 * Diag1X + n1 * Diag1Y + n2 * Diag1Z);
    const double TX0 = cxold + ParaT * Diag1X, TY0 = cyold + ParaT * Diag1Y, TZ0 = czold + ParaT * Diag1Z;
    const double TX1 = cxold + ParaT * Diag2X, TY1 = cyold + ParaT * Diag2Y, TZ1 = czold + ParaT * Diag2Z;
    const double TX2 = cxold + ParaT * Diag3X, TY2 = cyold + ParaT * Diag3Y, TZ2 = czold + ParaT * Diag3Z;
    const double tqx = q3 == 0 ? TX0 : (q3 == 1 ? TX1 : TX2), tqy = q3 == 0 ? TY0 : (q3 == 1 ? TY1 : TY2),
                 tqz = q3 == 0 ? TZ0 : (q3 == 1 ? TZ1 : TZ2);
    const float distq =
        sqrtf((float)(((tqx - xp) * (tqx - xp)) + ((tqy - yp) * (tqy - yp)) + ((tqz - zp) * (tqz - zp))));
    const double Dist0 = __shfl_sync(kAll, distq, 0), Dist1 = __shfl_sync(kAll, distq, 1), Dist2 = __shfl_sync(kAll, distq, 2);
    int x = (Dist0 < Dist1);
    int y = (Dist1 < Dist2);
    int z = (Dist2 < Dist0);
    int idx = 2 * (z - y) * z + (y - x) * y;
    const bool p0 = idx == 0, p1 = idx == 1;
    double mindist = p0 ? Dist0 : (p1 ? Dist1 : Dist2);
    double xc = p0 ? TX0 : (p1 ? TX1 : TX2), yc = p0 ? TY0 : (p1 ? TY1 : TY2), zc = p0 ? TZ0 : (p1 ? TZ1 : TZ2);
    double x1 = p0 ? TX1 : (p1 ? TX2 : TX0), y1 = p0 ? TY1 : (p1 ? TY2 : TY0), z1 = p0 ? TZ1 : (p1 ? TZ2 : TZ0);
    double x2 = p0 ? TX2 : (p1 ? TX0 : TX1), y2 = p0 ? TY2 : (p1 ? TY0 : TY1), z2 = p0 ? TZ2 : (p1 ? TZ0 : TZ1);
    // D1..D4 on lanes 0..3: D1 = |p - v2|, D2 = |c - v2|, D3 = |p - v1|, D4 = |c - v1|
    const double ax = (lane & 1) ? xc : xp, ay = (lane & 1) ? yc : yp, az = (lane & 1) ? zc : zp;
    const double bx = (lane & 2) ? x1 : x2, by = (lane & 2) ? y1 : y2, bz = (lane & 2) ? z1 : z2;
    const float dq = sqrtf((float)(((ax - bx) * (ax - bx)) + ((ay - by) * (ay - by)) + ((az - bz) * (az - bz))));
    double D1 = __shfl_sync(kAll, dq, 0), D2 = __shfl_sync(kAll, dq, 1), D3 = __shfl_sync(kAll, dq, 2),
           D4 = __shfl_sync(kAll, dq, 3);
    double I1 = 0, I2 = D2, J1 = 0, J2 = D4;
    if (mindist != 0) {
        // I1 on lane 0, J1 on lane 1
        const bool j = lane & 1;
        const double ex = j ? x1 : x2, ey = j ? y1 : y2, ez = j ? z1 : z2;
        const double Da = j ? D3 : D1, Db = j ? D4 : D2;
        const double ij = Da * ((xp - ex) * (xc - ex) + (yp - ey) * (yc - ey) + (zp - ez) * (zc - ez)) / (Da * Db);
        I1 = __shfl_sync(kAll, ij, 0);
        I2 = D2 - I1;
        J1 = __shfl_sync(kAll, ij, 1);
        J2 = D4 - J1;
    }
    const double sqrt3 = sqrt(3.0);
    double L12 = 0.5 * (dmin(I1, sqrt3) + dmin(I2, sqrt3));
    double L13 = 0.5 * (dmin(J1, sqrt3) + dmin(J2, sqrt3));
    double NewODiagL = sqrt(2.0) * dmax(L12, L13);
    double cd0 = xc - cxold, cd1 = yc - cyold, cd2 = zc - czold;
    double nd = sqrt(cd0 * cd0 + cd1 * cd1 + cd2 * cd2);
    const double uvq = (q3 == 0 ? cd0 : (q3 == 1 ? cd1 : cd2)) / nd;
    CaptureItem o;
    o.cx = xc - NewODiagL * __shfl_sync(kAll, uvq, 0);
    o.cy = yc - NewODiagL * __shfl_sync(kAll, uvq, 1);
    o.cz = zc - NewODiagL * __shfl_sync(kAll, uvq, 2);
    o.dl = (float)NewODiagL;
    o.liq = liq;
    taken = __shfl_sync(kAll, taken, 0);
    n_free = __shfl_sync(kAll, n_free, 0);
    appended_at = __shfl_sync(kAll, appended_at, 0);
    unsigned int slot = kNoRecord;
    if (taken < n_free)
        slot = B.free_slots[n_free - 1u - taken];
    else if (appended_at < B.X.capacity)
        slot = (unsigned int)appended_at;
    else
        atomicOr(&P->error, kErrListOverflow);
    capture_lengths(D, L, WinItem{t, c, dom << 5, h, cts, head.y, head.z, head.w, slot}, o, 32, (int)lane, kAll, st);
    if (act && !(old & (kMaskFresh | kMaskDead | kMaskKeep)) && (old & kDirBits) == opp && (old & kMaskGrown)) {
        st.rechecks++;
        D.ctype[a] = kSolid;
        atomicOr(&L.rec[p].stat, kMaskDead);
    }
}

// Capture pass of the persistent kernel, by the first `threads` threads of the block (its other warps
// start the domains' next cycle). Each block keeps the winners among its own claims (one per
// thread) and captures them.
template <int kFamily>
__device__ __forceinline__ void capture_block(PoolState *P, BlockShared &B, unsigned int threads, int app,
                                              unsigned long long base, unsigned long long *appended, int8_t also_liquid,
                                              CycleStats &st) {
    const unsigned int n = claim_count(B), lane = threadIdx.x & 31;
    if (kFamily == kShortList && n * 32 <= threads) {
        if (threadIdx.x / 32 < n)
            capture_claim(P, B, threadIdx.x / 32, app, base, appended, also_liquid, st);
        return;
    }
    for (unsigned int r0 = 0; r0 < n; r0 += threads) {
        const unsigned int i = r0 + threadIdx.x;
        WinItem w;
        const bool win = i < n && load_win(B.X, B.X.list[app], claim_at(B, i),
                                           i < (unsigned int)kBlockClaims ? B.claim_pos[i] : kNoRecord, w);
        const unsigned int winners = __ballot_sync(0xffffffffu, win);
        unsigned int first = 0;
        if (lane == 0 && winners)
            first = atomicAdd(&B.n_wins, __popc(winners));
        first = __shfl_sync(0xffffffffu, first, 0);
        if (win)
            B.wins[first + __popc(winners & ((1u << lane) - 1u))] = w;
        capture_sync(threads);
        capture_winners<kFamily == kLongList ? 6 : 2>(
            B.X, B.wins, B.captures, threads, B.n_wins, app, base, also_liquid,
            [&](WinItem *q, unsigned int m) { take_slots(P, B, q, m, base, appended); }, st);
        if (r0 + threads < n) {
            capture_sync(threads);
            if (threadIdx.x == 0)
                B.n_wins = 0;
            capture_sync(threads);
        }
    }
}

// Capture pass over the sharded claim list (the separate kernels): claim j of the cycle gets record slot
// base + j (a tombstone unless it won), and the count grows by T when the cycle finishes.
struct CaptureShared {
    WinItem wins[kBlock];
    CaptureItem captures[kCaptureItems];
    unsigned int n_wins;
};
__device__ void capture_pass(PoolState *P, const PassCtx &X, CaptureShared &C, CycleStats &st) {
    __shared__ unsigned long long s_pre[kShards + 1];
    const unsigned long long cap = P->shard_cap;
    shard_prefix(P->tcnt_s, cap, s_pre);
    const int app = P->pending; // list of the next cycle
    const unsigned long long T = s_pre[kShards];
    const unsigned long long base = P->cnt[app];
    if (base + T > P->capacity) {
        if (threadIdx.x == 0 && blockIdx.x == 0)
            atomicOr(&P->error, kErrListOverflow);
        return;
    }
    unsigned int losers = 0;
    const unsigned int lane = threadIdx.x & 31;
    // consecutive claims on different blocks (spread over all SMs)
    for (unsigned long long j0 = 0; j0 < T; j0 += (unsigned long long)gridDim.x * kBlock) {
        const unsigned long long j = j0 + (unsigned long long)threadIdx.x * gridDim.x + blockIdx.x;
        if (threadIdx.x == 0)
            C.n_wins = 0;
        __syncthreads();
        WinItem w;
        bool win = false;
        if (j < T) {
            win = load_win(X, X.list[app], __ldcg(P->tgt + shard_entry(s_pre, cap, j)), kNoRecord, w);
            w.slot = (unsigned int)(base + j);
            if (!win) {
                // a lower-index claimant captures t; this claim's slot stays a dropped record
                X.list[app].rec[base + j].stat = kMaskTomb;
                losers++;
            }
        }
        const unsigned int winners = __ballot_sync(0xffffffffu, win);
        unsigned int first = 0;
        if (lane == 0 && winners)
            first = atomicAdd(&C.n_wins, __popc(winners));
        first = __shfl_sync(0xffffffffu, first, 0);
        if (win) {
            C.wins[first + __popc(winners & ((1u << lane) - 1u))] = w;
            atomicAdd((unsigned long long *)&X.desc[w.dom_dir >> 5].liquid_shard[(blockIdx.x + j) & (kLiquidShards - 1)],
                      (unsigned long long)(-1ll));
        }
        __syncthreads();
        capture_winners<2>(X, C.wins, C.captures, kBlock, C.n_wins, app, base, (int8_t)kLiquid, [](WinItem *, unsigned int) {}, st);
        __syncthreads();
    }
    add_tombs(P, losers);
}

// End of a cycle: the record slots of this cycle's claims join the list.
__device__ void finish_capture(PoolState *P) {
    if (threadIdx.x < 32) {
        unsigned long long T = shard_count(P->tcnt_s[threadIdx.x], P->shard_cap);
#pragma unroll
        for (int o = 16; o; o >>= 1)
            T += __shfl_down_sync(0xffffffffu, T, o);
        if (threadIdx.x == 0) {
            const int app = P->pending;
            if (P->cnt[app] + T <= P->capacity)
                P->cnt[app] += T;
        }
    }
    __syncthreads();
}

template <int kBatch> __global__ void __launch_bounds__(kBlock) k_grow(PoolState *P) {
    __shared__ PassCtx X;
    load_ctx(P, X, 0);
    __syncthreads();
    CycleStats st;
    unsigned int tombs = 0;
    const int cur = P->cur;
    grow_pass<kBatch, false, kLongList, false>(P, X, nullptr, load_dyn(X.desc[0]), cur, P->cnt[cur], P->compact != 0, false, st, tombs);
    add_tombs(P, tombs);
    flush_stats(P, st);
}

__global__ void __launch_bounds__(kBlock) k_claim(PoolState *P) {
    __shared__ PassCtx X;
    load_ctx(P, X, 0);
    __syncthreads();
    CycleStats st;
    unsigned int tombs = 0;
    claim_pass<false>(P, X, nullptr, P->pending, st, tombs);
    if (!P->compact) // a compacted list starts without dropped records
        add_tombs(P, tombs);
    flush_stats(P, st);
}

// Capture pass as its own kernel; the last block to finish closes the cycle and, with kBegin,
// starts the next one.
template <bool kBegin> __global__ void __launch_bounds__(kBlock) k_capture_pass(PoolState *P) {
    __shared__ PassCtx X;
    load_ctx(P, X, 0);
    __syncthreads();
    __shared__ CaptureShared C;
    CycleStats st;
    capture_pass(P, X, C, st);
    flush_stats(P, st);
    __shared__ int s_last;
    __threadfence(); // this block's writes are visible device-wide before it is counted
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int prev = atomicAdd(&P->blocks_done, 1u);
        s_last = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        if (threadIdx.x == 0)
            P->blocks_done = 0;
        if (kBegin)
            begin_cycle(P, true, P->desc, P->n_domains, AliveSet{-1, {}}, false);
        else
            finish_capture(P);
    }
}

// ---------------------------------------------------------------------------------------------
// Grid-wide meeting point of the persistent kernel (all blocks co-resident: cooperative launch).
// Meeting k uses word k % 3: every block adds 2^56 (one arrival) and its share of what the grid
// needs to know (release), and polls the word (acquire) until every block has arrived; the low 56
// bits are then the sums over the grid, so the counts travel with the arrivals and no block works
// alone while the others wait. With the last block running the cycle's start before it released the
// others through a second word, an idle cycle took 9.7 us on 148 blocks. The word of meeting k + 2
// was last polled for meeting k - 1, which every block has passed once meeting k is complete: block
// 0 clears it then, before its own next arrival.
// Every wait is bounded: after kMeetTimeoutNs (or kMeetSpinCap polls) the block sets kErrBarrier and
// the kernel ends.
constexpr unsigned long long kMeetTimeoutNs = 1000000000ull;
constexpr unsigned int kMeetSpinCap = 1u << 26;
constexpr int kMeetShift = 56;
constexpr int kMeetMaxGrid = 255; // arrivals in the top byte
constexpr unsigned long long kMeetSums = (1ull << kMeetShift) - 1;

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Meeting number k (counted by the caller). share() gives this block's sums, in thread 0 after the
// block's other threads have arrived. total: the grid's sums. With tl set, meeting point `tag`
// records its first and last arrival and when block 0 left it. False: gave up waiting.
template <class Share>
__device__ bool grid_meet(PoolState *P, unsigned int &k, unsigned long long *tl, int tag, Share &&share,
                          unsigned long long &total) {
    __shared__ unsigned long long s_word;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long *word = &P->meet.word[k % 3].v;
        const unsigned long long add = (1ull << kMeetShift) + share();
        if (tl) {
            const unsigned long long now = global_ns();
            atomicMin(tl + 3 * tag + 0, now);
            atomicMax(tl + 3 * tag + 1, now);
        }
        red_release_u64(word, add);
        unsigned long long v = ld_acquire_u64(word);
        if ((v >> kMeetShift) != gridDim.x) {
            const unsigned long long t0 = global_ns();
            unsigned int it = 0;
            while (((v = ld_acquire_u64(word)) >> kMeetShift) != gridDim.x) {
                ++it;
                if (it >= kMeetSpinCap || ((it & 255u) == 0 && global_ns() - t0 > kMeetTimeoutNs)) {
                    atomicOr(&P->error, kErrBarrier);
                    v = 0;
                    break;
                }
            }
        }
        if (blockIdx.x == 0 && v) {
            P->meet.word[(k + 2) % 3].v = 0;
            if (tl)
                tl[3 * tag + 2] = global_ns();
        }
        s_word = v;
    }
    __syncthreads();
    k++;
    total = s_word & kMeetSums;
    return s_word != 0;
}

// ---------------------------------------------------------------------------------------------
// Start of domain d's cycle c + 1 (launch-local index) by one warp, while the rest of the grid runs
// the capture pass of cycle c: the device-side termination check, the cycle advance and the
// nucleation of the sites whose time has come, as start_domain does at the start of a launch. What
// makes that possible:
//   - the liquid count after cycle c is known before the captures (make_claims counts the cells
//     claimed; `claimed` are the hot domain's);
//   - a site that fires was marked (mark_code) during the capture pass before this one, when its
//     type was liquid. A claim made since has overwritten the mark, so the site fires iff the mark
//     is still there, and the captures, which see the mark or the site already active, leave it out
//     of a captured cell's liquid mask either way;
//   - a firing site flags its active neighbours' records (kMaskNuc) instead of clearing their mask
//     bits, which still count in cycle c; the growth pass of cycle c + 1 clears them.
// Sites due in cycle c + 2 are marked at the end. cycle0: the domain's cycle c when the caller has
// counted cycles whose start was not run (k_cycles), else -1.
__device__ __noinline__ void start_next(PoolState *P, BlockShared &B, unsigned int d, int cycle0, unsigned long long claimed,
                                        int app, unsigned long long base, unsigned long long *appended, int c,
                                        int n_cycles) {
    DomainDesc &D = B.X.desc[d];
    const unsigned int lane = threadIdx.x & 31;
    DomainStart s = load_start(D);
    if (s.ctype == nullptr || s.done)
        return;
    if (cycle0 >= 0)
        s.cycle0 = cycle0;
    const long long liquid0 = __ldcg(&D.liquid) - (long long)claimed;
    if (c + 1 >= n_cycles) {
        if (lane == 0)
            D.liquid = liquid0;
        return;
    }
    // rest of the descriptor
    const NucleationView V = nucleation_view(D);
    const int mark0 = __ldcg(&D.nuc_mark), nn0 = __ldcg(&D.nn), layer_no = D.layer_no;
    const long long active_size = D.active_size;
    const unsigned int epoch0 = __ldcg(&D.epoch);
    const bool check = s.check_mode && s.cycle0 > 0 && s.cycle0 % 1000 == 0;
    const bool probe = s.check_mode && (s.cycle0 & 63) == 0;
    const int dry_since = probe ? __ldcg(&D.dry_since) : 0;
    const int cts_max = probe ? D.cts_max : INT_MAX;
    long long liquid = 1;
    if (check || probe) {
        liquid = lane < kLiquidShards ? __ldcg(&D.liquid_shard[lane]) : 0;
#pragma unroll
        for (int o = 16; o; o >>= 1)
            liquid += __shfl_xor_sync(0xffffffffu, liquid, o);
        liquid += liquid0;
    }
    if (check && liquid == 0) {
        // src/CAupdate.cpp:782-783: no superheated or undercooled liquid left
        if (lane == 0) {
            D.liquid = liquid0;
            D.done = 1;
        }
        return;
    }
    const int cycle = s.cycle0 + 1;
    const RecordList &L = B.X.list[app];
    int fired_total = 0;
    for (int q = s.cursor0; q < mark0; q += 32) {
        const int idx = q + (int)lane;
        const int l = idx < mark0 ? __ldg(s.nuc_loc + idx) : -1;
        bool fire = false;
        int h = 0, cts = 0;
        if (l >= 0 && l < active_size) {
            fire = __ldcg(s.ctype + l) == mark_code(c + 1);
            h = __ldcg(V.gid + l);
            cts = V.cts_run[l];
        }
        const unsigned int firing = __ballot_sync(0xffffffffu, fire);
        if (!firing)
            continue;
        const unsigned int n_fire = __popc(firing);
        unsigned long long slot0 = 0;
        if (lane == 0) {
            slot0 = base + atomicAdd(appended, (unsigned long long)n_fire);
            atomicAdd(&B.n_appended, n_fire);
            if (slot0 + n_fire > B.X.capacity) {
                atomicOr(&P->error, kErrListOverflow);
                for (; slot0 < B.X.capacity; slot0++) // what is left of the list holds no record
                    L.rec[slot0].stat = kMaskTomb;
                slot0 = ULLONG_MAX;
            }
        }
        slot0 = __shfl_sync(0xffffffffu, slot0, 0);
        for (unsigned int todo = firing; todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            const unsigned int rank = __popc(firing & ((1u << src) - 1u));
            nucleate_site(V, s.ctype, L, d,
                          (unsigned int)__shfl_sync(0xffffffffu, l, src), __shfl_sync(0xffffffffu, h, src),
                          __shfl_sync(0xffffffffu, cts, src), slot0 == ULLONG_MAX ? ULLONG_MAX : slot0 + rank,
                          [&](unsigned int nb_pos, int) {
                              if (nb_pos < base)
                                  atomicOr(&L.rec[nb_pos].stat, kMaskNuc);
                          });
        }
        fired_total += (int)n_fire;
    }
    bool ended = false;
    if (probe && s.cycle0 - 2 >= cts_max && liquid == 0 && fired_total == 0) {
        // see start_domain
        if (dry_since != 0)
            ended = true;
        else if (lane == 0)
            D.dry_since = s.cycle0;
    }
    const int mark = (c + 2 < n_cycles && !ended) ? mark_sites(D, s, mark0, cycle + 1, mark_code(c + 2), layer_no, active_size)
                                                   : mark0;
    if (lane != 0)
        return;
    D.liquid = liquid0 - fired_total;
    if (ended) {
        D.cycle = (s.cycle0 + 999) / 1000 * 1000;
        D.done = 1;
        return;
    }
    D.cycle = cycle;
    D.epoch = epoch0 + 1;
    D.next_start = next_start_of(s, cycle, mark0, mark);
    D.nuc_cursor = mark0;
    D.nuc_mark = mark;
    D.nn = nn0 + fired_total;
    if (fired_total)
        atomicAdd(&P->stat[blockIdx.x & (kStatShards - 1)][kStatNucleated], (unsigned long long)fired_total);
}

constexpr int kTellLeast = 16;              // dropped records for which a block asks for a meeting (k_cycles)
constexpr unsigned int kTellFlag = 1u << 8; // in BlockShared::busy: it does

// n_cycles complete CA cycles (start, grow/claim, capture) in one cooperative launch.
//
// With one running domain a cycle is cut short where nothing is left of it. A cycle without claims
// whose successor's start is not needed (next_start_of) has no capture pass and one meeting. When
// besides no record was grown or dropped, the following cycles do nothing until the first of them that
// is past some record's CritTimeStep or needs its start: they only advance the cycle number. Of the
// cycles of a 64^3 solve 32 % make no claim (19 % grow nothing), of 3 x 3 spot melts 57 % (57 %), of
// small three-layer ones 86 % (74 %); an idle cycle took 4.8 us, one with growth and no claim about 7.
template <int kFamily, int kBatch, bool kMany>
__global__ void __launch_bounds__(kBlock, 1) k_cycles(PoolState *P, int n_cycles, AliveSet alive) {
    __shared__ BlockShared B;
    __shared__ ShortView views[kMany ? kViews : 1];
    CycleStats st;
    // the start of the launch's first cycle: one block for a few domains, a warp per domain across
    // the grid for many; later cycles are started under the capture pass (start_next)
    DomainDesc *const desc = P->desc;
    const int n_domains = P->n_domains;
    const bool spread = kMany || alive.n < 0;
    const int n_start = spread ? n_domains : alive.n;
    unsigned long long *const tl = P->timeline;
    unsigned int meet = 0;
    unsigned long long total = 0;
    const auto no_share = [] { return 0ull; };
    if (threadIdx.x == 0)
    {
        B.n_items = B.n_claims = B.n_wins = B.n_first = B.n_appended = B.n_free = B.n_taken = B.busy = 0;
        B.tombs = 0;
        B.min_cts = INT_MAX;
    }
    if (blockIdx.x == 0) {
        if (threadIdx.x < 3)
            *reinterpret_cast<int *>(&P->meet.min_cts[threadIdx.x].v) = INT_MAX;
        if (spread)
            begin_lists(P, false);
        else
            begin_cycle(P, false, desc, n_domains, alive, n_cycles > 1);
    }
    bool ok = grid_meet(P, meet, tl, 0, no_share, total);
    if (ok && spread) {
        begin_domains(P, desc, n_domains, (threadIdx.x >> 5) * gridDim.x + blockIdx.x, gridDim.x * (kBlock / 32),
                      n_cycles > 1);
        ok = grid_meet(P, meet, nullptr, 0, no_share, total);
    }
    load_ctx(P, B.X, alive.n > 0 ? (unsigned int)alive.idx[0] : 0u);
    // the list's state, the same in every block
    int cur = __ldcg(&P->cur);
    unsigned long long n = __ldcg(&P->cnt[cur]), tombs = __ldcg(&P->tombs);
    // the warps that start domains: the last of the blocks 0 .. n_start - 1
    const int start_warps = min(8, (n_start + (int)gridDim.x - 1) / (int)gridDim.x);
    const unsigned int threads = (int)blockIdx.x < n_start ? (unsigned int)(kBlock - 32 * start_warps) : (unsigned int)kBlock;
    __syncthreads();
    const bool solo = alive.n == 1;
    DomainDyn dyn{};
    bool started = true;                 // the last cycle's capture pass, with the start of this one, was run
    unsigned int passes = 0, starts = 0; // growth passes and capture passes so far
    for (int c = 0; ok && c < n_cycles; c++, passes++) {
        if (passes % kStatCycles == kStatCycles - 1) {
            flush_stats(P, st);
            st = CycleStats();
        }
        if (started)
            dyn = load_dyn(B.X.desc[B.X.hot]);
        else if (!dyn.done)
            dyn.cycle++;
        // compact when dropped records exceed a quarter of the list, as lists_start
        const bool compact = tombs * 4 > n;
        const int app = compact ? cur ^ 1 : cur; // list of the next cycle
        if (compact && threadIdx.x == 0) {
            // positions in the old list; counted again, for the new one, after grow_pass's block barrier
            B.n_free = 0;
            B.tombs = 0;
        }
        // growth with each block's claims right after its own growth; the global claim pass only
        // when some block's queue overflowed this cycle (the same answer for every block)
        unsigned int dropped = 0;
        if (kMany) {
            for (unsigned int d = threadIdx.x; d < min((unsigned int)n_domains, kViews); d += kBlock)
                views[d] = short_view(B.X.desc[d], B.X.extras);
            __syncthreads();
        }
        grow_pass<kBatch, true, kFamily, kMany>(P, B.X, &B, dyn, cur, n, compact, passes == 0, st, dropped, views);
        dropped = __reduce_add_sync(0xffffffffu, dropped);
        // A block tells its dropped records at the meeting after the captures, which a lone domain's cycle without
        // claims leaves out; it asks for that meeting when the list would be due for compaction if every block
        // had dropped as many as itself: were it due, a block with the mean or more would ask. Fewer than
        // kTellLeast wait for the next meeting or the launch's end (all blocks' together are at most one more
        // group of 32 for a few of the warps). The warp that adds last sees the sum (asked by thread 0 on its way
        // to the meeting instead: three-layer spots 0.2 % slower, melt tracks 0.3 %). (In a cycle that compacts the difference wraps
        // to a large one.)
        if ((threadIdx.x & 31) == 0 && dropped) {
            const unsigned int untold = (unsigned int)(atomicAdd(&B.tombs, (int)dropped) + (int)dropped);
            if ((int)untold >= kTellLeast && untold * gridDim.x > (unsigned int)(n >> 2) - (unsigned int)tombs)
                atomicOr(&B.busy, kTellFlag); // every store of 1 lies before grow_pass's block barrier
        }
        // sums: first claims of the hot domain (32 bits, as cell indices), blocks whose queue overflowed, blocks that
        // are busy, blocks that would tell
        constexpr int kOverflowShift = 32, kBusyShift = 40;
        static_assert(kTellFlag == 1u << 8, "the byte above the busy blocks");
        int *const grid_min = reinterpret_cast<int *>(&P->meet.min_cts[passes % 3].v);
        const auto claim_share = [&] {
            const unsigned long long v = B.n_first;
            B.n_first = 0;
            return v;
        };
        ok = grid_meet(
            P, meet, tl, 3 * c + 1,
            [&] {
                const unsigned long long v = claim_share() + (B.n_items > (unsigned int)kBlockQueue ? 1ull << kOverflowShift : 0ull) +
                                             ((unsigned long long)B.busy << kBusyShift);
                if (!B.busy && B.min_cts != INT_MAX)
                    atomicMin(grid_min, B.min_cts);
                B.n_items = B.busy = 0;
                B.min_cts = INT_MAX;
                return v;
            },
            total);
        if (!ok)
            break;
        unsigned long long claimed = total & 0xffffffffull;
        const bool asked = (total & ~(0xffull << kBusyShift)) != 0; // claims, an overflow, drops to tell
        const bool overflow = ((total >> kOverflowShift) & 0xffu) != 0, busy = ((total >> kBusyShift) & 0xffu) != 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) // read after the previous cycle's meeting, used two cycles on
            *reinterpret_cast<int *>(&P->meet.min_cts[(passes + 2) % 3].v) = INT_MAX;
        if (overflow) {
            dropped = 0;
            claim_pass<true>(P, B.X, &B, app, st, dropped);
            dropped = __reduce_add_sync(0xffffffffu, dropped);
            if ((threadIdx.x & 31) == 0 && dropped)
                atomicAdd(&B.tombs, (int)dropped);
            ok = grid_meet(P, meet, tl, 3 * c + 2, claim_share, total);
            if (!ok)
                break;
            claimed += total;
        }
        const unsigned long long base = compact ? __ldcg(&P->cnt[app]) : n;
        if (blockIdx.x == 0 && threadIdx.x < 32) {
            // counters that the grid has done with, or needs from the next meeting on
            if (threadIdx.x == 0 && compact)
                P->cnt[cur] = 0;
            if (overflow)
                P->qcnt_s[threadIdx.x].v = 0;
        }
        started = !solo || asked || (!dyn.done && c + 1 < n_cycles && dyn.cycle + 1 >= dyn.next_start);
        if (!started) {
            n = base;
            if (compact)
                tombs = 0;
            cur = app;
            if (!busy) {
                // cycles dyn.cycle + 1 .. + skip do nothing, nor do the starts up to the one after them
                long long skip = n_cycles - 1 - c;
                if (!dyn.done)
                    skip = min(skip, min((long long)__ldcg(grid_min) - dyn.cycle, (long long)dyn.next_start - 2 - dyn.cycle));
                if (skip > 0) {
                    c += (int)skip;
                    if (!dyn.done)
                        dyn.cycle += (int)skip;
                }
            }
            continue;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0)
            P->meet.appended[(starts + 1) % 3].v = 0;
        unsigned long long *const appended = &P->meet.appended[starts % 3].v;
        starts++;
        if (threadIdx.x >= threads) {
            const unsigned int w = (threadIdx.x - threads) / 32;
            for (int i = (int)(w * gridDim.x + blockIdx.x); i < n_start; i += start_warps * (int)gridDim.x) {
                const unsigned int d = spread ? (unsigned int)i : (unsigned int)alive.idx[i];
                start_next(P, B, d, solo ? dyn.cycle : -1, d == B.X.hot ? claimed : 0ull, app, base, appended, c, n_cycles);
            }
        }
        else {
            capture_block<kFamily>(P, B, threads, app, base, appended, mark_code(c + 2), st);
        }
        // sums: records appended (32 bits, as list positions), change of the number of dropped records
        // (24 bits: 2^15 more from each block, which keeps what exceeds its share for the next time)
        constexpr int kTombShift = 32, kTombBias = 1 << 15;
        ok = grid_meet(
            P, meet, tl, 3 * c + 3,
            [&] {
                const unsigned int free = min(B.n_free, (unsigned int)kFreeSlots), reused = min(B.n_taken, free);
                B.n_free = free - reused;
                B.tombs -= (int)reused;
                const int delta = min(max(B.tombs, 1 - kTombBias), kTombBias - 1);
                const unsigned long long v = B.n_appended + ((unsigned long long)(delta + kTombBias) << kTombShift);
                B.tombs -= delta;
                B.n_claims = B.n_wins = B.n_taken = B.n_appended = 0;
                return v;
            },
            total);
        n = base + (total & 0xffffffffull);
        if (n > B.X.capacity)
            n = B.X.capacity; // overflowed: flagged
        const long long change = (long long)(total >> kTombShift) - (long long)gridDim.x * kTombBias;
        tombs = (unsigned long long)max((long long)(compact ? 0 : tombs) + change, 0ll);
        cur = app;
    }
    // what the block has not told, for the next launch's start (lists_start)
    if (ok && threadIdx.x == 0 && B.tombs)
        atomicAdd(&P->tomb_s[blockIdx.x % kShards].v, (unsigned long long)(long long)B.tombs);
    if (ok && blockIdx.x == 0 && threadIdx.x == 0) {
        P->cur = P->pending = cur;
        P->cnt[cur] = n;
        P->cnt[cur ^ 1] = 0;
        P->tombs = tombs;
        P->compact = 0;
        if (solo && !dyn.done)
            B.X.desc[B.X.hot].cycle = dyn.cycle;
    }
    flush_stats(P, st);
}

// The bounded wait of the meeting point taken to its limit: a cooperative launch of two blocks in
// which block 0 leaves without arriving, so block 1's wait can only end by its time limit (it sets
// kErrBarrier and returns, and the context stays usable).
__global__ void __launch_bounds__(kBlock) k_meet_probe(PoolState *P) {
    if (blockIdx.x == 0)
        return;
    unsigned int k = 0;
    unsigned long long total;
    grid_meet(P, k, nullptr, 0, [] { return 0ull; }, total);
}

// Compiled launch shapes.
struct StepKernels {
    const void *cycles, *cycles_many; // up to kSerialDomains running, more
    void (*grow)(PoolState *);
    void (*capture_begin)(PoolState *);
    void (*capture_end)(PoolState *);
};
template <int kF, int kB> StepKernels step_kernels() {
    return {(const void *)k_cycles<kF, kB, false>, (const void *)k_cycles<kF, kB, true>, k_grow<kB>,
            k_capture_pass<true>, k_capture_pass<false>};
}
static_assert(kStepVariants == 4, "the shapes below");
const StepKernels kStepKernel[kStepVariants] = {
    step_kernels<kLongList, kBatchChoices[0]>(), step_kernels<kLongList, kBatchChoices[1]>(),
    step_kernels<kMidList, kBatchChoices[0]>(), step_kernels<kShortList, kBatchChoices[1]>()};

// ---------------------------------------------------------------------------------------------
// Census of src/CAupdate.cpp:738-808 for one domain and its current layer; the smallest
// CritTimeStep is taken over liquid cells of the layer inside the active window. Each thread reads
// 16 cells per step with 16-byte loads (the field arrays start on 256-byte boundaries); the tail of
// fewer than 16 cells is read cell by cell.
struct CensusCount {
    unsigned int superheated = 0, undercooled = 0, active = 0, solid = 0, remaining = 0;
    unsigned long long mn = ULLONG_MAX;
    __device__ __forceinline__ void cell(long long c, int t, int ly, int cts, int cycle, int layer, long long w_lo,
                                         long long w_hi) {
        if (ly == layer) {
            if (t == kLiquid) {
                if (cts > cycle)
                    superheated++;
                else
                    undercooled++;
                const unsigned long long u = (unsigned long long)(long long)cts;
                if (c >= w_lo && c < w_hi && u < mn)
                    mn = u;
            }
            else if (t == kActive)
                active++;
            else if (t == kSolid)
                solid++;
        }
        else if (t == kLiquid) {
            remaining++;
        }
    }
};

__global__ void __launch_bounds__(256) k_census(const DomainDesc *Dp, Census *out) {
    const DomainDesc &D = *Dp;
    const int8_t *ctype = D.ctype, *lay = D.layer;
    const int32_t *ctsp = D.cts;
    const long long N = D.domain_size;
    const int cycle = D.cycle, layer = D.layer_no;
    const long long plane = (long long)D.mx * D.my;
    const long long w_lo = plane * D.z_lo, w_hi = plane * D.z_end;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    CensusCount k;
    const long long n16 = N / 16;
    for (long long q = tid; q < n16; q += stride) {
        const int4 t16 = __ldcs(reinterpret_cast<const int4 *>(ctype) + q);
        const int4 l16 = __ldcs(reinterpret_cast<const int4 *>(lay) + q);
        int4 c4[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
            c4[u] = __ldcs(reinterpret_cast<const int4 *>(ctsp) + 4 * q + u);
        const int tw[4] = {t16.x, t16.y, t16.z, t16.w}, lw[4] = {l16.x, l16.y, l16.z, l16.w};
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int cv[4] = {c4[u].x, c4[u].y, c4[u].z, c4[u].w};
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const int t = (int)(int8_t)(tw[u] >> (8 * b)), ly = (int)(int8_t)(lw[u] >> (8 * b));
                k.cell(16 * q + 4 * u + b, t, ly, cv[b], cycle, layer, w_lo, w_hi);
            }
        }
    }
    for (long long c = 16 * n16 + tid; c < N; c += stride)
        k.cell(c, ctype[c], lay[c], ctsp[c], cycle, layer, w_lo, w_hi);
    const unsigned int counts[5] = {k.superheated, k.undercooled, k.active, k.solid, k.remaining};
#pragma unroll
    for (int q = 0; q < 5; q++) {
        unsigned long long v = counts[q];
        for (int o = 16; o; o >>= 1)
            v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0 && v)
            atomicAdd((unsigned long long *)out + q, v);
    }
    unsigned long long mn = k.mn;
    for (int o = 16; o; o >>= 1) {
        unsigned long long v = __shfl_down_sync(0xffffffffu, mn, o);
        mn = v < mn ? v : mn;
    }
    if ((threadIdx.x & 31) == 0)
        atomicMin(&out->next_cts, mn);
}

// Voronoi baseplate (src/CAinitialize.cpp:1646-1677): nearest seed by float distance, the first
// seed in draw order wins ties.
__global__ void k_voronoi(DomainDesc *Dp, const int32_t *seeds, int nseeds, float init_min) {
    extern __shared__ int s_seed[];
    const DomainDesc &D = *Dp;
    long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool mine = c < D.domain_size && D.gid[c] == kVoronoiPending;
    int gx = 0, gy = 0, k = 0;
    if (mine) {
        int plane = D.mx * D.my;
        k = (int)(c / plane);
        int rem = (int)(c - (long long)k * plane);
        gx = rem / D.my + D.xoff;
        gy = rem % D.my + D.yoff;
    }
    float best = init_min;
    int best_i = -1;
    for (int base = 0; base < nseeds; base += 1024) {
        int cnt = min(1024, nseeds - base);
        __syncthreads();
        for (int q = threadIdx.x; q < 3 * cnt; q += blockDim.x)
            s_seed[q] = seeds[3 * base + q];
        __syncthreads();
        if (mine) {
            for (int q = 0; q < cnt; q++) {
                float dx = (float)(abs(s_seed[3 * q] - gx));
                float dy = (float)(abs(s_seed[3 * q + 1] - gy));
                float dz = (float)(abs(s_seed[3 * q + 2] - k));
                float dist = sqrtf(dx * dx + dy * dy + dz * dz);
                if (dist < best) {
                    best_i = base + q;
                    best = dist;
                }
            }
        }
    }
    if (mine)
        D.gid[c] = best_i + 1;
}

// Active cells of the active window: fresh octahedra and their records. At admission these are
// the initially active cells (src/CAinitialize.cpp:1929-2044); at the start of a later layer, the
// active cells of the moved window (LayerSetup, src/CAinitialize.cpp:2840-2982).
__global__ void k_init_active(PoolState *P, int dom, int list_slot) {
    if (list_slot < 0)
        list_slot = P->pending; // the list the next cycle consumes
    DomainDesc &D = P->desc[dom];
    long long plane = (long long)D.mx * D.my;
    long long lo = plane, hi = plane * (D.nz - 1);
    if (lo < plane * D.z_lo)
        lo = plane * D.z_lo;
    if (hi > plane * D.z_end)
        hi = plane * D.z_end;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long c0 = lo + (long long)blockIdx.x * blockDim.x; c0 < hi; c0 += stride) {
        long long c = c0 + threadIdx.x;
        bool act = c < hi && D.ctype[c] == kActive;
        if (act)
            make_fresh_octahedron(D, (unsigned int)c);
        bool listed = act;
        unsigned long long pos = block_reserve(P, list_slot, listed ? 1u : 0u);
        if (listed && pos != ULLONG_MAX) {
            const RecordList L = list_of(P, list_slot);
            L.rec[pos] = ActiveRec{0.01f, 0.0f, D.cts_run[c], kMaskFresh};
            L.cell[pos] = (unsigned int)c;
            L.dom[pos] = dom_word((unsigned int)dom, kNoDir);
            L.min2[pos] = 0.0f;
            D.pos[c] = (unsigned int)pos;
            if (pos < L.body_cap) {
                RecordBody &b = L.body[pos];
                body_head(b) = make_float4(__int_as_float(D.gid[c]), D.doc[3ull * c], D.doc[3ull * c + 1], D.doc[3ull * c + 2]);
                for (int l = 0; l < 26; l++)
                    b.cdl[l] = D.cdl[26ull * c + l];
            }
        }
    }
}

// Re-labels every record of one domain in the list the next cycle consumes with the pool's
// always-finished placeholder domain (used when a slot is retired, before the slot is reused).
__global__ void k_drop_domain(PoolState *P, unsigned int dom, unsigned int placeholder) {
    const int nxt = P->pending;
    unsigned long long n = P->cnt[nxt];
    unsigned int *d = P->rdom[nxt];
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x)
        if (word_dom(d[i]) == dom)
            d[i] = dom_word(placeholder, kNoDir);
}

// Diagonal lengths held in the pending records back to the per-cell arrays.
__global__ void k_flush_records(PoolState *P) {
    const int nxt = P->pending;
    unsigned long long n = P->cnt[nxt];
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const ActiveRec r = P->rec[nxt][i];
        if (r.stat & kMaskTomb)
            continue; // a dropped record's other fields are not kept up to date
        const DomainDesc &D = P->desc[word_dom(P->rdom[nxt][i])];
        if (D.dl)
            D.dl[P->rcell[nxt][i]] = r.dl;
    }
}

// ---------------------------------------------------------------------------------------------
// Cell fields of a type-C problem made on the device (src/CAinitialize.cpp:1025-1055, 1460-1529,
// 1834-2247): walls on the ghost ring and the bottom and top planes, liquid elsewhere, the plane's
// CritTimeStep, LayerID 0, one UndercoolingChange value; then the substrate seeds (active, GrainID
// rank + 1) and the nuclei (GrainID -(rank + 1), in index order).
__global__ void k_fill_directional(int8_t *ctype, int32_t *gid, int32_t *cts, int8_t *layer, float *du, long long n,
                                   int mx, int my, int nz, const int32_t *plane_cts, float du_value) {
    const long long plane = (long long)mx * my;
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(c / plane);
        const int rem = (int)(c - (long long)k * plane);
        const int i = rem / my, j = rem - (rem / my) * my;
        const bool wall = i == 0 || i == mx - 1 || j == 0 || j == my - 1 || k == 0 || k == nz - 1;
        ctype[c] = wall ? kWall : kLiquid;
        gid[c] = 0;
        cts[c] = __ldg(plane_cts + k);
        layer[c] = 0;
        du[c] = du_value;
    }
}

__global__ void k_widen_types(const int8_t *ctype, int32_t *out, long long n) {
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x)
        out[c] = ctype[c];
}

__global__ void k_scatter_seeds(int8_t *ctype, int32_t *gid, const long long *active, long long n_active,
                                const int32_t *nuclei, long long n_nuclei) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n_active) {
        ctype[active[q]] = kActive;
        gid[active[q]] = (int32_t)(q + 1);
    }
    else if (q < n_active + n_nuclei) {
        const long long r = q - n_active;
        gid[nuclei[r]] = -(int32_t)(r + 1);
    }
}

// ---------------------------------------------------------------------------------------------
// Layer change of a multilayer domain (src/runCA.cpp:344-411).

// Undercooling updates of the ending layer, carried into the next: every liquid or active cell of
// the window whose LayerID <= layer had UndercoolingCurrent += UndercoolingChange once per executed
// cycle past its CritTimeStep (src/CAupdate.cpp:228-237).
__global__ void k_layer_base(const DomainDesc *Dp) {
    const DomainDesc &D = *Dp;
    const long long plane = (long long)D.mx * D.my;
    const long long hi = plane * D.z_end;
    const long long end = executed_upto(D, D.cycle);
    for (long long c = plane * D.z_lo + (long long)blockIdx.x * blockDim.x + threadIdx.x; c < hi;
         c += (long long)gridDim.x * blockDim.x) {
        const int t = D.ctype[c];
        if ((t != kLiquid && t != kActive) || D.layer[c] > D.layer_no)
            continue;
        const long long n = end - executed_upto(D, D.cts[c]);
        if (n > 0)
            D.nu_base[c] += (int32_t)n;
    }
}

// DomainShiftAndResize's two reductions (src/CAinitialize.cpp:2781-2812): the lowest z of an
// active cell and the highest z of a cell of the next layer. out = {INT_MAX, INT_MIN} on entry.
__global__ void k_layer_bounds(const DomainDesc *Dp, int next_layer, int *out) {
    const DomainDesc &D = *Dp;
    const long long plane = (long long)D.mx * D.my;
    int zmin = INT_MAX, zmax = INT_MIN;
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < D.domain_size;
         c += (long long)gridDim.x * blockDim.x) {
        const int z = (int)(c / plane);
        if (D.ctype[c] == kActive)
            zmin = min(zmin, z);
        if (D.layer[c] == next_layer)
            zmax = max(zmax, z);
    }
    for (int o = 16; o; o >>= 1) {
        zmin = min(zmin, __shfl_down_sync(0xffffffffu, zmin, o));
        zmax = max(zmax, __shfl_down_sync(0xffffffffu, zmax, o));
    }
    if ((threadIdx.x & 31) == 0) {
        if (zmin != INT_MAX)
            atomicMin(out, zmin);
        if (zmax != INT_MIN)
            atomicMax(out + 1, zmax);
    }
}

// The CritTimeStep the step uses this layer: the cell's own inside the window for LayerID <= layer,
// INT_MAX elsewhere (src/CAupdate.cpp:218-231 visits only window cells, and grows those with
// LayerID <= layernumber).
__global__ void k_layer_gate(const DomainDesc *Dp) {
    const DomainDesc &D = *Dp;
    const long long plane = (long long)D.mx * D.my;
    const long long lo = plane * D.z_lo, hi = plane * D.z_end;
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < D.domain_size;
         c += (long long)gridDim.x * blockDim.x)
        D.cts_run[c] = (c >= lo && c < hi && D.layer[c] <= D.layer_no) ? D.cts[c] : INT_MAX;
}

// ---------------------------------------------------------------------------------------------
// Pool runtime

namespace {
inline cudaStream_t S(void *s) { return (cudaStream_t)s; }
template <class T> T *dalloc(size_t n, std::vector<void *> &allocs, size_t &bytes) {
    void *p = nullptr;
    size_t b = std::max<size_t>(n * sizeof(T), 16);
    CUDA_OK(cudaMalloc(&p, b));
    allocs.push_back(p);
    bytes += b;
    return (T *)p;
}

// true when p is page-locked (or registered) host memory that a copy engine writes directly
bool host_pinned(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

// Moves one staged piece into the caller's buffer on several host threads: len bytes, or with
// widen len int8 values sign-extended to int32.
void stage_move(char *dst, const char *src, size_t len, bool widen) {
    constexpr size_t kPerThread = size_t(1) << 20;
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    const size_t nt = std::max<size_t>(1, std::min<size_t>({(size_t)hw, 8, len / kPerThread}));
    auto part = [&](size_t t) {
        const size_t lo = len * t / nt, hi = len * (t + 1) / nt;
        if (widen) {
            int32_t *o = (int32_t *)dst;
            const int8_t *i = (const int8_t *)src;
            for (size_t k = lo; k < hi; k++)
                o[k] = i[k];
        } else {
            std::memcpy(dst + lo, src + lo, hi - lo);
        }
    };
    std::vector<std::thread> workers;
    for (size_t t = 1; t < nt; t++)
        workers.emplace_back(part, t);
    part(0);
    for (auto &w : workers)
        w.join();
}
} // namespace

void Pool::to_host(const std::vector<HostCopy> &copies, void *stream) {
    constexpr size_t kStageBytes = size_t(32) << 20;
    cudaStream_t st = S(stream);
    // page-locked destinations take their DMA as they are; the rest go through the staging pieces
    struct Piece {
        char *dst;
        const char *src;
        size_t len;
        bool widen;
    };
    std::vector<Piece> pieces;
    for (const HostCopy &c : copies) {
        if (!c.dst || !c.bytes)
            continue;
        if (!c.widen && host_pinned(c.dst)) {
            CUDA_OK(cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToHost, st));
            continue;
        }
        for (size_t off = 0; off < c.bytes; off += kStageBytes)
            pieces.push_back({(char *)c.dst + (c.widen ? 4 * off : off), (const char *)c.src + off,
                              std::min(kStageBytes, c.bytes - off), c.widen});
    }
    if (pieces.empty())
        return;
    // The pieces are as large as this copy or the largest domain's GrainID needs, up to kStageBytes:
    // page-locking 64 MB takes some 30 ms (a new pool's first 64^3 solve 71 -> 38 ms), but each growth also
    // waits for what runs on the device. No piece is in flight here.
    size_t need = 0;
    for (const Piece &q : pieces)
        need = std::max(need, q.len);
    for (const auto &q : slots_)
        if (q.used)
            need = std::max(need, (size_t)q.problem->g.domain_size * 4);
    need = std::min(kStageBytes, need);
    if (need > stage_bytes_) {
        need = std::min(kStageBytes, std::max(2 * stage_bytes_, (need + (size_t(1) << 20) - 1) >> 20 << 20));
        stage_bytes_ = 0;
        for (int b = 0; b < 2; b++) {
            if (stage_[b]) {
                void *old = stage_[b];
                stage_[b] = nullptr;
                CUDA_OK(cudaFreeHost(old));
            }
            CUDA_OK(cudaMallocHost(&stage_[b], need));
            if (!stage_ev_[b]) {
                cudaEvent_t e;
                CUDA_OK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
                stage_ev_[b] = e;
            }
        }
        stage_bytes_ = need;
    }
    // two pieces in flight: the DMA of piece k+1 runs while the host threads move piece k out
    auto issue = [&](size_t k) {
        CUDA_OK(cudaMemcpyAsync(stage_[k & 1], pieces[k].src, pieces[k].len, cudaMemcpyDeviceToHost, st));
        CUDA_OK(cudaEventRecord((cudaEvent_t)stage_ev_[k & 1], st));
    };
    issue(0);
    for (size_t k = 0; k < pieces.size(); k++) {
        if (k + 1 < pieces.size())
            issue(k + 1);
        CUDA_OK(cudaEventSynchronize((cudaEvent_t)stage_ev_[k & 1]));
        stage_move(pieces[k].dst, (const char *)stage_[k & 1], pieces[k].len, pieces[k].widen);
    }
}

void pin_problem(Problem &p) {
    auto reg = [](void *ptr, size_t bytes) {
        if (bytes == 0)
            return;
        cudaError_t e = cudaHostRegister(ptr, bytes, cudaHostRegisterDefault);
        if (e != cudaSuccess && e != cudaErrorHostMemoryAlreadyRegistered)
            throw DeviceError(std::string("CUDA error ") + cudaGetErrorString(e) + " at cudaHostRegister");
        cudaGetLastError();
    };
    reg(p.cell_type.data(), p.cell_type.size());
    reg(p.grain_id.data(), p.grain_id.size() * 4);
    reg(p.cts.data(), p.cts.size() * 4);
    reg(p.layer_id.data(), p.layer_id.size());
    reg(p.du.data(), p.du.size() * 4);
    p.pinned = true;
}

void unpin_problem(Problem &p) {
    if (!p.pinned)
        return;
    for (void *ptr : {(void *)p.cell_type.data(), (void *)p.grain_id.data(), (void *)p.cts.data(),
                      (void *)p.layer_id.data(), (void *)p.du.data()})
        if (ptr)
            cudaHostUnregister(ptr);
    cudaGetLastError();
    p.pinned = false;
}

// Multilayer problems keep the per-cell octahedron state for the whole domain (the active window
// moves up layer by layer), plus the per-layer CritTimeStep gate and the undercooling carried over.
static size_t octahedron_cells(const Problem &p) {
    return p.cfg.number_of_layers > 1 ? (size_t)p.g.domain_size : (size_t)p.g.active_size;
}

size_t Pool::slot_bytes(const Problem &p) {
    size_t N = (size_t)p.g.domain_size, A = octahedron_cells(p);
    size_t multilayer = p.cfg.number_of_layers > 1 ? N * 8 : 0;
    size_t classes = p.du_values.size() > 1 ? N * 2 : 0;
    return N * (1 + 4 + 4 + 1 + 4) + A * (4 + 12 + 104 + 8 + 4) + multilayer + classes + p.nuclei_loc.size() * 8 +
           64 * 1024;
}

Pool::Pool(int device, size_t budget_bytes, unsigned long long list_capacity)
    : device_(device), budget_(budget_bytes) {
    CUDA_OK(cudaSetDevice(device));
    cudaDeviceProp prop;
    CUDA_OK(cudaGetDeviceProperties(&prop, device));
    num_sms_ = prop.multiProcessorCount;
    cudaStream_t s;
    CUDA_OK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    stream_ = s;
    // the device's edge masks (edge_mask) are the reference's ItList cases
    int it[9][26], lens[9];
    build_itlist(it, lens);
    for (int b = 0; b < 9; b++) {
        unsigned int m = 0, want = (1u << 26) - 1u;
        for (int q = 0; q < lens[b]; q++)
            m |= 1u << it[b][q];
        if (b == 1 || b == 5 || b == 6)
            want &= ~kDirYM;
        if (b == 2 || b == 7 || b == 8)
            want &= ~kDirYP;
        if (b == 3 || b == 5 || b == 7)
            want &= ~kDirXM;
        if (b == 4 || b == 6 || b == 8)
            want &= ~kDirXP;
        if (m != want)
            throw std::logic_error("edge masks differ from ItList");
    }
    max_domains_ = 8192;
    // list positions are 32-bit in the passes' block-local queues
    if (list_capacity > 0xffffffffull)
        throw Unsupported("list capacity above 2^32 - 1 records");
    capacity_ = std::max<unsigned long long>(list_capacity, 1024);
    int coop = 0;
    CUDA_OK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
    if (!coop)
        throw DeviceError("device does not support cooperative launches");
    int b = 0;
    for (int v = 0; v < kStepVariants; v++) {
        CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kStepKernel[v].cycles, kBlock, 0));
        int many = 0;
        CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&many, kStepKernel[v].cycles_many, kBlock, 0));
        b = std::min(b, many);
        if (b < 1)
            throw DeviceError("persistent kernel does not fit on an SM");
        grid_cycles_[v] = num_sms_ * b;
        CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, (const void *)kStepKernel[v].grow, kBlock, 0));
        grid_grow_[v] = num_sms_ * std::max(b, 1);
        CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, (const void *)kStepKernel[v].capture_end, kBlock, 0));
        grid_capture_[v] = num_sms_ * std::max(b, 1);
    }
    CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_claim, kBlock, 0));
    grid_claim_ = num_sms_ * std::max(b, 1);
    if (const char *m = std::getenv("EXACA_STEP_MODE"))
        step_mode_ = std::string(m) == "graph" ? 1 : 0;
    {
        // Domain slabs and growth tables come from the device's stream-ordered pool: admission and
        // retirement then queue behind running cycles instead of synchronising the device, and
        // freed slabs are reused by later admissions (the pool keeps what it has reserved until
        // this process ends).
        cudaMemPool_t mp;
        CUDA_OK(cudaDeviceGetDefaultMemPool(&mp, device));
        unsigned long long keep = ~0ull;
        CUDA_OK(cudaMemPoolSetAttribute(mp, cudaMemPoolAttrReleaseThreshold, &keep));
    }
    CUDA_OK(cudaMalloc(&dstate_, sizeof(PoolState)));
    CUDA_OK(cudaMalloc(&ddesc_, sizeof(DomainDesc) * (max_domains_ + 1)));
    CUDA_OK(cudaMemsetAsync(ddesc_, 0, sizeof(DomainDesc) * (max_domains_ + 1), s));
    {
        // descriptor max_domains_ is a placeholder that is always finished
        DomainDesc ph;
        std::memset(&ph, 0, sizeof(ph));
        ph.done = 1;
        CUDA_OK(cudaMemcpyAsync(ddesc_ + max_domains_, &ph, sizeof(ph), cudaMemcpyHostToDevice, s));
    }
    PoolState ps;
    std::memset(&ps, 0, sizeof(ps));
    for (int q = 0; q < 2; q++) {
        CUDA_OK(cudaMalloc(&ps.rec[q], capacity_ * sizeof(ActiveRec)));
        CUDA_OK(cudaMalloc(&ps.rdom[q], capacity_ * sizeof(unsigned int)));
        CUDA_OK(cudaMalloc(&ps.rcell[q], capacity_ * sizeof(unsigned int)));
        CUDA_OK(cudaMalloc(&ps.rmin2[q], capacity_ * sizeof(float)));
        CUDA_OK(cudaMalloc(&ps.body[q], std::min(capacity_, kBodyRecords) * sizeof(RecordBody)));
    }
    ps.body_cap = (unsigned int)std::min(capacity_, kBodyRecords);
    // a shard takes the entries of 1/kShards of the warps: room for its share of the list plus slack
    ps.shard_cap = capacity_ / kShards + 8192;
    const size_t qn = (size_t)kShards * ps.shard_cap;
    // the persistent kernel splits the claim list into one segment per block of its grid
    ps.tgt_len = qn + 4096ull * (unsigned long long)num_sms_;
    CUDA_OK(cudaMalloc(&ps.tgt, ps.tgt_len * sizeof(unsigned long long)));
    CUDA_OK(cudaMalloc(&ps.qpos, qn * sizeof(unsigned int)));
    CUDA_OK(cudaMalloc(&ps.qdom, qn * sizeof(unsigned int)));
    CUDA_OK(cudaMalloc(&ps.qmask, qn * sizeof(unsigned int)));
    CUDA_OK(cudaMalloc(&ps.qdl, qn * sizeof(float)));
    ps.capacity = capacity_;
    ps.cur = 0;
    ps.pending = 0;
    ps.n_domains = 0;
    ps.desc = ddesc_;
    CUDA_OK(cudaMemcpyAsync(dstate_, &ps, sizeof(ps), cudaMemcpyHostToDevice, s));
    CUDA_OK(cudaMalloc(&census_buf_, sizeof(Census)));
}

Pool::~Pool() {
    cudaSetDevice(device_);
    cudaStreamSynchronize(S(stream_));
    if (graph_exec_)
        cudaGraphExecDestroy((cudaGraphExec_t)graph_exec_);
    for (auto &s : slots_) {
        for (void *p : s.allocs)
            cudaFree(p);
        if (s.growth)
            cudaFree(s.growth);
    }
    for (auto &kv : tables_) {
        cudaFree(kv.second.guv);
        cudaFree(kv.second.mis);
        cudaFree(kv.second.cdl_table);
    }
    if (dstate_) {
        PoolState ps;
        if (cudaMemcpy(&ps, dstate_, sizeof(ps), cudaMemcpyDeviceToHost) == cudaSuccess) {
            for (int q = 0; q < 2; q++) {
                cudaFree(ps.rec[q]);
                cudaFree(ps.rdom[q]);
                cudaFree(ps.rcell[q]);
                cudaFree(ps.rmin2[q]);
                cudaFree(ps.body[q]);
            }
            cudaFree(ps.tgt);
            cudaFree(ps.qpos);
            cudaFree(ps.qdom);
            cudaFree(ps.qmask);
            cudaFree(ps.qdl);
        }
        cudaFree(dstate_);
    }
    cudaFree(ddesc_);
    cudaFree(census_buf_);
    if (copy_stream_)
        cudaStreamSynchronize(S(copy_stream_));
    for (int b = 0; b < 2; b++) {
        if (stage_[b])
            cudaFreeHost(stage_[b]);
        if (stage_ev_[b])
            cudaEventDestroy((cudaEvent_t)stage_ev_[b]);
    }
    cudaStreamDestroy(S(stream_));
    if (copy_stream_)
        cudaStreamDestroy(S(copy_stream_));
}

const DeviceTables &Pool::tables_for(const Problem &p) {
    auto it = tables_.find(p.cfg.orientation_file);
    if (it != tables_.end())
        return it->second;
    DeviceTables t;
    CUDA_OK(cudaMalloc(&t.guv, p.guv.size() * sizeof(float)));
    CUDA_OK(cudaMalloc(&t.cdl_table, p.cdl_table.size() * sizeof(float)));
    // on the pool's stream, as everything that its kernels read: it does not wait for the legacy stream, where
    // a copy from pageable memory may still be under way when the call returns
    cudaStream_t st = S(stream_);
    CUDA_OK(cudaMemcpyAsync(t.guv, p.guv.data(), p.guv.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    CUDA_OK(cudaMemcpyAsync(t.cdl_table, p.cdl_table.data(), p.cdl_table.size() * sizeof(float), cudaMemcpyHostToDevice,
                            st));
    h2d_bytes_ += (p.guv.size() + p.cdl_table.size()) * sizeof(float);
    return tables_[p.cfg.orientation_file] = t;
}

void Pool::push_desc(int slot) {
    // pageable source: staged before the call returns
    CUDA_OK(cudaMemcpyAsync(ddesc_ + slot, &host_desc_[slot], sizeof(DomainDesc), cudaMemcpyHostToDevice, S(stream_)));
}

void Pool::ensure_growth(int slot, long long needed) {
    SlotHost &s = slots_[slot];
    if (needed < s.growth_len)
        return;
    long long len = std::max<long long>(needed + 1, std::max<long long>(2LL * s.growth_len, 4096));
    if (len > INT_MAX / 2)
        throw Unsupported("growth table too long");
    // one table per distinct UndercoolingChange value, table c at c * len
    const Problem &p = *s.problem;
    const size_t n_tables = std::max<size_t>(1, p.du_values.size());
    std::vector<double> g(n_tables * (size_t)len);
    if (p.du_values.size() > 1) {
        for (size_t c = 0; c < n_tables; c++)
            build_growth_table(p, p.du_values[c], (int)len, g.data() + c * (size_t)len);
    }
    else {
        build_growth_table(p, p.du_value, (int)len, g.data());
    }
    double *d = nullptr;
    CUDA_OK(cudaMallocAsync((void **)&d, g.size() * sizeof(double), S(stream_)));
    CUDA_OK(cudaMemcpyAsync(d, g.data(), g.size() * sizeof(double), cudaMemcpyHostToDevice, S(stream_)));
    h2d_bytes_ += g.size() * sizeof(double);
    if (s.growth) {
        // queued work may still read the old table: it is freed in stream order after that work
        CUDA_OK(cudaFreeAsync(s.growth, S(stream_)));
    }
    s.growth = d;
    s.growth_len = (int)len;
    // patch only the table fields of the device descriptor
    DomainDesc &h = host_desc_[slot];
    h.growth = d;
    h.growth_len = (int)len;
    CUDA_OK(cudaMemcpyAsync((char *)(ddesc_ + slot) + offsetof(DomainDesc, growth), &h.growth, sizeof(h.growth),
                            cudaMemcpyHostToDevice, S(stream_)));
    CUDA_OK(cudaMemcpyAsync((char *)(ddesc_ + slot) + offsetof(DomainDesc, growth_len), &h.growth_len,
                            sizeof(h.growth_len), cudaMemcpyHostToDevice, S(stream_)));
}

// Named range on the host timeline for profilers (NVTX; inert when no tool is attached).
struct TraceRange {
    explicit TraceRange(const char *name) { nvtxRangePushA(name); }
    ~TraceRange() { nvtxRangePop(); }
    TraceRange(const TraceRange &) = delete;
    TraceRange &operator=(const TraceRange &) = delete;
};

int Pool::admit(std::shared_ptr<const Problem> pp, int check_mode) {
    TraceRange trace("exaca admit");
    CUDA_OK(cudaSetDevice(device_));
    const Problem &p = *pp;
    if (p.g.zbound_low != 0)
        throw Unsupported("active window must start at z = 0");
    size_t need = slot_bytes(p);
    if (bytes_in_use_ + need > budget_)
        throw AdmissionRefused("admission refused: HBM budget exceeded");
    int slot = -1;
    for (int s = 0; s < (int)slots_.size(); s++)
        if (!slots_[s].used) {
            slot = s;
            break;
        }
    if (slot < 0) {
        if ((int)slots_.size() >= max_domains_)
            throw AdmissionRefused("admission refused: too many domains");
        slot = (int)slots_.size();
        slots_.emplace_back();
        host_desc_.emplace_back();
    }
    SlotHost &s = slots_[slot];
    s = SlotHost();
    s.used = true;
    s.problem = pp;
    const Geometry &g = p.g;
    const int n_layers = p.cfg.number_of_layers;
    const bool multilayer = n_layers > 1;
    const bool classes = p.du_values.size() > 1;
    if (check_mode && p.cfg.simulation_type != "C")
        throw Unsupported("device-side termination covers type-C problems (types S and R jump cycles, stop at "
                          "finish time steps or change layers between launches): admit with device_check 0 "
                          "and run the plain path");
    const size_t N = g.domain_size, A = octahedron_cells(p), P = p.nuclei_loc.size();
    // every field of the slot in one allocation (256-byte aligned sub-arrays)
    size_t off = 0;
    auto carve = [&](size_t bytes) {
        size_t o = off;
        off += (std::max<size_t>(bytes, 16) + 255) & ~(size_t)255;
        return o;
    };
    const size_t o_ct = carve(N), o_gid = carve(N * 4), o_cts = carve(N * 4), o_ly = carve(N), o_du = carve(N * 4),
                 o_dl = carve(A * 4), o_doc = carve(A * 12), o_cdl = carve(A * 104), o_claim = carve(A * 8),
                 o_pos = carve(A * 4), o_nl = carve(P * 4), o_nt = carve(P * 4),
                 o_run = multilayer ? carve(N * 4) : 0, o_base = multilayer ? carve(N * 4) : 0,
                 o_cls = classes ? carve(N * 2) : 0;
    char *slab = nullptr;
    CUDA_OK(cudaMallocAsync((void **)&slab, off, S(stream_)));
    s.allocs.push_back(slab);
    s.bytes = off;
    DomainDesc d;
    std::memset(&d, 0, sizeof(d));
    d.ctype = (int8_t *)(slab + o_ct);
    d.gid = (int32_t *)(slab + o_gid);
    d.cts = (int32_t *)(slab + o_cts);
    d.layer = (int8_t *)(slab + o_ly);
    d.du = (float *)(slab + o_du);
    d.dl = (float *)(slab + o_dl);
    d.doc = (float *)(slab + o_doc);
    d.cdl = (float *)(slab + o_cdl);
    d.claim = (unsigned long long *)(slab + o_claim);
    d.pos = (unsigned int *)(slab + o_pos);
    d.cts_run = multilayer ? (int32_t *)(slab + o_run) : d.cts;
    d.nu_base = multilayer ? (int32_t *)(slab + o_base) : nullptr;
    d.du_class = classes ? (const uint16_t *)(slab + o_cls) : nullptr;
    int32_t *dnl = (int32_t *)(slab + o_nl);
    int32_t *dnt = (int32_t *)(slab + o_nt);
    // nuclei in time order; ties keep the reference's order (order does not change results)
    std::vector<int> order(P);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return p.nuclei_time[a] < p.nuclei_time[b]; });
    std::vector<int32_t> nl(P), nt(P);
    for (size_t q = 0; q < P; q++) {
        nl[q] = p.nuclei_loc[order[q]];
        nt[q] = p.nuclei_time[order[q]];
    }
    // host->device copies on the pool stream; pageable sources are staged before each call returns
    cudaStream_t st = S(stream_);
    if (p.dir.used) {
        // type C: the cell fields are made here from the plane CritTimeSteps, the substrate seeds and
        // the nuclei (a few KB cross PCIe instead of 14 bytes per cell)
        const size_t nk = p.dir.plane_cts.size(), na = p.dir.active.size(), nn = p.nuclei_loc.size();
        const size_t bytes = nk * 4 + na * 8 + nn * 4;
        // one upload: the 8-byte seed indices first (the allocation is 256-byte aligned), then the
        // 4-byte plane CritTimeSteps and nucleus indices
        std::vector<char> host(bytes);
        std::memcpy(host.data(), p.dir.active.data(), na * 8);
        std::memcpy(host.data() + na * 8, p.dir.plane_cts.data(), nk * 4);
        std::memcpy(host.data() + na * 8 + nk * 4, p.nuclei_loc.data(), nn * 4);
        char *dseed = nullptr;
        CUDA_OK(cudaMallocAsync((void **)&dseed, std::max<size_t>(bytes, 16), st));
        CUDA_OK(cudaMemcpyAsync(dseed, host.data(), bytes, cudaMemcpyHostToDevice, st));
        h2d_bytes_ += bytes;
        const long long *active = (const long long *)dseed;
        const int32_t *plane_cts = (const int32_t *)(dseed + na * 8);
        const int32_t *nuc = (const int32_t *)(dseed + na * 8 + nk * 4);
        const unsigned blocks = (unsigned)std::min<long long>((N + 255) / 256, (long long)num_sms_ * 16);
        k_fill_directional<<<blocks, 256, 0, st>>>(d.ctype, d.gid, d.cts, d.layer, d.du, (long long)N, g.mx, g.my,
                                                   g.nz, plane_cts, p.du_value);
        CUDA_OK(cudaGetLastError());
        const long long nseed = (long long)(na + nn);
        if (nseed)
            k_scatter_seeds<<<(unsigned)((nseed + 255) / 256), 256, 0, st>>>(d.ctype, d.gid, active, (long long)na,
                                                                             nuc, (long long)nn);
        CUDA_OK(cudaGetLastError());
        CUDA_OK(cudaFreeAsync(dseed, st));
    }
    else {
        CUDA_OK(cudaMemcpyAsync(d.ctype, p.cell_type.data(), N, cudaMemcpyHostToDevice, st));
        CUDA_OK(cudaMemcpyAsync(d.gid, p.grain_id.data(), N * 4, cudaMemcpyHostToDevice, st));
        CUDA_OK(cudaMemcpyAsync(d.cts, p.cts.data(), N * 4, cudaMemcpyHostToDevice, st));
        CUDA_OK(cudaMemcpyAsync(d.layer, p.layer_id.data(), N, cudaMemcpyHostToDevice, st));
        CUDA_OK(cudaMemcpyAsync(d.du, p.du.data(), N * 4, cudaMemcpyHostToDevice, st));
        h2d_bytes_ += N * 14;
    }
    CUDA_OK(cudaMemsetAsync(d.dl, 0, A * 4, st));
    CUDA_OK(cudaMemsetAsync(d.claim, 0xff, A * 8, st));
    CUDA_OK(cudaMemsetAsync(d.pos, 0xff, A * 4, st)); // kNoRecord
    if (multilayer)
        CUDA_OK(cudaMemsetAsync(d.nu_base, 0, N * 4, st));
    if (classes)
        CUDA_OK(cudaMemcpyAsync((void *)d.du_class, p.du_class.data(), N * 2, cudaMemcpyHostToDevice, st));
    if (P) {
        CUDA_OK(cudaMemcpyAsync(dnl, nl.data(), P * 4, cudaMemcpyHostToDevice, st));
        CUDA_OK(cudaMemcpyAsync(dnt, nt.data(), P * 4, cudaMemcpyHostToDevice, st));
    }
    h2d_bytes_ += (classes ? N * 2 : 0) + P * 8;
    const DeviceTables &tb = tables_for(p);
    d.guv = tb.guv;
    d.cdl_table = tb.cdl_table;
    d.nuc_loc = dnl;
    d.nuc_time = dnt;
    d.n_nuclei = (int)P;
    d.mx = g.mx;
    d.my = g.my;
    d.nz = g.nz;
    d.nz_active = g.nz_active;
    d.xoff = g.xoff;
    d.yoff = g.yoff;
    d.zbound_high = g.zbound_high;
    d.layer_no = 0;
    d.n_layers = n_layers;
    d.z_lo = g.zbound_low;
    d.z_end = g.zbound_low + g.nz_active;
    d.check_mode = check_mode;
    d.domain_size = g.domain_size;
    d.active_size = (long long)A;
    d.du_value = p.du_value;
    long long liquid = 0;
    int zero_du = 0, cts_max = INT_MIN;
    if (p.dir.used) {
        // every cell inside the wall ring is liquid except the substrate seeds
        liquid = (long long)(g.mx - 2) * (g.my - 2) * (g.nz - 2) - (long long)p.dir.active.size();
        zero_du = p.du_value == 0.0f ? 1 : 0;
        for (int32_t c : p.dir.plane_cts)
            cts_max = std::max(cts_max, c);
    }
    else {
        for (long i = 0; i < g.domain_size; i++) {
            int8_t t = p.cell_type[i];
            if (t == kLiquid && p.layer_id[i] == 0)
                liquid++;
            if ((t == kLiquid || t == kActive) && p.du[i] == 0.0f)
                zero_du = 1;
            cts_max = std::max(cts_max, p.cts[i]);
        }
    }
    d.liquid = liquid;
    d.zero_du = zero_du;
    d.cts_max = cts_max == INT_MIN ? INT_MAX : cts_max;
    host_desc_[slot] = d;
    push_desc(slot);
    if (multilayer) {
        k_layer_gate<<<num_sms_ * 4, 256, 0, st>>>(ddesc_ + slot);
        CUDA_OK(cudaGetLastError());
    }
    if (multilayer || classes) {
        static const int one = 1;
        CUDA_OK(cudaMemcpyAsync((char *)dstate_ + offsetof(PoolState, extras), &one, sizeof(int),
                                cudaMemcpyHostToDevice, st));
    }
    ensure_growth(slot, 4096);
    if (!p.voronoi_seeds.empty() || p.cfg.simulation_type != "C") {
        int nseeds = (int)(p.voronoi_seeds.size() / 3);
        int32_t *dseeds = nullptr;
        if (nseeds) {
            CUDA_OK(cudaMallocAsync((void **)&dseeds, p.voronoi_seeds.size() * 4, st));
            CUDA_OK(cudaMemcpyAsync(dseeds, p.voronoi_seeds.data(), p.voronoi_seeds.size() * 4,
                                    cudaMemcpyHostToDevice, st));
        }
        long long blocks = (g.domain_size + 255) / 256;
        k_voronoi<<<(unsigned)blocks, 256, 3 * 1024 * sizeof(int), st>>>(ddesc_ + slot, dseeds, nseeds,
                                                                         (float)(g.active_size));
        CUDA_OK(cudaGetLastError());
        if (dseeds)
            CUDA_OK(cudaFreeAsync(dseeds, st));
    }
    // register the domain, then build its initial active list in the list the next cycle consumes
    n_domains_ = std::max(n_domains_, slot + 1);
    CUDA_OK(cudaMemcpyAsync((char *)dstate_ + offsetof(PoolState, n_domains), &n_domains_, sizeof(int),
                            cudaMemcpyHostToDevice, st));
    k_init_active<<<num_sms_ * 4, 256, 0, st>>>(dstate_, slot, -1);
    CUDA_OK(cudaGetLastError());
    bytes_in_use_ += s.bytes;
    // the list's length until the next state read: as then, with the new domain's first active cells
    list_read_ = false;
    last_records_ += p.dir.used ? p.dir.active.size() : 0;
    return slot;
}

void Pool::retire(int slot) {
    TraceRange trace("exaca retire");
    CUDA_OK(cudaSetDevice(device_));
    SlotHost &s = slots_.at(slot);
    if (!s.used)
        return;
    cudaStream_t st = S(stream_);
    // mark done and drop its list entries before the memory goes away
    int one = 1;
    CUDA_OK(cudaMemcpyAsync((char *)(ddesc_ + slot) + offsetof(DomainDesc, done), &one, sizeof(int),
                            cudaMemcpyHostToDevice, st));
    k_drop_domain<<<num_sms_ * 2, 256, 0, st>>>(dstate_, (unsigned)slot, (unsigned)max_domains_);
    CUDA_OK(cudaGetLastError());
    DomainDesc zero;
    std::memset(&zero, 0, sizeof(zero));
    zero.done = 1;
    host_desc_[slot] = zero;
    // the copies from host memory are staged before each call returns; everything below runs in
    // stream order after the cycles already queued, so nothing waits here
    CUDA_OK(cudaMemcpyAsync(ddesc_ + slot, &zero, sizeof(zero), cudaMemcpyHostToDevice, st));
    for (void *p : s.allocs)
        CUDA_OK(cudaFreeAsync(p, st));
    if (s.growth)
        CUDA_OK(cudaFreeAsync(s.growth, st));
    bytes_in_use_ -= s.bytes;
    s = SlotHost();
}

// The persistent shape for a list of n records (0: not known). us per cycle of whole directional solves
// (records in the mean; a front is longest in mid-solve), long list with two / four records per lane, middle,
// short: 64^3 (7.0e3) 11.3 / 12.0 / 9.2 / 8.7, 128^3 (3.5e4) 12.6 / 13.3 / 10.3 / 10.4, 192^3 (8.7e4) 14.5 / 14.9
// / 12.2 / 13.0, 320^3 (2.9e5) 21.5 / 21.9 / 20.8 / 21.8, 400^3 (4.7e5) 26.9 / 27.3 / 28.0 / 29.2, 512^3 (8.0e5)
// 36.8 / 36.8 / 40.5 / 42.1; by this rule 8.7, 10.2, 12.3, 20.8, 26.5, 36.4.
int Pool::shape_for(unsigned long long n) {
    if (n == 0)
        return 2;
    return n < (1ull << 15) ? 3 : (n < 350000 ? 2 : (n < 700000 ? 0 : 1));
}

// Blocks of a persistent launch of n cycles, of the `full` co-resident ones. A launch that holds every SM
// keeps out those of other pools that a program steps beside it, and a short list gains nothing by more
// than a block per 64 records: us per cycle of a lone 32^3 domain (1.6e3 records) 9.1 on all blocks and 8.9 on a
// quarter, 48^3 (4.2e3) 9.3 and 9.2 on half, 64^3 (7.5e3) 9.5 and 9.6. Eight pools of 32^3 stepped from as many
// threads: 7.1 -> 2.7 us per cycle and pool, of 48^3 8.3 -> 6.6. A list grows during a launch, so the rule
// takes short launches only, and a quarter at least: from a few records to 1e5 within 1000 cycles, such
// launches took 20-36 % longer on a quarter of the blocks than on all; of 250 cycles, as long.
constexpr int kShortLaunch = 250;
int Pool::grid_for(int n, int full, bool many) const {
    if (grid_fixed_)
        return std::max(1, full / grid_fixed_);
    if (!list_read_ || n > kShortLaunch)
        return full;
    const unsigned long long least = std::max<unsigned long long>((full + 3) / 4, many ? n_domains_ : 0); // a warp starts a domain
    return (int)std::min<unsigned long long>(full, std::max(last_records_ / 64 + 1, least));
}

// One cooperative launch of k_cycles over n cycles (at most the co-resident blocks).
void Pool::launch_persistent(int n) {
    cudaStream_t st = S(stream_);
    // the meeting point starts at zero arrivals (a launch that gave up waiting may have left some)
    CUDA_OK(cudaMemsetAsync((char *)dstate_ + offsetof(PoolState, meet), 0, sizeof(PoolState::meet), st));
    PoolState *ps = dstate_;
    // the domains still running at the last state read, when few (the one with most cells first);
    // one that ends during the launch is still started and returns at once, as in the spread start
    AliveSet alive{};
    for (int s = 0; s < (int)slots_.size() && alive.n >= 0; s++) {
        if (!slots_[s].used || host_desc_[s].done)
            continue;
        if (alive.n == kSerialDomains) {
            alive.n = -1;
            break;
        }
        alive.idx[alive.n++] = s;
    }
    for (int i = 1; i < alive.n; i++)
        if (host_desc_[alive.idx[i]].active_size > host_desc_[alive.idx[0]].active_size)
            std::swap(alive.idx[0], alive.idx[i]);
    void *args[] = {&ps, &n, &alive};
    const bool fixed =
        trial_ || (config_fixed_ && !(tuned_records_ && last_records_ && last_records_ * 4 < tuned_records_));
    const int v = fixed ? variant_ : shape_for(last_records_);
    const int grid = grid_for(n, std::min(kMeetMaxGrid, grid_cycles_[v]), alive.n < 0);
    // many domains: a round of loads more per cycle for the views, which up to kSerialDomains do not repay
    // (a map of 96: 14.5 -> 15.5 us per cycle with seven running)
    const void *const kernel = alive.n < 0 ? kStepKernel[v].cycles_many : kStepKernel[v].cycles;
    CUDA_OK(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kBlock), args, 0, st));
    launches_ += 1;
    config_cycles_[v] += (unsigned long long)n;
}

// n cycles as separate pass kernels: the start of cycles 2..n runs in the last block of the
// previous capture pass, so a cycle costs three launches.
void Pool::launch_passes(int n) {
    if (n <= 0)
        return;
    cudaStream_t st = S(stream_);
    const StepKernels &K = kStepKernel[variant_];
    k_step_begin<<<1, kBlock, 0, st>>>(dstate_);
    for (int q = 0; q < n; q++) {
        K.grow<<<grid_grow_[variant_], kBlock, 0, st>>>(dstate_);
        k_claim<<<grid_claim_, kBlock, 0, st>>>(dstate_);
        if (q + 1 < n)
            K.capture_begin<<<grid_capture_[variant_], kBlock, 0, st>>>(dstate_);
        else
            K.capture_end<<<grid_capture_[variant_], kBlock, 0, st>>>(dstate_);
    }
    launches_ += 1 + 3ull * n;
}

void Pool::build_graph() {
    if (graph_exec_)
        return;
    graph_steps_ = 50;
    cudaStream_t st = S(stream_);
    cudaGraph_t graph;
    CUDA_OK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    const unsigned long long before = launches_;
    launch_passes(graph_steps_);
    launches_ = before;
    CUDA_OK(cudaStreamEndCapture(st, &graph));
    cudaGraphExec_t ex;
    CUDA_OK(cudaGraphInstantiate(&ex, graph, 0));
    CUDA_OK(cudaGraphDestroy(graph));
    graph_exec_ = ex;
}

void Pool::step(int n) {
    TraceRange trace("exaca step");
    if (n <= 0)
        return;
    cycles_launched_ += (unsigned long long)n;
    CUDA_OK(cudaSetDevice(device_));
    for (int s = 0; s < (int)slots_.size(); s++) {
        // a domain known to have ended executes no further cycle
        if (!slots_[s].used || host_desc_[s].done)
            continue;
        slots_[s].steps_launched += n;
        ensure_growth(s, slots_[s].steps_launched + 1);
    }
    if (step_mode_ == 0) {
        launch_persistent(n);
    }
    else {
        build_graph();
        cudaStream_t st = S(stream_);
        const int full = n / graph_steps_, rest = n % graph_steps_;
        for (int q = 0; q < full; q++)
            CUDA_OK(cudaGraphLaunch((cudaGraphExec_t)graph_exec_, st));
        launches_ += (unsigned long long)full * (1 + 3ull * graph_steps_);
        launch_passes(rest);
        config_cycles_[config()] += (unsigned long long)n;
    }
    CUDA_OK(cudaGetLastError());
}

void Pool::sync_state() {
    CUDA_OK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    if (!host_desc_.empty())
        CUDA_OK(cudaMemcpyAsync(host_desc_.data(), ddesc_, sizeof(DomainDesc) * host_desc_.size(),
                                cudaMemcpyDeviceToHost, st));
    // the list counters (cnt[2], capacity, tombs, cur): the length of the list the next cycle reads
    constexpr size_t kCnt = offsetof(PoolState, cnt), kEnd = offsetof(PoolState, cur) + sizeof(int);
    unsigned char lists[kEnd - kCnt];
    CUDA_OK(cudaMemcpyAsync(lists, (char *)dstate_ + kCnt, sizeof(lists), cudaMemcpyDeviceToHost, st));
    CUDA_OK(cudaStreamSynchronize(st));
    unsigned long long cnt[2];
    int cur;
    std::memcpy(cnt, lists, sizeof(cnt));
    std::memcpy(&cur, lists + (offsetof(PoolState, cur) - kCnt), sizeof(cur));
    last_records_ = cnt[cur & 1];
    list_read_ = true;
}

int Pool::check_bounded_wait() {
    CUDA_OK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    CUDA_OK(cudaMemsetAsync((char *)dstate_ + offsetof(PoolState, meet), 0, sizeof(PoolState::meet), st));
    PoolState *ps = dstate_;
    void *args[] = {&ps};
    CUDA_OK(cudaLaunchCooperativeKernel((const void *)k_meet_probe, dim3(2), dim3(kBlock), args, 0, st));
    launches_ += 1;
    const int flags = pool_error();
    // the pool carries on: no flag and a meeting point with no arrivals
    const int zero = 0;
    CUDA_OK(cudaMemcpyAsync((char *)dstate_ + offsetof(PoolState, error), &zero, sizeof(int), cudaMemcpyHostToDevice,
                            st));
    CUDA_OK(cudaMemsetAsync((char *)dstate_ + offsetof(PoolState, meet), 0, sizeof(PoolState::meet), st));
    CUDA_OK(cudaStreamSynchronize(st));
    return flags;
}

int Pool::pool_error() {
    int e = 0;
    CUDA_OK(cudaMemcpyAsync(&e, (char *)dstate_ + offsetof(PoolState, error), sizeof(int), cudaMemcpyDeviceToHost,
                            S(stream_)));
    CUDA_OK(cudaStreamSynchronize(S(stream_)));
    return e;
}

unsigned long long Pool::list_count() {
    PoolState ps;
    CUDA_OK(cudaMemcpyAsync(&ps, dstate_, sizeof(ps), cudaMemcpyDeviceToHost, S(stream_)));
    CUDA_OK(cudaStreamSynchronize(S(stream_)));
    return ps.cnt[ps.pending];
}

PoolStats Pool::stats() {
    PoolState ps;
    CUDA_OK(cudaMemcpyAsync(&ps, dstate_, sizeof(ps), cudaMemcpyDeviceToHost, S(stream_)));
    CUDA_OK(cudaStreamSynchronize(S(stream_)));
    PoolStats r;
    std::memset(&r, 0, sizeof(r));
    r.cycles = cycles_launched_;
    r.launches = launches_;
    r.h2d_bytes = h2d_bytes_;
    r.d2h_bytes = d2h_bytes_;
    for (int q = 0; q < kStatShards; q++) {
        r.listed += ps.stat[q][kStatListed];
        r.grown += ps.stat[q][kStatGrown];
        r.captured += ps.stat[q][kStatCaptured];
        r.nucleated += ps.stat[q][kStatNucleated];
        r.claims += ps.stat[q][kStatClaims];
        r.row_reads += ps.stat[q][kStatRowReads];
        r.dropped += ps.stat[q][kStatDropped];
        r.fresh += ps.stat[q][kStatFresh];
        r.rechecks += ps.stat[q][kStatRechecks];
        r.flagged += ps.stat[q][kStatFlagged];
    }
    return r;
}

KernelTimes Pool::profile_cycles(int n) {
    CUDA_OK(cudaSetDevice(device_));
    KernelTimes kt;
    if (n <= 0)
        return kt;
    for (int s = 0; s < (int)slots_.size(); s++) {
        if (!slots_[s].used)
            continue;
        slots_[s].steps_launched += n;
        ensure_growth(s, slots_[s].steps_launched + 1);
    }
    cudaStream_t st = S(stream_);
    cudaEvent_t ev[5];
    for (auto &e : ev)
        CUDA_OK(cudaEventCreate(&e));
    for (int q = 0; q < n; q++) {
        CUDA_OK(cudaEventRecord(ev[0], st));
        k_step_begin<<<1, kBlock, 0, st>>>(dstate_);
        CUDA_OK(cudaEventRecord(ev[1], st));
        kStepKernel[variant_].grow<<<grid_grow_[variant_], kBlock, 0, st>>>(dstate_);
        CUDA_OK(cudaEventRecord(ev[2], st));
        k_claim<<<grid_claim_, kBlock, 0, st>>>(dstate_);
        CUDA_OK(cudaEventRecord(ev[3], st));
        kStepKernel[variant_].capture_end<<<grid_capture_[variant_], kBlock, 0, st>>>(dstate_);
        CUDA_OK(cudaEventRecord(ev[4], st));
        CUDA_OK(cudaEventSynchronize(ev[4]));
        float t[4];
        for (int k = 0; k < 4; k++)
            CUDA_OK(cudaEventElapsedTime(&t[k], ev[k], ev[k + 1]));
        kt.begin_ms += t[0];
        kt.grow_ms += t[1];
        kt.claim_ms += t[2];
        kt.capture_ms += t[3];
    }
    CUDA_OK(cudaGetLastError());
    for (auto &e : ev)
        CUDA_OK(cudaEventDestroy(e));
    kt.cycles = n;
    cycles_launched_ += (unsigned long long)n;
    launches_ += 4ull * n;
    return kt;
}

void Pool::profile_persistent(int n, double us[7]) {
    for (int k = 0; k < 7; k++)
        us[k] = 0;
    if (n <= 0)
        return;
    CUDA_OK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    const size_t words = 3 * (3 * (size_t)n + 1);
    unsigned long long *dtl = nullptr;
    CUDA_OK(cudaMalloc(&dtl, words * sizeof(unsigned long long)));
    // first arrivals take the minimum, last arrivals the maximum, departures are stored
    std::vector<unsigned long long> tl(words, 0);
    for (size_t m = 0; m < words; m += 3)
        tl[m] = ULLONG_MAX;
    CUDA_OK(cudaMemcpyAsync(dtl, tl.data(), words * sizeof(unsigned long long), cudaMemcpyHostToDevice, st));
    CUDA_OK(cudaMemcpyAsync((char *)dstate_ + offsetof(PoolState, timeline), &dtl, sizeof(dtl),
                            cudaMemcpyHostToDevice, st));
    step(n);
    unsigned long long *none = nullptr;
    CUDA_OK(cudaMemcpyAsync((char *)dstate_ + offsetof(PoolState, timeline), &none, sizeof(none),
                            cudaMemcpyHostToDevice, st));
    CUDA_OK(cudaMemcpyAsync(tl.data(), dtl, words * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    CUDA_OK(cudaStreamSynchronize(st));
    CUDA_OK(cudaFree(dtl));
    // meeting points 3c+1, 3c+2, 3c+3 close cycle c's growth (with the blocks' own claims), global
    // claim and capture passes; those that a cycle left out were never departed from
    const unsigned long long *prev = &tl[0];
    for (int c = 0; c < n; c++) {
        const unsigned long long *m1 = &tl[3 * (3 * c + 1)], *m2 = &tl[3 * (3 * c + 2)], *m3 = &tl[3 * (3 * c + 3)];
        if (m1[2]) {
            us[0] += (double)(m1[0] - prev[2]);
            us[1] += (double)(m1[1] - prev[2]);
            prev = m1;
        }
        if (m2[2]) {
            us[2] += (double)(m2[0] - prev[2]);
            us[3] += (double)(m2[1] - prev[2]);
            prev = m2;
        }
        if (m3[2]) {
            us[4] += (double)(m3[0] - prev[2]);
            us[5] += (double)(m3[1] - prev[2]);
            us[6] += (double)(m3[2] - m3[1]);
            prev = m3;
        }
    }
    for (int k = 0; k < 7; k++)
        us[k] /= 1e3 * n;
}

void Pool::set_config(int config) {
    apply_config(config);
    config_fixed_ = true;
    tuned_records_ = 0;
}

void Pool::set_grid(int divisor) {
    if (divisor < 0 || divisor > 32)
        throw std::invalid_argument("grid divisor must be 0 (the default rule) or 1-32");
    grid_fixed_ = divisor;
}

void Pool::apply_config(int config) {
    if (config < 0 || config >= kStepConfigs)
        throw std::invalid_argument("step configuration out of range");
    const int mode = config / kStepVariants, variant = config % kStepVariants;
    // the graph holds the pass kernels, which two shapes share
    if (kStepKernel[variant].grow != kStepKernel[variant_].grow && graph_exec_) {
        CUDA_OK(cudaStreamSynchronize(S(stream_)));
        CUDA_OK(cudaGraphExecDestroy((cudaGraphExec_t)graph_exec_));
        graph_exec_ = nullptr;
    }
    step_mode_ = mode;
    variant_ = variant;
}

int Pool::autotune(int trial_cycles, double *ms_per_cycle) {
    // The active list grows from trial to trial. Half of each configuration's cycles are run in this order and
    // half in the reverse, so that each has the same mean place in it (in one pass the first one won
    // whatever it was). Graph shapes that share their kernels are neighbours: three graphs are built.
    constexpr int kOrder[kStepConfigs] = {0, 1, 2, 3, 4, 6, 5, 7};
    struct Trial {
        bool &on;
        explicit Trial(bool &f) : on(f) { on = true; }
        ~Trial() { on = false; }
    };
    double ms[kStepConfigs] = {};
    const int half[2] = {trial_cycles - trial_cycles / 2, trial_cycles / 2};
    {
        const Trial trial(trial_); // every launch takes the configuration that is timed
        for (int k = 0; k < 2 * kStepConfigs; k++) {
            const int c = kOrder[k < kStepConfigs ? k : 2 * kStepConfigs - 1 - k], n = half[k / kStepConfigs];
            if (n == 0)
                continue;
            apply_config(c);
            if (step_mode_ == 1)
                build_graph(); // outside the timed trial
            ms[c] += timed_step(n) / trial_cycles;
        }
    }
    int best = 0;
    for (int c = 0; c < kStepConfigs; c++) {
        if (ms_per_cycle)
            ms_per_cycle[c] = ms[c];
        if (ms[c] < ms[best])
            best = c;
    }
    set_config(best);
    sync_state();
    tuned_records_ = last_records_;
    return best;
}

long long Pool::run_all(int chunk, long long max_cycles) {
    TraceRange trace("exaca run_all");
    if (chunk <= 0)
        throw std::invalid_argument("chunk must be positive");
    long long stepped = 0;
    while (true) {
        sync_state();
        bool all_done = true;
        for (int s = 0; s < (int)slots_.size(); s++) {
            if (!slots_[s].used)
                continue;
            const DomainDesc &d = host_desc_[s];
            if (d.error)
                throw DeviceError("device error flags " + std::to_string(d.error) + " in slot " + std::to_string(s));
            if (!d.check_mode)
                throw std::invalid_argument("slot " + std::to_string(s) + " was admitted without device termination");
            all_done = all_done && d.done;
        }
        const int perr = pool_error();
        if (perr)
            throw DeviceError("pool error flags " + std::to_string(perr));
        if (all_done)
            return stepped;
        if (stepped >= max_cycles)
            throw DeviceError("domains still running after " + std::to_string(stepped) + " cycles");
        step(chunk);
        stepped += chunk;
    }
}

double Pool::timed_step(int n) {
    CUDA_OK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    cudaEvent_t ev[2];
    for (auto &e : ev)
        CUDA_OK(cudaEventCreate(&e));
    CUDA_OK(cudaEventRecord(ev[0], st));
    step(n);
    CUDA_OK(cudaEventRecord(ev[1], st));
    CUDA_OK(cudaEventSynchronize(ev[1]));
    float ms = 0;
    CUDA_OK(cudaEventElapsedTime(&ms, ev[0], ev[1]));
    for (auto &e : ev)
        CUDA_OK(cudaEventDestroy(e));
    return ms;
}

long long Pool::liquid(int slot) const {
    const DomainDesc &d = host_desc_.at(slot);
    long long v = d.liquid;
    for (int q = 0; q < kLiquidShards; q++)
        v += d.liquid_shard[q];
    return v;
}

Census Pool::census(int slot) {
    CUDA_OK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    Census init;
    std::memset(&init, 0, sizeof(init));
    init.next_cts = ULLONG_MAX;
    CUDA_OK(cudaMemcpyAsync(census_buf_, &init, sizeof(init), cudaMemcpyHostToDevice, st));
    k_census<<<num_sms_ * 4, 256, 0, st>>>(ddesc_ + slot, (Census *)census_buf_);
    CUDA_OK(cudaGetLastError());
    Census out;
    CUDA_OK(cudaMemcpyAsync(&out, census_buf_, sizeof(out), cudaMemcpyDeviceToHost, st));
    CUDA_OK(cudaStreamSynchronize(st));
    return out;
}

void Pool::set_cycle(int slot, int cycle) {
    sync_state();
    DomainDesc &h = host_desc_[slot];
    if (cycle > h.cycle) {
        if (h.n_jumps >= kMaxJumps)
            throw Unsupported("too many cycle jumps");
        h.jump_lo[h.n_jumps] = h.cycle;
        h.jump_hi[h.n_jumps] = cycle;
        h.n_jumps++;
    }
    h.cycle = cycle;
    // only this slot's dynamic fields change; nothing else is in flight on the stream
    push_desc(slot);
}

void Pool::next_layer(int slot, std::string &log) {
    TraceRange trace("exaca next_layer");
    // src/runCA.cpp:344-405: DomainShiftAndResize, then LayerSetup on the moved window
    CUDA_OK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    sync_state();
    DomainDesc d = host_desc_.at(slot);
    if (d.layer_no + 1 >= d.n_layers || !d.nu_base)
        throw std::logic_error("next_layer: the slot has no further layer");
    const unsigned blocks = (unsigned)num_sms_ * 4;
    k_layer_base<<<blocks, 256, 0, st>>>(ddesc_ + slot);
    CUDA_OK(cudaGetLastError());
    int bounds[2] = {INT_MAX, INT_MIN};
    int *dbounds = nullptr;
    CUDA_OK(cudaMalloc(&dbounds, sizeof(bounds)));
    CUDA_OK(cudaMemcpyAsync(dbounds, bounds, sizeof(bounds), cudaMemcpyHostToDevice, st));
    k_layer_bounds<<<blocks, 256, 0, st>>>(ddesc_ + slot, d.layer_no + 1, dbounds);
    CUDA_OK(cudaGetLastError());
    CUDA_OK(cudaMemcpyAsync(bounds, dbounds, sizeof(bounds), cudaMemcpyDeviceToHost, st));
    CUDA_OK(cudaStreamSynchronize(st));
    CUDA_OK(cudaFree(dbounds));
    // the new bottom is one plane below the lowest active cell, the new top the highest cell of the
    // next layer (src/CAinitialize.cpp:2776-2820)
    if (bounds[0] == INT_MAX || bounds[1] == INT_MIN || bounds[0] - 1 > bounds[1] || bounds[1] >= d.nz)
        throw DeviceError("layer change: no active cell or no cell of the next layer");
    const int z_lo = bounds[0] - 1, z_hi = bounds[1];
    std::ostringstream s;
    s << "New domain bottom at Z = " << z_lo << ", a shift of " << z_lo - d.z_lo << " cells\n";
    s << "New domain top at Z = " << z_hi << "\n";
    s << "New active domain height is " << z_hi - z_lo + 1 << "\n";
    s << "Resize executed\n";
    d.layer_no += 1;
    d.z_lo = z_lo;
    d.z_end = z_hi + 1;
    d.nz_active = z_hi - z_lo + 1;
    d.zbound_high = z_hi;
    d.cycle = 0;
    d.nuc_cursor = 0;
    d.nn = 0;
    d.n_jumps = 0;
    host_desc_[slot] = d;
    push_desc(slot);
    k_layer_gate<<<blocks, 256, 0, st>>>(ddesc_ + slot);
    CUDA_OK(cudaGetLastError());
    // LayerSetup: the records of the ended layer leave the list (re-labelled to the pool's finished
    // placeholder domain, dropped by the next growth pass); the window's octahedron arrays start from
    // zero (src/CAinitialize.cpp:2850-2852); every active cell of the new window gets a fresh
    // octahedron and a record
    k_drop_domain<<<num_sms_ * 2, 256, 0, st>>>(dstate_, (unsigned)slot, (unsigned)max_domains_);
    CUDA_OK(cudaGetLastError());
    CUDA_OK(cudaMemsetAsync(d.pos, 0xff, (size_t)d.active_size * 4, st));
    {
        const size_t plane = (size_t)d.mx * d.my, o = plane * d.z_lo, n = plane * (d.z_end - d.z_lo);
        CUDA_OK(cudaMemsetAsync(d.dl + o, 0, n * 4, st));
        CUDA_OK(cudaMemsetAsync(d.doc + 3 * o, 0, n * 12, st));
        CUDA_OK(cudaMemsetAsync(d.cdl + 26 * o, 0, n * 104, st));
    }
    k_init_active<<<num_sms_ * 4, 256, 0, st>>>(dstate_, slot, -1);
    CUDA_OK(cudaGetLastError());
    s << "New layer setup, GN dimensions are " << d.mx << " " << 0 << " " << d.nz_active << "\n";
    s << "New layer ghost nodes initialized\n";
    log += s.str();
}

void Pool::copy_out_raw(int slot, int32_t *grain_id, int8_t *cell_type) {
    CUDA_OK(cudaSetDevice(device_));
    const DomainDesc &d = host_desc_.at(slot);
    size_t N = slots_.at(slot).problem->g.domain_size;
    cudaStream_t st = S(stream_);
    to_host({{grain_id, d.gid, N * 4, false}, {cell_type, d.ctype, N, false}}, stream_);
    d2h_bytes_ += (grain_id ? N * 4 : 0) + (cell_type ? N : 0);
    CUDA_OK(cudaStreamSynchronize(st));
}

void Pool::flush_records() {
    CUDA_OK(cudaSetDevice(device_));
    k_flush_records<<<num_sms_ * 2, 256, 0, S(stream_)>>>(dstate_);
    CUDA_OK(cudaGetLastError());
    CUDA_OK(cudaStreamSynchronize(S(stream_)));
}

void Pool::copy_octahedra(int slot, float *dl, float *doc, float *cdl) {
    flush_records();
    const DomainDesc &d = host_desc_.at(slot);
    // the current layer's window (the whole allocation's prefix for single-layer problems)
    const size_t plane = (size_t)d.mx * d.my, o = plane * d.z_lo, A = plane * (d.z_end - d.z_lo);
    cudaStream_t st = S(stream_);
    to_host({{dl, d.dl + o, A * 4, false}, {doc, d.doc + 3 * o, A * 12, false}, {cdl, d.cdl + 26 * o, A * 104, false}},
            stream_);
    d2h_bytes_ += (dl ? A * 4 : 0) + (doc ? A * 12 : 0) + (cdl ? A * 104 : 0);
    CUDA_OK(cudaStreamSynchronize(st));
}

void Pool::copy_out(int slot, int32_t *grain_id, int32_t *cell_type) {
    TraceRange trace("exaca copy_out");
    if (!cell_type) {
        copy_out_raw(slot, grain_id, nullptr);
        return;
    }
    // CellType is widened to int32 on the device (in stream order after the cycles); both fields
    // then go to the caller's buffers as one DMA each when those are page-locked, else through the
    // pinned staging pieces
    CUDA_OK(cudaSetDevice(device_));
    const DomainDesc &d = host_desc_.at(slot);
    const size_t N = slots_.at(slot).problem->g.domain_size;
    cudaStream_t st = S(stream_);
    int32_t *wide = nullptr;
    CUDA_OK(cudaMallocAsync((void **)&wide, std::max<size_t>(N * 4, 16), st));
    const unsigned blocks = (unsigned)std::min<size_t>((N + 255) / 256, (size_t)num_sms_ * 16);
    k_widen_types<<<blocks, 256, 0, st>>>(d.ctype, wide, (long long)N);
    CUDA_OK(cudaGetLastError());
    to_host({{grain_id, d.gid, N * 4, false}, {cell_type, wide, N * 4, false}}, stream_);
    CUDA_OK(cudaFreeAsync(wide, st));
    CUDA_OK(cudaStreamSynchronize(st));
    d2h_bytes_ += (grain_id ? N * 4 : 0) + N * 4;
}

void Pool::copy_out_concurrent(int slot, int32_t *grain_id, int32_t *cell_type) {
    TraceRange trace("exaca copy_out_concurrent");
    CUDA_OK(cudaSetDevice(device_));
    const SlotHost &s = slots_.at(slot);
    const DomainDesc &d = host_desc_.at(slot);
    if (!s.used || !(d.done || s.finished))
        throw std::invalid_argument("copy_out_concurrent: the slot's domain has not ended");
    if (!copy_stream_) {
        cudaStream_t cs;
        CUDA_OK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        copy_stream_ = cs;
    }
    // The domain's GrainID and CellType are final (an ended domain's records only leave the list),
    // and the host saw that state, so the copies need no ordering against the pool stream. Copy
    // engines only: no kernel runs beside the persistent cooperative one.
    // CellType is widened on the host as it leaves the staging pieces.
    cudaStream_t cs = S(copy_stream_);
    const size_t N = s.problem->g.domain_size;
    to_host({{grain_id, d.gid, N * 4, false}, {cell_type, d.ctype, N, true}}, copy_stream_);
    CUDA_OK(cudaStreamSynchronize(cs));
    d2h_bytes_ += (grain_id ? N * 4 : 0) + (cell_type ? N : 0);
}

int Pool::run_plain(int slot, std::string &log, double *nucl_s, double *capture_s) {
    TraceRange trace("exaca run_plain");
    // src/runCA.cpp:282-411: the layer loop, each layer's cycles until no liquid of the layer is left
    const Problem &p = *slots_.at(slot).problem;
    const bool type_r = p.cfg.simulation_type == "R";
    const bool jump_type = p.cfg.simulation_type == "S" || type_r;
    auto t0 = std::chrono::steady_clock::now();
    auto t_layer = t0;
    cudaEvent_t ev0, ev1;
    CUDA_OK(cudaEventCreate(&ev0));
    CUDA_OK(cudaEventCreate(&ev1));
    CUDA_OK(cudaEventRecord(ev0, S(stream_)));
    sync_state();
    int cycle = host_desc_[slot].cycle;
    while (true) {
        int n = 1000 - (cycle % 1000);
        if (!config_fixed_ && cycle == 0) {
            // a layer's list grows from its initial front: its length is read, and with it the launch
            // shape chosen, every 250 cycles of the first 1000
            for (; n > 250; n -= 250) {
                step(250);
                sync_state();
            }
        }
        step(n);
        sync_state();
        const DomainDesc &d = host_desc_[slot];
        int perr = pool_error();
        if (d.error || perr) {
            std::ostringstream e;
            e << "device error flags: domain " << d.error << " pool " << perr;
            throw DeviceError(e.str());
        }
        cycle = d.cycle;
        Census c = census(slot);
        std::ostringstream s;
        s << "cycle = " << cycle << " Superheated liquid cells = " << c.superheated
          << " Undercooled liquid cells = " << c.undercooled << " Number of nucleation events this layer " << d.nn
          << " Remaining liquid cells in future layers of this simulation = " << c.remaining << "\n";
        log += s.str();
        bool xswitch = c.superheated + c.undercooled == 0;
        if (!xswitch && jump_type && c.undercooled == 0) {
            unsigned long long next = c.next_cts;
            if ((next - (unsigned long long)(long long)cycle) > 5000) {
                int nc = (int)(next - 1);
                set_cycle(slot, nc);
                cycle = nc;
                log += "Jumping to cycle " + std::to_string(cycle + 1) + "\n";
            }
            // type R ends a layer at its finish time step (src/CAupdate.cpp:818-819)
            if (type_r && cycle >= p.finish_time_step.at(d.layer_no))
                xswitch = true;
        }
        if (xswitch) {
            if (d.layer_no + 1 >= d.n_layers)
                break;
            const int layer = d.layer_no;
            next_layer(slot, log);
            double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_layer).count();
            t_layer = std::chrono::steady_clock::now();
            std::ostringstream s2;
            s2 << "Time for layer number " << layer << " was " << secs << " s, starting layer " << layer + 1 << "\n";
            log += s2.str();
            cycle = 0;
            continue;
        }
    }
    CUDA_OK(cudaEventRecord(ev1, S(stream_)));
    CUDA_OK(cudaEventSynchronize(ev1));
    float ms = 0;
    CUDA_OK(cudaEventElapsedTime(&ms, ev0, ev1));
    last_run_ms_ = ms;
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (nucl_s)
        *nucl_s = 0.0;
    if (capture_s)
        *capture_s = secs;
    slots_[slot].finished = true;
    return cycle;
}

// ---------------------------------------------------------------------------------------------
// Grain statistics (analysis/src/GAprint.cpp:17-198) on the device: per region cell, melted count,
// misorientation of its grain's orientation to +Z (table built on the host with the reference's
// libm acos), its 1-degree histogram, nucleated cells, GrainID range; then distinct GrainIDs via a
// bitmap over that range.
struct GrainAcc {
    unsigned long long melted, nucleated, top_melted;
    double mis, mis_top;
    unsigned long long hist[kMisorientationBins];
    unsigned long long grains;
    int gmin, gmax;
};

struct Region {
    int x0, x1, y0, y1, z0, z1, mx, my, nz;
};

// A row of the region (fixed z and x) per warp at a time, consecutive lanes on consecutive cells: one
// division per row instead of four 64-bit ones per cell. Neighbouring cells mostly belong to one grain, so
// their lanes share a histogram bin and a bitmap bit: the bin is counted once per set of lanes (with an
// atomic per cell the lanes of a warp queued on one word), the bit set by lanes whose left neighbour has
// another grain, where it is not set already. melted null: a type-C problem, where every cell off the
// bottom and top planes and the ghost ring (outside any region) is melted. bits null: gmin / gmax only
// (the bitmap's range is not known yet), as codes of which gmin holds the complement (both start at zero).
// 192 x 160 x 128: the call takes 0.12 ms (a launch, a memset and two copies are most of it) instead of 4.5
// with four divisions and an atomic per cell, a table of arc cosines made per call and the melted flags uploaded.
__device__ __forceinline__ unsigned int grain_code(int g) { return (unsigned int)g ^ 0x80000000u; } // ordered as g

__global__ void __launch_bounds__(256) k_grain_region(const int32_t *gid, const int8_t *melted, const float *mis, Region R,
                                                      GrainAcc *acc, unsigned long long *bits, int bits_min,
                                                      long long n_bits) {
    __shared__ unsigned int s_hist[kMisorientationBins];
    for (int b = threadIdx.x; b < kMisorientationBins; b += blockDim.x)
        s_hist[b] = 0;
    __syncthreads();
    const unsigned int lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    unsigned long long m = 0, nuc = 0, top = 0;
    double ms = 0, mt = 0;
    unsigned int cmin = 0xffffffffu, cmax = 0;
    const unsigned int nxr = (unsigned int)(R.x1 - R.x0 + 1), rows = nxr * (unsigned int)(R.z1 - R.z0 + 1);
    const int nyr = R.y1 - R.y0 + 1;
    for (unsigned int row = blockIdx.x * 8u + threadIdx.x / 32; row < rows; row += gridDim.x * 8u) {
        const unsigned int kz = row / nxr;
        const int k = (int)kz + R.z0, i = (int)(row - kz * nxr) + R.x0;
        const long long c0 = ((long long)k * R.mx + (i + 1)) * R.my + (R.y0 + 1);
        const bool plane_melted = k != 0 && k != R.nz - 1;
        for (int j0 = 0; j0 < nyr; j0 += 32) {
            const bool in = j0 + (int)lane < nyr;
            const int g = in ? __ldcs(gid + c0 + j0 + lane) : 0;
            const bool melt = in && (melted ? __ldcs(melted + c0 + j0 + lane) == 1 : plane_melted);
            if (in) {
                const unsigned int code = grain_code(g);
                cmin = min(cmin, code);
                cmax = max(cmax, code);
                nuc += g < 0;
            }
            int bin = -1;
            if (melt) {
                int ori = (abs(g) - 1) % 10000;
                if (ori < 0)
                    ori += 10000;
                const float a = __ldg(mis + ori);
                m++;
                ms += a;
                bin = min((int)a, kMisorientationBins - 1);
                if (k == R.z1) {
                    top++;
                    mt += a;
                }
            }
            const unsigned int same = __match_any_sync(0xffffffffu, bin);
            if (bin >= 0 && (same & below) == 0)
                atomicAdd(&s_hist[bin], (unsigned int)__popc(same));
            if (bits) {
                const int left = __shfl_up_sync(0xffffffffu, g, 1);
                const long long off = (long long)g - bits_min;
                if (in && (lane == 0 || left != g) && off >= 0 && off < n_bits) {
                    const unsigned long long bit = 1ull << (off & 63);
                    if (!(bits[off >> 6] & bit))
                        atomicOr(bits + (off >> 6), bit);
                }
            }
        }
    }
    for (int o = 16; o; o >>= 1) {
        m += __shfl_down_sync(0xffffffffu, m, o);
        nuc += __shfl_down_sync(0xffffffffu, nuc, o);
        top += __shfl_down_sync(0xffffffffu, top, o);
        ms += __shfl_down_sync(0xffffffffu, ms, o);
        mt += __shfl_down_sync(0xffffffffu, mt, o);
    }
    cmin = __reduce_min_sync(0xffffffffu, cmin);
    cmax = __reduce_max_sync(0xffffffffu, cmax);
    if (lane == 0) {
        if (m)
            atomicAdd(&acc->melted, m);
        if (nuc)
            atomicAdd(&acc->nucleated, nuc);
        if (top)
            atomicAdd(&acc->top_melted, top);
        if (ms != 0)
            atomicAdd(&acc->mis, ms);
        if (mt != 0)
            atomicAdd(&acc->mis_top, mt);
        if (cmin <= cmax) {
            // both start at zero: the minimum as the maximum of its complement
            atomicMax((unsigned int *)&acc->gmin, ~cmin);
            atomicMax((unsigned int *)&acc->gmax, cmax);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < kMisorientationBins; b += blockDim.x)
        if (s_hist[b])
            atomicAdd(&acc->hist[b], (unsigned long long)s_hist[b]);
}

__global__ void k_grain_bits(const int32_t *gid, Region R, int gmin, unsigned long long *bits) {
    const unsigned int lane = threadIdx.x & 31;
    const unsigned int nxr = (unsigned int)(R.x1 - R.x0 + 1), rows = nxr * (unsigned int)(R.z1 - R.z0 + 1);
    const int nyr = R.y1 - R.y0 + 1;
    for (unsigned int row = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; row < rows;
         row += gridDim.x * (blockDim.x / 32)) {
        const unsigned int kz = row / nxr;
        const long long c0 =
            ((long long)((int)kz + R.z0) * R.mx + ((int)(row - kz * nxr) + R.x0 + 1)) * R.my + (R.y0 + 1);
        for (int j = (int)lane; j < nyr; j += 32) {
            const long long off = (long long)gid[c0 + j] - gmin;
            const unsigned long long bit = 1ull << (off & 63);
            if (!(bits[off >> 6] & bit))
                atomicOr(bits + (off >> 6), bit);
        }
    }
}

__global__ void k_popcount(const unsigned long long *bits, long long nwords, unsigned long long *count) {
    unsigned long long c = 0;
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += (long long)gridDim.x * blockDim.x)
        c += __popcll(bits[w]);
    for (int o = 16; o; o >>= 1)
        c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c)
        atomicAdd(count, c);
}

GrainStats Pool::grain_stats(int slot, const int *region) {
    CUDA_OK(cudaSetDevice(device_));
    if (!slot_used(slot))
        throw std::invalid_argument("bad slot");
    const Problem &p = *slots_[slot].problem;
    const Geometry &g = p.g;
    Region R;
    if (region) {
        R.x0 = region[0], R.x1 = region[1], R.y0 = region[2], R.y1 = region[3], R.z0 = region[4], R.z1 = region[5];
    }
    else {
        R.x0 = 1, R.x1 = g.nx - 2, R.y0 = 1, R.y1 = g.ny - 2, R.z0 = 1, R.z1 = g.nz - 2;
    }
    if (R.x0 < 0 || R.x1 >= g.nx || R.y0 < 0 || R.y1 >= g.ny || R.z0 < 0 || R.z1 >= g.nz || R.x0 > R.x1 ||
        R.y0 > R.y1 || R.z0 > R.z1)
        throw std::invalid_argument("region outside the domain");
    R.mx = g.mx;
    R.my = g.my;
    R.nz = g.nz;
    tables_for(p);
    DeviceTables &tb = tables_.at(p.cfg.orientation_file);
    if (!tb.mis) {
        // per-orientation misorientation to +Z with the reference's expression (GAprint.cpp:38-46)
        std::vector<float> mis(kNumOrientations);
        for (int n = 0; n < kNumOrientations; n++) {
            double amin = 62.7;
            for (int ll = 0; ll < 3; ll++) {
                // double acos of the float component, as the reference's unqualified call on a float
                double a = std::abs((180 / M_PI) * std::acos((double)p.guv[9 * n + 3 * ll + 2]));
                if (a < amin)
                    amin = a;
            }
            mis[n] = (float)amin;
        }
        float *d = nullptr;
        CUDA_OK(cudaMalloc(&d, mis.size() * sizeof(float)));
        // on the stream of the kernels that read it (tables_for); kept only once it is filled
        const cudaError_t filled =
            cudaMemcpyAsync(d, mis.data(), mis.size() * sizeof(float), cudaMemcpyHostToDevice, S(stream_));
        if (filled != cudaSuccess)
            cudaFree(d);
        CUDA_OK(filled);
        tb.mis = d;
    }
    cudaStream_t st = S(stream_);
    const size_t N = g.domain_size;
    // a type-C domain's grains are its seeds and nuclei (and 0), its melted cells those off the walls: one
    // pass; otherwise the melted flags are uploaded and a second pass marks the grains between the first's
    // smallest and largest
    const bool known = p.dir.used;
    long long gmin = -(long long)p.nuclei_loc.size(), gmax = known ? (long long)p.dir.active.size() : 0;
    GrainStats out;
    GrainAcc acc;
    char *work = nullptr; // freed in stream order
    try {
        const int32_t *gid = host_desc_[slot].gid;
        const auto words = [](long long lo, long long hi) { return (size_t)((hi - lo + 64) / 64); };
        const size_t nwords = known ? words(gmin, gmax) : 0, flags = known ? 0 : (N + 15) / 16 * 16;
        constexpr size_t kAccBytes = (sizeof(GrainAcc) + 255) / 256 * 256;
        CUDA_OK(cudaMallocAsync((void **)&work, kAccBytes + nwords * 8 + flags, st));
        GrainAcc *dacc = (GrainAcc *)work;
        unsigned long long *bits = (unsigned long long *)(work + kAccBytes);
        int8_t *dmel = (int8_t *)(work + kAccBytes + nwords * 8);
        CUDA_OK(cudaMemsetAsync(work, 0, kAccBytes + nwords * 8, st));
        if (!known)
            CUDA_OK(cudaMemcpyAsync(dmel, p.melted.data(), N, cudaMemcpyHostToDevice, st));
        k_grain_region<<<num_sms_ * 8, 256, 0, st>>>(gid, known ? nullptr : dmel, tb.mis, R, dacc, known ? bits : nullptr,
                                                     (int)gmin, (long long)nwords * 64);
        CUDA_OK(cudaGetLastError());
        if (known)
            k_popcount<<<32, 256, 0, st>>>(bits, (long long)nwords, &dacc->grains);
        CUDA_OK(cudaGetLastError());
        CUDA_OK(cudaMemcpyAsync(&acc, dacc, sizeof(acc), cudaMemcpyDeviceToHost, st));
        CUDA_OK(cudaStreamSynchronize(st));
        const long long seen_min = (long long)(int)(~(unsigned int)acc.gmin ^ 0x80000000u),
                        seen_max = (long long)(int)((unsigned int)acc.gmax ^ 0x80000000u);
        if (!known || seen_min < gmin || seen_max > gmax) {
            gmin = seen_min;
            gmax = seen_max;
            CUDA_OK(cudaMemsetAsync(&dacc->grains, 0, sizeof(dacc->grains), st));
            const size_t nw = words(gmin, gmax);
            unsigned long long *more = nullptr;
            CUDA_OK(cudaMallocAsync((void **)&more, nw * 8, st));
            cudaMemsetAsync(more, 0, nw * 8, st);
            k_grain_bits<<<num_sms_ * 8, 256, 0, st>>>(gid, R, (int)gmin, more);
            k_popcount<<<32, 256, 0, st>>>(more, (long long)nw, &dacc->grains);
            const cudaError_t launched = cudaGetLastError();
            CUDA_OK(cudaFreeAsync(more, st));
            CUDA_OK(launched);
            CUDA_OK(cudaMemcpyAsync(&acc.grains, &dacc->grains, sizeof(acc.grains), cudaMemcpyDeviceToHost, st));
            CUDA_OK(cudaStreamSynchronize(st));
        }
    }
    catch (...) {
        if (work)
            cudaFreeAsync(work, st);
        throw;
    }
    CUDA_OK(cudaFreeAsync(work, st));
    out.region_cells = (long long)(R.x1 - R.x0 + 1) * (R.y1 - R.y0 + 1) * (R.z1 - R.z0 + 1);
    out.melted_cells = (long long)acc.melted;
    out.nucleated_cells = (long long)acc.nucleated;
    out.top_melted = (long long)acc.top_melted;
    out.n_grains = (long long)acc.grains;
    out.misorientation_sum = acc.mis;
    out.misorientation_top_sum = acc.mis_top;
    out.deltax = p.cfg.deltax;
    for (int b = 0; b < kMisorientationBins; b++)
        out.hist[b] = (long long)acc.hist[b];
    return out;
}

} // namespace exaca
