// Wide-batch Brandes searches (sm_100a): 16 or 32 sources a job, for graphs
// whose searches are a few levels deep.
//
// What bounds it.  On a small-diameter graph nearly every vertex is in the
// frontier of some source of a batch at the two or three middle levels, so a
// level is a sparse-matrix times dense-matrix product: every vertex adds the
// 16 (32) values of each neighbour.  The rows are gathered from L2, and an SM
// takes in 64 bytes a clock from there.  So the design is about bytes per
// (edge, source) and about whole rows per request:
//   - 16 (32) sources share a row: 64 (128) bytes of 32-bit path counts
//     forward, 128 (256) of doubles backward, no level words in between.  A row holds the
//     value of the slots that sit exactly at the level being read and 0 in
//     the others, so a gather needs no test per slot: 4 lanes take a row with
//     one or two 16- or 32-byte loads each and add.  (Measured on an R-MAT graph of
//     31 M entries: 141 us and 201 us a pass, 14 and 20 TB/s out of L2, the
//     whole port; the 64-byte rows of levels and values of sweep.cu carry 6
//     sources and take about 500 us.)  The sweeps here reach 300 to 400 us:
//     what is left is the latency of ids, bits and rows (a warp waits half of
//     its time for a load and a fifth at the sweeps' ends; 0.27 instructions a
//     cycle and scheduler, the L2 28 % busy, hit rate 77 %).  32 sources a job
//     share what is not rows: 1,590 us a job of 16 and 2,690 us one of 32 on
//     the benchmark's graph, in the order given.
//   - a bit per vertex and level says whether any slot sits there, so a
//     gather skips the rows of other vertices, rows are never cleared, and
//     backward sweeps visit a level's vertices only.
//   - path counts are 64-bit; the 32-bit rows are used while every count of
//     the level is below 2^28 (the sweep that finds them says so), and otherwise the
//     sweep reads levels and 64-bit counts (kFwdFull), with overflow checked.
//   - level 1, whose counts are 1, is a word of bits a vertex (kFwdOnes).
// All forward sweeps pull: no atomics on values, sums in a fixed order.
//
// Work split.  Vertices are numbered by descending degree class
// (wide_form.cu).  A vertex of few entries (up to 32, or up to 256 where a warp
// has much to do) is taken by four lanes, eight vertices of like degree a
// warp; a heavier one by a warp, its edges dealt to the eight groups of four
// lanes; the heaviest in chunks of 256 to 2,048 entries by one warp each, whose
// sums meet in a buffer and are added in a fixed order by the chunk that
// arrives last.  Warps draw items from a counter in shared memory, heaviest
// first.
//
// Teams.  The CTAs of the launch are cut into teams; a team runs one job at
// a time on state of its own, with a barrier over its own CTAs only, and
// draws its next job from a counter.  On a small graph a team is one CTA and
// the barrier is __syncthreads; on a large one the team is the whole grid.
// Every job writes its dependencies to its own vector, and k_wide_reduce
// adds the vectors in job order, so the result does not depend on which team
// ran a job, nor on what else ran.
//
// Coherence.  Levels and counts are read with .cg loads.  The bitmaps and rows
// are read through L1: they are written in one sweep and read in later ones,
// and the barrier's acquire and fences order the two.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "bcg_common.hpp"
#include "engine_internal.hpp"
#include "wide.cuh"

namespace bcg {

namespace {

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kNone = 0xffffffffu;
constexpr uint32_t kUnseen = 0xFFu;  // level byte of a vertex not reached yet
constexpr uint32_t kEmpty = 0xFEu;   // level byte of a slot without a source
constexpr double kWide32 = 1.5;      // time of a 32-source job's entries over a 16-source job's

// What a sweep does: forward over 32-bit rows, forward over levels and
// 64-bit counts, backward, backward at the deepest level (no child exists),
// forward from level 1 where every count is 1.
enum : int { kFwd32 = 0, kFwdFull = 1, kBack = 2, kBackLast = 3, kFwdOnes = 4 };

struct WideCtx {
    uint32_t T, rank;  // CTAs of the team, this one's place
    unsigned char *lvl;
    uint32_t *done, *act;  // bitmaps: all slots reached; by level: some slot at it
    uint32_t *bits;        // by vertex: the slots that are at level 1 (of vertices where some slot is)
    size_t words;
    unsigned long long *sig;
    unsigned char *g0;  // rows of even levels,
    ptrdiff_t g01;      // and how far behind them the odd levels' are
    unsigned long long *part;
    uint32_t *hcnt;
    double *bc;
};

// The rows of level d.
__device__ __forceinline__ unsigned char *rows_of(const WideCtx &x, uint32_t d) { return x.g0 + ((d & 1u) ? x.g01 : 0); }

// What follows from a job's number of slots NS (16 or 32): a lane holds LS of
// them, in a group of four lanes that takes a row together.
template <int NS>
struct Slots {
    static constexpr int LS = NS / 4;
    static constexpr int kLevels = LS / 4;    // words of a lane's levels
    static constexpr int kRow32 = NS * 4;     // bytes of a row of counts,
    static constexpr int kRow64 = NS * 8;     // of a row of doubles
};

template <int NS>
struct WideSmem {
    WideSub sub;
    WideCtx x;
    uint32_t roots[NS];
    double mult[NS];
    uint32_t nmed;      // end of the vertices a warp takes alone (WideSub::nmed by degree bound)
    uint32_t far;       // lists are brought to L2 ahead (kWideFar)
    uint32_t next;      // items drawn in the current sweep
    uint32_t found;     // this CTA's part of WideTeam::any
    uint32_t any;       // the team's, after the barrier
    unsigned long long count;   // this CTA's part of WideTeam::count
    uint32_t met[kWideLevels];  // vertices that some slot holds at a level, at most
    uint32_t left;              // vertices that some slot has not reached
    int ok;
    uint32_t edges[NS + 1];             // entries of the sources before each
    unsigned long long reach[3 * NS];   // this CTA's part of the sources' totals
    unsigned char list[kWideWarps][32];
};

__device__ __forceinline__ unsigned long long wide_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void ld32(const void *p, uint32_t (&w)[8]) {
    asm volatile("ld.global.cg.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "l"(p));
}
__device__ __forceinline__ void st32(void *p, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.u32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "l"(p)
                 : "memory");
}
// A lane's part of row u of doubles, or of 32-bit counts.  Not volatile: rows
// do not change during the sweep that reads them, so the loads may move.
// Through L1, which keeps the row of zeros that stands for ids to be left out:
// no load or add needs a test.  Except for the doubles of 32 slots, where a row
// of zeros costs as much as another (its 256 bytes go through the register
// port all the same) and the rows drive the bitmaps out of L1: they are tested
// and read past it.  (Benchmark's graph, the two large forward sweeps of a job
// of 32: 377 and 493 us tested, 347 and 415 us with zeros; the two large
// backward ones 437 and 664 us tested, 608 and 745 us with zeros.  4M-vertex
// graph, job of 16, forward 1,442 -> 1,040 us, backward 1,702 -> 1,425 us.)
template <int N>
__device__ __forceinline__ void ld_row(uint32_t u, uint32_t zero, const unsigned char *rows, double (&r)[N]) {
    if constexpr (N == 4) {
        asm("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
            : "=d"(r[0]), "=d"(r[1]), "=d"(r[2]), "=d"(r[3])
            : "l"(rows + (size_t)u * 128));
    } else {
#pragma unroll
        for (int k = 0; k < N; ++k) r[k] = 0.0;
        if (u != zero) {
#pragma unroll
            for (int k = 0; k < N; k += 4)
                asm("ld.global.cg.v4.f64 {%0,%1,%2,%3}, [%4];"
                    : "=d"(r[k]), "=d"(r[k + 1]), "=d"(r[k + 2]), "=d"(r[k + 3])
                    : "l"(rows + (size_t)u * 256 + 8 * k));
        }
    }
}
template <int N>
__device__ __forceinline__ void ld_row(uint32_t u, uint32_t, const unsigned char *rows, uint32_t (&r)[N]) {
    if constexpr (N == 4)
        asm("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
            : "l"(rows + (size_t)u * 64));
    else
        asm("ld.global.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
            : "l"(rows + (size_t)u * 128));
}
// An adjacency entry: streamed, so evicted before the rows.
__device__ __forceinline__ uint32_t ld_adj(const uint32_t *p, unsigned long long pol) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ bool wide_stopped(const WideCtrl *c) {
    const volatile int *p = &c->error;
    return p[0] | p[1] | p[2];
}

// Barrier of a team: one arrival per CTA on the team's counter.  Returns
// false when any CTA of the launch recorded an error; a waiting CTA sees that
// too, so nobody waits for one that has left.
template <int NS>
__device__ bool team_sync(const WideArgs &a, const WideCtx &x, WideTeam *t, WideSmem<NS> &sm, uint32_t slot,
                          uint32_t level = 0) {
    __syncthreads();
    if (threadIdx.x == 0) {
        bool ok = true;
        uint32_t any = sm.found;
        unsigned long long met = sm.count;
        if (x.T > 1) {
            if (slot < 4) {
                if (any) atomicOr(&t->any[slot], any);
                if (met) atomicAdd(&t->count[slot], met);
            }
            __threadfence();
            const unsigned long long arrived = atomicAdd(&t->arrived, 1ull) + 1ull;
            const unsigned long long target = (arrived + x.T - 1) / x.T * x.T;
            if (arrived != target) {
                const unsigned long long t0 = wide_ns();
                uint32_t spins = 0;
                for (;;) {
                    unsigned long long v;
                    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&t->arrived) : "memory");
                    if (v >= target) break;
                    if ((++spins & 63u) == 0) {
                        if (wide_stopped(a.ctrl)) break;
                        if (wide_ns() - t0 > kDefaultWaitNs) {
                            atomicCAS(&a.ctrl->error, 0, BCG_ERR_TIMEOUT);
                            if (a.poison) *a.poison = 1;
                            break;
                        }
                    }
                }
            }
            __threadfence();
            if (slot < 4) {
                any = *reinterpret_cast<volatile uint32_t *>(&t->any[slot]);
                met = *reinterpret_cast<volatile unsigned long long *>(&t->count[slot]);
            }
            ok = !wide_stopped(a.ctrl);
        } else {
            __threadfence();
            if (slot == 5) ok = !wide_stopped(a.ctrl);  // a team of one looks once a job
        }
        sm.next = 0;
        sm.found = 0;
        sm.count = 0;
        sm.any = any;
        if (slot < 4) {
            sm.met[level] = (uint32_t)met;
            sm.left -= (uint32_t)(met >> 32);
        }
        sm.ok = ok;
    }
    __syncthreads();
    return sm.ok != 0;
}

template <int KIND>
struct AccOf { using T = unsigned long long; };
template <>
struct AccOf<kBack> { using T = double; };
template <>
struct AccOf<kBackLast> { using T = double; };

template <int KIND, class T>
__device__ __forceinline__ T wide_add(T x, T y, bool &ovf) {
    const T s = x + y;
    if (KIND == kFwdFull) ovf |= s < y;
    return s;
}

// Lists of so many entries (16 MB) do not stay in L2 beside the rows, and an id
// is a trip to HBM: they are brought to L2 an item ahead of their loads.
// (Kernel without -> with: 1024 sources of the 1M-vertex graph, 30 M entries, 34.9 ->
// 34.0 ms; 260k vertices, 7 M, 3.78 -> 3.71; 4M vertices 5.55 -> 5.51; lists that
// stay, 97 k entries 0.82 -> 0.84, 1 M 0.256 -> 0.261, 2.3 M 2.49 -> 2.48.)
constexpr uint32_t kWideFar = 1u << 22;

// Entries [b, e) of the lists on their way to L2 (in whole 16 bytes: the lists
// lie in memory rounded to 256).
__device__ __forceinline__ void prefetch_adj(const uint32_t *adj, uint32_t b, uint32_t e, unsigned long long pol) {
    const uintptr_t p0 = (uintptr_t)(adj + b) & ~uintptr_t(15), p1 = ((uintptr_t)(adj + e) + 15) & ~uintptr_t(15);
    if (e > b)
        asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;" ::"l"(p0), "r"((uint32_t)(p1 - p0)), "l"(pol));
}

// The ids of a lane's edges base + step * j, j < 4, below end; past it zero,
// the id of the row of zeros (the graph's number of vertices).
__device__ __forceinline__ void load_ids(uint32_t (&id)[4], const uint32_t *__restrict__ adj, uint32_t base,
                                         uint32_t end, uint32_t step, uint32_t zero, unsigned long long pol) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t e = base + step * j;
        id[j] = e < end ? ld_adj(adj + e, pol) : zero;
    }
}

// Sets of rows that a lane holds, one being added and the others on their way
// (a set: 16 registers).  Each sweep is a matter of rows in flight: with 512
// threads of 128 registers three sets against two take 13.4 against 14.5 ms on
// an Erdos-Renyi graph of 500k vertices (200 sources, jobs of 32), 2.48 against
// 2.61 on a 100k-vertex R-MAT one, the same on the benchmark's; a fourth spills
// (14.0, 2.70).  Jobs of 16: 5.86, 6.00 and 5.58 ms with two, three and four
// sets at 4M vertices.
template <int LS>
constexpr int row_sets() { return LS == 4 ? 4 : 3; }

// The first J of a lane's four edges: a group of four lanes takes its lanes'
// edges one after the other, each lane LS slots of a row, the next rows in
// flight while the last are added.
template <int KIND, int J, int LS, class T>
__device__ __forceinline__ void add_rows(const unsigned char *rows, uint32_t zero, const uint32_t (&id)[4],
                                         T (&acc)[LS]) {
    const unsigned sh = threadIdx.x & 28u;
    if constexpr (KIND == kFwd32) {
        constexpr int U = 16 / LS;  // rows of a step
        uint32_t part[LS];          // at most 16 counts below 2^28
        constexpr int P = row_sets<LS>();
        uint32_t r[P][U][LS];
#pragma unroll
        for (int k = 0; k < LS; ++k) part[k] = 0u;
        auto fetch = [&](int s, uint32_t (&o)[U][LS]) {
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int e = s * U + q;
                ld_row(__shfl_sync(kFull, id[e >> 2], sh + (e & 3)), zero, rows, o[q]);
            }
        };
        constexpr int steps = 4 * J / U;
#pragma unroll
        for (int s = 0; s < P - 1 && s < steps; ++s) fetch(s, r[s]);
#pragma unroll
        for (int s = 0; s < steps; ++s) {
            if (s + P - 1 < steps) fetch(s + P - 1, r[(s + P - 1) % P]);
#pragma unroll
            for (int k = 0; k < LS; ++k) {
                uint32_t t = r[s % P][0][k] + r[s % P][1][k];
                if constexpr (U == 4) t += r[s % P][2][k] + r[s % P][3][k];
                part[k] += t;
            }
        }
#pragma unroll
        for (int k = 0; k < LS; ++k) acc[k] += (T)part[k];
    } else if constexpr (KIND == kBack) {
        constexpr int U = 8 / LS;
        constexpr int P = row_sets<LS>();
        double r[P][U][LS];
        auto fetch = [&](int s, double (&o)[U][LS]) {
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int e = s * U + q;
                ld_row(__shfl_sync(kFull, id[e >> 2], sh + (e & 3)), zero, rows, o[q]);
            }
        };
        constexpr int steps = 4 * J / U;
#pragma unroll
        for (int s = 0; s < P - 1 && s < steps; ++s) fetch(s, r[s]);
#pragma unroll
        for (int s = 0; s < steps; ++s) {
            if (s + P - 1 < steps) fetch(s + P - 1, r[(s + P - 1) % P]);
#pragma unroll
            for (int q = 0; q < U; ++q)
#pragma unroll
                for (int k = 0; k < LS; ++k) acc[k] += r[s % P][q][k];
        }
    }
}

// Adds the rows of a block's neighbours: every lane holds the ids of its own
// four edges.  Ids that no slot holds at the level become the row of zeros.
template <int KIND, int NS, class T>
__device__ __forceinline__ void add_block(const WideCtx &x, uint32_t d, uint32_t zero, uint32_t (&id)[4],
                                          T (&acc)[NS / 4], bool &ovf) {
    constexpr int LS = NS / 4;
    const unsigned l = threadIdx.x & 3u, sh = threadIdx.x & 28u;
    const uint32_t *act = x.act + (size_t)(KIND == kBack ? d + 1 : d) * x.words;
    uint32_t wd[4];
    // (zero's word may be the next level's first: in the array, and without effect)
#pragma unroll
    for (int j = 0; j < 4; ++j) wd[j] = act[id[j] >> 5];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (!((wd[j] >> (id[j] & 31u)) & 1u)) id[j] = zero;
    if constexpr (KIND == kFwdFull) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll 1
            for (int q = 0; q < 4; ++q) {
                const uint32_t u = __shfl_sync(kFull, id[j], sh + q);
                if (u == zero) continue;
#pragma unroll
                for (int h = 0; h < LS; h += 4) {
                    uint32_t r[8];
                    ld32(x.sig + (size_t)u * NS + l * LS + h, r);
                    const uint32_t lv =
                        __ldcg(reinterpret_cast<const uint32_t *>(x.lvl) + (size_t)u * (NS / 4) + l * (LS / 4) + h / 4);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (((lv >> (8 * k)) & 0xFFu) == d)
                            acc[h + k] = wide_add<KIND>(acc[h + k], (T)((unsigned long long)r[2 * k + 1] << 32 | r[2 * k]), ovf);
                }
            }
    } else {
        const unsigned char *rows = rows_of(x, KIND == kBack ? d + 1 : d) + l * (KIND == kFwd32 ? 4 * LS : 8 * LS);
        const bool low = id[0] != zero || id[1] != zero, high = id[2] != zero || id[3] != zero;
        if (__any_sync(kFull, high)) add_rows<KIND, 4>(rows, zero, id, acc);
        else if (__any_sync(kFull, low)) add_rows<KIND, 2>(rows, zero, id, acc);
    }
}

// Level 1.  Its counts are 1 (unless a list names a neighbour twice), so a row
// is a word of 32 slots' bits, and a lane adds the words of its edges bit by bit
// in kPlanes words: bit k of word p is bit p of slot k's sum.  Four edges take
// about 20 instructions where their rows take 80 and 512 bytes.
// (The sweep, 1M-vertex graph, 658 sources: 250 -> 196 us a job; kernel 35.7 ->
// 34.8 ms, 100k-vertex R-MAT 2.56 -> 2.49, 48 small graphs 5.28 -> 5.17, a
// 500k-vertex Erdos-Renyi graph, whose level 1 is next to empty, 13.4 -> 13.6.)
constexpr int kPlanes = 7;  // a lane has at most 64 edges: a chunk's by 32 lanes, or a light vertex's by 4
static_assert(8 * kWideChunk / 32 < 1 << kPlanes && (kWideLight << 3) / 4 < 1 << kPlanes, "planes of a lane's sums");

__device__ __forceinline__ void add_ones(const WideCtx &x, uint32_t d, const uint32_t (&id)[4], uint32_t (&pl)[kPlanes]) {
    const uint32_t *act = x.act + (size_t)d * x.words;
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = act[id[j] >> 5];
    uint32_t hit = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        w[j] = (w[j] >> (id[j] & 31u)) & 1u;
        hit |= w[j];
    }
    if (!__any_sync(kFull, hit)) return;  // most blocks, where the sources have few neighbours
    // (an id past the end is n: its bit may be another level's, its word is 0)
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = w[j] ? x.bits[id[j]] : 0u;
    const uint32_t s = w[0] ^ w[1] ^ w[2], c = (w[0] & w[1]) | (w[2] & (w[0] ^ w[1]));
    const uint32_t ones = s ^ w[3], c2 = s & w[3], twos = c ^ c2, fours = c & c2;
    uint32_t k = pl[0] & ones;
    pl[0] ^= ones;
    const uint32_t k1 = (pl[1] & twos) | (k & (pl[1] ^ twos));
    pl[1] ^= twos ^ k;
    k = (pl[2] & fours) | (k1 & (pl[2] ^ fours));
    pl[2] ^= fours ^ k1;
#pragma unroll
    for (int p = 3; p < kPlanes; ++p) {
        const uint32_t up = pl[p] & k;
        pl[p] ^= k;
        k = up;
    }
}

// Bit l of lane k's result is bit k of lane l's word.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x) {
    const unsigned lane = threadIdx.x & 31;
    constexpr uint32_t low[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const int s = 16 >> i;
        const uint32_t y = __shfl_xor_sync(kFull, x, s);
        x = (lane & (unsigned)s) ? (x & ~low[i]) | ((y >> s) & low[i]) : (x & low[i]) | ((y & low[i]) << s);
    }
    return x;
}

// A group's sums: slot LS * l + i of the four lanes' words into lane l's acc[i].
template <int LS>
__device__ __forceinline__ void ones_to_group(const uint32_t (&pl)[kPlanes], unsigned long long (&acc)[LS]) {
    const unsigned l = threadIdx.x & 3u, sh = threadIdx.x & 28u;
    uint32_t sum[LS];
#pragma unroll
    for (int i = 0; i < LS; ++i) sum[i] = 0u;
#pragma unroll
    for (int p = 0; p < kPlanes; ++p) {
        if (!__any_sync(kFull, pl[p] != 0u)) continue;
        uint32_t b[LS / 4];  // four slots' bytes each
#pragma unroll
        for (int h = 0; h < LS / 4; ++h) b[h] = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t y = __shfl_sync(kFull, pl[p], sh + q) >> (LS * l);
#pragma unroll
            for (int h = 0; h < LS / 4; ++h) b[h] += (((y >> (4 * h)) & 15u) * 0x00204081u) & 0x01010101u;
        }
#pragma unroll
        for (int i = 0; i < LS; ++i) sum[i] += ((b[i / 4] >> (8 * (i & 3))) & 0xFFu) << p;
    }
#pragma unroll
    for (int i = 0; i < LS; ++i) acc[i] = sum[i];
}

// The eight groups' sums of a warp's vertex, added in a fixed order and dealt
// out one slot a lane (own_slot): lane 4g + l gets one of the slots LS * l ..,
// which one by g's bits (16 slots: groups g and g ^ 1 get the same).
template <int NS>
__device__ __forceinline__ uint32_t own_slot() {
    const unsigned lane = threadIdx.x & 31, l = lane & 3u, g = lane >> 2;
    if (NS == 16) return 4u * l + (g >> 1);
    return 8u * l + g;
}
// Whether the lane is the one that stores its slot.
template <int NS>
__device__ __forceinline__ bool own_store() { return NS == 32 || !(threadIdx.x & 4u); }

template <int KIND, int NS, class T>
__device__ __forceinline__ T wide_fold(const T (&acc)[NS / 4], bool &ovf) {
    constexpr int LS = NS / 4;
    const unsigned lane = threadIdx.x & 31;
    T a[LS];
#pragma unroll
    for (int k = 0; k < LS; ++k) a[k] = acc[k];
#pragma unroll
    for (int n = LS / 2, o = 16; n >= 1; n /= 2, o /= 2) {
        const bool up = lane & (unsigned)o;
#pragma unroll
        for (int k = 0; k < n; ++k) {
            const T keep = up ? a[n + k] : a[k], give = up ? a[k] : a[n + k];
            a[k] = wide_add<KIND>(keep, (T)__shfl_xor_sync(kFull, give, o), ovf);
        }
    }
    if (NS == 16) a[0] = wide_add<KIND>(a[0], (T)__shfl_xor_sync(kFull, a[0], 4), ovf);
    return a[0];
}

// The warp's sums in the same places.
template <int NS>
__device__ __forceinline__ unsigned long long ones_to_warp(const uint32_t (&pl)[kPlanes]) {
    uint32_t sum = 0;
#pragma unroll
    for (int p = 0; p < kPlanes; ++p)
        if (__any_sync(kFull, pl[p] != 0u)) sum += (uint32_t)__popc(transpose_bits(pl[p])) << p;
    return __shfl_sync(kFull, sum, own_slot<NS>());
}

// Finishing a vertex whose sums lie one slot a lane (wide_fold's order): the
// whole warp calls.
template <int NS>
__device__ __forceinline__ uint32_t finish_fwd_warp(const WideCtx &x, uint32_t v, unsigned long long sum, uint32_t d,
                                                    uint32_t &found) {
    const uint32_t k = own_slot<NS>();
    unsigned char *lp = x.lvl + (size_t)v * NS + k;
    const uint32_t lv = __ldcg(lp);
    const bool fresh = lv == kUnseen && sum != 0ull;
    const bool got = __any_sync(kFull, fresh), left = __any_sync(kFull, lv == kUnseen && !fresh);
    if (got) {
        found |= 1u;
        if (own_store<NS>()) {
            reinterpret_cast<uint32_t *>(rows_of(x, d + 1))[(size_t)v * NS + k] = fresh ? (uint32_t)sum : 0u;
            if (fresh) {
                *lp = (unsigned char)(d + 1);
                x.sig[(size_t)v * NS + k] = sum;
                if (sum >> 28) found |= 2u;
            }
        }
    }
    return (got ? 1u : 0u) | (left ? 0u : 2u);
}

template <int NS>
__device__ __forceinline__ void finish_back_warp(const WideCtx &x, const double *mult, uint32_t v, uint32_t reach,
                                                 double sum, uint32_t d) {
    const uint32_t k = own_slot<NS>();
    const uint32_t lv = __ldcg(x.lvl + (size_t)v * NS + k);
    double s = 0.0, xo = 0.0;
    if (lv == d) {
        const double sg = (double)__ldcg(x.sig + (size_t)v * NS + k);
        const double delta = (double)reach + sg * sum;
        xo = (1.0 + delta) / sg;
        s = mult[k] * delta;
    }
    if (own_store<NS>()) reinterpret_cast<double *>(rows_of(x, d))[(size_t)v * NS + k] = xo;
#pragma unroll
    for (int o = 1; o <= 16; o *= 2)
        if (NS == 32 || o != 4) s += __shfl_xor_sync(kFull, s, o);
    // one add per vertex and sweep, sweeps ordered by the barrier
    if ((threadIdx.x & 31) == 0) atomicAdd(x.bc + v, s);
}

// Finishes vertex v from its sums (lane l of its group holds slots LS * l ..);
// every lane of the warp calls it, the ones without a vertex with valid =
// false.  Forward: the slots not reached yet whose sum is not 0 are at level d
// + 1.  Returns the bits of v's group: 1 some slot was reached, 2 none is left.
template <int NS>
__device__ __forceinline__ uint32_t finish_fwd(const WideCtx &x, uint32_t v, const unsigned long long (&acc)[NS / 4],
                                               bool valid, uint32_t d, uint32_t &found) {
    constexpr int LS = NS / 4, LW = LS / 4;
    const unsigned lane = threadIdx.x & 31, l = lane & 3u, sh = lane & 28u;
    uint32_t *lp = reinterpret_cast<uint32_t *>(x.lvl) + (size_t)v * (NS / 4) + l * LW;
    uint32_t nl[LW], f[LS];
    bool got = false, left = false;
#pragma unroll
    for (int h = 0; h < LW; ++h) {
        const uint32_t lv = valid ? __ldcg(lp + h) : 0u;
        nl[h] = lv;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = 4 * h + k;
            const bool fresh = ((lv >> (8 * k)) & 0xFFu) == kUnseen && acc[i] != 0ull;
            f[i] = fresh ? (uint32_t)acc[i] : 0u;
            if (fresh) {
                nl[h] = (nl[h] & ~(0xFFu << (8 * k))) | ((d + 1) << (8 * k));
                x.sig[(size_t)v * NS + LS * l + i] = acc[i];
                if (acc[i] >> 28) found |= 2u;
            }
        }
        if (nl[h] != lv) {
            lp[h] = nl[h];
            got = true;
        }
        left |= valid && __vcmpeq4(nl[h], kFull) != 0u;
    }
    const bool any = (__ballot_sync(kFull, got) >> sh) & 15u, rest = (__ballot_sync(kFull, left) >> sh) & 15u;
    if (any) {
        found |= 1u;
        uint4 *row = reinterpret_cast<uint4 *>(rows_of(x, d + 1) + (size_t)v * (NS * 4) + l * (4 * LS));
#pragma unroll
        for (int h = 0; h < LW; ++h) row[h] = make_uint4(f[4 * h], f[4 * h + 1], f[4 * h + 2], f[4 * h + 3]);
    }
    return (any ? 1u : 0u) | (rest ? 0u : 2u);
}

// Backward: delta = reach + sigma * sum of X over the children, X = (1 +
// delta) / sigma for the slots at level d, and the weighted delta into the
// job's vector.
template <int NS>
__device__ __forceinline__ void finish_back(const WideCtx &x, const WideSmem<NS> &sm, uint32_t v,
                                            const double (&acc)[NS / 4], bool valid, uint32_t d) {
    constexpr int LS = NS / 4, LW = LS / 4;
    const unsigned l = threadIdx.x & 3u;
    double s = 0.0;
    if (valid) {
#pragma unroll
        for (int h = 0; h < LW; ++h) {
            const uint32_t lv = __ldcg(reinterpret_cast<const uint32_t *>(x.lvl) + (size_t)v * (NS / 4) + l * LW + h);
            uint32_t w[8];
            uint32_t r[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k] = 0u;
            if (__vcmpeq4(lv, d * 0x01010101u)) {
                const double reach = (double)sm.sub.vinfo[v].y;
                ld32(x.sig + (size_t)v * NS + LS * l + 4 * h, r);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (((lv >> (8 * k)) & 0xFFu) != d) continue;
                    const double sg = (double)((unsigned long long)r[2 * k + 1] << 32 | r[2 * k]);
                    const double delta = reach + sg * acc[4 * h + k];
                    const double xo = (1.0 + delta) / sg;
                    w[2 * k] = (uint32_t)__double2loint(xo);
                    w[2 * k + 1] = (uint32_t)__double2hiint(xo);
                    s += sm.mult[LS * l + 4 * h + k] * delta;
                }
            }
            st32(rows_of(x, d) + (size_t)v * (NS * 8) + l * (8 * LS) + 32 * h, w);
        }
    }
    s += __shfl_xor_sync(kFull, s, 1);
    s += __shfl_xor_sync(kFull, s, 2);
    // one add per vertex and sweep, sweeps ordered by the barrier
    if (valid && l == 0) atomicAdd(x.bc + v, s);
}

// One sweep over the team's share of the job's vertices.
// (Not inlined: each kind then has the registers to itself.)
template <int KIND, int NS>
__device__ __noinline__ void wide_sweep(WideSmem<NS> &sm, uint32_t d) {
    const WideCtx &x = sm.x;
    using T = typename AccOf<KIND>::T;
    constexpr bool kForward = KIND == kFwd32 || KIND == kFwdFull || KIND == kFwdOnes;
    constexpr bool kOnes = KIND == kFwdOnes;
    constexpr int side = kForward ? 0 : 1;
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const WideSub &g = sm.sub;
    const uint32_t *offs = g.offs[side], *adj = g.adj[side];
    const uint32_t W = x.T * kWideWarps;
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    // items: chunks of the heavy vertices, runs of medium ones, (parts of)
    // words of light ones; as many a draw as leave every warp about four draws
    constexpr bool kGather = KIND != kBackLast;  // nothing to gather: every vertex is a light one
    const uint32_t nchunk = kGather ? g.nchunk[side] : 0u;
    const uint32_t light0 = kGather ? sm.nmed : 0u;
    const uint32_t nmedv = kGather ? sm.nmed - g.nheavy : 0u;
    const uint32_t left = kForward ? sm.left : sm.met[d];  // vertices the sweep does something for, at most
    const uint32_t thin = left >= g.n ? 1u : min(32u, g.n / max(1u, left));  // 1 in so many
    // (the few are the heavy ones first, so chunks are not drawn in larger lots)
    const uint32_t cb = min(4u, max(1u, nchunk / (4u * W)));
    const uint32_t mb = min(8u, max(1u, nmedv / (4u * W)));
    const uint32_t nl = g.n - light0;
    const uint32_t lp = thin > 1u ? 1u : (nl >= 128u * W ? 1u : (nl >= 64u * W ? 2u : 4u));  // parts of a word
    const uint32_t lw = min(thin, max(1u, nl / (64u * W)));  // or words of a draw
    const uint32_t nci = (nchunk + cb - 1) / cb, nmi = (nmedv + mb - 1) / mb;
    const uint32_t w0 = light0 >> 5, nli = nl ? ((((g.n + 31u) >> 5) - w0) * lp + lw - 1u) / lw : 0u;
    const uint32_t total = nci + nmi + nli;
    const uint32_t *need_map = kForward ? x.done : x.act + (size_t)d * x.words;
    uint32_t found = 0, fresh = 0, gone = 0;  // of the lane
    bool ovf = false;
    for (;;) {
        uint32_t c = 0;
        if (lane == 0) c = atomicAdd(&sm.next, 1u);
        c = __shfl_sync(kFull, c, 0);
        if (c >= total) break;  // so that c * T below cannot wrap
        const uint32_t it = x.rank + c * x.T;
        if (it >= total) break;
        if (it < nci + nmi) {
            // up to 32 segments of a warp each, lane i holding the i-th: chunks
            // of heavy vertices, or whole medium vertices
            const bool heavy = it < nci;
            uint32_t v = 0, e0 = 0, e1 = 0;
            bool need = false;
            if (heavy) {
                const uint32_t i = it * cb + lane;
                if (lane < cb && i < nchunk) {
                    const uint2 ch = g.chunk[side][i];
                    v = ch.x - g.base;
                    e0 = offs[v] + ch.y * g.chunk_len;
                    e1 = min(offs[v + 1], e0 + g.chunk_len);
                    need = true;
                }
            } else {
                v = g.nheavy + (it - nci) * mb + lane;
                if (lane < mb && v < sm.nmed) {
                    e0 = offs[v];
                    e1 = offs[v + 1];
                    need = true;
                }
            }
            if (need) {
                const uint32_t w = need_map[v >> 5] >> (v & 31u);
                need = kForward ? !(w & 1u) : (w & 1u) != 0u;
            }
            unsigned todo = __ballot_sync(kFull, need);
            if (need && sm.far) prefetch_adj(adj, e0, e1, pol);
            uint32_t nxt[4];
            uint32_t sb = 0, se = 0;
            if (todo) {
                sb = __shfl_sync(kFull, e0, __ffs(todo) - 1);
                se = __shfl_sync(kFull, e1, __ffs(todo) - 1);
                load_ids(nxt, adj, sb + lane, se, 32u, g.n, pol);
            }
#pragma unroll 1
            while (todo) {
                const int i = __ffs(todo) - 1;
                todo &= todo - 1;
                const uint32_t vi = __shfl_sync(kFull, v, i), end = se;
                T acc[NS / 4] = {};
                uint32_t pl[kPlanes] = {};
                uint32_t at = sb;
                bool more;
#pragma unroll 1
                do {
                    // the next block of this segment, or the next segment's
                    // first, is on its way while this one is added
                    uint32_t id[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) id[j] = nxt[j];
                    at += 128u;
                    more = at < end;
                    if (more) {
                        load_ids(nxt, adj, at + lane, end, 32u, g.n, pol);
                    } else if (todo) {
                        sb = __shfl_sync(kFull, e0, __ffs(todo) - 1);
                        se = __shfl_sync(kFull, e1, __ffs(todo) - 1);
                        load_ids(nxt, adj, sb + lane, se, 32u, g.n, pol);
                    }
                    if constexpr (kOnes) add_ones(x, d, id, pl);
                    else if constexpr (kGather) add_block<KIND, NS>(x, d, g.n, id, acc, ovf);
                } while (more);
                T sum;
                if constexpr (kOnes) sum = ones_to_warp<NS>(pl);
                else sum = wide_fold<KIND, NS>(acc, ovf);
                if (heavy) {
                    const uint32_t ci = it * cb + i;
                    const uint32_t c0 = g.cbeg[side][vi] - g.chunk0[side], nc = g.cbeg[side][vi + 1] - g.chunk0[side] - c0;
                    if (nc > 1) {
                        // the chunks meet: the one that arrives last adds them in
                        // order (16 slots: half warps the even and the odd ones)
                        const uint32_t k = own_slot<NS>();
                        T *part = reinterpret_cast<T *>(x.part);
                        if (own_store<NS>()) __stcg(part + (size_t)ci * NS + k, sum);
                        __syncwarp();
                        uint32_t last = 0;
                        if (lane == 0) {
                            __threadfence();
                            last = atomicAdd(x.hcnt + vi, 1u) == nc - 1u;
                            if (last) __threadfence();
                        }
                        last = __shfl_sync(kFull, last, 0);
                        if (!last) continue;
                        if (lane == 0) x.hcnt[vi] = 0u;
                        sum = 0;
                        constexpr uint32_t step = NS == 16 ? 2u : 1u;
#pragma unroll 4
                        for (uint32_t q = NS == 16 ? (lane >> 2) & 1u : 0u; q < nc; q += step)
                            sum = wide_add<KIND>(sum, __ldcg(part + (size_t)(c0 + q) * NS + k), ovf);
                        if (NS == 16) sum = wide_add<KIND>(sum, (T)__shfl_xor_sync(kFull, sum, 4), ovf);
                    }
                }
                if constexpr (kForward) {
                    const uint32_t b = finish_fwd_warp<NS>(x, vi, sum, d, found);
                    if (lane == 0) {
                        if (b & 1u) {
                            atomicOr(x.act + (size_t)(d + 1) * x.words + (vi >> 5), 1u << (vi & 31u));
                            ++fresh;
                        }
                        if (b & 2u) {
                            atomicOr(x.done + (vi >> 5), 1u << (vi & 31u));
                            ++gone;
                        }
                    }
                } else {
                    finish_back_warp<NS>(x, sm.mult, vi, g.vinfo[vi].y, sum, d);
                }
            }
        } else {
            // lw words, one a lane, or part of one
            const uint32_t li = (it - nci - nmi) * lw, wl = w0 + li / lp + lane;
            uint32_t ml = 0;
            if (lane < lw && wl << 5 < g.n) {
                const uint32_t vl = wl << 5;
                ml = need_map[wl];
                if (kForward) ml = ~ml;
                if (lp > 1) ml &= ((1u << (32u / lp)) - 1u) << ((li % lp) * (32u / lp));
                if (kGather && vl < light0) ml &= kFull << (light0 - vl);
                if (vl + 32u > g.n) ml &= (1u << (g.n - vl)) - 1u;
            }
#pragma unroll 1
            for (unsigned full = __ballot_sync(kFull, ml != 0u); full; full &= full - 1) {
            const int wi = __ffs(full) - 1;
            const uint32_t w = w0 + li / lp + wi, vb = w << 5, m = __shfl_sync(kFull, ml, wi);
            uint32_t e0 = 0, e1 = 0;
            if (kGather && vb + lane < g.n) {
                e0 = offs[vb + lane];
                e1 = offs[vb + lane + 1];
            }
            if (kGather && sm.far) {  // four of eight vertices or more: the eight's lists
                const uint32_t q0 = __shfl_sync(kFull, e0, (8u * lane) & 31u), q1 = __shfl_sync(kFull, e1, (8u * lane + 7u) & 31u);
                if (lane < 4 && __popc((m >> (8u * lane)) & 0xFFu) >= 4) prefetch_adj(adj, q0, q1, pol);
            }
            if ((m >> lane) & 1u) sm.list[wid][__popc(m & ((1u << lane) - 1u))] = (unsigned char)lane;
            __syncwarp();
            const uint32_t cnt = __popc(m);
            // eight vertices at a time, four lanes each
            auto pick = [&](uint32_t i0, bool &ok, uint32_t &p, uint32_t &b, uint32_t &e) {
                const uint32_t i = i0 + (lane >> 2);
                ok = i < cnt;
                p = ok ? sm.list[wid][i] : 0u;
                b = __shfl_sync(kFull, e0, p);
                e = __shfl_sync(kFull, e1, p);
                if (!ok) e = b;
            };
            bool ok;
            uint32_t p, sb, se, nxt[4];
            pick(0, ok, p, sb, se);
            if constexpr (kGather) load_ids(nxt, adj, sb + (lane & 3u), se, 4u, g.n, pol);
#pragma unroll 1
            for (uint32_t i0 = 0; i0 < cnt; i0 += 8) {
                const bool valid = ok;
                const uint32_t v = vb + p;
                T acc[NS / 4] = {};
                uint32_t pl[kPlanes] = {};
                if constexpr (kGather) {
                    const uint32_t b = sb, e = se;
                    const uint32_t nblk = max(1u, __reduce_max_sync(kFull, (e - b + 15u) / 16u));
#pragma unroll 1
                    for (uint32_t k = 1; k <= nblk; ++k) {
                        uint32_t id[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) id[j] = nxt[j];
                        if (k < nblk) {
                            load_ids(nxt, adj, b + 16u * k + (lane & 3u), e, 4u, g.n, pol);
                        } else if (i0 + 8 < cnt) {
                            pick(i0 + 8, ok, p, sb, se);
                            load_ids(nxt, adj, sb + (lane & 3u), se, 4u, g.n, pol);
                        }
                        if constexpr (kOnes) add_ones(x, d, id, pl);
                        else add_block<KIND, NS>(x, d, g.n, id, acc, ovf);
                    }
                    if constexpr (kOnes) ones_to_group<NS / 4>(pl, acc);
                } else {
                    pick(i0 + 8, ok, p, sb, se);
                }
                if constexpr (kForward) {
                    const uint32_t b = finish_fwd<NS>(x, v, acc, valid, d, found);
                    const uint32_t bit = valid ? 1u << (v & 31u) : 0u;
                    const uint32_t am = __reduce_or_sync(kFull, (b & 1u) ? bit : 0u);
                    const uint32_t dm = __reduce_or_sync(kFull, (b & 2u) ? bit : 0u);
                    if (lane == 0) {
                        if (am) {
                            atomicOr(x.act + (size_t)(d + 1) * x.words + w, am);
                            fresh += __popc(am);
                        }
                        if (dm) {
                            atomicOr(x.done + w, dm);
                            gone += __popc(dm);
                        }
                    }
                } else {
                    finish_back<NS>(x, sm, v, acc, valid, d);
                }
            }
            __syncwarp();
            }
        }
    }
    if (KIND == kFwdFull && ovf) found |= 4u;
    if (kForward) {
        found = __reduce_or_sync(kFull, found);
        if (lane == 0 && found) atomicOr(&sm.found, found);
        if (lane == 0 && (fresh | gone)) atomicAdd(&sm.count, (unsigned long long)gone << 32 | fresh);
    }
}

// Whether a path count at level d + 1 passed 2^64, asked after a forward
// sweep in which some sum did: the sweep sums every slot of a vertex, and what
// a slot that was reached before sums is no count.  Summed again for the slots
// that were open then (not reached now, or at level d + 1): a warp a vertex, a
// lane a slot.  (Telling them apart in the sweep itself takes registers from
// all of its kinds: 1 % of every run.)
template <int NS>
__device__ __noinline__ bool count_overflows(const WideSmem<NS> &sm, uint32_t d) {
    const WideCtx &x = sm.x;
    const WideSub &g = sm.sub;
    const unsigned lane = threadIdx.x & 31;
    const uint32_t w = x.rank * kWideWarps + (threadIdx.x >> 5);
    bool ovf = false;
    for (uint32_t v = w; v < g.n; v += x.T * kWideWarps) {
        const uint32_t lv = lane < NS ? __ldcg(x.lvl + (size_t)v * NS + lane) : kEmpty;
        const bool open = lv == kUnseen || lv == d + 1u;
        if (!__any_sync(kFull, open)) continue;
        unsigned long long sum = 0;
        const uint32_t e1 = g.offs[0][v + 1];
        for (uint32_t e = g.offs[0][v]; e < e1; ++e) {
            const size_t at = (size_t)g.adj[0][e] * NS + lane;
            if (open && __ldcg(x.lvl + at) == d) sum = wide_add<kFwdFull>(sum, __ldcg(x.sig + at), ovf);
        }
    }
    return ovf;
}

__device__ __forceinline__ void wide_trace(const WideArgs &a, uint32_t job, uint32_t kind, uint32_t level,
                                           uint32_t info) {
    if (!a.trace || blockIdx.x != 0 || threadIdx.x != 0) return;
    const unsigned int i = *a.trace_cnt;
    if (i >= a.trace_cap) return;
    a.trace[i] = TraceRec{wide_ns(), job, kind, level, info, 0ull};
    *a.trace_cnt = i + 1;
}

template <int NS>
__global__ void __launch_bounds__(kWideThreads, 1) bc_wide_kernel(WideArgs a) {
    __shared__ WideSmem<NS> sm;
    WideCtx &x = sm.x;
    const uint32_t team = blockIdx.x / a.team_ctas;
    if (team >= a.teams) return;
    if (a.poison && *reinterpret_cast<volatile int *>(a.poison)) return;
    WideTeam *t = a.team + team;
    if (threadIdx.x == 0) {
        unsigned char *st = a.state + (size_t)team * a.stride;
        x.T = a.team_ctas;
        x.rank = blockIdx.x % a.team_ctas;
        x.lvl = st;
        x.done = reinterpret_cast<uint32_t *>(st + a.o_done);
        x.act = reinterpret_cast<uint32_t *>(st + a.o_act);
        x.words = a.words;
        x.bits = reinterpret_cast<uint32_t *>(st + a.o_bits);
        x.sig = reinterpret_cast<unsigned long long *>(st + a.o_sig);
        x.g0 = st + a.o_g0;
        x.g01 = (ptrdiff_t)(a.o_g1 - a.o_g0);
        x.part = reinterpret_cast<unsigned long long *>(st + a.o_part);
        x.hcnt = reinterpret_cast<uint32_t *>(st + a.o_hcnt);
    }
    __syncthreads();
    const unsigned lane = threadIdx.x & 31;
    const uint32_t tid = x.rank * kWideThreads + threadIdx.x, nt = x.T * kWideThreads;
    if (threadIdx.x == 0) {
        sm.next = 0;
        sm.found = 0;
        sm.count = 0;
    }
    uint32_t job = team;
    for (uint32_t par = 0; job < a.njobs; par ^= 1u) {
        WideJob J{0u, 0u, 0u, 0u, 0ull};
        if (a.jobs) {
            J = a.jobs[job];
        } else {  // one graph's sources in order
            J.root0 = (a.job0 + job) * NS;
            J.nroots = min((uint32_t)NS, a.nroots - J.root0);
            J.out = (unsigned long long)job * a.subs[0].n;
        }
        if (threadIdx.x < sizeof(WideSub) / 4)
            reinterpret_cast<uint32_t *>(&sm.sub)[threadIdx.x] =
                reinterpret_cast<const uint32_t *>(a.subs + J.sub)[threadIdx.x];
        __syncthreads();
        if (threadIdx.x == 0) {
            // four lanes take a vertex while its blocks are no more than
            // about half of a warp's share of a sweep
            const uint32_t share = 128u * kWideWarps * (a.split_ctas ? a.split_ctas : x.T);
            const uint32_t entries = sm.sub.offs[1][sm.sub.n] - sm.sub.offs[1][0], blocks = entries / share;
            sm.far = entries >= kWideFar;
            sm.nmed = sm.sub.nmed[blocks >= 32 ? 3 : (blocks >= 16 ? 2 : (blocks >= 8 ? 1 : 0))];
        }
        if (threadIdx.x < NS) {
            const bool has = threadIdx.x < J.nroots;
            uint32_t r = kNone;
            if (has) r = sm.sub.inv[a.roots[J.root0 + threadIdx.x]];
            sm.roots[threadIdx.x] = r;
            sm.mult[threadIdx.x] = !has ? 0.0 : (a.mult ? a.mult[J.root0 + threadIdx.x] : 1.0);
        }
        if (threadIdx.x == 0) x.bc = a.jobbc + J.out;
        __syncthreads();
        const uint32_t n = sm.sub.n;
        const uint32_t *offs1 = sm.sub.offs[1], *adj1 = sm.sub.adj[1];
        if (threadIdx.x == 0) sm.left = n;
        if (threadIdx.x < 32) {
            // (16 lists of one graph: the sum may pass 2^32 only on graphs refused on the host)
            const uint32_t r = lane < NS ? sm.roots[lane] : kNone;
            uint32_t s = r != kNone ? offs1[r + 1] - offs1[r] : 0u;
#pragma unroll
            for (int o = 1; o < NS; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, s, o);
                if (lane >= (unsigned)o) s += y;
            }
            if (lane < NS) sm.edges[lane + 1] = s;
            if (lane == 0) sm.edges[0] = 0;
        }
        __syncthreads();
        // f(k, w) for every neighbour w of the source in slot k
        auto each_first = [&](auto f) {
            for (uint32_t i = tid; i < sm.edges[NS]; i += nt) {
                int k = 0;
                while (sm.edges[k + 1] <= i) ++k;
                f(k, adj1[offs1[sm.roots[k]] + (i - sm.edges[k])]);
            }
        };
        // reset: levels, the bitmaps of levels 0 and 1, the job's vector; the
        // sources at level 0 with one path
        if (x.rank == 0 && threadIdx.x == 0) {
            t->job[par] = a.teams + atomicAdd(&a.ctrl->next_job, 1u);
            for (int i = 0; i < 4; ++i) {
                t->any[i] = 0;
                t->count[i] = 0ull;
            }
        }
        for (uint32_t v = tid; v < n; v += nt) {
            uint32_t w[NS / 4];
#pragma unroll
            for (int k = 0; k < NS / 4; ++k) w[k] = kFull;
            bool root = false;
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                const uint32_t r = sm.roots[k];
                if (r == kNone) w[k >> 2] = (w[k >> 2] & ~(0xFFu << (8 * (k & 3)))) | (kEmpty << (8 * (k & 3)));
                if (r == v) {
                    w[k >> 2] &= ~(0xFFu << (8 * (k & 3)));
                    root = true;
                }
            }
#pragma unroll
            for (int h = 0; h < NS / 16; ++h)
                reinterpret_cast<uint4 *>(x.lvl)[(size_t)v * (NS / 16) + h] =
                    make_uint4(w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3]);
            x.bc[v] = 0.0;
            if (root) {
                uint32_t *row = reinterpret_cast<uint32_t *>(x.g0) + (size_t)v * NS;
                for (int k = 0; k < NS; ++k) {
                    row[k] = sm.roots[k] == v;
                    if (sm.roots[k] == v) x.sig[(size_t)v * NS + k] = 1ull;
                }
            }
        }
        for (uint32_t w = tid; w < (n + 31u) >> 5; w += nt) {
            uint32_t m = 0;
            for (int k = 0; k < NS; ++k)
                if (sm.roots[k] >> 5 == w && sm.roots[k] != kNone) m |= 1u << (sm.roots[k] & 31u);
            x.done[w] = 0;
            x.act[w] = m;
            x.act[x.words + w] = 0;
        }
        if (x.rank == 0 && threadIdx.x == 0) x.bits[n] = 0u;
        for (uint32_t i = tid; i < sm.sub.nheavy; i += nt) x.hcnt[i] = 0;
        // the rows of zeros: row n of the counts' rows and of the doubles'
        if (x.rank == 0 && threadIdx.x < NS) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                reinterpret_cast<uint32_t *>(rows_of(x, h))[(size_t)n * NS + threadIdx.x] = 0u;
                reinterpret_cast<double *>(rows_of(x, h))[(size_t)n * NS + threadIdx.x] = 0.0;
            }
        }
        // the rows of level 1 start from 0
        each_first([&](int k, uint32_t w) {
            if (w != sm.roots[k]) x.sig[(size_t)w * NS + k] = 0ull;
            x.bits[w] = 0u;
            uint4 *row = reinterpret_cast<uint4 *>(rows_of(x, 1) + (size_t)w * (NS * 4));
#pragma unroll
            for (int h = 0; h < NS / 4; ++h) row[h] = make_uint4(0u, 0u, 0u, 0u);
        });
        if (!team_sync(a, x, t, sm, 5)) return;
        wide_trace(a, job, 0, 0, n);

        // ---- forward
        uint32_t d = 0;
        bool big = false;  // some count of level d is 2^28 or more
        bool ones = false;  // every count of level 1 is 1
        for (;; ++d) {
            if (d + 2 >= kWideLevels) {
                if (!a.deep_jobs) {
                    if (threadIdx.x == 0) {
                        a.ctrl->deep = 1;
                        if (a.poison) *a.poison = 1;
                    }
                    return;
                }
                if (x.rank == 0 && threadIdx.x == 0) a.deep_jobs[job] = 1u;
                d = kWideLevels;  // the job is left
                break;
            }
            for (uint32_t w = tid; w < (n + 31u) >> 5; w += nt) x.act[(size_t)(d + 2) * x.words + w] = 0;
            if (x.rank == 0 && threadIdx.x == 0) {
                t->any[(d + 2) & 3] = 0;
                t->count[(d + 2) & 3] = 0ull;
            }
            if (d == 0) {
                // level 1: the sources' neighbours, one path for each time
                // they are listed
                each_first([&](int k, uint32_t w) {
                    if (w == sm.roots[k]) return;
                    x.lvl[(size_t)w * NS + k] = 1;
                    if (atomicAdd(x.sig + (size_t)w * NS + k, 1ull)) atomicOr(&sm.found, 8u);  // listed before
                    atomicOr(x.bits + w, 1u << k);
                    atomicAdd(reinterpret_cast<uint32_t *>(rows_of(x, 1)) + (size_t)w * NS + k, 1u);
                    atomicOr(x.act + x.words + (w >> 5), 1u << (w & 31u));
                });
                if (threadIdx.x == 0 && sm.edges[NS]) {
                    atomicOr(&sm.found, 1u);
                    if (x.rank == 0) sm.count = sm.edges[NS];  // at most
                }
            } else if (big) wide_sweep<kFwdFull, NS>(sm, d);
            else if (d == 1 && ones) wide_sweep<kFwdOnes, NS>(sm, d);
            else wide_sweep<kFwd32, NS>(sm, d);
            if (!team_sync(a, x, t, sm, d & 3, d + 1)) return;
            const uint32_t any = sm.any;
            wide_trace(a, job, 2, d, any);
            if (any & 4u) {
                if (count_overflows<NS>(sm, d)) {
                    a.ctrl->overflow = 1;
                    if (a.poison) *a.poison = 1;
                }
                if (!team_sync(a, x, t, sm, 5)) return;
            }
            if (!(any & 1u)) break;
            big = (any & 2u) != 0;
            ones = d == 0 && !(any & 8u);
        }
        const uint32_t D = d == kWideLevels ? 0u : d;

        // ---- what each source reached: a thread's vertices, four slots each
        // (a job is left by callers that do not ask)
        const bool counted = a.rstat || a.total;
        if (threadIdx.x < 3 * NS) sm.reach[threadIdx.x] = 0ull;
        __syncthreads();
        if (counted) {
            uint32_t vis[4] = {0, 0, 0, 0};
            unsigned long long ws[4] = {0, 0, 0, 0}, mc[4] = {0, 0, 0, 0};
            for (uint32_t i = tid; i < n * (NS / 4u); i += nt) {  // below 2^32 (checked on the host)
                const uint32_t lv = __ldcg(reinterpret_cast<const uint32_t *>(x.lvl) + i);
                const uint2 vi = sm.sub.vinfo[i / (NS / 4u)];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (((lv >> (8 * k)) & 0xFFu) >= kWideLevels) continue;
                    ++vis[k];
                    ws[k] += 1ull + vi.y;
                    mc[k] += (unsigned long long)vi.x + 2ull * vi.y;
                }
            }
            // nt is a multiple of 8, so a thread's words all belong to the same four slots
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                unsigned long long s0 = vis[k], s1 = ws[k], s2 = mc[k];
#pragma unroll
                for (int o = NS / 4; o <= 16; o <<= 1) {
                    s0 += __shfl_xor_sync(kFull, s0, o);
                    s1 += __shfl_xor_sync(kFull, s1, o);
                    s2 += __shfl_xor_sync(kFull, s2, o);
                }
                if (lane < NS / 4 && s0) {
                    atomicAdd(&sm.reach[4 * lane + k], s0);
                    atomicAdd(&sm.reach[NS + 4 * lane + k], s1);
                    atomicAdd(&sm.reach[2 * NS + 4 * lane + k], s2);
                }
            }
        }
        __syncthreads();
        if (threadIdx.x < NS && sm.reach[threadIdx.x] && a.total) {
            atomicAdd(&a.total->visited, sm.reach[threadIdx.x]);
            atomicAdd(&a.total->wsum, sm.reach[NS + threadIdx.x]);
            atomicAdd(&a.total->mc2, sm.reach[2 * NS + threadIdx.x]);
            atomicMax(&a.total->depth, D);
        } else if (threadIdx.x < NS && sm.reach[threadIdx.x] && a.rstat) {
            RootStat *rs = a.rstat + (size_t)job * NS + threadIdx.x;
            atomicAdd(&rs->visited, sm.reach[threadIdx.x]);
            atomicAdd(&rs->wsum, sm.reach[NS + threadIdx.x]);
            atomicAdd(&rs->mc2, sm.reach[2 * NS + threadIdx.x]);
            rs->depth = D;
        }

        // ---- backward
        for (uint32_t e = D; e >= 1; --e) {
            if (e == D) wide_sweep<kBackLast, NS>(sm, e);
            else wide_sweep<kBack, NS>(sm, e);
            if (!team_sync(a, x, t, sm, 4)) return;
            wide_trace(a, job, 3, e, 0);
        }
        if (D == 0 && !team_sync(a, x, t, sm, 4)) return;
        job = *reinterpret_cast<volatile uint32_t *>(&t->job[par]);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Adding up the jobs: vertex v of a graph gets its jobs' dependencies, eight
// interleaved partial sums in job order, then those in order.
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_wide_reduce(const WideCtrl *__restrict__ ctrl,
                                                     const int *__restrict__ poison,
                                                     const WideOut *__restrict__ outs, WideOut one,
                                                     const double *__restrict__ jobbc) {
    __shared__ double part[8][32];
    if (ctrl->error | ctrl->overflow | ctrl->deep) return;  // nothing of a stopped launch is kept
    if (poison && *poison) return;
    WideOut o = outs ? outs[blockIdx.y] : one;
    if (o.sub) o.n = o.sub->n;
    const unsigned lane = threadIdx.x & 31, p = threadIdx.x >> 5;
    for (uint32_t v0 = blockIdx.x * 32; v0 < o.n; v0 += gridDim.x * 32) {
        const uint32_t v = v0 + lane;
        double s = 0.0;
        if (v < o.n) {
            const double *q = jobbc + o.out0 + v;
#pragma unroll 4
            for (uint32_t j = p; j < o.njobs; j += 8) s += __ldcs(q + (size_t)j * o.n);
        }
        part[p][lane] = s;
        __syncthreads();
        if (p == 0 && v < o.n) {
#pragma unroll
            for (int k = 1; k < 8; ++k) s += part[k][lane];
            o.bc[o.map[v]] += s;
        }
        __syncthreads();
    }
}

// The same in strict job order, so that the bits do not depend on how the
// jobs of a graph are spread over launches.
__global__ void __launch_bounds__(256) k_wide_chain(const int *__restrict__ poison, const WideOut *__restrict__ outs,
                                                    const double *__restrict__ jobbc,
                                                    const uint32_t *__restrict__ deep_jobs) {
    if (*poison) return;
    const WideOut o = outs[blockIdx.y];
    bool left = false;
    for (uint32_t j = threadIdx.x; j < o.njobs; j += 256) left |= deep_jobs[o.job0 + j] != 0u;
    if (__syncthreads_or(left)) return;
    for (uint32_t v = blockIdx.x * 256 + threadIdx.x; v < o.n; v += gridDim.x * 256) {
        const double *q = jobbc + o.out0 + v;
        double *b = o.bc + o.map[v];
        double s = *b;
#pragma unroll 4
        for (uint32_t j = 0; j < o.njobs; ++j) s += __ldcs(q + (size_t)j * o.n);
        *b = s;
    }
}

// ---------------------------------------------------------------------------
// Which sources share a job.  A vertex costs a sweep of its list's rows at
// every level at which some slot of the job holds it, so slots whose searches
// run in step cost less: the levels of a source next to a hub come one
// earlier than those of a source two steps away.  Sources are ordered by what
// their second level reaches, the sum of their neighbours' degrees (of 512 of
// them, evenly spaced, where there are more), in the searched graph.  (Kernel
// time as given -> by their own degree -> by this, keys and order included: 174
// roots of a 260k-vertex R-MAT graph 4.89 -> 4.23 -> 3.90 ms, 658 of a 1M-vertex
// one with pendant trees 54.2 -> 48.2 -> 37.8, all 2,839 of a 4096-vertex one
// 0.98 -> 0.85 -> 0.85.)
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_wide_keys(const WideSub *__restrict__ sub, const uint32_t *__restrict__ roots,
                                                   uint32_t nroots, uint32_t *__restrict__ key) {
    const uint32_t i = (blockIdx.x * 256u + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (i >= nroots) return;
    const uint32_t v = sub->inv[roots[i]], b = sub->offs[1][v], deg = sub->offs[1][v + 1] - b, m = min(deg, 512u);
    unsigned long long s = 0;
#pragma unroll 4
    for (uint32_t j = lane; j < m; j += 32u) {
        const uint32_t e = m == deg ? j : (uint32_t)((unsigned long long)j * deg / m);
        s += sub->vinfo[sub->adj[1][b + e]].x;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    if (m < deg) s = s / m * deg;
    if (lane == 0) key[i] = (uint32_t)min(s, 0xFFFFFFFFull);
}

// Orders every kWideWindow sources by descending key, the given order among
// equals (a place is the number of sources before it: each is compared with all).
constexpr uint32_t kWideWindow = 8192;
__global__ void __launch_bounds__(256) k_wide_rank(const uint32_t *__restrict__ key, const uint32_t *__restrict__ roots,
                                                   const double *__restrict__ mult, uint32_t nroots,
                                                   uint32_t *__restrict__ roots_to, double *__restrict__ mult_to,
                                                   uint32_t *__restrict__ order) {
    __shared__ uint32_t k[256];
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;  // a block lies in one window
    const uint32_t w0 = blockIdx.x * 256u / kWideWindow * kWideWindow, w1 = min(nroots, w0 + kWideWindow);
    const uint32_t mine = i < nroots ? key[i] : 0u;
    uint32_t place = w0;
    for (uint32_t t = w0; t < w1; t += 256u) {
        __syncthreads();
        k[threadIdx.x] = t + threadIdx.x < w1 ? key[t + threadIdx.x] : 0u;
        __syncthreads();
        const uint32_t m = min(256u, w1 - t);
        for (uint32_t j = 0; j < m; ++j) place += k[j] > mine || (k[j] == mine && t + j < i);
    }
    if (i >= nroots) return;
    roots_to[place] = roots[i];
    if (mult) mult_to[place] = mult[i];
    if (order) order[place] = i;
}

#define CKW(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return set_error(e_ == cudaErrorMemoryAllocation ? BCG_ERR_OOM : BCG_ERR_CUDA, "%s failed: %s", \
                             #call, cudaGetErrorString(e_));                                       \
    } while (0)

size_t up256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

void preload_wide() {
    cudaFuncAttributes at;
    cudaFuncGetAttributes(&at, (const void *)bc_wide_kernel<16>);
    cudaFuncGetAttributes(&at, (const void *)bc_wide_kernel<32>);
    cudaFuncGetAttributes(&at, (const void *)k_wide_reduce);
    preload_wide_form();
}

int wide_order(const WideSub *sub, const uint32_t *roots, const double *mult, uint32_t nroots, uint32_t *key,
               uint32_t *roots_to, double *mult_to, uint32_t *order, cudaStream_t st) {
    k_wide_keys<<<(unsigned)(((size_t)nroots + 7) / 8), 256, 0, st>>>(sub, roots, nroots, key);
    k_wide_rank<<<(nroots + 255u) / 256u, 256, 0, st>>>(key, roots, mult, nroots, roots_to, mult_to, order);
    CKW(cudaGetLastError());
    return BCG_OK;
}

size_t wide_layout(WideArgs &a, uint32_t slots, size_t n, size_t nchunk, size_t nheavy) {
    const size_t words = (n + 31) / 32;
    size_t o = up256(n * slots);
    a.slots = slots;
    a.o_done = o; o += up256(words * 4);
    a.o_act = o; o += up256(words * 4 * kWideLevels);
    a.o_sig = o; o += up256(n * slots * 8);
    a.o_g0 = o; o += up256((n + 1) * slots * 8);
    a.o_g1 = o; o += up256((n + 1) * slots * 8);
    a.o_part = o; o += up256(std::max<size_t>(1, nchunk) * slots * 8);
    a.o_hcnt = o; o += up256(std::max<size_t>(1, nheavy) * 4);
    a.o_bits = o; o += up256((n + 1) * 4);
    a.stride = o;
    a.words = words;
    return o;
}

double wide_teams(WideArgs &a, uint64_t njobs, uint64_t entries, size_t state_bytes) {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // A job on a team of T CTAs takes about 70 us of barriers and latency, and
    // its entries at 9 ns an entry and CTA, 1.1 times that once the teams'
    // rows are well beyond L2 (fitted on 16-source jobs of R-MAT graphs: 0.1 M
    // entries 540 us on 1 CTA; 7.1 M entries 6,050 us on 13 and 590 us on 148;
    // 30 M entries 8,800 us on 29 and 1,590 us on 148), and a job of 32
    // sources 1.3 to 1.7 times one of 16 (414 us on 3 CTAs, 2,690 us on 148).  The number of teams that ends first, its
    // states within state_bytes.
    const double entry = a.slots == 32 ? 0.009 * kWide32 : 0.009, fixed = 70.0, beyond = 1.1;
    double best = 0.0;
    for (uint64_t t = 1; t <= std::min<uint64_t>({njobs, (uint64_t)nsm, kWideTeams}); ++t) {
        if (t > 1 && a.stride * t > state_bytes) break;
        const double rows = (double)t * (double)a.words * 32.0 * 8.0 * a.slots;
        const double job = fixed + (double)entries * entry * (rows > 126e6 ? beyond : 1.0) / (double)(nsm / t);
        const double all = (double)((njobs + t - 1) / t) * job;
        if (t == 1 || all < best) {
            best = all;
            a.teams = (uint32_t)t;
        }
    }
    a.team_ctas = (uint32_t)nsm / a.teams;
    return best;
}

uint32_t wide_plan(WideArgs &a, uint64_t nroots, uint64_t entries, size_t n, size_t nchunk, size_t nheavy,
                   size_t state_bytes) {
    WideArgs b = a;
    wide_layout(a, 16, n, nchunk, nheavy);
    const double t16 = wide_teams(a, (nroots + 15) / 16, entries, state_bytes);
    wide_layout(b, 32, n, nchunk, nheavy);
    if (b.stride > state_bytes && a.stride <= state_bytes) return 16;
    if (wide_teams(b, (nroots + 31) / 32, entries, state_bytes) >= t16) return 16;
    a = b;
    return 32;
}

int wide_enqueue(const WideArgs &a, const WideOut *outs, uint32_t nouts, const WideOut &one, uint32_t nmax,
                 cudaStream_t st) {
    WideArgs args = a;
    void *params[] = {&args};
    CKW(cudaLaunchCooperativeKernel(a.slots == 32 ? (const void *)bc_wide_kernel<32> : (const void *)bc_wide_kernel<16>,
                                    dim3(a.teams * a.team_ctas), dim3(kWideThreads),
                                    params, 0, st));
    const unsigned bx = (unsigned)std::max<size_t>(1, ((size_t)nmax + 31) / 32);
    // (65535 graphs at most in the second dimension)
    for (uint32_t o = 0; o < nouts; o += 65535u)
        k_wide_reduce<<<dim3(bx, std::min(65535u, nouts - o)), 256, 0, st>>>(a.ctrl, a.poison, outs ? outs + o : nullptr,
                                                                           one, a.jobbc);
    CKW(cudaGetLastError());
    return BCG_OK;
}

int wide_chain(const WideArgs &a, const WideOut *outs, uint32_t nouts, uint32_t nmax, const uint32_t *deep_jobs,
               cudaStream_t st) {
    const unsigned bx = (unsigned)std::max<size_t>(1, std::min<size_t>(1024, ((size_t)nmax + 255) / 256));
    for (uint32_t o = 0; o < nouts; o += 65535u)
        k_wide_chain<<<dim3(bx, std::min(65535u, nouts - o)), 256, 0, st>>>(a.poison, outs + o, a.jobbc, deep_jobs);
    CKW(cudaGetLastError());
    return BCG_OK;
}

// What a graph keeps for its wide runs (bcg_graph::wide).
struct WideGraph {
    WideForm form;
};

void wide_free(bcg_graph *g) {
    WideGraph *w = g->wide;
    if (!w) return;
    wide_form_free(w->form);
    delete w;
    g->wide = nullptr;
}

WideInput wide_input(const bcg_graph *g) {
    WideInput in{};
    in.n = g->tile_n ? g->tile_n : g->n;
    in.nnz = g->nnz_pruned;
    in.offs = g->d_offs;
    in.adj = g->d_adj;
    in.vinfo = g->d_vinfo;
    in.ext = g->d_ext;
    in.directed = (g->flags & BCG_DIRECTED) != 0;
    in.graphs = 1;
    in.big_nnz = in.nnz;
    return in;
}

int wide_run(bcg_graph *g, const uint32_t *roots, const double *mult, uint64_t nroots, cudaStream_t st, WideResult *res) {
    *res = WideResult{};
    int rc;
    // (out of memory: the caller's other kernels need less)
    if (!g->wide) {
        g->wide = new WideGraph();
        if ((rc = wide_form_make(g->wide->form, wide_input(g), true))) {
            wide_free(g);
            if (rc != BCG_ERR_OOM) return rc;
            cudaGetLastError();
            clear_error();
            return BCG_OK;
        }
        if (st != 0) CKW(cudaStreamSynchronize(0));  // the form that stream 0 made is ready for any stream
    }
    WideGraph *w = g->wide;
    const WideSub &b = w->form.subs[0];  // (bounds, on a small graph)
    const size_t n = b.n;
    WideArgs a{};
    const uint32_t slots = wide_plan(a, nroots, g->nnz_pruned, n, std::max(b.nchunk[0], b.nchunk[1]), b.nheavy);
    const uint64_t njobs = (nroots + slots - 1) / slots;
    // jobs of one launch: their vectors stay under 512 MB
    const uint64_t jl = std::min(njobs, std::max<uint64_t>(a.teams, (512ull << 20) / (n * 8 + 1)));
    // control words, teams, per-source totals (cleared together), the order
    // the sources run in; weights and sources (one upload), the same in that
    // order, and its keys; job vectors; states
    // (jobs that all run at once end with the slowest: making them alike in
    // themselves makes them unlike one another, so the given order stays)
    const bool sorted = njobs > a.teams;
    const size_t o_team = sizeof(WideCtrl), o_rstat = o_team + a.teams * sizeof(WideTeam),
                 o_order = o_rstat + njobs * slots * sizeof(RootStat), stat = o_order + (sorted ? nroots * 4 : 0),
                 o_blob = up256(stat), o_roots = up256(nroots * 8), blob = o_roots + up256(nroots * 4),
                 o_sorted = o_blob + up256(blob), o_jobbc = o_sorted + (sorted ? blob + up256(nroots * 4) : 0),
                 o_state = o_jobbc + up256(jl * n * 8), need = o_state + a.stride * a.teams;
    Workspace ws;
    const cudaError_t took = ws.take(need, st);
    if (took == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return BCG_OK;
    }
    CKW(took);
    unsigned char *const mem = ws.mem;
    std::vector<unsigned char> h(blob), hs(stat);
    memcpy(h.data(), mult, nroots * 8);
    memcpy(h.data() + o_roots, roots, nroots * 4);
    CKW(cudaMemcpyAsync(mem + o_blob, h.data(), blob, cudaMemcpyHostToDevice, st));
    a.subs = w->form.d_subs;
    a.nroots = (uint32_t)nroots;
    a.mult = reinterpret_cast<const double *>(mem + o_blob);
    a.roots = reinterpret_cast<const uint32_t *>(mem + o_blob + o_roots);
    a.jobbc = reinterpret_cast<double *>(mem + o_jobbc);
    a.state = mem + o_state;
    a.ctrl = reinterpret_cast<WideCtrl *>(mem);
    a.team = reinterpret_cast<WideTeam *>(mem + o_team);
    TraceRec *d_trace = nullptr;
    unsigned int *d_tcnt = nullptr;
    const char *trace_path = getenv("BCG_TRACE_FILE");
    if (trace_path && *trace_path) {
        a.trace_cap = 1u << 20;
        CKW(dev_alloc(&d_trace, a.trace_cap * sizeof(TraceRec)));
        CKW(dev_alloc(&d_tcnt, sizeof(unsigned int)));
        CKW(cudaMemsetAsync(d_tcnt, 0, sizeof(unsigned int), 0));
        CKW(cudaStreamSynchronize(0));
        a.trace = d_trace;
        a.trace_cnt = d_tcnt;
    }
    CKW(cudaMemsetAsync(mem, 0, stat, st));
    CKW(cudaEventRecord(g->ev0, st));
    // The jobs are added into bc on the device only if none of them stopped.
    // Several launches add one after the other, so bc is saved before them.
    const bool several = jl < njobs;
    if (several) {
        if (!g->d_bc_save) CKW(tmp_alloc(&g->d_bc_save, (size_t)g->n * sizeof(double), st));
        CKW(cudaMemcpyAsync(g->d_bc_save, g->d_bc, (size_t)g->n * sizeof(double), cudaMemcpyDeviceToDevice, st));
    }
    if (sorted) {
        unsigned char *to = mem + o_sorted;
        if ((rc = wide_order(a.subs, a.roots, a.mult, (uint32_t)nroots, reinterpret_cast<uint32_t *>(to + blob),
                             reinterpret_cast<uint32_t *>(to + o_roots), reinterpret_cast<double *>(to),
                             reinterpret_cast<uint32_t *>(mem + o_order), st)))
            return rc;
        a.roots = reinterpret_cast<const uint32_t *>(to + o_roots);
        a.mult = reinterpret_cast<const double *>(to);
        res->launches += 2;
    }
    const WideCtrl *c = reinterpret_cast<const WideCtrl *>(hs.data());
    for (uint64_t j0 = 0; j0 < njobs; j0 += jl) {
        a.njobs = (uint32_t)std::min(jl, njobs - j0);
        a.job0 = (uint32_t)j0;
        a.rstat = reinterpret_cast<RootStat *>(mem + o_rstat) + j0 * slots;
        if (j0) CKW(cudaMemsetAsync(mem, 0, o_rstat, st));
        if ((rc = wide_enqueue(a, nullptr, 1, WideOut{0, a.njobs, (uint32_t)n, w->form.map, g->d_bc, w->form.d_subs}, (uint32_t)n, st)))
            return rc;
        res->launches += 2;
        const bool last = j0 + a.njobs >= njobs;
        if (last) CKW(cudaEventRecord(g->ev1, st));
        CKW(cudaMemcpyAsync(hs.data(), mem, last ? stat : sizeof(WideCtrl), cudaMemcpyDeviceToHost, st));
        CKW(cudaStreamSynchronize(st));
        ws.waited = last || c->error || c->overflow || c->deep;
        if (c->error || c->overflow || c->deep) break;
    }
    if (d_trace) {
        unsigned int cnt = 0;
        CKW(cudaMemcpy(&cnt, d_tcnt, sizeof(cnt), cudaMemcpyDeviceToHost));
        std::vector<TraceRec> recs(cnt);
        if (cnt) CKW(cudaMemcpy(recs.data(), d_trace, cnt * sizeof(TraceRec), cudaMemcpyDeviceToHost));
        if (FILE *f = fopen(trace_path, "a")) {
            fprintf(f, "# wide roots %zu vertices %zu teams %u x %u\n", (size_t)nroots, n, a.teams, a.team_ctas);
            for (const TraceRec &r : recs)
                fprintf(f, "%u,%u,%u,%u,%llu,%llu\n", r.batch, r.kind, r.level, r.nwork, r.disc, r.t_ns);
            fclose(f);
        }
        dev_free(d_trace);
        dev_free(d_tcnt);
    }
    if (c->error) return set_error(c->error, "device reported error %d (a bounded wait gave up)", c->error);
    if (c->overflow || c->deep) {
        // an overflowing count or a deep search: for the caller's other kernels
        if (several)
            CKW(cudaMemcpyAsync(g->d_bc, g->d_bc_save, (size_t)g->n * sizeof(double), cudaMemcpyDeviceToDevice, st));
        res->launches = 0;
        res->overflow = c->overflow != 0;
        res->deep = c->deep != 0;
        return BCG_OK;
    }
    res->rstat.resize(njobs * slots);
    const RootStat *rs = reinterpret_cast<const RootStat *>(hs.data() + o_rstat);
    const uint32_t *order = reinterpret_cast<const uint32_t *>(hs.data() + o_order);
    for (uint64_t i = 0; i < nroots; ++i) res->rstat[sorted ? order[i] : i] = rs[i];
    res->batches = njobs;
    res->slots = slots;
    res->done = true;
    return BCG_OK;
}

}  // namespace bcg
