// Searches of deep, sparse graphs (sm_100a): grids, meshes and chains, whose
// searches have thousands of levels of a few thousand vertices.
//
// What bounds it.  There is next to no data in a level (a 2048 x 2048 grid:
// 3,960 levels of about 1,060 vertices a source), so a level costs what its
// chain of dependent loads and its barrier cost.  A sweep over the whole
// chip pays a grid barrier and its work lists for every level and batch of
// six sources: about 28 us.  Here a CTA, or a cluster of up to 16 where there
// are fewer sources than would fill the chip, runs one source by itself: the
// barrier is __syncthreads or the cluster's, and sources are independent.
// A level's states lie far apart, each load its own sector: an SM issues one
// of those in about 3 cycles and an atomic in about 10, so large frontiers
// want several SMs.  (2048 x 2048 grid, a forward and a backward level
// together, clusters of 4, 5, 8, 12 and 16: 14.0, 12.5, 9.2, 7.9 and 7.5 us.
// 300 x 290 grid, 150 vertices a level: 9.1 us with one CTA, 6.3 with 4; there
// it is a chain of latencies: on the way forward two round trips to L2 (1,300
// cycles each), the sum and the queue (1,500), the barrier (1,600); on the way
// back one round trip, the sum (1,000) and the barrier.)
//   - vertices have at most 4 (or 8) neighbours, kept as one 16-byte (two)
//     row, so there is no row start to look up first;
//   - the frontier is a queue in shared memory that carries each vertex's
//     neighbour row, read when the vertex was found; in a cluster it stays in
//     the finder's CTA while the CTAs' shares are about even, and is dealt to
//     all by the warp otherwise;
//   - one pass a level: the vertices of level d read the states of their
//     neighbours once, which gives both the sum over the parents (level d - 1,
//     finished) and the neighbours not reached yet, which are claimed for
//     level d + 1 while their own neighbour rows are already being loaded.
//     Two dependent L2 round trips a level;
//     A vertex also notes which neighbours lie deeper, so that the backward
//     pass reads its children only;
//   - backward, the vertices of a level are loaded two levels ahead and their
//     rows and counts one ahead, so one round trip (the children's values) is
//     left.
// Sums run over a vertex's neighbours in list order, so they do not depend on
// the order of the queue.  Every source's dependencies go to a vector of
// their own, and k_deep_reduce adds the vectors in source order.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "bcg_common.hpp"
#include "engine_internal.hpp"
#include "ext64.cuh"

namespace cg = cooperative_groups;

namespace bcg {

namespace {

constexpr int kDeepThreads = 512;      // most of a CTA
constexpr uint32_t kDeepCluster = 16;  // most CTAs of a source
constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kNone = 0xffffffffu;    // no neighbour
constexpr uint32_t kUnseen = 0xffffffffu;  // level of a vertex not reached

// What is kept of a vertex for a source: forward the path count (0: not
// reached), the level and which neighbours are one level deeper; the backward
// pass replaces the count by X = (1 + delta) / count and the rest by delta.
struct alignas(16) DeepState {
    unsigned long long val;
    uint32_t lvl, kids;
};

struct DeepCtrl {
    int overflow, deep, full;  // full: a queue of a cluster ran over
    uint32_t pad[29];
};

struct DeepArgs {
    uint32_t n, nroots;
    const uint32_t *ell;    // n rows of D neighbours, kNone where there is none
    const uint2 *vinfo;     // {degree, reach}; nullptr: every reach is 0
    const uint32_t *roots;
    DeepState *state;       // per source: n
    uint32_t *order;        // per source: n, the vertices by level
    uint32_t *lbeg;         // per source: kMaxLevel + 3, where a level starts in order
    RootStat *rstat;        // per source (zeroed)
    DeepCtrl *ctrl;
    uint32_t cluster;       // CTAs of a source
};

template <int D>
struct Row {
    uint32_t u[D];
};

template <int D>
__device__ __forceinline__ Row<D> ell_row(const uint32_t *ell, uint32_t v) {
    Row<D> r;
#pragma unroll
    for (int h = 0; h < D / 4; ++h) {
        const uint4 t = __ldg(reinterpret_cast<const uint4 *>(ell + (size_t)v * D) + h);
        r.u[4 * h] = t.x; r.u[4 * h + 1] = t.y; r.u[4 * h + 2] = t.z; r.u[4 * h + 3] = t.w;
    }
    return r;
}

// States are written by other threads of the cluster: always read from L2.
__device__ __forceinline__ void ld_state(const DeepState *p, unsigned long long &val, uint32_t &lvl, uint32_t &kids) {
    uint32_t a, b;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(a), "=r"(b), "=r"(lvl), "=r"(kids) : "l"(p) : "memory");
    val = (unsigned long long)b << 32 | a;
}

// Adds the terms that bit q of `which` names, x[q], in order of q, one of
// them a step: a warp takes as many steps as one of its lanes has terms (two
// on most of a grid's levels, and the first costs no addition).
template <int D, class T, class Add>
__device__ __forceinline__ T add_terms(const unsigned long long (&x)[D], uint32_t which, Add add) {
    T sum = T();
#pragma unroll 1
    for (bool first = true; which; first = false) {
        const uint32_t q = (uint32_t)__ffs(which) - 1u;
        which &= which - 1u;
        unsigned long long t = x[0];
#pragma unroll
        for (int k = 1; k < D; ++k) t = q == (uint32_t)k ? x[k] : t;
        sum = add(sum, t, first);
    }
    return sum;
}

__device__ __forceinline__ unsigned long long ld_val(const DeepState *p) {
    unsigned long long v;
    asm volatile("ld.global.cg.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Entries a queue holds in shared memory (two queues); a larger frontier's
// tail is read back from the order list.
template <int D>
constexpr uint32_t queue_cap() { return D == 4 ? 5000u : 2700u; }

template <bool EXT>
struct SumOf { using T = double; };
template <>
struct SumOf<true> { using T = unsigned long long; };

template <int D>
struct DeepSmem {
    uint32_t v[2][queue_cap<D>()];
    Row<D> nb[2][queue_cap<D>()];
    uint32_t cnt[3];  // ring: vertices found for a level, cleared a level ahead
    uint32_t stop;    // level whose sums overflowed (all ones: none)
    unsigned long long tot[3];
};

// Barrier of the CTAs of a source.
__device__ __forceinline__ void source_sync(uint32_t C) {
    if (C == 1) __syncthreads();
    else cg::this_cluster().sync();
}
template <class T>
__device__ __forceinline__ T *peer(T *p, uint32_t C, uint32_t rank) {
    return C == 1 ? p : cg::this_cluster().map_shared_rank(p, rank);
}

template <int D, bool EXT>
__global__ void __launch_bounds__(kDeepThreads, 1) bc_deep_kernel(DeepArgs a) {
    extern __shared__ __align__(16) unsigned char deep_raw[];
    static_assert(D <= 8, "neighbours of a row");
    DeepSmem<D> &sm = *reinterpret_cast<DeepSmem<D> *>(deep_raw);
    constexpr uint32_t Q = queue_cap<D>();
    const uint32_t C = a.cluster, s = blockIdx.x / C, rank = blockIdx.x % C;
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    DeepState *state = a.state + (size_t)s * a.n;
    uint32_t *order = a.order + (size_t)s * a.n;
    uint32_t *lbeg = a.lbeg + (size_t)s * (kMaxLevel + 3);
    if (tid == 0) {
        sm.cnt[0] = rank == 0;
        sm.cnt[1] = sm.cnt[2] = 0;
        sm.stop = kNone;
        if (rank == 0) {
            const uint32_t root = a.roots[s];
            state[root] = DeepState{EXT ? kExtOne : 1ull, 0u, 0u};
            sm.v[0][0] = root;
            sm.nb[0][0] = ell_row<D>(a.ell, root);
        }
    }
    if (tid < 3) sm.tot[tid] = 0ull;
    source_sync(C);
    // ---- forward: one pass a level
    const uint32_t logC = 31u - __clz(C);
    uint32_t d = 0, base = 0;  // the level, its place in order
    unsigned long long vis = 0, wsum = 0, mc2 = 0;
    bool too_deep = false;
    for (;; ++d) {
        const uint32_t ring = d % 3u, cnt = sm.cnt[ring];  // the level's vertices in this CTA's queue,
        uint32_t size = cnt, first = base;                 // in all, and where this CTA's start in order
        // (the other CTAs' counts are asked for here and used once the level's
        // own loads are on their way)
        const uint32_t mine = C == 1 ? 0u : (lane < C ? *peer(&sm.cnt[ring], C, lane) : 0u);
        bool known = C == 1, deal = false;
        auto counts = [&]() {
            if (known) return;
            known = true;
            size = __reduce_add_sync(kFull, mine);
            first = base + __reduce_add_sync(kFull, lane < rank ? mine : 0u);
            // What a CTA finds stays with it while the CTAs' shares differ by
            // little and cannot outgrow a queue; else the warps' finds are
            // dealt to all.
            const uint32_t most = __reduce_max_sync(kFull, mine);
            deal = most > (size >> logC) + (size >> (logC + 2u)) + 32u || most > Q / (D - 1);
        };
        // (one barrier a level: what a faster thread has written since is the
        // next level's, in another entry of the ring, with a higher stop level)
        if (d && sm.stop < d) {
            if (tid == 0 && rank == 0) a.ctrl->overflow = 1;
            break;
        }
        const uint32_t c = d & 1u, to = (d + 1u) % 3u;
        int seen_stop = 0;
        if (tid == 0 && (d & 31u) == 0) seen_stop = *reinterpret_cast<volatile int *>(&a.ctrl->overflow);
        for (uint32_t i0 = tid & ~31u; i0 < cnt; i0 += blockDim.x) {
            const uint32_t i = i0 + lane;
            const bool has = i < cnt;
            uint32_t v = 0;
            Row<D> nb;
#pragma unroll
            for (int q = 0; q < D; ++q) nb.u[q] = kNone;
            if (has) {
                if (i < Q) {
                    v = sm.v[c][i];
                    nb = sm.nb[c][i];
                } else {
                    v = __ldcg(order + first + i);
                    nb = ell_row<D>(a.ell, v);
                }
            }
            uint32_t lv[D];
            unsigned long long val[D];
            Row<D> far[D];
#pragma unroll
            for (int q = 0; q < D; ++q) {
                lv[q] = d;
                val[q] = 0ull;
                uint32_t unused;
                if (nb.u[q] != kNone) ld_state(state + nb.u[q], val[q], lv[q], unused);
            }
            // claim the neighbours not reached yet, their rows on the way (an
            // SM issues an atomic in about 10 cycles: none is spent on others)
#pragma unroll
            for (int q = 0; q < D; ++q) {
                if (lv[q] == kUnseen) {
                    lv[q] = atomicExch(&state[nb.u[q]].lvl, d + 1u);
                    if (D == 4) far[q] = ell_row<D>(a.ell, nb.u[q]);
                }
            }
            uint32_t reach = 0;
            if (has && a.vinfo) reach = a.vinfo[v].y;
            counts();
            if (has && i < Q) order[first + i] = v;
            uint32_t won[D], total = 0;
#pragma unroll
            for (int q = 0; q < D; ++q) {
                won[q] = __ballot_sync(kFull, lv[q] == kUnseen);
                total += __popc(won[q]);
            }
            const uint32_t dest = deal ? ((i0 >> 5) + rank + d) & (C - 1u) : rank;
            uint32_t at = 0;
            if (total && lane == 0) at = dest == rank ? atomicAdd(&sm.cnt[to], total) : atomicAdd(peer(&sm.cnt[to], C, dest), total);
            if (has) {
                uint32_t kids = 0, parents = 0, deg = 0;
                bool ovf = false;
#pragma unroll
                for (int q = 0; q < D; ++q) {
                    if (nb.u[q] == kNone) continue;
                    ++deg;
                    if (lv[q] == kUnseen || lv[q] == d + 1u) kids |= 1u << q;
                    if (lv[q] + 1u == d) parents |= 1u << q;
                }
                unsigned long long sum = add_terms<D, unsigned long long>(
                    val, parents, [&](unsigned long long x, unsigned long long y, bool one) {
                        if (one) return y;
                        if (EXT) return ext_add(x, y);
                        ovf |= x + y < y;
                        return x + y;
                    });
                if (d == 0) sum = EXT ? kExtOne : 1ull;
                *reinterpret_cast<uint4 *>(state + v) = make_uint4((uint32_t)sum, (uint32_t)(sum >> 32), d, kids);
                if (ovf) seen_stop = 1;
                ++vis;
                wsum += 1ull + reach;
                mc2 += (unsigned long long)deg + 2ull * reach;
            }
            __syncwarp();
            if (total) {
                at = __shfl_sync(kFull, at, 0);
                uint32_t *qv = dest == rank ? &sm.v[c ^ 1u][0] : peer(&sm.v[c ^ 1u][0], C, dest);
                Row<D> *qn = dest == rank ? &sm.nb[c ^ 1u][0] : peer(&sm.nb[c ^ 1u][0], C, dest);
#pragma unroll
                for (int q = 0; q < D; ++q) {
                    if ((won[q] >> lane) & 1u) {
                        const uint32_t p = at + __popc(won[q] & ((1u << lane) - 1u));
                        if (p < Q) {
                            qv[p] = nb.u[q];
                            qn[p] = D == 4 ? far[q] : ell_row<D>(a.ell, nb.u[q]);
                        } else if (C == 1) {
                            order[base + size + p] = nb.u[q];
                        } else {
                            a.ctrl->full = 1;  // the host runs it again with one CTA a source
                            seen_stop = 1;
                        }
                    }
                    at += __popc(won[q]);
                }
            }
        }
        counts();
        too_deep = size && d > kMaxLevel;
        if (!size || too_deep) break;
        if (tid == 0 && rank == 0) lbeg[d] = base;
        if (seen_stop)
            for (uint32_t k = 0; k < C; ++k) *peer(&sm.stop, C, k) = d;
        // (last read two barriers ago)
        if (tid == 0) sm.cnt[(d + 2u) % 3u] = 0;
        source_sync(C);
        base += size;
    }
    if (too_deep || (d && sm.stop < d)) {
        if (too_deep && tid == 0 && rank == 0) a.ctrl->deep = 1;
        source_sync(C);  // no CTA leaves while another may still read its counts
        return;
    }
    const uint32_t depth = d - 1u;
    if (tid == 0 && rank == 0) lbeg[d] = base;
    // ---- what the source reached
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        vis += __shfl_xor_sync(kFull, vis, o);
        wsum += __shfl_xor_sync(kFull, wsum, o);
        mc2 += __shfl_xor_sync(kFull, mc2, o);
    }
    if (lane == 0) {
        atomicAdd(&sm.tot[0], vis);
        atomicAdd(&sm.tot[1], wsum);
        atomicAdd(&sm.tot[2], mc2);
    }
    source_sync(C);
    if (tid == 0) {
        RootStat *rs = a.rstat + s;
        atomicAdd(&rs->visited, sm.tot[0]);
        atomicAdd(&rs->wsum, sm.tot[1]);
        atomicAdd(&rs->mc2, sm.tot[2]);
        if (rank == 0) rs->depth = depth;
    }
    // ---- backward: levels depth .. 1.  Of level e - 1 the vertex of each
    // thread is known (v1) and its row and state are loaded while level e is
    // worked on; of level e - 2 the vertex is loaded.
    // (a level's warps are dealt to the CTAs in turn)
    const uint32_t t0 = ((tid >> 5) * C + rank) * 32u + lane, per = C * blockDim.x;
    using Sum = typename SumOf<EXT>::T;
    struct Item {
        uint32_t v;
        Row<D> nb;
        unsigned long long sig;
        uint32_t kids, reach;
    };
    auto load = [&](Item &it) {
        it.nb = ell_row<D>(a.ell, it.v);
        uint32_t lvl;
        ld_state(state + it.v, it.sig, lvl, it.kids);
        it.reach = a.vinfo ? a.vinfo[it.v].y : 0u;
    };
    auto kids_of = [&](const Item &it, unsigned long long (&x)[D]) {
#pragma unroll
        for (int q = 0; q < D; ++q)
            if ((it.kids >> q) & 1u) x[q] = ld_val(state + it.nb.u[q]);
    };
    auto finish = [&](const Item &it, const unsigned long long (&x)[D]) {
        const Sum sum = add_terms<D, Sum>(x, it.kids, [&](Sum s, unsigned long long y, bool one) -> Sum {
            if constexpr (EXT) return one ? y : ext_add(s, y);
            else return s + __longlong_as_double((long long)y);
        });
        double dl;
        unsigned long long xo;
        if constexpr (EXT) {
            dl = (double)it.reach + ext_to_double(ext_mul(it.sig, sum));
            xo = ext_div(1.0 + dl, it.sig);
        } else {
            dl = (double)it.reach + (double)it.sig * sum;
            xo = (unsigned long long)__double_as_longlong((1.0 + dl) / (double)it.sig);
        }
        *reinterpret_cast<uint4 *>(state + it.v) =
            make_uint4((uint32_t)xo, (uint32_t)(xo >> 32), (uint32_t)__double2loint(dl), (uint32_t)__double2hiint(dl));
    };
    // starts of levels e, e - 1, e - 2
    uint32_t end = base, b0 = __ldcg(lbeg + depth), b1 = depth >= 2u ? __ldcg(lbeg + depth - 1) : 0u;
    Item even{}, odd{};
    uint32_t v1 = 0;
    if (t0 < end - b0) {
        even.v = __ldcg(order + b0 + t0);
        load(even);
    }
    if (depth >= 2u && t0 < b0 - b1) v1 = __ldcg(order + b1 + t0);
    auto level = [&](uint32_t e, Item &it, Item &nx) {
        const uint32_t n0 = end - b0, n1 = e >= 2u ? b0 - b1 : 0u;
        const uint32_t b2 = e >= 3u ? __ldcg(lbeg + e - 2) : 0u;
        unsigned long long x[D];
        if (t0 < n0) kids_of(it, x);
        nx.v = v1;
        if (t0 < n1) load(nx);
        if (t0 < n0) finish(it, x);
        for (uint32_t i = t0 + per; i < n0; i += per) {
            it.v = __ldcg(order + b0 + i);
            load(it);
            kids_of(it, x);
            finish(it, x);
        }
        if (e >= 3u && t0 < b1 - b2) v1 = __ldcg(order + b2 + t0);
        end = b0;
        b0 = b1;
        b1 = b2;
        source_sync(C);
    };
    for (uint32_t e = depth; e >= 1u; --e) {
        level(e, even, odd);
        if (--e == 0u) break;
        level(e, odd, even);
    }
    // the source's own dependencies do not count
    if (rank == 0 && tid == 0) state[a.roots[s]] = DeepState{1ull, 0u, 0u};
}

__global__ void k_deep_init(uint64_t cells, DeepState *__restrict__ state) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cells; i += (uint64_t)gridDim.x * blockDim.x)
        *reinterpret_cast<uint4 *>(state + i) = make_uint4(0u, 0u, kUnseen, 0u);
}

__global__ void k_deep_reduce(const DeepCtrl *__restrict__ ctrl, uint32_t n, uint32_t nroots,
                              const double *__restrict__ mult, const DeepState *__restrict__ state,
                              const uint32_t *__restrict__ ext, double *__restrict__ bc) {
    if (ctrl->overflow | ctrl->deep | ctrl->full) return;  // nothing of a stopped launch is kept
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    double sum = 0.0;
#pragma unroll 4
    for (uint32_t s = 0; s < nroots; ++s) {
        const uint4 t = __ldcs(reinterpret_cast<const uint4 *>(state + (size_t)s * n + v));
        if (t.x | t.y) sum += mult[s] * __hiloint2double((int)t.w, (int)t.z);
    }
    if (sum != 0.0) bc[ext ? ext[v] : v] += sum;
}

// What a source's search says of searches from the vertices that it reached
// (k_levels_low's bound): order's first `reached`, by level from lbeg.
__global__ void k_deep_low(uint32_t reached, uint32_t depth, const uint32_t *__restrict__ order,
                           const uint32_t *__restrict__ lbeg, uint8_t *__restrict__ low) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= reached) return;
    uint32_t l = 0, end = depth;  // the last level that starts at i or before
    while (l < end) {
        const uint32_t mid = (l + end + 1) / 2;
        if (lbeg[mid] <= i) l = mid;
        else end = mid - 1;
    }
    low[order[i]] = (uint8_t)min(max(l, depth - l), 255u);
}

template <int D>
__global__ void k_deep_rows(uint32_t n, const uint32_t *__restrict__ offs, const uint32_t *__restrict__ adj,
                            uint32_t *__restrict__ ell) {
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const uint32_t e0 = offs[v], deg = offs[v + 1] - e0;
#pragma unroll
    for (int q = 0; q < D; ++q) ell[(size_t)v * D + q] = (uint32_t)q < deg ? adj[e0 + q] : kNone;
}

// ---------------------------------------------------------------------------
// Whether a search's frontier grows faster than a mesh's.  kProbes CTAs search
// from vertices spread over the graph until a level of more than 16 + 8 d^2
// vertices is met (a lattice in three dimensions has up to 6 d^2 + 2), or the
// growth is a plane's at level 16 (8 d at most), or kProbeDepth levels or
// kProbeVerts vertices hold neither.  About 2 us a level, once a graph.
// ---------------------------------------------------------------------------
constexpr uint32_t kProbes = 8, kProbeDepth = 40, kProbeVerts = 32768, kProbeScan = 65536;
constexpr int kProbeThreads = 512;

// seen: kProbes bitmaps of `words` words (zeroed); queue: kProbes x (kProbeVerts
// + 8 x kProbeThreads); vote: {probes that started, probes that met a level so
// wide} (zeroed).
template <int D>
__global__ void __launch_bounds__(kProbeThreads) k_deep_probe(uint32_t n, const uint32_t *__restrict__ ell, uint32_t words,
                                                              uint32_t *__restrict__ seen, uint32_t *__restrict__ queue,
                                                              uint32_t *__restrict__ vote) {
    __shared__ uint32_t start, end;
    const uint32_t b = blockIdx.x, tid = threadIdx.x;
    uint32_t *bits = seen + (size_t)b * words, *q = queue + (size_t)b * (kProbeVerts + 8 * kProbeThreads);
    if (tid == 0) {
        start = kNone;
        end = 1;
    }
    __syncthreads();
    // the first vertex with a neighbour in the probe's part
    const uint32_t v0 = (uint32_t)((unsigned long long)n * b / kProbes), v1 = (uint32_t)((unsigned long long)n * (b + 1) / kProbes);
    for (uint32_t v = v0; v < v1 && v - v0 < kProbeScan; v += kProbeThreads) {
        if (v + tid < v1 && ell[(size_t)(v + tid) * D] != kNone) atomicMin(&start, v + tid);
        __syncthreads();
        const bool found = start != kNone;
        __syncthreads();
        if (found) break;
    }
    if (start == kNone) return;
    if (tid == 0) {
        q[0] = start;
        bits[start >> 5] = 1u << (start & 31u);
        atomicAdd(vote, 1u);
    }
    __syncthreads();
    uint32_t d = 0, from = 0, to = 1;  // level d is q[from .. to)
    while (d < kProbeDepth && to < kProbeVerts) {
        for (uint32_t i = from + tid; i < to; i += kProbeThreads) {
            const Row<D> r = ell_row<D>(ell, q[i]);
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const uint32_t u = r.u[k];
                if (u == kNone) continue;
                const uint32_t bit = 1u << (u & 31u);
                if (atomicOr(bits + (u >> 5), bit) & bit) continue;
                const uint32_t at = atomicAdd(&end, 1u);
                if (at < kProbeVerts + 8 * kProbeThreads) q[at] = u;
            }
        }
        __syncthreads();
        const uint32_t last = min(end, kProbeVerts + 8 * kProbeThreads);
        __syncthreads();
        from = to;
        to = last;
        ++d;
        const uint32_t size = to - from;
        if (size > 16u + 8u * d * d) {
            if (tid == 0) atomicAdd(vote + 1, 1u);
            return;
        }
        if (!size || (d == 16 && size <= 8u * d)) return;
    }
}

#define CKD(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return set_error(e_ == cudaErrorMemoryAllocation ? BCG_ERR_OOM : BCG_ERR_CUDA, "%s failed: %s", \
                             #call, cudaGetErrorString(e_));                                       \
    } while (0)

// The launch of a.nroots sources in clusters of up to `most` CTAs (a.cluster):
// as many a source as leave every source room on the chip.  Clusters of more
// than 8 are not promised by the architecture, and fewer of them fit than the
// SMs would allow: the device is asked.
template <int D, bool EXT>
cudaError_t deep_config(DeepArgs &a, uint32_t most, uint32_t nsm, cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at) {
    const void *f = (const void *)bc_deep_kernel<D, EXT>;
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DeepSmem<D>));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    a.cluster = 1;
    while (a.cluster < most && a.nroots * 2 * a.cluster <= nsm) a.cluster *= 2;
    cfg.gridDim = dim3(a.nroots * a.cluster);
    // (threads, measured on 2048 x 2048 vertices: clusters of 16 25.1 ms with
    // 256 and 26.5 with 512, of 8 30.1 and 29.8, of 4 45.8 and 42.0; 148
    // sources of 1000 x 1000, a CTA each: 34.7 and 32.7)
    cfg.blockDim = dim3(a.cluster >= 8 ? kDeepThreads / 2 : kDeepThreads);
    cfg.dynamicSmemBytes = sizeof(DeepSmem<D>);
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = a.cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (a.cluster > 8) {
        int fit = 0;
        e = cudaOccupancyMaxActiveClusters(&fit, f, &cfg);
        if (e != cudaSuccess || (uint32_t)fit < a.nroots) {
            cudaGetLastError();
            at.val.clusterDim.x = a.cluster = 8;
            cfg.gridDim = dim3(a.nroots * 8u);
        }
    }
    return cudaSuccess;
}

template <int D, bool EXT>
cudaError_t launch_deep(DeepArgs &a, uint32_t most, uint32_t nsm, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    const cudaError_t e = deep_config<D, EXT>(a, most, nsm, cfg, at);
    if (e != cudaSuccess) return e;
    cfg.stream = st;
    DeepArgs args = a;
    void *params[] = {&args};
    return cudaLaunchKernelExC(&cfg, (const void *)bc_deep_kernel<D, EXT>, params);
}

}  // namespace

// What a graph keeps for its deep runs (bcg_graph::deep).
struct DeepGraph {
    Workspace ell;
    int width = 0;       // neighbours of a row
    bool broad = false;  // frontiers grow faster than a mesh's (k_deep_probe)
};

void deep_free(bcg_graph *g) {
    if (!g->deep) return;
    delete g->deep;
    g->deep = nullptr;
}

bool deep_takes(const bcg_graph *g) { return !(g->flags & BCG_DIRECTED) && g->max_deg >= 1 && g->max_deg <= 8; }

// Makes g->deep, unless it is there; stays nullptr where there is no memory.
static int deep_make(bcg_graph *g) {
    if (g->deep) return BCG_OK;
    const uint32_t n = g->tile_n ? g->tile_n : g->n, words = (n + 31u) / 32u;
    const int D = g->max_deg <= 4 ? 4 : 8;
    DeepGraph *w = g->deep = new DeepGraph();
    w->width = D;
    Workspace probe;
    const size_t o_seen = 256, o_queue = o_seen + (size_t)kProbes * words * 4,
                 probe_bytes = o_queue + (size_t)kProbes * (kProbeVerts + 8 * kProbeThreads) * 4;
    uint32_t vote[2] = {0, 0};
    cudaError_t e = w->ell.take((size_t)n * D * sizeof(uint32_t), 0, true);
    if (e == cudaSuccess) e = probe.take(probe_bytes, 0);
    if (e == cudaSuccess) e = cudaMemsetAsync(probe.mem, 0, o_queue, 0);
    if (e == cudaSuccess) {
        uint32_t *ell = reinterpret_cast<uint32_t *>(w->ell.mem), *at = reinterpret_cast<uint32_t *>(probe.mem);
        uint32_t *seen = reinterpret_cast<uint32_t *>(probe.mem + o_seen), *queue = reinterpret_cast<uint32_t *>(probe.mem + o_queue);
        if (D == 4) {
            k_deep_rows<4><<<(n + 255) / 256, 256>>>(n, g->d_offs, g->d_adj, ell);
            k_deep_probe<4><<<kProbes, kProbeThreads>>>(n, ell, words, seen, queue, at);
        } else {
            k_deep_rows<8><<<(n + 255) / 256, 256>>>(n, g->d_offs, g->d_adj, ell);
            k_deep_probe<8><<<kProbes, kProbeThreads>>>(n, ell, words, seen, queue, at);
        }
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpy(vote, at, sizeof(vote), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaDeviceSynchronize();  // ready for any stream
        probe.waited = e == cudaSuccess;
    }
    if (e != cudaSuccess) {
        deep_free(g);
        if (e != cudaErrorMemoryAllocation) CKD(e);
        cudaGetLastError();
    } else {
        w->broad = vote[1] && 2 * vote[1] >= vote[0];
    }
    return BCG_OK;
}

// Most sources of a launch: one a CTA, in what a workspace may keep.
static uint64_t deep_slots(uint32_t n, uint64_t nroots, uint32_t nsm) {
    const size_t per = 20 * (size_t)n + (kMaxLevel + 3) * sizeof(uint32_t);
    return std::max<uint64_t>(1, std::min<uint64_t>({nroots, (uint64_t)nsm, kWorkKeep / per}));
}

static int deep_launch(bcg_graph *g, const uint32_t *roots, const double *mult, uint64_t nroots, bool ext, bool note,
                       uint32_t most_ctas, cudaStream_t st, DeepResult *res) {
    *res = DeepResult{};
    const uint32_t n = g->tile_n ? g->tile_n : g->n;
    const int D = g->max_deg <= 4 ? 4 : 8;
    DeepGraph *w = g->deep;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // a source's share: states and order (20 bytes a vertex), level starts; half
    // as many sources where there is no memory; launches of like size (148 sources of 2048 x
    // 2048 vertices: 128 ms in one launch of 12.4 GB, 194 as 102 and 46, 151 as
    // 74 and 74)
    auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
    uint64_t slots = deep_slots(n, nroots, (uint32_t)nsm);
    size_t o = up(sizeof(DeepCtrl));
    const size_t o_rstat = o; o += up(nroots * sizeof(RootStat));
    const size_t o_mult = o; o += up(nroots * sizeof(double));
    const size_t o_roots = o; o += up(nroots * sizeof(uint32_t));
    const size_t o_state = o;
    Workspace ws;
    size_t o_order = 0, o_lbeg = 0;
    for (;; slots /= 2) {
        const uint64_t launches = (nroots + slots - 1) / slots;
        slots = (nroots + launches - 1) / launches;
        o_order = o_state + up(slots * n * sizeof(DeepState));
        o_lbeg = o_order + up(slots * n * sizeof(uint32_t));
        const cudaError_t e = ws.take(o_lbeg + up(slots * (kMaxLevel + 3) * sizeof(uint32_t)), st);
        if (e == cudaSuccess) break;
        if (e != cudaErrorMemoryAllocation) CKD(e);
        cudaGetLastError();
        if (slots == 1) return BCG_OK;
    }
    unsigned char *const mem = ws.mem;
    DeepArgs a{};
    a.n = n;
    a.ell = reinterpret_cast<const uint32_t *>(w->ell.mem);
    a.vinfo = g->trees ? g->d_vinfo : nullptr;
    a.state = reinterpret_cast<DeepState *>(mem + o_state);
    a.order = reinterpret_cast<uint32_t *>(mem + o_order);
    a.lbeg = reinterpret_cast<uint32_t *>(mem + o_lbeg);
    a.ctrl = reinterpret_cast<DeepCtrl *>(mem);
    std::vector<unsigned char> up_(o_state - o_mult), down(o_mult);
    memcpy(up_.data(), mult, nroots * sizeof(double));
    memcpy(up_.data() + (o_roots - o_mult), roots, nroots * sizeof(uint32_t));
    const bool several = slots < nroots;
    CKD(cudaEventRecord(g->ev0, st));
    CKD(cudaMemsetAsync(mem, 0, o_mult, st));  // control words and the sources' totals
    CKD(cudaMemcpyAsync(mem + o_mult, up_.data(), up_.size(), cudaMemcpyHostToDevice, st));
    if (several) {  // launches add to bc one after the other: what it was before them
        if (!g->d_bc_save) CKD(tmp_alloc(&g->d_bc_save, (size_t)g->n * sizeof(double), st));
        CKD(cudaMemcpyAsync(g->d_bc_save, g->d_bc, (size_t)g->n * sizeof(double), cudaMemcpyDeviceToDevice, st));
    }
    const DeepCtrl *c = reinterpret_cast<const DeepCtrl *>(down.data());
    for (uint64_t s0 = 0; s0 < nroots; s0 += slots) {
        a.nroots = (uint32_t)std::min<uint64_t>(slots, nroots - s0);
        a.roots = reinterpret_cast<const uint32_t *>(mem + o_roots) + s0;
        a.rstat = reinterpret_cast<RootStat *>(mem + o_rstat) + s0;
        k_deep_init<<<nsm * 8, 256, 0, st>>>((uint64_t)a.nroots * n, a.state);
        CKD(D == 4 ? (ext ? launch_deep<4, true>(a, most_ctas, nsm, st) : launch_deep<4, false>(a, most_ctas, nsm, st))
                   : (ext ? launch_deep<8, true>(a, most_ctas, nsm, st) : launch_deep<8, false>(a, most_ctas, nsm, st)));
        k_deep_reduce<<<(n + 255) / 256, 256, 0, st>>>(a.ctrl, n, a.nroots,
                                                       reinterpret_cast<const double *>(mem + o_mult) + s0, a.state,
                                                       g->d_ext, g->d_bc);
        CKD(cudaGetLastError());
        res->launches += 3;
        const bool last = s0 + a.nroots >= nroots;
        if (last) CKD(cudaEventRecord(g->ev1, st));
        CKD(cudaMemcpyAsync(down.data(), mem, last ? o_mult : sizeof(DeepCtrl), cudaMemcpyDeviceToHost, st));
        CKD(cudaStreamSynchronize(st));
        ws.waited = last || c->overflow || c->deep || c->full;
        if (c->overflow || c->deep || c->full) break;
    }
    if (c->overflow || c->deep || c->full) {
        if (several)
            CKD(cudaMemcpyAsync(g->d_bc, g->d_bc_save, (size_t)g->n * sizeof(double), cudaMemcpyDeviceToDevice, st));
        // frontiers that do not fit the clusters' queues: one CTA a source
        if (c->full) {
            ws.leave();
            return deep_launch(g, roots, mult, nroots, ext, note, 1, st, res);
        }
        res->overflow = c->overflow != 0;
        return BCG_OK;
    }
    res->rstat.resize(nroots);
    memcpy(res->rstat.data(), down.data() + o_rstat, nroots * sizeof(RootStat));
    res->done = true;
    if (note) {  // (the last launch's first source; its states are not needed any more)
        const RootStat &rs = res->rstat[(nroots - 1) / slots * slots];
        uint8_t *d_low = mem + o_state;
        std::vector<uint8_t> low(n);
        CKD(cudaMemsetAsync(d_low, 0, n, st));
        k_deep_low<<<(unsigned)((rs.visited + 255) / 256), 256, 0, st>>>((uint32_t)rs.visited, rs.depth, a.order, a.lbeg, d_low);
        CKD(cudaGetLastError());
        CKD(cudaMemcpyAsync(low.data(), d_low, n, cudaMemcpyDeviceToHost, st));
        CKD(cudaStreamSynchronize(st));
        merge_levels(g, low);
    }
    return BCG_OK;
}

// Where frontiers are broad the queues of a cluster run over, and one CTA a
// source takes 33 ns a vertex (of three neighbours) where the sweep kernel
// takes 0.3 to 0.5 ms and 1.3 ns a vertex for six sources at once.  The widest
// level of a random 3-regular graph or a binary tree has a quarter of the
// vertices, of a 4-regular one or a tree of 3 children a third, of a tree of 7
// children 0.72: queues that hold that with room for uneven shares do (at 0.80
// of them a tree's ran over, at 0.81 none of the others').  Random 3-regular graph, 1, 6, 24, 48 and 148
// sources, clusters or one CTA a source against the sweep kernel: 2^16 vertices
// 0.22, 0.23, 0.44, 1.3 and 2.2 ms against 0.36, 0.55, 1.9, 3.8 and 12; 2^18
// vertices 0.48, 0.50, 7.0, 8.1 and 10 against 0.49, 0.89, 3.4, 6.6 and 21; 2^20
// vertices 18, 29, 34, 36 and 45 against 0.9, 2.4, 9.2, 18 and 57.  Complete
// binary tree of 2^20 vertices 11, 14, 16, 16 and 17 against 0.7, 1.4, 4.8, 9.5
// and 27.  The rule takes the faster in all of these, or one within 8 % of it, as
// it does on 4-regular graphs and trees of 3 and 7 children (2^14 to 2^21
// vertices, 1 to 400 sources).
int deep_run(bcg_graph *g, const uint32_t *roots, const double *mult, uint64_t nroots, bool ext, bool note,
             cudaStream_t st, DeepResult *res) {
    *res = DeepResult{};
    const int rc = deep_make(g);
    if (rc || !g->deep) return rc;
    uint32_t most = kDeepCluster;
    if (g->deep->broad) {
        const uint32_t n = g->tile_n ? g->tile_n : g->n;
        int dev = 0, nsm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        const uint64_t slots = deep_slots(n, nroots, (uint32_t)nsm), rounds = (nroots + slots - 1) / slots;
        DeepArgs a{};
        a.nroots = (uint32_t)((nroots + rounds - 1) / rounds);
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at{};
        if (g->max_deg <= 4) CKD((deep_config<4, false>(a, kDeepCluster, (uint32_t)nsm, cfg, at)));
        else CKD((deep_config<8, false>(a, kDeepCluster, (uint32_t)nsm, cfg, at)));
        const double queues = (double)a.cluster * (g->max_deg <= 4 ? queue_cap<4>() : queue_cap<8>());
        if (a.cluster == 1 || n > queues * (g->max_deg <= 3 ? 3.3 : (g->max_deg == 4 ? 1.7 : 1.2))) {
            // a CTA's search of so many vertices takes as long as `ratio` of the
            // sweep kernel's for six sources, and those have a fixed part of so
            // many vertices more
            const double mean = (double)g->nnz_pruned / n;
            const double fixed = mean >= 3.5 ? 200e3 : (mean >= 2.5 ? 230e3 : (g->max_deg > 4 ? 400e3 : 600e3));
            const double ratio = mean >= 3.5 ? (n <= (1u << 17) ? 24.0 : 33.0) : (mean >= 2.5 ? 19.0 : (g->max_deg > 4 ? 24.0 : (g->max_deg > 3 ? 27.0 : 22.0)));
            if ((double)((nroots + 5) / 6) * (fixed + n) <= ratio * n * rounds) return BCG_OK;
            most = 1;
        }
    }
    return deep_launch(g, roots, mult, nroots, ext, note, most, st, res);
}

}  // namespace bcg
