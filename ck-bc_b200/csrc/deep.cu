// Searches of deep, sparse graphs (sm_100a): grids, meshes and chains, whose
// searches have thousands of levels of a few thousand vertices.
//
// What bounds it.  There is next to no data in a level (a 2048 x 2048 grid:
// 3,960 levels of about 1,060 vertices a source), so a level costs what its
// chain of dependent loads and its barrier cost.  A sweep over the whole
// chip pays a grid barrier and its work lists for every level and batch of
// six sources: about 28 us.  Here a CTA, or a cluster of up to 8 where there
// are fewer sources than would fill the chip, runs one source by itself: the
// barrier is __syncthreads or the cluster's, and sources are independent.
// (A level's states lie far apart, each load its own sector, and one SM has
// only so many misses in flight: on the 2048 x 2048 grid a forward level takes
// it 24 us and a backward one 13; clusters of 2, 4 and 8 take 16, 10 and 7,
// and 8, 5 and 4.  On a 300 x 290 grid, 150 vertices a level, all take about 6
// and 2.6: there it is the chain of latencies alone.)
//   - vertices have at most 4 (or 8) neighbours, kept as one 16-byte (two)
//     row, so there is no row start to look up first;
//   - the frontier is a queue in shared memory that carries each vertex's
//     neighbour row, read when the vertex was found; in a cluster every warp
//     sends what it found to the queue of one CTA, in turn;
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

constexpr int kDeepThreads = 1024;
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

// States are written by other threads of the CTA: always read from L2.
__device__ __forceinline__ void ld_state(const DeepState *p, unsigned long long &val, uint32_t &lvl, uint32_t &kids) {
    uint32_t a, b;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(a), "=r"(b), "=r"(lvl), "=r"(kids) : "l"(p) : "memory");
    val = (unsigned long long)b << 32 | a;
}

// Entries a queue holds in shared memory (two queues); a larger frontier's
// tail is read back from the order list.
template <int D>
constexpr uint32_t queue_cap() { return D == 4 ? 5000u : 2700u; }

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
    uint32_t d = 0, base = 0, size = 0;  // the level, its place in order, its size
    unsigned long long vis = 0, wsum = 0, mc2 = 0;
    bool too_deep = false;
    for (;; ++d) {
        // the level's vertices: cnt in this CTA's queue, at order[first ..]
        const uint32_t ring = d % 3u;
        uint32_t cnt, first = base;
        if (C == 1) {
            cnt = size = sm.cnt[ring];
        } else {
            const uint32_t mine = lane < C ? *peer(&sm.cnt[ring], C, lane) : 0u;
            cnt = __shfl_sync(kFull, mine, rank);
            size = __reduce_add_sync(kFull, mine);
            first += __reduce_add_sync(kFull, lane < rank ? mine : 0u);
        }
        // (one barrier a level: what a faster thread has written since is the
        // next level's, in another entry of the ring, with a higher stop level)
        if (d && sm.stop < d) {
            if (tid == 0 && rank == 0) a.ctrl->overflow = 1;
            break;
        }
        too_deep = size && d > kMaxLevel;
        if (!size || too_deep) break;
        if (tid == 0 && rank == 0) lbeg[d] = base;
        const uint32_t c = d & 1u, to = (d + 1u) % 3u, next = base + size;
        int seen_stop = 0;
        if (tid == 0 && (d & 31u) == 0) seen_stop = *reinterpret_cast<volatile int *>(&a.ctrl->overflow);
        for (uint32_t i0 = tid & ~31u; i0 < cnt; i0 += kDeepThreads) {
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
                    order[first + i] = v;
                } else {
                    v = __ldcg(order + first + i);
                    nb = ell_row<D>(a.ell, v);
                }
            }
            uint32_t lv[D];
            unsigned long long val[D];
#pragma unroll
            for (int q = 0; q < D; ++q) {
                lv[q] = 0u;
                uint32_t unused;
                if (nb.u[q] != kNone) ld_state(state + nb.u[q], val[q], lv[q], unused);
            }
            uint32_t reach = 0;
            if (has && a.vinfo) reach = a.vinfo[v].y;
            // claim the neighbours not reached yet, their rows on the way
            uint32_t old[D];
            Row<D> far[D];
#pragma unroll
            for (int q = 0; q < D; ++q) {
                old[q] = 0u;
                if (nb.u[q] != kNone && lv[q] == kUnseen) {
                    old[q] = atomicExch(&state[nb.u[q]].lvl, d + 1u);
                    if (D == 4) far[q] = ell_row<D>(a.ell, nb.u[q]);
                }
            }
            if (has) {
                unsigned long long sum = 0ull;
                uint32_t kids = 0, deg = 0;
                bool ovf = false;
#pragma unroll
                for (int q = 0; q < D; ++q) {
                    if (nb.u[q] == kNone) continue;
                    ++deg;
                    if (lv[q] == kUnseen || lv[q] == d + 1u) kids |= 1u << q;
                    if (lv[q] + 1u != d) continue;
                    if (EXT) {
                        sum = ext_add(sum, val[q]);
                    } else {
                        sum += val[q];
                        ovf |= sum < val[q];
                    }
                }
                if (d == 0) sum = EXT ? kExtOne : 1ull;
                *reinterpret_cast<uint4 *>(state + v) = make_uint4((uint32_t)sum, (uint32_t)(sum >> 32), d, kids);
                if (ovf) seen_stop = 1;
                ++vis;
                wsum += 1ull + reach;
                mc2 += (unsigned long long)deg + 2ull * reach;
            }
            unsigned won[D];
            uint32_t total = 0;
#pragma unroll
            for (int q = 0; q < D; ++q) {
                won[q] = __ballot_sync(kFull, old[q] == kUnseen);
                total += __popc(won[q]);
            }
            if (total) {
                // a warp's finds go to one queue, the warps' in turn
                const uint32_t dest = C == 1 ? 0u : ((i0 >> 5) + rank + d) % C;
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(peer(&sm.cnt[to], C, dest), total);
                at = __shfl_sync(kFull, at, 0);
                uint32_t *qv = peer(&sm.v[c ^ 1u][0], C, dest);
                Row<D> *qn = peer(&sm.nb[c ^ 1u][0], C, dest);
#pragma unroll
                for (int q = 0; q < D; ++q) {
                    if ((won[q] >> lane) & 1u) {
                        const uint32_t p = at + __popc(won[q] & ((1u << lane) - 1u));
                        if (p < Q) {
                            qv[p] = nb.u[q];
                            qn[p] = D == 4 ? far[q] : ell_row<D>(a.ell, nb.u[q]);
                        } else if (C == 1) {
                            order[next + p] = nb.u[q];
                        } else {
                            a.ctrl->full = 1;  // the host runs it again with one CTA a source
                            seen_stop = 1;
                        }
                    }
                    at += __popc(won[q]);
                }
            }
        }
        if (seen_stop)
            for (uint32_t k = 0; k < C; ++k) *peer(&sm.stop, C, k) = d;
        // (last read two barriers ago)
        if (tid == 0) sm.cnt[(d + 2u) % 3u] = 0;
        source_sync(C);
        base = next;
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
    const uint32_t t0 = ((tid >> 5) * C + rank) * 32u + lane, per = C * kDeepThreads;
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
    auto finish = [&](const Item &it, const unsigned long long (&x)[D]) {
        double dl;
        unsigned long long xo;
        if (EXT) {
            unsigned long long sum = 0ull;
#pragma unroll
            for (int q = 0; q < D; ++q)
                if ((it.kids >> q) & 1u) sum = ext_add(sum, x[q]);
            dl = (double)it.reach + ext_to_double(ext_mul(it.sig, sum));
            xo = ext_div(1.0 + dl, it.sig);
        } else {
            double sum = 0.0;
#pragma unroll
            for (int q = 0; q < D; ++q)
                if ((it.kids >> q) & 1u) sum += __longlong_as_double((long long)x[q]);
            dl = (double)it.reach + (double)it.sig * sum;
            xo = (unsigned long long)__double_as_longlong((1.0 + dl) / (double)it.sig);
        }
        *reinterpret_cast<uint4 *>(state + it.v) =
            make_uint4((uint32_t)xo, (uint32_t)(xo >> 32), (uint32_t)__double2loint(dl), (uint32_t)__double2hiint(dl));
    };
    auto kids_of = [&](const Item &it, unsigned long long (&x)[D]) {
#pragma unroll
        for (int q = 0; q < D; ++q)
            if ((it.kids >> q) & 1u) x[q] = __ldcg(&state[it.nb.u[q]].val);
    };
    // starts of levels e, e - 1, e - 2
    uint32_t end = base, b0 = __ldcg(lbeg + depth), b1 = depth >= 2u ? __ldcg(lbeg + depth - 1) : 0u;
    Item it{};
    uint32_t v1 = 0;
    if (t0 < end - b0) {
        it.v = __ldcg(order + b0 + t0);
        load(it);
    }
    if (depth >= 2u && t0 < b0 - b1) v1 = __ldcg(order + b1 + t0);
    for (uint32_t e = depth; e >= 1u; --e) {
        const uint32_t n0 = end - b0, n1 = e >= 2u ? b0 - b1 : 0u;
        const uint32_t b2 = e >= 3u ? __ldcg(lbeg + e - 2) : 0u;
        unsigned long long x[D];
        if (t0 < n0) kids_of(it, x);
        Item nx{};
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
        it = nx;
        end = b0;
        b0 = b1;
        b1 = b2;
        source_sync(C);
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

template <int D>
__global__ void k_deep_rows(uint32_t n, const uint32_t *__restrict__ offs, const uint32_t *__restrict__ adj,
                            uint32_t *__restrict__ ell) {
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const uint32_t e0 = offs[v], deg = offs[v + 1] - e0;
#pragma unroll
    for (int q = 0; q < D; ++q) ell[(size_t)v * D + q] = (uint32_t)q < deg ? adj[e0 + q] : kNone;
}

#define CKD(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return set_error(e_ == cudaErrorMemoryAllocation ? BCG_ERR_OOM : BCG_ERR_CUDA, "%s failed: %s", \
                             #call, cudaGetErrorString(e_));                                       \
    } while (0)

template <int D, bool EXT>
cudaError_t launch_deep(const DeepArgs &a, cudaStream_t st) {
    const void *f = (const void *)bc_deep_kernel<D, EXT>;
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DeepSmem<D>));
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(a.nroots * a.cluster);
    cfg.blockDim = dim3(kDeepThreads);
    cfg.dynamicSmemBytes = sizeof(DeepSmem<D>);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = a.cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    DeepArgs args = a;
    void *params[] = {&args};
    return cudaLaunchKernelExC(&cfg, f, params);
}

}  // namespace

// What a graph keeps for its deep runs (bcg_graph::deep).
struct DeepGraph {
    uint32_t *ell = nullptr;
    int width = 0;         // neighbours of a row
    unsigned char *mem = nullptr;
    size_t cap = 0;
};

void deep_free(bcg_graph *g) {
    if (!g->deep) return;
    dev_free(g->deep->ell);
    dev_free(g->deep->mem);
    delete g->deep;
    g->deep = nullptr;
}

bool deep_takes(const bcg_graph *g) { return !(g->flags & BCG_DIRECTED) && g->max_deg >= 1 && g->max_deg <= 8; }

static int deep_launch(bcg_graph *g, const uint32_t *roots, const double *mult, uint64_t nroots, bool ext,
                       uint32_t most_ctas, cudaStream_t st, DeepResult *res) {
    *res = DeepResult{};
    const uint32_t n = g->tile_n ? g->tile_n : g->n;
    const int D = g->max_deg <= 4 ? 4 : 8;
    if (!g->deep) {
        DeepGraph *w = g->deep = new DeepGraph();
        w->width = D;
        const cudaError_t e = dev_alloc(&w->ell, (size_t)n * D * sizeof(uint32_t));
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            deep_free(g);
            return BCG_OK;
        }
        CKD(e);
        if (D == 4) k_deep_rows<4><<<(n + 255) / 256, 256>>>(n, g->d_offs, g->d_adj, w->ell);
        else k_deep_rows<8><<<(n + 255) / 256, 256>>>(n, g->d_offs, g->d_adj, w->ell);
        CKD(cudaGetLastError());
        CKD(cudaDeviceSynchronize());  // ready for any stream
    }
    DeepGraph *w = g->deep;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // a source's share: states and order (20 bytes a vertex), level starts; up to one source a CTA, 16 GiB in all
    auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t per = 20 * (size_t)n + (kMaxLevel + 3) * sizeof(uint32_t);
    const uint64_t slots = std::max<uint64_t>(1, std::min<uint64_t>({nroots, (uint64_t)nsm, (16ull << 30) / per}));
    size_t o = up(sizeof(DeepCtrl));
    const size_t o_rstat = o; o += up(nroots * sizeof(RootStat));
    const size_t o_mult = o; o += up(nroots * sizeof(double));
    const size_t o_roots = o; o += up(nroots * sizeof(uint32_t));
    const size_t o_state = o; o += up(slots * n * sizeof(DeepState));
    const size_t o_order = o; o += up(slots * n * sizeof(uint32_t));
    const size_t o_lbeg = o; o += up(slots * (kMaxLevel + 3) * sizeof(uint32_t));
    if (w->cap < o) {
        CKD(cudaDeviceSynchronize());  // earlier runs (any stream) are done with the old buffer
        dev_free(w->mem);
        w->mem = nullptr;
        w->cap = 0;
        const cudaError_t e = dev_alloc(&w->mem, o);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            return BCG_OK;
        }
        CKD(e);
        CKD(cudaDeviceSynchronize());
        w->cap = o;
    }
    DeepArgs a{};
    a.n = n;
    a.ell = w->ell;
    a.vinfo = g->trees ? g->d_vinfo : nullptr;
    a.state = reinterpret_cast<DeepState *>(w->mem + o_state);
    a.order = reinterpret_cast<uint32_t *>(w->mem + o_order);
    a.lbeg = reinterpret_cast<uint32_t *>(w->mem + o_lbeg);
    a.ctrl = reinterpret_cast<DeepCtrl *>(w->mem);
    std::vector<unsigned char> up_(o_state - o_mult), down(o_mult);
    memcpy(up_.data(), mult, nroots * sizeof(double));
    memcpy(up_.data() + (o_roots - o_mult), roots, nroots * sizeof(uint32_t));
    const bool several = slots < nroots;
    // as many CTAs a source as leave every source room on the chip
    a.cluster = 1;
    while (a.cluster < most_ctas && slots * 2 * a.cluster <= (uint64_t)nsm) a.cluster *= 2;
    CKD(cudaEventRecord(g->ev0, st));
    CKD(cudaMemsetAsync(w->mem, 0, o_mult, st));  // control words and the sources' totals
    CKD(cudaMemcpyAsync(w->mem + o_mult, up_.data(), up_.size(), cudaMemcpyHostToDevice, st));
    if (several) {  // launches add to bc one after the other: what it was before them
        if (!g->d_bc_save) CKD(dev_alloc(&g->d_bc_save, (size_t)g->n * sizeof(double)));
        CKD(cudaMemcpyAsync(g->d_bc_save, g->d_bc, (size_t)g->n * sizeof(double), cudaMemcpyDeviceToDevice, st));
    }
    const DeepCtrl *c = reinterpret_cast<const DeepCtrl *>(down.data());
    for (uint64_t s0 = 0; s0 < nroots; s0 += slots) {
        a.nroots = (uint32_t)std::min<uint64_t>(slots, nroots - s0);
        a.roots = reinterpret_cast<const uint32_t *>(w->mem + o_roots) + s0;
        a.rstat = reinterpret_cast<RootStat *>(w->mem + o_rstat) + s0;
        k_deep_init<<<nsm * 8, 256, 0, st>>>((uint64_t)a.nroots * n, a.state);
        CKD(D == 4 ? (ext ? launch_deep<4, true>(a, st) : launch_deep<4, false>(a, st))
                   : (ext ? launch_deep<8, true>(a, st) : launch_deep<8, false>(a, st)));
        k_deep_reduce<<<(n + 255) / 256, 256, 0, st>>>(a.ctrl, n, a.nroots,
                                                       reinterpret_cast<const double *>(w->mem + o_mult) + s0, a.state,
                                                       g->d_ext, g->d_bc);
        CKD(cudaGetLastError());
        res->launches += 3;
        const bool last = s0 + a.nroots >= nroots;
        if (last) CKD(cudaEventRecord(g->ev1, st));
        CKD(cudaMemcpyAsync(down.data(), w->mem, last ? o_mult : sizeof(DeepCtrl), cudaMemcpyDeviceToHost, st));
        CKD(cudaStreamSynchronize(st));
        if (c->overflow || c->deep || c->full) break;
    }
    if (c->overflow || c->deep || c->full) {
        if (several)
            CKD(cudaMemcpyAsync(g->d_bc, g->d_bc_save, (size_t)g->n * sizeof(double), cudaMemcpyDeviceToDevice, st));
        // frontiers that do not fit the clusters' queues: one CTA a source
        if (c->full) return deep_launch(g, roots, mult, nroots, ext, 1, st, res);
        res->overflow = c->overflow != 0;
        return BCG_OK;
    }
    res->rstat.resize(nroots);
    memcpy(res->rstat.data(), down.data() + o_rstat, nroots * sizeof(RootStat));
    res->done = true;
    return BCG_OK;
}

int deep_run(bcg_graph *g, const uint32_t *roots, const double *mult, uint64_t nroots, bool ext, cudaStream_t st,
             DeepResult *res) {
    return deep_launch(g, roots, mult, nroots, ext, 8, st, res);
}

}  // namespace bcg
