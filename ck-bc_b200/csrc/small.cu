// Searches of small graphs from few sources (sm_100a): a CTA runs one source
// with everything in its shared memory.
//
// What bounds it.  A search of a graph of a thousand vertices moves next to no
// data; it is a chain of some ten levels, and over the whole chip a level costs
// a grid barrier and half a dozen dependent round trips to L2 (7 to 10 us on a
// 1024-vertex R-MAT graph).  Here the list starts, the neighbour ids (16 bits
// each), the levels, the path counts and the queue lie in shared memory, a
// barrier is __syncthreads, and nothing is made of the graph beforehand: kernel
// 80 -> 35 us, the whole call 138 -> 83.
//   - forward, the vertices of a level add their counts to the neighbours that
//     are not reached yet, and a look at all vertices finds the ones that got
//     some.  While counts are small an addition is one 32-bit atomic that
//     nobody waits for; otherwise two, the upper one only when it or the carry
//     is not 0 (whole numbers: the order does not matter, and a carry out of
//     the upper word shows that the sum passed 2^64);
//   - backward, a vertex sums X = (1 + delta) / count over its neighbours one
//     level deeper, lane by lane and then in a fixed order: the same bits in
//     every run.
// Eight lanes take a vertex, a warp one of more than kSmallHeavy entries.
#include <algorithm>
#include <cstring>

#include "bcg_common.hpp"
#include "engine_internal.hpp"

namespace bcg {

namespace {

constexpr int kSmallThreads = 1024;
constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kSmallHeavy = 128;
constexpr uint32_t kUnseen = 0xFFFFu;       // level of a vertex not reached
constexpr size_t kSmallShared = 220 << 10;  // of the 227 KB a CTA can have

struct SmallCtrl {
    int overflow;
    uint32_t pad[31];
};

struct SmallArgs {
    uint32_t n, nnz;
    const uint32_t *offs, *adj;
    const uint2 *vinfo;   // {degree, reach}; nullptr: every reach is 0
    const uint32_t *ext;  // vertex -> place in bc (nullptr: the same)
    const uint32_t *roots;
    const double *mult;
    double *out;          // per source: n (nullptr: one source, added to bc)
    double *bc;
    RootStat *rstat;      // per source (zeroed)
    SmallCtrl *ctrl;      // zeroed
};

// Places in a CTA's shared memory.
struct SmallLayout {
    uint32_t offs, lvl, order, lbeg, adj, bytes;
};
__host__ __device__ inline SmallLayout small_layout(uint32_t n, uint32_t nnz) {
    SmallLayout l;
    uint32_t o = n * 8;  // counts come first
    l.offs = o; o += (n + 1) * 4;
    l.adj = o = (o + 7) & ~7u; o += (nnz + 3) / 4 * 8;
    l.lvl = o; o += n * 2;
    l.order = o; o += n * 2;
    l.lbeg = o; o += (n + 2) * 2;
    l.bytes = (o + 15) & ~15u;
    return l;
}

__global__ void __launch_bounds__(kSmallThreads, 1) bc_small_kernel(SmallArgs a) {
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ uint32_t cnt[3];  // ring: vertices found for a level, cleared a level ahead
    __shared__ uint32_t large;  // latest level with a count beyond 32-bit sums
    __shared__ uint32_t stop;  // level at which a count overflowed (all ones: none)
    const SmallLayout l = small_layout(a.n, a.nnz);
    unsigned long long *val = reinterpret_cast<unsigned long long *>(raw);
    uint32_t *offs = reinterpret_cast<uint32_t *>(raw + l.offs);
    uint16_t *ids = reinterpret_cast<uint16_t *>(raw + l.adj), *lvl = reinterpret_cast<uint16_t *>(raw + l.lvl);
    uint16_t *order = reinterpret_cast<uint16_t *>(raw + l.order), *lbeg = reinterpret_cast<uint16_t *>(raw + l.lbeg);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5, n = a.n;
    const uint32_t gl = lane & 7u, g0 = lane & 24u;  // place in the group of eight, its first lane
    const uint32_t root = a.roots[blockIdx.x];
    const double mult = a.mult[blockIdx.x];
    double *out = a.out ? a.out + (size_t)blockIdx.x * n : nullptr;
    for (uint32_t i = tid; i <= n; i += kSmallThreads) offs[i] = a.offs[i];
    const uint32_t quads = a.nnz / 4;
    for (uint32_t i = tid; i < quads; i += kSmallThreads) {
        const uint4 t = __ldg(reinterpret_cast<const uint4 *>(a.adj) + i);
        reinterpret_cast<uint2 *>(ids)[i] = make_uint2(t.x | t.y << 16, t.z | t.w << 16);
    }
    for (uint32_t i = quads * 4 + tid; i < a.nnz; i += kSmallThreads) ids[i] = (uint16_t)a.adj[i];
    for (uint32_t i = tid; i < n; i += kSmallThreads) {
        lvl[i] = (uint16_t)kUnseen;
        val[i] = 0ull;
        if (out) out[i] = 0.0;
    }
    if (tid < 3) cnt[tid] = 0u;
    if (tid == 0) {
        stop = kFull;
        large = 0;
    }
    __syncthreads();
    if (tid == 0) {
        lvl[root] = 0;
        val[root] = 1ull;
        order[0] = (uint16_t)root;
        lbeg[0] = 0;
    }
    __syncthreads();
    // ---- forward: level d is order[b .. e)
    uint32_t d = 0, b = 0, e = 1;
    // counts below this, added up over any list, stay below 2^32
    const uint32_t plain = kFull / max(1u, a.nnz);
    bool big = false;  // some count of the level is not below it
    for (;; ++d) {
        const uint32_t to = (d + 1u) % 3u;
        // count s to the neighbour at an entry, if it is not reached
        auto push = [&](uint32_t at, unsigned long long s) {
            const uint32_t w = ids[at];
            if (lvl[w] != kUnseen) return;
            uint32_t *c = reinterpret_cast<uint32_t *>(val + w);
            const uint32_t lo = (uint32_t)s;
            if (!big) {
                atomicAdd(c, lo);
                return;
            }
            const uint32_t was = atomicAdd(c, lo);
            const unsigned long long up = (s >> 32) + (was + lo < was ? 1ull : 0ull);
            if (up) {
                const uint32_t hi = (uint32_t)up, old = atomicAdd(c + 1, hi);
                if (up >> 32 || old + hi < old) stop = d;
            }
        };
        for (uint32_t i = b + wid * 4u; i < e; i += kSmallThreads / 8u) {
            const uint32_t at = i + (lane >> 3);
            uint32_t e0 = 0, e1 = 0;
            unsigned long long s = 0;
            if (at < e) {
                const uint32_t v = order[at];
                e0 = offs[v];
                e1 = offs[v + 1];
                s = val[v];
            }
            for (unsigned heavy = __ballot_sync(kFull, gl == 0 && e1 - e0 > kSmallHeavy); heavy; heavy &= heavy - 1u) {
                const int k = __ffs(heavy) - 1;
                const uint32_t h0 = __shfl_sync(kFull, e0, k), h1 = __shfl_sync(kFull, e1, k);
                const unsigned long long hs = __shfl_sync(kFull, s, k);
#pragma unroll 4
                for (uint32_t q = h0 + lane; q < h1; q += 32u) push(q, hs);
            }
            if (e1 - e0 <= kSmallHeavy)
#pragma unroll 4
                for (uint32_t q = e0 + gl; q < e1; q += 8u) push(q, s);
            __syncwarp();
        }
        __syncthreads();
        // the vertices that got a count are level d + 1
        for (uint32_t v0 = wid * 32u; v0 < n; v0 += kSmallThreads) {
            const uint32_t v = v0 + lane;
            const unsigned long long s = v < n && lvl[v] == kUnseen ? val[v] : 0ull;
            const unsigned got = __ballot_sync(kFull, s != 0ull);
            if (!got) continue;
            uint32_t p = 0;
            if (lane == 0) p = atomicAdd(&cnt[to], (uint32_t)__popc(got));
            p = __shfl_sync(kFull, p, 0) + e + __popc(got & ((1u << lane) - 1u));
            if (s) {
                order[p] = (uint16_t)v;
                lvl[v] = (uint16_t)(d + 1u);
                if (s >= plain) large = d + 1u;
            }
        }
        if (tid == 0) {
            cnt[(d + 2u) % 3u] = 0;  // (last read two levels ago)
            lbeg[d + 1] = (uint16_t)e;
        }
        __syncthreads();
        // (what a faster warp may have written since is a higher level)
        if (stop <= d) {
            if (tid == 0) a.ctrl->overflow = 1;
            return;
        }
        const uint32_t found = cnt[to];
        if (!found) break;
        big = large == d + 1u;
        b = e;
        e += found;
    }
    // ---- what the source reached
    {
        unsigned long long ws = 0, mc = 0;
        for (uint32_t i = tid; i < e; i += kSmallThreads) {
            const uint32_t v = order[i];
            const uint32_t reach = a.vinfo ? a.vinfo[v].y : 0u, deg = a.vinfo ? a.vinfo[v].x : offs[v + 1] - offs[v];
            ws += 1ull + reach;
            mc += (unsigned long long)deg + 2ull * reach;
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            ws += __shfl_xor_sync(kFull, ws, o);
            mc += __shfl_xor_sync(kFull, mc, o);
        }
        RootStat *rs = a.rstat + blockIdx.x;
        if (lane == 0 && ws) {
            atomicAdd(&rs->wsum, ws);
            atomicAdd(&rs->mc2, mc);
        }
        if (tid == 0) {
            rs->visited = e;
            rs->depth = d;
        }
    }
    // ---- backward: levels d .. 1
    for (uint32_t k = d; k >= 1u; --k) {
        const uint32_t b0 = lbeg[k], b1 = lbeg[k + 1];
        auto child = [&](uint32_t at) -> double {
            const uint32_t w = ids[at];
            return lvl[w] == k + 1u ? __longlong_as_double((long long)val[w]) : 0.0;
        };
        for (uint32_t i = b0 + wid * 4u; i < b1; i += kSmallThreads / 8u) {
            const uint32_t at = i + (lane >> 3);
            uint32_t v = 0, e0 = 0, e1 = 0, reach = 0;
            unsigned long long sig = 1;
            if (at < b1) {
                v = order[at];
                if (k < d) {  // (the deepest level has no children)
                    e0 = offs[v];
                    e1 = offs[v + 1];
                }
                sig = val[v];
                if (gl == 0 && a.vinfo) reach = a.vinfo[v].y;
            }
            double sum = 0.0;
            for (unsigned heavy = __ballot_sync(kFull, gl == 0 && e1 - e0 > kSmallHeavy); heavy; heavy &= heavy - 1u) {
                const int o = __ffs(heavy) - 1;
                const uint32_t h0 = __shfl_sync(kFull, e0, o), h1 = __shfl_sync(kFull, e1, o);
                double t = 0.0;
#pragma unroll 4
                for (uint32_t q = h0 + lane; q < h1; q += 32u) t += child(q);
#pragma unroll
                for (int x = 8; x <= 16; x <<= 1) t += __shfl_xor_sync(kFull, t, x);
                if (g0 == (uint32_t)o) sum = t;  // eight sums are left: added below like a light vertex's
            }
            if (e1 - e0 <= kSmallHeavy)
#pragma unroll 4
                for (uint32_t q = e0 + gl; q < e1; q += 8u) sum += child(q);
            __syncwarp();
#pragma unroll
            for (int x = 1; x <= 4; x <<= 1) sum += __shfl_xor_sync(kFull, sum, x);
            if (gl == 0 && at < b1) {
                const double sg = (double)sig, delta = (double)reach + sg * sum;
                val[v] = (unsigned long long)__double_as_longlong((1.0 + delta) / sg);
                if (out) out[v] = mult * delta;
                else a.bc[a.ext ? a.ext[v] : v] += mult * delta;
            }
        }
        __syncthreads();
    }
}

// bc of vertex v: the sources' dependencies, eight interleaved sums in source
// order, then those in order.
__global__ void __launch_bounds__(256) k_small_reduce(const SmallCtrl *__restrict__ ctrl, uint32_t n, uint32_t nroots,
                                                      const double *__restrict__ out, const uint32_t *__restrict__ ext,
                                                      double *__restrict__ bc) {
    __shared__ double part[8][32];
    if (ctrl->overflow) return;  // nothing of a stopped launch is kept
    const uint32_t lane = threadIdx.x & 31u, p = threadIdx.x >> 5, v = blockIdx.x * 32u + lane;
    double s = 0.0;
    if (v < n)
#pragma unroll 4
        for (uint32_t k = p; k < nroots; k += 8u) s += __ldcs(out + (size_t)k * n + v);
    part[p][lane] = s;
    __syncthreads();
    if (p || v >= n) return;
#pragma unroll
    for (int k = 1; k < 8; ++k) s += part[k][lane];
    bc[ext ? ext[v] : v] += s;
}

#define CKM(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return set_error(e_ == cudaErrorMemoryAllocation ? BCG_ERR_OOM : BCG_ERR_CUDA, "%s failed: %s", \
                             #call, cudaGetErrorString(e_));                                       \
    } while (0)

}  // namespace

// Everything of a source must fit a CTA's shared memory, and two rounds of the
// SMs must do: one source or 148 take the same time, 296 twice that, while the
// wide searches' time hardly grows.  (Whole call, these against the wide
// searches: R-MAT graph of 1024 vertices, 21,098 entries, 1, 148, 296 and 600
// sources 83 us against 135, 102 against 211, 143 against 202, 220 against 239;
// 2048 vertices, 45,656 entries 110 against 141, 121 against 210, 182 against
// 223, 298 against 283; with the ids left in L2, where they do not fit, 4096
// vertices, 96,820 entries, one source 200 against 143.)
bool small_takes(const bcg_graph *g, uint64_t nroots) {
    const uint32_t n = g->tile_n ? g->tile_n : g->n;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return n <= 16384 && g->nnz_pruned <= (1u << 17) && nroots <= 2ull * (unsigned)nsm &&
           small_layout(n, (uint32_t)g->nnz_pruned).bytes <= kSmallShared;
}

int small_run(bcg_graph *g, const uint32_t *roots, const double *mult, uint64_t nroots, cudaStream_t st,
              SmallResult *res) {
    *res = SmallResult{};
    SmallArgs a{};
    a.n = g->tile_n ? g->tile_n : g->n;
    a.nnz = (uint32_t)g->nnz_pruned;
    const uint32_t shared = small_layout(a.n, a.nnz).bytes;
    // control words and totals (uploaded as zeros), weights, sources; the
    // sources' dependencies
    auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t o_rstat = sizeof(SmallCtrl), o_mult = o_rstat + nroots * sizeof(RootStat),
                 o_roots = o_mult + nroots * sizeof(double), blob = o_roots + nroots * sizeof(uint32_t), o_out = up(blob),
                 need = o_out + (nroots > 1 ? nroots * a.n * sizeof(double) : 0);
    Workspace ws;
    const cudaError_t took = ws.take(need, st);
    if (took == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return BCG_OK;
    }
    CKM(took);
    unsigned char *const mem = ws.mem;
    std::vector<unsigned char> h(blob);
    memcpy(h.data() + o_mult, mult, nroots * sizeof(double));
    memcpy(h.data() + o_roots, roots, nroots * sizeof(uint32_t));
    CKM(cudaMemcpyAsync(mem, h.data(), blob, cudaMemcpyHostToDevice, st));
    a.offs = g->d_offs;
    a.adj = g->d_adj;
    a.vinfo = g->trees ? g->d_vinfo : nullptr;
    a.ext = g->d_ext;
    a.ctrl = reinterpret_cast<SmallCtrl *>(mem);
    a.rstat = reinterpret_cast<RootStat *>(mem + o_rstat);
    a.mult = reinterpret_cast<const double *>(mem + o_mult);
    a.roots = reinterpret_cast<const uint32_t *>(mem + o_roots);
    a.out = nroots > 1 ? reinterpret_cast<double *>(mem + o_out) : nullptr;
    a.bc = g->d_bc;
    const void *f = (const void *)bc_small_kernel;
    // (the limit belongs to the kernel, not to the launch: the same for every
    // graph, so that threads running graphs of different sizes do not lower it
    // for one another)
    CKM(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallShared));
    CKM(cudaEventRecord(g->ev0, st));
    void *params[] = {&a};
    CKM(cudaLaunchKernel(f, dim3((unsigned)nroots), dim3(kSmallThreads), params, shared, st));
    if (nroots > 1) {
        k_small_reduce<<<(a.n + 31u) / 32u, 256, 0, st>>>(a.ctrl, a.n, (uint32_t)nroots, a.out, a.ext, a.bc);
        CKM(cudaGetLastError());
    }
    CKM(cudaEventRecord(g->ev1, st));
    CKM(cudaMemcpyAsync(h.data(), mem, o_mult, cudaMemcpyDeviceToHost, st));
    CKM(cudaStreamSynchronize(st));
    ws.waited = true;
    res->overflow = reinterpret_cast<const SmallCtrl *>(h.data())->overflow != 0;
    if (res->overflow) return BCG_OK;  // the caller's other kernels extend the counts
    res->rstat.resize(nroots);
    memcpy(res->rstat.data(), h.data() + o_rstat, nroots * sizeof(RootStat));
    res->launches = nroots > 1 ? 2 : 1;
    res->done = true;
    return BCG_OK;
}

}  // namespace bcg
