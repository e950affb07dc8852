// The wide numbering of a graph or a union of graphs: vertices by descending
// degree class, graph by graph, built on the device in one pass of stable
// counting sort (so the numbering, and with it every sum's order, depends on
// the graph alone), and the lists rewritten in it.
#include <algorithm>

#include "bcg_common.hpp"
#include "engine_internal.hpp"
#include "wide.cuh"

namespace bcg {

namespace {

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kClasses = 112;     // key of degree class c: kClasses - 1 - c
constexpr uint32_t kKeyZero = kClasses - 1u;
constexpr uint32_t kSortVerts = 2048;  // vertices of a sorting block

// Degrees up to 32 are classes of their own (a warp takes eight vertices of
// one class), then eights up to 256, then two classes an octave; 0 is last.
__device__ __forceinline__ uint32_t degree_key(uint32_t d) {
    uint32_t c;
    if (d <= 32u) c = d;
    else if (d <= 256u) c = 33u + (d - 33u) / 8u;
    else {
        const uint32_t lg = 31u - __clz(d);
        c = 61u + 2u * (lg - 8u) + ((d >> (lg - 1u)) & 1u);
    }
    return kClasses - 1u - c;
}

// One graph of the union: its vertices [base, base + n) and its part of the
// histogram, kClasses rows of nb block counts from hist on.
struct FormGraph {
    uint32_t base, n, hist, nb;
};
// One sorting block: vertices [v0, v1) of graph g, the blk-th of its blocks.
struct FormBlock {
    uint32_t v0, v1, g, blk;
};

__device__ __forceinline__ uint32_t sort_degree(const uint32_t *offs, const uint32_t *toffs, uint32_t v) {
    const uint32_t d = offs[v + 1] - offs[v];
    return toffs ? max(d, toffs[v + 1] - toffs[v]) : d;
}
// (blocks nullptr: one graph, block b its b-th)
__device__ __forceinline__ FormBlock block_of(const FormBlock *blocks, uint32_t n) {
    if (blocks) return blocks[blockIdx.x];
    const uint32_t v0 = blockIdx.x * kSortVerts;
    return FormBlock{v0, min(n, v0 + kSortVerts), 0u, blockIdx.x};
}

__global__ void __launch_bounds__(256) k_form_hist(uint32_t n, const FormBlock *__restrict__ blocks,
                                                   const FormGraph *__restrict__ graphs, FormGraph one,
                                                   const uint32_t *__restrict__ offs,
                                                   const uint32_t *__restrict__ toffs, uint32_t *__restrict__ hist) {
    __shared__ uint32_t cnt[kClasses];
    for (uint32_t i = threadIdx.x; i < kClasses; i += 256) cnt[i] = 0;
    __syncthreads();
    const FormBlock b = block_of(blocks, n);
    const FormGraph g = graphs ? graphs[b.g] : one;
    for (uint32_t v = b.v0 + threadIdx.x; v < b.v1; v += 256) atomicAdd(&cnt[degree_key(sort_degree(offs, toffs, v))], 1u);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kClasses; i += 256) hist[g.hist + i * g.nb + b.blk] = cnt[i];
}

// hist: exclusive prefix sums, which are union positions (the graphs' parts
// follow one another and each sums up to its vertices).  Stable: vertices of a
// class keep their order.  perm: position -> vertex, inv: vertex -> position
// within its graph.
__global__ void __launch_bounds__(256) k_form_number(uint32_t n, const FormBlock *__restrict__ blocks,
                                                     const FormGraph *__restrict__ graphs, FormGraph one,
                                                     const uint32_t *__restrict__ offs,
                                                     const uint32_t *__restrict__ toffs,
                                                     const uint32_t *__restrict__ hist, uint32_t *__restrict__ perm,
                                                     uint32_t *__restrict__ inv) {
    __shared__ uint32_t base[kClasses], cnt[8][kClasses];
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const FormBlock b = block_of(blocks, n);
    const FormGraph g = graphs ? graphs[b.g] : one;
    for (uint32_t i = threadIdx.x; i < kClasses; i += 256) base[i] = hist[g.hist + i * g.nb + b.blk];
    for (uint32_t i = threadIdx.x; i < 8 * kClasses; i += 256) (&cnt[0][0])[i] = 0;
    __syncthreads();
    for (uint32_t v0 = b.v0; v0 < b.v1; v0 += 256) {
        const uint32_t v = v0 + threadIdx.x;
        const bool ok = v < b.v1;
        const uint32_t key = ok ? degree_key(sort_degree(offs, toffs, v)) : kClasses;
        const unsigned peers = __match_any_sync(kFull, key);
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        if (ok && rank == 0) cnt[wid][key] = __popc(peers);
        __syncthreads();
        if (ok) {
            uint32_t pos = base[key] + rank;
            for (unsigned w = 0; w < wid; ++w) pos += cnt[w][key];
            perm[pos] = v;
            inv[v] = pos - g.base;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kClasses; i += 256) {
            uint32_t s = 0;
            for (unsigned w = 0; w < 8; ++w) {
                s += cnt[w][i];
                cnt[w][i] = 0;
            }
            base[i] += s;
        }
        __syncthreads();
    }
}

// By position: row lengths (0 at n, for the scan), the degree and reach words,
// where a vertex's bc goes, and the chunks of the heavy vertices, at least one
// each (a heavy vertex has a degree of the classes from chunk's octave on).
__global__ void k_form_rows(uint32_t n, const uint32_t *__restrict__ perm, const uint32_t *__restrict__ offs,
                            const uint32_t *__restrict__ toffs, const uint2 *__restrict__ vinfo,
                            const uint32_t *__restrict__ ext, uint32_t chunk, uint32_t *__restrict__ len0,
                            uint32_t *__restrict__ len1, uint32_t *__restrict__ ch0, uint32_t *__restrict__ ch1,
                            uint2 *__restrict__ vi2, uint32_t *__restrict__ map) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n) return;
    if (i == n) {
        len1[n] = ch1[n] = 0;
        if (toffs) len0[n] = ch0[n] = 0;
        return;
    }
    const uint32_t v = perm[i];
    const uint32_t out = offs[v + 1] - offs[v], in = toffs ? toffs[v + 1] - toffs[v] : out;
    const bool heavy = degree_key(max(out, in)) <= degree_key(chunk + 1u);
    len1[i] = out;
    ch1[i] = heavy ? max(1u, (out + chunk - 1u) / chunk) : 0u;
    if (toffs) {
        len0[i] = in;
        ch0[i] = heavy ? max(1u, (in + chunk - 1u) / chunk) : 0u;
    }
    vi2[i] = vinfo[v];
    map[i] = ext ? ext[v] : v;
}

// The lists in the new numbering (ids within the graph), one warp a vertex,
// order kept, and the chunk table.
__global__ void k_form_fill(uint32_t n, const uint32_t *__restrict__ perm, const uint32_t *__restrict__ inv,
                            const uint32_t *__restrict__ offs, const uint32_t *__restrict__ adj,
                            const uint32_t *__restrict__ offs2, uint32_t *__restrict__ adj2,
                            const uint32_t *__restrict__ cbeg, uint2 *__restrict__ chunk) {
    const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned lane = threadIdx.x & 31;
    if (w >= n) return;
    const uint32_t v = perm[w], e0 = offs[v], len = offs[v + 1] - e0, o = offs2[w];
    for (uint32_t i = lane; i < len; i += 32) adj2[o + i] = inv[adj[e0 + i]];
    const uint32_t c0 = cbeg[w], c1 = cbeg[w + 1];
    for (uint32_t c = c0 + lane; c < c1; c += 32) chunk[c] = make_uint2((uint32_t)w, c - c0);
}

// One warp a vertex.
__global__ void k_form_loops(uint32_t n, const uint32_t *__restrict__ offs, const uint32_t *__restrict__ adj,
                             uint32_t *__restrict__ loops) {
    const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= n) return;
    for (uint32_t e = offs[w] + (threadIdx.x & 31u); e < offs[w + 1]; e += 32)
        if (adj[e] == (uint32_t)w) *loops = 1;
}

// The graphs' descriptions.  proto: everything that is the same for all, with
// pointers to the union's arrays.
__global__ void k_form_subs(uint32_t graphs, const FormGraph *__restrict__ list, FormGraph one,
                            const uint32_t *__restrict__ hist, WideSub proto, WideSub *__restrict__ subs) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= graphs) return;
    const FormGraph g = list ? list[i] : one;
    WideSub s = proto;
    auto before = [&](uint32_t key) { return hist[g.hist + key * g.nb] - g.base; };  // vertices of lower keys
    s.base = g.base;
    s.n = before(kKeyZero);
    s.nheavy = before(degree_key(proto.chunk_len + 1u) + 1u);
    for (uint32_t b = 0; b < 4; ++b) s.nmed[b] = max(s.nheavy, before(degree_key(kWideLight << b)));
    for (int d = 0; d < 2; ++d) {
        s.offs[d] = proto.offs[d] + g.base;
        s.cbeg[d] = proto.cbeg[d] + g.base;
        s.chunk0[d] = s.cbeg[d][0];
        s.nchunk[d] = s.cbeg[d][g.n] - s.chunk0[d];
        s.chunk[d] = proto.chunk[d] + s.chunk0[d];
    }
    s.vinfo = proto.vinfo + g.base;
    subs[i] = s;
}

// Transposed lists of a directed graph (the order within a list is free: path
// counts are integers).
__global__ void k_form_indeg(uint64_t nnz, const uint32_t *__restrict__ adj, uint32_t *__restrict__ deg) {
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(deg + adj[e], 1u);
}
__global__ void k_form_transpose(uint32_t n, const uint32_t *__restrict__ offs, const uint32_t *__restrict__ adj,
                                 uint32_t *__restrict__ cursor, uint32_t *__restrict__ tadj) {
    const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned lane = threadIdx.x & 31;
    if (w >= n) return;
    for (uint32_t e = offs[w] + lane; e < offs[w + 1]; e += 32) tadj[atomicAdd(cursor + adj[e], 1u)] = (uint32_t)w;
}

#define CKF(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return set_error(e_ == cudaErrorMemoryAllocation ? BCG_ERR_OOM : BCG_ERR_CUDA, "%s failed: %s", \
                             #call, cudaGetErrorString(e_));                                       \
    } while (0)

inline unsigned fblocks(uint64_t work, unsigned per) { return (unsigned)std::max<uint64_t>(1, (work + per - 1) / per); }

// Memory of a form and of its building, as offsets.
struct FormPlan {
    uint32_t chunk = kWideChunk;
    uint32_t blocks = 0;
    // form
    size_t subs, inv, map, vinfo, offs[2], adj[2], cbeg[2], chunks[2], bytes;
    // scratch
    size_t perm, hist, scan, toffs, tadj, cursor, fblocks, fgraphs, scratch;
};

FormPlan plan_form(const WideInput &in) {
    FormPlan p;
    // entries of a warp's share of a heavy vertex: longer ones meet less
    // often, shorter ones leave more warps something to do
    while (p.chunk < 8 * kWideChunk && in.big_nnz / (148ull * kWideWarps * 8) >= p.chunk) p.chunk *= 2;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (std::max<size_t>(bytes, 16) + 255) & ~size_t(255);
        return at;
    };
    const size_t n = in.n, n1 = n + 1, nnz = in.nnz;
    // heavy vertices have chunk entries or more in one direction
    const size_t maxchunk = (in.directed ? 3 : 2) * (nnz / p.chunk) + 1;
    p.subs = take(in.graphs * sizeof(WideSub));
    p.inv = take(n * 4);
    p.map = take(n * 4);
    p.vinfo = take(n * 8);
    for (int d = in.directed ? 0 : 1; d < 2; ++d) {
        p.offs[d] = take(n1 * 4);
        p.adj[d] = take(nnz * 4);
        p.cbeg[d] = take(n1 * 4);
        p.chunks[d] = take(maxchunk * 8);
    }
    if (!in.directed) {
        p.offs[0] = p.offs[1]; p.adj[0] = p.adj[1]; p.cbeg[0] = p.cbeg[1]; p.chunks[0] = p.chunks[1];
    }
    p.bytes = o;
    o = 0;
    if (in.base)
        for (uint32_t i = 0; i < in.graphs; ++i) p.blocks += fblocks(in.base[i + 1] - in.base[i], kSortVerts);
    else
        p.blocks = fblocks(n, kSortVerts);
    p.perm = take(n * 4);
    p.hist = take((size_t)kClasses * p.blocks * 4);
    p.scan = take(scan_scratch(std::max<uint64_t>(n1, (uint64_t)kClasses * p.blocks)) * 4);
    p.toffs = take(in.directed ? n1 * 4 : 0);
    p.tadj = take(in.directed ? nnz * 4 : 0);
    p.cursor = take(in.directed ? n1 * 4 : 0);
    p.fblocks = take(in.base ? (size_t)p.blocks * sizeof(FormBlock) : 0);
    p.fgraphs = take(in.base ? (size_t)in.graphs * sizeof(FormGraph) : 0);
    p.scratch = o;
    return p;
}

}  // namespace

void preload_wide_form() {
    cudaFuncAttributes at;
    for (const void *k : {(const void *)k_form_hist, (const void *)k_form_number, (const void *)k_form_rows,
                          (const void *)k_form_fill, (const void *)k_form_subs})
        cudaFuncGetAttributes(&at, k);
    preload_scan();
}

size_t wide_form_bytes(const WideInput &in, size_t *scratch) {
    const FormPlan p = plan_form(in);
    *scratch = p.scratch;
    return p.bytes;
}

int wide_form_enqueue(WideForm &f, const WideInput &in, unsigned char *mem, unsigned char *scratch, cudaStream_t st) {
    const FormPlan p = plan_form(in);
    const uint32_t n = in.n;
    auto u32 = [](unsigned char *b, size_t o) { return reinterpret_cast<uint32_t *>(b + o); };
    uint32_t *perm = u32(scratch, p.perm), *hist = u32(scratch, p.hist), *scan = u32(scratch, p.scan);
    uint32_t *toffs = nullptr, *tadj = nullptr;
    int rc;
    if (in.directed) {
        toffs = u32(scratch, p.toffs);
        tadj = u32(scratch, p.tadj);
        uint32_t *cursor = u32(scratch, p.cursor);
        CKF(cudaMemsetAsync(cursor, 0, ((size_t)n + 1) * sizeof(uint32_t), st));
        k_form_indeg<<<148 * 8, 256, 0, st>>>(in.nnz, in.adj, cursor);
        if ((rc = scan_exclusive(cursor, toffs, (uint64_t)n + 1, scan, st))) return rc;
        CKF(cudaMemcpyAsync(cursor, toffs, (size_t)n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
        k_form_transpose<<<fblocks((uint64_t)n * 32, 256), 256, 0, st>>>(n, in.offs, in.adj, cursor, tadj);
        CKF(cudaGetLastError());
    }
    FormGraph one{0, n, 0, p.blocks};
    FormBlock *blocks = nullptr;
    FormGraph *graphs = nullptr;
    if (in.base) {
        std::vector<FormBlock> hb;
        std::vector<FormGraph> hg(in.graphs);
        hb.reserve(p.blocks);
        uint32_t hbase = 0;
        for (uint32_t i = 0; i < in.graphs; ++i) {
            const uint32_t b = in.base[i], m = in.base[i + 1] - b, nb = fblocks(m, kSortVerts);
            hg[i] = FormGraph{b, m, hbase, nb};
            hbase += kClasses * nb;
            for (uint32_t k = 0; k < nb; ++k)
                hb.push_back(FormBlock{b + k * kSortVerts, std::min(b + m, b + (k + 1) * kSortVerts), i, k});
        }
        blocks = reinterpret_cast<FormBlock *>(scratch + p.fblocks);
        graphs = reinterpret_cast<FormGraph *>(scratch + p.fgraphs);
        CKF(cudaMemcpyAsync(blocks, hb.data(), hb.size() * sizeof(FormBlock), cudaMemcpyHostToDevice, st));
        CKF(cudaMemcpyAsync(graphs, hg.data(), hg.size() * sizeof(FormGraph), cudaMemcpyHostToDevice, st));
    }
    f.inv = u32(mem, p.inv);
    f.map = u32(mem, p.map);
    f.d_subs = reinterpret_cast<WideSub *>(mem + p.subs);
    uint2 *vinfo = reinterpret_cast<uint2 *>(mem + p.vinfo);
    k_form_hist<<<p.blocks, 256, 0, st>>>(n, blocks, graphs, one, in.offs, toffs, hist);
    if ((rc = scan_exclusive(hist, hist, (uint64_t)kClasses * p.blocks, scan, st))) return rc;
    k_form_number<<<p.blocks, 256, 0, st>>>(n, blocks, graphs, one, in.offs, toffs, hist, perm, f.inv);
    k_form_rows<<<fblocks((uint64_t)n + 1, 256), 256, 0, st>>>(n, perm, in.offs, toffs, in.vinfo, in.ext, p.chunk,
                                                               u32(mem, p.offs[0]), u32(mem, p.offs[1]),
                                                               u32(mem, p.cbeg[0]), u32(mem, p.cbeg[1]), vinfo, f.map);
    CKF(cudaGetLastError());
    WideSub proto{};
    proto.chunk_len = p.chunk;
    proto.vinfo = vinfo;
    proto.inv = f.inv;
    for (int d = 0; d < 2; ++d) {
        // 0: who leads to v (the transposed lists of a directed graph), 1: where v leads
        proto.offs[d] = u32(mem, p.offs[d]);
        proto.adj[d] = u32(mem, p.adj[d]);
        proto.cbeg[d] = u32(mem, p.cbeg[d]);
        proto.chunk[d] = reinterpret_cast<const uint2 *>(mem + p.chunks[d]);
    }
    for (int d = in.directed ? 0 : 1; d < 2; ++d) {
        uint32_t *o = u32(mem, p.offs[d]), *c = u32(mem, p.cbeg[d]);
        if ((rc = scan_exclusive(o, o, (uint64_t)n + 1, scan, st))) return rc;
        if ((rc = scan_exclusive(c, c, (uint64_t)n + 1, scan, st))) return rc;
        const bool t = in.directed && d == 0;
        k_form_fill<<<fblocks((uint64_t)n * 32, 256), 256, 0, st>>>(n, perm, f.inv, t ? toffs : in.offs, t ? tadj : in.adj,
                                                                    o, u32(mem, p.adj[d]), c,
                                                                    reinterpret_cast<uint2 *>(mem + p.chunks[d]));
    }
    k_form_subs<<<fblocks(in.graphs, 128), 128, 0, st>>>(in.graphs, graphs, one, hist, proto, f.d_subs);
    CKF(cudaGetLastError());
    return BCG_OK;
}

int wide_form_make(WideForm &f, const WideInput &in, bool bounds) {
    size_t scratch_bytes = 0;
    const size_t bytes = wide_form_bytes(in, &scratch_bytes);
    f.subs.resize(in.graphs);
    // One small graph whose bounds do: everything in one block, and the first
    // run does not wait for the building.
    const bool small = bounds && in.graphs == 1 && !in.directed && in.n <= (1u << 16);
    CKF(f.mem.take(small ? bytes + scratch_bytes : bytes, 0, true));
    if (small) {
        WideSub &s = f.subs[0];
        s = WideSub{};
        s.n = in.n;
        s.nheavy = (uint32_t)(in.nnz / kWideChunk + 1);
        s.nchunk[0] = s.nchunk[1] = (uint32_t)(2 * (in.nnz / kWideChunk) + 1);
        return wide_form_enqueue(f, in, f.mem.mem, f.mem.mem + bytes, 0);
    }
    Workspace scratch;
    CKF(scratch.take(scratch_bytes, 0));
    int rc = wide_form_enqueue(f, in, f.mem.mem, scratch.mem, 0);
    if (!rc && cudaMemcpy(f.subs.data(), f.d_subs, in.graphs * sizeof(WideSub), cudaMemcpyDeviceToHost) != cudaSuccess)
        rc = set_error(BCG_ERR_CUDA, "reading the wide form: %s", cudaGetErrorString(cudaGetLastError()));
    scratch.waited = rc == BCG_OK;
    return rc;
}

int wide_loops(const WideInput &in, bool *loops) {
    Workspace ws;
    uint32_t found = 0;
    CKF(ws.take(4, 0));
    uint32_t *d_found = reinterpret_cast<uint32_t *>(ws.mem);
    CKF(cudaMemsetAsync(d_found, 0, 4, 0));
    k_form_loops<<<fblocks((uint64_t)in.n * 32, 256), 256>>>(in.n, in.offs, in.adj, d_found);
    CKF(cudaGetLastError());
    CKF(cudaMemcpy(&found, d_found, 4, cudaMemcpyDeviceToHost));
    ws.waited = true;
    *loops = found != 0;
    return BCG_OK;
}

void wide_form_free(WideForm &f) {
    f.mem.leave();
    f.d_subs = nullptr;
    f.inv = f.map = nullptr;
    f.subs.clear();
}

}  // namespace bcg
