// Batched form: exact all-sources BC of many independent graphs in one
// persistent launch (no counterpart in the reference, whose program runs one
// graph per process; the per-graph computation is the same as bcg_run's).
//
// The graphs are laid out on the device as one disjoint union (graph g's
// vertex v is union vertex base[g] + v), ordered by their count of
// non-isolated vertices, largest first.  Brandes on a disjoint union is Brandes
// on each component, so each graph's slice of the union's bc is that graph's
// bc.  Sources are packed per component: batch i puts, in slot k, the
// (i*S + k)-th non-isolated vertex of every graph that has that many, so one
// batch advances every active graph at once and the sweeps of small graphs
// share the grid barriers of the large ones.  Graphs still active in batch i
// are a prefix of the union and tiles never cross a graph boundary, so a
// batch resets and first pulls only the rows and tiles of that prefix.  The whole schedule runs in one cooperative launch,
// captured once into a CUDA graph and replayed by every bcg_batch_run.
//
// Sets of shallow graphs (wide_shallow: every graph of mean degree 6 and up, or
// of a few vertices) do not run that schedule: their sources go to the
// wide-batch searches (wide.cu), 32 of one graph a job, a CTA or a few to a
// job, largest graphs first, in as many launches as the job vectors' memory
// asks for, captured the same way.  One with a search of more than 62 levels
// goes back to the packed schedule, and one with loops stays there.  (48 graphs
// of 250 to 2,500 vertices: the packed schedule advances all by six sources a
// batch and pays about 13 barriers of the whole chip for it, 108 ms; a CTA that
// runs 32 sources of one graph has no such barrier: 5.2 ms.)
//
// The autotuner times a prefix of the schedule for each candidate batch width
// S in {1, 3, 6} and tile shape (vertices x adjacency entries per tile), keeps
// the fastest per root, and rebuilds the schedule for it.
#include <algorithm>
#include <cstring>
#include <numeric>
#include <vector>

#include "bcg_common.hpp"
#include "engine_internal.hpp"
#include "wide.cuh"

using namespace bcg;

struct bcg_batch {
    bcg_graph *g = nullptr;
    uint32_t ngraphs = 0;
    std::vector<uint32_t> base, gn;  // per caller graph: first union vertex, vertex count
    std::vector<uint32_t> order;     // union position -> caller graph
    std::vector<uint32_t> hdeg;      // union degrees
    uint32_t width = 3;
    // device schedule of the current width and tile shape
    uint32_t *d_xbeg = nullptr, *d_xroots = nullptr, *d_xtiles = nullptr, *d_xrbeg = nullptr;
    uint2 *d_xrange = nullptr;
    unsigned char *d_xslot = nullptr;
    unsigned long long *d_xpf = nullptr, *d_xpu = nullptr;
    RootStat *d_rstat = nullptr;
    uint32_t nbatch = 0;
    uint64_t nroots = 0;
    std::vector<uint32_t> hxbeg;  // host copy of the batch starts
    cudaStream_t stream = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int captured = 0;  // 1: runs replay a captured CUDA graph; 0: direct launches
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // the wide searches of the set (wide = false: the packed schedule runs)
    bool wide = false, packed = false;  // packed: its schedule is built
    WideForm form;
    struct Launch {
        WideArgs a;
        size_t outs;  // offset of its WideOut entries in d_wide
        uint32_t nouts, nmax;
    };
    std::vector<Launch> launches;
    uint64_t njobs = 0;
    unsigned char *d_wide = nullptr, *d_stat = nullptr, *d_state = nullptr;
    double *d_jobbc = nullptr, *d_save = nullptr;
    size_t stat_bytes = 0, o_total = 0;
};

namespace {

#define CKB(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return set_error(e_ == cudaErrorMemoryAllocation ? BCG_ERR_OOM : BCG_ERR_CUDA, "%s failed: %s", \
                             #call, cudaGetErrorString(e_));                                       \
    } while (0)

void free_schedule(bcg_batch *b) {
    cudaFree(b->d_xbeg); cudaFree(b->d_xroots); cudaFree(b->d_xtiles); cudaFree(b->d_xslot);
    cudaFree(b->d_xpf); cudaFree(b->d_xpu); cudaFree(b->d_rstat); cudaFree(b->d_xrbeg); cudaFree(b->d_xrange);
    b->d_xbeg = b->d_xroots = b->d_xtiles = b->d_xrbeg = nullptr;
    b->d_xrange = nullptr;
    b->d_xslot = nullptr;
    b->d_xpf = b->d_xpu = nullptr;
    b->d_rstat = nullptr;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
    b->captured = 0;
    b->packed = false;
}

constexpr uint32_t kBatchSlots = 32;  // sources of a job: every graph has all its vertices searched

void free_wide(bcg_batch *b) {
    wide_form_free(b->form);
    dev_free(b->d_wide); dev_free(b->d_stat); dev_free(b->d_state); dev_free(b->d_jobbc); dev_free(b->d_save);
    b->d_wide = b->d_stat = b->d_state = nullptr;
    b->d_jobbc = b->d_save = nullptr;
    b->launches.clear();
    b->wide = false;
}

// The set's jobs and launches (b->wide = true), if every graph is shallow.
// Running out of memory leaves the packed schedule to do the work.
int build_wide(bcg_batch *b) {
    bcg_graph *g = b->g;
    const uint32_t G = b->ngraphs;
    std::vector<uint32_t> ubase(G + 1);
    std::vector<uint32_t> act(G, 0);
    std::vector<uint64_t> gnnz(G, 0);
    WideInput in = wide_input(g);
    in.graphs = G;
    in.base = ubase.data();
    in.big_nnz = 0;
    uint64_t nroots = 0;
    for (uint32_t p = 0; p < G; ++p) {
        const uint32_t v0 = ubase[p] = b->base[b->order[p]], nv = b->gn[b->order[p]];
        uint64_t &nnz = gnnz[p];
        for (uint32_t v = v0; v < v0 + nv; ++v) {
            nnz += b->hdeg[v];
            act[p] += b->hdeg[v] != 0;
        }
        if (!wide_shallow(act[p], nnz)) return BCG_OK;
        in.big_nnz = std::max(in.big_nnz, nnz);
        nroots += act[p];
    }
    ubase[G] = g->n;
    if (nroots == 0 || g->n >= (1u << 28)) return BCG_OK;
    auto give_up = [&](int rc) {
        free_wide(b);
        return rc == BCG_ERR_OOM ? (cudaGetLastError(), BCG_OK) : rc;
    };
    // (the total of edges below is a half of all sources' entries together,
    // which takes an even number of each: the packed schedule halves its own)
    bool loops = false;
    int rc = wide_loops(in, &loops);
    if (rc || loops) return give_up(rc);
    rc = wide_form_make(b->form, in, false);
    if (rc) return give_up(rc);
    // jobs in union order (largest graphs first); a launch ends when its jobs'
    // vectors take 512 MB, or when the graphs have become a quarter of its
    // first one's size and it has work for four rounds of the chip
    constexpr uint64_t kCells = (512ull << 20) / 8;
    std::vector<WideJob> jobs;
    std::vector<uint32_t> roots;
    std::vector<WideOut> outs;
    struct Span { size_t job0, njobs, out0, nouts; uint64_t cells, entries; uint32_t nmax, nch, nheavy; };
    std::vector<Span> spans;
    uint64_t most_cells = 0;
    roots.reserve(nroots);
    for (uint32_t p = 0; p < G; ++p) {
        const WideSub &s = b->form.subs[p];
        if (!act[p]) continue;
        const size_t r0 = roots.size();
        for (uint32_t v = ubase[p]; v < ubase[p + 1]; ++v)
            if (b->hdeg[v]) roots.push_back(v);
        for (uint32_t r = 0; r < act[p]; r += kBatchSlots) {
            if (spans.empty() || spans.back().cells + s.n > kCells ||
                (r == 0 && s.n < spans.back().nmax / 4 && spans.back().njobs >= 4 * 148))
                spans.push_back(Span{jobs.size(), 0, outs.size(), 0, 0, 0, s.n, 1, 1});
            Span &l = spans.back();
            if (l.nouts == 0 || r == 0) {
                outs.push_back(WideOut{l.cells, 0, s.n, b->form.map + s.base, g->d_bc, nullptr});
                ++l.nouts;
            }
            ++outs.back().njobs;
            jobs.push_back(WideJob{p, (uint32_t)(r0 + r), std::min<uint32_t>(kBatchSlots, act[p] - r), 0, l.cells});
            ++l.njobs;
            l.cells += s.n;
            l.entries += gnnz[p];
            l.nmax = std::max(l.nmax, s.n);
            l.nch = std::max({l.nch, s.nchunk[0], s.nchunk[1]});
            l.nheavy = std::max(l.nheavy, s.nheavy);
            most_cells = std::max(most_cells, l.cells);
        }
    }
    auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t o_roots = up(jobs.size() * sizeof(WideJob)), o_outs = o_roots + up(roots.size() * 4),
                 blob = o_outs + outs.size() * sizeof(WideOut);
    size_t stat = 0, state = 0;
    for (const Span &l : spans) {
        bcg_batch::Launch L{};
        state = std::max(state, (wide_layout(L.a, kBatchSlots, l.nmax, l.nch, l.nheavy), wide_teams(L.a, l.njobs, l.entries / l.njobs),
                                 L.a.stride * L.a.teams));
        L.a.njobs = (uint32_t)l.njobs;
        L.outs = o_outs + l.out0 * sizeof(WideOut);
        L.nouts = (uint32_t)l.nouts;
        L.nmax = l.nmax;
        b->launches.push_back(L);
        stat += sizeof(WideCtrl) + L.a.teams * sizeof(WideTeam);
    }
    b->o_total = stat;
    b->stat_bytes = stat + sizeof(RootStat);
    cudaError_t e;
    if ((e = dev_alloc(&b->d_wide, blob)) != cudaSuccess || (e = dev_alloc(&b->d_stat, b->stat_bytes)) != cudaSuccess ||
        (e = dev_alloc(&b->d_state, state)) != cudaSuccess ||
        (e = dev_alloc(&b->d_jobbc, most_cells * sizeof(double))) != cudaSuccess ||
        (spans.size() > 1 && (e = dev_alloc(&b->d_save, (size_t)g->n * sizeof(double))) != cudaSuccess))
        return give_up(set_error(e == cudaErrorMemoryAllocation ? BCG_ERR_OOM : BCG_ERR_CUDA, "wide searches: %s",
                                 cudaGetErrorString(e)));
    CKB(cudaMemcpy(b->d_wide, jobs.data(), jobs.size() * sizeof(WideJob), cudaMemcpyHostToDevice));
    CKB(cudaMemcpy(b->d_wide + o_roots, roots.data(), roots.size() * 4, cudaMemcpyHostToDevice));
    CKB(cudaMemcpy(b->d_wide + o_outs, outs.data(), outs.size() * sizeof(WideOut), cudaMemcpyHostToDevice));
    // a graph's sources in the order its jobs should take them, if there is
    // memory for a second list (a set's jobs are of many graphs: 6.2 -> 5.6 ms
    // on 48 R-MAT graphs)
    uint32_t *tmp = nullptr;
    if ((e = dev_alloc(&tmp, roots.size() * 8)) == cudaSuccess) {
        CKB(cudaMemcpy(tmp, roots.data(), roots.size() * 4, cudaMemcpyHostToDevice));
        uint32_t *to = reinterpret_cast<uint32_t *>(b->d_wide + o_roots);
        size_t r = 0;
        for (uint32_t p = 0; p < G && !rc; r += act[p], ++p)
            if (act[p] > kBatchSlots)
                rc = wide_order(b->form.d_subs + p, tmp + r, nullptr, act[p], tmp + roots.size() + r, to + r, nullptr, nullptr, 0);
        dev_free(tmp);
        if (rc) return give_up(rc);
    } else {
        cudaGetLastError();
    }
    CKB(cudaDeviceSynchronize());  // everything is ready for the batch's stream
    size_t at = 0;
    for (size_t i = 0; i < spans.size(); ++i) {
        WideArgs &a = b->launches[i].a;
        a.subs = b->form.d_subs;
        a.jobs = reinterpret_cast<const WideJob *>(b->d_wide) + spans[i].job0;
        a.roots = reinterpret_cast<const uint32_t *>(b->d_wide + o_roots);
        a.jobbc = b->d_jobbc;
        a.state = b->d_state;
        a.ctrl = reinterpret_cast<WideCtrl *>(b->d_stat + at);
        a.team = reinterpret_cast<WideTeam *>(b->d_stat + at + sizeof(WideCtrl));
        a.total = reinterpret_cast<RootStat *>(b->d_stat + b->o_total);
        at += sizeof(WideCtrl) + a.teams * sizeof(WideTeam);
    }
    b->njobs = jobs.size();
    b->nroots = nroots;
    b->wide = true;
    return BCG_OK;
}

// Enqueues the wide launches on b->stream.
int enqueue_wide(bcg_batch *b) {
    CKB(cudaMemsetAsync(b->d_stat, 0, b->stat_bytes, b->stream));
    if (b->d_save)  // launches add to bc one after the other: what it was before them
        CKB(cudaMemcpyAsync(b->d_save, b->g->d_bc, (size_t)b->g->n * sizeof(double), cudaMemcpyDeviceToDevice, b->stream));
    for (const bcg_batch::Launch &l : b->launches) {
        const int rc = wide_enqueue(l.a, reinterpret_cast<const WideOut *>(b->d_wide + l.outs), l.nouts, WideOut{}, l.nmax,
                                    b->stream);
        if (rc) return rc;
    }
    return BCG_OK;
}

// Builds and uploads the packed schedule for width b->width and the graph's
// current tiles.
int build_schedule(bcg_batch *b) {
    free_schedule(b);
    const uint32_t S = b->width;
    bcg_graph *g = b->g;
    std::vector<uint32_t> tile_of(g->n);
    CKB(cudaMemcpy(tile_of.data(), g->d_tile_of, (size_t)g->n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    // per union position: its non-isolated vertices, and the graph's entries
    const uint32_t G = b->ngraphs;
    std::vector<std::vector<uint32_t>> act(G);
    std::vector<uint64_t> gnnz(G, 0);
    uint32_t maxc = 0;
    for (uint32_t p = 0; p < G; ++p) {
        const uint32_t gi = b->order[p];
        const uint32_t v0 = b->base[gi], nv = b->gn[gi];
        for (uint32_t v = v0; v < v0 + nv; ++v) {
            gnnz[p] += b->hdeg[v];
            if (b->hdeg[v]) act[p].push_back(v);
        }
        maxc = std::max<uint32_t>(maxc, (uint32_t)act[p].size());
    }
    const uint32_t nb = (maxc + S - 1) / S;
    std::vector<uint32_t> xbeg(nb + 1, 0), xroots, xtiles(nb);
    std::vector<unsigned char> xslot;
    std::vector<unsigned long long> xpf(nb, 0), xpu(nb, 0);
    for (uint32_t i = 0; i < nb; ++i) {
        uint32_t last_active = 0;  // union positions [0, last_active) have roots in batch i
        for (uint32_t p = 0; p < G; ++p) {
            if (act[p].size() <= (size_t)i * S) break;  // sorted: no later graph is active
            last_active = p + 1;
            for (uint32_t k = 0; k < S; ++k) {
                const size_t j = (size_t)i * S + k;
                if (j >= act[p].size()) break;
                const uint32_t r = act[p][j];
                xroots.push_back(r);
                xslot.push_back((unsigned char)k);
                xpf[i] += b->hdeg[r];
                xpu[i] += gnnz[p] - b->hdeg[r];
            }
        }
        xbeg[i + 1] = (uint32_t)xroots.size();
        // tiles of the active prefix: every tile before the first inactive
        // graph's (tiles never cross a graph boundary)
        xtiles[i] = (last_active >= G) ? g->ntiles : (tile_of[b->base[b->order[last_active]]] & ~kHubFlag);
    }
    b->nbatch = nb;
    b->nroots = xroots.size();
    b->hxbeg = xbeg;
    if (nb == 0) return BCG_OK;
    CKB(cudaMalloc(&b->d_xbeg, xbeg.size() * sizeof(uint32_t)));
    CKB(cudaMalloc(&b->d_xroots, std::max<size_t>(1, xroots.size()) * sizeof(uint32_t)));
    CKB(cudaMalloc(&b->d_xslot, std::max<size_t>(1, xslot.size())));
    CKB(cudaMalloc(&b->d_xtiles, nb * sizeof(uint32_t)));
    CKB(cudaMalloc(&b->d_xpf, nb * sizeof(unsigned long long)));
    CKB(cudaMalloc(&b->d_xpu, nb * sizeof(unsigned long long)));
    CKB(cudaMalloc(&b->d_rstat, (size_t)nb * S * sizeof(RootStat)));
    CKB(cudaMemcpy(b->d_xbeg, xbeg.data(), xbeg.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    if (!xroots.empty()) {
        CKB(cudaMemcpy(b->d_xroots, xroots.data(), xroots.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
        CKB(cudaMemcpy(b->d_xslot, xslot.data(), xslot.size(), cudaMemcpyHostToDevice));
    }
    CKB(cudaMemcpy(b->d_xtiles, xtiles.data(), nb * sizeof(uint32_t), cudaMemcpyHostToDevice));
    CKB(cudaMemcpy(b->d_xpf, xpf.data(), nb * sizeof(unsigned long long), cudaMemcpyHostToDevice));
    CKB(cudaMemcpy(b->d_xpu, xpu.data(), nb * sizeof(unsigned long long), cudaMemcpyHostToDevice));
    // one tile range per batch: the active prefix [0, xtiles[i])
    std::vector<uint32_t> xrbeg(nb + 1);
    std::iota(xrbeg.begin(), xrbeg.end(), 0u);
    std::vector<uint2> xrange(nb, make_uint2(0u, 0u));
    CKB(cudaMalloc(&b->d_xrbeg, (nb + 1) * sizeof(uint32_t)));
    CKB(cudaMalloc(&b->d_xrange, nb * sizeof(uint2)));
    CKB(cudaMemcpy(b->d_xrbeg, xrbeg.data(), (nb + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice));
    CKB(cudaMemcpy(b->d_xrange, xrange.data(), nb * sizeof(uint2), cudaMemcpyHostToDevice));
    b->packed = true;
    return ensure_state(g, S);
}

PackedRun packed_prefix(const bcg_batch *b, uint32_t nbatch) {
    PackedRun p{};
    p.xbeg = b->d_xbeg;
    p.xroots = b->d_xroots;
    p.xslot = b->d_xslot;
    p.xpf = b->d_xpf;
    p.xpu = b->d_xpu;
    p.xtiles = b->d_xtiles;
    p.xrbeg = b->d_xrbeg;
    p.xrange = b->d_xrange;
    p.nbatch = nbatch;
    p.rstat = b->d_rstat;
    return p;
}

// One run of the first nbatch batches on b->stream, timed with events.
int timed_run(bcg_batch *b, uint32_t nbatch, float *ms) {
    CKB(cudaEventRecord(b->ev0, b->stream));
    int rc = enqueue_packed(b->g, packed_prefix(b, nbatch), b->width, b->stream);
    if (rc) return rc;
    CKB(cudaEventRecord(b->ev1, b->stream));
    rc = check_ctrl(b->g, b->stream);
    if (rc) return rc;
    CKB(cudaEventElapsedTime(ms, b->ev0, b->ev1));
    return BCG_OK;
}

}  // namespace

namespace bcg {

int make_union(uint32_t ngraphs, const uint32_t *const *offsets, const uint32_t *const *adj, const uint32_t *n,
               bool by_active, std::vector<uint32_t> &order, std::vector<uint32_t> &base,
               std::vector<uint32_t> &hdeg, bcg_graph **out) {
    *out = nullptr;
    if (ngraphs == 0 || !offsets || !adj || !n) return set_error(BCG_ERR_ARG, "no graphs or null arrays");
    uint64_t N = 0, NNZ = 0;
    for (uint32_t i = 0; i < ngraphs; ++i) {
        if (!offsets[i] || n[i] == 0) return set_error(BCG_ERR_ARG, "graph %u: null offsets or n == 0", i);
        if (offsets[i][n[i]] && !adj[i]) return set_error(BCG_ERR_ARG, "graph %u: null adjacency", i);
        N += n[i];
        NNZ += offsets[i][n[i]];
    }
    if (N > 0xFFFFFFFEull || NNZ > 0xFFFFFFFFull)
        return set_error(BCG_ERR_RANGE, "union of %u graphs exceeds 32-bit ids/offsets", ngraphs);
    order.resize(ngraphs);
    std::iota(order.begin(), order.end(), 0u);
    if (by_active) {
        // most non-isolated vertices first
        std::vector<uint32_t> act(ngraphs, 0);
        for (uint32_t i = 0; i < ngraphs; ++i)
            for (uint32_t v = 0; v < n[i]; ++v) act[i] += (offsets[i][v + 1] > offsets[i][v]);
        std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return act[x] > act[y]; });
    }
    base.assign(ngraphs, 0);
    std::vector<uint32_t> uoffs(N + 1), uadj(NNZ);
    hdeg.resize(N);
    uint64_t vpos = 0, epos = 0;
    for (uint32_t p = 0; p < ngraphs; ++p) {
        const uint32_t gi = order[p];
        const uint32_t vb = (uint32_t)vpos;
        base[gi] = vb;
        const uint32_t *o = offsets[gi];
        for (uint32_t v = 0; v < n[gi]; ++v) {
            uoffs[vpos] = (uint32_t)epos;
            hdeg[vpos] = o[v + 1] - o[v];
            for (uint32_t e = o[v]; e < o[v + 1]; ++e) {
                const uint32_t w = adj[gi][e];
                if (w >= n[gi]) return set_error(BCG_ERR_ARG, "graph %u: adj[%u] = %u >= n=%u", gi, e, w, n[gi]);
                uadj[epos++] = vb + w;
            }
            ++vpos;
        }
    }
    uoffs[N] = (uint32_t)epos;
    return bcg_graph_create(uoffs.data(), uadj.data(), (uint32_t)N, NNZ, 0, out);
}

}  // namespace bcg

extern "C" {

int bcg_batch_create(uint32_t ngraphs, const uint32_t *const *offsets, const uint32_t *const *adj,
                     const uint32_t *n, bcg_batch **out) {
    clear_error();
    if (!out) return set_error(BCG_ERR_ARG, "null output handle");
    *out = nullptr;
    bcg_batch *b = new bcg_batch();
    int rc = make_union(ngraphs, offsets, adj, n, true, b->order, b->base, b->hdeg, &b->g);
    if (rc) {
        delete b;
        return rc;
    }
    b->ngraphs = ngraphs;
    b->gn.assign(n, n + ngraphs);
    // tiles never cross a graph boundary: a batch then reaches exactly the
    // rows of its active graphs, and only those are reset and walked
    std::vector<uint32_t> breaks(b->base);
    std::sort(breaks.begin(), breaks.end());
    b->g->tile_breaks = breaks;
    rc = graph_retile(b->g, b->g->tile_vcap, b->g->tile_ecap, true);
    if (rc) {
        bcg_batch_destroy(b);
        return rc;
    }
    auto fail = [&](int code) {
        bcg_batch_destroy(b);
        return code;
    };
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaEventCreate(&b->ev0)) != cudaSuccess || (e = cudaEventCreate(&b->ev1)) != cudaSuccess)
        return fail(set_error(BCG_ERR_CUDA, "stream/event: %s", cudaGetErrorString(e)));
    rc = build_wide(b);
    if (!rc && !b->wide) rc = build_schedule(b);
    if (rc) return fail(rc);
    *out = b;
    return BCG_OK;
}

int bcg_batch_destroy(bcg_batch *b) {
    clear_error();
    if (!b) return set_error(BCG_ERR_ARG, "null handle");
    if (b->stream) cudaStreamSynchronize(b->stream);
    free_schedule(b);
    free_wide(b);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->stream) cudaStreamDestroy(b->stream);
    if (b->g) bcg_graph_destroy(b->g);
    delete b;
    return BCG_OK;
}

// Runs the set's launches on b->stream, captured into a CUDA graph by the
// first run and replayed; if the capture cannot be made, runs launch directly
// (b->captured says which).
static int replay(bcg_batch *b) {
    auto enqueue = [&]() {
        return b->wide ? enqueue_wide(b) : enqueue_packed(b->g, packed_prefix(b, b->nbatch), b->width, b->stream);
    };
    if (!b->exec) {
        cudaGraph_t graph = nullptr;
        int rc = BCG_ERR_CUDA;
        if (cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeRelaxed) == cudaSuccess) {
            rc = enqueue();
            const cudaError_t ee = cudaStreamEndCapture(b->stream, &graph);
            if (rc == BCG_OK && ee == cudaSuccess && graph && cudaGraphInstantiate(&b->exec, graph, 0) == cudaSuccess) {
                b->graph = graph;
                b->captured = 1;
            } else {
                if (graph) cudaGraphDestroy(graph);
                b->exec = nullptr;
            }
        }
        cudaGetLastError();  // a refused capture leaves no sticky error
        clear_error();
    }
    CKB(cudaEventRecord(b->ev0, b->stream));
    if (b->exec) {
        CKB(cudaGraphLaunch(b->exec, b->stream));
    } else {
        const int rc = enqueue();
        if (rc) return rc;
    }
    CKB(cudaEventRecord(b->ev1, b->stream));
    return BCG_OK;
}

int bcg_batch_run(bcg_batch *b, bcg_stats *stats) {
    clear_error();
    if (!b) return set_error(BCG_ERR_ARG, "null handle");
    if (stats) *stats = bcg_stats{};
    uint64_t teps = 0, vis = 0, cv = 0;
    uint32_t md = 0, width = 0;
    uint64_t batches = 0;
    if (b->wide) {
        int rc = replay(b);
        if (rc) return rc;
        std::vector<unsigned char> hs(b->stat_bytes);
        CKB(cudaMemcpyAsync(hs.data(), b->d_stat, b->stat_bytes, cudaMemcpyDeviceToHost, b->stream));
        CKB(cudaStreamSynchronize(b->stream));
        bool deep = false, overflow = false;
        int error = 0;
        for (const bcg_batch::Launch &l : b->launches) {
            const WideCtrl *c =
                reinterpret_cast<const WideCtrl *>(hs.data() + (reinterpret_cast<unsigned char *>(l.a.ctrl) - b->d_stat));
            deep |= c->deep != 0;
            overflow |= c->overflow != 0;
            if (c->error) error = c->error;
        }
        if ((deep || overflow || error) && b->d_save) {
            CKB(cudaMemcpyAsync(b->g->d_bc, b->d_save, (size_t)b->g->n * sizeof(double), cudaMemcpyDeviceToDevice, b->stream));
            CKB(cudaStreamSynchronize(b->stream));
        }
        if (error) return set_error(error, "device reported error %d (a bounded wait gave up)", error);
        if (overflow) return set_error(BCG_ERR_OVERFLOW, "a shortest-path count exceeded 2^64");
        if (deep) {  // from here on the packed schedule runs
            free_schedule(b);
            free_wide(b);
            rc = build_schedule(b);
            if (rc) return rc;
        } else {
            const RootStat *t = reinterpret_cast<const RootStat *>(hs.data() + b->o_total);
            teps = t->mc2 / 2;  // every source's share is even (no loops)
            vis = t->visited;
            cv = t->wsum;
            md = t->depth;
            batches = b->njobs;
            width = kBatchSlots;
        }
    }
    if (!b->wide) {
        batches = b->nbatch;
        width = b->width;
        if (b->nbatch) {
            int rc = replay(b);
            if (!rc) rc = check_ctrl(b->g, b->stream);
            if (rc) return rc;
        }
        if (stats) {
            std::vector<RootStat> rs((size_t)b->nbatch * b->width);
            if (!rs.empty())
                CKB(cudaMemcpy(rs.data(), b->d_rstat, rs.size() * sizeof(RootStat), cudaMemcpyDeviceToHost));
            for (const RootStat &r : rs) {
                teps += r.mc2 / 2;
                vis += r.visited;
                cv += r.wsum;
                md = std::max(md, r.depth);
            }
        }
    }
    if (stats) {
        uint64_t nsrc = 0;
        for (uint32_t i = 0; i < b->ngraphs; ++i) nsrc += b->gn[i];
        float ms = 0.f;
        if (batches) cudaEventElapsedTime(&ms, b->ev0, b->ev1);
        stats->sources = nsrc;
        stats->roots = b->nroots;
        stats->skipped = nsrc - b->nroots;
        stats->batches = batches;
        stats->teps_edges = teps;
        stats->visited = vis;
        stats->comp_vertices = cv;
        stats->max_depth = md;
        stats->batch_width = width;
        stats->kernel_ms = ms;
    }
    return BCG_OK;
}

int bcg_batch_reset_bc(bcg_batch *b) {
    clear_error();
    if (!b) return set_error(BCG_ERR_ARG, "null handle");
    return bcg_reset_bc(b->g);
}

int bcg_batch_get_bc(bcg_batch *b, uint32_t graph, double *bc_host) {
    clear_error();
    if (!b || !bc_host) return set_error(BCG_ERR_ARG, "null argument");
    if (graph >= b->ngraphs) return set_error(BCG_ERR_ARG, "graph %u >= %u graphs", graph, b->ngraphs);
    double *d_bc = nullptr;
    int rc = bcg_bc_device_ptr(b->g, &d_bc);
    if (rc) return rc;
    CKB(cudaMemcpy(bc_host, d_bc + b->base[graph], (size_t)b->gn[graph] * sizeof(double), cudaMemcpyDeviceToHost));
    return BCG_OK;
}

int bcg_batch_autotune(bcg_batch *b, uint32_t sample_batches, uint32_t *width, uint32_t *tile_vertices,
                       uint32_t *tile_entries) {
    clear_error();
    if (!b) return set_error(BCG_ERR_ARG, "null handle");
    static const uint32_t widths[] = {1, 3, 6};
    static const uint32_t shapes[][2] = {{32, 512}, {32, 256}, {32, 128}, {16, 128}, {16, 64}};
    if (b->wide) {  // nothing to tune: the widths and tiles are the packed schedule's
        if (width) *width = b->width;
        if (tile_vertices) *tile_vertices = b->g->tile_vcap;
        if (tile_entries) *tile_entries = b->g->tile_ecap;
        return bcg_reset_bc(b->g);
    }
    double best = 0.0;
    uint32_t bw = b->width, bv = b->g->tile_vcap, be = b->g->tile_ecap;
    for (const auto &sh : shapes) {
        int rc = graph_retile(b->g, sh[0], sh[1]);
        if (rc) return rc;
        for (uint32_t S : widths) {
            b->width = S;
            rc = build_schedule(b);
            if (rc) return rc;
            if (!b->nbatch) continue;
            const uint32_t nb = std::max(1u, std::min(b->nbatch, sample_batches ? sample_batches : 4u));
            float ms = 0.f;
            rc = timed_run(b, nb, &ms);  // warm-up (module, state, caches)
            if (!rc) rc = timed_run(b, nb, &ms);
            if (rc) return rc;
            const double per_root = ms / std::max<uint32_t>(1, b->hxbeg[nb]);
            if (best == 0.0 || per_root < best) {
                best = per_root;
                bw = S;
                bv = sh[0];
                be = sh[1];
            }
        }
    }
    int rc = graph_retile(b->g, bv, be);
    if (rc) return rc;
    b->width = bw;
    rc = build_schedule(b);
    if (rc) return rc;
    rc = bcg_reset_bc(b->g);  // the timing runs added into the accumulators
    if (rc) return rc;
    if (width) *width = bw;
    if (tile_vertices) *tile_vertices = bv;
    if (tile_entries) *tile_entries = be;
    return BCG_OK;
}

int bcg_batch_info(bcg_batch *b, uint32_t *nbatch, uint32_t *width, uint32_t *tile_vertices,
                   uint32_t *tile_entries, int *captured) {
    clear_error();
    if (!b) return set_error(BCG_ERR_ARG, "null handle");
    if (nbatch) *nbatch = b->wide ? (uint32_t)std::min<uint64_t>(b->njobs, 0xFFFFFFFFull) : b->nbatch;
    if (width) *width = b->width;
    if (tile_vertices) *tile_vertices = b->g->tile_vcap;
    if (tile_entries) *tile_entries = b->g->tile_ecap;
    if (captured) *captured = b->captured;
    return BCG_OK;
}

}  // extern "C"
