// Types of the wide-batch searches (wide.cu): 16 or 32 sources a job, jobs
// spread over teams of CTAs.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "engine.cuh"
#include "workspace.hpp"

struct bcg_graph;

namespace bcg {

// One CTA per SM.  Registers hold rows in flight, and 640 threads leave 96 a
// thread, with spills in every sweep: 512 with 128 take 35.7 against 37.4 ms on
// the benchmark's graph (1024 sources), 5.3 against 5.6 for 48 small graphs; 576
// and 768 are slower than either.
constexpr int kWideThreads = 512;
constexpr int kWideWarps = kWideThreads / 32;
constexpr uint32_t kWideTeams = 148;  // most teams of a launch
constexpr uint32_t kWideLevels = 64;  // levels a job can hold (deeper searches run elsewhere)
constexpr uint32_t kWideLight = 32;   // four lanes take a vertex of up to so many entries, or 2, 4, 8 times that
constexpr uint32_t kWideChunk = 256;  // entries of a warp's share of a heavy vertex, at least

// One searched graph (or one graph of a union), its vertices numbered by
// descending degree class: [0, nheavy) have chunk_len entries or more in
// some direction and are cut into chunks of so many, [nheavy, nmed[i]) more
// than kWideLight << i, [nmed[i], n) the rest.  Index 0 of a pair: the lists a forward
// sweep sums over (who leads to v), 1: the lists of a backward sweep (where v
// leads); the same arrays on an undirected graph.
struct WideSub {
    uint32_t n, nheavy, chunk_len, pad;
    uint32_t nmed[4];
    uint32_t nchunk[2];
    uint32_t base, pad2;       // the graph's first position in its union
    uint32_t chunk0[2];        // its first chunk there
    const uint32_t *offs[2], *adj[2];  // entries from offs[..][v] on in adj
    const uint2 *chunk[2];     // {union position of the vertex, index of the chunk within it}
    const uint32_t *cbeg[2];   // first chunk (of the union's) of a vertex
    const uint2 *vinfo;        // {out-degree, reach}
    const uint32_t *inv;       // the engine's vertex id -> this numbering
};

// One job: up to `slots` sources of one searched graph.
struct WideJob {
    uint32_t sub, root0, nroots, pad;
    unsigned long long out;  // its dependencies: bc[out .. out + n) of WideArgs::jobbc
};

// Words the CTAs of a team share (one cache line each).
struct WideTeam {
    unsigned long long arrived;  // barrier arrivals since the launch (monotone)
    uint32_t job[2];             // next job, by parity of the current one
    uint32_t any[4];             // ring: the forward sweep found a vertex (1), a count of 2^28 or more (2), a sum past 2^64 (4:
                                 // count_overflows tells whether it is a count), a neighbour listed twice at level 1 (8)
    unsigned long long count[4];  // ring: vertices the forward sweep found, and finished (upper half)
    uint32_t pad[16];
};
static_assert(sizeof(WideTeam) == 128, "one line per team");

struct WideCtrl {
    int error, overflow, deep;   // any of them set ends the launch
    uint32_t next_job;           // first job not handed out
    uint32_t pad[28];
};
static_assert(sizeof(WideCtrl) == 128, "one line");

struct WideArgs {
    const WideSub *subs;
    const WideJob *jobs;    // nullptr: subs[0]'s sources roots[0 .. nroots) in order, from job job0 on,
                            // job j's vector at j * n
    uint32_t njobs, job0, nroots;
    uint32_t slots;         // sources of a job: 16 or 32
    uint32_t teams, team_ctas;
    uint32_t split_ctas;    // team size the split of vertices by degree is made for (0: team_ctas);
                            // fixed, a job's sums do not depend on the launch it runs in
    const uint32_t *roots;  // engine ids, by WideJob::root0
    const double *mult;     // weights, likewise (nullptr: 1)
    double *jobbc;
    int *poison;            // several launches' stop word (nullptr: none): set by a launch that
                            // stops, and a launch that finds it set does nothing
    uint32_t *deep_jobs;    // njobs words (zeroed): a job with a search of more levels than it holds
                            // sets its word and is left; nullptr: such a job stops the launch
    RootStat *rstat;        // njobs * slots, zeroed (nullptr: not wanted)
    RootStat *total;        // or the sums over all sources, and the deepest level (zeroed)
    WideCtrl *ctrl;
    WideTeam *team;
    // per-team state, each array sized for the launch's largest graph
    unsigned char *state;
    size_t stride;          // bytes of a team's state
    size_t o_done, o_act, o_bits, o_sig, o_g0, o_g1, o_part, o_hcnt;
    size_t words;           // 32-vertex words of the largest graph (row length of act)
    TraceRec *trace;
    unsigned int trace_cap;
    unsigned int *trace_cnt;
};

// Adding the jobs of a graph: bc[map[v]] += sum over j < njobs of
// jobbc[out0 + j * n + v].
struct WideOut {
    unsigned long long out0;
    uint32_t njobs, n;
    const uint32_t *map;
    double *bc;
    const WideSub *sub;  // set: n is its n (not known to the host)
    uint32_t job0, pad;  // its first job's word of deep_jobs (wide_chain)
};

// The lists a wide form is made from (device arrays; vinfo and ext by engine
// id, ext nullptr: bc is indexed by engine id).  A union of several graphs has
// base[graphs + 1] (host), the first vertex of each.
struct WideInput {
    uint32_t n;
    uint64_t nnz;
    const uint32_t *offs, *adj;
    const uint2 *vinfo;
    const uint32_t *ext;
    bool directed;
    const uint32_t *base;
    uint32_t graphs;
    uint64_t big_nnz;  // entries of the largest graph
};

WideInput wide_input(const bcg_graph *g);  // of a graph's searched lists

// A graph's (or union's) lists in the wide numbering.
struct WideForm {
    Workspace mem;                 // everything below on the device (empty: the caller's memory)
    WideSub *d_subs = nullptr;     // one a graph
    uint32_t *inv = nullptr, *map = nullptr;
    std::vector<WideSub> subs;     // the host's copy (wide_form_make)
};

// Bytes of a form, and of the scratch that building it takes.
size_t wide_form_bytes(const WideInput &in, size_t *scratch);
// Enqueues the building in memory of that size on st; f.subs stays empty.
int wide_form_enqueue(WideForm &f, const WideInput &in, unsigned char *mem, unsigned char *scratch, cudaStream_t st);
// Allocates and builds on stream 0, and reads subs back.  bounds: the caller
// takes subs' n, nheavy and nchunk for upper bounds (n counts the vertices
// without an entry too) and its WideOut names the device's sub; of one small
// graph nothing is read back then, and the building is not waited for.
int wide_form_make(WideForm &f, const WideInput &in, bool bounds);
void wide_form_free(WideForm &f);
// Whether some list names its own vertex (waits).
int wide_loops(const WideInput &in, bool *loops);

// Loads the wide searches' kernels on the current device (CUDA would load each
// at its first launch, which takes device memory).
void preload_wide();
void preload_wide_form();
void preload_scan();

// Fills a's state layout for jobs of 16 or 32 slots on graphs of up to n
// vertices; returns the stride.
size_t wide_layout(WideArgs &a, uint32_t slots, size_t n, size_t nchunk, size_t nheavy);
// Whether a graph with so many vertices that have an entry, and so many
// entries, is shallow enough to be tried: mean degree 6 and up, or too few
// vertices for more levels than a job holds.
inline bool wide_shallow(uint64_t active, uint64_t nnz) { return nnz >= 6 * active || active + 2 < kWideLevels; }
// Cuts the SMs into teams for njobs jobs on lists of so many entries (their
// mean), a's layout being set; returns the time in us this is expected to take.
// One team at least, also where its state alone is more than state_bytes: a
// caller whose buffer is fixed looks at a.stride itself.
double wide_teams(WideArgs &a, uint64_t njobs, uint64_t entries, size_t state_bytes = 512ull << 20);
// Layout and teams for nroots sources of one graph, in jobs of 16 or 32,
// whichever is expected to end first; returns which.
uint32_t wide_plan(WideArgs &a, uint64_t nroots, uint64_t entries, size_t n, size_t nchunk, size_t nheavy,
                   size_t state_bytes = 512ull << 20);
// Puts a graph's nroots sources (and weights, unless nullptr) in the order in
// which its jobs should take them; order (nullptr: not wanted) says which came
// to each place.  key: nroots words of scratch.  Windows of 8192 sources.
int wide_order(const WideSub *sub, const uint32_t *roots, const double *mult, uint32_t nroots, uint32_t *key,
               uint32_t *roots_to, double *mult_to, uint32_t *order, cudaStream_t st);
// One launch of a's jobs and the adding of their vectors: nouts entries of
// outs (device; nmax vertices at most; 0: nothing is added), or `one` when outs
// is nullptr.
int wide_enqueue(const WideArgs &a, const WideOut *outs, uint32_t nouts, const WideOut &one, uint32_t nmax,
                 cudaStream_t st);

// Adds the vectors in strict job order (a.poison unset); of an entry with a
// job that was left, none.
int wide_chain(const WideArgs &a, const WideOut *outs, uint32_t nouts, uint32_t nmax, const uint32_t *deep_jobs,
               cudaStream_t st);

}  // namespace bcg
