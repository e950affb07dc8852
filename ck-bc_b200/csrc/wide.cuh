// Types of the wide-batch searches (wide.cu): 16 sources a job, jobs spread
// over teams of CTAs.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "engine.cuh"

namespace bcg {

constexpr int kWideSlots = 16;       // sources of a job
constexpr int kWideThreads = 640;    // one CTA per SM, 96 registers a thread
constexpr int kWideWarps = kWideThreads / 32;
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
    const uint32_t *offs[2], *adj[2];
    const uint2 *chunk[2];     // {vertex, index of the chunk within it}
    const uint32_t *cbeg[2];   // nheavy + 1: first chunk of a heavy vertex
    const uint2 *vinfo;        // {out-degree, reach}
    const uint32_t *inv;       // the engine's vertex id -> this numbering
};

// One job: up to 16 sources of one searched graph.
struct WideJob {
    uint32_t sub, root0, nroots, pad;
    unsigned long long out;  // its dependencies: bc[out .. out + n) of WideArgs::jobbc
};

// Words the CTAs of a team share (one cache line each).
struct WideTeam {
    unsigned long long arrived;  // barrier arrivals since the launch (monotone)
    uint32_t job[2];             // next job, by parity of the current one
    uint32_t any[4];             // ring: the forward sweep found a vertex (1), a count of 2^32 or more (2)
    unsigned long long count[4];  // ring: vertices the forward sweep found, and finished (upper half)
    uint32_t pad[16];
};
static_assert(sizeof(WideTeam) == 128, "one line per team");

struct WideCtrl {
    int error, overflow, deep;   // any of them set ends the launch
    uint32_t next_job;           // first job not handed out
    unsigned long long wait_ns;
    uint32_t pad[26];
};
static_assert(sizeof(WideCtrl) == 128, "one line");

struct WideArgs {
    const WideSub *subs;
    const WideJob *jobs;
    uint32_t njobs;
    uint32_t teams, team_ctas;
    const uint32_t *roots;  // engine ids, by WideJob::root0
    const double *mult;
    double *jobbc;
    RootStat *rstat;        // njobs * 16, zeroed
    WideCtrl *ctrl;
    WideTeam *team;
    // per-team state, each array sized for the launch's largest graph
    unsigned char *state;
    size_t stride;          // bytes of a team's state
    size_t o_done, o_act, o_sig, o_g0, o_g1, o_part, o_hcnt;
    size_t words;           // 32-vertex words of the largest graph (row length of act)
    TraceRec *trace;
    unsigned int trace_cap;
    unsigned int *trace_cnt;
};

}  // namespace bcg
