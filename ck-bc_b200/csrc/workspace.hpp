// Large device buffers that outlive one use (defined in engine.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace bcg {

// The buffer of one run that waits for its results (states, job vectors), or of
// a graph's second form: taken from those that earlier ones on any graph of
// the device left, or allocated, and left for later ones.  What is left is at
// most kWorkKeep a device (4 GiB once no graph is alive) and goes when an
// allocation of the library would fail without it.
constexpr uint64_t kWorkKeep = 8ull << 30;
struct Workspace {
    unsigned char *mem = nullptr;
    size_t cap = 0;
    int device = 0;
    bool waited = false;  // the host has waited for all work on it
    Workspace() = default;
    Workspace(const Workspace &) = delete;
    Workspace &operator=(const Workspace &) = delete;
    ~Workspace() { leave(); }
    void leave();  // (waits for the device first unless `waited`)
    // Ready for stream st.  keep: it is held for long, so one of about the size.
    cudaError_t take(size_t bytes, cudaStream_t st, bool keep = false);
};

}  // namespace bcg
