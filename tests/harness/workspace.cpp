/*
 * workspace.cpp -- test harness: the library's workspace (csrc/workspace.cpp)
 * over an allocator of fixed size in host memory, in place of the CUDA calls
 * that it makes.  Built by tests/test_workspace_memory.py into a temporary
 * directory; not part of the library.
 */
#include "../../part_conc_spt_abc_gb300/csrc/workspace.cpp"

#include <cstdlib>
#include <map>
#include <thread>

namespace {
size_t g_limit = 0, g_used = 0;
std::map<void*, size_t> g_blocks;
} // namespace

extern "C" {

cudaError_t cudaMalloc(void** p, size_t n)
{
    if (g_used + n > g_limit) return cudaErrorMemoryAllocation;
    *p = std::malloc(1);
    g_blocks[*p] = n;
    g_used += n;
    return cudaSuccess;
}

cudaError_t cudaFree(void* p)
{
    g_used -= g_blocks.at(p);
    g_blocks.erase(p);
    std::free(p);
    return cudaSuccess;
}

cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }

void* ws_open(size_t limit)
{
    g_limit = limit;
    return new pcs::Workspace;
}

size_t ws_close(void* w) /* what is still allocated then */
{
    delete static_cast<pcs::Workspace*>(w);
    return g_used;
}

size_t ws_used() { return g_used; }
size_t ws_keep() { return pcs::Workspace::kKeep; }

/* a standalone call of `bytes`, and within it another thread's of `inner` (0: none): 1 where both got their memory */
int ws_call(void* w, size_t bytes, size_t inner)
{
    pcs::Workspace& ws = *static_cast<pcs::Workspace*>(w);
    try {
        pcs::Lease lease(ws, nullptr, bytes);
        int ok = 1;
        if (inner)
            std::thread([&] { ok = ws_call(w, inner, 0); }).join();
        lease.done();
        return ok;
    } catch (const pcs::Error& e) {
        return e.status == PCS_ERR_OUT_OF_MEMORY ? 0 : -1;
    }
}

/* a cap set (1) or lifted (0) */
void ws_cap(void* w, int on) { static_cast<pcs::Workspace*>(w)->set_keep(!on); }

/* a cap set during a call of `bytes`: what is allocated after it */
size_t ws_cap_during_call(void* w, size_t bytes)
{
    pcs::Workspace& ws = *static_cast<pcs::Workspace*>(w);
    {
        pcs::Lease lease(ws, nullptr, bytes);
        std::thread([&] { ws_cap(w, 1); }).join();
        lease.done();
    }
    return g_used;
}

/* a job's buffer, freed at once */
int ws_job(void* w, size_t bytes)
{
    pcs::DevBuf b;
    try {
        static_cast<pcs::Workspace*>(w)->alloc(b, bytes);
        return 1;
    } catch (const pcs::Error& e) {
        return e.status == PCS_ERR_OUT_OF_MEMORY ? 0 : -1;
    }
}

} // extern "C"
