/*
 * workspace.cpp -- device buffers, and the memory that the standalone entry
 * points keep between calls.
 */
#include "engine.h"

#include <algorithm>

namespace pcs {

void DevBuf::alloc(size_t n)
{
    release();
    if (n == 0) n = 16;
    cudaError_t e = cudaMalloc(&p, n);
    if (e != cudaSuccess) {
        p = nullptr;
        (void)cudaGetLastError();
        throw Error(PCS_ERR_OUT_OF_MEMORY, "device allocation of " + std::to_string(n) + " bytes failed");
    }
    bytes = n;
}

void DevBuf::release()
{
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
}

bool Workspace::give_back()
{
    std::unique_lock<std::mutex> held(mu, std::try_to_lock);
    if (!held.owns_lock() || !dev.p) return false;
    dev.release();
    return true;
}

void Workspace::set_keep(bool k)
{
    keep = k;
    if (!k) give_back();
}

void Workspace::alloc(DevBuf& b, size_t n)
{
    try {
        b.alloc(n);
    } catch (const Error& e) {
        if (e.status != PCS_ERR_OUT_OF_MEMORY || !give_back()) throw;
        b.alloc(n);
    }
}

Lease::Lease(Workspace& ws, cudaStream_t stream, size_t bytes) : ws_(ws), stream_(stream), held_(ws.mu, std::try_to_lock)
{
    size_ = std::max<size_t>(bytes, 256u);
    if (held_.owns_lock() && !ws_.keep) ws_.dev.release();
    if (held_.owns_lock() && ws_.keep && size_ <= Workspace::kKeep) {
        if (ws_.dev.bytes < size_) {
            size_t n = 1u << 20;
            while (n < size_) n <<= 1;
            ws_.dev.release();
            if (cudaMalloc(&ws_.dev.p, n) == cudaSuccess) {
                ws_.dev.bytes = n;
            } else { /* no room to keep that much: this call's own, below */
                (void)cudaGetLastError();
                ws_.dev.p = nullptr;
            }
        }
        base_ = ws_.dev.as<char>();
    }
    if (!base_) {
        own_alloc_();
        base_ = own_.as<char>();
    }
}

/* A block of the call's own; what is kept makes room for it if need be (the
 * lock on it is this call's, or Workspace::alloc tries for it). */
void Lease::own_alloc_()
{
    if (!held_.owns_lock()) return ws_.alloc(own_, size_);
    try {
        own_.alloc(size_);
    } catch (const Error& e) {
        if (e.status != PCS_ERR_OUT_OF_MEMORY || !ws_.dev.p) throw;
        ws_.dev.release();
        own_.alloc(size_);
    }
}

Lease::~Lease()
{
    /* a call that failed on its way may have left work that uses this memory */
    if (!done_) cudaStreamSynchronize(stream_);
    if (held_.owns_lock() && !ws_.keep) ws_.dev.release();
}

void* Lease::take(size_t bytes)
{
    if (used_ + bytes > size_) throw Error(PCS_ERR_INVALID_ARGUMENT, "workspace overflow");
    void* p = base_ + used_;
    used_ += bytes;
    return p;
}

char* Lease::stage(size_t n)
{
    n = (n + 63u) / 64u * 64u;
    if (!held_.owns_lock() || !ws_.pinned || staged_ + n > Workspace::kPinned) return nullptr;
    char* p = ws_.pinned + staged_;
    staged_ += n;
    return p;
}

} // namespace pcs
