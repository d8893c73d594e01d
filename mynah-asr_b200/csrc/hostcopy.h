// Copies between the device and host memory that a caller owns (hostcopy.cu).
#pragma once
#include <vector>

#include "common.cuh"

namespace mb {

// copy_in: ordered on `st`; when it returns the host memory may be reused, unless it is page-locked (as cudaMemcpyAsync).
// copy_out: what `st` holds so far is waited for; when it returns the host memory holds the data, unless it is page-locked.
int copy_in(void *dev, const void *host, size_t bytes, cudaStream_t st);
struct CopyOut { void *host; const void *dev; size_t bytes; };
int copy_out(const std::vector<CopyOut> &parts, cudaStream_t st);
static inline int copy_out(void *host, const void *dev, size_t bytes, cudaStream_t st) { return copy_out({CopyOut{host, dev, bytes}}, st); }

// Whoever makes copies says when it comes and goes: threads and page-locked pieces live as long as the last one.
void copy_user_made();
void copy_user_gone();
struct CopyUser {
    CopyUser() { copy_user_made(); }
    ~CopyUser() { copy_user_gone(); }
    CopyUser(const CopyUser &) = delete;
    CopyUser &operator=(const CopyUser &) = delete;
};

}  // namespace mb
