// runtime.h - error reporting shared by the C entry points.
#pragma once
#include "cwp_b200.h"
#include <cuda_runtime.h>

namespace cwpb {
// records a message for cwp_last_error() on this thread and returns code
int set_error(int code, const char* fmt, ...) __attribute__((format(printf, 2, 3)));
void clear_error();

// Several device arrays in one allocation: every cudaMalloc / cudaFree of a few MB costs 0.1 to 0.3 ms (and cudaFree waits for the
// device), which was three quarters of the time to load a batch. Declare the arrays twice with the same calls: once with
// base = nullptr for the size, once to place them.
struct Carver {
    char* base; size_t at = 0;
    explicit Carver(void* b) : base(static_cast<char*>(b)) {}
    template <class T> void take(T*& p, size_t count) { p = base ? reinterpret_cast<T*>(base + at) : nullptr; at += (count * sizeof(T) + 255) & ~(size_t)255; }
};
}  // namespace cwpb

#define CWPB_CUDA(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return ::cwpb::set_error(e_ == cudaErrorMemoryAllocation ? CWP_ERR_NOMEM : CWP_ERR_CUDA, "%s (%s:%d)", cudaGetErrorString(e_), __FILE__, __LINE__); } while (0)
#define CWPB_CHECK(cond, code, ...) do { if (!(cond)) return ::cwpb::set_error(code, __VA_ARGS__); } while (0)
