// Shared definitions for the opcuda-b200 library (sm_100a).
//
// Error model: every exported entry point returns an int status -- 0 on success, a
// negative OPB_E* code for an argument error detected on the host, or a positive
// cudaError_t.  The last status is also kept per host thread and can be read through
// opcuda_get_status(), which is how the reference's callers read it
// (oplib/opcuda/util.cu:59,204-207; oplib/opmodel/types/CArray.cs:577-578).
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stdint.h>

#define OPB_API extern "C" __attribute__((visibility("default")))

enum {
    OPB_OK = 0,
    OPB_E_ARG = -1,       // bad size / count
    OPB_E_NULL = -2,      // null pointer where one is required
    OPB_E_ALIGN = -3,     // pointer or size misaligned for the kernel's vector access
    OPB_E_UNSUPPORTED = -4,
    OPB_E_NOMEM = -5,
    OPB_E_TIMEOUT = -6,   // a bounded device wait ran out
    OPB_E_STATE = -7,     // call out of order (missing init, plan not built, ...)
};

namespace opb {

int set_status(int s);            // records and returns s
int set_cuda(cudaError_t e);      // records and returns (int)e
cudaStream_t stream();            // the calling thread's current library stream
int num_sms();                    // SM count of the current device (cached per device)
int launch_check();               // cudaGetLastError -> status

inline bool aligned(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// Profiler range over one library call (NVTX; a no-op unless a profiler is attached), so
// that a capture can select a call's kernels by name.
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

// Programmatic dependent launch.  A kernel launched by launch_pdl may be set up (its launch, and
// what it does before pdl_wait) while the kernel before it in the stream still runs; pdl_wait
// returns once that kernel has completed and its writes are visible, so every thread of a kernel
// launched this way calls it before it touches global memory.  pdl_next lets the kernel's own
// successor be set up in turn, once all its blocks have called it or ended.  It stands after the
// wait, so that one successor at most is resident and order stays transitive, and after the
// block's tensor memory is allocated: a successor may sit on tensor memory while it waits for
// this kernel, which therefore must not still be asking for its own.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
    pdl_wait();
    pdl_next();
}

template <class... P, class... A>
inline int launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#endif

}  // namespace opb

#define OPB_NVTX(name) opb::NvtxRange opb_nvtx_range_(name)

#define OPB_TRY(expr)                                  \
    do {                                               \
        cudaError_t _e = (expr);                       \
        if (_e != cudaSuccess) return opb::set_cuda(_e); \
    } while (0)

#define OPB_REQUIRE(cond, code)                        \
    do {                                               \
        if (!(cond)) return opb::set_status(code);     \
    } while (0)
