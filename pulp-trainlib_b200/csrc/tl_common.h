// Internal header of libtrainlib_b200: runtime context, staging scopes and launch helpers.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cstdint>
#include <cstddef>
#include <cstdio>
#include <utility>
#include <vector>

typedef __half fp16;   // device-side storage type of the ABI's fp16 (IEEE binary16)
#define TRAINLIB_NO_FP16_TYPEDEF
#include "../../include/trainlib_b200_abi.h"
#include "../../include/trainlib_b200.h"

namespace tl {

// ---------------------------------------------------------------- errors
void set_error(int code, const char *fmt, ...);
bool cuda_ok(cudaError_t e, const char *what);
bool ready();                       // lazily initialises the device; false => error latched

#define TL_CUDA(call) ::tl::cuda_ok((call), #call)

// ---------------------------------------------------------------- context
cudaStream_t stream();
int streams();                      // number of independent batch-1 streams (>= 1)
int sm_count();
int gemm_path();
void count_launch();
// Per-kernel timing (off by default): when on, every launch is bracketed by CUDA events on the
// library stream and its duration is added to the entry of its kernel name.
bool profiling();
void profile_begin(const char *kernel_name);
void profile_end();
// Useful floating-point operations of the launch begun last (2 per multiply-add of the operator's definition:
// zeros a kernel multiplies for its own convenience are not work).  No-op unless profiling is on.
void profile_add_flops(double flops);

// Launch a kernel on the library stream, count it, latch launch errors.
// Every launch carries the programmatic-serialization attribute and every thread of every kernel comes through pdl_wait(), also where its block
// leaves early: blocks are placed as the blocks of the kernel before leave, and wait there until that kernel has completed and its
// writes are visible.  In front of pdl_wait() stands nothing but what needs the arguments alone (indices, tables in shared memory,
// barriers, tensor memory): no global memory is read or written there.  The
// order of memory operations is that of plain launches; what goes is the launch latency between two kernels of a stream,
// which is longer than most kernels of a single layer (measured: a 1.9 us kernel every 2.0 us instead of every 4.1 us in a
// stream, 1.76 instead of 1.95 in a graph).  No kernel lets its successor start early (griddepcontrol.launch_dependents): a
// successor that shares an SM with a persistent convolution kernel slowed both.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif
template <class... P, class... A> inline void launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A &&...args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream(); cfg.attrs = &attr; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
// The same as clusters of `cluster` blocks.
template <class... P, class... A> inline void launch_clusters(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, int cluster, A &&...args)
{
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream(); cfg.attrs = attr; cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
// Whether the device can place one cluster of that size (more than eight blocks are not portable).
template <class... P> inline bool clusters_fit(void (*kernel)(P...), int threads, size_t smem, int cluster)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)cluster; attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.attrs = &attr; cfg.numAttrs = 1;
    int n = 0;
    return cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
}
#define TL_LAUNCH_CLUSTER(kernel, grid, block, smem, cluster, ...)                  \
    do {                                                                            \
        const bool tl_prof_ = ::tl::profiling();                                    \
        if (tl_prof_) ::tl::profile_begin(#kernel);                                 \
        ::tl::launch_clusters(kernel, dim3(grid), dim3(block), (size_t)(smem), cluster, __VA_ARGS__); \
        if (tl_prof_) ::tl::profile_end();                                          \
        ::tl::count_launch();                                                       \
        ::tl::cuda_ok(cudaGetLastError(), #kernel);                                 \
    } while (0)
#define TL_LAUNCH(kernel, grid, block, smem, ...)                                   \
    do {                                                                            \
        const bool tl_prof_ = ::tl::profiling();                                    \
        if (tl_prof_) ::tl::profile_begin(#kernel);                                 \
        ::tl::launch_kernel(kernel, dim3(grid), dim3(block), (size_t)(smem), __VA_ARGS__); \
        if (tl_prof_) ::tl::profile_end();                                          \
        ::tl::count_launch();                                                       \
        ::tl::cuda_ok(cudaGetLastError(), #kernel);                                 \
    } while (0)

// ---------------------------------------------------------------- staging
// A Scope maps the pointers of one entry-point call to device addresses.
// Device pointers pass through; host pointers get a mirror in the staging arena that is
// filled before (in / inout) and copied back after (out / inout) the kernels of the call.
class Scope {
public:
    Scope();
    ~Scope();                       // copies outputs back, synchronises if anything was staged
    template <class T> const T *in(const T *p, size_t n) { return (const T *)map((void *)p, n * sizeof(T), true, false); }
    template <class T> T *out(T *p, size_t n) { return (T *)map((void *)p, n * sizeof(T), false, true); }
    template <class T> T *inout(T *p, size_t n) { return (T *)map((void *)p, n * sizeof(T), true, true); }
    template <class T> T *scratch(size_t n) { return (T *)alloc(n * sizeof(T), true); }   // device-only temporary
    // the same for a path that has another one to fall back on: no memory is no error
    template <class T> T *try_scratch(size_t n) { return (T *)alloc(n * sizeof(T), false); }
    bool ok() const;                // also sends the uploads that wait: asked in front of a call's kernels
    bool staged() const { return staged_; }   // some buffer of this call lives in host memory (mirrored in the arena)
    // a reduction of this call may be deferred: every buffer is the caller's own device memory and the call does not go
    // on to read the result itself
    bool may_defer() const { return !staged_ && !no_defer_; }
    void no_deferral() { no_defer_ = true; }
private:
    struct Entry { void *host; void *dev; void *pinned; size_t bytes; bool write_back; bool copied_in; };
    bool upload(Entry &e);
    void *map(void *p, size_t bytes, bool copy_in, bool copy_out);
    void *alloc(size_t bytes, bool needed);
    std::vector<Entry> entries_;
    size_t arena_mark_, pinned_mark_;
    unsigned stage_mark_;
    bool ok_;
    bool staged_;
    bool no_defer_ = false;
};

bool is_device_pointer(const void *p);
bool arena_pinned();                // a captured graph holds addresses of library-owned device memory: it must stay where it is
bool capturing();                   // between trainlib_graph_begin and _end
void scratch_touch();               // library-owned memory that calls of two streams share is in use on the current stream
void scratch_mark();                // behind such a use: what a stream set later waits for

// deferred reductions (tl_defer.cu): partial results kept until one batched launch sums them all
bool defer_enabled();
float *defer_alloc(size_t floats);
void defer_plain(const float *part, float *out, long long n, int groups);
void defer_columns(const float *part, float *out, int rows, int dim, int pairs);
void defer_wgt(const float *part, float *out, int groups, long long group_floats, int Cin, int Cout, int s2, int xg, int cigs, int ncopy);
void defer_settle(const void *out); // before a gradient is written again: its pending sum, if there is one, runs first
void defer_flush();
void defer_release();               // the last captured graph is gone

static inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

} // namespace tl
