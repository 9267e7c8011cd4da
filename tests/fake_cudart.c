/* A CUDA runtime without a device, for tests of the library's host code on the CPU: memory is the host's, launches do nothing
 * but are counted, and one of them can be made to fail.  Preloaded in front of libcudart. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

static struct { char *p; size_t n; } blocks[256];
static cudaError_t last = cudaSuccess;
static int launches, fail_at, max_cluster, max_blocks, cluster_limit = 16;

void fake_reset(int fail) { launches = max_cluster = max_blocks = 0; fail_at = fail; }   /* fail: number of the launch that fails, from 1; 0: none */
void fake_cluster_limit(int n) { cluster_limit = n; }
int fake_launches(void) { return launches; }
int fake_max_cluster(void) { return max_cluster; }
int fake_max_blocks(void) { return max_blocks; }           /* of a launch, along x and y */

cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "made by the test"; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(struct cudaDeviceProp *p, int d) { (void)d; memset(p, 0, sizeof *p); p->multiProcessorCount = 148; p->major = 10; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) { (void)a; (void)d; *v = 148; return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n)
{
    if (posix_memalign(p, 256, n)) return cudaErrorMemoryAllocation;
    memset(*p, 0x55, n);
    for (int i = 0; i < 256; i++) if (!blocks[i].p) { blocks[i].p = *p; blocks[i].n = n; break; }
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    for (int i = 0; i < 256; i++) if (blocks[i].p == p) blocks[i].p = NULL;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return posix_memalign(p, 256, n) ? cudaErrorMemoryAllocation : cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f) { (void)f; return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p)
{
    memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    for (int i = 0; i < 256; i++) if (blocks[i].p && (char *)p >= blocks[i].p && (char *)p < blocks[i].p + blocks[i].n) a->type = cudaMemoryTypeDevice;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t q) { (void)k; (void)q; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t q) { (void)q; memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)malloc(8); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)malloc(8); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char *s, void **p, unsigned long long f, enum cudaDriverEntryPointQueryResult *r)
{
    (void)s; (void)f; *p = NULL;
    if (r) *r = cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *f, const cudaLaunchConfig_t *c)
{
    (void)f;
    *n = 9;
    for (unsigned i = 0; i < c->numAttrs; i++) if (c->attrs[i].id == cudaLaunchAttributeClusterDimension && (int)c->attrs[i].val.clusterDim.x > cluster_limit) *n = 0;
    return cudaSuccess;
}
static cudaError_t launch(int cluster, dim3 grid)
{
    if ((int)(grid.x * grid.y) > max_blocks) max_blocks = (int)(grid.x * grid.y);
    if (cluster > max_cluster) max_cluster = cluster;
    if (++launches == fail_at || cluster > cluster_limit) return last = cudaErrorLaunchOutOfResources;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args)
{
    int cluster = 1;
    (void)f; (void)args;
    for (unsigned i = 0; i < c->numAttrs; i++) if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = (int)c->attrs[i].val.clusterDim.x;
    return launch(cluster, c->gridDim);
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t n, cudaStream_t s) { (void)f; (void)b; (void)args; (void)n; (void)s; return launch(1, g); }
