// A CUDA runtime for tests of host code on a machine without a GPU: preloaded
// before libbmfp.so, it answers the runtime calls of the matrix and solver
// entry points from host memory. Kernels do nothing; memory is zeroed. A test
// asks for what happened, and makes calls fail, through the fake_* functions.
#include "solver.h"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>

namespace
{
std::map<cudaStream_t, int> g_pending; // operations queued since the stream was last waited for
int g_mallocs = 0, g_fail_malloc = -1, g_graphs = 0, g_coop_fault = 0, g_elapsed = 0;
int g_fast_from = -1, g_fast_to = -1;
// What the next copies of a solver's state report.
enum { kAsIs, kFault, kDone } g_state = kAsIs;

cudaError_t give (void **p, size_t n)
{
  *p = aligned_alloc (256, (n + 256) / 256 * 256);
  memset (*p, 0, (n + 256) / 256 * 256);
  return cudaSuccess;
}
} // namespace

extern "C" {
int fake_pending (void *s) { return g_pending[(cudaStream_t) s]; }
int fake_mallocs () { return g_mallocs; }
// The n-th cudaMalloc from now on fails (-1: none).
void fake_fail_malloc (int n)
{
  g_mallocs = 0;
  g_fail_malloc = n;
}
int fake_graphs () { return g_graphs; }
// Cooperative launches leave a fault in the state, graphs a converged run.
void fake_cooperative_fault (int on) { g_coop_fault = on; }
// Event intervals number from .. to - 1 take 1 ms, the others 2 ms.
void fake_fast_intervals (int from, int to)
{
  g_elapsed = 0;
  g_fast_from = from;
  g_fast_to = to;
}
int fake_intervals () { return g_elapsed; }

cudaError_t cudaGetDevice (int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice (int) { return cudaSuccess; }
cudaError_t cudaGetLastError () { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute (int *v, cudaDeviceAttr a, int)
{
  *v = a == cudaDevAttrMultiProcessorCount               ? 152
       : a == cudaDevAttrMaxSharedMemoryPerBlockOptin    ? 227 << 10
       : a == cudaDevAttrL2CacheSize                     ? 1 << 20
                                                         : 1;
  return cudaSuccess;
}
cudaError_t cudaMalloc (void **p, size_t n)
{
  if (g_mallocs++ == g_fail_malloc)
    return cudaErrorMemoryAllocation;
  return give (p, n);
}
cudaError_t cudaFree (void *p) { return free (p), cudaSuccess; }
cudaError_t cudaMallocAsync (void **p, size_t n, cudaStream_t s) { return g_pending[s]++, give (p, n); }
cudaError_t cudaFreeAsync (void *p, cudaStream_t s) { return g_pending[s]++, free (p), cudaSuccess; }
cudaError_t cudaHostAlloc (void **p, size_t n, unsigned) { return give (p, n); }
cudaError_t cudaMallocHost (void **p, size_t n) { return give (p, n); }
cudaError_t cudaFreeHost (void *p) { return free (p), cudaSuccess; }
cudaError_t cudaMemGetInfo (size_t *f, size_t *t) { return *f = *t = (size_t) 1 << 38, cudaSuccess; }
cudaError_t cudaMemsetAsync (void *p, int v, size_t n, cudaStream_t s)
{
  memset (p, v, n);
  g_pending[s]++;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync (void *d, const void *p, size_t n, cudaMemcpyKind kind, cudaStream_t s)
{
  memmove (d, p, n);
  if (kind == cudaMemcpyDeviceToHost && n == sizeof (bmfp::DevState))
    {
      auto *st = static_cast<bmfp::DevState *> (d);
      st->fault = g_state == kFault;
      st->done = g_state == kDone;
      if (g_state == kDone)
        st->status = bmfp::kStateConverged;
    }
  g_pending[s]++;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags (cudaStream_t *s, unsigned) { return give ((void **) s, 8); }
cudaError_t cudaStreamDestroy (cudaStream_t s) { return free (s), cudaSuccess; }
cudaError_t cudaStreamSynchronize (cudaStream_t s) { return g_pending[s] = 0, cudaSuccess; }
cudaError_t cudaStreamWaitEvent (cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture (cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture (cudaStream_t, cudaGraph_t *g) { return give ((void **) g, 8); }
cudaError_t cudaGraphInstantiate (cudaGraphExec_t *e, cudaGraph_t, unsigned long long)
{
  g_graphs++;
  return give ((void **) e, 8);
}
cudaError_t cudaGraphDestroy (cudaGraph_t g) { return free (g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy (cudaGraphExec_t e) { return free (e), cudaSuccess; }
cudaError_t cudaGraphLaunch (cudaGraphExec_t, cudaStream_t s)
{
  g_pending[s]++;
  g_state = kDone;
  return cudaSuccess;
}
cudaError_t cudaEventCreate (cudaEvent_t *e) { return give ((void **) e, 8); }
cudaError_t cudaEventCreateWithFlags (cudaEvent_t *e, unsigned) { return give ((void **) e, 8); }
cudaError_t cudaEventDestroy (cudaEvent_t e) { return free (e), cudaSuccess; }
cudaError_t cudaEventRecord (cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize (cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime (float *ms, cudaEvent_t, cudaEvent_t)
{
  const int k = g_elapsed++;
  *ms = k >= g_fast_from && k < g_fast_to ? 1.0f : 2.0f;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute (const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor (int *n, const void *, int, size_t)
{
  return *n = 1, cudaSuccess;
}
cudaError_t __cudaGetKernel (cudaKernel_t *k, const void *f) { return *k = (cudaKernel_t) f, cudaSuccess; }
cudaError_t __cudaLaunchKernel (cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t s)
{
  return g_pending[s]++, cudaSuccess;
}
cudaError_t cudaLaunchKernel (const void *, dim3, dim3, void **, size_t, cudaStream_t s)
{
  return g_pending[s]++, cudaSuccess;
}
cudaError_t cudaLaunchKernelExC (const cudaLaunchConfig_t *c, const void *, void **)
{
  g_pending[c->stream]++;
  g_state = g_coop_fault ? kFault : kDone;
  return cudaSuccess;
}
}
