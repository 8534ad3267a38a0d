/* A CUDA runtime without a device, preloaded by test_host_faults.py: device
 * memory is host memory, copies are done at once, kernels do not run. It
 * keeps the mapped host ranges, so that a launch can be checked against them,
 * and lets launches fail on request. */
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>

#define RANGES 64
static struct { char *p; size_t n; } mapped[RANGES];

int fake_launches;       /* launches asked for */
int fake_fail_launch;    /* launches return an error */
int fake_syncs, fake_host_allocs;
long long fake_device_bytes;   /* device memory asked for */
/* 1: every launch is a grid lookup, done as out[i] = x of position i + 1; fake_stray counts those whose
 * positions or results lie outside the mapped ranges (and are left out) */
int fake_lookup, fake_stray;

static int map_add(void *p, size_t n)
{
  for (int i = 0; i < RANGES; i++)
    if (!mapped[i].p) {
      mapped[i].p = (char *)p;
      mapped[i].n = n;
      return 1;
    }
  return 0;
}

static int map_find(const void *p, size_t n)
{
  for (int i = 0; i < RANGES; i++)
    if (mapped[i].p && (char *)p >= mapped[i].p && (char *)p + n <= mapped[i].p + mapped[i].n) return i;
  return -1;
}

/* cudaDeviceReset: nothing stays mapped */
void fake_reset(void) { memset(mapped, 0, sizeof mapped); }

cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
static cudaError_t last = cudaSuccess;
cudaError_t cudaGetLastError(void)
{
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d)
{
  (void)d;
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 232448;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v)
{
  (void)f; (void)a; (void)v;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { fake_syncs++; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; fake_syncs++; return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n)
{
  fake_device_bytes += (long long)n;
  *p = calloc(1, n);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k)
{
  (void)k;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
  (void)st;
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) { (void)st; return cudaMemset(d, v, n); }

cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f)
{
  (void)f;
  fake_host_allocs++;
  *p = calloc(1, n);
  return *p && map_add(*p, n) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void *p)
{
  const int i = map_find(p, 1);
  if (i >= 0) mapped[i].p = NULL;
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostRegister(void *p, size_t n, unsigned f)
{
  (void)f;
  return map_add(p, n) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaHostUnregister(void *p)
{
  const int i = map_find(p, 1);
  if (i < 0) return cudaErrorHostMemoryNotRegistered;
  mapped[i].p = NULL;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p)
{
  memset(a, 0, sizeof *a);
  a->type = map_find(p, 1) >= 0 ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  if (a->type == cudaMemoryTypeHost) a->devicePointer = a->hostPointer = (void *)p;
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void **d, void *p, unsigned f)
{
  (void)f;
  *d = p;
  return map_find(p, 1) >= 0 ? cudaSuccess : cudaErrorInvalidValue;
}

static cudaError_t launch(void **args)
{
  fake_launches++;
  if (fake_fail_launch) return last = cudaErrorLaunchFailure;
  if (fake_lookup) {
    /* (grid, geometry, n, positions, results) */
    const int n = *(int *)args[2];
    const double *x = *(const double **)args[3];
    double *out = *(double **)args[4];
    if (map_find(x, sizeof(double) * 3 * n) < 0 || map_find(out, sizeof(double) * n) < 0) fake_stray++;
    else
      for (int i = 0; i < n; i++) out[i] = x[3 * i] + 1.0;
  }
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t m, cudaStream_t s)
{
  (void)f; (void)g; (void)b; (void)m; (void)s;
  return launch(args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args)
{
  (void)c; (void)f;
  return launch(args);
}
