// Which kernels a call is routed to, without a GPU: onefft_b200/csrc/onefft_api.cu (host code only)
// compiled as C++ and linked with this file, which stands in for the CUDA runtime (two devices, memory
// from malloc, streams and graphs as plain numbers) and for the kernel launchers, and prints one line per
// launch. Run by tests/test_dispatch.py with the name of a scenario.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "fft_launch.h"
#include "onefft_cuda.h"
#include "uneven.h"

static int g_device = 0;
static const float2 *g_in = nullptr;
static float2 *g_out = nullptr;

// ---- the runtime -----------------------------------------------------------------------------------

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = g_device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return d < 2 ? (g_device = d, cudaSuccess) : cudaErrorInvalidDevice; }
cudaError_t cudaMalloc(void **p, size_t n) { return *p = malloc(n), *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { return *d = h, cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
    return *s = cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *, const void *) { return cudaErrorInvalidValue; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) { return *n = 4, cudaSuccess; }
cudaError_t cudaGraphCreate(cudaGraph_t *g, unsigned) { return *g = (cudaGraph_t)1, cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
// a kernel node keeps the device that was current when it was added
cudaError_t cudaGraphAddKernelNode(cudaGraphNode_t *n, cudaGraph_t, const cudaGraphNode_t *, size_t, const cudaKernelNodeParams *) {
    return *n = (cudaGraphNode_t)(size_t)(1 + g_device), cudaSuccess;
}
static int g_graph_device = -1;
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    g_graph_device = g_device;
    return *e = (cudaGraphExec_t)1, cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphExecKernelNodeSetParams(cudaGraphExec_t, cudaGraphNode_t, const cudaKernelNodeParams *) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
    return printf("graph on device %d\n", g_graph_device), cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) {
    return printf("kernel on device %d\n", g_device), cudaSuccess;
}
}

// ---- the launchers ---------------------------------------------------------------------------------

namespace ofb {
static cudaError_t note(const char *kernel, int mode, int len, long long batch, const float2 *in, const float2 *out) {
    printf("%s mode %d len %d batch %lld in %lld out %lld\n", kernel, mode, len, batch, (long long)(in - g_in),
           (long long)(out - g_out));
    return cudaSuccess;
}
int batched_log_c(int m) { return m >= 12 ? 0 : 12 - m; }
bool batched_log_c_supported(int m, int c) { return c >= 0 && (c == batched_log_c(m) || (c + 1 >= batched_log_c(m) && c <= batched_log_c(m) + 1 && m + c <= 13)); }
int pass_log_c(int) { return 2; }
bool pass_tile_supported(int len, int c) { return len >= 4 && len <= 12 && len + c <= 14; }
bool pass_tma_supported(int len, int c) { return len >= 6 && len <= 12 && c <= 4 && len + c <= 14; }
bool pass_wide_weights(int mode, int len, const PassArgs &a) { return mode == 0 ? !a.pre || len <= 10 : mode == 1 || !a.post; }
bool pass01_fused_supported(int, int, int, int) { return true; }
bool batched_pipe_supported(int m) { return m == 12; }
bool batched_long_supported(int m) { return m == 13 || m == 14; }
int column_tma_log_c(int) { return -1; }
bool pass_columns_wide_supported(int, int, const PassArgs &) { return false; }
int stage_table_entries_host(int m) { return m < 4 ? 0 : 16 << m; }
int uneven_split(int m, int, int pass) { return pass ? m / 2 : m - m / 2; }
int uneven_tuned_split(int) { return 0; }
int uneven_smem_bytes() { return 40000; }
const void *uneven_kernel(const int *, bool) { return (const void *)1; }
cudaError_t set_expire_waits(int) { return cudaSuccess; }
cudaError_t launch_stage_table(float2 *, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_big_table(double2 *, double2 *, int, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_twiddle_probe(float2 *, unsigned, unsigned long long, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_power_loss_grad(int, const float2 *, const float *, float2 *, double *, long long, const float2 *, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launch_single_kernel(int m, const float2 *in, float2 *out, long long batch, const float2 *, int, cudaStream_t,
                                 const float2 *, const float2 *, int c) {
    return note("batched", c, m, batch, in, out);
}
cudaError_t launch_single_kernel_tc(int m, const float2 *in, float2 *out, long long batch, const float2 *, int, int, cudaStream_t) {
    return note("tc", 0, m, batch, in, out);
}
cudaError_t launch_batched_pipe(int m, const float2 *in, float2 *out, long long batch, const float2 *, int, unsigned *, cudaStream_t) {
    return note("pipe", 0, m, batch, in, out);
}
cudaError_t launch_batched_long(int m, const float2 *in, float2 *out, long long batch, const float2 *, int, unsigned *, cudaStream_t,
                                const float2 *, const float2 *) {
    return note("long", 0, m, batch, in, out);
}
cudaError_t launch_pass(int mode, int len, int, const PassArgs &a, int batch, cudaStream_t) {
    return note("pass", mode, len, batch, a.in, a.out);
}
cudaError_t launch_pass_tma(int mode, int len, int, const PassArgs &a, int batch, cudaStream_t) {
    return note("tma", mode, len, batch, a.in, a.out);
}
cudaError_t launch_pass_wide(int mode, int len, int, const PassArgs &a, int batch, cudaStream_t) {
    return note("wide", mode, len, batch, a.in, a.out);
}
cudaError_t launch_pass_tc(int mode, int len, const PassArgs &a, int batch, int, cudaStream_t) {
    return note("pass_tc", mode, len, batch, a.in, a.out);
}
cudaError_t launch_pass01_fused(int l0, int, int, int, const PassArgs &a, const PassArgs &, int, int, int, unsigned *, cudaStream_t) {
    return note("fused", 0, l0, 1, a.in, a.out);
}
cudaError_t launch_cluster(const PassArgs &a, const float2 *, int, long long batch, cudaStream_t) {
    return note("cluster", 0, a.log2n, batch, a.in, a.out);
}
cudaError_t launch_pass_columns(int, int, const PassArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_pass_columns_tma(int, int, const PassArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_pass_columns_wide(int, int, const PassArgs &, cudaStream_t) { return cudaSuccess; }
}  // namespace ofb

// ---- scenarios -------------------------------------------------------------------------------------

// Addresses that are never touched: input and output 2^44 bytes apart.
static void buffers(size_t shift) {
    g_in = (const float2 *)(((size_t)1 << 45) + 8 * shift);
    g_out = (float2 *)(((size_t)1 << 46) + 8 * shift);
}

static void forward(const onefft_plan *p, size_t batch, size_t shift) {
    buffers(shift);
    const int rc = onefft_dev_forward_batched(p, (const float *)g_in, (float *)g_out, batch, nullptr);
    if (rc) printf("error %d\n", rc);
}

int main(int argc, char **argv) {
    const char *what = argc > 1 ? argv[1] : "";
    if (!strcmp(what, "uneven_device")) {  // a batch made on device 0, executed with either device current
        for (int m : {10, 16}) {
            onefft_desc d[3] = {{m, 0, 0}, {m, 1, (int64_t)1 << m}, {m, 0, (int64_t)2 << m}};
            cudaSetDevice(0);
            onefft_uneven *u = onefft_uneven_create(d, 3);
            if (!u) return printf("%s\n", onefft_last_error()), 1;
            buffers(0);
            for (int dev : {0, 1}) {
                cudaSetDevice(dev);
                const int rc = onefft_uneven_execute(u, (const float *)g_in, (float *)g_out, nullptr);
                if (rc) printf("error %d\n", rc);
            }
            onefft_uneven_destroy(u);
        }
    } else if (!strcmp(what, "widths")) {  // argv: log2n, width (none: NULL), shift
        const int m = atoi(argv[2]), len = m, cols = argc > 4 ? atoi(argv[4]) : 0;
        onefft_plan *p = onefft_plan_create_tiles((size_t)1 << m, 1, &len, argc > 4 ? &cols : nullptr, 0, 0);
        if (!p) return printf("%s\n", onefft_last_error()), 0;
        forward(p, 7, atoi(argv[3]));
        onefft_plan_destroy(p);
    } else if (!strcmp(what, "default")) {  // argv: log2n, batch, shift
        onefft_plan *p = onefft_plan_create((size_t)1 << atoi(argv[2]));
        if (!p) return printf("%s\n", onefft_last_error()), 1;
        forward(p, strtoull(argv[3], nullptr, 10), atoi(argv[4]));
        onefft_plan_destroy(p);
    } else {
        return 2;
    }
    return 0;
}
