// The CUDA runtime calls and kernel launches of the host code, on host memory
// and with a log of what was queued, so that its error paths (a launch that
// fails, a stream being captured) can be tested without a GPU.  Kernels do
// nothing but what a test looks at: generation writes the parameter set's
// `pos`, Berlekamp-Massey takes its polynomial's last word from that, a product
// passes the first word of its chi on.  Built by fake_gpu.py with the library's own .cpp files.
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>

#include "../mtgp_gb300/csrc/batch.h"

namespace {

std::mutex g_mu;
std::string g_log, g_fail;
int g_fail_nth = 0;
void *g_capturing = nullptr;

void log(const char *fmt, ...) {
    char buf[256];
    va_list ap;
    va_start(ap, fmt);
    std::vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    std::lock_guard<std::mutex> lk(g_mu);
    g_log += buf;
    g_log += '\n';
}

// Whether this call of `name` is the one that a test asked to fail.
bool fails(const char *name) {
    std::lock_guard<std::mutex> lk(g_mu);
    return g_fail == name && --g_fail_nth == 0;
}

cudaError_t call(const char *name) {
    log("%s", name);
    return fails(name) ? cudaErrorUnknown : cudaSuccess;
}

// A kernel or an asynchronous operation on s.
cudaError_t queued(const char *name, cudaStream_t s, const char *fmt = "", ...) {
    char buf[160];
    va_list ap;
    va_start(ap, fmt);
    std::vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    log("%s%s %s", name, s && s == g_capturing ? " captured" : "", buf);
    return fails(name) ? cudaErrorUnknown : cudaSuccess;
}

}  // namespace

extern "C" {

// ---- the tests' side --------------------------------------------------------
void fake_clear(void) {
    std::lock_guard<std::mutex> lk(g_mu);
    g_log.clear();
    g_fail.clear();
    g_capturing = nullptr;
}
int fake_log(char *out, int cap) {
    std::lock_guard<std::mutex> lk(g_mu);
    std::snprintf(out, (size_t)cap, "%s", g_log.c_str());
    return (int)g_log.size();
}
// The nth call (from 1) of `name` from now on fails.
void fake_fail(const char *name, int nth) {
    std::lock_guard<std::mutex> lk(g_mu);
    g_fail = name;
    g_fail_nth = nth;
}
void fake_capture(void *s) { g_capturing = s; }

// ---- the runtime ------------------------------------------------------------
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = std::calloc(n ? n : 1, 1);
    return call("cudaMalloc");
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t s) {
    *p = std::calloc(n ? n : 1, 1);
    return queued("cudaMallocAsync", s);
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    *p = std::calloc(n ? n : 1, 1);
    return call("cudaHostAlloc");
}
cudaError_t cudaFree(void *p) {
    std::free(p);
    return p ? call("cudaFree") : cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) {
    std::free(p);
    return queued("cudaFreeAsync", s);
}
cudaError_t cudaFreeHost(void *p) {
    std::free(p);
    return p ? call("cudaFreeHost") : cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return call("cudaMemcpy");
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    std::memcpy(d, s, n);
    return queued("cudaMemcpyAsync", st);
}
cudaError_t cudaMemcpy2D(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h,
                         cudaMemcpyKind) {
    for (size_t k = 0; k < h; k++) std::memcpy((char *)d + k * dp, (const char *)s + k * sp, w);
    return call("cudaMemcpy2D");
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t st) {
    for (size_t k = 0; k < h; k++) std::memcpy((char *)d + k * dp, (const char *)s + k * sp, w);
    return queued("cudaMemcpy2DAsync", st);
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
    std::memset(p, v, n);
    return call("cudaMemset");
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) {
    std::memset(p, v, n);
    return queued("cudaMemsetAsync", s, "%zu", n);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = (cudaStream_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    log("cudaStreamSynchronize");
    if (s && s == g_capturing) return cudaErrorStreamCaptureUnsupported;
    return fails("cudaStreamSynchronize") ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return call("cudaDeviceSynchronize"); }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *st) {
    *st = s && s == g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t, unsigned) {
    return queued("cudaStreamWaitEvent", s);
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) {
    return cudaErrorNotSupported;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = (cudaEvent_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) { return queued("cudaEventRecord", s); }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
    *v = 152;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *, const void *) {
    return cudaErrorInvalidValue;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *) {
    return cudaErrorNotSupported;
}

}  // extern "C"

// ---- the kernels ------------------------------------------------------------
namespace mtgp {

bool shape32(int mexp, Shape *s) {
#define X(M, N, T, B) if (mexp == M) { *s = Shape{M, N, T, B}; return true; }
    MTGP_SHAPES32(X)
    return false;
}
bool shape64(int mexp, Shape *s) {
    MTGP_SHAPES64(X)
#undef X
    return false;
}
bool powOpsFits(int W) { return W > 0; }
bool powOpsWide(int W, int window) { return window != 2 && W < 3000; }
bool batchSplits32(int mexp) { return mexp == 11213 || mexp == 23209; }
bool batchSplits64(int mexp) { return mexp == 11213 || mexp == 23209; }
int batchResident32(int, bool, int) { return 1520; }
int batchResident64(int, bool, int) { return 1520; }

#define BOTH(X) X(32, uint32_t) X(64, uint64_t)
#define X(B, W)                                                                                  \
    cudaError_t launchSeed##B(const DevParams##B *, const int *, const W *, W, W *, int, int,    \
                              int, cudaStream_t s) {                                             \
        return queued("launchSeed" #B, s);                                                       \
    }                                                                                            \
    cudaError_t launchKeyed##B(const DevParams##B *, const int *, const W *, const uint64_t *,   \
                               W *, int, int, int, cudaStream_t s) {                             \
        return queued("launchKeyed" #B, s);                                                      \
    }                                                                                            \
    cudaError_t launchBM##B(const W *seqs, int n2, int nseq, int nw, uint32_t *C, int *L,        \
                            cudaStream_t s) {                                                    \
        for (int j = 0; j < nseq; j++) {                                                         \
            L[j] = n2 / 2;                                                                       \
            C[(size_t)j * nw] = 1;                                                               \
            C[(size_t)j * nw + n2 / 64] = (uint32_t)seqs[(size_t)j * n2];                        \
        }                                                                                        \
        return queued("launchBM" #B, s);                                                         \
    }                                                                                            \
    cudaError_t launchGen##B(int, int kind, const DevParams##B *p, const int *pi, W *, int n,    \
                             void *out, uint64_t, uint64_t os, cudaStream_t s, int) {            \
        for (int g = 0; g < n && out; g++)                                                       \
            ((W *)out)[(uint64_t)g * os] = (W)p[pi ? pi[g] : g].pos;                             \
        return queued("launchGen" #B, s, "kind %d", kind);                                       \
    }                                                                                            \
    cudaError_t launchJump##B(int, const DevParams##B *, W *, const JumpDesc *d, int n, int,     \
                              cudaStream_t s, const JumpDesc &row) {                             \
        return queued("launchJump" #B, s, "n %d poly %08x", n, (d ? *d : row).poly[0][0]);       \
    }                                                                                            \
    cudaError_t launchJumpFan##B(int, const DevParams##B *, const W *, const uint32_t *polys,    \
                                 int, W *, int, const JumpPart *, int n, int,                    \
                                 cudaStream_t s) {                                               \
        return queued("launchJumpFan" #B, s, "n %d poly %08x", n, polys[0]);                     \
    }                                                                                            \
    cudaError_t launchJumpParts##B(int, const DevParams##B *, const W *, const uint32_t *, int,  \
                                   W *, int, const JumpPart *, int n, cudaStream_t s) {          \
        return queued("launchJumpParts" #B, s, "n %d", n);                                       \
    }                                                                                            \
    cudaError_t launchBatch##B(const BatchLaunch &b, const DevParams##B *, W *,                  \
                               cudaStream_t s) {                                                 \
        return queued("launchBatch" #B, s, "grid %d core %d tasks %d", b.grid, b.core,           \
                      b.ntasks);                                                                 \
    }                                                                                            \
    cudaError_t launchUnstage##B(int, W *, const void *, const int *, int, cudaStream_t s) {     \
        return queued("launchUnstage" #B, s);                                                    \
    }
BOTH(X)
#undef X

cudaError_t launchBarrett(const uint32_t *, int, int, int, size_t, uint32_t *, cudaStream_t s) {
    return queued("launchBarrett", s);
}
cudaError_t launchMonomials(uint32_t *, size_t, int, int, int, cudaStream_t s) {
    return queued("launchMonomials", s);
}
cudaError_t launchGatherPow2(const uint32_t *, size_t, int, int, uint32_t *, cudaStream_t s) {
    return queued("launchGatherPow2", s);
}
static cudaError_t pow(const PowOp *ops, int n, cudaStream_t s) {
    for (int k = 0; k < n; k++) {
        ops[k].dst[0] = ops[k].tab[0];
        if (ops[k].D <= 0) log("pow with degree %d", ops[k].D);
    }
    return queued("launchPowOps", s, "n %d D %d chi %08x", n, n ? ops[0].D : 0,
                  n ? ops[0].tab[0] : 0u);
}
cudaError_t launchPowOps(const PowOp *ops, int n, const uint32_t *, int, cudaStream_t s, int) {
    return pow(ops, n, s);
}
cudaError_t launchFewPowOps(const PowOp *ops, int n, const uint32_t *, int, cudaStream_t s, int) {
    return pow(ops, n, s);
}

}  // namespace mtgp
