// A stand-in for the CUDA runtime and the kernel launchers, for tests of the
// host code without a GPU: device memory is host memory, kernels do nothing, and
// the call number fake_fail_at fails.  Copies stay pending on their stream until
// it is waited for.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

#include "gcz_kernels.h"

namespace {
struct Copy {
    const char *p;
    size_t n;
};
std::map<cudaStream_t, std::vector<Copy>> g_pending;
long g_calls = 0, g_fail_at = 0;
size_t g_handles = 0;
std::map<cudaStream_t, void *> g_last_to;

bool fails() { return ++g_calls == g_fail_at; }
cudaError_t done(cudaError_t e = cudaErrorUnknown) { return fails() ? e : cudaSuccess; }
}  // namespace

extern "C" {
void fake_fail_at(long call) { g_calls = 0, g_fail_at = call, g_last_to.clear(); }
long fake_calls() { return g_calls; }
// Whether the last copy of a stream went to p.
int fake_last_to(void *p) {
    for (auto &s : g_last_to)
        if (s.second == p) return 1;
    return 0;
}
// Copies not waited for that read or write [p, p + n).
long fake_pending(const char *p, size_t n) {
    long k = 0;
    for (auto &s : g_pending)
        for (const Copy &c : s.second) k += c.p < p + n && p < c.p + c.n;
    return k;
}

cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
    memset(p, 0, sizeof(*p));
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "fake failure"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) {
    if (fails()) return cudaErrorMemoryAllocation;
    return *p = calloc(1, n), cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { return memset(p, v, n), done(); }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), done(); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    if (fails()) return cudaErrorUnknown;
    memcpy(g_last_to[st] = d, s, n);
    g_pending[st].push_back({static_cast<const char *>(s), n});
    g_pending[st].push_back({static_cast<const char *>(d), n});
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    return *s = reinterpret_cast<cudaStream_t>(++g_handles), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return g_pending[s].clear(), done(); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return done(); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = reinterpret_cast<cudaEvent_t>(++g_handles), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return done(); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return done(); }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) { return memset(a, 0, sizeof(*a)), cudaSuccess; }
cudaError_t cudaLaunchHostFunc(cudaStream_t, cudaHostFn_t f, void *p) { return f(p), done(); }
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { return done(); }

// what the compiler's registration of the file's own kernel calls
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }

size_t gcz_zstd_frames_bound(size_t n) { return n + n / 128 + 1024; }
}

namespace gcz {
cudaError_t launch_zstd_match(const ZstdLaunch &, cudaStream_t) { return done(); }
cudaError_t launch_lzma_match(const LzmaLaunch &, cudaStream_t) { return done(); }
cudaError_t launch_cand_sweep(const uint8_t *, uint64_t, uint32_t, uint32_t, uint16_t *, uint32_t, int, cudaStream_t,
                              const WinDesc *, int, bool) {
    return done();
}
size_t zstd2_seg_scratch_entries(uint32_t n) { return n * 1024ull; }
cudaError_t launch_zstd_parse(const Zstd2Launch &, cudaStream_t) { return done(); }
cudaError_t launch_expand_seqs(const void *, const uint32_t *, uint64_t *offsets, uint32_t num, uint32_t, void *,
                               uint64_t, uint32_t *, int, cudaStream_t, bool, uint32_t *status_out) {
    memset(offsets, 0, (num + 1) * 8ull);
    if (status_out) *status_out = 0;
    return done();
}
cudaError_t launch_zstd_literals(const uint8_t *, uint64_t, uint32_t, uint32_t, const uint32_t *, const uint32_t *,
                                 uint32_t, uint8_t *, int, cudaStream_t) {
    return done();
}
cudaError_t launch_lzma_verify(const LzmaLaunch &, const uint16_t *, cudaStream_t) { return done(); }
cudaError_t launch_lzma_unpack(const uint32_t *, uint64_t, uint32_t, uint32_t, uint32_t, uint32_t *, uint32_t *,
                               uint32_t *, int, cudaStream_t) {
    return done();
}
cudaError_t launch_zenc(const ZencLaunch &, cudaStream_t) { return done(); }
cudaError_t launch_zenc_compact(const ZencLaunch &l, uint64_t *offsets, uint8_t *, uint64_t, cudaStream_t) {
    memset(offsets, 0, (l.num_windows + 1) * 8ull);
    return done();
}
}  // namespace gcz
