// The CUDA runtime and the kernels' launchers as host stand-ins, so that the
// library's host code (cvm_api.cpp, included after this header) runs without a
// device: memory is the host's, work is "done" at once, and what a test wants
// to see -- live memory, waits, launches -- is recorded.  A test injects its
// events through `on_call` (by function name, before the call takes effect;
// a value other than cudaSuccess is returned in the call's place).
#pragma once

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

#include "cvm_internal.h"

namespace fake {

struct State {
    std::recursive_mutex mu;
    std::map<char *, size_t> device, pinned;  // live memory (device: pool and plain)
    size_t deviceBytes = 0, devicePeak = 0, frees = 0;
    std::set<void *> capturing;
    std::multiset<void *> synced;             // streams waited for
    std::map<std::string, long> calls;
    std::function<cudaError_t(const std::string &)> on_call;
    std::function<void(const char *, const cvm::FftClass &)> on_launch;
    uintptr_t next = 64;
    // host memory that the device can read: all of it, or one page-locked range
    int pageable = 1;
    const char *lockedFrom = nullptr, *lockedTo = nullptr;
    // what launch_den_poor and launch_tally report: blocks without a bound per
    // member, and the rows' steps that formed den, per source
    int poor = 0;
    std::function<unsigned long long(int)> formed;
};
inline State &state() {
    static State *s = new State;  // outlives the library's own statics
    return *s;
}

inline cudaError_t called(const char *name) {
    State &s = state();
    std::lock_guard<std::recursive_mutex> lk(s.mu);
    s.calls[name]++;
    return s.on_call ? s.on_call(name) : cudaSuccess;
}

inline cudaError_t alloc(void **p, size_t n, std::map<char *, size_t> &live, bool device) {
    State &s = state();
    std::lock_guard<std::recursive_mutex> lk(s.mu);
    *p = aligned_alloc(256, (n + 255) / 256 * 256);
    live[static_cast<char *>(*p)] = n;
    if (device) {
        s.deviceBytes += n;
        s.devicePeak = std::max(s.devicePeak, s.deviceBytes);
    }
    return cudaSuccess;
}
inline cudaError_t release(void *p, std::map<char *, size_t> &live, bool device) {
    State &s = state();
    std::lock_guard<std::recursive_mutex> lk(s.mu);
    auto it = live.find(static_cast<char *>(p));
    if (it == live.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    if (device) s.deviceBytes -= it->second;
    s.frees++;
    live.erase(it);
    free(p);
    return cudaSuccess;
}
// Whether [p, p + n) lies in one live device allocation.
inline bool inside(const void *p, size_t n) {
    State &s = state();
    std::lock_guard<std::recursive_mutex> lk(s.mu);
    char *c = static_cast<char *>(const_cast<void *>(p));
    auto it = s.device.upper_bound(c);
    if (it == s.device.begin()) return false;
    --it;
    return c >= it->first && c + n <= it->first + it->second;
}
inline cudaError_t handle(void **out) {
    State &s = state();
    std::lock_guard<std::recursive_mutex> lk(s.mu);
    *out = reinterpret_cast<void *>(s.next += 64);
    return cudaSuccess;
}
inline cudaError_t launched(const char *name, const cvm::FftClass *fc, const void *p, size_t n) {
    if (p && !inside(p, n)) {
        fprintf(stderr, "%s writes outside its allocation\n", name);
        abort();
    }
    State &s = state();
    std::lock_guard<std::recursive_mutex> lk(s.mu);
    cvm::count_launches(1);
    if (fc && s.on_launch) s.on_launch(name, *fc);
    return called(name);
}

}  // namespace fake

#define FAKE_CALL(name)                              \
    do {                                             \
        const cudaError_t e_ = fake::called(#name);  \
        if (e_ != cudaSuccess) return e_;            \
    } while (0)

extern "C" {
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    memset(static_cast<void *>(p), 0, sizeof *p);
    p->major = 10;
    p->minor = 3;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrPageableMemoryAccess ? fake::state().pageable : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *least, int *greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { return fake::handle(reinterpret_cast<void **>(p)); }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { FAKE_CALL(cudaMalloc); return fake::alloc(p, n, fake::state().device, true); }
cudaError_t cudaFree(void *p) { FAKE_CALL(cudaFree); return fake::release(p, fake::state().device, true); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) {
    FAKE_CALL(cudaMallocFromPoolAsync);
    return fake::alloc(p, n, fake::state().device, true);
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { FAKE_CALL(cudaFreeAsync); return fake::release(p, fake::state().device, true); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { FAKE_CALL(cudaHostAlloc); return fake::alloc(p, n, fake::state().pinned, false); }
cudaError_t cudaFreeHost(void *p) { FAKE_CALL(cudaFreeHost); return fake::release(p, fake::state().pinned, false); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    memset(static_cast<void *>(a), 0, sizeof *a);
    const char *c = static_cast<const char *>(p);
    if (c >= fake::state().lockedFrom && c < fake::state().lockedTo) {
        a->type = cudaMemoryTypeHost;
        a->devicePointer = a->hostPointer = const_cast<char *>(c);
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *, const void *, size_t, cudaMemcpyKind) { FAKE_CALL(cudaMemcpy); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    FAKE_CALL(cudaMemcpyAsync);
    if (n <= 16) memcpy(d, s, n);  // (counters are real, pixels and maps are not)
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *, size_t, const void *, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) {
    FAKE_CALL(cudaMemcpy2DAsync);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
    FAKE_CALL(cudaMemsetAsync);
    if (!fake::inside(p, n)) abort();
    (void)v;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return fake::handle(reinterpret_cast<void **>(s)); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return fake::handle(reinterpret_cast<void **>(s)); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    FAKE_CALL(cudaStreamSynchronize);
    fake::state().synced.insert(s);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return fake::handle(reinterpret_cast<void **>(e)); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return fake::handle(reinterpret_cast<void **>(e)); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    std::lock_guard<std::recursive_mutex> lk(fake::state().mu);
    fake::state().capturing.insert(s);
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
    std::lock_guard<std::recursive_mutex> lk(fake::state().mu);
    fake::state().capturing.erase(s);
    return fake::handle(reinterpret_cast<void **>(g));
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *st) {
    std::lock_guard<std::recursive_mutex> lk(fake::state().mu);
    *st = fake::state().capturing.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
    FAKE_CALL(cudaGraphInstantiate);
    return fake::handle(reinterpret_cast<void **>(x));
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { FAKE_CALL(cudaGraphLaunch); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { FAKE_CALL(cudaGraphExecDestroy); return cudaSuccess; }
}  // extern "C"

namespace cvm {

cudaError_t launch_gray(const uint8_t *, long long, int, int, uint8_t *d, long long dp, cudaStream_t) {
    return fake::launched("gray", nullptr, d, (size_t)dp);
}
cudaError_t launch_alpha_scan(const uint8_t *, long long, int, int, unsigned int *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_prep(const uint8_t *, long long, int, int, int, int, const uint8_t *, long long, int, int, DevParams *P, int n,
                        int, int, int, DevFrame *F, cudaStream_t, const DevParams *) {
    if (!fake::inside(F, sizeof *F)) abort();
    return fake::launched("prep", nullptr, P, (size_t)n * sizeof *P);
}
cudaError_t launch_fwd_rows(const uint8_t *, long long, int, int, const int *, const TileGeom &, const FftClass &fc, float2 *spec,
                            int cnS, cudaStream_t, int, const char *label, float, const float *, const unsigned long long *, float,
                            int) {
    return fake::launched(label ? label : "fwd_rows", &fc, spec, (size_t)fc.ntiles * cnS * fc.dftH * fc.hwp * 8);
}
cudaError_t launch_cols(int mode, const float2 *in, float2 *, int cnS, const TileGeom &, const FftClass &fc, int cls, int, const int *,
                        float, const MemberSet &ms, int nmembers, cudaStream_t, const char *) {
    const size_t one = (size_t)fc.ntiles * fc.dftH * fc.hwp * 8;
    if (!fake::inside(in, one * cnS)) abort();
    if (mode >= 2 && !fake::inside(ms.scratch[cls], one * nmembers)) abort();
    return fake::launched("cols", &fc, nullptr, 0);
}
bool den_table_rows(const FftClass &fc) { return fc.log2n >= 7 && fc.log2n <= 11; }
int inv_rows_ctas_per_tile(const FftClass &fc, int rowsMax, int *pairs, int, int, int, int) {
    *pairs = 4;
    return (std::min(rowsMax, fc.dftH) + 7) / 8;
}
cudaError_t launch_inv_rows(const TileGeom &, const FftClass &fc, int, int, const MemberSet &ms, int nmembers, int, int, int nparts,
                            Partial *p, int *, cvm_result *, cudaStream_t, int, unsigned int *, int) {
    if (ms.lanes && !ms.table && !fake::inside(ms.lanes, (size_t)ms.solo.rw * ms.solo.rh * 8)) abort();
    (void)nmembers;
    return fake::launched(ms.sat ? "inv_rows_table" : "inv_rows", &fc, p, (size_t)nparts * sizeof *p);
}
SepGrid sep_grid(int rwMax, int rhMax) {
    SepGrid g;
    memset(static_cast<void *>(&g), 0, sizeof g);
    g.ncx = (rwMax + 255) / 256;
    g.hp = (rwMax + 255) / 256 * 256;
    g.rhMax = rhMax;
    return g;
}
cudaError_t launch_sep_stats(const uint8_t *, long long, int, int, int ih, const MemberSet &, int, int, int, const SepGrid &sg, int,
                             int cnMax, unsigned int *H, size_t, cudaStream_t, int, cudaStream_t, cudaEvent_t, unsigned int *, int,
                             cudaEvent_t) {
    return fake::launched("sep_stats", nullptr, H, (size_t)ih * sg.hp * (cnMax == 1 ? 2 : 4) * 4);
}
cudaError_t launch_vblock(const unsigned int *, unsigned int *B, int nblk, size_t n, cudaStream_t) {
    return fake::launched("vblock", nullptr, B, (size_t)nblk * n * 4);
}
cudaError_t launch_den_poor(const MemberSet &ms, int n, int *poor, cudaStream_t) {
    if (!fake::inside(ms.table, (size_t)n * sizeof(DevMember))) abort();
    *poor = fake::state().poor * n;
    return fake::launched("den_poor", nullptr, poor, 4);
}
cudaError_t launch_tally(const unsigned int *words, DenTally *out, unsigned int seq, int source, cudaStream_t) {
    const auto &formed = fake::state().formed;
    out->source = source;
    out->poor = words[0];
    out->formed = formed ? formed(source) : 0;
    out->seq = seq;
    return fake::launched("tally", nullptr, words, kTallyWords * 4);
}
cudaError_t launch_row_prefix(const uint8_t *, long long, int, int, int, int, unsigned int *P, int, cudaStream_t) {
    return fake::launched("row_prefix", nullptr, P, 4);
}
size_t sat_scratch_elems(int ih, int hp, int np) { return (size_t)((ih + 3) / 4) * hp * (np == 4 ? 6 : 2); }
cudaError_t launch_sat(const uint8_t *, long long, int, int ih, int hp, int np, const int *, unsigned int *B, unsigned int *S,
                       cudaStream_t) {
    if (!fake::inside(S, (size_t)(ih + 1) * hp * (np == 4 ? 6 : 2) * 4)) abort();
    return fake::launched("sat", nullptr, B, sat_scratch_elems(ih, hp, np) * 4);
}
cudaError_t upload_bytes(void *, const void *, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ingest(void *d, size_t p, const void *, size_t, size_t, int rows, cudaStream_t) {
    return fake::launched("ingest", nullptr, d, p * rows);
}
cudaError_t launch_ingest_solo(const SoloSource *, uint8_t *d, long long ip, int, int ih, uint8_t *t, long long tp, int, int th, int,
                               int, unsigned int *z, int zw, cudaStream_t) {
    if (!fake::inside(t, (size_t)tp * th) || !fake::inside(z, (size_t)zw * 4)) abort();
    return fake::launched("ingest_solo", nullptr, d, (size_t)ip * ih);
}
cudaError_t launch_shrink_gather(const float2 *, int, float2 *, int, int, int, cudaStream_t) { return cudaSuccess; }
size_t peaks_scratch_ints(int w, int h) { return (size_t)h * ((w + 255) / 256) * 9; }
cudaError_t launch_peaks(const float *, int w, int h, float, int, int, int *s, int32_t *, int, int *, cudaStream_t) {
    return fake::launched("peaks", nullptr, s, peaks_scratch_ints(w, h) * 4);
}
cudaError_t tc_selftest(double *, double *) { return cudaSuccess; }
cudaError_t tc_init() { return cudaSuccess; }
int tc_error_read_clear() { return 0; }
int rows_error_read_clear() { return 0; }
void profile_enable(int) {}
bool profile_on() { return false; }
int profile_read(int, char *, size_t, double *, unsigned long long *) { return -1; }
int profile_span(int, char *, size_t, double *, double *) { return -1; }

}  // namespace cvm

#define EXPECT(c)                                                                \
    do {                                                                         \
        if (!(c)) {                                                              \
            fprintf(stderr, "%s:%d: expected %s\n", __FILE__, __LINE__, #c);     \
            exit(1);                                                             \
        }                                                                        \
    } while (0)
