// engine_host.h -- the engine's host code (csrc/engine.cu) on a fake CUDA
// runtime and fake kernels, for checks that need no GPU: "device" memory is
// host memory, every stream operation happens at once and takes the next
// number of one sequence, an event holds the number at which it was
// recorded, and any call can be told to fail.  Include once per program.
#pragma once
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <cuda_runtime.h>

namespace fake {

struct Event {
    long long at = 0;
};

long long seq = 0;          // stream operations so far
long long waited_for = 0;   // the latest operation a host wait covered
int fail_malloc = -1;       // cudaMalloc calls until one fails (-1: none)
bool fail_force = false;    // the next force launch fails
int prepared = 0;           // prepare_small_force calls
long long force_at = 0;     // number of the last force launch
int one_launch_calls = 0, small_calls = 0, force_calls = 0, predictions = 0, scatters = 0;
int small_fits = 1;         // what small_force_fits answers
int nsplit = 4;             // splits of every shape
unsigned *word = nullptr;   // status word of the last force launch
unsigned report = 0;        // what the next force launch leaves there

}  // namespace fake

cudaError_t fake_cudaSetDevice(int) { return cudaSuccess; }
cudaError_t fake_cudaGetLastError() { return cudaSuccess; }
const char *fake_cudaGetErrorString(cudaError_t) { return "injected"; }
cudaError_t fake_cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t fake_cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = reinterpret_cast<cudaStream_t>(1); return cudaSuccess; }
cudaError_t fake_cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t fake_cudaStreamSynchronize(cudaStream_t) { fake::waited_for = fake::seq; return cudaSuccess; }
cudaError_t fake_cudaStreamQuery(cudaStream_t) { fake::waited_for = fake::seq; return cudaSuccess; }
cudaError_t fake_cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t fake_cudaEventCreate(cudaEvent_t *e) { *e = reinterpret_cast<cudaEvent_t>(new fake::Event); return cudaSuccess; }
cudaError_t fake_cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return fake_cudaEventCreate(e); }
cudaError_t fake_cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<fake::Event *>(e); return cudaSuccess; }
cudaError_t fake_cudaEventRecord(cudaEvent_t e, cudaStream_t) { reinterpret_cast<fake::Event *>(e)->at = fake::seq; return cudaSuccess; }
cudaError_t fake_cudaEventSynchronize(cudaEvent_t e) {
    fake::waited_for = std::max(fake::waited_for, reinterpret_cast<fake::Event *>(e)->at);
    return cudaSuccess;
}
cudaError_t fake_cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
template <class T>
cudaError_t fake_cudaMalloc(T **q, size_t n) {
    void **p = reinterpret_cast<void **>(q);
    if (fake::fail_malloc >= 0 && fake::fail_malloc-- == 0) return cudaErrorMemoryAllocation;
    *p = calloc(1, n ? n : 1);
    return cudaSuccess;
}
template <class T>
cudaError_t fake_cudaMallocHost(T **p, size_t n) {
    *p = static_cast<T *>(calloc(1, n ? n : 1));
    return cudaSuccess;
}
cudaError_t fake_cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t fake_cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t fake_cudaMemset(void *p, int v, size_t n) { ++fake::seq; memset(p, v, n); return cudaSuccess; }
cudaError_t fake_cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return fake_cudaMemset(p, v, n); }
cudaError_t fake_cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { ++fake::seq; memcpy(d, s, n); return cudaSuccess; }
cudaError_t fake_cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) { return fake_cudaMemcpy(d, s, n, k); }
cudaError_t fake_cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h,
                                     cudaMemcpyKind, cudaStream_t) {
    ++fake::seq;
    for (size_t r = 0; r < h; ++r) memcpy(static_cast<char *>(d) + r * dp, static_cast<const char *>(s) + r * sp, w);
    return cudaSuccess;
}

#define cudaDeviceGetAttribute fake_cudaDeviceGetAttribute
#define cudaEventCreate fake_cudaEventCreate
#define cudaEventCreateWithFlags fake_cudaEventCreateWithFlags
#define cudaEventDestroy fake_cudaEventDestroy
#define cudaEventElapsedTime fake_cudaEventElapsedTime
#define cudaEventRecord fake_cudaEventRecord
#define cudaEventSynchronize fake_cudaEventSynchronize
#define cudaFree fake_cudaFree
#define cudaFreeHost fake_cudaFreeHost
#define cudaGetErrorString fake_cudaGetErrorString
#define cudaGetLastError fake_cudaGetLastError
#define cudaMalloc fake_cudaMalloc
#define cudaMallocHost fake_cudaMallocHost
#define cudaMemcpy fake_cudaMemcpy
#define cudaMemcpy2DAsync fake_cudaMemcpy2DAsync
#define cudaMemcpyAsync fake_cudaMemcpyAsync
#define cudaMemset fake_cudaMemset
#define cudaMemsetAsync fake_cudaMemsetAsync
#define cudaSetDevice fake_cudaSetDevice
#define cudaStreamCreateWithFlags fake_cudaStreamCreateWithFlags
#define cudaStreamDestroy fake_cudaStreamDestroy
#define cudaStreamQuery fake_cudaStreamQuery
#define cudaStreamSynchronize fake_cudaStreamSynchronize
#define cudaStreamWaitEvent fake_cudaStreamWaitEvent
#include "engine.cu"

namespace fake {

void apply(const g6::SmallCall &sc, double *jraw, int *jindex) {
    for (int k = 0; k < sc.n_upd; ++k) {
        for (int f = 0; f < g6::JF_COUNT; ++f) jraw[(size_t)f * sc.cap + sc.addr[k]] = sc.vals[k][f];
        jindex[sc.addr[k]] = sc.index[k];
    }
}

// The fake force of i = the sum of the masses of the j it was given records
// of, as its potential; no acc, jerk or neighbour.
void force(const g6::ForceParams &p) {
    force_at = ++seq;
    if (p.nsplit == 0 && nsplit > 1) memset(p.part, 0, (size_t)nsplit * p.ni * sizeof(g6::Partial));
    const g6::JRecF64 *r = static_cast<const g6::JRecF64 *>(p.jrec);
    for (int i = 0; i < p.ni; ++i) {
        double m = 0;
        for (int j = 0; j < p.nj; ++j) m += r[j].pos.w;
        p.out_pot[i] = m;
        for (int c = 0; c < 3; ++c) p.out_acc[3 * i + c] = p.out_jerk[3 * i + c] = 0;
        p.out_nn[i] = 0;
    }
    word = p.status;
    *p.status |= report;
    report = 0;
}

void predict(const double *jraw, int cap, int nj, int nj_pad, void *jrec) {
    ++predictions;
    g6::JRecF64 *r = static_cast<g6::JRecF64 *>(jrec);
    for (int j = 0; j < nj_pad; ++j) r[j].pos.w = j < nj ? jraw[(size_t)g6::JF_M * cap + j] : 0.0;
}

}  // namespace fake

namespace g6 {
int tile_size(int kmode) { return tile_of(kmode); }
ForceConfig fill_config(int, int, int, int) {
    ForceConfig c{32, 1, 8, 8, fake::nsplit};
    return c;
}
ForceConfig choose_config(int k, int ni, int nj_pad, int sms, bool) { return fill_config(k, ni, nj_pad, sms); }
size_t partial_bytes(const ForceConfig &c, int ni) { return c.nsplit > 1 ? (size_t)c.nsplit * ni * sizeof(Partial) : 0; }
size_t partial_bytes_fixed(int jper, int nj_pad, int ni) {
    return (size_t)std::max(1, (nj_pad + jper - 1) / jper) * ni * sizeof(Partial);
}
bool small_force_fits(const ForceConfig &, ForceParams) { return fake::small_fits; }
int small_force_variant(const ForceConfig &cfg, bool ident, bool nb, bool g4) { return nb + 2 * ident + 4 * g4; }
cudaError_t prepare_small_force(int) {
    ++fake::prepared;
    return cudaSuccess;
}
cudaError_t launch_force(cudaStream_t, int, const ForceConfig &, ForceParams p, bool, bool, bool, bool) {
    if (fake::fail_force) return fake::fail_force = false, cudaErrorLaunchFailure;
    ++fake::force_calls;
    if (p.status_clear) *p.status_clear = 0;
    fake::force(p);
    return cudaSuccess;
}
cudaError_t launch_small_force(cudaStream_t, const ForceConfig &, ForceParams p, const SmallCall &sc, double *jraw,
                               int *jindex, unsigned *status2, bool, bool) {
    if (fake::fail_force) return fake::fail_force = false, cudaErrorLaunchFailure;
    ++fake::one_launch_calls;
    fake::apply(sc, jraw, jindex);
    fake::predict(jraw, sc.cap, sc.nj, sc.nj_pad, const_cast<void *>(p.jrec));
    status2[sc.parity ^ 1] = 0;
    fake::force(p);
    return cudaSuccess;
}
void launch_small_call(cudaStream_t, int, const SmallCall &sc, double *jraw, int *jindex, void *jrec, IRec *irec,
                       double *, unsigned *status2) {
    ++fake::seq;
    ++fake::small_calls;
    fake::apply(sc, jraw, jindex);
    if (sc.predict) fake::predict(jraw, sc.cap, sc.nj, sc.nj_pad, jrec);
    memcpy(irec, sc.irec, sizeof(IRec) * sc.ni);
    status2[sc.parity ^ 1] = 0;
}
void launch_predict(cudaStream_t, int, const double *jraw, const int *, int cap, int nj, int nj_pad, double,
                    const FixedScale &, void *jrec, unsigned *) {
    ++fake::seq;
    fake::predict(jraw, cap, nj, nj_pad, jrec);
}
void launch_scatter(cudaStream_t, int n, const StagedJ *staged, double *jraw, int *jindex, int cap, unsigned *copied,
                    unsigned seq) {
    ++fake::seq;
    *copied = seq;
    ++fake::scatters;
    for (int k = 0; k < n; ++k) {
        for (int f = 0; f < JF_COUNT; ++f) jraw[(size_t)f * cap + staged[k].addr] = staged[k].vals[f];
        jindex[staged[k].addr] = staged[k].index;
    }
}
// not reached by these checks
void launch_scatter_bulk(cudaStream_t, int, const BulkJ &, double *, int *, int) { abort(); }
void launch_irec_from_j(cudaStream_t, const double *, const int *, int, int, int, double, IRec *) { ++fake::seq; }
void launch_energy(cudaStream_t, int, int, const IRec *, const double *, int, const double *, double *) { ++fake::seq; }
void launch_refine_v2(cudaStream_t, const double *, int, int, double *) { abort(); }
cudaError_t launch_refine(cudaStream_t, const RefineArgs &, int) { abort(); }
int split_log2_blocks(long long) { return 0; }
void launch_split_agree(cudaStream_t, int, int, const Partial *, long long *) { abort(); }
void launch_split_fix(cudaStream_t, int, int, int, long long, const Partial *, const long long *, long long *,
                      long long *) { abort(); }
void launch_split_finish(cudaStream_t, int, int, long long, const long long *, const long long *, const long long *,
                         double *, double *, double *, int *) { abort(); }
cudaError_t launch_nb_compact(cudaStream_t, int ni, const int *, const int *, int, long long *off, int *) {
    memset(off, 0, sizeof(long long) * (ni + 1));
    return cudaSuccess;
}
cudaError_t launch_nb_full_g4(cudaStream_t, const void *, int, const IRec &, double, int *, int, int *) { abort(); }
void launch_copy_wait_selftest(cudaStream_t, unsigned *, unsigned long long) { abort(); }
}  // namespace g6
