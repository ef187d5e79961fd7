/* A CUDA runtime on the host for cb_api.cpp, cb_pool.cpp and cb_ensemble.cu: "device" memory is
 * host memory, kernels do nothing, and copies to the host stay queued on their
 * stream until it is waited for. A test can make one of those copies fail. Built
 * and run by test_host_path.py, which needs no GPU. */
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <malloc.h>
#include <mutex>
#include <vector>

#include "cb_handle.h"

using namespace cb;

namespace {

struct Copy {
    cudaStream_t stream;
    void *dst;
    const void *src;
    size_t bytes;
};
std::mutex mu;
std::vector<Copy> queued;
size_t fail_bytes = 0;    /* copies to the host of this size count ... */
int fail_at = -1;         /* ... and this one of them fails */

int waits = 0, ones = 0, twos = 0;   /* waits for a stream or event, one-step and two-step launches */
bool two_step = false;               /* the two-step pass applies */
size_t room = (size_t)-1;            /* bytes of an allocation that still fit */
int timed_out = 0;                   /* error word that a step leaves in the record */

void run_stream(cudaStream_t s) {
    std::lock_guard<std::mutex> lock(mu);
    std::vector<Copy> rest;
    for (const Copy &c : queued) {
        if (c.stream == s) std::memcpy(c.dst, c.src, c.bytes);
        else rest.push_back(c);
    }
    queued = rest;
}

size_t queued_for(const void *dst, size_t bytes) {
    std::lock_guard<std::mutex> lock(mu);
    size_t n = 0;
    for (const Copy &c : queued) n += (const char *)c.dst >= (const char *)dst && (const char *)c.dst < (const char *)dst + bytes;
    return n;
}

}  // namespace

/* memory that was used before */
extern "C" void *aligned_alloc(size_t align, size_t bytes) {
    void *p = memalign(align, bytes);
    if (p) std::memset(p, 0x5a, bytes);
    return p;
}

extern "C" {
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) {
    return n <= room && (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaMalloc(void **p, size_t n) { return cudaMallocAsync(p, n, nullptr); }
cudaError_t cudaFree(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, cudaMemcpyKind) { return std::memcpy(dst, src, n), cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind kind, cudaStream_t s) {
    if (kind != cudaMemcpyDeviceToHost) return std::memcpy(dst, src, n), cudaSuccess;
    std::lock_guard<std::mutex> lock(mu);
    if (n == fail_bytes && fail_at-- == 0) return cudaErrorUnknown;
    queued.push_back({s, dst, src, n});
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = (cudaStream_t)std::malloc(1), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return run_stream(s), std::free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return ++waits, run_stream(s), cudaSuccess; }
/* an event is the stream it was recorded on */
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)std::calloc(1, sizeof(cudaStream_t)), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return *(cudaStream_t *)e = s, cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) { return run_stream(*(cudaStream_t *)e), cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return ++waits, cudaEventQuery(e); }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorName(cudaError_t) { return "fake"; }
const char *cudaGetErrorString(cudaError_t) { return "a fake's error"; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaErrorNotSupported; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

/* a start without the initial condition */
int cb_create_from_seed(const cb_params *p, const cb_ic_params *, const char *, cb_sums *first, char *, size_t, size_t *,
                        cb_handle **out) {
    size_t n = 1;
    for (int i = 0; i < p->d; ++i) n *= (size_t)p->n_grids;
    return cb_create_from_ic(p, std::vector<double>(n, 1.0).data(), nullptr, first, out);
}
}

namespace cb {
int finish_writer(cb_handle *) { return CB_OK; }
void free_fft(cb_handle *) {}
size_t ic_blocks(const StepConst &) { return 1; }
size_t step_blocks(const StepConst &) { return 1; }
int step2tb_steps(const StepConst &, int, int, bool) { return 0; }
bool step3df_applies(const StepConst &, int) { return false; }
bool step3tb_geometry(const StepConst &, int, int tl, int &, int &, size_t &, unsigned &, int &) { return two_step && tl == 2; }
/* no member of these tests is batched */
int batch2_kind(const StepConst &, int) { return 0; }
int batch2_steps(const std::vector<int> &, int, int, int) { return 0; }
int batch2_threads(const std::vector<int> &, int, int, int) { return 0; }
std::vector<int> batch2_tiles(const std::vector<int> &, int, int, int) { return {}; }
cudaError_t launch_step2_batch(int, int, const Batch2Member *, const std::vector<int> &, int, int, int, double *, cudaStream_t) {
    return cudaErrorNotSupported;
}
cudaError_t launch_convert(int, int, const void *, void *, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_flush_drift(int, const StepConst &, const void *, const void *, void *, DevState *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ic_backkick(int, const StepConst &, const void *, void *, DevState *, double *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ic_energies(int, const StepConst &, const void *, const void *, void *, void *, void *, DevState *, double *,
                               cudaStream_t) { return cudaSuccess; }
/* between rows of doubles */
cudaError_t launch_repitch(int from, int to, const void *src, size_t sp, void *dst, size_t dp, int n, size_t rows, cudaStream_t s) {
    run_stream(s);
    for (size_t r = 0; from == P_FP64 && to == P_FP64 && r < rows; ++r)
        std::memcpy((double *)dst + r * dp, (const double *)src + r * sp, n * sizeof(double));
    return cudaSuccess;
}
cudaError_t launch_step(int, const StepConst &, bool, int, const void *, const void *, void *, void *, void *, void *, void *,
                        DevState *st, double *, cudaStream_t) {
    if (timed_out) st->err = timed_out;
    return ++ones, cudaSuccess;
}
cudaError_t launch_step2_tb(int, const StepConst &, int, bool, const void *, const void *, void *, void *, DevState *, double *,
                            cudaStream_t) { return cudaSuccess; }
cudaError_t launch_step3_df(int, const StepConst &, int, bool, void *, void *, void *, void *, DevState *, double *,
                            cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t launch_step3_ms(int, const StepConst &, int, void *, void *, void *, void *, DevState *, double *, cudaStream_t) {
    return cudaErrorNotSupported;
}
cudaError_t launch_step3_tb(int, const StepConst &, int, const void *, const void *, void *, void *, DevState *, cudaStream_t) {
    return ++twos, cudaSuccess;
}
}  // namespace cb

namespace {

#define CHECK(x)                                                                      \
    do {                                                                              \
        if (!(x)) return std::printf("line %d: not so: %s\n", __LINE__, #x), 1;        \
    } while (0)

cb_params params(int d, int n, int precision) {
    cb_params p;
    std::memset(&p, 0, sizeof p);
    p.d = d;
    p.n_grids = n;
    p.L = n / 8.0;
    p.c = 3.0;
    p.dt = 0.0125;
    p.mpl = 200.0;
    p.delta_v = 1.0;
    p.precision = precision;
    p.memorysave = 1;
    return p;
}

/* A download whose second field cannot be queued: no copy into the caller's
 * buffers is under way when the call returns. */
int download(int d, int n, int precision) {
    const cb_params p = params(d, n, precision);
    size_t sites = 1;
    for (int i = 0; i < d; ++i) sites *= (size_t)n;
    std::vector<double> start(sites, 0.5);
    cb_handle *h = nullptr;
    CHECK(cb_create_from_ic(&p, start.data(), nullptr, nullptr, &h) == CB_OK);
    std::vector<float> phi(sites), pi(sites);
    fail_bytes = sites * sizeof(float);
    fail_at = 1;
    CHECK(cb_get_fields_f32(h, phi.data(), pi.data(), nullptr, nullptr, nullptr) == CB_EDEVICE);
    CHECK(queued_for(phi.data(), fail_bytes) == 0 && queued_for(pi.data(), fail_bytes) == 0);
    fail_at = -1;
    CHECK(cb_get_fields_f32(h, phi.data(), pi.data(), nullptr, nullptr, nullptr) == CB_OK);
    CHECK(queued_for(phi.data(), fail_bytes) == 0 && queued_for(pi.data(), fail_bytes) == 0);
    return cb_destroy(h) == CB_OK ? 0 : 1;
}

/* A served run whose fields could not be downloaded hands out zeros, not what
 * their memory held before. */
int served(int n, int which) {
    cb_request req;
    std::memset(&req, 0, sizeof req);
    req.params = params(2, n, CB_FP32C);
    req.nt = 4;
    req.want_fields = 1;
    cb_pool *pool = nullptr;
    int64_t id = 0;
    const size_t sites = (size_t)n * n;
    fail_bytes = sites * sizeof(float);
    fail_at = which;
    CHECK(cb_pool_create(8ll << 30, 2, &pool) == CB_OK);
    CHECK(cb_pool_submit(pool, &req, nullptr, &id) == CB_OK);
    CHECK(cb_pool_wait(pool, id, 20000) == CB_OK);
    std::vector<float> phi(sites, 7.f), pi(sites, 7.f);
    int state = -1;
    CHECK(cb_pool_status(pool, id, &state, nullptr) == CB_OK && state == CB_REQ_FAILED);
    CHECK(cb_pool_result(pool, id, nullptr, 0, nullptr, phi.data(), pi.data(), nullptr, nullptr, 0) == CB_EDEVICE);
    for (size_t i = 0; i < sites; ++i) CHECK(phi[i] == 0.f && pi[i] == 0.f);
    return cb_pool_destroy(pool) == CB_OK ? 0 : 1;
}

/* The first steps of a static 3-D run: the launches of those steps and no others,
 * and no wait. */
int first_steps(int n, int precision) {
    const cb_params p = params(3, n, precision);
    std::vector<double> start((size_t)n * n * n, 0.5);
    cb_handle *h = nullptr;
    two_step = true;
    CHECK(cb_create_from_ic(&p, start.data(), nullptr, nullptr, &h) == CB_OK);
    waits = ones = twos = 0;
    CHECK(cb_step(h, 8, 0, nullptr) == CB_OK);
    CHECK(waits == 0 && ones == 0 && twos == 4);
    CHECK(cb_step(h, 3, 0, nullptr) == CB_OK);
    CHECK(waits == 0 && ones == 1 && twos == 5);
    int64_t launches = 0, steps = 0;
    CHECK(cb_get_counters(h, &launches, &steps) == CB_OK && launches == 6 && steps == 11);
    return cb_destroy(h) == CB_OK ? 0 : 1;
}

/* Padded rows on a device with little room beside the fields: they go up and come
 * down in smaller pieces. */
int little_room(int n) {
    const cb_params p = params(3, n, CB_FP64);
    const size_t sites = (size_t)n * n * n, field = (size_t)n * n * (n + 1) * sizeof(double);
    std::vector<double> start(sites), phi(sites), pi(sites);
    for (size_t i = 0; i < sites; ++i) start[i] = 0.25 + (double)i;
    cb_handle *h = nullptr;
    CHECK(cb_create_from_ic(&p, start.data(), start.data(), nullptr, &h) == CB_OK);
    room = field / 7;   /* the staging buffer was released after the set-up */
    CHECK(cb_get_fields(h, phi.data(), pi.data(), nullptr, nullptr, nullptr) == CB_OK);
    CHECK(phi == start && pi == start);
    room = (size_t)-1;
    return cb_destroy(h) == CB_OK ? 0 : 1;
}

/* An ensemble whose member's step ended in a wait that ran out says so. */
int ensemble_timeout() {
    const cb_params p = params(3, 16, CB_FP64);
    std::vector<double> start(16 * 16 * 16, 0.5);
    cb_handle *h = nullptr;
    cb_ensemble *e = nullptr;
    cb_sums lines[4];
    CHECK(cb_create_from_ic(&p, start.data(), nullptr, nullptr, &h) == CB_OK);
    CHECK(cb_ensemble_create(1, &h, &e) == CB_OK);
    CHECK(cb_ensemble_step(e, 4, 2, lines) == CB_OK);
    timed_out = 0x71;
    CHECK(cb_ensemble_step(e, 4, 2, lines) == CB_ETIMEOUT);
    timed_out = 0;
    CHECK(cb_ensemble_destroy(e) == CB_OK);
    return cb_destroy(h) == CB_OK ? 0 : 1;
}

}  // namespace

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    int bad = 0;
    if (what == "download") bad = download(2, 64, CB_FP32C) || download(2, 64, CB_FP64) || download(3, 65, CB_FP32C);
    else if (what == "served") bad = served(1500, 0) || served(1500, 1) || served(64, 1);
    else if (what == "first") bad = first_steps(64, CB_FP64) || first_steps(65, CB_FP32C) || first_steps(128, CB_FP32C);
    else if (what == "ensemble") bad = ensemble_timeout();
    else if (what == "room") bad = little_room(65);
    else bad = std::printf("what?\n");
    std::printf(bad ? "failed\n" : "ok\n");
    return bad ? 1 : 0;
}
