// Failing CUDA calls, on the host: this program defines the runtime's functions that
// the library uses (its own definitions come first in the dynamic linker's order),
// over host memory and without running a kernel, and lets chosen ones fail.  Copies
// back to the host land when their stream is waited for, as on a device.
// Usage: test_faults CASE [ARGUMENT...]
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../par2-rs_b200/csrc/common.cuh"

// ---- the runtime -----------------------------------------------------------

namespace {
std::mutex g_mu;
std::map<void *, size_t> g_device;  // live device allocations
size_t g_used = 0, g_room = size_t(1) << 40;
int g_fail_syncs = 0;  // cudaStreamSynchronize calls that fail from now on
struct Copy {
    void *dst;
    const void *src;
    size_t n;
};
std::vector<Copy> g_pending;

// launches by kernel (the library registers its kernels before main starts)
std::map<const void *, std::string> &kernels()
{
    static std::map<const void *, std::string> m;
    return m;
}
std::map<std::string, int> g_launches;
cudaError_t launched(const void *fn)
{
    ++g_launches[kernels()[fn]];
    return cudaSuccess;
}
int launches(const char *part)
{
    int n = 0;
    for (const auto &x : g_launches)
        if (x.first.find(part) != std::string::npos)
            n += x.second;
    return n;
}

void land()
{
    for (const Copy &c : g_pending)
        memcpy(c.dst, c.src, c.n);
    g_pending.clear();
}
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
    std::lock_guard<std::mutex> l(g_mu);
    if (g_used + n > g_room)
        return cudaErrorMemoryAllocation;
    *p = aligned_alloc(256, (n + 255) / 256 * 256);
    memset(*p, 0, n < 65536 ? n : 65536);  // larger ones are not read by the cases
    g_device[*p] = n;
    g_used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    std::lock_guard<std::mutex> l(g_mu);
    land();
    g_used -= g_device[p];
    g_device.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n)
{
    *p = calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void *p)
{
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
    std::lock_guard<std::mutex> l(g_mu);
    if (k == cudaMemcpyDeviceToHost)
        g_pending.push_back({d, s, n});
    else
        memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t)
{
    for (size_t i = 0; i < h; ++i)
        memcpy(static_cast<char *>(d) + i * dp, static_cast<const char *>(s) + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t)
{
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    std::lock_guard<std::mutex> l(g_mu);
    if (g_fail_syncs > 0) {
        --g_fail_syncs;
        return cudaErrorUnknown;
    }
    land();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t)
{
    std::lock_guard<std::mutex> l(g_mu);
    land();
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 1.f;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int)
{
    memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int)
{
    *v = 10;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 1;
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "injected"; }
#define OK(name, ...) \
    cudaError_t name(__VA_ARGS__) { return cudaSuccess; }
OK(cudaGetLastError, void)
OK(cudaSetDevice, int)
OK(cudaStreamDestroy, cudaStream_t)
OK(cudaStreamWaitEvent, cudaStream_t, cudaEvent_t, unsigned)
OK(cudaEventDestroy, cudaEvent_t)
OK(cudaEventRecord, cudaEvent_t, cudaStream_t)
OK(cudaEventQuery, cudaEvent_t)
OK(cudaFuncSetAttribute, const void *, cudaFuncAttribute, int)
#undef OK
cudaError_t cudaLaunchKernel(const void *fn, dim3, dim3, void **, size_t, cudaStream_t) { return launched(fn); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *fn, void **) { return launched(fn); }
void **__cudaRegisterFatBinary(void *)
{
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *)
{
    kernels()[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    static char stream;
    *s = reinterpret_cast<cudaStream_t>(&stream);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    static char event;
    *e = reinterpret_cast<cudaEvent_t>(&event);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
}

// ---- the cases -------------------------------------------------------------

#define CHECK(c)                                                                        \
    do {                                                                                \
        if (!(c)) {                                                                     \
            printf("%s:%d: %s (last error: %s)\n", __FILE__, __LINE__, #c, p2g_last_error()); \
            return 1;                                                                   \
        }                                                                               \
    } while (0)

// A "device" buffer of n slices of S bytes and their addresses.
static std::vector<uint8_t *> slices(size_t n, size_t S)
{
    void *p = nullptr;
    const size_t pitch = (S + 15) / 16 * 16;
    cudaMalloc(&p, n * pitch);
    std::vector<uint8_t *> v(n);
    for (size_t i = 0; i < n; ++i)
        v[i] = static_cast<uint8_t *>(p) + i * pitch;
    return v;
}

// The last wait of a device repair fails: the call reports that, not a singular
// matrix read from a word that never arrived.
static int repair_sync(p2g_ctx *ctx)
{
    const size_t k = 60, m = 5, S = 4096;
    const auto present = slices(k - m, S), rec = slices(m, S), out = slices(m, S);
    uint64_t missing[m];
    uint32_t exps[m];
    for (size_t i = 0; i < m; ++i) {
        missing[i] = 3 * i;
        exps[i] = static_cast<uint32_t>(i);
    }
    auto repair = [&] {
        return p2g_repair(ctx, k, S, missing, m, present.data(), exps, rec.data(), out.data(), P2G_DEVICE_PTRS);
    };
    CHECK(repair() == P2G_OK);
    g_fail_syncs = 1;
    CHECK(repair() == P2G_ECUDA);
    CHECK(strstr(p2g_last_error(), "cudaStreamSynchronize"));
    CHECK(repair() == P2G_OK);
    return 0;
}

// A batch of one CREATE job; returns p2g_batch_create's or p2g_batch_run's code.
static int run_create(p2g_ctx *ctx, const std::vector<uint8_t *> &src, const std::vector<uint8_t *> &out, size_t S)
{
    std::vector<uint32_t> exps(out.size());
    for (size_t i = 0; i < exps.size(); ++i)
        exps[i] = static_cast<uint32_t>(i);
    p2g_job J = {};
    J.kind = P2G_JOB_CREATE;
    J.k = src.size();
    J.slice_bytes = S;
    J.src = src.data();
    J.n = out.size();
    J.exps = exps.data();
    J.out = out.data();
    p2g_batch *b = nullptr;
    if (const int rc = p2g_batch_create(ctx, &J, 1, 0, &b))
        return rc;
    const int rc = p2g_batch_run(b);
    p2g_batch_destroy(b);
    return rc;
}

// Forms that are all -1 are the heuristic's, tensor cores included, as NULL is.
static int forms(p2g_ctx *ctx)
{
    const size_t S = 65536;
    const auto src = slices(2000, S), out = slices(100, S);
    const int none[P2G_BATCH_CLASSES] = {-1, -1, -1, -1, -1, -1, -1, -1};
    const int one[P2G_BATCH_CLASSES] = {-1, -1, -1, P2G_FORM_WIDE, -1, -1, -1, -1};
    const int *tries[] = {nullptr, none, one, none};
    for (const int *f : tries) {
        CHECK(p2g_batch_set_forms(ctx, f) == P2G_OK);
        g_launches.clear();
        CHECK(run_create(ctx, src, out, S) == P2G_OK);
        CHECK(launches("tensor_muladd") == (f == one ? 0 : 1));
        CHECK(launches("muladd_persistent") == (f == one ? 1 : 0));
    }
    return 0;
}

// A batch tuner that fails leaves the pinned forms pinned.
static int tune_fails(p2g_ctx *ctx)
{
    const size_t S = 65536;
    const auto src = slices(2000, S), out = slices(100, S);
    const int wide[P2G_BATCH_CLASSES] = {0, 0, 0, 0, 0, 0, 0, 0};
    CHECK(p2g_batch_set_forms(ctx, wide) == P2G_OK);
    g_room = g_used + (1 << 20);
    CHECK(p2g_batch_autotune(ctx, 1, nullptr, nullptr) == P2G_ENOMEM);
    g_room = size_t(1) << 40;
    g_launches.clear();
    CHECK(run_create(ctx, src, out, S) == P2G_OK);
    CHECK(launches("tensor_muladd") == 0 && launches("muladd_persistent") == 1);
    return 0;
}

// A batch whose tensor-core operands do not fit falls back to the tables, also where
// the first of the two buffers did fit (and would leave no room for the tables').
static int batch_room(p2g_ctx *&ctx)
{
    const size_t S = 65536;
    const auto src = slices(2000, S), out = slices(100, S);
    // forms 252 MB and coefficients 6.9 MB; planes 131 MB and records 6.4 MB; each
    // with a quarter of headroom
    for (const size_t mb : {1000, 318, 200}) {
        g_room = g_used + mb * 1000000;
        g_launches.clear();
        CHECK(run_create(ctx, src, out, S) == P2G_OK);
        CHECK(launches("tensor_muladd") == (mb == 1000 ? 1 : 0));
        CHECK(launches("muladd_persistent") == (mb == 1000 ? 0 : 1));
        // a fresh context: no spare buffers
        CHECK(p2g_destroy(ctx) == P2G_OK);
        g_room = size_t(1) << 40;
        CHECK(p2g_create(0, &ctx) == P2G_OK);
    }
    return 0;
}

// An autotuner without room for the tensor cores' operands tunes the tables.
static int tune_room(p2g_ctx *ctx)
{
    // planes 134 MB and records 6.3 MB; coefficients for the tensor cores 31 MB
    p2g_plan plan;
    g_room = g_used + 150000000;
    CHECK(p2g_autotune(ctx, 65535, 1, 64, 1, &plan) == P2G_OK);
    CHECK(plan.tile_symbols == 1024 && !strcmp(p2g_last_error(), ""));
    // less than the tables take is still an error
    g_room = g_used + (1 << 20);
    CHECK(p2g_autotune(ctx, 65535, 30, 4096, 1, &plan) == P2G_ENOMEM);
    return 0;
}

// Prints the device bytes that a batch of one job takes, without the quarter of
// headroom of its large buffers.
static int job_bytes(p2g_ctx *ctx, const char *kind, size_t k, size_t n, size_t S)
{
    const bool repair = !strcmp(kind, "repair");
    const auto src = slices(k, S), rec = slices(n, S), out = slices(n, S);
    std::vector<uint32_t> exps(n);
    std::vector<uint64_t> missing(n);
    for (size_t i = 0; i < n; ++i) {
        exps[i] = static_cast<uint32_t>(i);
        missing[i] = i;
    }
    p2g_job J = {};
    J.kind = repair ? P2G_JOB_REPAIR : P2G_JOB_CREATE;
    J.k = k;
    J.slice_bytes = S;
    J.src = src.data();
    J.n = n;
    J.exps = exps.data();
    J.missing = missing.data();
    J.recovery = rec.data();
    J.out = out.data();
    // scratch of the context that a first batch grows (decode matrices) stays
    p2g_batch *b = nullptr;
    CHECK(p2g_batch_create(ctx, &J, 1, 0, &b) == P2G_OK);
    p2g_batch_destroy(b);
    for (p2g::DevBuf &d : ctx->spare)
        d.release();
    ctx->spare.clear();
    const size_t before = g_used;
    CHECK(p2g_batch_create(ctx, &J, 1, 0, &b) == P2G_OK);
    printf("%zu\n", (g_used - before) / 5 * 4);
    p2g_batch_destroy(b);
    return 0;
}

// The plan that p2g_get_plan names is the one that calls run.
static int get_plan(p2g_ctx *ctx)
{
    struct {
        size_t k, r, S;
    } const shapes[] = {{20, 2, 4096}, {2048, 205, 1 << 16}, {2048, 4, 1 << 16}, {256, 13, 1 << 16}, {64, 24, 1 << 16},
                        {64, 120, 1 << 12}, {400, 150, 4096}};
    for (const auto &x : shapes) {
        const auto src = slices(x.k, x.S), out = slices(x.r, x.S);
        std::vector<uint32_t> exps(x.r);
        p2g_plan p;
        for (int pinned = 0; pinned < 2; ++pinned) {
            CHECK(p2g_get_plan(ctx, x.k, x.r, x.S, &p) == P2G_OK);
            g_launches.clear();
            CHECK(p2g_encode(ctx, src.data(), x.k, x.S, exps.data(), x.r, out.data(), P2G_DEVICE_PTRS) == P2G_OK);
            CHECK(launches("tensor_muladd") == (p.tile_symbols == 256));
            CHECK(launches("muladd_paired") == (p.tile_symbols == 512));
            CHECK(launches("muladd_bitsliced") == (p.tile_symbols == 1024));
            p.input_splits = 3;
            CHECK(p2g_set_plan(ctx, x.k, x.r, x.S, &p) == P2G_OK);
            p2g_plan q;
            CHECK(p2g_get_plan(ctx, x.k, x.r, x.S, &q) == P2G_OK);
            CHECK(!memcmp(&p, &q, sizeof p));
        }
    }
    p2g_plan p;
    CHECK(p2g_get_plan(ctx, 0, 1, 64, &p) == P2G_EINVAL && p2g_get_plan(ctx, 65536, 1, 64, &p) == P2G_ERANGE);
    return 0;
}

// Closed-form inverses: one CTA up to 64 rows where the call waits for them, up to 96
// beside a repair's first pass, up to 128 where repairs of a batch share the launch.
static int inverse_routes(p2g_ctx *ctx)
{
    const size_t S = 4096;
    for (const size_t m : {1, 64, 65, 96, 97, 128, 129}) {
        const size_t k = 3 * m + 5;
        std::vector<uint64_t> missing(m);
        std::vector<uint32_t> exps(m);
        std::vector<uint16_t> inv(m * m);
        for (size_t i = 0; i < m; ++i) {
            missing[i] = 2 * i;
            exps[i] = static_cast<uint32_t>(i);
        }
        const auto present = slices(k - m, S), rec = slices(m, S), out = slices(m, S);
        g_launches.clear();
        CHECK(p2g_reconstruction_matrix(ctx, k, missing.data(), m, exps.data(), inv.data()) == P2G_OK);
        CHECK(launches("vdm_small") == (m <= 64) && launches("vdm_quotients") == (m > 64));
        g_launches.clear();
        CHECK(p2g_repair(ctx, k, S, missing.data(), m, present.data(), exps.data(), rec.data(), out.data(),
                         P2G_DEVICE_PTRS) == P2G_OK);
        CHECK(launches("vdm_small") == (m <= 96) && launches("vdm_quotients") == (m > 96));
        p2g_job jobs[2] = {};
        for (p2g_job &J : jobs) {
            J.kind = P2G_JOB_REPAIR;
            J.k = k;
            J.slice_bytes = S;
            J.src = present.data();
            J.n = m;
            J.exps = exps.data();
            J.missing = missing.data();
            J.recovery = rec.data();
            J.out = out.data();
        }
        for (const int n : {1, 2}) {
            p2g_batch *b = nullptr;
            g_launches.clear();
            CHECK(p2g_batch_create(ctx, jobs, n, 0, &b) == P2G_OK);
            const bool one = m <= (n == 1 ? 64 : 128);
            CHECK(launches("vdm_small") == one && launches("vdm_quotients") == (one ? 0 : n));
            p2g_batch_destroy(b);
        }
    }
    return 0;
}

// Inputs from the host: problems that upload in many small parts are not multiplied
// in as many tensor-core launches, and go to the tables where those end sooner; where
// the link is what takes the time, the parts stay as many as they can.
static int upload_parts(p2g_ctx *ctx)
{
    struct {
        size_t k, r, S;
        int least, most;  // tensor_muladd launches of an encode
    } const shapes[] = {{1487, 185, 10716, 1, 8},  {200, 40, 200 << 10, 0, 0},  {256, 13, 64 << 10, 0, 0},
                        {1024, 102, 65536, 10, 32}, {100, 30, 64 << 10, 0, 1}};
    for (const auto &x : shapes) {
        std::vector<uint8_t> in(x.k * x.S), back(x.r * x.S);
        std::vector<const uint8_t *> src(x.k);
        std::vector<uint8_t *> out(x.r);
        std::vector<uint32_t> exps(x.r);
        std::vector<uint64_t> missing(x.r);
        for (size_t i = 0; i < x.k; ++i)
            src[i] = in.data() + i * x.S;
        for (size_t i = 0; i < x.r; ++i) {
            out[i] = back.data() + i * x.S;
            exps[i] = static_cast<uint32_t>(i);
            missing[i] = i;
        }
        g_launches.clear();
        CHECK(p2g_encode(ctx, src.data(), x.k, x.S, exps.data(), x.r, out.data(), 0) == P2G_OK);
        const int n = launches("tensor_muladd");
        CHECK(n >= x.least && n <= x.most);
        CHECK(n > 0 || launches("muladd_") > 0);
        // a pinned plan is kept, whatever the parts
        p2g_plan p;
        CHECK(p2g_get_plan(ctx, x.k, x.r, x.S, &p) == P2G_OK);
        CHECK(p2g_set_plan(ctx, x.k, x.r, x.S, &p) == P2G_OK);
        g_launches.clear();
        CHECK(p2g_encode(ctx, src.data(), x.k, x.S, exps.data(), x.r, out.data(), 0) == P2G_OK);
        CHECK((launches("tensor_muladd") > 0) == (p.tile_symbols == 256));
        g_launches.clear();
        CHECK(p2g_repair(ctx, x.k, x.S, missing.data(), x.r, src.data(), exps.data(), src.data(), out.data(), 0) ==
              P2G_OK);
        // and one launch for the second pass, or one a slab
        CHECK(launches("tensor_muladd") <= 2 * x.most + 2);
    }
    return 0;
}

int main(int argc, char **argv)
{
    p2g_ctx *ctx = nullptr;
    CHECK(p2g_create(0, &ctx) == P2G_OK);
    int rc = 2;
    if (argc == 2 && !strcmp(argv[1], "repair_sync"))
        rc = repair_sync(ctx);
    if (argc == 2 && !strcmp(argv[1], "tune_fails"))
        rc = tune_fails(ctx);
    if (argc == 2 && !strcmp(argv[1], "batch_room"))
        rc = batch_room(ctx);
    if (argc == 2 && !strcmp(argv[1], "tune_room"))
        rc = tune_room(ctx);
    if (argc == 6 && !strcmp(argv[1], "job_bytes"))
        rc = job_bytes(ctx, argv[2], strtoull(argv[3], nullptr, 10), strtoull(argv[4], nullptr, 10),
                       strtoull(argv[5], nullptr, 10));
    if (argc == 2 && !strcmp(argv[1], "upload_parts"))
        rc = upload_parts(ctx);
    if (argc == 2 && !strcmp(argv[1], "inverse_routes"))
        rc = inverse_routes(ctx);
    if (argc == 2 && !strcmp(argv[1], "get_plan"))
        rc = get_plan(ctx);
    if (argc == 2 && !strcmp(argv[1], "forms"))
        rc = forms(ctx);
    if (rc == 0) {
        CHECK(p2g_destroy(ctx) == P2G_OK);
        printf("ok\n");
    }
    return rc;
}
