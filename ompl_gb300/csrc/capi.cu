// C ABI of libgbompl (include/gbompl.h): object lifetimes, argument checking, guard-band bounds,
// the uniform grid over world spheres, staging for host-memory calls, and kernel launches.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include <random>

#include <nvtx3/nvToolsExt.h>

#include "chain_state.cuh"
#include "nn_device.cuh"
#include "tma.cuh"

using namespace gbo;

namespace
{
thread_local std::string g_err;
std::atomic<unsigned long long> g_launches{0};

gbo_status fail(gbo_status s, const std::string &msg)
{
    g_err = msg;
    return s;
}

#define CUDA_TRY(expr)                                                                                               \
    do                                                                                                               \
    {                                                                                                                \
        cudaError_t _e = (expr);                                                                                     \
        if (_e != cudaSuccess)                                                                                       \
        {                                                                                                            \
            cudaGetLastError(); /* reported here, not by the next call's launch check */                             \
            return fail(_e == cudaErrorMemoryAllocation ? GBO_ERR_OUT_OF_MEMORY : GBO_ERR_CUDA,                      \
                        std::string(#expr) + ": " + cudaGetErrorString(_e));                                         \
        }                                                                                                            \
    } while (0)

#define CHECK_LAUNCH()                                                                                               \
    do                                                                                                               \
    {                                                                                                                \
        cudaError_t _e = cudaGetLastError();                                                                         \
        if (_e != cudaSuccess)                                                                                       \
            return fail(GBO_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(_e));                      \
    } while (0)

int g_sm_count = 0;
int g_device_ok = -1;  // -1 unknown, 0 no, 1 yes

gbo_status ensure_device()
{
    if (g_device_ok == 1)
        return GBO_OK;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0)
    {
        cudaGetLastError();
        g_device_ok = 0;
        return fail(GBO_ERR_NO_DEVICE, "no CUDA device");
    }
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceProp p;
    if (cudaGetDeviceProperties(&p, dev) != cudaSuccess)
        return fail(GBO_ERR_NO_DEVICE, "cudaGetDeviceProperties failed");
    if (!(p.major == 10 && p.minor == 3))
        return fail(GBO_ERR_NO_DEVICE, "libgbompl is built for sm_103a only; device is sm_" +
                                           std::to_string(p.major) + std::to_string(p.minor));
    g_sm_count = p.multiProcessorCount;
    g_device_ok = 1;
    return GBO_OK;
}

LaunchCfg lcfg(gbo_stream s)
{
    LaunchCfg lc;
    lc.stream = (cudaStream_t)s;
    lc.sm_count = g_sm_count;
    return lc;
}

constexpr double kU32 = 5.9604644775390625e-08;  // 2^-24, FP32 unit roundoff
// Bound on |cos/sin FP32 - exact| of one link direction (sincos_ff, chain_warp.cuh): Horner rounding
// <= 2 ulp (1.2e-7), Taylor truncation <= 2e-9, reduction and low-part terms < 1e-12.
constexpr double kEpsDir = 1.3e-7;
constexpr double kPiH = 3.141592653589793238462643383279502884;

bool valid_layout(int layout, int64_t n, int64_t ld, int dim)
{
    if (layout == GBO_LAYOUT_SOA)
        return ld >= n;
    if (layout == GBO_LAYOUT_AOS)
        return ld >= dim;
    return false;
}

// Ring of device counter slots so that calls in flight on different streams do not share one.
struct CounterRing
{
    RunCounters *dev = nullptr;
    std::atomic<unsigned> next{0};
    unsigned last = 0;
    static constexpr unsigned kSlots = 64;
    gbo_status init()
    {
        CUDA_TRY(cudaMalloc(&dev, sizeof(RunCounters) * kSlots));
        CUDA_TRY(cudaMemset(dev, 0, sizeof(RunCounters) * kSlots));
        return GBO_OK;
    }
    RunCounters *take(cudaStream_t s)
    {
        unsigned i = next.fetch_add(1) % kSlots;
        last = i;
        cudaMemsetAsync(dev + i, 0, sizeof(RunCounters), s);
        return dev + i;
    }
    ~CounterRing()
    {
        if (dev)
            cudaFree(dev);
    }
};

struct Pinned
{
    void *p = nullptr;
    size_t bytes = 0;
    gbo_status reserve(size_t b)
    {
        if (b <= bytes)
            return GBO_OK;
        if (p)
            cudaFreeHost(p);
        p = nullptr;
        bytes = 0;
        CUDA_TRY(cudaMallocHost(&p, b));
        bytes = b;
        return GBO_OK;
    }
    ~Pinned()
    {
        if (p)
            cudaFreeHost(p);
    }
};

// Whether work enqueued on s is being captured into a graph (and does not run now)
bool capturing(cudaStream_t s)
{
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) == cudaSuccess)
        return st != cudaStreamCaptureStatusNone;
    cudaGetLastError();  // the legacy stream beside another stream's capture
    return false;
}

// Per-object device scratch that grows geometrically with the stream-ordered allocator. Outgrown
// buffers are kept until the object is destroyed: freeing them during a call would synchronise the
// whole device (cudaFree) and stall every other stream. Grown in a call that is being captured, a buffer is
// ordinary memory: a stream-ordered allocation would be the graph's, gone for later calls.
struct DevBuf
{
    void *p = nullptr;
    size_t bytes = 0;
    std::vector<void *> outgrown;
    gbo_status reserve(size_t b, cudaStream_t stream = nullptr)
    {
        if (b <= bytes)
            return GBO_OK;
        const size_t want = std::max(b, 2 * bytes);
        void *np = nullptr;
        if (capturing(stream))
        {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            CUDA_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
            const cudaError_t e = cudaMalloc(&np, want);
            cudaThreadExchangeStreamCaptureMode(&mode);
            CUDA_TRY(e);
        }
        else
            CUDA_TRY(cudaMallocAsync(&np, want, stream));
        if (p)
            outgrown.push_back(p);
        p = np;
        bytes = want;
        return GBO_OK;
    }
    ~DevBuf()
    {
        if (p || !outgrown.empty())
            cudaDeviceSynchronize();
        if (p)
            cudaFree(p);
        for (void *q : outgrown)
            cudaFree(q);
    }
};

// Staging of the *_rows calls: buffers per call in flight, so that a thread waiting for its stream holds up no other.
// As many as calls have overlapped, freed with the object. Page-locked memory is made by a call that overlaps none, and
// at once as large as a small batch can need: making it waits for all the device's work.
constexpr size_t kRowBytes = 128 * 1024;
struct RowBuffers
{
    Pinned pin;
    void *plain = nullptr;
    size_t plain_bytes = 0;
    DevBuf dev;
    bool pinned = false;
    RowBuffers *next = nullptr;  // idle ones of a pool
    ~RowBuffers() { std::free(plain); }
};
struct RowPool
{
    std::mutex mu;
    RowBuffers *idle = nullptr;
    int out = 0;
    ~RowPool()
    {
        while (RowBuffers *b = idle)
        {
            idle = b->next;
            delete b;
        }
    }
};
struct RowCall
{
    RowPool &pool;
    cudaStream_t s;
    RowBuffers *b;
    bool enqueued = false;
    RowCall(RowPool &p, cudaStream_t stream) : pool(p), s(stream)
    {
        std::lock_guard<std::mutex> lk(pool.mu);
        b = pool.idle;
        if (b)
            pool.idle = b->next;
        else if ((b = new (std::nothrow) RowBuffers()))
            b->pinned = pool.out == 0;
        ++pool.out;
    }
    // before the buffers are another call's, what this one enqueued on them is done, also after an error
    ~RowCall()
    {
        if (enqueued && cudaStreamSynchronize(s) != cudaSuccess)
            cudaGetLastError();
        std::lock_guard<std::mutex> lk(pool.mu);
        if (b)
        {
            b->next = pool.idle;
            pool.idle = b;
        }
        --pool.out;
    }
    gbo_status reserve(size_t bytes)
    {
        bytes = std::max(bytes, kRowBytes);
        if (!b)
            return fail(GBO_ERR_OUT_OF_MEMORY, "staging allocation failed");
        if (b->pinned)
        {
            if (auto e = b->pin.reserve(bytes))
                return e;
        }
        else if (b->plain_bytes < bytes)
        {
            std::free(b->plain);
            b->plain = std::malloc(bytes);
            b->plain_bytes = b->plain ? bytes : 0;
            if (!b->plain)
                return fail(GBO_ERR_OUT_OF_MEMORY, "staging allocation failed");
        }
        return b->dev.reserve(bytes, s);
    }
    char *host() const { return (char *)(b->pinned ? b->pin.p : b->plain); }
    char *device() const { return (char *)b->dev.p; }
    gbo_status copy_in(size_t bytes)
    {
        enqueued = true;
        CUDA_TRY(cudaMemcpyAsync(device(), host(), bytes, cudaMemcpyHostToDevice, s));
        return GBO_OK;
    }
    gbo_status copy_out(size_t at, size_t bytes)
    {
        CUDA_TRY(cudaMemcpyAsync(host() + at, device() + at, bytes, cudaMemcpyDeviceToHost, s));
        enqueued = false;
        CUDA_TRY(cudaStreamSynchronize(s));
        return GBO_OK;
    }
};

size_t pad16(size_t b)
{
    return (b + 15) & ~size_t(15);
}
}  // namespace

struct gbo_space
{
    SpaceParams sp{};
    double extent = 0.0;
};

struct gbo_checker
{
    SpaceParams sp{};
    int kind = 0;
    int precision = GBO_PRECISION_FP64;
    WorldArgs wa{};
    void *d64 = nullptr, *d32 = nullptr;
    int *cell_start = nullptr, *cell_items = nullptr;
    float *cell_items4 = nullptr;
    __half *clr = nullptr;
    ArmTail *tail = nullptr;  // one list per counter slot
    unsigned *test_order = nullptr;
    unsigned long long *masks = nullptr;
    CounterRing ctr;
    int tuned_schedule = -1;
    std::mutex mu, tune_mu;
    cudaStream_t host_stream = nullptr;
    Pinned pin_in, pin_out;
    DevBuf dev_in, dev_out;
    RowPool rows;
    ~gbo_checker()
    {
        if (d64)
            cudaFree(d64);
        if (d32)
            cudaFree(d32);
        if (cell_start)
            cudaFree(cell_start);
        if (cell_items)
            cudaFree(cell_items);
        if (cell_items4)
            cudaFree(cell_items4);
        if (clr)
            cudaFree(clr);
        if (tail)
            cudaFree(tail);
        if (test_order)
            cudaFree(test_order);
        if (masks)
            cudaFree(masks);
        if (host_stream)
            cudaStreamDestroy(host_stream);
    }
};

struct gbo_sampler
{
    SpaceParams sp{};
    SamplerState *st = nullptr;
    std::mutex mu;
    cudaStream_t host_stream = nullptr;
    Pinned pin;
    DevBuf dev, words;  // words: the word-stream scratch of the device calls
    DevBuf gwork;       // GaussChunk, per-CTA counts and pairs of sampleGaussian
    bool has_saved = false;  // mirrors SamplerState::has_saved (a cached Gaussian value is pending)
    ~gbo_sampler()
    {
        if (host_stream)
            cudaStreamDestroy(host_stream);
        if (st)
            cudaFree(st);
    }
};

// Cell index of a gbo_nn over a RealVector / wrapped space (kernels_nn_cells.cu), over its first `size` elements:
// built by the first large batch after a change of the element set (add / remove / clear clear `size`).
struct NNBoxCells
{
    int64_t size = 0;
    BoxCellShape shape{};
    DevBuf start, cstart, skey, kmin, pts8, box, extent;
    gbo_status reserve(int64_t n, cudaStream_t s)
    {
        const size_t sub = (size_t)shape.C << shape.bits, chunks = (size_t)n / 32 + shape.C + 1;
        for (auto r : {start.reserve((sub + 1) * sizeof(int), s), cstart.reserve(((size_t)shape.C + 1) * sizeof(int), s),
                       skey.reserve((size_t)n * sizeof(int), s), kmin.reserve(chunks * sizeof(int), s),
                       pts8.reserve((size_t)n * 2 * sizeof(float4), s), box.reserve(chunks * 4 * sizeof(float4), s),
                       extent.reserve(16 * sizeof(float), s)})
            if (r)
                return r;
        return GBO_OK;
    }
    BoxCellArgs args() const
    {
        return BoxCellArgs{shape.L, shape.C, shape.bits, shape.dA, shape.nA, shape.nB, (const int *)start.p,
                           (const int *)cstart.p, (const int *)skey.p, (const int *)kmin.p, (const float4 *)pts8.p,
                           (const float4 *)box.p, (const float *)extent.p};
    }
};
constexpr int kCellLevels = 12;  // indexes over size, size / 2, ... elements (prefix limits)

// Cell index of a kinematic-chain gbo_nn (kernels_nn.cu), built like NNBoxCells.
struct NNChainCells
{
    bool valid = false;
    DevBuf key, count, start, fill, skey, sfeat, box, cstart, cbox;
};

struct gbo_nn
{
    SpaceParams sp{};
    int precision = GBO_PRECISION_FP32_GUARDED;
    int64_t cap = 0, size = 0, alive_count = 0;
    int F = 0;
    double *pts64 = nullptr;
    float *feat32 = nullptr;
    float4 *feat4 = nullptr;
    int *outside = nullptr;  // device flag: an element lies outside the bounds eps32 was derived for
    unsigned char *alive = nullptr;
    float eps32 = 0.f;
    NNBoxCells cells[kCellLevels];
    int64_t forgone = 0;  // pairs above the cell search's worth that batches took without an index
    DevBuf cwork;  // scratch of the cell builds and query orders
    NNChainCells ccells;
    DevBuf qfeat, fb_list, part, qorder;
    DevBuf ranks;  // keys of the present elements in order (approximate nearest after removals)
    CounterRing ctr;
    unsigned long long queries = 0;
    std::mutex mu;
    std::mutex search_mu;  // the set, its indexes and the scratch, while a call enqueues (SearchOrder)
    cudaEvent_t searched = nullptr;
    unsigned long long searched_on = 0;
    bool in_flight = false;
    cudaStream_t host_stream = nullptr;
    Pinned pin;
    DevBuf dev;
    RowPool rows;
    ~gbo_nn()
    {
        if (searched)
            cudaEventDestroy(searched);
        if (host_stream)
            cudaStreamDestroy(host_stream);
        if (pts64)
            cudaFree(pts64);
        if (feat32)
            cudaFree(feat32);
        if (feat4)
            cudaFree(feat4);
        if (outside)
            cudaFree(outside);
        if (alive)
            cudaFree(alive);
    }
};

namespace
{
// NVTX range over a C-ABI call (visible to ncu / Nsight; no cost without an attached tool)
struct Trace
{
    explicit Trace(const char *name) { nvtxRangePushA(name); }
    ~Trace() { nvtxRangePop(); }
};
}  // namespace

namespace gbo
{
void note_launch()
{
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

int persistent_grid(const void *kernel, int block, unsigned smem, const LaunchCfg &lc, int64_t max_blocks)
{
    static std::mutex mu;
    static std::map<std::pair<const void *, std::pair<unsigned, int>>, int> occ;
    static std::map<const void *, bool> raised;
    int per_sm = 0;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (smem > 48 * 1024 && !raised[kernel])
        {
            // raise the kernel's dynamic shared-memory limit once, to the device's opt-in maximum, so
            // that launches with any world size up to it remain valid
            int dev = 0, optin = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 1024);
            raised[kernel] = true;
        }
        auto key = std::make_pair(kernel, std::make_pair(smem, block));
        auto it = occ.find(key);
        if (it == occ.end())
        {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem);
            if (per_sm < 1)
                per_sm = 1;
            occ[key] = per_sm;
        }
        else
            per_sm = it->second;
    }
    int64_t g = (int64_t)per_sm * lc.sm_count;
    if (max_blocks < g)
        g = max_blocks;
    return (int)(g < 1 ? 1 : g);
}

unsigned world_smem_bytes(const WorldArgs &wa, int precision)
{
    if (precision == GBO_PRECISION_FP32_GUARDED &&
        (wa.kind == GBO_CHECK_CHAIN_SEGMENTS || wa.kind == GBO_CHECK_DH_SPHERES))
        return wa.stage32 ? wa.bytes32 : 0;
    return wa.stage64 ? wa.bytes64 : 0;
}
}  // namespace gbo

namespace
{
// Guard-band bounds of the FP32 kinematic-chain test (see checkers.cuh). All bounds are
// worst-case: eps_dir covers float conversion of the reduced angle (u*pi) plus the sincosf error
// (2 ulp); link vectors VX = c*L have error L*(eps_dir + 2u); a position after k links has error
// k*(L*(eps_dir + u) + u*R) with R the reach; a cross product a x b of vectors with component
// magnitudes <= A, B and component errors da, db has error 2*(da*B + db*A + da*db) + 3u*A*B.
// Each bound is inflated by a safety factor of 2.
void chain_bounds(const SpaceParams &sp, const double *w, int n, ChainGuard &g, std::vector<ChainSegF32> &segs,
                  float &e_dist)
{
    const double u = kU32, L = sp.link, nl = sp.dim;
    const double eps_dir = kEpsDir;
    const double R = nl * L + 0.001;
    const double dV = L * (eps_dir + 2 * u) + 1e-15;
    const double dP = (nl + 1) * (L * (eps_dir + u) + u * R) + 1e-15;
    auto cross = [&](double A, double B, double da, double db) {
        return 2.0 * (da * B + db * A + da * db) + 3.0 * u * A * B + 1e-15;
    };
    const double safety = 2.0;
    // one bound e for the four numerator comparisons (that of s_numer - denom or t_numer - denom,
    // which include the others), stored as the thresholds FLT_EPSILON -/+ e rounded outward
    const double flt_eps = std::ldexp(1.0, -23);
    auto down = [](double x) {
        float f = (float)x;
        return (double)f > x ? std::nextafter(f, -INFINITY) : f;
    };
    auto up = [](double x) {
        float f = (float)x;
        return (double)f < x ? std::nextafter(f, INFINITY) : f;
    };
    auto numer_bound = [&](double A, double B, double C, double eden, double es, double et) {
        const double eu = es + eden + u * 2 * (A * C + A * B), ev = et + eden + u * 2 * (B * C + A * B);
        return safety * std::max(std::max(es, et), std::max(eu, ev));
    };
    g.eps_dir = (float)eps_dir;
    {
        const double A = L, B = L, C = 2 * R, dC = 2 * dP + 2 * u * R;
        const double eden = cross(A, B, dV, dV), es = cross(A, C, dV, dC), et = cross(B, C, dV, dC);
        const double e = numer_bound(A, B, C, eden, es, et);
        g.self_den = up(safety * eden + 1e-12);
        g.self_lo = down(flt_eps - e);
        g.self_hi = up(flt_eps + e);
    }
    segs.resize(n);
    for (int j = 0; j < n; ++j)
    {
        const double x0 = w[4 * j], y0 = w[4 * j + 1], x1 = w[4 * j + 2], y1 = w[4 * j + 3];
        const double sx = x1 - x0, sy = y1 - y0;
        const double B = std::max(std::fabs(sx), std::fabs(sy));
        const double W0 = std::max(std::fabs(x0), std::fabs(y0));
        const double A = L, C = R + W0;
        const double dB = u * B, dC = dP + u * W0 + u * C;
        const double eden = cross(A, B, dV, dB), es = cross(A, C, dV, dC), et = cross(B, C, dB, dC);
        ChainSegF32 s{};
        s.x0 = (float)x0;
        s.y0 = (float)y0;
        s.sx = (float)sx;
        s.sy = (float)sy;
        const double e = numer_bound(A, B, C, eden, es, et);
        s.e_den = up(safety * eden + 1e-12);
        s.lo = down(flt_eps - e);
        s.hi = up(flt_eps + e);
        segs[j] = s;
    }
    // workspace distance (segment_count, FP32 form): dx_i accumulates 2i direction errors and i
    // roundings of partial sums bounded by 2i; the norm adds |ddx| + |ddy| and a relative 2^-22.
    double e = 0.0;
    for (int i = 1; i <= sp.dim; ++i)
    {
        const double ddx = 2.0 * i * eps_dir + u * 2.0 * i * i;
        e += 2.0 * ddx + std::ldexp(1.0, -21) * 2.0 * i;
    }
    e = L * (e + u * sp.dim * 2.0 * sp.dim) + u * L * 2.0 * sp.dim * sp.dim;
    e_dist = (float)(safety * e);
}

// Chain kNN features X_i = sum_{m<=i} cos(theta_m) accumulate i direction errors and i roundings.
float chain_knn_eps(const SpaceParams &sp)
{
    const double u = kU32, L = sp.link;
    const double eps_dir = kEpsDir;
    double e = 0.0;
    for (int i = 1; i <= sp.dim; ++i)
    {
        const double dX = i * eps_dir + u * i * i;            // one feature
        const double ddx = 2.0 * dX + u * 2.0 * i;            // difference of features
        e += 2.0 * ddx + std::ldexp(1.0, -21) * 2.0 * i + u * 2.0 * i * sp.dim;
    }
    return (float)(2.0 * L * e * 1.01 + 1e-12);
}

// Box / wrapped spaces: features are coordinates rounded to FP32 (error u*|x|), squared distance
// accumulated with FMA (relative error <= (dim + 2) u); bound on |sqrt(s32) - d64|.
float box_knn_eps(const SpaceParams &sp)
{
    double m2 = 0.0, span2 = 0.0;
    for (int d = 0; d < sp.dim; ++d)
    {
        const double lo = sp.kind == GBO_SPACE_REAL_VECTOR ? sp.low[d] : -kPiH;
        const double hi = sp.kind == GBO_SPACE_REAL_VECTOR ? sp.high[d] : kPiH;
        const double m = std::max(std::fabs(lo), std::fabs(hi));
        m2 += m * m;
        span2 += (hi - lo) * (hi - lo);
    }
    const double coord = 2.0 * kU32 * std::sqrt(m2) + (sp.kind == GBO_SPACE_REAL_VECTOR ? 0.0 : 4.0 * kU32 * 7.0);
    const double rel = (sp.dim + 4) * kU32 * std::sqrt(span2);
    return (float)(2.0 * (coord + rel) + 1e-12);
}
}  // namespace

// Segment-test order of a kinematic-chain checker. The validity result does not depend on the order in
// which the segment tests run; the warp-cooperative kernels stop at the first round of 32 tests that
// holds a definite intersection, so tests that are likely to intersect go first. The order is a greedy
// cover of the definite intersections found (FP32, guarded) in 8192 states drawn uniformly from the
// joint bounds: repeatedly take the test that intersects in most states not yet covered.
static gbo_status order_chain_tests(gbo_checker *c)
{
    const SpaceParams &sp = c->sp;
    const int n = sp.dim, m = n + 1, nw = c->wa.n;
    const int n_tests = (m - 1) * (m - 2) / 2 + m * nw;
    const int words = (n_tests + 31) / 32;
    const int S = 8192;
    std::mt19937_64 rng(0x9e3779b97f4a7c15ull);
    std::uniform_real_distribution<double> U(-kPiH, kPiH);
    std::vector<double> st((size_t)n * S);
    for (auto &x : st)
        x = U(rng);
    double *dst = nullptr;
    unsigned *dbits = nullptr;
    CUDA_TRY(cudaMalloc(&dst, st.size() * sizeof(double)));
    if (cudaMalloc(&dbits, (size_t)S * words * sizeof(unsigned)) != cudaSuccess)
    {
        cudaFree(dst);
        return fail(GBO_ERR_OUT_OF_MEMORY, "test-order scratch allocation failed");
    }
    cudaMemcpy(dst, st.data(), st.size() * sizeof(double), cudaMemcpyHostToDevice);
    WorldArgs wa = c->wa;
    wa.test_order = nullptr;
    launch_chain_hits(nullptr, sp, wa, dst, S, dbits, words);
    std::vector<unsigned> bits((size_t)S * words);
    cudaError_t e = cudaMemcpy(bits.data(), dbits, bits.size() * sizeof(unsigned), cudaMemcpyDeviceToHost);
    cudaFree(dst);
    cudaFree(dbits);
    if (e != cudaSuccess)
        return fail(GBO_ERR_CUDA, std::string("test ordering: ") + cudaGetErrorString(e));
    // transpose to per-test state bitsets
    const int sw = S / 64;
    std::vector<uint64_t> tb((size_t)n_tests * sw, 0);
    for (int s = 0; s < S; ++s)
        for (int t = 0; t < n_tests; ++t)
            if (bits[(size_t)s * words + t / 32] >> (t % 32) & 1u)
                tb[(size_t)t * sw + s / 64] |= 1ull << (s % 64);
    std::vector<uint64_t> covered(sw, 0);
    std::vector<char> used(n_tests, 0);
    std::vector<unsigned> order;
    order.reserve(n_tests);
    for (int step = 0; step < n_tests; ++step)
    {
        int best = -1;
        long best_gain = -1;
        for (int t = 0; t < n_tests; ++t)
        {
            if (used[t])
                continue;
            long g = 0;
            for (int w = 0; w < sw; ++w)
                g += __builtin_popcountll(tb[(size_t)t * sw + w] & ~covered[w]);
            if (g > best_gain)
            {
                best_gain = g;
                best = t;
            }
        }
        if (best_gain <= 0)
            break;
        used[best] = 1;
        order.push_back(chain_test_entry(best, n, nw));
        for (int w = 0; w < sw; ++w)
            covered[w] |= tb[(size_t)best * sw + w];
    }
    for (int t = 0; t < n_tests; ++t)
        if (!used[t])
            order.push_back(chain_test_entry(t, n, nw));
    CUDA_TRY(cudaMalloc(&c->test_order, order.size() * sizeof(unsigned)));
    CUDA_TRY(cudaMemcpy(c->test_order, order.data(), order.size() * sizeof(unsigned), cudaMemcpyHostToDevice));
    c->wa.test_order = c->test_order;
    return GBO_OK;
}

// The masks of ChainMasks for a world of at most 64 finite segments.
static gbo_status build_chain_masks(gbo_checker *c, const double *world, int n)
{
    const double L = c->sp.link;
    if (n > 64 || !(L > 1e-3 && L < 1e3))
        return GBO_OK;
    for (int i = 0; i < 4 * n; ++i)
        if (!(std::fabs(world[i]) < 1e3 * L))
            return GBO_OK;
    constexpr int G = kChainMaskCells, K = kChainMaskBins;
    std::vector<unsigned long long> m((size_t)G * G + K, 0);
    const double half = c->sp.dim * L * 1.01, cell = 2.0 * half / G;
    const double reach = L * 33.0 / 64.0 + cell * 0.70711 + 1e-3 * L;
    const double eps = std::ldexp(1.0, -23);
    // position of a direction in [0, 1): 0.5 - 0.5 cos / (|cos| + |sin|) over the half turn [0, pi)
    auto place = [&](double t) {
        const double x = std::cos(t), y = std::sin(t);
        return 0.5 - 0.5 * (y < 0.0 ? -x : x) / (std::fabs(x) + std::fabs(y));
    };
    for (int j = 0; j < n; ++j)
    {
        const double dx = world[4 * j + 2] - world[4 * j], dy = world[4 * j + 3] - world[4 * j + 1];
        const double ax = world[4 * j] - dx / 64.0, ay = world[4 * j + 1] - dy / 64.0;  // lengthened at both ends
        const double bx = dx * (33.0 / 32.0), by = dy * (33.0 / 32.0), B = std::hypot(dx, dy);
        // the cells whose middle lies in the segment's box widened by `reach`
        const double b2 = bx * bx + by * by, far2 = reach * reach * (1.0 + 1e-12);
        auto first = [&](double lo) { return std::max(0, (int)std::floor((lo - reach + half) / cell - 0.5)); };
        auto last = [&](double hi) { return std::min(G - 1, (int)std::ceil((hi + reach + half) / cell - 0.5)); };
        const int p1 = last(std::max(ax, ax + bx)), q1 = last(std::max(ay, ay + by));
        for (int p = first(std::min(ax, ax + bx)); p <= p1; ++p)
            for (int q = first(std::min(ay, ay + by)); q <= q1; ++q)
            {
                const double x = -half + (p + 0.5) * cell - ax, y = -half + (q + 0.5) * cell - ay;
                const double t = b2 > 0.0 ? std::min(1.0, std::max(0.0, (x * bx + y * by) / b2)) : 0.0;
                const double ex = x - t * bx, ey = y - t * by;
                if (ex * ex + ey * ey <= far2)
                    m[(size_t)p * G + q] |= 1ull << j;
            }
        // |denom| = L B |sin|, 66 FLT_EPSILON against the rounding of the FP32 direction (and 1e-5 of an angle)
        const double s = L * B > 0.0 ? 66.0 * eps / (L * B) : 2.0;
        if (s >= 0.5)
        {
            for (int k = 0; k < K; ++k)
                m[(size_t)G * G + k] |= 1ull << j;
            continue;
        }
        const double d = std::asin(s) + 1e-5, phi = std::atan2(dy, dx);
        const int k0 = (int)std::floor(place(phi - d) * K) - 1, k1 = (int)std::floor(place(phi + d) * K) + 1;
        // increasing over the half turn; past its end the bins start again
        const int count = (k1 - k0 + 2 * K) % K;
        for (int k = 0; k <= count; ++k)
            m[(size_t)G * G + ((k0 + k) % K + K) % K] |= 1ull << j;
    }
    CUDA_TRY(cudaMalloc(&c->masks, m.size() * sizeof(m[0])));
    CUDA_TRY(cudaMemcpy(c->masks, m.data(), m.size() * sizeof(m[0]), cudaMemcpyHostToDevice));
    c->wa.masks = ChainMasks{c->masks, c->masks + G * G, (float)half, (float)(G / (2.0 * half))};
    return GBO_OK;
}

// Uniform grid over the circles' bounding box: as many cells a side (at most 256) as keep the lists below 16
// entries a circle (plus a floor for small worlds). None for a world with a value that is not finite.
static gbo_status build_circle_grid(gbo_checker *c, const double *world, int64_t n)
{
    CircleGrid &g = c->wa.circles;
    double lo[2] = {1e300, 1e300}, hi[2] = {-1e300, -1e300};
    for (int64_t i = 0; i < n; ++i)
        for (int d = 0; d < 2; ++d)
        {
            const double x = world[3 * i + d], r = std::fabs(world[3 * i + 2]);
            if (!(std::fabs(x) < 1e100 && r < 1e100))
                return GBO_OK;
            lo[d] = std::min(lo[d], x - r);
            hi[d] = std::max(hi[d], x + r);
        }
    if (n == 0 || !(hi[0] - lo[0] > 0.0) || !(hi[1] - lo[1] > 0.0))
        return GBO_OK;
    for (int d = 0; d < 2; ++d)
    {
        const double pad = 1e-6 * (hi[d] - lo[d]) + 1e-12 * std::max(std::fabs(lo[d]), std::fabs(hi[d]));
        lo[d] -= pad;
        hi[d] += pad;
    }
    std::vector<int> start, items;
    for (int G = 256; G >= 2; G /= 2)
    {
        const double cell[2] = {(hi[0] - lo[0]) / G, (hi[1] - lo[1]) / G};
        // the cells a thousandth of a cell around circle i: a row's run of cells follows from its distance in x
        const double inv[2] = {1.0 / cell[0], 1.0 / cell[1]};
        auto visit = [&](int64_t i, auto &&emit) {
            const double x = world[3 * i] - lo[0], y = world[3 * i + 1] - lo[1], r = std::fabs(world[3 * i + 2]);
            const double r2 = r * r * (1.0 + 1e-9);
            auto first = [&](double at) { return std::max(0, (int)std::floor(at - 2e-3)); };
            auto last = [&](double at) { return std::min(G - 1, (int)std::floor(at + 2e-3)); };
            const int p1 = last((x + r) * inv[0]);
            for (int p = first((x - r) * inv[0]); p <= p1; ++p)
            {
                const double b0 = (p - 1e-3) * cell[0], b1 = (p + 1.0 + 1e-3) * cell[0];
                const double gap = x < b0 ? b0 - x : (x > b1 ? x - b1 : 0.0);
                if (gap * gap > r2)
                    continue;
                const double w = std::sqrt(r2 - gap * gap);
                const int q1 = last((y + w) * inv[1]);
                for (int q = first((y - w) * inv[1]); q <= q1; ++q)
                    emit(p * G + q);
            }
        };
        const size_t most = 4096 + 16 * (size_t)n;
        size_t total = 0;
        start.assign((size_t)G * G + 1, 0);
        for (int64_t i = 0; i < n && total <= most; ++i)
            visit(i, [&](int k) {
                ++start[k + 1];
                ++total;
            });
        if (total > most)
            continue;
        for (size_t k = 0; k < (size_t)G * G; ++k)
            start[k + 1] += start[k];
        std::vector<int> fill(start.begin(), start.end() - 1);
        items.assign(std::max<size_t>(total, 1), 0);
        for (int64_t i = 0; i < n; ++i)
            visit(i, [&](int k) { items[fill[k]++] = (int)i; });
        CUDA_TRY(cudaMalloc(&c->cell_start, start.size() * sizeof(int)));
        CUDA_TRY(cudaMalloc(&c->cell_items, items.size() * sizeof(int)));
        CUDA_TRY(cudaMemcpy(c->cell_start, start.data(), start.size() * sizeof(int), cudaMemcpyHostToDevice));
        CUDA_TRY(cudaMemcpy(c->cell_items, items.data(), items.size() * sizeof(int), cudaMemcpyHostToDevice));
        g.n = G;
        for (int d = 0; d < 2; ++d)
        {
            g.lo[d] = lo[d];
            g.inv[d] = G / (hi[d] - lo[d]);
        }
        g.start = c->cell_start;
        g.items = c->cell_items;
        return GBO_OK;
    }
    return GBO_OK;
}

extern "C" {

const char *gbo_status_string(gbo_status s)
{
    switch (s)
    {
        case GBO_OK:
            return "ok";
        case GBO_ERR_INVALID_ARGUMENT:
            return "invalid argument";
        case GBO_ERR_CUDA:
            return "CUDA error";
        case GBO_ERR_NO_DEVICE:
            return "no usable device";
        case GBO_ERR_OUT_OF_MEMORY:
            return "out of memory";
        case GBO_ERR_TIMEOUT:
            return "device wait timed out";
        case GBO_ERR_UNSUPPORTED:
            return "unsupported";
        default:
            return "unknown status";
    }
}

const char *gbo_last_error(void)
{
    return g_err.c_str();
}

uint64_t gbo_launch_count(void)
{
    return g_launches.load();
}

gbo_status gbo_selftest_bounded_wait(int64_t limit_ns, double *elapsed_ms)
{
    if (limit_ns <= 0 || limit_ns > 2000000000ll)
        return fail(GBO_ERR_INVALID_ARGUMENT, "wait limit must be in (0, 2 s]");
    if (auto st = ensure_device())
        return st;
    unsigned long long *d = nullptr;
    CUDA_TRY(cudaMalloc(&d, 2 * sizeof(unsigned long long)));
    launch_wait_probe((unsigned long long)limit_ns, d);
    unsigned long long h[2] = {0, 0};
    const cudaError_t e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess)
        return fail(GBO_ERR_CUDA, std::string("bounded-wait self-test: ") + cudaGetErrorString(e));
    if (elapsed_ms)
        *elapsed_ms = (double)h[1] * 1e-6;
    return h[0] ? fail(GBO_ERR_TIMEOUT, "the probe's wait ran out, as intended") : GBO_OK;
}

gbo_status gbo_device_check(int *sm_count, int *cc_major, int *cc_minor)
{
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0)
    {
        cudaGetLastError();
        return fail(GBO_ERR_NO_DEVICE, "no CUDA device");
    }
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceProp p;
    CUDA_TRY(cudaGetDeviceProperties(&p, dev));
    if (sm_count)
        *sm_count = p.multiProcessorCount;
    if (cc_major)
        *cc_major = p.major;
    if (cc_minor)
        *cc_minor = p.minor;
    return ensure_device();
}

// ---------------------------------------------------------------- spaces
gbo_status gbo_space_create(int kind, int dim, const double *low, const double *high, double param, double lvs,
                            double lvs_fraction, unsigned factor, gbo_space **out)
{
    if (!out)
        return fail(GBO_ERR_INVALID_ARGUMENT, "out is NULL");
    if (kind < GBO_SPACE_REAL_VECTOR || kind > GBO_SPACE_WRAP_L2)
        return fail(GBO_ERR_INVALID_ARGUMENT, "unknown space kind");
    if (dim < 1 || dim > GBO_MAXD)
        return fail(dim > GBO_MAXD ? GBO_ERR_UNSUPPORTED : GBO_ERR_INVALID_ARGUMENT, "dimension must be 1..16");
    if (kind == GBO_SPACE_SO2 && dim != 1)
        return fail(GBO_ERR_INVALID_ARGUMENT, "SO2 has dimension 1");
    if (kind == GBO_SPACE_REAL_VECTOR && (!low || !high))
        return fail(GBO_ERR_INVALID_ARGUMENT, "RealVector bounds required");
    if (factor < 1)
        return fail(GBO_ERR_INVALID_ARGUMENT,
                    "The multiplicative factor for the valid segment count between two states must be strictly positive");
    auto *s = new gbo_space();
    s->sp.kind = kind;
    s->sp.dim = dim;
    s->sp.factor = factor;
    s->sp.link = param;
    for (int d = 0; d < dim; ++d)
    {
        if (kind == GBO_SPACE_REAL_VECTOR)
        {
            if (!(low[d] <= high[d]))
            {
                delete s;
                return fail(GBO_ERR_INVALID_ARGUMENT, "lower bound above upper bound");
            }
            s->sp.low[d] = low[d];
            s->sp.high[d] = high[d];
        }
        else
        {
            s->sp.low[d] = -kPiH;
            s->sp.high[d] = kPiH;
        }
    }
    // StateSpace::setup (StateSpace.cpp:237-249) with the kind's getMaximumExtent
    double e = 0.0;
    if (kind == GBO_SPACE_SO2)
        e = kPiH;
    else
    {
        for (int d = 0; d < dim; ++d)
        {
            const double r = kind == GBO_SPACE_WRAP_L2 ? kPiH : s->sp.high[d] - s->sp.low[d];
            e += r * r;
        }
        e = std::sqrt(e);
    }
    s->extent = e;
    if (lvs <= 0.0)
    {
        const double eps = 2.220446049250313e-16;
        if (lvs_fraction < eps || lvs_fraction > 1.0 - eps)
        {
            delete s;
            return fail(GBO_ERR_INVALID_ARGUMENT, "The fraction of the extent must be larger than 0 and less than 1");
        }
        lvs = e * lvs_fraction;
    }
    if (!(lvs >= 2.220446049250313e-16))
    {
        delete s;
        return fail(GBO_ERR_INVALID_ARGUMENT, "The longest valid segment must be positive.");
    }
    s->sp.lvs = lvs;
    *out = s;
    return GBO_OK;
}

gbo_status gbo_space_destroy(gbo_space *s)
{
    delete s;
    return GBO_OK;
}

gbo_status gbo_space_info(const gbo_space *s, double *max_extent, double *lvs)
{
    if (!s)
        return fail(GBO_ERR_INVALID_ARGUMENT, "space is NULL");
    if (max_extent)
        *max_extent = s->extent;
    if (lvs)
        *lvs = s->sp.lvs;
    return GBO_OK;
}

gbo_status gbo_space_distance(const gbo_space *s, const double *a, const double *b, int64_t n, int64_t ld, int layout,
                              double *out, gbo_stream stream)
{
    if (!s || (n > 0 && (!a || !b || !out)) || n < 0 || !valid_layout(layout, n, ld, s->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad distance arguments");
    if (auto st = ensure_device())
        return st;
    launch_distance(lcfg(stream), s->sp, make_view(a, ld, layout), make_view(b, ld, layout), n, out);
    CHECK_LAUNCH();
    return GBO_OK;
}

gbo_status gbo_space_interpolate(const gbo_space *s, const double *a, const double *b, const double *t, int64_t n,
                                 int64_t ld, int layout, double *out, gbo_stream stream)
{
    if (!s || (n > 0 && (!a || !b || !t || !out)) || n < 0 || !valid_layout(layout, n, ld, s->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad interpolate arguments");
    if (auto st = ensure_device())
        return st;
    StatesView ov = make_view(out, ld, layout);
    launch_interpolate(lcfg(stream), s->sp, make_view(a, ld, layout), make_view(b, ld, layout), t, n,
                       MutStatesView{out, ov.si, ov.sd});
    CHECK_LAUNCH();
    return GBO_OK;
}

gbo_status gbo_get_motion_states(const gbo_space *s, const double *s1, const double *s2, int64_t n, int64_t ld,
                                 int layout, unsigned count, int endpoints, double *out, int64_t out_ld,
                                 gbo_stream stream)
{
    const int64_t m = endpoints ? (int64_t)count + 2 : (int64_t)count;
    if (!s || n < 0 || (n > 0 && (!s1 || !s2 || (m > 0 && !out))) || !valid_layout(layout, n, ld, s->sp.dim) ||
        !valid_layout(layout, n * m, out_ld, s->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad getMotionStates arguments");
    if (n == 0 || m == 0)
        return GBO_OK;
    if (auto st = ensure_device())
        return st;
    StatesView ov = make_view(out, out_ld, layout);
    launch_motion_states(lcfg(stream), s->sp, make_view(s1, ld, layout), make_view(s2, ld, layout), n, count,
                         endpoints ? 1 : 0, MutStatesView{out, ov.si, ov.sd});
    CHECK_LAUNCH();
    return GBO_OK;
}

// ---------------------------------------------------------------- checkers
gbo_status gbo_checker_create(const gbo_space *space, int kind, const double *world, int64_t n_world,
                              const double *dh, int n_joints, int spheres_per_link, double sphere_radius,
                              gbo_checker **out)
{
    if (!space || !out)
        return fail(GBO_ERR_INVALID_ARGUMENT, "space/out is NULL");
    if (kind < GBO_CHECK_ALL_VALID || kind > GBO_CHECK_DH_BOXES)
        return fail(GBO_ERR_INVALID_ARGUMENT, "unknown checker kind");
    // boxes use the DH sphere-arm kernels with a box narrow phase (WorldArgs::boxes)
    const bool boxes = kind == GBO_CHECK_DH_BOXES;
    const int stride = boxes ? 6 : 4;
    if (n_world < 0 || (n_world > 0 && !world) || n_world > (1 << 24))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad world");
    const SpaceParams &sp = space->sp;
    if (kind == GBO_CHECK_CIRCLES && sp.dim != 2)
        return fail(GBO_ERR_INVALID_ARGUMENT, "the circle checker needs a 2-D space");
    if (kind == GBO_CHECK_CHAIN_SEGMENTS && sp.kind != GBO_SPACE_KINEMATIC_CHAIN)
        return fail(GBO_ERR_INVALID_ARGUMENT, "the chain checker needs a kinematic-chain space");
    if ((kind == GBO_CHECK_DH_SPHERES || boxes) &&
        (!dh || n_joints < 1 || n_joints > 8 || n_joints != sp.dim || spheres_per_link < 1 || sphere_radius < 0))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad DH arm (1..8 joints = space dimension)");
    if (auto st = ensure_device())
        return st;
    auto *c = new gbo_checker();
    c->sp = sp;
    c->kind = kind;
    WorldArgs &wa = c->wa;
    wa.kind = boxes ? GBO_CHECK_DH_SPHERES : kind;
    wa.boxes = boxes ? 1 : 0;
    wa.n = (int)n_world;
    wa.inv_lvs32 = (float)(1.0 / sp.lvs);
    auto cleanup = [&](gbo_status s) {
        delete c;
        return s;
    };
    if (c->ctr.init() != GBO_OK)
        return cleanup(GBO_ERR_OUT_OF_MEMORY);
    std::vector<double> w64;
    if (kind == GBO_CHECK_CIRCLES)
    {
        for (int64_t i = 0; i < n_world; ++i)
        {
            w64.push_back(world[3 * i]);
            w64.push_back(world[3 * i + 1]);
            w64.push_back(world[3 * i + 2] * world[3 * i + 2]);  // circles2D.h:51 r2_ = r * r
        }
    }
    else if (kind != GBO_CHECK_ALL_VALID)
        w64.assign(world, world + stride * n_world);
    size_t b64 = pad16(w64.size() * sizeof(double));
    if (b64)
    {
        if (cudaMalloc(&c->d64, b64) != cudaSuccess)
            return cleanup(fail(GBO_ERR_OUT_OF_MEMORY, "world allocation failed"));
        cudaMemset(c->d64, 0, b64);
        cudaMemcpy(c->d64, w64.data(), w64.size() * sizeof(double), cudaMemcpyHostToDevice);
    }
    wa.data64 = c->d64;
    wa.bytes64 = (unsigned)b64;
    if (kind == GBO_CHECK_CIRCLES)
        if (auto st = build_circle_grid(c, world, n_world))
            return cleanup(st);
    wa.stage64 = (b64 > 0 && !wa.circles.n && b64 <= 96 * 1024 && wa.kind != GBO_CHECK_DH_SPHERES) ? 1 : 0;
    if (kind == GBO_CHECK_CHAIN_SEGMENTS)
    {
        std::vector<ChainSegF32> segs;
        chain_bounds(sp, world, (int)n_world, wa.guard, segs, wa.e_dist);
        // trig hazard bound of the FP64 forms: joint k's position is a sum of k link vectors cos/sin * L;
        // the device's sines and cosines (CUDA's FP64 sincos, within 2 ulps, or the correctly rounded
        // ones) and the C library's (within 1 ulp) differ by at most 4 ulps (<= 4 * 2^-52), which moves
        // each product by at most 4 L 2^-52 plus its rounding, and each partial sum by its rounding
        // (2^-53 of the reach); safety factor 2
        {
            const double L = sp.link, reach = sp.dim * std::fabs(L) + 0.001;
            wa.hz_pos = 2.0 * (sp.dim + 1) * (std::fabs(L) * 0x1p-50 + std::fabs(L) * 0x1p-53 + reach * 0x1p-53);
        }
        size_t b32 = pad16(segs.size() * sizeof(ChainSegF32));
        if (b32)
        {
            if (cudaMalloc(&c->d32, b32) != cudaSuccess)
                return cleanup(fail(GBO_ERR_OUT_OF_MEMORY, "world allocation failed"));
            cudaMemcpy(c->d32, segs.data(), segs.size() * sizeof(ChainSegF32), cudaMemcpyHostToDevice);
        }
        wa.data32 = c->d32;
        wa.bytes32 = (unsigned)b32;
        wa.stage32 = b32 > 0 && b32 <= 96 * 1024;
        if (!wa.stage32 && b32)
            return cleanup(fail(GBO_ERR_UNSUPPORTED, "segment world too large for shared memory"));
        if (b32 && sp.dim <= 31)
            if (auto st = order_chain_tests(c))
                return cleanup(st);
        if (b32)
            if (auto st = build_chain_masks(c, world, (int)n_world))
                return cleanup(st);
    }
    if (wa.kind == GBO_CHECK_DH_SPHERES)
    {
        DHArm &arm = wa.arm;
        arm.joints = n_joints;
        arm.spl = spheres_per_link;
        arm.rs = sphere_radius;
        for (int i = 0; i < n_joints; ++i)
        {
            arm.a[i] = dh[3 * i];
            arm.d[i] = dh[3 * i + 1];
            const int code = (int)dh[3 * i + 2];
            if (code < -1 || code > 1)
                return cleanup(fail(GBO_ERR_INVALID_ARGUMENT, "alpha code must be -1, 0 or +1"));
            arm.ca[i] = code == 0 ? 1.f : 0.f;
            arm.sa[i] = code == 0 ? 0.f : (float)code;
            arm.af[i] = (float)arm.a[i];
            arm.dfl[i] = (float)arm.d[i];
            arm.len[i] = (float)(1.000001 * std::sqrt(arm.a[i] * arm.a[i] + arm.d[i] * arm.d[i]));
        }
        arm.rsf = (float)sphere_radius;
        arm.inv_spl = 1.0f / (float)spheres_per_link;
        // FP32 obstacles (rows as given)
        std::vector<float> s32(stride * n_world);
        double rmax = 0.0;
        for (int64_t i = 0; i < stride * n_world; ++i)
            s32[i] = (float)world[i];
        for (int64_t i = 0; i < n_world; ++i)
            rmax = std::max(rmax, boxes ? 0.0 : world[4 * i + 3]);
        size_t b32 = pad16(s32.size() * sizeof(float));
        if (b32)
        {
            if (cudaMalloc(&c->d32, b32) != cudaSuccess)
                return cleanup(fail(GBO_ERR_OUT_OF_MEMORY, "world allocation failed"));
            cudaMemcpy(c->d32, s32.data(), s32.size() * sizeof(float), cudaMemcpyHostToDevice);
        }
        wa.data32 = c->d32;
        wa.bytes32 = (unsigned)b32;
        wa.stage32 = 0;  // the FP32 narrow phase reads the spheres listed in the grid cells (cell_items4)
        // FK error bound in FP32 (spectral-norm propagation): |dR_k| <= k (2 eps_t + 16u),
        // |dp| <= sum_k (|dR_k| |pA| + |pA| (eps_t + u) + 4u (|p| + |pA|)); centres add 3u|p|.
        // angles: |q| <= qmax (the space's bounds; states beyond them are re-checked in FP64), rounded to
        // FP32 (u |q|, +1% for the float-float interpolation), sincosf within 2 ulp
        double qmax = kPiH;
        if (sp.kind == GBO_SPACE_REAL_VECTOR)
        {
            qmax = 0.0;
            for (int d = 0; d < sp.dim; ++d)
                qmax = std::max(qmax, std::max(std::fabs(sp.low[d]), std::fabs(sp.high[d])));
        }
        wa.dh_qmax = (float)qmax;
        const double u = kU32, eps_t = u * qmax * 1.01 + 2.0 * std::ldexp(1.0, -23);
        double dR = 0.0, dp = 0.0, reach = 0.0;
        for (int i = 0; i < n_joints; ++i)
        {
            const double pa = std::sqrt(arm.a[i] * arm.a[i] + arm.d[i] * arm.d[i]);
            reach += pa;
            dp += dR * pa + pa * (eps_t + u) * 2.0 + 4.0 * u * (reach + pa);
            dR += 2.0 * eps_t + 16.0 * u;
        }
        const double dc = (dp + 3.0 * u * reach) * std::sqrt(3.0);  // Euclidean centre error
        // the same propagation for the FP64 forms when every sine and cosine moves by 4 ulps (4 * 2^-52,
        // CUDA's FP64 sincos against the C library's): the trig hazard bound of a sphere centre
        // (safety factor 2)
        {
            const double u64 = 0x1p-53, et = 0x1p-50;
            double dR64 = 0.0, dp64 = 0.0, reach64 = 0.0;
            for (int i = 0; i < n_joints; ++i)
            {
                const double pa = std::sqrt(arm.a[i] * arm.a[i] + arm.d[i] * arm.d[i]);
                reach64 += pa;
                dp64 += dR64 * pa + pa * (et + u64) * 2.0 + 4.0 * u64 * (reach64 + pa);
                dR64 += 2.0 * et + 16.0 * u64;
            }
            wa.hz_dh = 2.0 * (dp64 + 3.0 * u64 * reach64) * std::sqrt(3.0);
        }
        // The grid below lists an obstacle in every cell within rs (+ r) + margin of it, so a listed
        // obstacle lies within D = rs (+ rmax) + margin + one cell diagonal of the robot sphere centre:
        // |d^2 - d_ref^2| <= 2|d| dc + dc^2 (+ rounding of d^2, rr^2). Boxes: the distance of a point
        // from a box is 1-Lipschitz per axis; each axis adds the roundings of |c - centre| - half
        // extent and of the FP32 box (<= 40u for coordinates below 4, 10u of them above).
        // The margin covers the error of a centre's cell in FP32: dc, and 5u of the coordinates (the box's end
        // rounded, the subtraction, the product with 64 / width). The same coordinates bound the roundings of a
        // box.
        double size = reach;
        for (int64_t i = 0; i < n_world; ++i)
            for (int r = 0; r < 3; ++r)
            {
                const double x = std::fabs(world[stride * i + r]) + std::fabs(world[stride * i + (boxes ? 3 + r : 3)]);
                if (std::isfinite(x))
                    size = std::max(size, x + sphere_radius);
            }
        const double margin = std::max(1e-3, 2.0 * (dc + 5.0 * u * 3.0 * size));
        const int G = 64;
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        // world obstacle i: centre o(i, r), half extent h(i, r) (boxes) or radius (spheres), and the
        // reach added around it (rs + margin for boxes, rs + r + margin for spheres)
        auto o_of = [&](int64_t i, int r) { return world[stride * i + r]; };
        auto half = [&](int64_t i, int r) { return boxes ? world[stride * i + 3 + r] : 0.0; };
        auto grow = [&](int64_t i) { return (boxes ? 0.0 : world[4 * i + 3]) + sphere_radius + margin; };
        for (int64_t i = 0; i < n_world; ++i)
            for (int r = 0; r < 3; ++r)
            {
                const double ext = grow(i) + half(i, r);
                lo[r] = std::min(lo[r], o_of(i, r) - ext);
                hi[r] = std::max(hi[r], o_of(i, r) + ext);
            }
        if (n_world == 0)
            for (int r = 0; r < 3; ++r)
            {
                lo[r] = -1;
                hi[r] = 1;
            }
        double diag2 = 0.0;
        for (int r = 0; r < 3; ++r)
        {
            lo[r] -= margin;
            hi[r] += margin;
            diag2 += ((hi[r] - lo[r]) / G) * ((hi[r] - lo[r]) / G);
        }
        const double D = 1.01 * (sphere_radius + rmax + margin + std::sqrt(diag2));
        const double dcx = boxes ? dc + 10.0 * u * std::max(4.0, size) * std::sqrt(3.0) : dc;
        const double E = 2.0 * D * dcx + dcx * dcx + 8.0 * u * D * D + 4.0 * u * (D * D);
        wa.dh_e = (float)(2.0 * E);
        // uniform 64^3 grid: a sphere is listed in every cell whose box lies within rs + ro + margin of its
        // centre (exact sphere-box distance), so the cell holding a robot sphere centre lists every world
        // sphere that can touch it; cells store the index (FP64 path) and the FP32 sphere itself.
        double inv[3], cell[3];
        for (int r = 0; r < 3; ++r)
        {
            inv[r] = G / (hi[r] - lo[r]);
            cell[r] = (hi[r] - lo[r]) / G;
            wa.glo64[r] = lo[r];
            wa.ginv64[r] = inv[r];
            wa.glo[r] = (float)lo[r];
            wa.ginv[r] = (float)inv[r];
        }
        const size_t ncell = (size_t)G * G * G;
        std::vector<int> start(ncell + 1, 0);
        auto visit = [&](int64_t i, auto &&emit) {
            const double ext = grow(i);
            int c0[3], c1[3];
            for (int r = 0; r < 3; ++r)
            {
                c0[r] = std::max(0, (int)std::floor((o_of(i, r) - half(i, r) - ext - lo[r]) * inv[r]) - 1);
                c1[r] = std::min(G - 1, (int)std::floor((o_of(i, r) + half(i, r) + ext - lo[r]) * inv[r]) + 1);
            }
            for (int x = c0[0]; x <= c1[0]; ++x)
                for (int y = c0[1]; y <= c1[1]; ++y)
                    for (int z = c0[2]; z <= c1[2]; ++z)
                    {
                        const int ix[3] = {x, y, z};
                        double d2 = 0.0;
                        for (int r = 0; r < 3; ++r)
                        {
                            const double b0 = lo[r] + ix[r] * cell[r], b1 = b0 + cell[r];
                            const double o0 = o_of(i, r) - half(i, r), o1 = o_of(i, r) + half(i, r);
                            const double g = o1 < b0 ? b0 - o1 : (o0 > b1 ? o0 - b1 : 0.0);
                            d2 += g * g;
                        }
                        if (d2 <= ext * ext * (1.0 + 1e-9))
                            emit(((size_t)x * G + y) * G + z);
                    }
        };
        for (int64_t i = 0; i < n_world; ++i)
            visit(i, [&](size_t k) { start[k + 1]++; });
        for (size_t k = 0; k < ncell; ++k)
            start[k + 1] += start[k];
        std::vector<int> fill(start.begin(), start.end() - 1), items(std::max(1, start[ncell]));
        const int per_item = boxes ? 8 : 4;
        std::vector<float> items4(per_item * items.size(), 0.f);
        for (int64_t i = 0; i < n_world; ++i)
            visit(i, [&](size_t k) {
                const int pos = fill[k]++;
                items[pos] = (int)i;
                for (int r = 0; r < stride; ++r)
                    items4[per_item * (size_t)pos + r] = (float)world[stride * i + r];
            });
        if (cudaMalloc(&c->cell_start, start.size() * sizeof(int)) != cudaSuccess ||
            cudaMalloc(&c->cell_items, items.size() * sizeof(int)) != cudaSuccess ||
            cudaMalloc(&c->cell_items4, items4.size() * sizeof(float)) != cudaSuccess)
            return cleanup(fail(GBO_ERR_OUT_OF_MEMORY, "grid allocation failed"));
        cudaMemcpy(c->cell_start, start.data(), start.size() * sizeof(int), cudaMemcpyHostToDevice);
        cudaMemcpy(c->cell_items, items.data(), items.size() * sizeof(int), cudaMemcpyHostToDevice);
        cudaMemcpy(c->cell_items4, items4.data(), items4.size() * sizeof(float), cudaMemcpyHostToDevice);
        wa.cell_items4 = (const float4 *)c->cell_items4;
        wa.cell_start = c->cell_start;
        wa.cell_items = c->cell_items;
        wa.grid_n = G;
        // Clearance grid over the same box. Its distances hold for finite obstacles whose reach |rs + r| is
        // not larger than rs + r (the box and its margins follow r); otherwise nothing is proven free.
        {
            const int CG = 128;  // a multiple of 8
            bool ok = true;
            double scale = reach;
            for (int64_t i = 0; i < stride * n_world; ++i)
                ok &= std::isfinite(world[i]);
            for (int64_t i = 0; i < n_world && !boxes; ++i)
                ok &= world[4 * i + 3] >= -sphere_radius;
            for (int64_t i = 0; i < n_world && boxes; ++i)
                for (int r = 3; r < 6; ++r)
                    ok &= world[6 * i + r] >= 0.0;
            for (int r = 0; r < 3; ++r)
                scale = std::max(scale, std::max(std::fabs(lo[r]), std::fabs(hi[r])) + (hi[r] - lo[r]));
            ok &= scale < 1e15;  // its square in FP32
            // the halves hold up to 65,504: distances are stored in units of a power of two (1 below 1e3)
            wa.clr_unit = ok && scale >= 1e3 ? (float)std::exp2(std::ceil(std::log2(scale * 1e-3))) : 1.f;
            wa.clr_n = CG;
            for (int r = 0; r < 3; ++r)
            {
                wa.clr_lo[r] = (float)lo[r];
                wa.clr_cell[r] = (float)((hi[r] - lo[r]) / CG);
                wa.clr_inv[r] = (float)(CG / (hi[r] - lo[r]));
            }
            wa.clr_margin = ok ? (float)(2.0 * dc + 4e-6 * scale + 1e-6) : 1e6f;
            wa.clr_out = ok ? (float)sphere_radius - wa.clr_margin : -1e6f;
            if (cudaMalloc(&c->clr, sizeof(__half) * CG * CG * CG) != cudaSuccess ||
                cudaMalloc(&c->tail, sizeof(ArmTail) * kArmTailRoom * CounterRing::kSlots) != cudaSuccess)
                return cleanup(fail(GBO_ERR_OUT_OF_MEMORY, "clearance grid allocation failed"));
            wa.clr = c->clr;
            launch_arm_clearance(lcfg(nullptr), wa, c->clr);
            cudaStreamSynchronize(nullptr);
        }
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return cleanup(fail(GBO_ERR_CUDA, cudaGetErrorString(e)));
    if (cudaStreamCreateWithFlags(&c->host_stream, cudaStreamNonBlocking) != cudaSuccess)
        return cleanup(fail(GBO_ERR_CUDA, "stream creation failed"));
    *out = c;
    return GBO_OK;
}

gbo_status gbo_checker_destroy(gbo_checker *c)
{
    if (c)
        cudaDeviceSynchronize();
    delete c;
    return GBO_OK;
}

gbo_status gbo_checker_set_precision(gbo_checker *c, int precision)
{
    if (!c || (precision != GBO_PRECISION_FP64 && precision != GBO_PRECISION_FP32_GUARDED))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad precision");
    c->precision = precision;
    return GBO_OK;
}

gbo_status gbo_checker_stats(const gbo_checker *c, uint64_t *evaluated, uint64_t *rechecked)
{
    if (!c)
        return fail(GBO_ERR_INVALID_ARGUMENT, "checker is NULL");
    RunCounters h{};
    CUDA_TRY(cudaMemcpy(&h, c->ctr.dev + c->ctr.last, sizeof(h), cudaMemcpyDeviceToHost));
    if (evaluated)
        *evaluated = h.evaluated;
    if (rechecked)
        *rechecked = h.rechecked;
    if (h.timeout)
        return fail(GBO_ERR_TIMEOUT, "a device-side wait ran out in the last call");
    if (h.error)
        return fail(GBO_ERR_CUDA, "a kernel refused to stage its world into shared memory in the last call");
    return GBO_OK;
}

gbo_status gbo_checker_counters(const gbo_checker *c, uint64_t *evaluated, uint64_t *rechecked, uint64_t *hazards)
{
    if (!c)
        return fail(GBO_ERR_INVALID_ARGUMENT, "checker is NULL");
    RunCounters h{};
    CUDA_TRY(cudaMemcpy(&h, c->ctr.dev + c->ctr.last, sizeof(h), cudaMemcpyDeviceToHost));
    if (evaluated)
        *evaluated = h.evaluated;
    if (rechecked)
        *rechecked = h.rechecked;
    if (hazards)
        *hazards = h.hazards;
    return GBO_OK;
}

gbo_status gbo_is_valid(gbo_checker *c, const double *states, int64_t n, int64_t ld, int layout, uint8_t *out,
                        gbo_stream stream)
{
    Trace trace("gbo_is_valid");
    if (!c || n < 0 || (n > 0 && (!states || !out)) || !valid_layout(layout, n, ld, c->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad isValid arguments");
    if (n == 0)
        return GBO_OK;
    LaunchCfg lc = lcfg(stream);
    RunCounters *ctr = c->ctr.take(lc.stream);
    launch_validity(lc, c->precision, c->sp, c->wa, make_view(states, ld, layout), n, out, ctr);
    CHECK_LAUNCH();
    return GBO_OK;
}

static gbo_status motion_impl(gbo_checker *c, const double *s1, const double *s2, int64_t n, int64_t ld, int layout,
                              int schedule, uint8_t *ok, int32_t *first_j, int32_t *nd, const LaunchCfg &lc)
{
    RunCounters *ctr = c->ctr.take(lc.stream);
    launch_motion(lc, c->precision, schedule, c->sp, c->wa, make_view(s1, ld, layout), make_view(s2, ld, layout), n,
                  ok, first_j, nd, ctr, c->tail ? c->tail + (ctr - c->ctr.dev) * kArmTailRoom : nullptr);
    CHECK_LAUNCH();
    return GBO_OK;
}

// checkMotion's schedule and launch; host_rows: s1 and s2 are page-locked host memory read in place.
static gbo_status motion_call(gbo_checker *c, const double *s1, const double *s2, int64_t n, int64_t ld, int layout,
                              int schedule, uint8_t *ok, int32_t *first_j, int32_t *nd, gbo_stream stream,
                              bool host_rows)
{
    LaunchCfg lc = lcfg(stream);
    lc.host_rows = host_rows;
    if (schedule == GBO_SCHEDULE_AUTO && c->wa.kind == GBO_CHECK_DH_SPHERES)
        schedule = GBO_SCHEDULE_WARP;  // one form for every schedule
    if (schedule == GBO_SCHEDULE_AUTO && c->precision == GBO_PRECISION_FP32_GUARDED &&
        chain_motion_lanes(lc, c->sp, c->wa, n))
        schedule = GBO_SCHEDULE_WARP;  // a large chain batch: its own form, nothing to tune
    if (schedule == GBO_SCHEDULE_AUTO)
    {
        std::lock_guard<std::mutex> lk(c->tune_mu);
        if (c->tuned_schedule < 0)
        {
            // autotune: time both persistent schedules on (a prefix of) this batch
            const int64_t m = std::min<int64_t>(n, 65536);
            cudaEvent_t e0, e1;
            cudaEventCreate(&e0);
            cudaEventCreate(&e1);
            float best = 1e30f;
            int pick = GBO_SCHEDULE_TILE;
            for (int sch : {GBO_SCHEDULE_TILE, GBO_SCHEDULE_WARP})
            {
                for (int rep = 0; rep < 2; ++rep)
                {
                    cudaEventRecord(e0, lc.stream);
                    if (auto st = motion_impl(c, s1, s2, m, ld, layout, sch, ok, first_j, nd, lc))
                        return st;
                    cudaEventRecord(e1, lc.stream);
                    cudaEventSynchronize(e1);
                    float ms = 0.f;
                    cudaEventElapsedTime(&ms, e0, e1);
                    if (rep == 1 && ms < best)
                    {
                        best = ms;
                        pick = sch;
                    }
                }
            }
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            c->tuned_schedule = pick;
        }
        schedule = c->tuned_schedule;
    }
    return motion_impl(c, s1, s2, n, ld, layout, schedule, ok, first_j, nd, lc);
}

gbo_status gbo_check_motion(gbo_checker *c, const double *s1, const double *s2, int64_t n, int64_t ld, int layout,
                            int schedule, uint8_t *ok, int32_t *first_j, int32_t *nd, gbo_stream stream)
{
    Trace trace("gbo_check_motion");
    if (!c || n < 0 || (n > 0 && (!s1 || !s2 || !ok)) || !valid_layout(layout, n, ld, c->sp.dim) ||
        schedule < GBO_SCHEDULE_PLAIN || schedule > GBO_SCHEDULE_AUTO)
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad checkMotion arguments");
    if (n == 0)
        return GBO_OK;
    return motion_call(c, s1, s2, n, ld, layout, schedule, ok, first_j, nd, stream, false);
}

gbo_status gbo_last_valid(const gbo_space *s, const double *s1, const double *s2, const int32_t *first_j,
                          const int32_t *nd, int64_t n, int64_t ld, int layout, double *last_t, double *last_state,
                          gbo_stream stream)
{
    if (!s || n < 0 || (n > 0 && (!s1 || !s2 || !first_j || !nd)) || !valid_layout(layout, n, ld, s->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad lastValid arguments");
    StatesView ov = make_view(last_state, ld, layout);
    launch_last_valid(lcfg(stream), s->sp, make_view(s1, ld, layout), make_view(s2, ld, layout), first_j, nd, n,
                      last_t, MutStatesView{last_state, ov.si, ov.sd});
    CHECK_LAUNCH();
    return GBO_OK;
}

__global__ void finish_states_chain(const unsigned long long *first, int64_t count, uint8_t *ok, int64_t *fi)
{
    const unsigned long long f = *first;
    const bool good = f >= (unsigned long long)count;
    *ok = good ? 1 : 0;
    if (fi)
        *fi = good ? -1 : (int64_t)f;
}

gbo_status gbo_check_motion_states(gbo_checker *c, const double *states, int64_t count, int64_t ld, int layout,
                                   uint8_t *ok, int64_t *first_invalid, gbo_stream stream)
{
    if (!c || count < 0 || (count > 0 && !states) || !ok || !valid_layout(layout, count, ld, c->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad checkMotion(states) arguments");
    LaunchCfg lc = lcfg(stream);
    RunCounters *ctr = c->ctr.take(lc.stream);
    unsigned long long *first = &ctr->queue;  // slot's queue word doubles as the running minimum
    CUDA_TRY(cudaMemsetAsync(first, 0xff, sizeof(unsigned long long), lc.stream));
    if (count > 0)
        launch_states_chain(lc, c->sp, c->wa, make_view(states, ld, layout), count, first, ctr);
    finish_states_chain<<<1, 1, 0, lc.stream>>>(first, count, ok, first_invalid);
    note_launch();
    CHECK_LAUNCH();
    return GBO_OK;
}

// Device address of a page-locked host array (cudaMallocHost / cudaHostRegister), or null for
// pageable or device memory. Kernels read and write such arrays in place over the coherent host
// link, so the transfer overlaps with the work inside the launch instead of preceding it.
static void *mapped_host(const void *p)
{
    cudaPointerAttributes a{};
    if (!p || cudaPointerGetAttributes(&a, p) != cudaSuccess)
    {
        cudaGetLastError();
        return nullptr;
    }
    return a.type == cudaMemoryTypeHost ? a.devicePointer : nullptr;
}

gbo_status gbo_is_valid_host(gbo_checker *c, const double *states, int64_t n, uint8_t *out)
{
    Trace trace("gbo_is_valid_host");
    if (!c || n < 0 || (n > 0 && (!states || !out)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad isValid arguments");
    if (n == 0)
        return GBO_OK;
    std::lock_guard<std::mutex> lk(c->mu);
    const size_t bin = (size_t)n * c->sp.dim * sizeof(double);
    const double *din = (const double *)mapped_host(states);
    uint8_t *dout = (uint8_t *)mapped_host(out);
    // a lane per state would read the rows across the host link a few bytes at a time: copied first (400,000
    // chain states: 391 us; a warp per state in place 518)
    if (!din || (c->precision == GBO_PRECISION_FP32_GUARDED && chain_validity_lanes(c->sp, c->wa, n)))
    {
        if (auto st = c->dev_in.reserve(bin, c->host_stream))
            return st;
        const void *src = states;
        if (!din)
        {
            if (auto st = c->pin_in.reserve(bin))
                return st;
            std::memcpy(c->pin_in.p, states, bin);
            src = c->pin_in.p;
        }
        CUDA_TRY(cudaMemcpyAsync(c->dev_in.p, src, bin, cudaMemcpyHostToDevice, c->host_stream));
        din = (const double *)c->dev_in.p;
    }
    if (!dout)
    {
        if (auto st = c->dev_out.reserve((size_t)n, c->host_stream))
            return st;
    }
    if (auto st = gbo_is_valid(c, din, n, c->sp.dim, GBO_LAYOUT_AOS, dout ? dout : (uint8_t *)c->dev_out.p,
                               c->host_stream))
        return st;
    if (!dout)
        CUDA_TRY(cudaMemcpyAsync(out, c->dev_out.p, (size_t)n, cudaMemcpyDeviceToHost, c->host_stream));
    CUDA_TRY(cudaStreamSynchronize(c->host_stream));
    return GBO_OK;
}

gbo_status gbo_check_motion_host(gbo_checker *c, const double *s1, const double *s2, int64_t n, uint8_t *ok,
                                 double *last_t, double *last_state)
{
    Trace trace("gbo_check_motion_host");
    if (!c || n < 0 || (n > 0 && (!s1 || !s2 || !ok)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad checkMotion arguments");
    if (n == 0)
        return GBO_OK;
    std::lock_guard<std::mutex> lk(c->mu);
    const int dim = c->sp.dim;
    const size_t bst = (size_t)n * dim * sizeof(double);
    // page-locked arrays are used in place (mapped_host); the others go through device buffers
    const double *m1 = (const double *)mapped_host(s1), *m2 = (const double *)mapped_host(s2);
    // the arm's lanes read their edges' rows, the chain's warps in place (chain_motion_lanes)
    const bool arm = c->wa.kind == GBO_CHECK_DH_SPHERES;
    const bool in_place = m1 && m2 && !arm;
    uint8_t *mok = arm ? nullptr : (uint8_t *)mapped_host(ok);
    double *mlt = (double *)mapped_host(last_t), *mls = (double *)mapped_host(last_state);
    // device layout: [s1 | s2 (copy path)] | first_j | nd | ok | last_t | last_state
    const size_t off_fj = in_place ? 0 : 2 * bst, off_nd = off_fj + 4 * (size_t)n, off_ok = off_nd + 4 * (size_t)n;
    const size_t off_lt = pad16(off_ok + (size_t)n), off_ls = off_lt + 8 * (size_t)n, total = off_ls + bst;
    if (auto st = c->dev_in.reserve(total, c->host_stream))
        return st;
    char *d = (char *)c->dev_in.p;
    if (!in_place)
    {
        // straight from the caller's arrays to the device (no staging copy on the host)
        CUDA_TRY(cudaMemcpyAsync(d, s1, bst, cudaMemcpyHostToDevice, c->host_stream));
        CUDA_TRY(cudaMemcpyAsync(d + bst, s2, bst, cudaMemcpyHostToDevice, c->host_stream));
        m1 = (const double *)d;
        m2 = (const double *)(d + bst);
    }
    uint8_t *okd = mok ? mok : (uint8_t *)(d + off_ok);
    int32_t *fj = (int32_t *)(d + off_fj), *ndv = (int32_t *)(d + off_nd);
    const int sched = c->precision == GBO_PRECISION_FP64 ? GBO_SCHEDULE_PLAIN : GBO_SCHEDULE_AUTO;
    if (auto st = motion_call(c, m1, m2, n, dim, GBO_LAYOUT_AOS, sched, okd, fj, ndv, c->host_stream, in_place))
        return st;
    double *ltd = mlt ? mlt : (double *)(d + off_lt), *lsd = mls ? mls : (double *)(d + off_ls);
    if (last_t || last_state)
    {
        launch_last_valid(lcfg(c->host_stream), c->sp, make_view(m1, dim, GBO_LAYOUT_AOS),
                          make_view(m2, dim, GBO_LAYOUT_AOS), fj, ndv, n, ltd,
                          MutStatesView{last_state ? lsd : nullptr, dim, 1});
        CHECK_LAUNCH();
    }
    if (!mok)
        CUDA_TRY(cudaMemcpyAsync(ok, okd, (size_t)n, cudaMemcpyDeviceToHost, c->host_stream));
    if (last_t && !mlt)
        CUDA_TRY(cudaMemcpyAsync(last_t, ltd, 8 * (size_t)n, cudaMemcpyDeviceToHost, c->host_stream));
    if (last_state && !mls)
        CUDA_TRY(cudaMemcpyAsync(last_state, lsd, bst, cudaMemcpyDeviceToHost, c->host_stream));
    CUDA_TRY(cudaStreamSynchronize(c->host_stream));
    return GBO_OK;
}

// Small batches in host memory on the caller's stream (ordered after its earlier work, unlike the *_host
// calls' own stream): one copy in, the kernels, one copy out through the object's page-locked buffers.
gbo_status gbo_is_valid_rows(gbo_checker *c, const double *states, int64_t n, uint8_t *out, gbo_stream stream)
{
    if (!c || n < 0 || (n > 0 && (!states || !out)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad isValid arguments");
    if (n == 0)
        return GBO_OK;
    const size_t bin = (size_t)n * c->sp.dim * sizeof(double);
    RowCall call(c->rows, (cudaStream_t)stream);
    if (auto e = call.reserve(bin + (size_t)n))
        return e;
    char *h = call.host(), *d = call.device();
    std::memcpy(h, states, bin);
    if (auto e = call.copy_in(bin))
        return e;
    if (auto e = gbo_is_valid(c, (const double *)d, n, c->sp.dim, GBO_LAYOUT_AOS, (uint8_t *)d + bin, stream))
        return e;
    if (auto e = call.copy_out(bin, (size_t)n))
        return e;
    std::memcpy(out, h + bin, (size_t)n);
    return GBO_OK;
}

gbo_status gbo_check_motion_rows(gbo_checker *c, const double *s1, const double *s2, int64_t n, int schedule,
                                 uint8_t *ok, int32_t *first_j, int32_t *nd, gbo_stream stream)
{
    if (!c || n < 0 || (n > 0 && (!s1 || !s2 || !ok || !first_j || !nd)) || schedule < GBO_SCHEDULE_PLAIN ||
        schedule > GBO_SCHEDULE_AUTO)
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad checkMotion arguments");
    if (n == 0)
        return GBO_OK;
    const size_t bst = (size_t)n * c->sp.dim * sizeof(double), out = 9 * (size_t)n;
    RowCall call(c->rows, (cudaStream_t)stream);
    if (auto e = call.reserve(2 * bst + out))
        return e;
    char *h = call.host(), *d = call.device();
    std::memcpy(h, s1, bst);
    std::memcpy(h + bst, s2, bst);
    if (auto e = call.copy_in(2 * bst))
        return e;
    int32_t *fj = (int32_t *)(d + 2 * bst), *ndv = fj + n;
    uint8_t *okd = (uint8_t *)(ndv + n);
    if (auto e = gbo_check_motion(c, (const double *)d, (const double *)(d + bst), n, c->sp.dim, GBO_LAYOUT_AOS,
                                  schedule, okd, fj, ndv, stream))
        return e;
    if (auto e = call.copy_out(2 * bst, out))
        return e;
    std::memcpy(first_j, h + 2 * bst, 4 * (size_t)n);
    std::memcpy(nd, h + 2 * bst + 4 * (size_t)n, 4 * (size_t)n);
    std::memcpy(ok, h + 2 * bst + 8 * (size_t)n, (size_t)n);
    return GBO_OK;
}

// ---------------------------------------------------------------- samplers
gbo_status gbo_sampler_create(const gbo_space *space, uint32_t local_seed, gbo_sampler **out)
{
    if (!space || !out)
        return fail(GBO_ERR_INVALID_ARGUMENT, "space/out is NULL");
    if (auto st = ensure_device())
        return st;
    auto *s = new gbo_sampler();
    s->sp = space->sp;
    // mt19937 seeding (std::mersenne_twister_engine::seed): x0 = seed, x_i = f * (x_{i-1} ^ (x_{i-1} >> 30)) + i
    SamplerState h{};
    h.mt[0] = local_seed;
    for (unsigned i = 1; i < 624; ++i)
        h.mt[i] = 1812433253u * (h.mt[i - 1] ^ (h.mt[i - 1] >> 30)) + i;
    h.pos = 624;
    if (cudaMalloc(&s->st, sizeof(SamplerState)) != cudaSuccess)
    {
        delete s;
        return fail(GBO_ERR_OUT_OF_MEMORY, "sampler allocation failed");
    }
    cudaMemcpy(s->st, &h, sizeof(h), cudaMemcpyHostToDevice);
    if (cudaStreamCreateWithFlags(&s->host_stream, cudaStreamNonBlocking) != cudaSuccess)
    {
        delete s;
        return fail(GBO_ERR_CUDA, "stream creation failed");
    }
    *out = s;
    return GBO_OK;
}

gbo_status gbo_sampler_destroy(gbo_sampler *s)
{
    delete s;
    return GBO_OK;
}

// Word-stream scratch of a sampling call of n states (stream-ordered growth): 2 words per value, at
// most 16M words (larger calls run in chunks).
static gbo_status sampler_words(gbo_sampler *s, int64_t n, gbo_stream stream, int64_t &cap)
{
    cap = std::max<int64_t>(2, std::min<int64_t>(2 * n * s->sp.dim, (int64_t)1 << 24));
    return s->words.reserve((size_t)cap * sizeof(unsigned), (cudaStream_t)stream);
}

// sampleUniform / sampleUniformNear over n states. Calls of at least 2^18 stream words run on segments
// of the stream generated side by side from jump-ahead windows (segments of L = 2^m words, m >= 15, the
// smallest m that keeps them at most 160); smaller calls run the recurrence on one CTA.
static gbo_status sample_uniform_call(gbo_sampler *s, const double *near, StatesView nearv, double distance,
                                      int64_t n, MutStatesView out, gbo_stream stream)
{
    const int64_t values = n * s->sp.dim, W = 2 * values;
    if (W >= ((int64_t)1 << 18) && values < ((int64_t)1 << 31) && mt_field_ready())
    {
        int m = 15;
        while (m < 24 && W > ((int64_t)160 << m))
            ++m;
        const int64_t L = (int64_t)1 << m;
        const int nseg = (int)((W + L - 1) / L);
        const uint32_t *polys = nullptr;
        if (nseg > 1)
            if (auto st = mt_jump_table((uint64_t)L, nseg - 1, &polys))
                return fail(st, "jump-ahead polynomials could not be prepared");
        if (auto st = s->words.reserve((size_t)sample_jump_words(nseg, W) * sizeof(unsigned), (cudaStream_t)stream))
            return st;
        launch_sample_uniform_jump(lcfg(stream), s->st, s->sp, near, nearv, distance, n, out, (unsigned *)s->words.p,
                                   polys, L, nseg);
        CHECK_LAUNCH();
        return GBO_OK;
    }
    int64_t cap = 0;
    if (auto st = sampler_words(s, n, stream, cap))
        return st;
    launch_sample_uniform(lcfg(stream), s->st, s->sp, near, nearv, distance, n, out, (unsigned *)s->words.p, cap);
    CHECK_LAUNCH();
    return GBO_OK;
}

gbo_status gbo_sample_uniform(gbo_sampler *s, int64_t n, double *out, int64_t ld, int layout, gbo_stream stream)
{
    Trace trace("gbo_sample_uniform");
    if (!s || n < 0 || (n > 0 && !out) || !valid_layout(layout, n, ld, s->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sampleUniform arguments");
    StatesView ov = make_view(out, ld, layout);
    return sample_uniform_call(s, nullptr, StatesView{}, 0.0, n, MutStatesView{out, ov.si, ov.sd}, stream);
}

gbo_status gbo_sample_uniform_near(gbo_sampler *s, const double *near, double distance, int64_t n, int64_t ld,
                                   int layout, double *out, gbo_stream stream)
{
    if (!s || n < 0 || (n > 0 && (!out || !near)) || !valid_layout(layout, n, ld, s->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sampleUniformNear arguments");
    StatesView ov = make_view(out, ld, layout);
    return sample_uniform_call(s, near, make_view(near, ld, layout), distance, n, MutStatesView{out, ov.si, ov.sd},
                               stream);
}

// StateSampler::sampleGaussian (StateSampler.h:96-100) for n states, state i drawn around mean row i
// (mean and out share ld and layout). Returns after the call's stream work: the number of candidate
// draws is data dependent and the host reads each chunk's progress.
gbo_status gbo_sample_gaussian(gbo_sampler *s, const double *mean, double stddev, int64_t n, int64_t ld, int layout,
                               double *out, gbo_stream stream)
{
    Trace trace("gbo_sample_gaussian");
    if (!s || n < 0 || (n > 0 && (!out || !mean)) || !valid_layout(layout, n, ld, s->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sampleGaussian arguments");
    const int64_t M = n * s->sp.dim;
    if (M == 0)
        return GBO_OK;
    // raw words for the expected candidates plus a margin and one whole block (capped; larger calls
    // run in several chunks)
    const double mu = (double)((M + 1) / 2) / 0.7853981633974483;
    const int64_t cap = std::min<int64_t>(((int64_t)1 << 25) + 628,
                                          4 * (int64_t)std::ceil(mu + 8.0 * std::sqrt(mu) + 64.0) + 628);
    cudaStream_t st = (cudaStream_t)stream;
    // large chunks draw their candidates' words on jump-ahead segments (segment length chosen as for
    // sampleUniform from the first chunk's words; later chunks are shorter and use fewer segments)
    const int64_t W0 = 4 * ((cap - 624) / 4);  // the most words a chunk draws (4 per candidate)
    const uint32_t *polys = nullptr;
    int64_t L = 0, jump_words = 0;
    if (W0 >= ((int64_t)1 << 18) && mt_field_ready())
    {
        int m = 15;
        while (m < 24 && W0 > ((int64_t)160 << m))
            ++m;
        L = (int64_t)1 << m;
        const int nseg = (int)((W0 + L - 1) / L);
        if (nseg > 1)
            if (auto e = mt_jump_table((uint64_t)L, nseg - 1, &polys))
                return fail(e, "jump-ahead polynomials could not be prepared");
        if (nseg == 1)
            polys = nullptr;
        jump_words = sample_jump_words(nseg, 0);
    }
    const int64_t cap_al = (cap + 3) & ~(int64_t)3;
    if (auto e = s->words.reserve((size_t)(cap_al + jump_words) * sizeof(unsigned), st))
        return e;
    const size_t cnt_bytes = pad16(sizeof(GaussChunk) + sizeof(long long) * (size_t)(cap / 4096 + 2));
    const size_t slots = (size_t)gauss_pair_slots(cap);
    if (auto e = s->gwork.reserve(cnt_bytes + slots * (sizeof(double2) + sizeof(unsigned short) + 2 * sizeof(unsigned)),
                                  st))
        return e;
    double2 *pair = (double2 *)((char *)s->gwork.p + cnt_bytes);
    const StatesView ov = make_view(out, ld, layout);
    const int64_t chunks = launch_sample_gaussian(
        lcfg(st), s->st, s->has_saved, s->sp, make_view(mean, ld, layout), stddev, n, MutStatesView{out, ov.si, ov.sd},
        (unsigned *)s->words.p, cap, (GaussChunk *)s->gwork.p, (long long *)((char *)s->gwork.p + sizeof(GaussChunk)),
        pair, (unsigned short *)(pair + slots), (unsigned *)((unsigned short *)(pair + slots) + slots),
        polys ? (unsigned *)s->words.p + cap_al : nullptr, polys, L);
    if (chunks < 0)
        return fail(GBO_ERR_CUDA, std::string("sampleGaussian: ") + cudaGetErrorString(cudaGetLastError()));
    CHECK_LAUNCH();
    s->has_saved = ((M - (s->has_saved ? 1 : 0)) & 1) != 0;
    return GBO_OK;
}

// UniformValidStateSampler::sample, n calls. A call draws until a valid state or `attempts` draws;
// the stream must end where OMPL's would, so no draw is made that no call consumes. Each round draws
// one state per unresolved call (every such call consumes at least one more), checks them, and walks
// the flags on the host; after 8 rounds the rest is drawn speculatively up to its upper bound
// (attempts per call) from a saved copy of the generator, which is then restored and advanced by
// exactly the draws consumed.
gbo_status gbo_sample_valid(gbo_sampler *s, gbo_checker *c, int64_t n, unsigned attempts, double *out, int64_t ld,
                            int layout, uint8_t *ok, gbo_stream stream)
{
    Trace trace("gbo_sample_valid");
    if (!s || !c || n < 0 || (n > 0 && (!out || !ok)) || !valid_layout(layout, n, ld, s->sp.dim) ||
        c->sp.dim != s->sp.dim)
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sampleValid arguments");
    if (n == 0)
        return GBO_OK;
    const int64_t A = attempts > 0 ? attempts : 1;  // do { ... } while: one draw at least
    const int dim = s->sp.dim;
    cudaStream_t st = (cudaStream_t)stream;
    const StatesView ov = make_view(out, ld, layout);
    const LaunchCfg lc = lcfg(st);
    std::vector<uint8_t> flags, okh;
    std::vector<int64_t> src;
    int64_t done = 0, open = 0;  // calls resolved; draws of the unresolved call so far
    constexpr int64_t kSpeculativeCap = 1ll << 26;
    for (int round = 0; done < n; ++round)
    {
        const int64_t r = n - done;
        const bool spec = round >= 8 && r * A - open <= kSpeculativeCap;
        const int64_t gen = spec ? r * A - open : r;
        double *buf = nullptr;
        uint8_t *fl = nullptr;
        int64_t *idx = nullptr;
        SamplerState *ckpt = nullptr;
        CUDA_TRY(cudaMallocAsync((void **)&buf, (size_t)gen * dim * sizeof(double), st));
        CUDA_TRY(cudaMallocAsync((void **)&fl, (size_t)gen, st));
        CUDA_TRY(cudaMallocAsync((void **)&idx, (size_t)r * sizeof(int64_t), st));
        if (spec)
        {
            CUDA_TRY(cudaMallocAsync((void **)&ckpt, sizeof(SamplerState), st));
            CUDA_TRY(cudaMemcpyAsync(ckpt, s->st, sizeof(SamplerState), cudaMemcpyDeviceToDevice, st));
        }
        if (auto e = gbo_sample_uniform(s, gen, buf, dim, GBO_LAYOUT_AOS, stream))
            return e;
        if (auto e = gbo_is_valid(c, buf, gen, dim, GBO_LAYOUT_AOS, fl, stream))
            return e;
        flags.resize((size_t)gen);
        CUDA_TRY(cudaMemcpyAsync(flags.data(), fl, (size_t)gen, cudaMemcpyDeviceToHost, st));
        CUDA_TRY(cudaStreamSynchronize(st));
        src.clear();
        okh.clear();
        int64_t q = 0;
        while (done + (int64_t)src.size() < n && q < gen)
        {
            ++open;
            if (flags[(size_t)q] || open == A)
            {
                src.push_back(q);
                okh.push_back(flags[(size_t)q] ? 1 : 0);
                open = 0;
            }
            ++q;
        }
        if (spec)
        {
            // back to the saved generator, advanced by exactly the q draws consumed (same values)
            CUDA_TRY(cudaMemcpyAsync(s->st, ckpt, sizeof(SamplerState), cudaMemcpyDeviceToDevice, st));
            if (auto e = gbo_sample_uniform(s, q, buf, dim, GBO_LAYOUT_AOS, stream))
                return e;
        }
        const int64_t m = (int64_t)src.size();
        if (m)
        {
            CUDA_TRY(cudaMemcpyAsync(idx, src.data(), (size_t)m * sizeof(int64_t), cudaMemcpyHostToDevice, st));
            CUDA_TRY(cudaMemcpyAsync(ok + done, okh.data(), (size_t)m, cudaMemcpyHostToDevice, st));
            launch_gather_rows(lc, StatesView{buf, dim, 1}, idx, m, dim,
                               MutStatesView{out + done * ov.si, ov.si, ov.sd});
            CHECK_LAUNCH();
        }
        cudaFreeAsync(buf, st);
        cudaFreeAsync(fl, st);
        cudaFreeAsync(idx, st);
        if (ckpt)
            cudaFreeAsync(ckpt, st);
        CUDA_TRY(cudaStreamSynchronize(st));  // src / okh are reused by the next round
        done += m;
    }
    return GBO_OK;
}

// ---------------------------------------------------------------- nearest neighbours
gbo_status gbo_nn_create(const gbo_space *space, int64_t capacity, gbo_nn **out)
{
    if (!space || !out || capacity < 1)
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad nn arguments");
    if (auto st = ensure_device())
        return st;
    auto *nn = new gbo_nn();
    nn->sp = space->sp;
    nn->cap = capacity;
    nn->F = space->sp.kind == GBO_SPACE_KINEMATIC_CHAIN ? 2 * space->sp.dim : space->sp.dim;
    nn->eps32 = space->sp.kind == GBO_SPACE_KINEMATIC_CHAIN ? chain_knn_eps(space->sp) : box_knn_eps(space->sp);
    if (cudaMalloc(&nn->pts64, sizeof(double) * space->sp.dim * capacity) != cudaSuccess ||
        cudaMalloc(&nn->feat32, sizeof(float) * nn->F * capacity) != cudaSuccess ||
        cudaMalloc(&nn->feat4, sizeof(float4) * ((nn->F + 3) / 4) * capacity) != cudaSuccess ||
        cudaMalloc(&nn->outside, sizeof(int)) != cudaSuccess ||
        cudaMalloc(&nn->alive, capacity) != cudaSuccess || nn->ctr.init() != GBO_OK)
    {
        delete nn;
        return fail(GBO_ERR_OUT_OF_MEMORY, "nearest-neighbour index allocation failed");
    }
    cudaMemset(nn->alive, 0, capacity);
    cudaMemset(nn->outside, 0, sizeof(int));
    if (cudaStreamCreateWithFlags(&nn->host_stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&nn->searched, cudaEventDisableTiming) != cudaSuccess)
    {
        delete nn;
        return fail(GBO_ERR_CUDA, "stream creation failed");
    }
    *out = nn;
    return GBO_OK;
}

gbo_status gbo_nn_destroy(gbo_nn *nn)
{
    if (nn)
        cudaDeviceSynchronize();
    delete nn;
    return GBO_OK;
}

gbo_status gbo_nn_set_precision(gbo_nn *nn, int precision)
{
    if (!nn || (precision != GBO_PRECISION_FP64 && precision != GBO_PRECISION_FP32_GUARDED))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad precision");
    nn->precision = precision;
    return GBO_OK;
}

gbo_status gbo_nn_add(gbo_nn *nn, const double *states, int64_t n, int64_t ld, int layout, int64_t *first_key,
                      gbo_stream stream)
{
    if (!nn || n < 0 || (n > 0 && !states) || !valid_layout(layout, n, ld, nn->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad add arguments");
    std::lock_guard<std::mutex> lk(nn->search_mu);
    if (nn->size + n > nn->cap)
        return fail(GBO_ERR_OUT_OF_MEMORY, "nearest-neighbour index capacity exceeded");
    if (first_key)
        *first_key = nn->size;
    LaunchCfg lc = lcfg(stream);
    StatesView v = make_view(states, ld, layout);
    launch_store_points(lc, nn->sp, v, n, nn->pts64, nn->cap, nn->size, nn->alive, nn->outside);
    // features of the new elements, written at column offset `size` of the [F][cap] array
    launch_features(lc, nn->sp, v, n, nn->feat32 + nn->size, nn->cap, nn->feat4 + nn->size);
    CHECK_LAUNCH();
    nn->size += n;
    if (nn->alive_count >= 0)  // else recounted on demand
        nn->alive_count += n;
    for (auto &c : nn->cells)
        c.size = 0;
    nn->forgone = 0;
    nn->ccells.valid = false;
    return GBO_OK;
}

gbo_status gbo_nn_remove(gbo_nn *nn, const int64_t *keys, int64_t n, gbo_stream stream)
{
    if (!nn || n < 0 || (n > 0 && !keys))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad remove arguments");
    std::lock_guard<std::mutex> lk(nn->search_mu);
    launch_remove(lcfg(stream), keys, n, nn->size, nn->alive);
    CHECK_LAUNCH();
    nn->alive_count = -1;  // recounted on demand
    for (auto &c : nn->cells)
        c.size = 0;
    nn->forgone = 0;
    nn->ccells.valid = false;
    return GBO_OK;
}

gbo_status gbo_nn_clear(gbo_nn *nn)
{
    if (!nn)
        return fail(GBO_ERR_INVALID_ARGUMENT, "nn is NULL");
    std::lock_guard<std::mutex> lk(nn->search_mu);
    CUDA_TRY(cudaDeviceSynchronize());
    CUDA_TRY(cudaMemset(nn->alive, 0, nn->cap));
    CUDA_TRY(cudaMemset(nn->outside, 0, sizeof(int)));
    nn->size = 0;
    nn->alive_count = 0;
    for (auto &c : nn->cells)
        c.size = 0;
    nn->forgone = 0;
    nn->ccells.valid = false;
    return GBO_OK;
}

gbo_status gbo_nn_size(const gbo_nn *nn, int64_t *size)
{
    if (!nn || !size)
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad size arguments");
    auto *m = const_cast<gbo_nn *>(nn);
    std::lock_guard<std::mutex> lk(m->search_mu);
    if (m->alive_count < 0)
    {
        std::vector<unsigned char> h(m->size);
        CUDA_TRY(cudaDeviceSynchronize());
        if (m->size)
            CUDA_TRY(cudaMemcpy(h.data(), m->alive, m->size, cudaMemcpyDeviceToHost));
        int64_t c = 0;
        for (auto x : h)
            c += x;
        m->alive_count = c;
    }
    *size = m->alive_count;
    return GBO_OK;
}

// One nearestK at a time enqueues its work, and the work of one on another stream waits for it: the cell indexes, which
// a search may have to build, and the scratch belong to the gbo_nn. A call being captured only takes the lock (an event
// from outside may not enter a capture): its replays are the caller's to order.
struct SearchOrder
{
    gbo_nn *nn;
    cudaStream_t s;
    bool captured;
    unsigned long long id = 0;
    std::lock_guard<std::mutex> lk;
    SearchOrder(gbo_nn *n, cudaStream_t stream) : nn(n), s(stream), captured(capturing(stream)), lk(n->search_mu)
    {
        if (captured)
            return;
        cudaStreamGetId(s, &id);
        if (nn->in_flight && id != nn->searched_on)
            cudaStreamWaitEvent(s, nn->searched, 0);
    }
    ~SearchOrder()
    {
        if (captured)
            return;
        cudaEventRecord(nn->searched, s);
        nn->searched_on = id;
        nn->in_flight = true;
    }
};

static NNArgs nn_args(const gbo_nn *nn)
{
    NNArgs a;
    a.pts64 = nn->pts64;
    a.feat32 = nn->feat32;
    a.feat4 = nn->feat4;
    a.alive = nn->alive;
    a.cap = nn->cap;
    a.size = nn->size;
    a.eps32 = nn->eps32;
    return a;
}

// Prefix levels of a batch: limits in (size / 2, size] at each; without limits, and below 65,536 elements, all that
// are left
static int box_cell_levels(int64_t size, bool prefix)
{
    int n = 1;
    while (prefix && size / 2 >= 32768 && n < kCellLevels)
    {
        size /= 2;
        ++n;
    }
    return n;
}

// Whether the indexes that a batch searches are built
static bool cells_built(const gbo_nn *nn, bool prefix)
{
    if (nn->sp.kind == GBO_SPACE_KINEMATIC_CHAIN)
        return nn->ccells.valid;
    int64_t size = nn->size;
    for (int level = 0, n = box_cell_levels(size, prefix); level < n; ++level, size /= 2)
        if (nn->cells[level].size != size)
            return false;
    return true;
}

// The cell search of a batch over a RealVector / wrapped gbo_nn, building the indexes it needs in stream order.
static gbo_status box_cells_call(gbo_nn *nn, const LaunchCfg &lc, const float *qf, int64_t nq, const int64_t *prefix,
                                 int k, const KnnOut &out)
{
    const cudaStream_t s = lc.stream;
    int64_t size = nn->size;
    for (int level = 0, n = box_cell_levels(size, prefix); level < n; ++level)
    {
        NNBoxCells &c = nn->cells[level];
        KnnOut o = out;
        o.nn.size = size;
        const BoxCellShape shape = cell_shape(nn->sp.dim, size);
        const size_t sub = (size_t)shape.C << shape.bits, sums = sub / 4096 + 2;
        // [element or query keys | counts | fill | block sums | query starts | query order]
        const size_t words = (size_t)std::max(size, nq) + 2 * sub + sums + (size_t)shape.C + 1 + (size_t)nq;
        if (auto e = nn->cwork.reserve(words * sizeof(int), s))
            return e;
        int *key = (int *)nn->cwork.p, *count = key + std::max(size, nq), *fill = count + sub, *bs = fill + sub;
        int *qstart = bs + sums, *qorder = qstart + shape.C + 1;
        if (c.size != size)
        {
            c.shape = shape;
            if (auto e = c.reserve(size, s))
                return e;
            launch_cell_build(lc, o.nn, nn->sp, shape, key, count, bs, fill, c.args());
            CHECK_LAUNCH();
            c.size = size;
        }
        launch_knn_cells(lc, c.args(), nn->sp, qf, nq, prefix, size / 2, level == 0, k, key, count, qstart, fill,
                         qorder, bs, o);
        CHECK_LAUNCH();
        if (level + 1 < n)
            size /= 2;
    }
    if (prefix && !launch_knn_group(lc, out.nn, nn->sp, out.qv, nq, k, prefix, size / 2, out.idx, out.dist, out.fb_list,
                                    out.fb_n, out.ctr))
        return fail(GBO_ERR_UNSUPPORTED, "nearestK: no form for the low prefix limits");
    CHECK_LAUNCH();
    return GBO_OK;
}

static gbo_status ensure_chain_cells(gbo_nn *nn, const LaunchCfg &lc)
{
    NNChainCells &c = nn->ccells;
    if (c.valid)
        return GBO_OK;
    const int64_t n = std::max<int64_t>(nn->size, 1);
    const cudaStream_t s = lc.stream;
    for (auto r : {c.key.reserve((size_t)n * sizeof(int), s), c.count.reserve(kQueryKeys * sizeof(int), s),
                   c.start.reserve(kQueryKeys * sizeof(int), s), c.fill.reserve(kQueryKeys * sizeof(int), s),
                   c.skey.reserve((size_t)n * sizeof(int64_t), s), c.sfeat.reserve((size_t)n * 5 * sizeof(float4), s),
                   c.box.reserve((size_t)kQueryKeys * 5 * sizeof(uint4), s),
                   c.cstart.reserve((size_t)(kQueryKeys + 1) * sizeof(int), s),
                   c.cbox.reserve((size_t)(n / 32 + kQueryKeys) * 5 * sizeof(uint4), s)})
        if (r)
            return r;
    launch_ccell_build(lc, nn_args(nn), nn->sp, (int *)c.key.p, (int *)c.count.p, (int *)c.start.p, (int *)c.fill.p,
                       (int64_t *)c.skey.p, (float4 *)c.sfeat.p, (uint4 *)c.box.p, (int *)c.cstart.p,
                       (uint4 *)c.cbox.p);
    CHECK_LAUNCH();
    c.valid = true;
    return GBO_OK;
}

gbo_status gbo_nn_nearest_k(gbo_nn *nn, const double *q, int64_t nq, int64_t ld, int layout, int k,
                            const int64_t *prefix, int64_t *idx, double *dist, gbo_stream stream)
{
    Trace trace("gbo_nn_nearest_k");
    if (!nn || nq < 0 || k < 1 || (nq > 0 && (!q || !idx)) || !valid_layout(layout, nq, ld, nn->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad nearestK arguments");
    if (k > 64)
        return fail(GBO_ERR_UNSUPPORTED, "nearestK supports k <= 64");
    if (nq == 0)
        return GBO_OK;
    LaunchCfg lc = lcfg(stream);
    const SearchOrder order(nn, lc.stream);
    NNArgs a = nn_args(nn);
    StatesView qv = make_view(q, ld, layout);
    RunCounters *ctr = nn->ctr.take(lc.stream);
    nn->queries += nq;
    if (nn->precision == GBO_PRECISION_FP32_GUARDED && k <= knn_fp32_max_k(nn->sp))
    {
        if (auto st = nn->fb_list.reserve(sizeof(unsigned long long) * nq, lc.stream))
            return st;
        unsigned long long *fb_n = &ctr->queue;
        // The cell searches take batches that are worth more than their fixed cost (query order, the longest
        // search), counted in query-element pairs. Measured, cells / group kernel: 3-D, 200,000 elements, 512
        // queries (1e8 pairs) 102 / 162 us; wrapped 5-D, 100,000, 1,024 (1e8) 155 / 212 us; 6-D, 600,000, 256
        // (1.5e8) 265 us by the group kernel, 512 (3e8) 249 / 482 us; wrapped 7-D, 200,000, 1,024 (2e8) 446 us by
        // the group kernel, 2,048 (4e8) 466 / 800 us; chain, 200,000, 4,096 (8e8) 2.1 ms, 2,048 (4e8) 1.5 ms by
        // the group kernel.
        // An index that is not built yet costs 50 us (70,000 elements) to 95 us (600,000), what the group kernel
        // takes for 5e7 pairs: it is built by the batch that exceeds `worth` by as much, or by the batches since
        // the last change of the set together.
        const bool chain = nn->sp.kind == GBO_SPACE_KINEMATIC_CHAIN;
        const int dim = nn->sp.dim;
        constexpr int64_t kBuildPairs = 50000000ll;
        constexpr int64_t kBoxWorth[9] = {0,        30000000,  30000000,  30000000, 50000000,
                                          50000000, 120000000, 250000000, 400000000};
        const int64_t worth = chain ? 800000000ll : kBoxWorth[std::min(dim, 8)];
        const int64_t pairs = nq * nn->size;
        bool cells = nn->size >= (chain ? 65536 : 16384) && nn->size < (1ll << 30) && nq < (1ll << 31) &&
                     nq >= (chain ? 1024 : 64) && pairs >= worth && !(chain && prefix);
        if (cells && !chain && nn->cells[0].size != nn->size)
        {
            nn->forgone += std::min(pairs - worth, kBuildPairs);
            cells = nn->forgone >= kBuildPairs;
        }
        // a captured call builds none: the build would run with each replay, and not before later calls
        if (cells && order.captured && !cells_built(nn, prefix != nullptr))
            cells = false;
        // a huge batch over a tiny index: thread per query (100 elements, 20,000 queries: 148 us against
        // 186 us wrapped, 0.62 ms against 0.91 ms on the chain)
        const bool tiny = nq >= 16384 && nn->size <= 256;
        if (!cells && !tiny)
        {
            NNArgs g = a;
            if (nn->alive_count == nn->size)
                g.alive = nullptr;
            if (launch_knn_group(lc, g, nn->sp, qv, nq, k, prefix, INT64_MAX, idx, dist,
                                 (unsigned long long *)nn->fb_list.p, fb_n, ctr))
            {
                launch_knn_exact(lc, a, nn->sp, qv, nq, k, prefix, idx, dist,
                                 (const unsigned long long *)nn->fb_list.p, fb_n, std::min<int64_t>(nq, 4096));
                CHECK_LAUNCH();
                return GBO_OK;
            }
        }
        if (auto st = nn->qfeat.reserve(sizeof(float) * nn->F * nq, lc.stream))
            return st;
        launch_features(lc, nn->sp, qv, nq, (float *)nn->qfeat.p, nq);
        // large batches over a large RealVector / wrapped index: cell search (PRM's prefix kNN)
        if (cells && (nn->sp.kind == GBO_SPACE_WRAP_L2 || nn->sp.kind == GBO_SPACE_REAL_VECTOR) && nn->sp.dim <= 8)
        {
            if (auto st = box_cells_call(nn, lc, (const float *)nn->qfeat.p, nq, prefix, k,
                                         KnnOut{a, qv, idx, dist, (unsigned long long *)nn->fb_list.p, fb_n, ctr}))
                return st;
            launch_knn_exact(lc, a, nn->sp, qv, nq, k, prefix, idx, dist,
                             (const unsigned long long *)nn->fb_list.p, fb_n, std::min<int64_t>(nq, 4096));
            CHECK_LAUNCH();
            return GBO_OK;
        }
        // a large chain index: the cell search, one warp per query (the query order's keys are the cells)
        if (cells && chain && nn->sp.dim <= 10 && k <= 20)
        {
            const size_t wb = ((size_t)3 * kQueryKeys + nq) * sizeof(int);
            if (auto st = nn->qorder.reserve(wb + (size_t)nq * sizeof(int64_t) + 16, lc.stream))
                return st;
            int *work = (int *)nn->qorder.p;
            int64_t *ord = (int64_t *)((char *)nn->qorder.p + pad16(wb));
            launch_query_order(lc, nn->sp, (const float *)nn->qfeat.p, nq, work, ord);
            if (auto st = ensure_chain_cells(nn, lc))
                return st;
            NNChainCells &c = nn->ccells;
            const ChainCellArgs ci{(const int *)c.start.p,  (const int *)c.count.p, (const int64_t *)c.skey.p,
                                   (const float4 *)c.sfeat.p, nn->size,  (const uint4 *)c.box.p,
                                   (const int *)c.cstart.p,   (const uint4 *)c.cbox.p};
            if (launch_knn_ccell(lc, a, ci, nn->sp, qv, (const float *)nn->qfeat.p, nq, ord, work + 3 * kQueryKeys, k,
                                 idx, dist, (unsigned long long *)nn->fb_list.p, fb_n, ctr))
            {
                launch_knn_exact(lc, a, nn->sp, qv, nq, k, prefix, idx, dist,
                                 (const unsigned long long *)nn->fb_list.p, fb_n, std::min<int64_t>(nq, 4096));
                CHECK_LAUNCH();
                return GBO_OK;
            }
        }
        const int P = knn_chunks(lc, nq, nn->size);
        const int keep = knn_keep(k);
        const size_t pl = (size_t)P * nq * keep;
        if (auto st = nn->part.reserve(pl * (sizeof(float) + sizeof(int64_t)) + 64, lc.stream))
            return st;
        int64_t *part_k = (int64_t *)nn->part.p;
        float *part_d = (float *)(part_k + pl);
        if (launch_knn_fp32(lc, a, nn->sp, qv, (const float *)nn->qfeat.p, nq, k, prefix, idx, dist,
                            (unsigned long long *)nn->fb_list.p, fb_n, ctr, part_d, part_k, P))
        {
            // queries whose FP32 band overflowed: exact FP64 scan (count read on the device)
            launch_knn_exact(lc, a, nn->sp, qv, nq, k, prefix, idx, dist, (const unsigned long long *)nn->fb_list.p,
                             fb_n, std::min<int64_t>(nq, 4096));
            CHECK_LAUNCH();
            return GBO_OK;
        }
    }
    launch_knn_exact(lc, a, nn->sp, qv, nq, k, prefix, idx, dist, nullptr, nullptr, nq);
    CHECK_LAUNCH();
    return GBO_OK;
}

// counts, or with offsets the filled and sorted segments
static void radius_call(gbo_nn *nn, StatesView qv, int64_t nq, double r, int64_t *counts, const int64_t *offsets,
                        int64_t *idx, double *dist, gbo_stream stream)
{
    std::lock_guard<std::mutex> lk(nn->search_mu);
    NNArgs a = nn_args(nn);
    if (nn->alive_count == nn->size)
        a.alive = nullptr;
    if (nn->precision == GBO_PRECISION_FP32_GUARDED &&
        launch_radius_group(lcfg(stream), a, nn->sp, qv, nq, r, nn->outside, counts, offsets, idx, dist))
        return;
    launch_radius(lcfg(stream), nn_args(nn), nn->sp, qv, nq, r, counts, offsets, idx, dist);
}

gbo_status gbo_nn_nearest_r_count(gbo_nn *nn, const double *q, int64_t nq, int64_t ld, int layout, double r,
                                  int64_t *counts, gbo_stream stream)
{
    if (!nn || nq < 0 || (nq > 0 && (!q || !counts)) || !valid_layout(layout, nq, ld, nn->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad nearestR arguments");
    radius_call(nn, make_view(q, ld, layout), nq, r, counts, nullptr, nullptr, nullptr, stream);
    CHECK_LAUNCH();
    return GBO_OK;
}

gbo_status gbo_nn_nearest_r_fill(gbo_nn *nn, const double *q, int64_t nq, int64_t ld, int layout, double r,
                                 const int64_t *offsets, int64_t *idx, double *dist, gbo_stream stream)
{
    if (!nn || nq < 0 || (nq > 0 && (!q || !offsets || !idx || !dist)) || !valid_layout(layout, nq, ld, nn->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad nearestR arguments");
    radius_call(nn, make_view(q, ld, layout), nq, r, nullptr, offsets, idx, dist, stream);
    CHECK_LAUNCH();
    return GBO_OK;
}

// NearestNeighborsSqrtApprox::nearest (NearestNeighborsSqrtApprox.h:91-115) for nq queries made one after
// another. checks = 1 + floor(sqrt(n)) for the n present elements; *offset is the structure's offset
// before the first query and after the last. Positions count the present elements in insertion order
// (NearestNeighborsLinear's vector, whose remove erases); with removals a table of their keys is built
// on the host.
gbo_status gbo_nn_nearest_sqrt_approx(gbo_nn *nn, const double *q, int64_t nq, int64_t ld, int layout,
                                      uint64_t *offset, int64_t *idx, double *dist, gbo_stream stream)
{
    Trace trace("gbo_nn_nearest_sqrt_approx");
    if (!nn || !offset || nq < 0 || (nq > 0 && (!q || !idx || !dist)) ||
        !(layout == GBO_LAYOUT_SOA ? ld >= nq : (layout == GBO_LAYOUT_AOS && ld >= nn->sp.dim)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad nearest arguments");
    if (nq == 0)
        return GBO_OK;
    int64_t n = 0;
    if (auto st = gbo_nn_size(nn, &n))
        return st;
    if (n == 0)
        return fail(GBO_ERR_INVALID_ARGUMENT, "No elements found in nearest neighbors data structure");
    const int64_t checks = 1 + (int64_t)std::floor(std::sqrt((double)n));
    const cudaStream_t s = (cudaStream_t)stream;
    const int64_t *rank = nullptr;
    if (n != nn->size)
    {
        std::vector<unsigned char> alive((size_t)nn->size);
        CUDA_TRY(cudaStreamSynchronize(s));
        CUDA_TRY(cudaMemcpy(alive.data(), nn->alive, (size_t)nn->size, cudaMemcpyDeviceToHost));
        std::vector<int64_t> keys;
        keys.reserve((size_t)n);
        for (int64_t k = 0; k < nn->size; ++k)
            if (alive[(size_t)k])
                keys.push_back(k);
        if ((int64_t)keys.size() != n)
            return fail(GBO_ERR_INVALID_ARGUMENT, "element count changed during the call");
        if (auto st = nn->ranks.reserve(keys.size() * sizeof(int64_t), s))
            return st;
        CUDA_TRY(cudaMemcpyAsync(nn->ranks.p, keys.data(), keys.size() * sizeof(int64_t), cudaMemcpyHostToDevice, s));
        rank = (const int64_t *)nn->ranks.p;
    }
    launch_sqrt_approx(lcfg(stream), nn_args(nn), nn->sp, make_view(q, ld, layout), nq, n, checks,
                       (unsigned long long)*offset, rank, idx, dist);
    CHECK_LAUNCH();
    if (rank)
        CUDA_TRY(cudaStreamSynchronize(s));  // the key table is host memory's copy
    *offset = (*offset + (uint64_t)nq) % (uint64_t)checks;
    return GBO_OK;
}

gbo_status gbo_nn_error_stats(const gbo_nn *nn, float *max_abs_error, float *bound)
{
    if (!nn)
        return fail(GBO_ERR_INVALID_ARGUMENT, "nn is NULL");
    RunCounters h{};
    CUDA_TRY(cudaMemcpy(&h, nn->ctr.dev + nn->ctr.last, sizeof(h), cudaMemcpyDeviceToHost));
    if (max_abs_error)
    {
        float e;
        std::memcpy(&e, &h.max_err_bits, sizeof(e));
        *max_abs_error = e;
    }
    if (bound)
        *bound = nn->eps32;
    return GBO_OK;
}

gbo_status gbo_nn_stats(const gbo_nn *nn, uint64_t *queries, uint64_t *rechecked, uint64_t *fallbacks)
{
    if (!nn)
        return fail(GBO_ERR_INVALID_ARGUMENT, "nn is NULL");
    RunCounters h{};
    CUDA_TRY(cudaMemcpy(&h, nn->ctr.dev + nn->ctr.last, sizeof(h), cudaMemcpyDeviceToHost));
    if (queries)
        *queries = nn->queries;
    if (rechecked)
        *rechecked = h.rechecked;
    if (fallbacks)
        *fallbacks = h.fallbacks;
    return GBO_OK;
}

gbo_status gbo_nn_search_bytes(const gbo_nn *nn, uint64_t *bytes)
{
    if (!nn || !bytes)
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad search-bytes arguments");
    RunCounters h{};
    CUDA_TRY(cudaMemcpy(&h, nn->ctr.dev + nn->ctr.last, sizeof(h), cudaMemcpyDeviceToHost));
    *bytes = h.bytes;
    return GBO_OK;
}

gbo_status gbo_nn_add_host(gbo_nn *nn, const double *states, int64_t n, int64_t *first_key)
{
    if (!nn || n < 0 || (n > 0 && !states))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad add arguments");
    std::lock_guard<std::mutex> lk(nn->mu);
    const size_t b = (size_t)n * nn->sp.dim * sizeof(double);
    if (auto st = nn->pin.reserve(b + 16))
        return st;
    if (auto st = nn->dev.reserve(b + 16, nn->host_stream))
        return st;
    std::memcpy(nn->pin.p, states, b);
    CUDA_TRY(cudaMemcpyAsync(nn->dev.p, nn->pin.p, b, cudaMemcpyHostToDevice, nn->host_stream));
    if (auto st = gbo_nn_add(nn, (const double *)nn->dev.p, n, nn->sp.dim, GBO_LAYOUT_AOS, first_key,
                             nn->host_stream))
        return st;
    CUDA_TRY(cudaStreamSynchronize(nn->host_stream));
    return GBO_OK;
}

gbo_status gbo_nn_remove_host(gbo_nn *nn, const int64_t *keys, int64_t n)
{
    if (!nn || n < 0 || (n > 0 && !keys))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad remove arguments");
    std::lock_guard<std::mutex> lk(nn->mu);
    const size_t b = (size_t)n * sizeof(int64_t);
    if (auto st = nn->dev.reserve(b + 16, nn->host_stream))
        return st;
    CUDA_TRY(cudaMemcpyAsync(nn->dev.p, keys, b, cudaMemcpyHostToDevice, nn->host_stream));
    if (auto st = gbo_nn_remove(nn, (const int64_t *)nn->dev.p, n, nn->host_stream))
        return st;
    CUDA_TRY(cudaStreamSynchronize(nn->host_stream));
    return GBO_OK;
}

gbo_status gbo_nn_nearest_k_host(gbo_nn *nn, const double *q, int64_t nq, int k, int64_t *idx, double *dist)
{
    if (!nn || nq < 0 || k < 1 || (nq > 0 && (!q || !idx)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad nearestK arguments");
    std::lock_guard<std::mutex> lk(nn->mu);
    const size_t bq = (size_t)nq * nn->sp.dim * sizeof(double), bo = (size_t)nq * k * 8;
    if (auto st = nn->pin.reserve(std::max(bq, 2 * bo) + 16))
        return st;
    if (auto st = nn->dev.reserve(bq + 2 * bo + 32, nn->host_stream))
        return st;
    char *d = (char *)nn->dev.p;
    std::memcpy(nn->pin.p, q, bq);
    CUDA_TRY(cudaMemcpyAsync(d, nn->pin.p, bq, cudaMemcpyHostToDevice, nn->host_stream));
    int64_t *di = (int64_t *)(d + pad16(bq));
    double *dd = (double *)(d + pad16(bq) + bo);
    if (auto st = gbo_nn_nearest_k(nn, (const double *)d, nq, nn->sp.dim, GBO_LAYOUT_AOS, k, nullptr, di,
                                   dist ? dd : nullptr, nn->host_stream))
        return st;
    CUDA_TRY(cudaMemcpyAsync(nn->pin.p, di, bo, cudaMemcpyDeviceToHost, nn->host_stream));
    if (dist)
        CUDA_TRY(cudaMemcpyAsync((char *)nn->pin.p + bo, dd, bo, cudaMemcpyDeviceToHost, nn->host_stream));
    CUDA_TRY(cudaStreamSynchronize(nn->host_stream));
    std::memcpy(idx, nn->pin.p, bo);
    if (dist)
        std::memcpy(dist, (char *)nn->pin.p + bo, bo);
    return GBO_OK;
}

gbo_status gbo_nn_nearest_k_rows(gbo_nn *nn, const double *q, int64_t nq, int k, int64_t *idx, double *dist,
                                 gbo_stream stream)
{
    if (!nn || nq < 0 || k < 1 || (nq > 0 && (!q || !idx || !dist)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad nearestK arguments");
    if (k > 64)
        return fail(GBO_ERR_UNSUPPORTED, "nearestK supports k <= 64");
    if (nq == 0)
        return GBO_OK;
    const size_t bq = (size_t)nq * nn->sp.dim * sizeof(double), bo = (size_t)nq * k * 8;
    RowCall call(nn->rows, (cudaStream_t)stream);
    if (auto e = call.reserve(bq + 2 * bo))
        return e;
    char *h = call.host(), *d = call.device();
    std::memcpy(h, q, bq);
    if (auto e = call.copy_in(bq))
        return e;
    if (auto e = gbo_nn_nearest_k(nn, (const double *)d, nq, nn->sp.dim, GBO_LAYOUT_AOS, k, nullptr,
                                  (int64_t *)(d + bq), (double *)(d + bq + bo), stream))
        return e;
    if (auto e = call.copy_out(bq, 2 * bo))
        return e;
    std::memcpy(idx, h + bq, bo);
    std::memcpy(dist, h + bq + bo, bo);
    return GBO_OK;
}

gbo_status gbo_nn_nearest_sqrt_approx_host(gbo_nn *nn, const double *q, int64_t nq, uint64_t *offset, int64_t *idx,
                                           double *dist)
{
    if (!nn || !offset || nq < 0 || (nq > 0 && (!q || !idx)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad nearest arguments");
    std::lock_guard<std::mutex> lk(nn->mu);
    const size_t bq = (size_t)nq * nn->sp.dim * sizeof(double), bo = (size_t)nq * 8;
    if (auto st = nn->pin.reserve(std::max(bq, 2 * bo) + 16))
        return st;
    if (auto st = nn->dev.reserve(bq + 2 * bo + 32, nn->host_stream))
        return st;
    char *d = (char *)nn->dev.p;
    std::memcpy(nn->pin.p, q, bq);
    CUDA_TRY(cudaMemcpyAsync(d, nn->pin.p, bq, cudaMemcpyHostToDevice, nn->host_stream));
    int64_t *di = (int64_t *)(d + pad16(bq));
    double *dd = (double *)(d + pad16(bq) + bo);
    if (auto st = gbo_nn_nearest_sqrt_approx(nn, (const double *)d, nq, nn->sp.dim, GBO_LAYOUT_AOS, offset, di, dd,
                                             nn->host_stream))
        return st;
    CUDA_TRY(cudaMemcpyAsync(nn->pin.p, di, bo, cudaMemcpyDeviceToHost, nn->host_stream));
    CUDA_TRY(cudaMemcpyAsync((char *)nn->pin.p + bo, dd, bo, cudaMemcpyDeviceToHost, nn->host_stream));
    CUDA_TRY(cudaStreamSynchronize(nn->host_stream));
    std::memcpy(idx, nn->pin.p, bo);
    if (dist)
        std::memcpy(dist, (char *)nn->pin.p + bo, bo);
    return GBO_OK;
}

gbo_status gbo_nn_nearest_r_host(gbo_nn *nn, const double *q, double r, int64_t cap, int64_t *count, int64_t *idx,
                                 double *dist)
{
    if (!nn || !q || !count || cap < 0 || (cap > 0 && (!idx || !dist)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad nearestR arguments");
    std::lock_guard<std::mutex> lk(nn->mu);
    const int dim = nn->sp.dim;
    if (auto st = nn->dev.reserve(64 + 16 * (size_t)(nn->size + 1) + 16 * (size_t)dim, nn->host_stream))
        return st;
    char *d = (char *)nn->dev.p;
    double *dq = (double *)d;
    int64_t *dcount = (int64_t *)(d + 16 * ((dim * 8 + 15) / 16));
    int64_t *doff = dcount + 1;
    int64_t *didx = dcount + 2;
    double *ddist = (double *)(didx + nn->size + 1);
    CUDA_TRY(cudaMemcpyAsync(dq, q, dim * sizeof(double), cudaMemcpyHostToDevice, nn->host_stream));
    CUDA_TRY(cudaMemsetAsync(doff, 0, sizeof(int64_t), nn->host_stream));
    if (auto st = gbo_nn_nearest_r_count(nn, dq, 1, dim, GBO_LAYOUT_AOS, r, dcount, nn->host_stream))
        return st;
    if (auto st = gbo_nn_nearest_r_fill(nn, dq, 1, dim, GBO_LAYOUT_AOS, r, doff, didx, ddist, nn->host_stream))
        return st;
    int64_t c = 0;
    CUDA_TRY(cudaMemcpyAsync(&c, dcount, sizeof(int64_t), cudaMemcpyDeviceToHost, nn->host_stream));
    CUDA_TRY(cudaStreamSynchronize(nn->host_stream));
    *count = c;
    const int64_t m = std::min(c, cap);
    if (m > 0)
    {
        CUDA_TRY(cudaMemcpy(idx, didx, m * sizeof(int64_t), cudaMemcpyDeviceToHost));
        CUDA_TRY(cudaMemcpy(dist, ddist, m * sizeof(double), cudaMemcpyDeviceToHost));
    }
    return GBO_OK;
}

gbo_status gbo_sample_uniform_host(gbo_sampler *s, int64_t n, double *out)
{
    if (!s || n < 0 || (n > 0 && !out))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sampleUniform arguments");
    std::lock_guard<std::mutex> lk(s->mu);
    const size_t b = (size_t)n * s->sp.dim * sizeof(double);
    if (auto st = s->dev.reserve(b + 16, s->host_stream))
        return st;
    if (auto st = s->pin.reserve(b + 16))
        return st;
    if (auto st = gbo_sample_uniform(s, n, (double *)s->dev.p, s->sp.dim, GBO_LAYOUT_AOS, s->host_stream))
        return st;
    CUDA_TRY(cudaMemcpyAsync(s->pin.p, s->dev.p, b, cudaMemcpyDeviceToHost, s->host_stream));
    CUDA_TRY(cudaStreamSynchronize(s->host_stream));
    std::memcpy(out, s->pin.p, b);
    return GBO_OK;
}

gbo_status gbo_sample_valid_host(gbo_sampler *s, gbo_checker *c, int64_t n, unsigned attempts, double *out,
                                 uint8_t *ok)
{
    if (!s || !c || n < 0 || (n > 0 && (!out || !ok)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sampleValid arguments");
    if (n == 0)
        return GBO_OK;
    std::lock_guard<std::mutex> lk(s->mu);
    const size_t b = (size_t)n * s->sp.dim * sizeof(double);
    if (auto st = s->dev.reserve(b + (size_t)n + 16, s->host_stream))
        return st;
    double *d = (double *)s->dev.p;
    uint8_t *dok = (uint8_t *)s->dev.p + b;
    if (auto st = gbo_sample_valid(s, c, n, attempts, d, s->sp.dim, GBO_LAYOUT_AOS, dok, s->host_stream))
        return st;
    CUDA_TRY(cudaMemcpyAsync(out, d, b, cudaMemcpyDeviceToHost, s->host_stream));
    CUDA_TRY(cudaMemcpyAsync(ok, dok, (size_t)n, cudaMemcpyDeviceToHost, s->host_stream));
    CUDA_TRY(cudaStreamSynchronize(s->host_stream));
    return GBO_OK;
}

gbo_status gbo_sample_uniform_near_host(gbo_sampler *s, const double *near, double distance, int64_t n, double *out)
{
    if (!s || n < 0 || (n > 0 && (!out || !near)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sampleUniformNear arguments");
    std::lock_guard<std::mutex> lk(s->mu);
    const size_t b = (size_t)n * s->sp.dim * sizeof(double);
    if (auto st = s->dev.reserve(2 * b + 32, s->host_stream))
        return st;
    if (auto st = s->pin.reserve(b + 16))
        return st;
    double *dn = (double *)s->dev.p, *dout = (double *)((char *)s->dev.p + pad16(b));
    std::memcpy(s->pin.p, near, b);
    CUDA_TRY(cudaMemcpyAsync(dn, s->pin.p, b, cudaMemcpyHostToDevice, s->host_stream));
    if (auto st = gbo_sample_uniform_near(s, dn, distance, n, s->sp.dim, GBO_LAYOUT_AOS, dout, s->host_stream))
        return st;
    CUDA_TRY(cudaMemcpyAsync(s->pin.p, dout, b, cudaMemcpyDeviceToHost, s->host_stream));
    CUDA_TRY(cudaStreamSynchronize(s->host_stream));
    std::memcpy(out, s->pin.p, b);
    return GBO_OK;
}

gbo_status gbo_sample_gaussian_host(gbo_sampler *s, const double *mean, double stddev, int64_t n, double *out)
{
    if (!s || n < 0 || (n > 0 && (!out || !mean)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sampleGaussian arguments");
    std::lock_guard<std::mutex> lk(s->mu);
    const size_t b = (size_t)n * s->sp.dim * sizeof(double);
    if (auto st = s->dev.reserve(2 * b + 32, s->host_stream))
        return st;
    if (auto st = s->pin.reserve(b + 16))
        return st;
    double *dm = (double *)s->dev.p, *dout = (double *)((char *)s->dev.p + pad16(b));
    std::memcpy(s->pin.p, mean, b);
    CUDA_TRY(cudaMemcpyAsync(dm, s->pin.p, b, cudaMemcpyHostToDevice, s->host_stream));
    if (auto st = gbo_sample_gaussian(s, dm, stddev, n, s->sp.dim, GBO_LAYOUT_AOS, dout, s->host_stream))
        return st;
    CUDA_TRY(cudaMemcpyAsync(s->pin.p, dout, b, cudaMemcpyDeviceToHost, s->host_stream));
    CUDA_TRY(cudaStreamSynchronize(s->host_stream));
    std::memcpy(out, s->pin.p, b);
    return GBO_OK;
}

// PRM::uniteComponents over a roadmap's edges in the order PRM adds them (PRM.cpp:580-609): boost's
// disjoint_sets, every vertex first its own set; union_set(n, m) links the two roots by rank (the root of
// higher rank becomes the parent of the other; on a tie the root of m's set becomes the parent and its
// rank grows), finds compress paths. root[v] = find_set(v) after the last union: the component tag that
// PRM::getPlannerData gives each vertex (PRM.cpp:734-754). Host memory, no device work.
gbo_status gbo_prm_component_roots(const int64_t *src, const int64_t *dst, int64_t n_edges, int64_t n_vertices,
                                   int64_t *root)
{
    if (n_edges < 0 || n_vertices < 0 || (n_edges && (!src || !dst)) || (n_vertices && !root))
        return GBO_ERR_INVALID_ARGUMENT;
    std::vector<int64_t> parent((size_t)n_vertices);
    std::vector<uint32_t> rank((size_t)n_vertices, 0);
    for (int64_t v = 0; v < n_vertices; ++v)
        parent[(size_t)v] = v;
    auto find = [&](int64_t x) {
        int64_t r = x;
        while (parent[(size_t)r] != r)
            r = parent[(size_t)r];
        while (parent[(size_t)x] != r)
        {
            const int64_t next = parent[(size_t)x];
            parent[(size_t)x] = r;
            x = next;
        }
        return r;
    };
    for (int64_t e = 0; e < n_edges; ++e)
    {
        if (src[e] < 0 || src[e] >= n_vertices || dst[e] < 0 || dst[e] >= n_vertices)
            return GBO_ERR_INVALID_ARGUMENT;
        const int64_t i = find(src[e]), j = find(dst[e]);
        if (i == j)
            continue;
        if (rank[(size_t)i] > rank[(size_t)j])
            parent[(size_t)j] = i;
        else
        {
            parent[(size_t)i] = j;
            if (rank[(size_t)i] == rank[(size_t)j])
                ++rank[(size_t)j];
        }
    }
    for (int64_t v = 0; v < n_vertices; ++v)
        root[v] = find(v);
    return GBO_OK;
}

gbo_status gbo_measure_fp32_peak(double *flops, gbo_stream stream)
{
    if (!flops)
        return fail(GBO_ERR_INVALID_ARGUMENT, "flops is NULL");
    if (auto st = ensure_device())
        return st;
    *flops = measure_fp32_peak(lcfg(stream));
    CHECK_LAUNCH();
    return GBO_OK;
}

gbo_status gbo_sincos32(const double *theta, int64_t n, float *cos_out, float *sin_out, gbo_stream stream)
{
    if (n < 0 || (n > 0 && (!theta || !cos_out || !sin_out)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sincos32 arguments");
    if (auto st = ensure_device())
        return st;
    launch_sincos32(lcfg(stream), theta, n, cos_out, sin_out);
    CHECK_LAUNCH();
    return GBO_OK;
}

gbo_status gbo_log_rn(const double *x, int64_t n, double *out, gbo_stream stream)
{
    if (n < 0 || n > (int64_t)INT32_MAX * 256 || (n > 0 && (!x || !out)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad log_rn arguments");
    if (auto st = ensure_device())
        return st;
    launch_log_rn(lcfg(stream), x, n, out);
    CHECK_LAUNCH();
    return GBO_OK;
}

gbo_status gbo_sincos_cr(const double *x, int64_t n, double *sin_out, double *cos_out, gbo_stream stream)
{
    if (n < 0 || (n > 0 && (!x || !sin_out || !cos_out)))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad sincos_cr arguments");
    if (auto st = ensure_device())
        return st;
    launch_sincos_cr(lcfg(stream), x, n, sin_out, cos_out);
    CHECK_LAUNCH();
    return GBO_OK;
}

gbo_status gbo_checker_precision_stats(gbo_checker *c, const double *states, int64_t n, int64_t ld, int layout,
                                       gbo_precision_stats *out, gbo_stream stream)
{
    if (!c || !out || n < 0 || (n > 0 && !states) || !valid_layout(layout, n, ld, c->sp.dim))
        return fail(GBO_ERR_INVALID_ARGUMENT, "bad precision_stats arguments");
    if (c->wa.kind != GBO_CHECK_CHAIN_SEGMENTS && c->wa.kind != GBO_CHECK_DH_SPHERES)
        return fail(GBO_ERR_UNSUPPORTED, "this checker has no FP32 form");
    struct Tally
    {
        unsigned long long states, flips, ambiguous;
        unsigned int max_err_bits;
    } h{};
    void *d = nullptr;
    if (cudaMalloc(&d, sizeof(Tally)) != cudaSuccess)
        return fail(GBO_ERR_OUT_OF_MEMORY, "precision_stats buffer");
    LaunchCfg lc = lcfg(stream);
    cudaMemsetAsync(d, 0, sizeof(Tally), lc.stream);
    const bool launched = n > 0 && launch_precision_stats(lc, c->sp, c->wa, make_view(states, ld, layout), n, d);
    cudaMemcpyAsync(&h, d, sizeof(Tally), cudaMemcpyDeviceToHost, lc.stream);
    const cudaError_t e = cudaStreamSynchronize(lc.stream);
    cudaFree(d);
    if (e != cudaSuccess)
        return fail(GBO_ERR_CUDA, cudaGetErrorString(e));
    if (n > 0 && !launched)
        return fail(GBO_ERR_UNSUPPORTED, "precision statistics not available for this checker's size");
    float mx;
    std::memcpy(&mx, &h.max_err_bits, sizeof(mx));
    out->states = h.states;
    out->flips = h.flips;
    out->ambiguous = h.ambiguous;
    out->max_abs_err = mx;
    return GBO_OK;
}

gbo_status gbo_measure_fp64_peak(double *flops, gbo_stream stream)
{
    if (!flops)
        return fail(GBO_ERR_INVALID_ARGUMENT, "flops is NULL");
    if (auto st = ensure_device())
        return st;
    *flops = measure_fp64_peak(lcfg(stream));
    CHECK_LAUNCH();
    return GBO_OK;
}

}  // extern "C"

// ---------------------------------------------------------------- internal accessors (noalloc.cu)
namespace gbo
{
gbo_status internal_fail(gbo_status s, const char *msg)
{
    return fail(s, msg);
}

gbo_status internal_ensure_device(int *sm_count)
{
    if (auto st = ensure_device())
        return st;
    *sm_count = g_sm_count;
    return GBO_OK;
}

gbo_status internal_request_dim(const gbo_request *r, int *dim)
{
    if (r->kind == GBO_REQ_KNN)
    {
        if (!r->nn)
            return GBO_ERR_INVALID_ARGUMENT;
        *dim = r->nn->sp.dim;
        return GBO_OK;
    }
    if ((r->kind != GBO_REQ_VALIDITY && r->kind != GBO_REQ_MOTION) || !r->checker)
        return GBO_ERR_INVALID_ARGUMENT;
    *dim = r->checker->sp.dim;
    return GBO_OK;
}

bool internal_nn_view(const gbo_nn *nn, NNArgs *a, SpaceParams *sp, int *precision, int *features)
{
    if (!nn)
        return false;
    *a = nn_args(nn);
    *sp = nn->sp;
    *precision = nn->precision;
    *features = nn->F;
    return true;
}
}  // namespace gbo
