// Cell search for nearestK over large RealVector / wrapped indexes, one warp per query.
//
// Index: a uniform grid of L levels per coordinate (about 40 to 280 elements a cell). Inside a cell the elements
// are in the order of `sub` further bits, one per coordinate (the half of the level they lie in), and every 32
// of them are a chunk with a box and its smallest key.
//
// Search: a query seeds its threshold T with the k-th FP32 distance found in its own cell (an upper bound on
// its k-th overall), then visits the cells in three rings of growing distance, so that T has tightened before
// the many far cells are looked at. A cell's distance is a sum of per-coordinate distances to its levels'
// intervals; the sums over the first half of the coordinates and over the rest are tabulated per query, so a
// lane's cell test is two shared-memory reads and an add. A visited cell's chunks are tested by their boxes, 32
// at a time, and the needed ones scanned, 32 elements at a time. The kept list lives in the lanes and is decided
// there in FP64 (warp_finish).
//
// Prefix limits (PRM: query m sees the first m elements): queries with a limit in (S / 2, S] use an index over
// the first S elements, S = size, size / 2, ..., so that at most half of what a query meets lies past its limit;
// the lowest limits go to knn_group_kernel.
//
// PRM of 2M samples (620,000 milestones, wrapped 7-D, k = 10): 90 ms with all cells' boxes tested in index order,
// every element of a needed cell scanned and limits below a quarter left to a thread-per-query scan (28 of the
// 90); 40 ms, index builds included. 200,000 wrapped 5-D elements, 4,096 queries: 136 us. Bound: instruction issue of
// the chunk scans and box tests.
#include <algorithm>

#include "nn_device.cuh"

namespace gbo
{

constexpr int kSubMax = 1 << 19;  // cells times sub-cells

// Lower bound of the metric distance of x from a point of [lo, hi] on the circle. The metric folds t = |x - y| to
// min(t, 2 pi - t), which is negative from 2 pi on (elements outside [-pi, pi], an interval widened past the wrap) and
// counts by its square: 0 inside and where an end lies that far, else the nearer end's. (Outside, the nearer end is
// max(p, r) away, the other max(|p|, |r|).)
__device__ __forceinline__ float wrap_gap(float x, float lo, float hi)
{
    const float p = lo - x, r = x - hi;
    return fmaxf(fminf(fmaxf(p, r), 6.28318530717958647692f - fmaxf(fabsf(p), fabsf(r))), 0.f);
}

// distance from query q to the box (lo, hi per coordinate), squared, scaled down by (1 - 1e-5) against
// the rounding of both sides
template <int KIND, int MAXF>
__device__ __forceinline__ float bcell_lb(const float4 *b, const float *q, int dim)
{
    const float4 l0 = b[0], l1 = b[1], h0 = b[2], h1 = b[3];
    const float lo[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
    const float hi[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < MAXF; ++i)
        if (i < dim)
        {
            const float x = q[i];
            float d;
            if constexpr (KIND == GBO_SPACE_WRAP_L2 || KIND == GBO_SPACE_SO2)
                d = wrap_gap(x, lo[i], hi[i]);
            else
                d = fmaxf(fmaxf(lo[i] - x, x - hi[i]), 0.f);
            s = fmaf(d, d, s);
        }
    return s * (1.0f - 1e-5f);
}

__device__ __forceinline__ void cell_range(const SpaceParams &sp, int d, float &lo, float &hi)
{
    if (sp.kind == GBO_SPACE_REAL_VECTOR)
    {
        lo = (float)sp.low[d];
        hi = (float)sp.high[d];
    }
    else
    {
        lo = -3.14159265358979f;
        hi = 3.14159265358979f;
    }
}

// Level of value x of coordinate d, and the half of the level it lies in
__device__ __forceinline__ int cell_level(const SpaceParams &sp, int L, int d, float x, int &half)
{
    float lo, hi;
    cell_range(sp, d, lo, hi);
    half = 0;
    if (!(hi > lo))
        return 0;
    const float g = (x - lo) * ((float)L / (hi - lo));
    const float f = fminf(fmaxf(floorf(g), 0.f), (float)(L - 1));  // NaN: 0
    half = g - f >= 0.5f;
    return (int)f;
}

__device__ __forceinline__ int cell_of(const SpaceParams &sp, int L, const float *f, int64_t ld, int64_t i, int &sub)
{
    int c = 0;
    sub = 0;
    for (int d = sp.dim - 1; d >= 0; --d)
    {
        int h;
        c = c * L + cell_level(sp, L, d, f[(int64_t)d * ld + i], h);
        sub = 2 * sub + h;
    }
    return c;
}

__device__ __forceinline__ int float_order(float x)
{
    const int b = __float_as_int(x);
    return b >= 0 ? b : b ^ 0x7fffffff;
}

// key[i] = cell << bits | sub of the present elements (else -1), their counts, and each coordinate's extremes
__global__ void __launch_bounds__(256) cell_assign_kernel(SpaceParams sp, int L, int bits, const float *feat,
                                                          int64_t cap, const unsigned char *alive, int64_t n, int *key,
                                                          int *count, int *extent)
{
    __shared__ int mn[8], mx[8];
    if (threadIdx.x < 8)
    {
        mn[threadIdx.x] = INT_MAX;
        mx[threadIdx.x] = INT_MIN;
    }
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
        int k = -1;
        if (alive[i])
        {
            int sub;
            const int c = cell_of(sp, L, feat, cap, i, sub);
            k = c << bits | (sub & ((1 << bits) - 1));
            atomicAdd(&count[k], 1);
            for (int d = 0; d < sp.dim; ++d)
            {
                const float x = feat[(int64_t)d * cap + i];
                const int v = float_order(x);
                if (x != x)
                    continue;
                if (v < mn[d])
                    atomicMin(&mn[d], v);
                if (v > mx[d])
                    atomicMax(&mx[d], v);
            }
        }
        key[i] = k;
    }
    __syncthreads();
    if (threadIdx.x < sp.dim)
    {
        atomicMin(&extent[2 * threadIdx.x], mn[threadIdx.x]);
        atomicMax(&extent[2 * threadIdx.x + 1], mx[threadIdx.x]);
    }
}

// the extremes from their integer order back to floats
__global__ void cell_extent_kernel(int *extent)
{
    if (threadIdx.x < 16)
    {
        const int b = extent[threadIdx.x];
        extent[threadIdx.x] = b >= 0 ? b : b ^ 0x7fffffff;
    }
}

__global__ void cell_clear_kernel(int *extent)
{
    if (threadIdx.x < 16)
        extent[threadIdx.x] = threadIdx.x & 1 ? INT_MIN : INT_MAX;
}

// Exclusive scan of n counts in two launches: block sums, then every block adds up the blocks before it.
// start[0 .. n]; fill[0 .. n - 1] = start.
constexpr int kScanBlock = 4096;

__global__ void __launch_bounds__(1024) scan_sums_kernel(const int *count, int n, int *sums)
{
    __shared__ int part[32];
    const int i0 = blockIdx.x * kScanBlock + threadIdx.x * 4;
    int s = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        s += i0 + j < n ? count[i0 + j] : 0;
    s = __reduce_add_sync(0xffffffffu, s);
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32)
    {
        s = __reduce_add_sync(0xffffffffu, part[threadIdx.x]);
        if (threadIdx.x == 0)
            sums[blockIdx.x] = s;
    }
}

__global__ void __launch_bounds__(1024) scan_kernel(const int *count, int n, const int *sums, int *start, int *fill)
{
    __shared__ int part[32];
    __shared__ int base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
        base = 0;
    __syncthreads();
    int before = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += 1024)
        before += sums[b];
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0 && before)
        atomicAdd(&base, before);
    const int i0 = blockIdx.x * kScanBlock + threadIdx.x * 4;
    int v[4], s = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        v[j] = i0 + j < n ? count[i0 + j] : 0;
        s += v[j];
    }
    int incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
            incl += t;
    }
    if (lane == 31)
        part[warp] = incl;
    __syncthreads();
    if (warp == 0)
    {
        int t = part[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o)
                t += u;
        }
        part[lane] = t;
    }
    __syncthreads();
    int run = base + (warp ? part[warp - 1] : 0) + incl - s;
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        if (i0 + j < n)
        {
            start[i0 + j] = run;
            fill[i0 + j] = run;
        }
        run += v[j];
        if (i0 + j == n - 1)
            start[n] = run;
    }
}

__global__ void cell_scatter_kernel(const int *key, int64_t n, int *fill, int *out)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
        const int c = key[i];
        if (c >= 0)
            out[atomicAdd(&fill[c], 1)] = (int)i;
    }
}

// chunks per cell (cell c holds positions start[c << bits] .. start[(c + 1) << bits])
__global__ void cell_chunks_kernel(const int *start, int bits, int C, int *chunks)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < C)
        chunks[c] = (start[(c + 1) << bits] - start[c << bits] + 31) / 32;
}

// sorted coordinates pts8[2p], pts8[2p + 1] (unused ones 0), and each chunk's box (min of coordinates 0-3, 4-7,
// then max) and smallest key: a warp per cell
__global__ void __launch_bounds__(256) cell_fill_kernel(const float *feat, int64_t cap, int dim, const int *start, int bits,
                                                        int C, const int *cstart, const int *skey, float4 *pts8,
                                                        float4 *box, int *kmin)
{
    const int lane = threadIdx.x & 31;
    for (int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); c < C; c += (int)((gridDim.x * blockDim.x) >> 5))
    {
        const int s0 = start[c << bits], s1 = start[(c + 1) << bits];
        for (int p0 = s0, ch = cstart[c]; p0 < s1; p0 += 32, ++ch)
        {
            const int p = p0 + lane;
            const bool in = p < s1;
            const int key = in ? skey[p] : INT_MAX;
            float v[8], mn[8], mx[8];
#pragma unroll
            for (int d = 0; d < 8; ++d)
            {
                v[d] = in && d < dim ? feat[(int64_t)d * cap + key] : 0.f;
                mn[d] = in ? v[d] : __int_as_float(0x7f800000);
                mx[d] = in ? v[d] : -__int_as_float(0x7f800000);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                {
                    mn[d] = fminf(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
                    mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
                }
            }
            const int km = __reduce_min_sync(0xffffffffu, key);
            if (in)
            {
                pts8[2 * (int64_t)p] = make_float4(v[0], v[1], v[2], v[3]);
                pts8[2 * (int64_t)p + 1] = make_float4(v[4], v[5], v[6], v[7]);
            }
            if (lane == 0)
            {
                box[4 * (int64_t)ch] = make_float4(mn[0], mn[1], mn[2], mn[3]);
                box[4 * (int64_t)ch + 1] = make_float4(mn[4], mn[5], mn[6], mn[7]);
                box[4 * (int64_t)ch + 2] = make_float4(mx[0], mx[1], mx[2], mx[3]);
                box[4 * (int64_t)ch + 3] = make_float4(mx[4], mx[5], mx[6], mx[7]);
                kmin[ch] = km;
            }
        }
    }
}

// cell of the queries with a limit in (above, size] (all without limits), else -1
__global__ void cell_query_kernel(SpaceParams sp, int L, const float *qf, int64_t nq, const int64_t *prefix,
                                  int64_t above, int64_t size, bool top, int *key, int *count)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += (int64_t)gridDim.x * blockDim.x)
    {
        int k = -1;
        if (!prefix || (prefix[i] > above && (top || prefix[i] <= size)))
        {
            int sub;
            k = cell_of(sp, L, qf, nq, i, sub);
            atomicAdd(&count[k], 1);
        }
        key[i] = k;
    }
}

template <int KIND, int MAXF, int K_KEEP>
__global__ void __launch_bounds__(128, 8) knn_cell_kernel(const __grid_constant__ BoxCellArgs ci,
                                                          const __grid_constant__ SpaceParams sp, const float *qf,
                                                          int64_t nq, const int *qorder, const int *qcount, int k,
                                                          const int64_t *prefix, const __grid_constant__ KnnOut out)
{
    extern __shared__ float table[];  // per warp: nA + nB sums
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t qs = (int64_t)blockIdx.x * 4 + warp;
    if (qs >= *qcount)
        return;
    const int64_t qi = qorder[qs];
    const float inf = __int_as_float(0x7f800000);
    float q[MAXF];
#pragma unroll
    for (int f = 0; f < MAXF; ++f)
        q[f] = f < sp.dim ? qf[(int64_t)f * nq + qi] : 0.f;
    const int limit = prefix ? (int)min((int64_t)INT_MAX, prefix[qi]) : INT_MAX;
    float *A = table + warp * (ci.nA + ci.nB), *B = A + ci.nA;
    const int L = ci.L;
    // squared distance of coordinate d's value x from level l's interval: the grid's, widened against the rounding
    // of the level, the outermost ones reaching the data's extremes (elements outside the bounds are in them)
    auto level_d2 = [&](int d, float x, int l) {
        float lo, hi;
        cell_range(sp, d, lo, hi);
        // the level of a value is off by up to 2^-22 L of a level, the ends by a few roundings of the bounds
        const float w = (hi - lo) / (float)L, pad = 1e-3f * w + 1e-6f * fmaxf(fabsf(lo), fabsf(hi));
        float a = lo + (float)l * w - pad, b = lo + (float)(l + 1) * w + pad;
        if (l == 0)
            a = fminf(a, ci.extent[2 * d]);
        if (l == L - 1 || !(hi > lo))  // bounds that fix the coordinate: every value is in level 0
            b = fmaxf(b, ci.extent[2 * d + 1]);
        float s;
        if constexpr (KIND == GBO_SPACE_WRAP_L2)
            s = wrap_gap(x, a, b);
        else
            s = fmaxf(fmaxf(a - x, x - b), 0.f);
        return s * s;
    };
    // T[i + l size] = T[i] + (level l of the next coordinate), from the back: entries 0 .. size - 1 are read by
    // all and replaced last
    auto tabulate = [&](float *T, int d0, int d1) {
        if (lane == 0)
            T[0] = 0.f;
        __syncwarp();
        int size = 1;
        for (int d = d0; d < d1; ++d)
        {
            float x = 0.f;
#pragma unroll
            for (int f = 0; f < MAXF; ++f)
                if (f == d)
                    x = q[f];
            const int total = size * L;
            for (int e0 = (total - 1) / 32 * 32; e0 >= 0; e0 -= 32)
            {
                const int e = e0 + lane;
                float v = 0.f;
                if (e < total)
                {
                    const int l = e / size;
                    v = T[e - l * size] + level_d2(d, x, l);
                }
                __syncwarp();
                if (e < total)
                    T[e] = v;
                __syncwarp();
            }
            size = total;
        }
    };
    tabulate(A, 0, ci.dA);
    tabulate(B, ci.dA, sp.dim);
    WarpList<K_KEEP> list;
    list.init();
    float T = inf;
    auto tighten = [&]() {
        const float dk = list.at(k - 1);
        if (dk < inf)
        {
            const float r = sqrtf(dk) + 2.f * out.nn.eps32;
            T = fminf(T, r * r * (1.0f + 1e-5f));
        }
    };
    // a query that is not finite has no neighbours, and its bounds are 0: nothing is searched
    bool finite = true;
#pragma unroll
    for (int f = 0; f < MAXF; ++f)
        finite = finite && fabsf(q[f]) < inf;
    auto scan_chunk = [&](int p0, int s1) {
        const int p = p0 + lane;
        float d = inf;
        int key = -1;
        if (p < s1)
        {
            key = ci.skey[p];
            const float4 a = ci.pts8[2 * (int64_t)p];
            float pf[8] = {a.x, a.y, a.z, a.w, 0.f, 0.f, 0.f, 0.f};
            if (MAXF > 4)
            {
                const float4 b = ci.pts8[2 * (int64_t)p + 1];
                pf[4] = b.x;
                pf[5] = b.y;
                pf[6] = b.z;
                pf[7] = b.w;
            }
            d = key < limit ? box_dist2<KIND, MAXF>(pf, q, MAXF) : inf;
        }
        unsigned m = __ballot_sync(0xffffffffu, d < list.last() && d <= T);
        while (m)
        {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const float dc = __shfl_sync(0xffffffffu, d, src);
            const int kc = __shfl_sync(0xffffffffu, key, src);
            if (dc < list.last())
                list.insert(dc, kc, lane);
        }
    };
    auto scan_cell = [&](int c) {
        const int s0 = ci.start[c << ci.bits], s1 = ci.start[(c + 1) << ci.bits];
        if (s0 == s1)
            return;
        const int chunks = (s1 - s0 + 31) / 32, ch0 = ci.cstart[c];
        for (int b = 0; b < chunks; b += 32)
        {
            const int ch = b + lane;
            float lb = inf;
            if (ch < chunks && ci.kmin[ch0 + ch] < limit)
                lb = bcell_lb<KIND, MAXF>(ci.box + 4 * (int64_t)(ch0 + ch), q, sp.dim);
            unsigned m = __ballot_sync(0xffffffffu, lb < fminf(T, list.last()));
            while (m)
            {
                const int src = __ffs(m) - 1;
                m &= m - 1;
                if (__shfl_sync(0xffffffffu, lb, src) < fminf(T, list.last()))
                {
                    scan_chunk(s0 + 32 * (b + src), s1);
                    tighten();
                }
            }
        }
    };
    int own = 0, h;
#pragma unroll
    for (int d = MAXF - 1; d >= 0; --d)
        if (d < sp.dim)
            own = own * L + cell_level(sp, L, d, q[d], h);
    if (finite)
        scan_cell(own);
    // rings of a tenth and a third of the threshold's square, then the rest (an infinite T: all at once)
    float from = -1.f;
#pragma unroll 1
    for (int ring = 0; finite && ring < 3; ++ring)
    {
        const float cut = fminf(T, list.last());
        const float to = ring == 2 || !(cut < inf) ? inf : (ring == 0 ? 0.1f : 0.33f) * cut;
        for (int j = 0; j < ci.nB; ++j)
        {
            const float tb = B[j] * (1.0f - 1e-5f), near = fminf(to, fminf(T, list.last()));
            if (!(tb < near))
                continue;
            for (int i0 = 0; i0 < ci.nA; i0 += 32)
            {
                const int i = i0 + lane;
                const float lb = i < ci.nA ? (A[i] + B[j]) * (1.0f - 1e-5f) : inf;
                const float now = fminf(to, fminf(T, list.last()));
                unsigned m = __ballot_sync(0xffffffffu, lb >= from && lb < now);
                while (m)
                {
                    const int src = __ffs(m) - 1;
                    m &= m - 1;
                    const int c = j * ci.nA + i0 + src;
                    if (c != own && __shfl_sync(0xffffffffu, lb, src) < fminf(T, list.last()))
                        scan_cell(c);
                }
            }
        }
        if (to == inf)
            break;
        from = fmaxf(from, to);  // T may have shrunk past the ring: no cell is visited twice
    }
    warp_finish<KIND, MAXF, K_KEEP>(out, sp, qi, k, list, lane);
}

int cell_levels(int dim, int64_t n)
{
    // about 40 elements per cell, at most 65536 cells (1024 on one coordinate)
    int L = 2;
    while (true)
    {
        int64_t c = 1;
        for (int d = 0; d < dim; ++d)
            c *= L + 1;
        if (c > (dim == 1 ? 1024 : 65536) || c * 40 > n)
            break;
        ++L;
    }
    return L;
}

static int grid_for(const LaunchCfg &lc, int64_t n)
{
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)lc.sm_count * 8));
}

static void launch_scan(const LaunchCfg &lc, const int *count, int n, int *sums, int *start, int *fill)
{
    const int blocks = (n + kScanBlock - 1) / kScanBlock;
    scan_sums_kernel<<<blocks, 1024, 0, lc.stream>>>(count, n, sums);
    scan_kernel<<<blocks, 1024, 0, lc.stream>>>(count, n, sums, start, fill);
}

BoxCellShape cell_shape(int dim, int64_t n)
{
    BoxCellShape s;
    s.L = cell_levels(dim, n);
    s.C = 1;
    for (int d = 0; d < dim; ++d)
        s.C *= s.L;
    s.bits = 0;
    while (s.bits < dim && ((int64_t)s.C << (s.bits + 1)) <= kSubMax)
        ++s.bits;
    s.dA = (dim + 1) / 2;
    s.nA = 1;
    for (int d = 0; d < s.dA; ++d)
        s.nA *= s.L;
    s.nB = s.C / s.nA;
    return s;
}

void launch_cell_build(const LaunchCfg &lc, const NNArgs &nn, const SpaceParams &sp, const BoxCellShape &s, int *key,
                       int *count, int *sums, int *fill, const BoxCellArgs &ci)
{
    const int sub = s.C << s.bits;
    int *start = const_cast<int *>(ci.start), *cstart = const_cast<int *>(ci.cstart), *skey = const_cast<int *>(ci.skey);
    int *extent = (int *)const_cast<float *>(ci.extent);
    cudaMemsetAsync(count, 0, (size_t)sub * sizeof(int), lc.stream);
    cell_clear_kernel<<<1, 32, 0, lc.stream>>>(extent);
    cell_assign_kernel<<<grid_for(lc, nn.size), 256, 0, lc.stream>>>(sp, s.L, s.bits, nn.feat32, nn.cap, nn.alive,
                                                                     nn.size, key, count, extent);
    launch_scan(lc, count, sub, sums, start, fill);
    cell_scatter_kernel<<<grid_for(lc, nn.size), 256, 0, lc.stream>>>(key, nn.size, fill, skey);
    cell_extent_kernel<<<1, 32, 0, lc.stream>>>(extent);
    cell_chunks_kernel<<<(s.C + 255) / 256, 256, 0, lc.stream>>>(start, s.bits, s.C, count);
    launch_scan(lc, count, s.C, sums, cstart, fill);
    cell_fill_kernel<<<grid_for(lc, (int64_t)s.C * 32), 256, 0, lc.stream>>>(
        nn.feat32, nn.cap, sp.dim, start, s.bits, s.C, cstart, skey, const_cast<float4 *>(ci.pts8),
        const_cast<float4 *>(ci.box), const_cast<int *>(ci.kmin));
    for (int i = 0; i < 10; ++i)
        note_launch();
}

template <int KIND, int MAXF, int K_KEEP>
static void launch_cell_t(const LaunchCfg &lc, const BoxCellArgs &ci, const SpaceParams &sp, const float *qf, int64_t nq,
                          const int *qorder, const int *qcount, int k, const int64_t *prefix, const KnnOut &out)
{
    const size_t smem = (size_t)4 * (ci.nA + ci.nB) * sizeof(float);
    knn_cell_kernel<KIND, MAXF, K_KEEP><<<(int)((nq + 3) / 4), 128, smem, lc.stream>>>(ci, sp, qf, nq, qorder, qcount, k,
                                                                                      prefix, out);
    note_launch();
}

void launch_knn_cells(const LaunchCfg &lc, const BoxCellArgs &ci, const SpaceParams &sp, const float *qf, int64_t nq,
                      const int64_t *prefix, int64_t above, bool top, int k, int *qkey, int *qcount, int *qstart,
                      int *qfill, int *qorder, int *sums, const KnnOut &out)
{
    cudaMemsetAsync(qcount, 0, (size_t)ci.C * sizeof(int), lc.stream);
    cell_query_kernel<<<grid_for(lc, nq), 256, 0, lc.stream>>>(sp, ci.L, qf, nq, prefix, above, out.nn.size, top, qkey,
                                                               qcount);
    launch_scan(lc, qcount, ci.C, sums, qstart, qfill);
    cell_scatter_kernel<<<grid_for(lc, nq), 256, 0, lc.stream>>>(qkey, nq, qfill, qorder);
    for (int i = 0; i < 4; ++i)
        note_launch();
#define GBO_CELL(KIND, MAXF, KK) launch_cell_t<KIND, MAXF, KK>(lc, ci, sp, qf, nq, qorder, qstart + ci.C, k, prefix, out)
#define GBO_CELL_K(KIND, MAXF)                                                                                         \
    do                                                                                                                \
    {                                                                                                                 \
        if (k <= 12)                                                                                                  \
            GBO_CELL(KIND, MAXF, 16);                                                                                 \
        else if (k <= 20)                                                                                             \
            GBO_CELL(KIND, MAXF, 24);                                                                                 \
        else if (k <= 40)                                                                                             \
            GBO_CELL(KIND, MAXF, 48);                                                                                 \
        else                                                                                                          \
            GBO_CELL(KIND, MAXF, 72);                                                                                 \
    } while (0)
    if (sp.kind == GBO_SPACE_WRAP_L2 && sp.dim <= 4)
        GBO_CELL_K(GBO_SPACE_WRAP_L2, 4);
    else if (sp.kind == GBO_SPACE_WRAP_L2)
        GBO_CELL_K(GBO_SPACE_WRAP_L2, 8);
    else if (sp.dim <= 4)
        GBO_CELL_K(GBO_SPACE_REAL_VECTOR, 4);
    else
        GBO_CELL_K(GBO_SPACE_REAL_VECTOR, 8);
#undef GBO_CELL_K
#undef GBO_CELL
}

}  // namespace gbo
