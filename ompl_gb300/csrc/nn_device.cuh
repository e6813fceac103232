// Device helpers shared by the nearest-neighbour kernels: element and query loads, the (distance, key)
// order and the FP32 metrics over features.
#pragma once
#include <climits>

#include "kernels_nn.cuh"

namespace gbo
{

template <int MAXD>
__device__ __forceinline__ void load_point(const double *pts, int64_t cap, int dim, int64_t key, double *x)
{
#pragma unroll
    for (int d = 0; d < MAXD; ++d)
        x[d] = d < dim ? pts[(int64_t)d * cap + key] : 0.0;
}

template <int MAXD>
__device__ __forceinline__ void load_query(const StatesView &v, int64_t i, int dim, double *x)
{
#pragma unroll
    for (int d = 0; d < MAXD; ++d)
        x[d] = d < dim ? v(i, d) : 0.0;
}

__device__ __forceinline__ bool less_dk(double a, int64_t ka, double b, int64_t kb)
{
    return a < b || (a == b && ka < kb);
}

// Element features: REAL_VECTOR / WRAP_L2 / SO2: the coordinates (F = dim); KINEMATIC_CHAIN: the
// cumulative link-direction sums interleaved (X_1, Y_1, ..., X_n, Y_n), F = 2 dim, so that
// distance = L * sum_i |(X_i(a) - X_i(b), Y_i(a) - Y_i(b))|. All indices below are compile-time.
template <int KIND, int MAXF>
__device__ __forceinline__ float box_dist2(const float *a, const float *b, int dim)
{
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < MAXF; ++i)
        if (i < dim)
        {
            float d = a[i] - b[i];
            if constexpr (KIND == GBO_SPACE_WRAP_L2 || KIND == GBO_SPACE_SO2)
            {
                d = fabsf(d);
                d = fminf(d, 6.28318530717958647692f - d);
            }
            s = fmaf(d, d, s);
        }
    return s;
}

__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <int MAXF>
__device__ __forceinline__ float chain_dist32(const float *a, const float *b, int dim)
{
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < MAXF / 2; ++i)
        if (i < dim)
        {
            const float dx = a[2 * i] - b[2 * i], dy = a[2 * i + 1] - b[2 * i + 1];
            s += sqrt_approx(fmaf(dx, dx, dy * dy));
        }
    return s;
}

// The kept list spread over a warp: entry j = 32 s + lane in slot s of the lane (S = K_KEEP / 32
// rounded up slots), ascending, unused entries +inf / -1.
template <int K_KEEP>
struct WarpList
{
    static constexpr int S = (K_KEEP + 31) / 32;
    float d[S];
    int k[S];
    __device__ __forceinline__ void init()
    {
#pragma unroll
        for (int s = 0; s < S; ++s)
        {
            d[s] = __int_as_float(0x7f800000);
            k[s] = -1;
        }
    }
    // entry j of the list, in every lane
    __device__ __forceinline__ float at(int j) const
    {
        float v = d[0];
#pragma unroll
        for (int s = 1; s < S; ++s)
            if (j >> 5 == s)
                v = d[s];
        return __shfl_sync(0xffffffffu, v, j & 31);
    }
    __device__ __forceinline__ float last() const { return at(K_KEEP - 1); }
    // inserts (dd, kk) after the entries with a distance <= dd (those kept earlier stay first)
    __device__ __forceinline__ void insert(float dd, int kk, int lane)
    {
        int pos = 0;
#pragma unroll
        for (int s = 0; s < S; ++s)
            pos += __popc(__ballot_sync(0xffffffffu, 32 * s + lane < K_KEEP && d[s] <= dd));
        if (pos >= K_KEEP)
            return;
        float up_d[S];
        int up_k[S];
#pragma unroll
        for (int s = 0; s < S; ++s)
        {
            up_d[s] = __shfl_up_sync(0xffffffffu, d[s], 1);
            up_k[s] = __shfl_up_sync(0xffffffffu, k[s], 1);
            if (s > 0)
            {
                // lane 0 of slot s takes entry 32 s - 1: lane 31 of slot s - 1
                const float cd = __shfl_sync(0xffffffffu, d[s - 1], 31);
                const int ck = __shfl_sync(0xffffffffu, k[s - 1], 31);
                if (lane == 0)
                {
                    up_d[s] = cd;
                    up_k[s] = ck;
                }
            }
        }
#pragma unroll
        for (int s = 0; s < S; ++s)
        {
            const int j = 32 * s + lane;
            if (j >= pos && j < K_KEEP)
            {
                d[s] = j == pos ? dd : up_d[s];
                k[s] = j == pos ? kk : up_k[s];
            }
        }
    }
};

// Where a search's results go, and the index they are decided on
struct KnnOut
{
    NNArgs nn;
    StatesView qv;
    int64_t *idx;
    double *dist;
    unsigned long long *fb_list, *fb_n;
    RunCounters *ctr;
};

// Decides query qi's result from the kept list of a warp's search, in FP64: every entry within 2 * eps of the
// k-th FP32 distance is re-evaluated with the reference-order distance, one entry per lane, and ranked by
// (FP64 distance, key). A full list whose last entry lies inside that band may have dropped elements of it: the
// query goes to the FP64 scan.
template <int KIND, int MAXD, int K_KEEP>
__device__ __forceinline__ void warp_finish(const KnnOut &out, const SpaceParams &sp, int64_t qi, int k,
                                            const WarpList<K_KEEP> &L, int lane)
{
    constexpr int S = WarpList<K_KEEP>::S;
    const float eps = out.nn.eps32, kth = L.at(k - 1);
    float band;
    if constexpr (KIND == GBO_SPACE_KINEMATIC_CHAIN)
        band = kth + 2.f * eps;
    else
    {
        const float r = sqrtf(kth) + 2.f * eps;
        band = r * r * (1.0f + 1e-6f);
    }
    const int last_key = __shfl_sync(0xffffffffu, L.k[S - 1], (K_KEEP - 1) & 31);
    if (last_key >= 0 && !(L.last() > band))
    {
        if (lane == 0)
        {
            out.fb_list[atomicAdd(out.fb_n, 1ull)] = (unsigned long long)qi;
            atomicAdd(&out.ctr->fallbacks, 1ull);
        }
        return;
    }
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    double q64[MAXD], d64[S];
    load_query<MAXD>(out.qv, qi, sp.dim, q64);
    int key[S], rank[S];
    float max_err = 0.f;
    unsigned kept = 0;
#pragma unroll
    for (int s = 0; s < S; ++s)
    {
        d64[s] = inf;
        key[s] = INT_MAX;
        rank[s] = 0;
        if (32 * s + lane < K_KEEP && L.k[s] >= 0 && L.d[s] <= band)
        {
            double x[MAXD];
            load_point<MAXD>(out.nn.pts64, out.nn.cap, sp.dim, L.k[s], x);
            key[s] = L.k[s];
            d64[s] = distance64<MAXD, false>(sp, x, q64);
            const float d32 = KIND == GBO_SPACE_KINEMATIC_CHAIN ? L.d[s] : sqrtf(L.d[s]);
            max_err = fmaxf(max_err, fabsf((float)(d64[s] - (double)d32)));
            ++kept;
        }
    }
    kept = __reduce_add_sync(0xffffffffu, kept);
    max_err = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(max_err)));
    // the band's entries are the first `kept` of the list
#pragma unroll
    for (int t = 0; t < S; ++t)
        for (int l = 0; l < 32 && 32 * t + l < (int)kept; ++l)
        {
            const double d = __shfl_sync(0xffffffffu, d64[t], l);
            const int kk = __shfl_sync(0xffffffffu, key[t], l);
#pragma unroll
            for (int s = 0; s < S; ++s)
                rank[s] += less_dk(d, kk, d64[s], key[s]);
        }
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (key[s] != INT_MAX && rank[s] < k)
        {
            out.idx[qi * k + rank[s]] = key[s];
            if (out.dist)
                out.dist[qi * k + rank[s]] = d64[s];
        }
    for (int r = (int)kept + lane; r < k; r += 32)
    {
        out.idx[qi * k + r] = -1;
        if (out.dist)
            out.dist[qi * k + r] = inf;
    }
    if (lane == 0)
    {
        atomicAdd(&out.ctr->rechecked, (unsigned long long)kept);
        if (max_err > 0.f)
            atomicMax(&out.ctr->max_err_bits, __float_as_uint(max_err));
    }
}

}  // namespace gbo
