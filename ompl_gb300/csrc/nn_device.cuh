// Device helpers shared by the nearest-neighbour kernels: element and query loads, the (distance, key)
// order and the FP32 metrics over features.
#pragma once
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

}  // namespace gbo
