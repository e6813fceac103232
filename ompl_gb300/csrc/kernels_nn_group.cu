// nearestK in one launch for batches that the cell searches do not take: small query batches, small
// indexes, a planner's single query.
//
//   knn_group_kernel  a CTA (or a cluster of CTAs that split the elements) answers QG queries. The FP32
//                     distances of every element are computed once, coalesced, and only the minimum of
//                     each group of 32 m consecutive elements is kept. The K-th smallest of the
//                     minima of disjoint buckets of groups bounds the K-th smallest distance from above
//                     (T), so only groups whose minimum is at most T are read again, and their elements
//                     with a distance of at most T are the candidates: K plus a few, whatever the index's
//                     size. One warp then re-evaluates the candidates of the guard band in FP64, one per
//                     lane, and ranks them by (FP64 distance, key).
//
// A thread-per-query scan with kept lists (knn_scan_kernel + knn_finish_kernel) gives a small batch one
// thread per query and chunk, stops a warp for every lane's insertion and evaluates a query's FP64
// distances one after another. Here a query has 256 threads or more, nothing is inserted, and the finish
// runs side by side. Per call: 2,000 elements, one query, k = 10: 300 -> 33 us (the host's share);
// 60,000 wrapped 7-D elements, 500 queries: 814 -> 110 us; 10,000 planar points, 1,000 queries: 823 ->
// 44 us. Bound: at 500 queries the kernel issues on 36% of its cycles (57 warp instructions per 32
// pairs; the waves of CTAs are short); DRAM and L2 are below 10%.
#include <algorithm>
#include <climits>
#include <cstdint>

#include <cooperative_groups.h>

#include "nn_device.cuh"

namespace cg = cooperative_groups;

namespace gbo
{

namespace
{
constexpr float kInf = __builtin_huge_valf();

// per CTA: group minima a query can keep, buckets of groups, candidates a query can hold
template <int QG>
struct GroupCfg
{
    static constexpr int kGroups = QG == 1 ? 1024 : 512;
    static constexpr int kCand = QG == 1 ? 1024 : 256;
};
constexpr int kBuckets = 160;

template <int QG>
struct GroupSmem
{
    float gmin[QG][GroupCfg<QG>::kGroups];
    float bucket[QG][kBuckets];
    double c64[QG][GroupCfg<QG>::kCand];
    float cd[QG][GroupCfg<QG>::kCand];
    int ck[QG][GroupCfg<QG>::kCand];
    int cnt[QG];
    float T[QG];
};

// Smallest of a warp's non-negative (or infinite) values: their bits order like unsigned integers.
__device__ __forceinline__ float warp_min(float v)
{
    return __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(v)));
}

// rk[s]: how many of the 32 S values before v[s] of this lane in (value, position 32 s + lane) order
template <int S>
__device__ __forceinline__ void bucket_ranks(const float *v, int *rk, int lane)
{
#pragma unroll
    for (int t = 0; t < S; ++t)
#pragma unroll 8
        for (int l = 0; l < 32; ++l)
        {
            const float o = __shfl_sync(0xffffffffu, v[t], l);
#pragma unroll
            for (int s = 0; s < S; ++s)
                rk[s] += o < v[s] || (o == v[s] && (t < s || (t == s && l < lane)));
        }
}

// FP32 distance over all MAXF features (those past the space's are zero on both sides), squared for the
// box kinds.
template <int KIND, int MAXF>
__device__ __forceinline__ float group_dist(const float *a, const float *b, float link)
{
    if constexpr (KIND == GBO_SPACE_KINEMATIC_CHAIN)
        return chain_dist32<MAXF>(a, b, MAXF / 2) * link;
    else
        return box_dist2<KIND, MAXF>(a, b, MAXF);
}
// Query q's FP32 features, as features_kernel forms the elements'
template <int KIND, int MAXF>
__device__ __forceinline__ void query_features(const SpaceParams &sp, const StatesView &qv, int64_t q, float *qf)
{
    if constexpr (KIND == GBO_SPACE_KINEMATIC_CHAIN)
    {
        double theta = 0.;
        float X = 0.f, Y = 0.f;
#pragma unroll
        for (int d = 0; d < MAXF / 2; ++d)
            if (d < sp.dim)
            {
                theta = dadd(theta, qv(q, d));
                float c, s;
                dir32(theta, c, s);
                X += c;
                Y += s;
                qf[2 * d] = X;
                qf[2 * d + 1] = Y;
            }
    }
    else
    {
#pragma unroll
        for (int d = 0; d < MAXF; ++d)
            if (d < sp.dim)
                qf[d] = (float)qv(q, d);
    }
}

// Element `key`'s features: coalesced float4 planes, as many as the space's features fill (the index has
// no more), zero past them
template <int KIND, int MAXF>
__device__ __forceinline__ void element_features(const NNArgs &nn, const SpaceParams &sp, int key, float *pf)
{
    const int planes = ((KIND == GBO_SPACE_KINEMATIC_CHAIN ? 2 * sp.dim : sp.dim) + 3) / 4;
#pragma unroll
    for (int j = 0; j < (MAXF + 3) / 4; ++j)
    {
        const float4 v = j < planes ? nn.feat4[(int64_t)j * nn.cap + key] : make_float4(0.f, 0.f, 0.f, 0.f);
        pf[4 * j] = v.x;
        pf[4 * j + 1] = v.y;
        if (4 * j + 2 < MAXF)
        {
            pf[4 * j + 2] = v.z;
            pf[4 * j + 3] = v.w;
        }
    }
}
}  // namespace

// K: list length that bounds the band (knn_keep(k)); buckets: a multiple of 32, at least 2 K.
// nn.alive may be null: every element is present.
template <int KIND, int MAXF, int QG, int kThreads>
__global__ void __launch_bounds__(kThreads, QG == 4 ? (MAXF <= 8 ? 768 : 512) / kThreads : 2)
    knn_group_kernel(NNArgs nn, SpaceParams sp, StatesView qv, int64_t nq, int k, int K, int buckets,
                     const int64_t *prefix, int64_t max_limit, int64_t *idx, double *dist,
                     unsigned long long *fb_list, unsigned long long *fb_n, RunCounters *ctr)
{
    constexpr int MAXD = KIND == GBO_SPACE_KINEMATIC_CHAIN ? MAXF / 2 : MAXF;
    constexpr int kWarps = kThreads / 32;
    constexpr int GC = GroupCfg<QG>::kGroups, CC = GroupCfg<QG>::kCand;
    __shared__ GroupSmem<QG> sm;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), CS = (int)cluster.num_blocks();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t q0 = (int64_t)(blockIdx.x / CS) * QG;
    const float link = (float)sp.link;
    // queries of another launch (the same ones in every CTA of a cluster)
    unsigned skip = 0;
    if (prefix && max_limit < INT64_MAX)
    {
        bool any = false;
        for (int g = 0; g < QG && q0 + g < nq; ++g)
        {
            const bool theirs = prefix[q0 + g] > max_limit;
            skip |= theirs ? 1u << g : 0u;
            any |= !theirs;
        }
        if (!any)
            return;
    }

    // queries: their FP32 features (as features_kernel forms them) and the number of elements they see
    float qf[QG][MAXF];
    int lim[QG], top = 0;
#pragma unroll
    for (int g = 0; g < QG; ++g)
    {
        const int64_t q = q0 + g;
        int64_t l = 0;
        if (q < nq)
        {
            l = nn.size;
            if (prefix)
                l = skip >> g & 1u ? 0 : min(l, prefix[q]);
        }
        lim[g] = (int)max(l, (int64_t)0);
        top = max(top, lim[g]);
#pragma unroll
        for (int f = 0; f < MAXF; ++f)
            qf[g][f] = 0.f;
        if (q < nq)
            query_features<KIND, MAXF>(sp, qv, q, qf[g]);
    }
    if (threadIdx.x < QG)
        sm.cnt[threadIdx.x] = 0;

    // groups of 32 m elements, each computed by one warp. Small indexes: a quarter warp's 8 elements form
    // a group (sub), so that there are enough groups to bound the K-th distance; all are read again.
    const int W = kWarps * CS, gw = rank * kWarps + warp;
    const bool sub = top < 32 * buckets && top <= 8 * GC;
    int m = top < 256 * buckets ? 1 : (top < 768 * buckets ? 4 : 8);
    while ((top + 32 * m * W - 1) / (32 * m * W) * kWarps > GC)
        m *= 2;
    auto load = [&](int key, float *pf) { element_features<KIND, MAXF>(nn, sp, key, pf); };
    {
        int local = warp;
        for (int g0 = gw * 32 * m; g0 < top; g0 += W * 32 * m, local += kWarps)
        {
            float mn[QG];
#pragma unroll
            for (int g = 0; g < QG; ++g)
                mn[g] = kInf;
            const int g1 = min(g0 + 32 * m, top);
            int key = g0 + lane;
            auto fold = [&](const float *pf, int at, bool here) {
#pragma unroll
                for (int g = 0; g < QG; ++g)
                {
                    const float d = group_dist<KIND, MAXF>(pf, qf[g], link);
                    mn[g] = here && at < lim[g] ? fminf(mn[g], d) : mn[g];
                }
            };
            constexpr int U = MAXF <= 8 ? (QG == 1 ? 4 : 2) : 1;
            for (; key + 32 * (U - 1) < g1; key += 32 * U)
            {
                float pf[U][MAXF];
                bool here[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                {
                    load(key + 32 * u, pf[u]);
                    here[u] = !nn.alive || nn.alive[key + 32 * u];
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    fold(pf[u], key + 32 * u, here[u]);
            }
            for (; key < g1; key += 32)
            {
                float pf[MAXF];
                load(key, pf);
                fold(pf, key, !nn.alive || nn.alive[key]);
            }
            if (sub)
            {
                // 8-lane minima: four groups per warp iteration
#pragma unroll
                for (int g = 0; g < QG; ++g)
                {
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1)
                        mn[g] = fminf(mn[g], __shfl_xor_sync(0xffffffffu, mn[g], o));
                    if ((lane & 7) == 0)
                        sm.gmin[g][4 * local + (lane >> 3)] = mn[g];
                }
            }
            else
            {
#pragma unroll
                for (int g = 0; g < QG; ++g)
                {
                    const float v = warp_min(mn[g]);
                    if (lane == 0)
                        sm.gmin[g][local] = v;
                }
            }
        }
    }
    __syncthreads();

    // bucket minima over the groups of the whole cluster: group number (over the cluster) modulo `buckets`
    const int rounds = (top + 32 * m * W - 1) / (32 * m * W), per = sub ? 4 : 1, groups = rounds * kWarps * per;
    for (int b = threadIdx.x; b < QG * buckets; b += kThreads)
        sm.bucket[b / buckets][b % buckets] = kInf;
    __syncthreads();
    for (int i = threadIdx.x; i < QG * groups; i += kThreads)
    {
        const int g = i / groups, l = i - g * groups;
        // local group l: round l / (8 per), warp (l / per) % 8
        const int round = l / (kWarps * per), w = (l / per) % kWarps, e = l % per;
        const int64_t first = ((int64_t)round * W + rank * kWarps + w) * 32 * m;
        if (first < top)
        {
            const int id = (int)(((int64_t)round * W + rank * kWarps + w) * per + e);
            atomicMin((unsigned *)&sm.bucket[g][id % buckets], __float_as_uint(sm.gmin[g][l]));
        }
    }
    cluster.sync();
    // T: the K-th smallest bucket minimum (infinite when fewer than K buckets hold an element)
    if (warp < QG)
    {
        const int g = warp;
        float v[kBuckets / 32];
        int rk[kBuckets / 32];
#pragma unroll
        for (int s = 0; s < kBuckets / 32; ++s)
        {
            v[s] = kInf;
            rk[s] = 0;
            if (32 * s < buckets)
                for (int r = 0; r < CS; ++r)
                    v[s] = fminf(v[s], cluster.map_shared_rank(&sm, r)->bucket[g][32 * s + lane]);
        }
        // ranks, ties by bucket: buckets <= 64 need two of the slots
        if (buckets <= 64)
            bucket_ranks<2>(v, rk, lane);
        else
            bucket_ranks<kBuckets / 32>(v, rk, lane);
#pragma unroll
        for (int s = 0; s < kBuckets / 32; ++s)
            if (32 * s < buckets && rk[s] == K - 1)
                sm.T[g] = v[s];
    }
    __syncthreads();

    // second read: elements within T of the groups whose minimum is, appended to the query's list in the
    // CTA that finishes it (query g: CTA g mod CS)
#pragma unroll
    for (int g = 0; g < QG; ++g)
    {
        const float T = sm.T[g];
        GroupSmem<QG> *own = cluster.map_shared_rank(&sm, g % CS);
        int local = warp;
        for (int g0 = gw * 32 * m; g0 < lim[g]; g0 += W * 32 * m, local += kWarps)
        {
            if (!sub && !(sm.gmin[g][local] <= T))
                continue;
            const int g1 = min(g0 + 32 * m, lim[g]);
            for (int key = g0 + lane; key < g1; key += 32)
            {
                float pf[MAXF];
                load(key, pf);
                const float d = group_dist<KIND, MAXF>(pf, qf[g], link);
                if (d <= T && d < kInf && (!nn.alive || nn.alive[key]))
                {
                    const int pos = atomicAdd(&own->cnt[g], 1);
                    if (pos < CC)
                    {
                        own->cd[g][pos] = d;
                        own->ck[g][pos] = key;
                    }
                }
            }
        }
    }
    cluster.sync();

    // finish: warp w of the owning CTA takes query g with g / CS == w
    const int g = warp * CS + rank;
    if (g >= QG || q0 + g >= nq || (skip >> g & 1u))
        return;
    const int64_t qi = q0 + g;
    const float T = sm.T[g], eps = nn.eps32;
    const int n = sm.cnt[g];
    bool overflow = n > CC;
    float band = kInf;
    if (!overflow && n >= k)
    {
        // the k-th smallest FP32 distance
        float kth = 0.f;
        for (int i = lane; i < n; i += 32)
        {
            const float d = sm.cd[g][i];
            int r = 0;
#pragma unroll 8
            for (int j = 0; j < n; ++j)
            {
                const float o = sm.cd[g][j];
                r += o < d || (o == d && j < i);
            }
            if (r == k - 1)
                kth = d;
        }
        kth = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(kth)));
        if constexpr (KIND == GBO_SPACE_KINEMATIC_CHAIN)
            band = kth + 2.f * eps;
        else
        {
            const float r = sqrtf(kth) + 2.f * eps;
            band = r * r * (1.0f + 1e-6f);
        }
        overflow = !(band <= T);  // elements of the band may lie beyond the candidates
    }
    else if (!overflow)
        overflow = T < kInf;  // fewer than k candidates under a finite bound: never, by T's definition
    if (overflow)
    {
        if (lane == 0)
        {
            fb_list[atomicAdd(fb_n, 1ull)] = (unsigned long long)qi;
            atomicAdd(&ctr->fallbacks, 1ull);
        }
        return;
    }
    // FP64 distances of the band, one candidate per lane: the band's elements move to the front of the list
    double q64[MAXD];
    load_query<MAXD>(qv, qi, sp.dim, q64);
    const double inf64 = __longlong_as_double(0x7ff0000000000000ll);
    int kept = 0;
    float max_err = 0.f;
    for (int i0 = 0; i0 < n; i0 += 32)
    {
        const int i = i0 + lane;
        const float d32 = i < n ? sm.cd[g][i] : kInf;
        const int key = i < n ? sm.ck[g][i] : 0;
        const bool in = i < n && d32 <= band;
        const unsigned mask = __ballot_sync(0xffffffffu, in);
        if (in)
        {
            const int at = kept + __popc(mask & ((1u << lane) - 1u));
            sm.cd[g][at] = d32;
            sm.ck[g][at] = key;
        }
        kept += __popc(mask);
        __syncwarp();
    }
    for (int i = lane; i < kept; i += 32)
    {
        double x[MAXD];
        load_point<MAXD>(nn.pts64, nn.cap, sp.dim, sm.ck[g][i], x);
        const double d = distance64<MAXD, false>(sp, x, q64);
        sm.c64[g][i] = d;
        const float d32 = sm.cd[g][i], f = KIND == GBO_SPACE_KINEMATIC_CHAIN ? d32 : sqrtf(d32);
        max_err = fmaxf(max_err, fabsf((float)(d - (double)f)));
    }
    max_err = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(max_err)));
    __syncwarp();
    for (int i = lane; i < kept; i += 32)
    {
        const int key = sm.ck[g][i];
        const double d = sm.c64[g][i];
        int r = 0;
#pragma unroll 4
        for (int j = 0; j < kept; ++j)
            r += less_dk(sm.c64[g][j], sm.ck[g][j], d, key);
        if (r < k)
        {
            idx[qi * k + r] = key;
            if (dist)
                dist[qi * k + r] = d;
        }
    }
    for (int r = kept + lane; r < k; r += 32)
    {
        idx[qi * k + r] = -1;
        if (dist)
            dist[qi * k + r] = inf64;
    }
    if (lane == 0)
    {
        atomicAdd(&ctr->rechecked, (unsigned long long)kept);
        if (max_err > 0.f)
            atomicMax(&ctr->max_err_bits, __float_as_uint(max_err));
    }
}

namespace
{
template <int KIND, int MAXF, int QG, int kThreads>
void launch_group_t(const LaunchCfg &lc, const NNArgs &nn, const SpaceParams &sp, StatesView qv, int64_t nq, int k,
                    int K, int CS, const int64_t *prefix, int64_t max_limit, int64_t *idx, double *dist,
                    unsigned long long *fb_list, unsigned long long *fb_n, RunCounters *ctr)
{
    const int buckets = std::min(kBuckets, (2 * K + 31) / 32 * 32);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((nq + QG - 1) / QG * CS));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = lc.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)CS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, knn_group_kernel<KIND, MAXF, QG, kThreads>, nn, sp, qv, nq, k, K, buckets, prefix,
                       max_limit, idx, dist, fb_list, fb_n, ctr);
    note_launch();
}
}  // namespace

bool launch_knn_group(const LaunchCfg &lc, const NNArgs &nn, const SpaceParams &sp, StatesView qv, int64_t nq, int k,
                      const int64_t *prefix, int64_t max_limit, int64_t *idx, double *dist,
                      unsigned long long *fb_list, unsigned long long *fb_n, RunCounters *ctr)
{
    if (nq == 0 || k > knn_fp32_max_k(sp) || nn.size >= (1ll << 30))
        return false;
    // Four queries share an element's loads from 64 queries on (wrapped 7-D, 60,000 elements: 63 queries
    // 47 us with one per CTA, 64 queries 49 us with four). The elements are split over a cluster as long
    // as the CTAs fit on the GPU together, twice over for a large index (200,000 elements, 1,000 queries:
    // 431 us against 466 us with one CTA per four queries; 60,000: 186 us against 182 us), and a warp
    // still has eight or more rounds of 32 elements.
    const int QG = nq >= 64 ? 4 : 1;
    const int64_t ctas = (nq + QG - 1) / QG;
    const int threads = QG == 1 || ctas < 64 ? 256 : 128;
    const int64_t room = (int64_t)lc.sm_count * (QG == 1 ? 4 : 768 / threads) * (nn.size >= 131072 ? 2 : 1);
    int CS = 1;
    while (CS < 8 && ctas * 2 * CS <= room && nn.size >= (int64_t)CS * 2048)
        CS *= 2;
#define GBO_GROUP(KIND, MAXF)                                                                                          \
    do                                                                                                                \
    {                                                                                                                 \
        if (QG == 1)                                                                                                  \
            launch_group_t<KIND, MAXF, 1, 256>(lc, nn, sp, qv, nq, k, knn_keep(k), CS, prefix, max_limit, idx, dist,  \
                                               fb_list, fb_n, ctr);                                                   \
        else if (threads == 256)                                                                                      \
            launch_group_t<KIND, MAXF, 4, 256>(lc, nn, sp, qv, nq, k, knn_keep(k), CS, prefix, max_limit, idx, dist,  \
                                               fb_list, fb_n, ctr);                                                   \
        else                                                                                                          \
            launch_group_t<KIND, MAXF, 4, 128>(lc, nn, sp, qv, nq, k, knn_keep(k), CS, prefix, max_limit, idx, dist,  \
                                               fb_list, fb_n, ctr);                                                   \
    } while (0)
    if (sp.kind == GBO_SPACE_KINEMATIC_CHAIN && sp.dim <= 10)
        GBO_GROUP(GBO_SPACE_KINEMATIC_CHAIN, 20);
    else if (sp.kind == GBO_SPACE_WRAP_L2 && sp.dim <= 4)
        GBO_GROUP(GBO_SPACE_WRAP_L2, 4);
    else if (sp.kind == GBO_SPACE_WRAP_L2 && sp.dim <= 8)
        GBO_GROUP(GBO_SPACE_WRAP_L2, 8);
    else if (sp.kind == GBO_SPACE_REAL_VECTOR && sp.dim <= 2)
        GBO_GROUP(GBO_SPACE_REAL_VECTOR, 2);
    else if (sp.kind == GBO_SPACE_REAL_VECTOR && sp.dim <= 4)
        GBO_GROUP(GBO_SPACE_REAL_VECTOR, 4);
    else if (sp.kind == GBO_SPACE_REAL_VECTOR && sp.dim <= 8)
        GBO_GROUP(GBO_SPACE_REAL_VECTOR, 8);
    else
        return false;
#undef GBO_GROUP
    return true;
}

// ---------------------------------------------------------------- nearestR
// A CTA (or cluster) takes QG queries: the FP32 distance of every element decides all but those within
// the error bound of the radius, which are decided in FP64 (offsets null: counts only). The fill pass
// writes each hit's FP64 distance in arrival order and the first CTA of the cluster then sorts the
// query's segment by (distance, key), a total order, so the result does not depend on the arrival order.
// *outside: an element lies outside the bounds for which eps32 holds; then, and for such a query, every
// distance is decided in FP64. One warp per query computing every distance in FP64 and one lane sorting
// took 4.4 ms a pass for 1,000 queries over 50,000 7-D elements, bound by the FP64 pipe and 1,000 warps;
// the whole nearestR call went from 9.06 to 0.53 ms.
constexpr int kSortRoom = 1024;

template <int KIND, int MAXF, int QG, int kThreads>
__global__ void __launch_bounds__(kThreads) radius_group_kernel(NNArgs nn, SpaceParams sp, StatesView qv, int64_t nq,
                                                                double r, const int *outside, int64_t *counts,
                                                                const int64_t *offsets, int64_t *idx, double *dist)
{
    constexpr int MAXD = KIND == GBO_SPACE_KINEMATIC_CHAIN ? MAXF / 2 : MAXF;
    __shared__ int cnt[QG];
    __shared__ double s_d[kSortRoom];
    __shared__ int64_t s_k[kSortRoom];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), CS = (int)cluster.num_blocks();
    const int64_t q0 = (int64_t)(blockIdx.x / CS) * QG;
    const float link = (float)sp.link;
    const int lane = threadIdx.x & 31;
    float qf[QG][MAXF];
    float lo[QG], hi[QG];  // below lo: a hit; above hi: none; squared for the box kinds
#pragma unroll
    for (int g = 0; g < QG; ++g)
    {
        const int64_t q = q0 + g;
#pragma unroll
        for (int f = 0; f < MAXF; ++f)
            qf[g][f] = 0.f;
        lo[g] = -1.f;
        hi[g] = -1.f;  // no query: no element
        if (q < nq)
        {
            query_features<KIND, MAXF>(sp, qv, q, qf[g]);
            bool in = *outside == 0 && nn.eps32 > 0.f;
            for (int d = 0; d < sp.dim; ++d)
            {
                const double x = qv(q, d);
                in &= x >= sp.low[d] && x <= sp.high[d];
            }
            const double e = 1.5 * (double)nn.eps32;
            double a = r - e, b = r + e;
            if (KIND != GBO_SPACE_KINEMATIC_CHAIN)
            {
                a = a > 0.0 ? a * a : -1.0;
                b = b * b;
                if (r + e < 0.0)
                    b = -1.0;
            }
            lo[g] = in ? __double2float_rd(a - 1e-6 * fabs(a)) : -1.f;
            hi[g] = in ? __double2float_ru(b + 1e-6 * fabs(b)) : kInf;
        }
    }
    if (threadIdx.x < QG)
        cnt[threadIdx.x] = 0;
    cluster.sync();
    int mine[QG];
#pragma unroll
    for (int g = 0; g < QG; ++g)
        mine[g] = 0;
    const int step = kThreads * CS;
    for (int key = rank * kThreads + (int)threadIdx.x; key < (int)nn.size; key += step)
    {
        float pf[MAXF];
        element_features<KIND, MAXF>(nn, sp, key, pf);
        const bool here = !nn.alive || nn.alive[key];
        unsigned near = 0;  // queries whose FP64 distance is needed
#pragma unroll
        for (int g = 0; g < QG; ++g)
        {
            const float d = group_dist<KIND, MAXF>(pf, qf[g], link);
            // NaN distances: not a hit, except that an unbounded query decides everything in FP64
            const bool may = here && (d <= hi[g] || hi[g] == kInf);
            const bool sure = may && !offsets && d < lo[g];
            mine[g] += sure;
            near |= may && !sure ? 1u << g : 0u;
        }
        while (near)
        {
            const int g = __ffs(near) - 1;
            near &= near - 1;
            const int64_t q = q0 + g;
            double x[MAXD], q64[MAXD];
            load_query<MAXD>(qv, q, sp.dim, q64);
            load_point<MAXD>(nn.pts64, nn.cap, sp.dim, key, x);
            const double dd = distance64<MAXD, false>(sp, x, q64);
            if (!(dd <= r))
                continue;
            int *count = cluster.map_shared_rank(&cnt[g], 0);
            const int at = atomicAdd(count, 1);
            if (offsets)
            {
                idx[offsets[q] + at] = key;
                dist[offsets[q] + at] = dd;
            }
        }
    }
    if (!offsets)
    {
#pragma unroll
        for (int g = 0; g < QG; ++g)
        {
            const int t = __reduce_add_sync(0xffffffffu, mine[g]);
            if (lane == 0 && t)
                atomicAdd(cluster.map_shared_rank(&cnt[g], 0), t);
        }
    }
    __threadfence();
    cluster.sync();
    if (rank != 0)
        return;
    if (!offsets)
    {
        if (threadIdx.x < QG && q0 + threadIdx.x < nq && counts)
            counts[q0 + threadIdx.x] = cnt[threadIdx.x];
        return;
    }
    for (int g = 0; g < QG && q0 + g < nq; ++g)
    {
        const int n = cnt[g];
        int64_t *ki = idx + offsets[q0 + g];
        double *di = dist + offsets[q0 + g];
        if (n <= kSortRoom)
        {
            __syncthreads();
            for (int i = threadIdx.x; i < n; i += kThreads)
            {
                s_d[i] = __ldcg(di + i);
                s_k[i] = __ldcg((const long long *)ki + i);
            }
            __syncthreads();
            for (int i = threadIdx.x; i < n; i += kThreads)
            {
                const double d = s_d[i];
                const int64_t key = s_k[i];
                int at = 0;
#pragma unroll 4
                for (int j = 0; j < n; ++j)
                    at += less_dk(s_d[j], s_k[j], d, key);
                di[at] = d;
                ki[at] = key;
            }
            continue;
        }
        // long segments: bitonic sort in place; positions past n act as +infinity and never move (every
        // comparison is ascending: the first step of a merge pairs mirrored positions)
        volatile double *dv = di;
        volatile int64_t *kv = ki;
        int64_t p2 = 1;
        while (p2 < n)
            p2 <<= 1;
        for (int64_t w = 2; w <= p2; w <<= 1)
            for (int64_t h = w >> 1; h > 0; h >>= 1)
            {
                __syncthreads();
                for (int64_t t = threadIdx.x; t < p2 / 2; t += kThreads)
                {
                    const int64_t i = t / h * 2 * h + t % h;
                    const int64_t j = h == w >> 1 ? t / h * 2 * h + 2 * h - 1 - t % h : i + h;
                    if (j < n)
                    {
                        const double a = dv[i], b = dv[j];
                        const int64_t ka = kv[i], kb = kv[j];
                        if (less_dk(b, kb, a, ka))
                        {
                            dv[i] = b;
                            dv[j] = a;
                            kv[i] = kb;
                            kv[j] = ka;
                        }
                    }
                }
                __threadfence_block();
            }
        __syncthreads();
    }
}

namespace
{
template <int KIND, int MAXF, int QG, int kThreads>
void launch_radius_t(const LaunchCfg &lc, const NNArgs &nn, const SpaceParams &sp, StatesView qv, int64_t nq, double r,
                     const int *outside, int CS, int64_t *counts, const int64_t *offsets, int64_t *idx, double *dist)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((nq + QG - 1) / QG * CS));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = lc.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)CS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, radius_group_kernel<KIND, MAXF, QG, kThreads>, nn, sp, qv, nq, r, outside, counts,
                       offsets, idx, dist);
    note_launch();
}
}  // namespace

bool launch_radius_group(const LaunchCfg &lc, const NNArgs &nn, const SpaceParams &sp, StatesView qv, int64_t nq,
                         double r, const int *outside, int64_t *counts, const int64_t *offsets, int64_t *idx,
                         double *dist)
{
    if (nq == 0 || nq >= (1ll << 28) || nn.size >= (1ll << 30))
        return false;
    // four queries share an element's loads from 64 queries on; clusters split the elements while the
    // CTAs are fewer than six per SM (as in launch_knn_group)
    const int QG = nq >= 64 ? 4 : 1;
    const int64_t ctas = (nq + QG - 1) / QG;
    int CS = 1;
    while (CS < 8 && ctas * 2 * CS <= (int64_t)lc.sm_count * (QG == 1 ? 4 : 6) && nn.size >= (int64_t)CS * 2048)
        CS *= 2;
#define GBO_RADIUS(KIND, MAXF)                                                                                         \
    do                                                                                                                \
    {                                                                                                                 \
        if (QG == 1)                                                                                                  \
            launch_radius_t<KIND, MAXF, 1, 256>(lc, nn, sp, qv, nq, r, outside, CS, counts, offsets, idx, dist);      \
        else                                                                                                          \
            launch_radius_t<KIND, MAXF, 4, 128>(lc, nn, sp, qv, nq, r, outside, CS, counts, offsets, idx, dist);      \
    } while (0)
    if (sp.kind == GBO_SPACE_KINEMATIC_CHAIN && sp.dim <= 10)
        GBO_RADIUS(GBO_SPACE_KINEMATIC_CHAIN, 20);
    else if (sp.kind == GBO_SPACE_WRAP_L2 && sp.dim <= 8)
        GBO_RADIUS(GBO_SPACE_WRAP_L2, 8);
    else if (sp.kind == GBO_SPACE_REAL_VECTOR && sp.dim <= 4)
        GBO_RADIUS(GBO_SPACE_REAL_VECTOR, 4);
    else if (sp.kind == GBO_SPACE_REAL_VECTOR && sp.dim <= 8)
        GBO_RADIUS(GBO_SPACE_REAL_VECTOR, 8);
    else
        return false;
#undef GBO_RADIUS
    return true;
}

}  // namespace gbo
