// Kinematic-chain kernels built on the warp-cooperative FP32 evaluator (chain_warp.cuh).
//
//   chain_validity_warp_kernel  StateValidityChecker::isValid, one warp per state
//   chain_motion_warp_kernel    DiscreteMotionValidator::checkMotion, persistent, one warp per edge
//                               taken from the device work queue; states j = 1..nd-1 then s2 in order
//                               (DiscreteMotionValidator.cpp:48-91), stopping at the first invalid one.
// Interpolated joints are formed in float-float from exact splits of s1 and s2:
//   q_i(t) = s1_i + D_i t, D_i the shortest-arc difference of KinematicChain.h:150-176 (the wrap by
//   2*pi that interpolate applies changes no sine or cosine), t = j / nd in float-float; the link
//   angles theta_k(t) = sum_{i<=k} q_i(t) = A_k + t S_k come from per-edge prefix sums A_k of s1 and
//   S_k of D, so a state needs no scan of its joints.
// Anything the FP32 error bounds leave undecided is settled with the FP64 reference-order code: an
// ambiguous segment test (chain_round64), an undecided segment count (chain_nd64_warp), and the states of
// an edge whose joint difference lies within 1e-9 of pi, where the interpolation's own branch is not
// settled in FP32 (motion_joint64). All FP64 work sits in small out-of-line functions: an inlined or
// large call inside the edge loop costs the loop registers, and local-memory spills, on every edge.
#include "chain_state.cuh"
#include "kernels.cuh"
#include "tma.cuh"

namespace gbo
{

// Dynamic shared memory of the warp kernels: the world's ChainSegF32 records (bytes32 = 32 * nw),
// then (dim + 1) link records per warp, then one test table per warp (one u32 per test).
struct ChainSmem
{
    ChainSegF32 *w32;
    const unsigned *tab;  // this warp's table
    int nw;               // world segments
    int lb;               // index of this warp's first link record in w32
    ChainTables t;
};

__device__ bool chain_setup(const SpaceParams &sp, const WorldArgs &wa, unsigned char *smem, uint64_t *bar,
                            RunCounters *ctr, ChainSmem &cs)
{
    if (!stage_bulk(smem, wa.data32, wa.bytes32, bar, &ctr->timeout, &ctr->error))
        return false;
    ChainSegF32 *w = (ChainSegF32 *)smem;
    const int per_warp = sp.dim + 1, n_link_recs = (int)(blockDim.x >> 5) * per_warp;
    init_chain_links(w + wa.n, n_link_recs, wa.guard);
    unsigned *tabs = (unsigned *)(w + wa.n + n_link_recs);
    build_chain_tables(sp.dim, wa.n, wa.test_order, tabs, (int)(blockDim.x >> 5), cs.t);
    if (threadIdx.x == 0)
    {
        chain_hz_pos = wa.hz_pos;
        chain_hz = &ctr->hazards;
    }
    __syncthreads();
    cs.w32 = w;
    cs.tab = tabs + (threadIdx.x >> 5) * cs.t.n_tests;
    cs.nw = wa.n;
    cs.lb = wa.n + (int)(threadIdx.x >> 5) * per_warp;
    return true;
}

__device__ __forceinline__ ff lane_joint(const StatesView &v, int64_t i, int lane, int dim)
{
    return lane < dim ? split_double(v(i, lane)) : ff{0.f, 0.f};
}

// Cold FP64 paths (reference operation order), kept out of line so that the FP32 kernels keep a small
// register footprint.

// StateSpace::validSegmentCount of one edge in FP64 (StateSpace.cpp:851-854), warp-collective: the
// chain metric of distance64 (demos/KinematicChain.h:105-121) with the cumulative angles and the
// sums in the reference's order (lane by lane through shuffles) and the sines and cosines one joint
// per lane.
__device__ __noinline__ int chain_nd64_warp(const SpaceParams &sp, const StatesView &v1, const StatesView &v2,
                                            int64_t e, int lane)
{
    const int n = sp.dim;
    const double qa = lane < n ? v1(e, lane) : 0.0, qb = lane < n ? v2(e, lane) : 0.0;
    double t1 = 0., t2 = 0., m1 = 0., m2 = 0.;
    for (int i = 0; i < n; ++i)
    {
        t1 = dadd(t1, __shfl_sync(0xffffffffu, qa, i));
        t2 = dadd(t2, __shfl_sync(0xffffffffu, qb, i));
        if (i == lane)
        {
            m1 = t1;
            m2 = t2;
        }
    }
    double s1 = 0., c1 = 1., s2 = 0., c2 = 1.;
    if (lane < n)
    {
        sincos(m1, &s1, &c1);
        sincos(m2, &s2, &c2);
    }
    double dx = 0., dy = 0., dist = 0.;
    for (int i = 0; i < n; ++i)
    {
        dx = dadd(dx, dsub(__shfl_sync(0xffffffffu, c1, i), __shfl_sync(0xffffffffu, c2, i)));
        dy = dadd(dy, dsub(__shfl_sync(0xffffffffu, s1, i), __shfl_sync(0xffffffffu, s2, i)));
        dist = dadd(dist, dsqrt(dadd(dmul(dx, dx), dmul(dy, dy))));
    }
    return segment_count_from_distance(sp, dmul(dist, sp.link));
}

// Joint `ln` of checked state j of edge e in FP64, as DiscreteMotionValidator.cpp:63 forms it (j == top
// is s2 itself). Out of line: inlined, the compiler hoists the loop-invariant FP64 division j / nd out
// of the rarely taken re-check branch and executes it for every checked state.
__device__ __noinline__ double motion_joint64(const StatesView &v1, const StatesView &v2, int64_t e, int ln, int j,
                                              int nd, int top)
{
    if (j == top)
        return v2(e, ln);
    return interp_angle64(v1(e, ln), v2(e, ln), ddiv((double)j, (double)nd));
}

__global__ void __launch_bounds__(256, 4) chain_validity_warp_kernel(const __grid_constant__ SpaceParams sp,
                                                                  const __grid_constant__ WorldArgs wa,
                                                                  const __grid_constant__ StatesView v, int64_t n,
                                                                  uint8_t *out, RunCounters *ctr)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    ChainSmem cs;
    if (!chain_setup(sp, wa, smem, &bar, ctr, cs))
        return;
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const float L = (float)sp.link;
    const double L64 = sp.link;
    const int dim = sp.dim;
    const double *w64 = (const double *)wa.data64;
    unsigned rechecks = 0, evaluated = 0;
    for (int64_t i = warp; i < n; i += nwarps)
    {
        ++evaluated;
        float vx, vy, px, py;
        chain_segments32(lane_joint(v, i, lane, dim), lane, dim, L, vx, vy, px, py);
        auto q64 = [&](int ln) { return ln < dim ? v(i, ln) : 0.0; };
        const int r = chain_state_warp32(lane, dim, L64, vx, vy, px, py, cs.w32, cs.nw, cs.lb, w64, cs.tab, cs.t, q64,
                                         rechecks);
        if (lane == 0)
            out[i] = r == kValid ? 1 : 0;
    }
    if (lane == 0)
    {
        if (evaluated)
            atomicAdd(&ctr->evaluated, (unsigned long long)evaluated);
        if (rechecks)
            atomicAdd(&ctr->rechecked, (unsigned long long)rechecks);
    }
}

__global__ void __launch_bounds__(256, 4) chain_motion_warp_kernel(const __grid_constant__ SpaceParams sp,
                                                                const __grid_constant__ WorldArgs wa,
                                                                const __grid_constant__ StatesView v1,
                                                                const __grid_constant__ StatesView v2, int64_t n,
                                                                uint8_t *ok, int32_t *first_j, int32_t *nd_out,
                                                                RunCounters *ctr)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    ChainSmem cs;
    if (!chain_setup(sp, wa, smem, &bar, ctr, cs))
        return;
    const int lane = threadIdx.x & 31;
    const int dim = sp.dim;
    const float L = (float)sp.link;
    const double L64 = sp.link;
    const double *w64 = (const double *)wa.data64;
    constexpr float kPiF = 3.14159265358979323846f;
    unsigned evaluated = 0, rechecks = 0;
    for (;;)
    {
        unsigned long long ei = 0;
        if (lane == 0)
            ei = atomicAdd(&ctr->queue, 1ull);
        const int64_t e = (int64_t)__shfl_sync(0xffffffffu, ei, 0);
        if (e >= n)
            break;
        const double a64 = lane < dim ? v1(e, lane) : 0.0, b64 = lane < dim ? v2(e, lane) : 0.0;
        const ff a = split_double(a64), b = split_double(b64);
        // shortest-arc difference per joint; an edge whose |difference| is within 1e-9 of pi, or with a
        // joint that is not finite, is decided with the FP64 interpolation (the reference's branch on
        // fabs(diff) <= pi is not settled here)
        ff diff = two_sum(b.hi, -a.hi);
        diff = fast_two_sum(diff.hi, diff.lo + (b.lo - a.lo));
        // |diff| - pi in float-float: adh - float(pi) is exact, float(pi) - pi = 8.742278e-08 (the
        // constant's own error is ~3e-15); the whole is good to ~1e-13, far inside the 1e-9 window
        const float adh = fabsf(diff.hi);
        const float over_pi = ((adh - kPiF) + (diff.hi < 0.f ? -diff.lo : diff.lo)) + 8.742278e-08f;
        const bool finite =
            ((__double2hiint(a64) & 0x7ff00000) != 0x7ff00000) && ((__double2hiint(b64) & 0x7ff00000) != 0x7ff00000);
        const bool near_pi = lane < dim && !(fabsf(over_pi) >= 1e-9f && finite);
        // an edge with a joint difference within 1e-9 of pi builds its states with the FP64 reference
        // interpolation (motion_joint64): the branch on fabs(diff) <= pi is not settled in FP32
        const bool exact = __any_sync(0xffffffffu, near_pi);
        ff D = diff;
        if (lane < dim && over_pi > 0.f)  // the reference wraps when fabs(diff) > pi
        {
            // D = diff - sign(diff) * 2*pi in float-float
            const float sgn = diff.hi > 0.f ? -1.f : 1.f;
            const ff t1 = two_sum(diff.hi, sgn * 6.28125f);
            const ff t2 = two_sum(t1.hi, sgn * (519505.0f / 268435456.0f));
            D = fast_two_sum(t2.hi, (t1.lo + t2.lo) + (diff.lo + sgn * 2.4308403e-10f));
        }
        // absolute link angles of s1 and s2 and the prefix sums of the joint differences: state t has
        // theta_k(t) = ta_k + t * DS_k (the sum over joints of a_i + D_i t)
        // s2's angles ta + DS differ from its own prefix sums by whole turns (the wraps of D), which
        // leave every sine and cosine unchanged
        const ff ta = warp_scan_ff(a, lane), DS = warp_scan_ff(D, lane);
        const ff tb = ff_add(ta, DS);
        int nd = chain_segment_count_warp(ta, tb, lane, dim, L, wa.inv_lvs32, wa.e_dist, sp.factor);
        const bool nd64 = nd < 0;
        if (nd64)
        {
            // not decided by the FP32 distance bound. Identical finite end points: every term of the reference's
            // sum is exactly zero, so its count is; else the reference's FP64 count
            const bool same = __all_sync(0xffffffffu, lane >= dim || (a64 == b64 && finite));
            nd = same ? 0 : chain_nd64_warp(sp, v1, v2, e, lane);
        }
        if (exact || nd64)
            ++rechecks;
        const int top = nd > 1 ? nd : 1;
        // 1/nd in float-float
        const float ndf = float_of(nd > 0 ? nd : 1);
        const float inv_hi = __frcp_rn(ndf);
        const float inv_lo = fmaf(-inv_hi, ndf, 1.0f) * inv_hi;
        float jf = 0.f;
        int first = -1;
        for (int j = 1; j <= top; ++j)
        {
            jf += 1.0f;
            ff th;  // absolute link angle of lane < dim (j == top and exact are the same in every lane)
            if (j == top)
                th = tb;
            else if (exact)
                th = warp_scan_ff(lane < dim ? split_double(motion_joint64(v1, v2, e, lane, j, nd, top)) : ff{0.f, 0.f},
                                  lane);
            else
            {
                const float t_hi = jf * inv_hi;
                const float t_lo = fmaf(jf, inv_hi, -t_hi) + jf * inv_lo;
                const float p_hi = DS.hi * t_hi;
                const float p_lo = fmaf(DS.hi, t_hi, -p_hi) + fmaf(DS.hi, t_lo, DS.lo * t_hi);
                th = ff_add(ta, {p_hi, p_lo});
            }
            float vx, vy, px, py;
            chain_segments32_theta(th, lane, dim, L, vx, vy, px, py);
            auto q64 = [&](int ln) { return ln < dim ? motion_joint64(v1, v2, e, ln, j, nd, top) : 0.0; };
            const int r = chain_state_warp32(lane, dim, L64, vx, vy, px, py, cs.w32, cs.nw, cs.lb, w64, cs.tab, cs.t, q64,
                                             rechecks);
            ++evaluated;
            if (r == kInvalid)
            {
                first = j == top ? nd : j;
                break;
            }
        }
        if (lane == 0)
        {
            ok[e] = first < 0 ? 1 : 0;
            if (first_j)
                first_j[e] = first;
            if (nd_out)
                nd_out[e] = nd;
        }
    }
    if (lane == 0)
    {
        if (evaluated)
            atomicAdd(&ctr->evaluated, (unsigned long long)evaluated);
        if (rechecks)
            atomicAdd(&ctr->rechecked, (unsigned long long)rechecks);
    }
}

// ---------------------------------------------------------------- large batches: lane per state, then warp per state
// A warp evaluates 32 states at a time. Each lane forms its own state's links (no warp scans, all lanes busy) and
// writes them to the warp's records; then the warp walks the test table with all lanes on the same test, 16
// tests at a time, as long as that finds intersections: the order puts the likely ones first, so most
// invalid states end here at about one warp instruction a state and test. The states left (valid ones mostly)
// are finished one by one with 32 tests per round, as in chain_state_warp32. A definite intersection decides a
// state whatever other tests say; a state with an undecided test that no definite one follows is run
// through all tests again in rounds, where the FP64 code settles them.
//
// Worlds of at most 64 segments have masks (ChainMasks): a lane then tests its links against about 1.4 segments each
// instead of all, before the rounds, and the rounds are left with the link-link and tip tests.
//
// Against one warp per state or edge throughout, whose kinematics, scans and edge setup keep 10 of 32 lanes
// busy: a million states of 10 links among 32 segments 349 -> 101 us (worlds with hardly a valid state) and 367 ->
// 171 us (0.5% valid); edges at chain_motion_lanes. Bound: the ALU pipe (the guarded test's comparisons) and, for
// edges, the latency of the rounds at 20 warps an SM.
struct ChainLanes
{
    const ChainSegF32 *w;   // world segments
    const unsigned *tab;    // tests in order: chain_test_entry's format
    float4 *rec;            // this warp's links: state (lane) s, link k at s * stride + k: start point, vector
    float *edge;            // this warp's edges: rows of 32 (motion only)
    const unsigned *first;  // link-link and tip tests (with masks)
    int nw, n_tests, n_first, stride;
};

// Odd in float4 units: the 8 lanes of a 16-byte access phase then cover all banks
__host__ __device__ inline int chain_lane_stride(int dim)
{
    return (dim + 1) | 1;
}

__device__ bool chain_lanes_setup(const SpaceParams &sp, const WorldArgs &wa, unsigned char *smem, uint64_t *bar,
                                  RunCounters *ctr, ChainLanes &cl)
{
    if (!stage_bulk(smem, wa.data32, wa.bytes32, bar, &ctr->timeout, &ctr->error))
        return false;
    int n_self;
    cl.w = (const ChainSegF32 *)smem;
    cl.nw = wa.n;
    cl.n_tests = chain_test_count(sp.dim, wa.n, n_self);
    cl.stride = chain_lane_stride(sp.dim);
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
    float4 *rec = (float4 *)(smem + wa.bytes32);
    cl.rec = rec + (size_t)warp * 32 * cl.stride;
    unsigned *tab = (unsigned *)(rec + (size_t)warps * 32 * cl.stride);
    unsigned *first = tab + ((cl.n_tests + 3) & ~3);
    cl.first = first;
    cl.n_first = wa.masks.cell ? n_self + wa.n : 0;
    cl.edge = (float *)(first + ((cl.n_first + 3) & ~3)) + (size_t)warp * 4 * sp.dim * 32;
    for (int t = threadIdx.x; t < cl.n_first; t += blockDim.x)
        first[t] = t < n_self ? chain_test_entry(t, sp.dim, wa.n) : (unsigned)sp.dim | (unsigned)(t - n_self) << 8;
    for (int t = threadIdx.x; t < cl.n_tests; t += blockDim.x)
        tab[t] = wa.test_order ? wa.test_order[t] : chain_test_entry(t, sp.dim, wa.n);
    cl.tab = tab;
    if (threadIdx.x == 0)
    {
        chain_hz_pos = wa.hz_pos;
        chain_hz = &ctr->hazards;
    }
    __syncthreads();
    return true;
}

// One more link of the lane's state: angle th (float-float), start point x, y (moved on)
__device__ __forceinline__ void chain_lane_link(float4 *rec, int k, ff th, float L, float &c, float &s, float &x, float &y)
{
    sincos_ff(th, c, s);
    const float vx = c * L, vy = s * L;
    rec[k] = make_float4(x, y, vx, vy);
    x += vx;
    y += vy;
}

// The shared walk over the table: hit / amb of the lane's state (work lanes), tests done returned.
__device__ __forceinline__ int chain_lane_walk(const ChainLanes &cl, const ChainGuard &g, const float4 *rec, bool work,
                                               bool masks, bool &hit, bool &amb)
{
    int t = 0;
    hit = amb = false;
    unsigned left = __ballot_sync(0xffffffffu, work);
    while (left && t < cl.n_tests)
    {
        const int end = min(t + 16, cl.n_tests);
        for (; t < end; ++t)
        {
            const unsigned e = cl.tab[t];
            const float4 A = rec[chain_test_a(e)];
            float4 Bs;
            float lo, hi, den;
            if (e & 0x80000000u)
            {
                Bs = rec[chain_test_b(e)];
                lo = g.self_lo;
                hi = g.self_hi;
                den = g.self_den;
            }
            else
            {
                const ChainSegF32 ws = cl.w[chain_test_b(e)];
                Bs = make_float4(ws.x0, ws.y0, ws.sx, ws.sy);
                lo = ws.lo;
                hi = ws.hi;
                den = ws.e_den;
            }
            const int r = seg_intersect32(A.z, A.w, Bs.z, Bs.w, A.x - Bs.x, A.y - Bs.y, lo, hi, den);
            hit |= r == kInvalid;
            amb |= r == kAmbiguous;
        }
        hit = hit && work;
        const unsigned now = __ballot_sync(0xffffffffu, work && !hit);
        // a state left over costs about 250 instructions with masks (a warp's 16 tests: 650), 600 without
        const bool stop = __popc(left) - __popc(now) < (masks ? 3 : 1);
        left = now;
        if (stop)
            break;
    }
    return t;
}

// U tests per lane side by side (the warps are few, so each has to overlap its own latencies); act: the lane's
// test counts. kInvalid when one of them intersects, undecided ones settled in FP64, else kValid (all lanes).
template <int U, class Q64>
__device__ __forceinline__ int chain_lane_tests(const ChainLanes &cl, const ChainGuard &g, const float4 *rec,
                                                const unsigned (&e)[U], const bool (&act)[U], int lane, int n,
                                                double L64, const double *w64, Q64 q64, bool &have64)
{
    int r[U];
    bool clear = true;
#pragma unroll
    for (int u = 0; u < U; ++u)
    {
        const bool link = e[u] & 0x80000000u;
        const int b = chain_test_b(e[u]);
        const float4 A = rec[chain_test_a(e[u])];
        const float4 Bs = link ? rec[b] : *(const float4 *)&cl.w[b];
        const float4 Bb = link ? make_float4(g.self_lo, g.self_hi, g.self_den, 0.f) : *(const float4 *)&cl.w[b].lo;
        r[u] = seg_intersect32(A.z, A.w, Bs.z, Bs.w, A.x - Bs.x, A.y - Bs.y, Bb.x, Bb.y, Bb.z);
        r[u] = act[u] ? r[u] : kValid;
        clear &= r[u] == kValid;
    }
    if (!__ballot_sync(0xffffffffu, !clear))
        return kValid;
#pragma unroll
    for (int u = 0; u < U; ++u)
    {
        if (__any_sync(0xffffffffu, r[u] == kAmbiguous))
        {
            have64 = true;
            // chain_round64 takes record indices: links from nw on
            const unsigned ib = e[u] & 0x80000000u ? (unsigned)(cl.nw + chain_test_b(e[u])) : (unsigned)chain_test_b(e[u]);
            r[u] = chain_round64(lane, n, L64, q64(lane), (unsigned)(cl.nw + chain_test_a(e[u])) | ib << 16, cl.nw, cl.nw,
                                 r[u], w64);
        }
        if (__any_sync(0xffffffffu, r[u] == kInvalid))
            return kInvalid;
    }
    return kValid;
}

// World segments that a link (start point and vector in `l`) may have to be tested against: those within reach of
// its middle point, and those nearly parallel to it. All when the masks do not cover the link.
__device__ __forceinline__ unsigned long long chain_link_mask(const ChainMasks &m, const float4 l, unsigned long long all)
{
    const float mx = fmaf(0.5f, l.z, l.x), my = fmaf(0.5f, l.w, l.y);
    const float gx = (mx + m.half) * m.inv, gy = (my + m.half) * m.inv;
    const float d = fabsf(l.z) + fabsf(l.w);
    if (!(gx >= 0.f && gx < (float)kChainMaskCells && gy >= 0.f && gy < (float)kChainMaskCells && d > 0.f))
        return all;
    const float a = __fdividef(l.w < 0.f ? -l.z : l.z, d);  // cosine-like, decreasing over the half turn
    const int bin = min(kChainMaskBins - 1, max(0, (int)((0.5f - 0.5f * a) * (float)kChainMaskBins)));
    return __ldg(m.cell + (int)gx * kChainMaskCells + (int)gy) | __ldg(m.bin + bin);
}

// Each lane's own link-world tests by the masks (undecided lanes; the tip's tests are among the warp's rounds)
__device__ __forceinline__ void chain_lane_world(const ChainLanes &cl, const ChainMasks &masks, const float4 *rec, int n,
                                                 bool undecided, bool &hit, bool &amb)
{
    const unsigned long long all = ~0ull >> (64 - cl.nw);
    unsigned long long m = 0;
    float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
    int link = undecided ? 0 : n;
    while (__any_sync(0xffffffffu, link < n || m))
    {
        // a lane takes its next test, from the next link that has one
        while (!m && link < n)
        {
            A = rec[link++];
            m = chain_link_mask(masks, A, all);
        }
        if (m)
        {
            const ChainSegF32 B = cl.w[__ffsll((long long)m) - 1];
            m &= m - 1;
            const int r = seg_intersect32(A.z, A.w, B.sx, B.sy, A.x - B.x0, A.y - B.y0, B.lo, B.hi, B.e_den);
            amb |= r == kAmbiguous;
            if (r == kInvalid)
            {
                hit = true;
                m = 0;
                link = n;
            }
        }
    }
}

// The rest of the state in records `rec`: kInvalid or kValid in all lanes. With masks: the link-link and tip
// tests, then (world: not done by chain_lane_world, or left undecided there) each link's own world segments,
// several lanes a link; what is left out cannot intersect. Without
// (more than 64 segments): the table from test `t` on (t = 0 for a state with an undecided test).
template <class Q64>
__device__ __forceinline__ int chain_lane_rounds(const ChainLanes &cl, const WorldArgs &wa, const float4 *rec, int t,
                                                 bool world, int lane, int n, double L64, const double *w64, Q64 q64,
                                                 unsigned &rechecked)
{
    const ChainGuard &g = wa.guard;
    bool have64 = false;
    int r = kValid;
    if (wa.masks.cell)
    {
        const int n2 = cl.n_first;
        for (int base = 0; base < n2 && r == kValid; base += 96)
        {
            unsigned e[3];
            bool act[3];
#pragma unroll
            for (int u = 0; u < 3; ++u)
            {
                act[u] = base + 32 * u + lane < n2;
                e[u] = cl.first[min(base + 32 * u + lane, n2 - 1)];
            }
            r = chain_lane_tests<3>(cl, g, rec, e, act, lane, n, L64, w64, q64, have64);
        }
        if (r == kValid && world)
        {
            const int parts = 32 / n, link = lane / parts, part = lane - link * parts;  // n <= 15: at least 2 lanes
            const int bits = (64 + parts - 1) / parts;
            unsigned long long m = 0;
            if (link < n)
                m = chain_link_mask(wa.masks, rec[link], ~0ull >> (64 - cl.nw)) >> (bits * part) & ((1ull << bits) - 1);
            while (r == kValid && __any_sync(0xffffffffu, m != 0))
            {
                const bool act[1] = {m != 0};
                const int j = act[0] ? bits * part + __ffsll((long long)m) - 1 : 0;
                const unsigned e[1] = {(unsigned)(act[0] ? link : 0) | (unsigned)j << 8};
                m &= m - 1;
                r = chain_lane_tests<1>(cl, g, rec, e, act, lane, n, L64, w64, q64, have64);
            }
        }
    }
    else
        for (int base = t; base < cl.n_tests && r == kValid; base += 96)
        {
            unsigned e[3];
            bool act[3];
#pragma unroll
            for (int u = 0; u < 3; ++u)
            {
                act[u] = base + 32 * u + lane < cl.n_tests;
                e[u] = cl.tab[min(base + 32 * u + lane, cl.n_tests - 1)];
            }
            r = chain_lane_tests<3>(cl, g, rec, e, act, lane, n, L64, w64, q64, have64);
        }
    rechecked += have64 && lane == 0;
    return r;
}

__global__ void __launch_bounds__(128, 5) chain_validity_lane_kernel(const __grid_constant__ SpaceParams sp,
                                                                  const __grid_constant__ WorldArgs wa,
                                                                  const __grid_constant__ StatesView v, int64_t n,
                                                                  uint8_t *out, RunCounters *ctr)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    ChainLanes cl;
    if (!chain_lanes_setup(sp, wa, smem, &bar, ctr, cl))
        return;
    const int lane = threadIdx.x & 31, dim = sp.dim;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const float L = (float)sp.link;
    const double *w64 = (const double *)wa.data64;
    float4 *mine = cl.rec + lane * cl.stride;
    unsigned rechecks = 0, evaluated = 0;
    for (int64_t i0 = warp * 32; i0 < n; i0 += nwarps * 32)
    {
        const int64_t i = i0 + lane;
        const bool work = i < n;
        __syncwarp();  // the previous states' records are no longer read
        if (work)
        {
            ++evaluated;
            ff th{0.f, 0.f};
            float c = 1.f, s = 0.f, x = 0.f, y = 0.f;
            for (int d = 0; d < dim; ++d)
            {
                th = ff_add(th, split_double(v(i, d)));
                chain_lane_link(mine, d, th, L, c, s, x, y);
            }
            mine[dim] = make_float4(x, y, c * 0.001f, s * 0.001f);
        }
        __syncwarp();
        bool hit, amb;
        const int t = chain_lane_walk(cl, wa.guard, mine, work, wa.masks.cell != nullptr, hit, amb);
        if (wa.masks.cell)
            chain_lane_world(cl, wa.masks, mine, dim, work && !hit, hit, amb);
        unsigned left = __ballot_sync(0xffffffffu, work && !hit && (amb || t < cl.n_tests));
        const unsigned unsure = __ballot_sync(0xffffffffu, amb);
        while (left)
        {
            const int src = __ffs(left) - 1;
            left &= left - 1;
            auto q64 = [&](int ln) { return ln < dim ? v(i0 + src, ln) : 0.0; };
            const int r = chain_lane_rounds(cl, wa, cl.rec + src * cl.stride, unsure >> src & 1u ? 0 : t,
                                            unsure >> src & 1u, lane, dim,
                                            sp.link, w64, q64, rechecks);
            if (lane == src)
                hit = r == kInvalid;
        }
        if (work)
            out[i] = hit ? 0 : 1;
    }
    evaluated = __reduce_add_sync(0xffffffffu, evaluated);
    if (lane == 0)
    {
        if (evaluated)
            atomicAdd(&ctr->evaluated, (unsigned long long)evaluated);
        if (rechecks)
            atomicAdd(&ctr->rechecked, (unsigned long long)rechecks);
    }
}

// Each lane owns an edge of the work queue (refilled when half are idle); with half or fewer live, the lanes
// are spread over the live edges' next states. An edge's states are settled in order.
__global__ void __launch_bounds__(128, 5) chain_motion_lane_kernel(const __grid_constant__ SpaceParams sp,
                                                                const __grid_constant__ WorldArgs wa,
                                                                const __grid_constant__ StatesView v1,
                                                                const __grid_constant__ StatesView v2, int64_t n,
                                                                uint8_t *ok, int32_t *first_j, int32_t *nd_out,
                                                                RunCounters *ctr)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    __shared__ unsigned char order[4][32];
    ChainLanes cl;
    if (!chain_lanes_setup(sp, wa, smem, &bar, ctr, cl))
        return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, dim = sp.dim;
    const float L = (float)sp.link;
    const double *w64 = (const double *)wa.data64;
    constexpr float kPiF = 3.14159265358979323846f;
    float4 *mine = cl.rec + lane * cl.stride;
    unsigned rechecks = 0, evaluated = 0;
    int64_t e = 0;
    int nd = 0, top = 0, next = 1, first = -1;
    bool live = false, more = true, exact = false;
    for (;;)
    {
        const unsigned idle = __ballot_sync(0xffffffffu, !live && more);
        if (idle && (__popc(idle) >= 16 || !__any_sync(0xffffffffu, live)))
        {
            unsigned long long q = 0;
            if (lane == __ffs(idle) - 1)
                q = atomicAdd(&ctr->queue, (unsigned long long)__popc(idle));
            q = __shfl_sync(0xffffffffu, q, __ffs(idle) - 1);
            bool nd64 = false;
            const bool fresh = idle >> lane & 1u;
            if (fresh)
            {
                e = (int64_t)q + __popc(idle & ((1u << lane) - 1u));
                more = e < n;
                live = more;
            }
            if (fresh && live)
            {
                // as chain_motion_warp_kernel, joint by joint: shortest-arc differences, absolute angles of s1, their
                // changes over the edge, and the segment count by the FP32 metric
                exact = false;
                bool same = true;  // identical finite end points
                ff ta{0.f, 0.f}, DS{0.f, 0.f};
                float dx = 0.f, dy = 0.f, dist = 0.f;
                for (int d = 0; d < dim; ++d)
                {
                    const double a64 = v1(e, d), b64 = v2(e, d);
                    const ff a = split_double(a64), b = split_double(b64);
                    ff diff = two_sum(b.hi, -a.hi);
                    diff = fast_two_sum(diff.hi, diff.lo + (b.lo - a.lo));
                    const float adh = fabsf(diff.hi);
                    const float over_pi = ((adh - kPiF) + (diff.hi < 0.f ? -diff.lo : diff.lo)) + 8.742278e-08f;
                    const bool finite = ((__double2hiint(a64) & 0x7ff00000) != 0x7ff00000) &&
                                        ((__double2hiint(b64) & 0x7ff00000) != 0x7ff00000);
                    exact |= !(fabsf(over_pi) >= 1e-9f && finite);
                    same &= a64 == b64 && finite;
                    ff D = diff;
                    if (over_pi > 0.f)
                    {
                        const float sgn = diff.hi > 0.f ? -1.f : 1.f;
                        const ff t1 = two_sum(diff.hi, sgn * 6.28125f);
                        const ff t2 = two_sum(t1.hi, sgn * (519505.0f / 268435456.0f));
                        D = fast_two_sum(t2.hi, (t1.lo + t2.lo) + (diff.lo + sgn * 2.4308403e-10f));
                    }
                    ta = ff_add(ta, a);
                    DS = ff_add(DS, D);
                    cl.edge[(4 * d) * 32 + lane] = ta.hi;
                    cl.edge[(4 * d + 1) * 32 + lane] = ta.lo;
                    cl.edge[(4 * d + 2) * 32 + lane] = DS.hi;
                    cl.edge[(4 * d + 3) * 32 + lane] = DS.lo;
                    float c1, s1, c2, s2;
                    sincos_ff(ta, c1, s1);
                    sincos_ff(ff_add(ta, DS), c2, s2);
                    dx += c1 - c2;
                    dy += s1 - s2;
                    dist += sqrtf(fmaf(dx, dx, dy * dy));
                }
                dist *= L;
                const float lo = (dist - wa.e_dist) * wa.inv_lvs32 * (1.0f - 4.0f * 5.96e-8f);
                const float hi = (dist + wa.e_dist) * wa.inv_lvs32 * (1.0f + 4.0f * 5.96e-8f);
                const float cl_ = ceilf(lo), ch = ceilf(hi);
                nd64 = !(lo > 0.f) || !(hi < 4.0e6f) || cl_ != ch;
                if (!nd64)
                    nd = (int)(sp.factor * (unsigned)cl_);
                else if (same)
                    nd = 0;  // every term of the reference's sum is exactly zero
                rechecks += exact || nd64;
                nd64 &= !same;
            }
            unsigned todo = __ballot_sync(0xffffffffu, nd64);
            while (todo)
            {
                const int src = __ffs(todo) - 1;
                todo &= todo - 1;
                const int c = chain_nd64_warp(sp, v1, v2, __shfl_sync(0xffffffffu, e, src), lane);
                if (lane == src)
                    nd = c;
            }
            if (fresh && live)
            {
                top = nd > 1 ? nd : 1;
                next = 1;
                first = -1;
            }
        }
        const unsigned M = __ballot_sync(0xffffffffu, live);
        if (!M)
        {
            if (__any_sync(0xffffffffu, more))
                continue;
            break;
        }
        const int cnt = __popc(M), reps = 32 / cnt;
        int owner = lane, rep = 0;
        bool work = live;
        if (reps > 1)
        {
            if (live)
                order[warp][__popc(M & ((1u << lane) - 1u))] = (unsigned char)lane;
            __syncwarp();
            rep = lane / cnt;
            owner = order[warp][lane - rep * cnt];
            work = rep < reps;
        }
        const int o_next = __shfl_sync(0xffffffffu, next, owner), o_top = __shfl_sync(0xffffffffu, top, owner);
        const int o_nd = __shfl_sync(0xffffffffu, nd, owner);
        const int64_t o_e = __shfl_sync(0xffffffffu, e, owner);
        const bool o_exact = __shfl_sync(0xffffffffu, (int)exact, owner);
        work = work && o_top - o_next >= rep;
        const int j = work ? o_next + rep : o_next;
        __syncwarp();  // the previous states' records are no longer read
        if (work)
        {
            ++evaluated;
            const float ndf = float_of(o_nd > 0 ? o_nd : 1);
            const float inv_hi = __frcp_rn(ndf), inv_lo = fmaf(-inv_hi, ndf, 1.0f) * inv_hi;
            const float jf = float_of(j);
            const float t_hi = jf * inv_hi, t_lo = fmaf(jf, inv_hi, -t_hi) + jf * inv_lo;
            ff run{0.f, 0.f};
            float c = 1.f, s = 0.f, x = 0.f, y = 0.f;
            for (int d = 0; d < dim; ++d)
            {
                const ff ta{cl.edge[(4 * d) * 32 + owner], cl.edge[(4 * d + 1) * 32 + owner]};
                const ff DS{cl.edge[(4 * d + 2) * 32 + owner], cl.edge[(4 * d + 3) * 32 + owner]};
                ff th;
                if (j == o_top)
                    th = ff_add(ta, DS);
                else if (o_exact)
                    th = run = ff_add(run, split_double(motion_joint64(v1, v2, o_e, d, j, o_nd, o_top)));
                else
                {
                    const float p_hi = DS.hi * t_hi;
                    const float p_lo = fmaf(DS.hi, t_hi, -p_hi) + fmaf(DS.hi, t_lo, DS.lo * t_hi);
                    th = ff_add(ta, {p_hi, p_lo});
                }
                chain_lane_link(mine, d, th, L, c, s, x, y);
            }
            mine[dim] = make_float4(x, y, c * 0.001f, s * 0.001f);
        }
        __syncwarp();
        bool hit, amb;
        const int t = chain_lane_walk(cl, wa.guard, mine, work, wa.masks.cell != nullptr, hit, amb);
        if (wa.masks.cell)
            chain_lane_world(cl, wa.masks, mine, dim, work && !hit, hit, amb);
        // the states that are left, in order; those behind a colliding state of their edge do not matter
        unsigned left = __ballot_sync(0xffffffffu, work && !hit && (amb || t < cl.n_tests));
        const unsigned unsure = __ballot_sync(0xffffffffu, amb);
        const int mate = reps > 1 ? cnt : 32;  // lanes of one owner are `mate` apart
        while (left)
        {
            const int src = __ffs(left) - 1;
            left &= left - 1;
            // a state before it on the same edge already collides
            const unsigned hits = __ballot_sync(0xffffffffu, hit);
            bool behind = false;
            for (int l = src - mate; l >= 0; l -= mate)
                behind |= hits >> l & 1u;
            if (behind)
                continue;
            const int64_t se = __shfl_sync(0xffffffffu, o_e, src);
            const int sj = __shfl_sync(0xffffffffu, j, src), snd = __shfl_sync(0xffffffffu, o_nd, src);
            const int stop = __shfl_sync(0xffffffffu, o_top, src);
            auto q64 = [&](int ln) { return ln < dim ? motion_joint64(v1, v2, se, ln, sj, snd, stop) : 0.0; };
            const int r = chain_lane_rounds(cl, wa, cl.rec + src * cl.stride, unsure >> src & 1u ? 0 : t,
                                            unsure >> src & 1u, lane, dim,
                                            sp.link, w64, q64, rechecks);
            if (lane == src)
                hit = r == kInvalid;
        }
        // the owner takes its states in order
        const unsigned hits = __ballot_sync(0xffffffffu, hit && work), worked = __ballot_sync(0xffffffffu, work);
        if (live)
        {
            const int rank = __popc(M & ((1u << lane) - 1u));
            for (int i = 0; i < reps && first < 0; ++i)
            {
                const int l = reps > 1 ? rank + i * cnt : lane;
                if (!(worked >> l & 1u))
                    break;
                if (hits >> l & 1u)
                    first = next;
                else
                    ++next;
            }
            if (first >= 0 || next > top)
            {
                ok[e] = first < 0 ? 1 : 0;
                if (first_j)
                    first_j[e] = first < 0 ? -1 : (first == top ? nd : first);
                if (nd_out)
                    nd_out[e] = nd;
                live = false;
            }
        }
    }
    evaluated = __reduce_add_sync(0xffffffffu, evaluated);
    rechecks = __reduce_add_sync(0xffffffffu, rechecks);
    if (lane == 0)
    {
        if (evaluated)
            atomicAdd(&ctr->evaluated, (unsigned long long)evaluated);
        if (rechecks)
            atomicAdd(&ctr->rechecked, (unsigned long long)rechecks);
    }
}

static unsigned chain_lane_smem(const SpaceParams &sp, const WorldArgs &wa, bool motion)
{
    const int m = sp.dim + 1, n_self = (m - 1) * (m - 2) / 2, n_tests = n_self + m * wa.n;
    const int n_first = wa.masks.cell ? n_self + wa.n : 0;
    return wa.bytes32 + 4 * 32 * chain_lane_stride(sp.dim) * 16 + (((n_tests + 3) & ~3) + ((n_first + 3) & ~3)) * 4 +
           (motion ? 4 * 4 * sp.dim * 32 * 4 : 0);
}

// Hit bitmaps of n states (SoA FP64, ld = n) for the host's test ordering: one warp per state.
__global__ void __launch_bounds__(256) chain_hits_kernel(SpaceParams sp, WorldArgs wa, const double *states, int n,
                                                         unsigned *bits, int words)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    RunCounters *none = nullptr;
    (void)none;
    __shared__ unsigned timeout, error;
    if (threadIdx.x == 0)
        timeout = error = 0;
    __syncthreads();
    if (!stage_bulk(smem, wa.data32, wa.bytes32, &bar, &timeout, &error))
        return;
    const ChainSegF32 *w = (const ChainSegF32 *)smem;
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    int n_self;
    const int n_tests = chain_test_count(sp.dim, wa.n, n_self);
    StatesView v{states, 1, (int64_t)n};
    for (int i = warp; i < n; i += nwarps)
    {
        float vx, vy, px, py;
        chain_segments32(lane_joint(v, i, lane, sp.dim), lane, sp.dim, (float)sp.link, vx, vy, px, py);
        chain_state_hits32(lane, vx, vy, px, py, w, sp.dim, wa.n, n_tests, wa.guard, bits + (size_t)i * words);
    }
}

void launch_chain_hits(cudaStream_t s, const SpaceParams &sp, const WorldArgs &wa, const double *states, int n,
                       unsigned *bits, int words)
{
    if (wa.bytes32 > 48 * 1024)
    {
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        cudaFuncSetAttribute((const void *)chain_hits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin - 1024);
    }
    chain_hits_kernel<<<64, 256, wa.bytes32, s>>>(sp, wa, states, n, bits, words);
    note_launch();
}

static unsigned chain_smem(const SpaceParams &sp, const WorldArgs &wa, int block)
{
    const int m = sp.dim + 1;
    const int n_tests = (m - 1) * (m - 2) / 2 + m * wa.n;
    return wa.bytes32 + (unsigned)((block / 32) * m * sizeof(ChainSegF32)) +
           (unsigned)((4 * (block / 32) * n_tests + 15) & ~15);
}

// The dynamic shared memory limit of a persistent kernel is raised to the opt-in maximum - 1 KB.
static bool chain_smem_fits(unsigned bytes)
{
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return (int64_t)bytes + 1024 <= (int64_t)optin;
}

// Block size of the warp kernels: 256 threads, or fewer warps per CTA when the per-warp test tables of
// a large world would not fit in shared memory (down to one warp, which needs what a single shared
// table did). Returns 0 when even that does not fit.
static int chain_block(const SpaceParams &sp, const WorldArgs &wa, unsigned &sm)
{
    for (int block = 256; block >= 32; block /= 2)
    {
        sm = chain_smem(sp, wa, block);
        if (chain_smem_fits(sm))
            return block;
    }
    return 0;
}

static bool chain_lanes_fit(const SpaceParams &sp, const WorldArgs &wa, bool motion)
{
    // dim <= 15: link angles of interpolated states inside sincos_ff's range, two lanes a link in the rounds
    return sp.dim <= 15 && wa.stage32 && chain_smem_fits(chain_lane_smem(sp, wa, motion));
}

// Lane per edge once the batch fills every lane the GPU holds (97,280 at 10 links): below that a warp waits for its
// slowest edge with few others to hide it (65,536 edges between valid states of the benchmark's world: 187 us against
// 173 us a warp per edge; 100,000: 248 against 245; 400,000: 673 against 871; 100,000 edges that end at their first
// state: 35 against 92). Not for rows read across the host link, where a lane's reads come a few bytes at a time
// (100,000 edges of that world, page-locked: 270 us a warp per edge in place, 660 a lane per edge in place, 350 a
// lane per edge after a copy to the device).
bool chain_motion_lanes(const LaunchCfg &lc, const SpaceParams &sp, const WorldArgs &wa, int64_t n)
{
    if (lc.host_rows || wa.kind != GBO_CHECK_CHAIN_SEGMENTS || n < 32768 || !chain_lanes_fit(sp, wa, true))
        return false;
    return n >= 128ll * persistent_grid((const void *)chain_motion_lane_kernel, 128, chain_lane_smem(sp, wa, true), lc,
                                        INT64_MAX / 2);
}

// Lane per state from the batch on that fills them (32,768 states: the same 27 us; 65,536: 41 against 27).
bool chain_validity_lanes(const SpaceParams &sp, const WorldArgs &wa, int64_t n)
{
    return wa.kind == GBO_CHECK_CHAIN_SEGMENTS && n >= 32768 && chain_lanes_fit(sp, wa, false);
}

bool launch_chain_validity_warp(const LaunchCfg &lc, const SpaceParams &sp, const WorldArgs &wa, StatesView v,
                                int64_t n, uint8_t *out, RunCounters *ctr)
{
    if (chain_validity_lanes(sp, wa, n))
    {
        const unsigned bytes = chain_lane_smem(sp, wa, false);
        const int grid = persistent_grid((const void *)chain_validity_lane_kernel, 128, bytes, lc, (n + 127) / 128);
        chain_validity_lane_kernel<<<grid, 128, bytes, lc.stream>>>(sp, wa, v, n, out, ctr);
        note_launch();
        return true;
    }
    unsigned sm = 0;
    const int block = sp.dim > 31 || !wa.stage32 ? 0 : chain_block(sp, wa, sm);
    if (!block)
        return false;
    const int grid =
        persistent_grid((const void *)chain_validity_warp_kernel, block, sm, lc, (n * 32 + block - 1) / block);
    chain_validity_warp_kernel<<<grid, block, sm, lc.stream>>>(sp, wa, v, n, out, ctr);
    note_launch();
    return true;
}

bool launch_chain_motion_warp(const LaunchCfg &lc, const SpaceParams &sp, const WorldArgs &wa, StatesView v1,
                              StatesView v2, int64_t n, uint8_t *ok, int32_t *fj, int32_t *nd, RunCounters *ctr)
{
    if (chain_motion_lanes(lc, sp, wa, n))
    {
        const unsigned bytes = chain_lane_smem(sp, wa, true);
        const int grid = persistent_grid((const void *)chain_motion_lane_kernel, 128, bytes, lc, (n + 127) / 128);
        chain_motion_lane_kernel<<<grid, 128, bytes, lc.stream>>>(sp, wa, v1, v2, n, ok, fj, nd, ctr);
        note_launch();
        return true;
    }
    unsigned sm = 0;
    // link angles of interpolated states reach |theta| <= 2 dim pi, inside sincos_ff's range for dim <= 15
    const int block = sp.dim > 15 || !wa.stage32 ? 0 : chain_block(sp, wa, sm);
    if (!block)
        return false;
    const int grid =
        persistent_grid((const void *)chain_motion_warp_kernel, block, sm, lc, (n * 32 + block - 1) / block);
    chain_motion_warp_kernel<<<grid, block, sm, lc.stream>>>(sp, wa, v1, v2, n, ok, fj, nd, ctr);
    note_launch();
    return true;
}

}  // namespace gbo
