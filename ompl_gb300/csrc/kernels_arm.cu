// DH arm motion checking (DiscreteMotionValidator.cpp:48-91) by clearance: few of an edge's states are
// evaluated, the others are proven free.
//
//   arm_clearance_kernel  per cell of a uniform grid over the world, the distance from the cell's centre to
//                         the nearest obstacle surface (half, rounded down). Distance is 1-Lipschitz, so a
//                         point's clearance is at least that minus its distance from the centre.
//   arm_motion_kernel     evaluates state j of an edge: forward kinematics, and for each link the clearance of
//                         its halves (four spheres each at eight spheres a link). Halves with clearance above
//                         their extent plus the sphere radius need no narrow phase; the others test their
//                         spheres one by one as the definition does. What the clearances exceed is slack s.
//                         Along the motion a point of link i moves with velocity at most v (from the state's
//                         joint rates, at both link ends) and acceleration at most
//                         B = 1.5 sum_j W_j^2 len_j, W_j the sum of the joints' rates up to j (|Omega'| <=
//                         W^2/2 for the angular velocity Omega, |l''| <= |Omega'| len + |Omega|^2 len), so no
//                         state within r steps, v r + B r^2 / 2 <= s for every link, can collide: the next
//                         state to evaluate is j + r + 1. First invalid index, ok and nd are those of the
//                         state-by-state check.
//
// Work: a warp owns up to `per` edges, refilled from the device work queue. With as many live edges as
// lanes, each lane advances its own edge; with fewer, the lanes are spread over the live edges, `rep` of
// them evaluating states a stride apart, and the covered prefix of the strided states counts. Small batches
// and what is left when the queue has run empty go to arm_chunk_kernel, where many warps share an edge. The
// undecided states are settled by the whole warp in FP64, one at a time. In the FP64 form these are all
// states that may touch an obstacle: FP32 proves spheres free there, by bounds on its error, and decides
// nothing else.
//
// 256,000 edges of 2..2,000 states (48 checked in order, 9.6 evaluated) among 4,096 spheres: 3.20 ms for one
// warp per edge evaluating every state, 1.20 ms; 3,001 edges among 2,048 boxes in the FP64 form: 6.7 to 8.4 ms
// with every state and sphere in FP64, 0.37 to 0.43 ms. Bound: instruction issue of the FP32 evaluation (about 3,000
// instructions per 32 states) and the longest edges' rounds. Cells: 64^3 12.1 evaluations per edge, 128^3 9.6,
// 192^3 8.8 (not taken: 14 MB a world).
#include <algorithm>
#include <climits>

#include <cuda_fp16.h>

#include "arm_device.cuh"

namespace gbo
{

constexpr int kLateRounds = 8;   // rounds of a warp after the queue ran empty
constexpr int kArmChunks = 32;   // most runs that an edge is cut into, and
constexpr int kArmRun = 32;      // fewest states of a run

// Signed distance of obstacle i's surface from (x, y, z); the definition compares sphere distances with
// (rs + r)^2, so a negative radius acts by |rs + r|.
__device__ __forceinline__ float obstacle_distance(const WorldArgs &wa, int i, float x, float y, float z)
{
    const float *w = (const float *)wa.data32;  // rows of 4 (spheres) or 6 (boxes)
    if (wa.boxes)
    {
        const float *o = w + 6 * (int64_t)i;
        const float dx = fmaxf(fabsf(x - o[0]) - o[3], 0.f), dy = fmaxf(fabsf(y - o[1]) - o[4], 0.f);
        const float dz = fmaxf(fabsf(z - o[2]) - o[5], 0.f);
        return sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
    }
    const float4 o = ((const float4 *)w)[i];
    const float dx = x - o.x, dy = y - o.y, dz = z - o.z;
    return sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) - fmaxf(o.w, fabsf(wa.arm.rsf + o.w) - wa.arm.rsf);
}

// A CTA fills a block of 8 x 8 x 4 cells: the nearest obstacle of every cell is among those whose distance
// from the block's centre is at most the smallest such distance plus twice the block's half diagonal, so
// the CTA collects these first (both passes with the threads over the obstacles) and each cell looks at
// them alone. 128^3 cells among 16,384 spheres: 2 x 64 obstacles a thread instead of 16,384. Where the list is too
// long (a dense cluster, seen from blocks all around it) and the block far, the obstacles are divided among 8 lanes
// instead, whose 2 x 4 cells share one distance: a checker of 4,096 (100,000) spheres in a tenth of the world's width
// is made in 5.0 (110) ms instead of 8.6 (200) with every obstacle for every cell; edges evaluate 1% more states.
constexpr int kNearRoom = 2048;

__global__ void __launch_bounds__(256) arm_clearance_kernel(const __grid_constant__ WorldArgs wa, __half *out)
{
    __shared__ int near[kNearRoom];
    __shared__ float s_min[8];
    __shared__ int s_n;
    const int G = wa.clr_n, t = threadIdx.x;
    const int b = blockIdx.x, bz = b % (G / 4), by = b / (G / 4) % (G / 8), bx = b / (G / 4) / (G / 8);
    const float *lo = wa.clr_lo, *cell = wa.clr_cell;
    const float cx = lo[0] + (float)(8 * bx + 4) * cell[0], cy = lo[1] + (float)(8 * by + 4) * cell[1];
    const float cz = lo[2] + (float)(4 * bz + 2) * cell[2];
    const float hd = sqrtf(16.f * cell[0] * cell[0] + 16.f * cell[1] * cell[1] + 4.f * cell[2] * cell[2]);
    const float most = 30000.f * wa.clr_unit;
    float m = most;
    for (int i = t; i < wa.n; i += 256)
        m = fminf(m, obstacle_distance(wa, i, cx, cy, cz));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((t & 31) == 0)
        s_min[t >> 5] = m;
    if (t == 0)
        s_n = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k)
        m = fminf(m, s_min[k]);
    const float cut = m + 2.f * hd + wa.clr_margin;
    for (int i = t; i < wa.n; i += 256)
        if (obstacle_distance(wa, i, cx, cy, cz) <= cut)
        {
            const int at = atomicAdd(&s_n, 1);
            if (at < kNearRoom)
                near[at] = i;
        }
    __syncthreads();
    const int ix = 8 * bx + t / 32, iy = 8 * by + t / 4 % 8, iz = 4 * bz + t % 4;
    const float x = lo[0] + ((float)ix + 0.5f) * cell[0], y = lo[1] + ((float)iy + 0.5f) * cell[1];
    const float z = lo[2] + ((float)iz + 0.5f) * cell[2];
    float best = most;
    if (s_n <= kNearRoom)
        for (int k = 0; k < s_n; ++k)
            best = fminf(best, obstacle_distance(wa, near[k], x, y, z));
    else if (m >= 2.f * hd)
    {
        // 8 lanes, 2 x 4 cells: the distance from their middle, less each cell's from there
        const float gy = lo[1] + (float)(8 * by + (t / 8 % 4) * 2 + 1) * cell[1];
        for (int i = t % 8; i < wa.n; i += 8)
            best = fminf(best, obstacle_distance(wa, i, x, gy, cz));
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
            best = fminf(best, __shfl_xor_sync(0xffffffffu, best, o));
        best -= 1.000001f * sqrtf(fmaf(y - gy, y - gy, (z - cz) * (z - cz)));
    }
    else
        for (int i = 0; i < wa.n; ++i)
            best = fminf(best, obstacle_distance(wa, i, x, y, z));
    out[(ix * G + iy) * G + iz] = __float2half_rd(fmaxf(best - wa.clr_margin, -most) / wa.clr_unit);
}

void launch_arm_clearance(const LaunchCfg &lc, const WorldArgs &wa, __half *out)
{
    arm_clearance_kernel<<<wa.clr_n / 8 * (wa.clr_n / 8) * (wa.clr_n / 4), 256, 0, lc.stream>>>(wa, out);
    note_launch();
}

// Settles the lanes whose state is undecided with the warp's FP64 test, in lane order; the lanes of the same
// owner after a colliding state are left (their states come later on the edge).
__device__ __forceinline__ void arm_settle(const SpaceParams &sp, const WorldArgs &wa, const StatesView &v1,
                                           const StatesView &v2, int64_t e, int j, int nd, int top, int owner, int lane,
                                           double *wq, double (*wpos)[3], int &verdict, int &free, unsigned &rechecks,
                                           RunCounters *ctr)
{
    unsigned A = __ballot_sync(0xffffffffu, verdict == kAmbiguous);
    while (A)
    {
        const int src = __ffs(A) - 1;
        A &= A - 1;
        if (lane == src)
            arm_state64(sp, v1, v2, e, j, nd, top, wq);
        __syncwarp();
        const bool hit = dh_valid64_warp(wa.arm, wq, (const double *)wa.data64, wa, wpos, lane, &ctr->hazards);
        if (lane == src)
        {
            verdict = hit ? kInvalid : kValid;
            free = 0;
            ++rechecks;
        }
        if (hit)
            A &= ~(__ballot_sync(0xffffffffu, owner == __shfl_sync(0xffffffffu, owner, src)) & (0xfffffffeu << src));
        __syncwarp();
    }
}

// start angle a and difference to b of joint d, for arm_eval32's table. Not finite (or far out of range): NaN,
// which sends the states to FP64.
__device__ __forceinline__ void arm_store_joint(const SpaceParams &sp, float (*edge)[32], int col, int d, double a,
                                                double b)
{
    const double diff = joint_difference(sp, a, b);
    const ff A = split_double(a), D = split_double(diff);
    const bool fine = fabs(a) <= 1e6 && fabs(diff) <= 1e6;
    edge[4 * d][col] = fine ? A.hi : __int_as_float(0x7fc00000);
    edge[4 * d + 1][col] = A.lo;
    edge[4 * d + 2][col] = D.hi;
    edge[4 * d + 3][col] = D.lo;
}

__device__ __forceinline__ int arm_segments(const SpaceParams &sp, const StatesView &v1, const StatesView &v2, int64_t e,
                                            double *a, double *b)
{
#pragma unroll
    for (int d = 0; d < 8; ++d)
    {
        a[d] = d < sp.dim ? v1(e, d) : 0.0;
        b[d] = d < sp.dim ? v2(e, d) : 0.0;
    }
    return segment_count_from_distance(sp, distance64<8>(sp, a, b));
}

__device__ __forceinline__ void arm_write(int64_t e, int first, int nd, int top, uint8_t *ok, int32_t *first_j,
                                          int32_t *nd_out)
{
    ok[e] = first < 0 ? 1 : 0;
    if (first_j)
        first_j[e] = first < 0 ? -1 : (first == top ? nd : first);
    if (nd_out)
        nd_out[e] = nd;
}

__device__ __forceinline__ void arm_counts(RunCounters *ctr, unsigned evaluated, unsigned rechecks, int lane)
{
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

// 128 threads: four warps, each with its own edges; an edge's start angles and differences (float-float) are in
// the owner lane's column of the warp's table.
template <int PREC>
__global__ void __launch_bounds__(128, 5)
    arm_motion_kernel(const __grid_constant__ SpaceParams sp, const __grid_constant__ WorldArgs wa,
                      const __grid_constant__ StatesView v1, const __grid_constant__ StatesView v2, int64_t n, int per,
                      ArmTail *tail, uint8_t *ok, int32_t *first_j, int32_t *nd_out, RunCounters *ctr)
{
    __shared__ float tab[4][32][32];
    __shared__ ArmChain chain[4];
    __shared__ double wq[4][8];
    __shared__ double wpos[4][9][3];
    __shared__ unsigned char order[4][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float(*edge)[32] = tab[warp];
    unsigned evaluated = 0, rechecks = 0;
    // the owner lane's edge
    int64_t e = 0;
    int nd = 0, top = 0, next = 1, stride = 1, first = -1, late = 0;
    bool live = false, more = true, done = false;
    for (;;)
    {
        // refill once a quarter of the owners are idle
        const unsigned idle = __ballot_sync(0xffffffffu, lane < per && !live && more);
        if (idle && (4 * __popc(idle) >= per || !__any_sync(0xffffffffu, live)))
        {
            unsigned long long q = 0;
            if (lane == __ffs(idle) - 1)
                q = atomicAdd(&ctr->queue, (unsigned long long)__popc(idle));
            q = __shfl_sync(0xffffffffu, q, __ffs(idle) - 1);
            if (idle >> lane & 1u)
            {
                e = (int64_t)q + __popc(idle & ((1u << lane) - 1u));
                more = e < n;
                if (more)
                {
                    double a[8], b[8];
                    nd = arm_segments(sp, v1, v2, e, a, b);
                    top = nd > 1 ? nd : 1;
                    next = 1;
                    stride = 1;
                    first = -1;
                    live = true;
                    done = false;
#pragma unroll
                    for (int d = 0; d < 8; ++d)
                        if (d < sp.dim)
                            arm_store_joint(sp, edge, lane, d, a[d], b[d]);
                }
            }
            __syncwarp();
        }
        const unsigned M = __ballot_sync(0xffffffffu, live);
        if (!M)
        {
            if (__any_sync(0xffffffffu, lane < per && more))
                continue;
            break;
        }
        // lanes over the live edges: lane works on state next + rep * stride of `owner`
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
        const int o_nd = __shfl_sync(0xffffffffu, nd, owner), o_stride = __shfl_sync(0xffffffffu, stride, owner);
        const int64_t o_e = __shfl_sync(0xffffffffu, e, owner);
        const int64_t j64 = (int64_t)o_next + (int64_t)rep * o_stride;
        work = work && j64 <= o_top;
        const int j = (int)(work ? j64 : o_next);
        int verdict = kValid, free = 0;  // `free` states on each side of j are proven free
        if (work)
        {
            verdict = arm_eval32<PREC>(wa, chain[warp], lane, edge, owner, j, o_nd, free);
            ++evaluated;
        }
        arm_settle(sp, wa, v1, v2, o_e, j, o_nd, o_top, owner, lane, wq[warp], wpos[warp], verdict, free, rechecks,
                   ctr);
        if (reps == 1)
        {
            if (live)
            {
                if (verdict == kInvalid)
                    first = next;
                else if ((int64_t)next + free >= top)
                    done = true;
                else
                    next += free + 1;
            }
        }
        else
        {
            // the owner takes its strided states in order while they continue the covered prefix
            const int mine = __popc(M & ((1u << lane) - 1u));
            const int spacing = stride;
            int covered = next - 1;
            bool open = live;
            for (int i = 0; i < reps; ++i)
            {
                const int src = (mine + i * cnt) & 31;
                const int vi = __shfl_sync(0xffffffffu, verdict, src), fi = __shfl_sync(0xffffffffu, free, src);
                const int64_t x = (int64_t)next + (int64_t)i * spacing;
                if (open && x <= top)
                {
                    if (vi == kInvalid)
                    {
                        if (x == (int64_t)covered + 1)
                            first = (int)x;
                        open = false;
                    }
                    else if (x - fi <= (int64_t)covered + 1)
                    {
                        covered = (int)min(max((int64_t)covered, x + fi), (int64_t)top);
                        stride = 1 + fi + fi / 2;
                    }
                    else
                    {
                        open = false;
                        stride = 1 + spacing / 3;
                    }
                }
            }
            if (covered >= top)
                done = true;
            else
                next = covered + 1;
        }
        if (live && (first >= 0 || done))
        {
            arm_write(e, first, nd, top, ok, first_j, nd_out);
            live = false;
        }
        // the queue is empty: after a few more rounds the edges that are left go to the chunk kernel, where
        // many warps share each, as far as its list has room
        if (!__any_sync(0xffffffffu, lane < per && more) && ++late == kLateRounds)
        {
            const unsigned L = __ballot_sync(0xffffffffu, live);
            unsigned at = 0;
            if (lane == 0 && L)
                at = atomicAdd(&ctr->deferred, (unsigned)__popc(L));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(L & ((1u << lane) - 1u));
            if (live && at < (unsigned)kArmTailRoom)
            {
                tail[at] = ArmTail{(unsigned)e, next, INT_MAX, nd};
                live = false;
            }
        }
    }
    arm_counts(ctr, evaluated, rechecks, lane);
}

// Edges shared by many warps: a batch (tail null; first_j holds the smallest colliding state found, nd_out the segment
// counts) or a list: what arm_motion_kernel left, or a batch without those outputs. The states left of an edge are cut into at most `chunks` runs of
// kArmRun states or more; work item c * count + i is run c of edge i, so that every edge's early runs go first and the
// later runs of an edge that has already collided before them are passed over, as are those that a short edge does not
// have. A run's 32 lanes evaluate states a stride apart, as above. arm_finish_kernel then writes the results.
template <int PREC>
__global__ void __launch_bounds__(128, 5)
    arm_chunk_kernel(const __grid_constant__ SpaceParams sp, const __grid_constant__ WorldArgs wa,
                     const __grid_constant__ StatesView v1, const __grid_constant__ StatesView v2, int n, int chunks,
                     ArmTail *tail, int32_t *first_j, const int32_t *nd_out, RunCounters *ctr)
{
    __shared__ float tab[4][32][32];
    __shared__ ArmChain chain[4];
    __shared__ double wq[4][8];
    __shared__ double wpos[4][9][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float(*edge)[32] = tab[warp];
    unsigned evaluated = 0, rechecks = 0;
    const int count = tail ? (int)min(ctr->deferred, (unsigned)kArmTailRoom) : n;
    const int items = count * chunks, warps = (int)gridDim.x * 4;
    for (int item = (int)blockIdx.x * 4 + warp; item < items; item += warps)
    {
        const int c = item / count, i = item % count;
        const int64_t e = tail ? tail[i].e : i;
        const int nd = tail ? tail[i].nd : nd_out[i], start = tail ? tail[i].next : 1;
        int *first = tail ? &tail[i].first : first_j + i;
        const int top = nd > 1 ? nd : 1;
        const int64_t len = max(((int64_t)top - start + chunks) / chunks, (int64_t)kArmRun);
        int64_t lo = start + c * len;
        const int64_t end = min(lo + len - 1, (int64_t)top);
        // the smallest colliding state found so far, the same in every lane
        auto found = [&]() {
            const int f = lane == 0 ? *(volatile int *)first : 0;
            return __shfl_sync(0xffffffffu, f, 0);
        };
        if (lo <= end && found() > lo)
        {
            __syncwarp();
            if (lane < sp.dim)
                arm_store_joint(sp, edge, 0, lane, v1(e, lane), v2(e, lane));
            __syncwarp();
            int64_t stride = 1;
            while (lo <= end && found() > lo)
            {
                const int64_t j = lo + lane * stride;
                const bool work = j <= end;
                int verdict = kValid, free = 0;
                if (work)
                {
                    verdict = arm_eval32<PREC>(wa, chain[warp], lane, edge, 0, (int)j, nd, free);
                    ++evaluated;
                }
                arm_settle(sp, wa, v1, v2, e, (int)j, nd, top, 0, lane, wq[warp], wpos[warp], verdict, free, rechecks,
                           ctr);
                // covered prefix: the running maximum of what the lanes before proved free must reach the lane
                int64_t reach = work && verdict == kValid ? min(j + free, end) : lo - 1;
                for (int o = 1; o < 32; o <<= 1)
                {
                    const int64_t r = __shfl_up_sync(0xffffffffu, reach, o);
                    if (lane >= o)
                        reach = max(reach, r);
                }
                int64_t before = __shfl_up_sync(0xffffffffu, reach, 1);
                if (lane == 0)
                    before = lo - 1;
                const bool gap = work && (verdict == kInvalid || j - free > before + 1);
                const unsigned bad = __ballot_sync(0xffffffffu, gap);
                const int stop = bad ? __ffs(bad) - 1 : 31;
                const int64_t covered =
                    bad ? __shfl_sync(0xffffffffu, before, stop) : __shfl_sync(0xffffffffu, reach, 31);
                if (bad && __shfl_sync(0xffffffffu, verdict, stop) == kInvalid &&
                    __shfl_sync(0xffffffffu, j, stop) == covered + 1)
                {
                    if (lane == 0)
                        atomicMin(first, (int)(covered + 1));
                    break;
                }
                const int f = __shfl_sync(0xffffffffu, free, bad ? max(stop - 1, 0) : 0);
                stride = bad ? 1 + stride / 3 : 1 + (int64_t)f + f / 2;
                lo = covered + 1;
            }
        }
        __syncwarp();
    }
    arm_counts(ctr, evaluated, rechecks, lane);
}

// a batch that the chunk kernel checks, in the outputs or (without them) as a list
__global__ void arm_begin_kernel(const __grid_constant__ SpaceParams sp, StatesView v1, StatesView v2, int n,
                                 ArmTail *tail, int32_t *first_j, int32_t *nd_out, RunCounters *ctr)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    double a[8], b[8];
    const int nd = arm_segments(sp, v1, v2, i, a, b);
    if (tail)
    {
        tail[i] = ArmTail{(unsigned)i, 1, INT_MAX, nd};
        if (i == 0)
            ctr->deferred = (unsigned)n;
        return;
    }
    nd_out[i] = nd;
    first_j[i] = INT_MAX;
}

// results of the edges that the chunk kernel checked
__global__ void arm_finish_kernel(int n, const ArmTail *tail, uint8_t *ok, int32_t *first_j, int32_t *nd_out,
                                  const RunCounters *ctr)
{
    const int count = tail ? (int)min(ctr->deferred, (unsigned)kArmTailRoom) : n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count)
        return;
    const ArmTail t = tail ? tail[i] : ArmTail{(unsigned)i, 1, first_j[i], nd_out[i]};
    arm_write(t.e, t.first == INT_MAX ? -1 : t.first, t.nd, t.nd > 1 ? t.nd : 1, ok, first_j, nd_out);
}

template <int PREC>
static void launch_arm_motion_t(const LaunchCfg &lc, const SpaceParams &sp, const WorldArgs &wa, StatesView v1,
                                StatesView v2, int64_t n, ArmTail *tail, uint8_t *ok, int32_t *fj, int32_t *nd,
                                RunCounters *ctr)
{
    // CTAs the GPU holds (the same shared memory and registers in both kernels)
    const int full = persistent_grid((const void *)arm_motion_kernel<PREC>, 128, 0, lc, INT64_MAX / 2);
    // Few edges: a lane each would leave the GPU empty and wait for the longest edge; cut in runs instead. Runs / lanes,
    // among 1,500 spheres: 1,500 edges of 120 states 138 / 226 us, of 2..2,000 states 157 / 275 us; 4,000 edges of 12
    // states 121 / 108 us, of 120 172 / 283 us, of 2..2,000 226 / 353 us; 6,000 of 12 states 177 / 155 us, of 120 222 /
    // 245 us; 20,000 of 120 451 / 320 us.
    constexpr int kFewEdges = 4096;
    if (n <= (fj && nd ? kFewEdges : kArmTailRoom))
    {
        ArmTail *list = fj && nd ? nullptr : tail;
        arm_begin_kernel<<<(int)((n + 63) / 64), 64, 0, lc.stream>>>(sp, v1, v2, (int)n, list, fj, nd, ctr);
        const int grid = (int)std::min<int64_t>(full, (n * kArmChunks + 3) / 4);
        arm_chunk_kernel<PREC><<<grid, 128, 0, lc.stream>>>(sp, wa, v1, v2, (int)n, kArmChunks, list, fj, nd, ctr);
        arm_finish_kernel<<<(int)((n + 127) / 128), 128, 0, lc.stream>>>((int)n, list, ok, fj, nd, ctr);
    }
    else
    {
        // edges per warp: enough warps for the whole GPU first, then lanes
        int per = 1;
        while (per < 32 && n > (int64_t)full * 4 * per)
            per *= 2;
        const int grid = (int)std::min<int64_t>(full, (n + 4 * per - 1) / (4 * per));
        arm_motion_kernel<PREC><<<grid, 128, 0, lc.stream>>>(sp, wa, v1, v2, n, per, tail, ok, fj, nd, ctr);
        arm_chunk_kernel<PREC><<<full, 128, 0, lc.stream>>>(sp, wa, v1, v2, 0, kArmChunks, tail, nullptr, nullptr, ctr);
        arm_finish_kernel<<<kArmTailRoom / 128, 128, 0, lc.stream>>>(0, tail, ok, fj, nd, ctr);
    }
    for (int i = 0; i < 3; ++i)
        note_launch();
}

void launch_arm_motion(const LaunchCfg &lc, int precision, const SpaceParams &sp, const WorldArgs &wa, StatesView v1,
                       StatesView v2, int64_t n, ArmTail *tail, uint8_t *ok, int32_t *fj, int32_t *nd, RunCounters *ctr)
{
    if (precision == GBO_PRECISION_FP64)
        launch_arm_motion_t<GBO_PRECISION_FP64>(lc, sp, wa, v1, v2, n, tail, ok, fj, nd, ctr);
    else
        launch_arm_motion_t<GBO_PRECISION_FP32_GUARDED>(lc, sp, wa, v1, v2, n, tail, ok, fj, nd, ctr);
}

}  // namespace gbo
