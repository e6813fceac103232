// State evaluation of the DH arm with clearance (kernels_arm.cu): verdict of one checked state of an edge
// and the number of states on each side of it that the clearance proves free.
#pragma once
#include <cuda_fp16.h>

#include "kernels.cuh"

namespace gbo
{

// Lower bound of the distance from (x, y, z) to the nearest obstacle surface. Cells hold the distance
// from their centre less clr_margin (FP32 rounding of both sides and of the position); every obstacle
// lies at least rs inside the grid's box, which bounds points outside it. NaN for NaN.
// The approximate square root and quotient (a few ulp) are far inside clr_margin and free_steps' slack.
__device__ __forceinline__ float arm_sqrt(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float arm_clearance(const WorldArgs &wa, float x, float y, float z)
{
    const float gx = (x - wa.clr_lo[0]) * wa.clr_inv[0], gy = (y - wa.clr_lo[1]) * wa.clr_inv[1];
    const float gz = (z - wa.clr_lo[2]) * wa.clr_inv[2];
    const float N = (float)wa.clr_n, m = N - 0.5f, h = 0.5f * N;
    const float ix = floorf(fminf(fmaxf(gx, 0.f), m)), iy = floorf(fminf(fmaxf(gy, 0.f), m));
    const float iz = floorf(fminf(fmaxf(gz, 0.f), m));
    const float dx = (gx - (ix + 0.5f)) * wa.clr_cell[0], dy = (gy - (iy + 0.5f)) * wa.clr_cell[1];
    const float dz = (gz - (iz + 0.5f)) * wa.clr_cell[2];
    const float v = __half2float(wa.clr[((int)ix * wa.clr_n + (int)iy) * wa.clr_n + (int)iz]);
    float c = fmaf(v, wa.clr_unit, -arm_sqrt(fmaf(dx, dx, fmaf(dy, dy, dz * dz))));
    if (fmaxf(fabsf(gx - h), fmaxf(fabsf(gy - h), fabsf(gz - h))) > h && c == c)
    {
        // outside the box: at least the distance to it plus rs
        const float ox = (fabsf(gx - h) - h) * wa.clr_cell[0], oy = (fabsf(gy - h) - h) * wa.clr_cell[1];
        const float oz = (fabsf(gz - h) - h) * wa.clr_cell[2];
        c = fmaxf(c, fmaxf(ox, fmaxf(oy, oz)) + wa.clr_out);
    }
    return c;
}

// States within `r` of the current one that a link with slack s, speed v and acceleration bound B per step
// cannot leave: the largest r with v r + B r^2 / 2 <= s (1e-3 relative slack for the FP32 evaluation).
__device__ __forceinline__ float free_steps(float s, float v, float B)
{
    v *= 1.001f;
    B *= 1.001f;
    const float q = v + arm_sqrt(fmaf(v, v, 2.f * B * s));
    return q > 1e-20f ? fminf(__fdividef(1.998f * s, q), 1e9f) : 1e9f;
}

// the joint difference that interpolate multiplies by t (RealVector: to - from; else the shortest arc,
// with the sign that is added to `from`; adding 2 pi to an angle changes no transform)
__device__ __forceinline__ double joint_difference(const SpaceParams &sp, double a, double b)
{
    const double d = dsub(b, a);
    if (sp.kind == GBO_SPACE_REAL_VECTOR || fabs(d) <= kPi || !(d == d))
        return d;
    return d > 0.0 ? -dsub(kTwoPi, d) : -dsub(-kTwoPi, d);
}

// checked state j of an edge in FP64, as the reference interpolates it (j == top is s2 itself)
__device__ __forceinline__ double arm_angle64(const SpaceParams &sp, double a, double b, double t, bool last)
{
    if (last)
        return b;
    return sp.kind == GBO_SPACE_REAL_VECTOR ? dadd(a, dmul(dsub(b, a), t)) : interp_angle64(a, b, t);
}

static __device__ __noinline__ void arm_state64(const SpaceParams &sp, const StatesView &v1, const StatesView &v2,
                                                int64_t e, int j, int nd, int top, double *q)
{
    const double t = j == top ? 1.0 : ddiv((double)j, (double)nd);
    for (int d = 0; d < sp.dim; ++d)
        q[d] = arm_angle64(sp, v1(e, d), v2(e, d), t, j == top);
}

// Angles above this (float-float reduction of sincos_ff) and edges of more steps (j and nd exact in FP32)
// go to FP64.
constexpr float kArmMaxAngle = 96.f;
constexpr int kArmMaxSteps = 1 << 22;

// A warp's joint positions of the states its lanes evaluate, with each link's speed and acceleration bound
struct ArmChain
{
    float p[9][3][32], v[8][32], B[8][32];
};

// Clearance of one link's halves (FP32 ends p and p + ln): `steps` shrinks to what they prove free; a half
// whose spheres must be tested one by one, or that proves less than one step free, is marked.
__device__ __forceinline__ void arm_halves(const WorldArgs &wa, int i, const float *p, const float *ln, float vmax,
                                           float B, float &steps, unsigned &must, unsigned &weak)
{
    const float inv_spl = wa.arm.inv_spl;
    const int h0 = wa.arm.spl >> 1;
    const float len = 1.00001f * arm_sqrt(fmaf(ln[0], ln[0], fmaf(ln[1], ln[1], ln[2] * ln[2])));
#pragma unroll
    for (int half = 0; half < 2; ++half)
    {
        const int k0 = half ? h0 : 0, k1 = half ? wa.arm.spl : h0;
        const float f = 0.5f * (float)(k0 + k1) * inv_spl;
        const float s = arm_clearance(wa, fmaf(f, ln[0], p[0]), fmaf(f, ln[1], p[1]), fmaf(f, ln[2], p[2])) -
                        0.5f * (float)(k1 - k0 - 1) * inv_spl * len - wa.arm.rsf;
        const float fs = free_steps(fmaxf(s, 0.f), vmax, B);
        const unsigned bit = k0 < k1 ? 1u << (2 * i + half) : 0u;
        if (!(s > 0.f))
            must |= bit;
        else if (!(fs >= 1.f))
            weak |= bit;
        else if (bit)
            steps = fminf(steps, fs);
    }
}

// The marked halves' spheres, one after another per lane (a lane's own list, so that a warp runs as long
// as its longest list and not through every half that any lane marked): test(c) is the narrow phase
// of a sphere with FP32 centre c and returns kValid, kInvalid or kAmbiguous.
template <bool kDecide, class Test>
__device__ __forceinline__ int arm_spheres(const WorldArgs &wa, const ArmChain &ch, int lane, unsigned must,
                                           unsigned weak, float &steps, Test test)
{
    const float inv_spl = wa.arm.inv_spl;
    const int h0 = wa.arm.spl >> 1;
    int k = 0, k1 = 0, i = 0;
    float p[3], ln[3], v = 0.f, B = 0.f;
    bool amb = false;
    for (;;)
    {
        if (k >= k1)
        {
            // a better bound does not matter once a sphere had to be tested
            const unsigned left = must ? must : (steps >= 1.f ? weak : 0u);
            if (!left)
                break;
            const int h = __ffs(left) - 1;
            must &= ~(1u << h);
            weak &= ~(1u << h);
            i = h >> 1;
            k = h & 1 ? h0 : 0;
            k1 = h & 1 ? wa.arm.spl : h0;
#pragma unroll
            for (int r = 0; r < 3; ++r)
            {
                p[r] = ch.p[i][r][lane];
                ln[r] = ch.p[i + 1][r][lane] - p[r];
            }
            v = ch.v[i][lane];
            B = ch.B[i][lane];
        }
        const float f = ((float)k + 0.5f) * inv_spl;
        const float c[3] = {fmaf(f, ln[0], p[0]), fmaf(f, ln[1], p[1]), fmaf(f, ln[2], p[2])};
        const float s = arm_clearance(wa, c[0], c[1], c[2]) - wa.arm.rsf;
        if (s > 0.f)
            steps = fminf(steps, free_steps(s, v, B));
        else
        {
            steps = 0.f;
            const int r = test(c);
            if (r == kInvalid || (!kDecide && r == kAmbiguous))
                return r;
            amb |= r == kAmbiguous;
        }
        ++k;
    }
    return amb ? kAmbiguous : kValid;
}

// The cell of an FP32 sphere centre in the obstacle grid, or -1 outside it (no obstacle near). Cells list the
// obstacles within rs + r + a margin of their box, which covers the centre's FP32 error.
__device__ __forceinline__ int arm_cell(const WorldArgs &wa, const float *c)
{
    const int G = wa.grid_n;
    int cell[3];
    bool inside = true;
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
        const float g = floorf((c[r] - wa.glo[r]) * wa.ginv[r]);
        inside &= (g >= 0.f && g < (float)G);
        cell[r] = (int)g;
    }
    return inside ? (cell[0] * G + cell[1]) * G + cell[2] : -1;
}

// FP32 squared distance of a sphere centre to listed obstacle `it`, less the squared reach
__device__ __forceinline__ float arm_pair32(const WorldArgs &wa, const float *c, int it)
{
    const float rs = wa.arm.rsf;
    if (wa.boxes)
    {
        const float4 o = __ldg(wa.cell_items4 + 2 * it), h = __ldg(wa.cell_items4 + 2 * it + 1);
        const float dx = fmaxf(fabsf(c[0] - o.x) - o.w, 0.f), dy = fmaxf(fabsf(c[1] - o.y) - h.x, 0.f);
        const float dz = fmaxf(fabsf(c[2] - o.z) - h.y, 0.f);
        return fmaf(dz, dz, fmaf(dy, dy, dx * dx)) - rs * rs;
    }
    const float4 o = __ldg(wa.cell_items4 + it);
    const float dx = c[0] - o.x, dy = c[1] - o.y, dz = c[2] - o.z;
    const float rr = rs + o.w;
    return fmaf(dz, dz, fmaf(dy, dy, dx * dx)) - rr * rr;
}

// Checked state j of the edge in column `col` of the warp's table (start angles and differences as
// float-float): kValid (then `free`), kAmbiguous (FP64 decides) or, in the FP32-guarded form only,
// kInvalid. FP32_GUARDED: dh_valid32's decision. FP64: FP32 only proves spheres free, by the clearance or by
// the pair test's error bound; every state that may touch is decided in FP64.
// nd <= 1: the only state is s2 (t = 1).
template <int PREC>
__device__ __forceinline__ int arm_eval32(const WorldArgs &wa, ArmChain &ch, int lane, const float (*edge)[32],
                                          int col, int j, int nd, int &free)
{
    const DHArm &arm = wa.arm;
    if (nd > kArmMaxSteps)
        return kAmbiguous;
    const float ndf = (float)(nd > 1 ? nd : 1);
    const float inv_hi = __frcp_rn(ndf), inv_lo = fmaf(-inv_hi, ndf, 1.0f) * inv_hi;
    const float jf = (float)j;
    const float t_hi = jf * inv_hi, t_lo = fmaf(jf, inv_hi, -t_hi) + jf * inv_lo;
    float R[3][3] = {{1.f, 0.f, 0.f}, {0.f, 1.f, 0.f}, {0.f, 0.f, 1.f}};
    float p[3] = {0.f, 0.f, 0.f}, om[3] = {0.f, 0.f, 0.f}, vel[3] = {0.f, 0.f, 0.f};
    float W = 0.f, B = 0.f, speed = 0.f, steps = 1e9f;
    unsigned must = 0, weak = 0;
#pragma unroll
    for (int r = 0; r < 3; ++r)
        ch.p[0][r][lane] = 0.f;
#pragma unroll 1
    for (int i = 0; i < arm.joints; ++i)
    {
        const ff A{edge[4 * i][col], edge[4 * i + 1][col]}, D{edge[4 * i + 2][col], edge[4 * i + 3][col]};
        const float p_hi = D.hi * t_hi;
        const float p_lo = fmaf(D.hi, t_hi, -p_hi) + fmaf(D.hi, t_lo, D.lo * t_hi);
        const ff q = ff_add(A, ff{p_hi, p_lo});
        if (!(fabsf(q.hi) <= kArmMaxAngle))
            return kAmbiguous;
        float cq, sq;
        sincos_ff(q, cq, sq);
        const float ca = arm.ca[i], sa = arm.sa[i], a = arm.af[i], d = arm.dfl[i];
        // joint rate per step, about R's third column
        const float u = D.hi * inv_hi;
        W += fabsf(u);
        B = fmaf(1.5f * W * W, arm.len[i], B);
        float ln[3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
        {
            om[r] = fmaf(u, R[r][2], om[r]);
            // columns of R * A: (c, s, 0), (-s ca, c ca, sa), (s sa, -c sa, ca)
            const float x = fmaf(R[r][1], sq, R[r][0] * cq), y = fmaf(R[r][1], cq, -R[r][0] * sq), z = R[r][2];
            ln[r] = fmaf(z, d, x * a);
            R[r][0] = x;
            R[r][1] = fmaf(z, sa, y * ca);
            R[r][2] = fmaf(z, ca, -y * sa);
        }
        vel[0] += om[1] * ln[2] - om[2] * ln[1];
        vel[1] += om[2] * ln[0] - om[0] * ln[2];
        vel[2] += om[0] * ln[1] - om[1] * ln[0];
        const float ns = arm_sqrt(fmaf(vel[0], vel[0], fmaf(vel[1], vel[1], vel[2] * vel[2])));
        const float vmax = fmaxf(speed, ns);
        speed = ns;
        arm_halves(wa, i, p, ln, vmax, B, steps, must, weak);
        ch.v[i][lane] = vmax;
        ch.B[i][lane] = B;
#pragma unroll
        for (int r = 0; r < 3; ++r)
        {
            p[r] += ln[r];
            ch.p[i + 1][r][lane] = p[r];
        }
    }
    constexpr bool kDecide = PREC == GBO_PRECISION_FP32_GUARDED;
    const float E = wa.dh_e;
    const int verdict = arm_spheres<kDecide>(wa, ch, lane, must, weak, steps, [&](const float *c) {
        const int cell = arm_cell(wa, c);
        if (cell < 0)
            return (int)kValid;
        const int b = __ldg(wa.cell_start + cell), e = __ldg(wa.cell_start + cell + 1);
        bool amb = false;
        for (int it = b; it < e; ++it)
        {
            const float t = arm_pair32(wa, c, it);
            if (kDecide && t < -E)
                return (int)kInvalid;
            amb |= !(t > E);
            if (!kDecide && amb)
                break;
        }
        return (int)(amb ? kAmbiguous : kValid);
    });
    free = (int)steps;
    return verdict;
}

}  // namespace gbo
