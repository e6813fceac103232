// State sampling: RealVectorStateSampler::sampleUniform / sampleUniformNear and SO2StateSampler
// (RealVectorStateSpace.cpp:45-65, SO2StateSpace.cpp:46-56) over one sampler's RNG stream.
//
// The stream is OMPL's RNG (RandomNumbers.h:66-76): std::mt19937 -> libstdc++
// generate_canonical<double, 53> (two 32-bit draws w0, w1: (w0 + w1 * 2^32) / 2^64, values >= 1
// replaced by the largest double below 1) -> uniformReal(lo, hi) = (hi - lo) * U + lo.
// mt19937 (Matsumoto & Nishimura 1998) is sequential across 624-word blocks. Calls of fewer than 2^18
// stream words run on one CTA that produces the sampler's word stream (mt_words_kernel) while the
// whole GPU converts word pairs into coordinates (words_to_states_kernel); larger calls cut their
// stretch of the stream into segments that start from jump-ahead windows and run side by side (below).
// sampleGaussian (further below) draws its polar candidates' words the same two ways.
#include <algorithm>
#include <cmath>

#include "crlog.cuh"
#include "kernels_nn.cuh"

namespace gbo
{

__device__ __forceinline__ unsigned temper(unsigned y)
{
    y ^= y >> 11;
    y ^= (y << 7) & 0x9d2c5680u;
    y ^= (y << 15) & 0xefc60000u;
    y ^= y >> 18;
    return y;
}

__device__ __forceinline__ unsigned twist_word(unsigned cur, unsigned next, unsigned far)
{
    const unsigned y = (cur & 0x80000000u) | (next & 0x7fffffffu);
    return far ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
}

__device__ __forceinline__ double canonical53(unsigned w0, unsigned w1)
{
    double sum = (double)w0;
    sum = __dadd_rn(sum, __dmul_rn((double)w1, 4294967296.0));
    double r = __dmul_rn(sum, 5.421010862427522170037264e-20);  // / 2^64 (exact power of two)
    if (r >= 1.0)
        r = 0.99999999999999988897769753748;                   // nextafter(1, 0)
    return r;
}

// The recurrence on the stream's own index: with x_0 .. x_623 the generator's block, the next words are
// x_n = x_(n-227) ^ f(x_(n-624), x_(n-623)), n >= 624. Thread t < 227 produces n = 624 + t, then every
// 227th: x_(n-227) is the word it produced last (a register), and the words n and n + 227 of one step need
// nothing later than x_(n-170), so a step makes 454 words between two barriers. The words live in a ring of
// four steps in shared memory (word n at slot mt_slot(n)), so each thread's addresses repeat every fourth
// step and are kept in registers. Bound by the chain barrier, load, f, store, barrier; the recurrence in
// blocks had three barriers to 624 words (one CTA, 240,000 words: 129 -> 53 us; 153 segments of 2^17 words:
// 60 us with tempering, now 25 without).
constexpr int kMtLag = 227, kMtStep = 2 * kMtLag, kMtRing = 4 * kMtStep;
static_assert(kMtRing >= 624 + kMtStep, "a step's inputs and outputs fit in the ring");

__device__ __forceinline__ int mt_slot(int64_t n)  // n >= 0; the block's words 0 .. 623 end the ring
{
    return (int)((n + kMtRing - 624) % kMtRing);
}

// Words [624, make) of the stream after the block in the ring (whole steps); those below keep are stored
// at o + n. Every thread of the CTA (at least 227) calls it; the ring is complete on return.
template <bool kTemper>
__device__ __forceinline__ void mt_run(unsigned *ring, int64_t make, int64_t keep, unsigned *o)
{
    const int t = threadIdx.x;
    const bool act = t < kMtLag;
    int in[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        const int at[4] = {624, 623, 397, 396};
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            const int r = kMtStep * j + (act ? t : 0) - at[q];
            in[j][q] = r < 0 ? r + kMtRing : r;
        }
    }
    unsigned v0 = 0u, v1 = act ? ring[mt_slot(397 + t)] : 0u;
    auto step = [&](int j) {
        const unsigned a = ring[in[j][0]], b = ring[in[j][1]], c = ring[in[j][2]], d = ring[in[j][3]];
        v0 = twist_word(a, b, v1);
        v1 = twist_word(c, d, v0);
        if (act)
        {
            ring[kMtStep * j + t] = v0;
            ring[kMtStep * j + kMtLag + t] = v1;
        }
        __syncthreads();
    };
    int64_t n = 624;
    unsigned *w = o + n + t;
    // whole rounds without a test; a step's words are stored after its barrier, under the next step's loads
    for (const int64_t whole = min(make, keep) - kMtRing; n <= whole; n += kMtRing, w += kMtRing)
    {
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            step(j);
            if (act)
            {
                w[kMtStep * j] = kTemper ? temper(v0) : v0;
                w[kMtStep * j + kMtLag] = kTemper ? temper(v1) : v1;
            }
        }
    }
    for (; n < make; n += kMtRing, w += kMtRing)  // the rest: make may be up to a block beyond keep
    {
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            if (n + kMtStep * j >= make)
                return;
            step(j);
            if (act && n + kMtStep * j + t < keep)
                w[kMtStep * j] = kTemper ? temper(v0) : v0;
            if (act && n + kMtStep * j + kMtLag + t < keep)
                w[kMtStep * j + kMtLag] = kTemper ? temper(v1) : v1;
        }
    }
}

// The word stream: one CTA continues the stream at st->pos and writes its next W tempered words to
// out, then saves the generator.
// kRaw (speculative draws): the words are stored untempered, every new block is stored whole (up to
// W + 623 words) and the generator is left unchanged, so that any prefix of the stream can later be
// committed by copying the block that holds its last word (gauss_advance_kernel).
template <bool kRaw>
__global__ void __launch_bounds__(256) mt_words_kernel(SamplerState *st, int64_t W, unsigned *out)
{
    __shared__ unsigned ring[kMtRing];
    const int t = threadIdx.x;
    for (int i = t; i < 624; i += blockDim.x)
        ring[mt_slot(i)] = st->mt[i];
    const int pos = (int)st->pos;  // next unused word of the block (624: none)
    __syncthreads();
    const int64_t end = pos + W;            // words [pos, end) of the stream
    const int64_t block = (end - 1) / 624;  // the block of the last one
    const int64_t whole = 624 * (block + 1);
    for (int i = pos + t; i < 624 && i < end; i += blockDim.x)
        out[i - pos] = kRaw ? ring[mt_slot(i)] : temper(ring[mt_slot(i)]);
    mt_run<!kRaw>(ring, whole, kRaw ? whole : end, out - pos);
    if (kRaw)
        return;
    for (int i = t; i < 624; i += blockDim.x)
        st->mt[i] = ring[mt_slot(624 * block + i)];
    if (t == 0)
        st->pos = (unsigned)(end - 624 * block);
}

// Values v0 .. v0 + nv - 1 of a sampling call (value v = coordinate v % dim of state v / dim) from the
// word pairs (2m, 2m + 1), m = v - v0, of the word stream: generate_canonical<double, 53> and
// uniformReal (or the near bounds), across the whole GPU.
__global__ void __launch_bounds__(256) words_to_states_kernel(const unsigned *words, int64_t v0, int64_t nv,
                                                              SpaceParams sp, StatesView nearv, int use_near,
                                                              double distance, MutStatesView out)
{
    for (int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; m < nv; m += (int64_t)gridDim.x * blockDim.x)
    {
        const double U = canonical53(words[2 * m], words[2 * m + 1]);
        const int64_t v = v0 + m;
        const int64_t i = v / sp.dim;
        const int d = (int)(v - i * sp.dim);
        double lo, hi;
        if (use_near)
        {
            const double c = nearv(i, d);
            if (sp.kind == GBO_SPACE_SO2)
            {
                lo = __dsub_rn(c, distance);
                hi = __dadd_rn(c, distance);
            }
            else
            {
                lo = fmax(sp.low[d], __dsub_rn(c, distance));
                hi = fmin(sp.high[d], __dadd_rn(c, distance));
            }
        }
        else
        {
            lo = sp.low[d];
            hi = sp.high[d];
        }
        double x = __dadd_rn(__dmul_rn(__dsub_rn(hi, lo), U), lo);
        if (use_near && sp.kind == GBO_SPACE_SO2)
        {
            // SO2StateSpace::enforceBounds (SO2StateSpace.cpp:79-87)
            double y = fmod(x, 2.0 * kPi);
            if (y < -kPi)
                y = __dadd_rn(y, 2.0 * kPi);
            else if (y >= kPi)
                y = __dsub_rn(y, 2.0 * kPi);
            x = y;
        }
        out(i, d) = x;
    }
}

void launch_sample_uniform(const LaunchCfg &lc, SamplerState *st, const SpaceParams &sp, const double *near,
                           StatesView nearv, double distance, int64_t n, MutStatesView out, unsigned *words,
                           int64_t cap_words)
{
    const int64_t total = n * sp.dim, chunk = cap_words / 2;
    for (int64_t v0 = 0; v0 < total; v0 += chunk)
    {
        const int64_t nv = std::min(chunk, total - v0);
        mt_words_kernel<false><<<1, 256, 0, lc.stream>>>(st, 2 * nv, words);
        const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((nv + 255) / 256, (int64_t)lc.sm_count * 8));
        words_to_states_kernel<<<grid, 256, 0, lc.stream>>>(words, v0, nv, sp, nearv, near != nullptr, distance, out);
        note_launch();
        note_launch();
    }
}

// ---------------------------------------------------------------- segmented stream (jump-ahead)
// Calls of many values cut their stretch of the stream, words [0, W) counted from the sampler's next
// word T0, into segments of L words (L even, so no value's word pair is split): segment s starts from
// the generator window at T0 - 1 + s L (position 1 of that window: its word 0 only carries its top
// bit). Window 0 is the sampler's own state. Window s >= 1 is A^(sL) applied to the window at T0 - 1
// (mt_jump.cu): with p = x^(sL) mod phi, its word w is the XOR over the set coefficients i of p of
// u_(i+w), u_t = x_(T0-1+t). One CTA per segment then runs the recurrence over its words and converts
// them to coordinates, so the call runs at the width of the GPU instead of one CTA's recurrence.

// RN(w1 * 2^32 + w0) / 2^64 (generate_canonical's value) in integer arithmetic: the same double as
// canonical53, including the largest double below 1 for sums that round up to 2^64.
__device__ __forceinline__ double canonical53_int(unsigned w0, unsigned w1)
{
    if (w1 == 0u)  // below 2^-32: the sum is exact
        return __dmul_rn((double)w0, 5.421010862427522170037264e-20);
    const int z = __clz((int)w1);
    const unsigned hi = __funnelshift_l(w0, w1, z), lo = w0 << z;  // leading one at bit 63
    // round to 53 bits, ties to even; value in [2^(-1-z), 2^-z), the leading one added to the exponent (a
    // carry out of the mantissa makes it a power of two)
    const unsigned inc = ((lo & 0x7ffu) + 0x3ffu + ((lo >> 11) & 1u)) >> 11;
    const unsigned long long b = ((unsigned long long)(hi >> 11) << 32 | __funnelshift_r(lo, hi, 11)) +
                                 ((unsigned long long)((1021u - (unsigned)z) << 20) << 32) + inc;
    return b == 0x3ff0000000000000ull ? 0.99999999999999988897769753748  // rounded to 1: nextafter(1, 0)
                                      : __longlong_as_double((long long)b);
}

// A factor prepared for span_times_canonical: its 53-bit mantissa with the leading one at bit 63 (0: not
// a normal number, or too small for every product to be one) and the rest as the bits of a power of two.
struct SpanFactor
{
    unsigned mant_hi, mant_lo;
    unsigned base;  // sign and exponent: the high word of +-2^e
    double value;
};

__device__ __forceinline__ SpanFactor span_factor(double v)
{
    const unsigned long long a = (unsigned long long)__double_as_longlong(v);
    const int e = (int)(a >> 52) & 0x7ff;
    const bool fits = e >= 66 && e != 0x7ff;  // U is 0 or at least 2^-64
    const unsigned long long m = fits ? (a << 11) | (1ull << 63) : 0ull;
    return {(unsigned)(m >> 32), (unsigned)m, (unsigned)(a >> 32) & 0xfff00000u, v};
}

// RN(span * U), U = generate_canonical's value for the word pair: both roundings to 53 bits on the integer
// pipe (an FP64 instruction holds an SM's pipe for 16 cycles). Factors that do not fit, a high word 0 and a U
// that rounds up to a power of two go through the doubles.
__device__ __forceinline__ double span_times_canonical(const SpanFactor &f, unsigned w0, unsigned w1)
{
    const int z = __clz((int)w1);
    const unsigned mh = __funnelshift_l(w0, w1, z), ml = w0 << (z & 31);  // w1 != 0: leading one at bit 63
    // U's mantissa: 53 bits at the top, ties to even
    const unsigned long long u =
        ((((unsigned long long)mh << 32) | (ml & 0xfffff800u)) +
         (((ml & 0x7ffu) + 0x3ffu + ((ml >> 11) & 1u)) & 0x800u));
    const unsigned uh = (unsigned)(u >> 32), ul = (unsigned)u;
    if (w1 == 0u || uh == 0u || f.mant_hi == 0u)
        return __dmul_rn(f.value, canonical53_int(w0, w1));
    // the 128-bit product of the mantissas, in [2^126, 2^128); no partial sum exceeds 64 bits
    const unsigned long long p0 = (unsigned long long)f.mant_lo * ul;
    const unsigned long long p1 = (unsigned long long)f.mant_lo * uh + (unsigned)(p0 >> 32);
    const unsigned long long p2 = (unsigned long long)f.mant_hi * ul + (unsigned)p1;
    const unsigned long long p3 = (unsigned long long)f.mant_hi * uh + ((p1 >> 32) + (p2 >> 32));
    unsigned h1 = (unsigned)(p3 >> 32), h0 = (unsigned)p3, l1 = (unsigned)p2;
    const unsigned down = (~h1) >> 31;  // product of the mantissas below 2: one bit lower
    h1 = __funnelshift_l(h0, h1, down);
    h0 = __funnelshift_l(l1, h0, down);
    l1 <<= down;
    const unsigned sticky = (l1 | (unsigned)p0) != 0u ? 1u : 0u;
    const unsigned inc = ((h0 & 0x7ffu) + 0x3ffu + (((h0 >> 11) & 1u) | sticky)) >> 11;
    // span = +-2^e times its mantissa, U = 2^(-1 - z) times its own: exponent e - z - down, less one because the
    // mantissa's leading one is added to it (a carry out of the rounded mantissa goes the same way)
    const unsigned long long m = (((unsigned long long)(h1 >> 11) << 32) | __funnelshift_r(h0, h1, 11)) + inc;
    const unsigned top = f.base - ((unsigned)(z + 1) << 20) - (down << 20);
    return __longlong_as_double((long long)(m + ((unsigned long long)top << 32)));
}

// Coordinate d of state i of a sampleUniformNear call from generate_canonical's U.
__device__ __forceinline__ double near_value(int64_t i, int d, double U, const SpaceParams &sp, StatesView nearv,
                                             double distance)
{
    const double c = nearv(i, d);
    double lo, hi;
    if (sp.kind == GBO_SPACE_SO2)
    {
        lo = __dsub_rn(c, distance);
        hi = __dadd_rn(c, distance);
    }
    else
    {
        lo = fmax(sp.low[d], __dsub_rn(c, distance));
        hi = fmin(sp.high[d], __dadd_rn(c, distance));
    }
    double x = __dadd_rn(__dmul_rn(__dsub_rn(hi, lo), U), lo);
    if (sp.kind == GBO_SPACE_SO2)
    {
        // SO2StateSpace::enforceBounds (SO2StateSpace.cpp:79-87)
        double y = fmod(x, 2.0 * kPi);
        if (y < -kPi)
            y = __dadd_rn(y, 2.0 * kPi);
        else if (y >= kPi)
            y = __dsub_rn(y, 2.0 * kPi);
        x = y;
    }
    return x;
}

// u_t = x_(T0-1+t), t < kJumpU, is what the jumps read: coefficients below 19968 + 32, words below 624
constexpr int64_t kJumpU = 19968 + 704;

// Windows of a call's nseg segments: the sampler's block and position (625 words), then words w of
// windows 1 .. nseg - 1 at w * ldw + window - 1 (side by side, so that a warp's 32 windows share a line).
__host__ __device__ inline int window_stride(int nseg)
{
    return (nseg - 1 + 31) & ~31;
}

// CTA 0: u and the sampler's block; the others clear the windows that the jumps add to.
__global__ void __launch_bounds__(256) mt_window_seq_kernel(const SamplerState *st, unsigned *u, unsigned *windows,
                                                            int cleared)
{
    const int t = threadIdx.x;
    if (blockIdx.x > 0)
    {
        for (int i = (blockIdx.x - 1) * 256 + t; i < cleared; i += (gridDim.x - 1) * 256)
            windows[625 + i] = 0u;
        return;
    }
    __shared__ unsigned ring[kMtRing];
    const int pos = (int)st->pos;  // 1..624
    for (int i = t; i < 624; i += blockDim.x)
    {
        const unsigned v = st->mt[i];
        ring[mt_slot(i)] = v;
        windows[i] = v;
        if (i >= pos - 1)
            u[i - (pos - 1)] = v;
    }
    if (t == 0)
        windows[624] = (unsigned)pos;
    __syncthreads();
    mt_run<false>(ring, kJumpU + pos - 1, kJumpU + pos - 1, u - (pos - 1));
}

// Windows 1..K by table lookup ("four Russians"): coefficients are taken 5 at a time (group g covers
// i = 5g .. 5g + 4), and for each stream position p the 32 XOR combinations of u[p .. p + 4] are tabulated:
// word w of a window adds, for group g, the entry of position 5g + w that the window's 5 coefficient bits
// select. A CTA covers kJW window words, one range of groups in phases of kJGB, and up to 32 NW windows
// (one thread per window, kJW accumulators each). The phase's groups and words share their positions:
// 5 (kJGB - 1) + kJW tables serve kJGB kJW lookups per window, so a call of one warp of windows spends 16% of
// its shared-memory accesses on building and one of five warps 3% (a table per group and word: 1 in 5 at
// five warps, half of them at one). Entry h of position p sits at word 33 p + h: the 32 lanes of a lookup
// (one p, any h) hit 32 banks or the same word, and so does a build (lane h). Bound by the lookups' shared-
// memory wavefronts, K 624 3988 / 32 of them: 1M 10-D states (K = 152) 83 -> 60 us (74% of the
// wavefront rate), 100,000 7-D Gaussian states (K = 55) 106 -> 28 us. Partial results go to the windows
// (zeroed before) by atomicXor, 32 windows to a line.
constexpr int kJG = 5;                                 // coefficients per lookup
constexpr int kJGroups = (19937 + kJG - 1) / kJG;      // 3988 groups (bits past 19936 are zero)
constexpr int kJGB = 16;                               // groups per phase: 80 coefficients, 2.5 words
constexpr int kJPhases = (kJGroups + kJGB - 1) / kJGB; // 250
constexpr int kJW = 48;                                // window words per CTA (624 = 13 * 48)
constexpr int kJumpWarps = 20;                         // warps per SM the grid aims at
constexpr int kJTables = kJG * (kJGB - 1) + kJW;       // positions tabulated per phase
static_assert(kJG * kJGB * kJPhases + 624 + kJG <= kJumpU, "every position a phase tabulates is in u");

// grid: (624 / kJW, ranges of per phases, window chunks)
template <int NW>
__global__ void __launch_bounds__(32 * NW) mt_jump_kernel(const unsigned *u, const unsigned *polys, int K, int ldw,
                                                          int per, unsigned *windows)
{
    __shared__ unsigned tab[33 * kJTables];
    constexpr int kPerWarp = (kJTables + NW - 1) / NW;
    const int w0 = blockIdx.x * kJW;
    const int p0 = blockIdx.y * per, p1 = min(p0 + per, kJPhases);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int k = blockIdx.z * 32 * NW + t;
    unsigned mask[kJG];
#pragma unroll
    for (int j = 0; j < kJG; ++j)
        mask[j] = 0u - ((unsigned)(lane >> j) & 1u);
    unsigned acc[kJW];
#pragma unroll
    for (int w = 0; w < kJW; ++w)
        acc[w] = 0u;
    // the 80 coefficient bits of a phase start at bit 0 or 16 of word 2.5 p (zero past word 623)
    const unsigned *crow = polys + (size_t)min(k, K - 1) * 624;
    auto coefficients = [&](int p, unsigned(&c)[4]) {
        const int q = (kJG * kJGB * p) >> 5;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            c[j] = q + j < 624 ? crow[q + j] : 0u;
    };
    unsigned next[4];
    coefficients(min(p0, kJPhases - 1), next);
#pragma unroll 1
    for (int p = p0; p < p1; ++p)
    {
        const int sh = (p & 1) * 16;
        const unsigned c[4] = {__funnelshift_r(next[0], next[1], sh), __funnelshift_r(next[1], next[2], sh),
                               __funnelshift_r(next[2], next[3], sh), 0u};
        if (p + 1 < p1)
            coefficients(p + 1, next);
        {
            const int first = warp * kPerWarp, last = min(first + kPerWarp, kJTables);
            const unsigned *x = u + kJG * kJGB * p + w0 + first;
            unsigned *T = tab + 33 * first + lane;
            unsigned r0 = x[0], r1 = x[1], r2 = x[2], r3 = x[3];
#pragma unroll 8
            for (int i = 0; i < last - first; ++i)
            {
                const unsigned r4 = x[i + 4];
                T[33 * i] = (r0 & mask[0]) ^ (r1 & mask[1]) ^ (r2 & mask[2]) ^ (r3 & mask[3]) ^ (r4 & mask[4]);
                r0 = r1;
                r1 = r2;
                r2 = r3;
                r3 = r4;
            }
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < kJGB; e += 2)  // two groups to one three-way XOR
        {
            const int b0 = kJG * e, b1 = b0 + kJG;
            const unsigned h0 = __funnelshift_r(c[b0 >> 5], c[(b0 >> 5) + 1], b0 & 31) & 31u;
            const unsigned h1 = __funnelshift_r(c[b1 >> 5], c[(b1 >> 5) + 1], b1 & 31) & 31u;
            const unsigned *T0 = tab + 33 * kJG * e + h0, *T1 = tab + 33 * kJG * (e + 1) + h1;
#pragma unroll
            for (int w = 0; w < kJW; ++w)
                acc[w] ^= T0[33 * w] ^ T1[33 * w];
        }
        __syncthreads();
    }
    if (k < K)
    {
        unsigned *o = windows + 625 + (size_t)w0 * ldw + k;
#pragma unroll
        for (int w = 0; w < kJW; ++w)
            atomicXor(o + (size_t)w * ldw, acc[w]);
    }
}

template <int NW>
static void launch_jump_t(const LaunchCfg &lc, const unsigned *u, const uint32_t *polys, int K, int ldw,
                          unsigned *windows)
{
    // ranges of phases fill the SMs with up to kJumpWarps warps each (12 warps: 61 us at K = 152, 20: 60)
    const int chunks = 624 / kJW * ((K + 32 * NW - 1) / (32 * NW));
    const int ctas = lc.sm_count * std::max(1, kJumpWarps / NW);
    const int ranges = std::max(1, std::min(kJPhases, ctas / chunks));
    const int per = (kJPhases + ranges - 1) / ranges;
    mt_jump_kernel<NW><<<dim3(624 / kJW, (kJPhases + per - 1) / per, (K + 32 * NW - 1) / (32 * NW)), 32 * NW, 0,
                         lc.stream>>>(u, polys, K, ldw, per, windows);
}

// The windows of nseg segments after the sampler's next word, in scratch; returns their address.
static const unsigned *launch_windows(const LaunchCfg &lc, const SamplerState *st, const uint32_t *polys, int nseg,
                                      unsigned *scratch)
{
    const int K = nseg - 1, ldw = window_stride(nseg);
    unsigned *u = scratch, *windows = scratch + kJumpU;
    const int cleared = 624 * ldw;
    mt_window_seq_kernel<<<1 + std::min((cleared + 1023) / 1024, lc.sm_count), 256, 0, lc.stream>>>(st, u, windows,
                                                                                                    cleared);
    note_launch();
    if (K > 0)
    {
        switch (std::min(8, (K + 31) / 32))
        {
        case 1: launch_jump_t<1>(lc, u, polys, K, ldw, windows); break;
        case 2: launch_jump_t<2>(lc, u, polys, K, ldw, windows); break;
        case 3: launch_jump_t<3>(lc, u, polys, K, ldw, windows); break;
        case 4: launch_jump_t<4>(lc, u, polys, K, ldw, windows); break;
        case 5: launch_jump_t<5>(lc, u, polys, K, ldw, windows); break;
        case 6: launch_jump_t<6>(lc, u, polys, K, ldw, windows); break;
        case 7: launch_jump_t<7>(lc, u, polys, K, ldw, windows); break;
        default: launch_jump_t<8>(lc, u, polys, K, ldw, windows); break;
        }
        note_launch();
    }
    return windows;
}

// One CTA per segment s: words [s L, min((s + 1) L, W)) of the call from window s, untempered, stored as the
// recurrence produces them (word j of the call at words[j]; tempering here took as long as the recurrence,
// 42 us against 25 for 153 segments of 2^17 words, and a few instructions where the words are read). kSave: the
// last segment leaves its generator in st; sampleGaussian's draws are speculative and committed afterwards.
template <bool kSave>
__global__ void __launch_bounds__(256) mt_segment_kernel(SamplerState *st, const unsigned *windows, int64_t L,
                                                         int64_t W, int nseg, unsigned *words)
{
    __shared__ unsigned ring[kMtRing];
    const int t = threadIdx.x, s = blockIdx.x;
    const unsigned *src = s == 0 ? windows : windows + 625 + (s - 1);
    const size_t stride = s == 0 ? 1 : (size_t)window_stride(nseg);
    for (int i = t; i < 624; i += blockDim.x)
        ring[mt_slot(i)] = src[i * stride];
    const int pos = s == 0 ? (int)windows[624] : 1;
    __syncthreads();
    const int64_t begin = (int64_t)s * L, end = pos + min(begin + L, W) - begin;
    const bool last = kSave && s == nseg - 1;
    const int64_t block = (end - 1) / 624;  // the block of the segment's last word
    unsigned *o = words + begin - pos;
    for (int i = pos + t; i < 624 && i < end; i += blockDim.x)
        o[i] = ring[mt_slot(i)];
    mt_run<false>(ring, last ? 624 * (block + 1) : end, end, o);
    if (last)
    {
        for (int i = t; i < 624; i += blockDim.x)
            st->mt[i] = ring[mt_slot(624 * block + i)];
        if (t == 0)
            st->pos = (unsigned)(end - 624 * block);
    }
}

// The call's values from the stored word pairs (value v = coordinate v % dim of state v / dim from pair v):
// tempering, generate_canonical in integer arithmetic, then uniformReal (or the near bounds), lanes over
// consecutive values. Bound by the integer pipe and the FP64 addition; with the product on the FP64 pipe it
// was bound there (1M 10-D states: 52 us on words already tempered, now 48 with the tempering). (Tiles of 128
// states turned in shared memory, for whole lines written to a coordinate-major output, took 58 us: the L2 merges
// the sectors, the barriers cost more.)
template <bool kNear>
__global__ void __launch_bounds__(256) pairs_to_states_kernel(const uint2 *pairs, int64_t nv, SpaceParams sp,
                                                              StatesView nearv, double distance,
                                                              MutStatesView out)
{
    __shared__ SpanFactor span[GBO_MAXD];
    __shared__ double low[GBO_MAXD];
    for (int d = threadIdx.x; d < sp.dim; d += blockDim.x)
    {
        span[d] = span_factor(__dsub_rn(sp.high[d], sp.low[d]));
        low[d] = sp.low[d];
    }
    __syncthreads();
    // this thread's values step by the grid: state and coordinate are carried instead of divided out
    const unsigned step = gridDim.x * blockDim.x, first = blockIdx.x * blockDim.x + threadIdx.x;
    const int di = (int)(step / (unsigned)sp.dim), dd = (int)(step % (unsigned)sp.dim);
    int64_t i = first / (unsigned)sp.dim;
    int d = (int)(first % (unsigned)sp.dim);
    double *o = &out(i, d);
    const int64_t hop = di * out.si + dd * out.sd, wrap = out.si - sp.dim * out.sd;
    uint2 next = first < nv ? pairs[first] : uint2{0u, 0u};
    for (int64_t m = first; m < nv; m += step)
    {
        const unsigned w0 = temper(next.x), w1 = temper(next.y);
        if (m + step < nv)
            next = pairs[m + step];
        *o = kNear ? near_value(i, d, canonical53_int(w0, w1), sp, nearv, distance)
                   : __dadd_rn(span_times_canonical(span[d], w0, w1), low[d]);
        i += di;
        d += dd;
        o += hop;
        if (d >= sp.dim)
        {
            d -= sp.dim;
            ++i;
            o += wrap;
        }
    }
}

int64_t sample_jump_words(int64_t nseg, int64_t W)
{
    return kJumpU + 625 + 624 * (int64_t)window_stride((int)nseg) + 4 + W;
}

void launch_sample_uniform_jump(const LaunchCfg &lc, SamplerState *st, const SpaceParams &sp, const double *near,
                                StatesView nearv, double distance, int64_t n, MutStatesView out, unsigned *scratch,
                                const uint32_t *polys, int64_t L, int nseg)
{
    const int64_t values = n * sp.dim, W = 2 * values;
    const unsigned *windows = launch_windows(lc, st, polys, nseg, scratch);
    unsigned *words = scratch + kJumpU + 625 + 624 * (int64_t)window_stride(nseg);
    words += (4 - ((uintptr_t)words / 4) % 4) % 4;  // 16-byte aligned
    mt_segment_kernel<true><<<nseg, 256, 0, lc.stream>>>(st, windows, L, W, nseg, words);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((values + 255) / 256, (int64_t)lc.sm_count * 16));
    (near ? pairs_to_states_kernel<true> : pairs_to_states_kernel<false>)<<<grid, 256, 0, lc.stream>>>(
        (const uint2 *)words, values, sp, nearv, distance, out);
    note_launch();
    note_launch();
}

// The next W raw (untempered) words of the stream after the sampler's next word into raw[0 .. W), the
// generator unchanged: the segmented generation of sampleUniform without the conversion.
static void launch_raw_words_jump(const LaunchCfg &lc, const SamplerState *st, int64_t W, unsigned *raw,
                                  unsigned *scratch, const uint32_t *polys, int64_t L)
{
    const int nseg = (int)((W + L - 1) / L);
    const unsigned *windows = launch_windows(lc, st, polys, nseg, scratch);
    mt_segment_kernel<false><<<nseg, 256, 0, lc.stream>>>(nullptr, windows, L, W, nseg, raw);
    note_launch();
}

// ---------------------------------------------------------------- sampleGaussian
// RealVectorStateSampler::sampleGaussian (RealVectorStateSpace.cpp:67-82: per coordinate
// rng_.gaussian(mean, stdDev) clamped to the bounds) and SO2StateSampler::sampleGaussian
// (SO2StateSpace.cpp:58-62: wrapped by enforceBounds). RNG::gaussian (RandomNumbers.h:98-101) is
// libstdc++'s normal_distribution, the polar method of Marsaglia and Bray (1964) with a cached pair:
// a candidate takes two uniform01 draws (4 stream words), x = 2U - 1, y = 2V - 1, r2 = x^2 + y^2, and is
// rejected while r2 > 1 or r2 == 0; an accepted one gives mult = sqrt(-2 log(r2) / r2) and the values
// y * mult (returned) then x * mult (cached for the next draw of the same RNG, across calls).
// Every operation is the same IEEE double operation except log, which is log_rn (crlog.cuh, rounded
// to nearest); glibc's log differs from the correctly rounded value in the last bit for a small
// fraction of arguments, and only the values of those pairs differ (by an ulp or two).
//
// Stream consumption is data dependent, so a chunk draws a bounded surplus of candidates
// speculatively (raw words, generator unchanged), evaluates every accepted candidate's pair once
// (gauss_pairs_kernel), ranks the CTAs' counts (gauss_scan_kernel), places the pairs the call needs
// (gauss_emit_kernel) and then commits exactly the words used (gauss_advance[_seg]_kernel).
constexpr int kGaussPerCta = 1024;  // candidates per CTA: 256 threads x 4

// 2U - 1 rounded to nearest for a generate_canonical value U in [0, 1): 2U by the exponent (exact; U is
// 0 or at least 2^-64), then one FP64 subtraction.
__device__ __forceinline__ double two_u_minus_1(double U)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(U);
    return __dsub_rn(__longlong_as_double((long long)(b ? b + (1ull << 52) : 0ull)), 1.0);
}

// The polar method's candidate from four stream words: generate_canonical in integer arithmetic (the
// same doubles as canonical53), and the rejection test r2 > 1 || r2 == 0 on the bits (r2 >= +0).
__device__ __forceinline__ bool polar_candidate(uint4 w, double &x, double &y, double &r2)
{
    x = two_u_minus_1(canonical53_int(temper(w.x), temper(w.y)));
    y = two_u_minus_1(canonical53_int(temper(w.z), temper(w.w)));
    r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
    const unsigned long long rb = (unsigned long long)__double_as_longlong(r2);
    return rb != 0ull && rb <= 0x3FF0000000000000ull;
}

// a < b for doubles as IEEE compares them, on the integer pipe (the FP64 pipe is this kernel's bound):
// false when either is NaN or both are zeros, else the order of the sign-magnitude bit patterns.
__device__ __forceinline__ bool dlt_bits(double a, double b)
{
    const long long ia = __double_as_longlong(a), ib = __double_as_longlong(b);
    const unsigned long long ma = (unsigned long long)ia & 0x7fffffffffffffffull;
    const unsigned long long mb = (unsigned long long)ib & 0x7fffffffffffffffull;
    if (ma > 0x7ff0000000000000ull || mb > 0x7ff0000000000000ull || (ma | mb) == 0ull)
        return false;
    return (ia ^ ((ia >> 63) & 0x7fffffffffffffffll)) < (ib ^ ((ib >> 63) & 0x7fffffffffffffffll));
}

// Value v of the call (coordinate v % dim of state v / dim) from a standard normal value g:
// normal_distribution's g * 1 + 0 (which only turns -0 into +0: done on the bits), then * stdDev + mean
// and the bounds.
__device__ __forceinline__ void gauss_emit(const SpaceParams &sp, StatesView mean, double stddev, MutStatesView out,
                                           int64_t v, double g)
{
    const int64_t i = v / sp.dim;
    const int d = (int)(v - i * sp.dim);
    const double g0 = __double_as_longlong(g) == (long long)0x8000000000000000ull ? 0.0 : g;
    double z = __dadd_rn(__dmul_rn(g0, stddev), mean(i, d));
    if (sp.kind == GBO_SPACE_SO2)
    {
        // SO2StateSpace::enforceBounds (SO2StateSpace.cpp:79-87)
        double r = fmod(z, 2.0 * kPi);
        if (r < -kPi)
            r = __dadd_rn(r, 2.0 * kPi);
        else if (r >= kPi)
            r = __dsub_rn(r, 2.0 * kPi);
        z = r;
    }
    else if (dlt_bits(z, sp.low[d]))
        z = sp.low[d];
    else if (dlt_bits(sp.high[d], z))
        z = sp.high[d];
    out(i, d) = z;
}

// Value 0 of a call from the cached value of the previous call.
__global__ void gauss_saved_kernel(SamplerState *st, SpaceParams sp, StatesView mean, double stddev, MutStatesView out)
{
    if (threadIdx.x == 0)
    {
        gauss_emit(sp, mean, stddev, out, 0, st->saved);
        st->has_saved = 0;
    }
}

// The pairs of CTA b's 1,024 candidates (k = 1024 b .. 1024 b + 1023): its threads rank the accepted
// candidates in stream order with ballots and keep their (x, y) compacted in shared memory, then
// evaluate consecutive pairs with no lane idle on a rejected candidate: accepted candidate q of the CTA
// gives pair[1024 b + q] = (y mult, x mult), mult = sqrt(-2 log(r2) / r2), and kidx[1024 b + q] = its
// candidate index within the CTA; cnt[b] = the CTA's accepted count. The pairs whose log the plain-FP64
// evaluation cannot round (about 3 %) are listed (b << 10 | q, one global atomic per CTA) for
// gauss_slow_kernel, which runs the double-double evaluation for all of them across the GPU; done here
// at the end of each CTA, it held the CTA's other warps in a long serial tail. gauss_emit_kernel places
// the pairs.
__global__ void __launch_bounds__(256) gauss_pairs_kernel(const uint4 *cand, int64_t G, long long *cnt,
                                                          double2 *pair, unsigned short *kidx, unsigned *slowlist,
                                                          GaussChunk *ctl)
{
    __shared__ double2 sxy[kGaussPerCta];          // accepted (x, y) by local pair index
    __shared__ double sr2[kGaussPerCta];           // and their x^2 + y^2
    __shared__ unsigned short slow[kGaussPerCta];  // local pair indices left to log_cr
    __shared__ int wcnt[4][8];
    __shared__ int nslow;
    __shared__ long long slow0;  // this CTA's first entry in slowlist
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0)
        nslow = 0;
    const int64_t base = (int64_t)blockIdx.x * kGaussPerCta;
    double xs[4], ys[4], rs[4];
    unsigned bal[4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
    {
        const int64_t k = base + r * 256 + t;
        bool acc = false;
        xs[r] = ys[r] = rs[r] = 0.0;
        if (k < G)
            acc = polar_candidate(cand[k], xs[r], ys[r], rs[r]);
        bal[r] = __ballot_sync(0xffffffffu, acc);
        if (lane == 0)
            wcnt[r][warp] = __popc(bal[r]);
    }
    __syncthreads();
    int np = 0;  // accepted candidates of this CTA in earlier rounds
#pragma unroll
    for (int r = 0; r < 4; ++r)
    {
        int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w)
        {
            before += w < warp ? wcnt[r][w] : 0;
            all += wcnt[r][w];
        }
        if ((bal[r] >> lane) & 1u)
        {
            const int q = np + before + __popc(bal[r] & ((1u << lane) - 1u));
            sxy[q] = make_double2(xs[r], ys[r]);
            sr2[q] = rs[r];
            kidx[base + q] = (unsigned short)(r * 256 + t);
        }
        np += all;
    }
    if (t == 0)
        cnt[blockIdx.x] = np;
    __syncthreads();
#pragma unroll 1
    for (int q = t; q < np; q += 256)
    {
        const double2 p = sxy[q];
        const double r2 = sr2[q];
        double lg;
        if (log_fast(r2, lg))
        {
            const double mult = __dsqrt_rn(__ddiv_rn(__dmul_rn(-2.0, lg), r2));
            pair[base + q] = make_double2(__dmul_rn(p.y, mult), __dmul_rn(p.x, mult));
        }
        else
            slow[atomicAdd(&nslow, 1)] = (unsigned short)q;
    }
    __syncthreads();
    const int ns = nslow;
    if (ns == 0)
        return;
    if (t == 0)
        slow0 = atomicAdd((unsigned long long *)&ctl->slow, (unsigned long long)ns);
    __syncthreads();
    for (int i = t; i < ns; i += 256)
        slowlist[slow0 + i] = (unsigned)blockIdx.x << 10 | slow[i];
}

// Pair v = b << 10 | q of the chunk from its candidate (formed again from its words) and lg = log(r2).
__device__ __forceinline__ void gauss_listed_pair(const uint4 *cand, const unsigned short *kidx, double2 *pair,
                                                  unsigned v, bool cr, unsigned *crlist, GaussChunk *ctl)
{
    const int64_t base = (int64_t)(v >> 10) * kGaussPerCta;
    const int q = (int)(v & 1023u);
    double x, y, r2, lg;
    polar_candidate(cand[base + kidx[base + q]], x, y, r2);
    if (cr)
        lg = log_cr(r2);
    else if (!log_med(r2, lg))
    {
        // left to gauss_cr_kernel (about 2 % of the list): one atomic per warp
        const unsigned act = __activemask(), lane = threadIdx.x & 31u;
        const unsigned lead = __ffs(act) - 1;
        unsigned long long at = 0;
        if (lane == lead)
            at = atomicAdd((unsigned long long *)&ctl->slow_cr, (unsigned long long)__popc(act));
        at = __shfl_sync(act, at, lead);
        crlist[at + __popc(act & ((1u << lane) - 1u))] = v;
        return;
    }
    const double mult = __dsqrt_rn(__ddiv_rn(__dmul_rn(-2.0, lg), r2));
    pair[base + q] = make_double2(__dmul_rn(y, mult), __dmul_rn(x, mult));
}

// The pairs gauss_pairs_kernel listed, with log_med; those it cannot round go to crlist. Consecutive warps of
// entries go to different CTAs: the list is a few warps an SM, and each is a serial FP64 chain (100,000 7-D
// states, about 10,000 entries; with gauss_cr_kernel's order the call takes 199 us instead of 209).
__global__ void __launch_bounds__(256) gauss_slow_kernel(const uint4 *cand, const unsigned short *kidx,
                                                         const unsigned *slowlist, unsigned *crlist,
                                                         GaussChunk *ctl, double2 *pair)
{
    const long long n = ctl->slow;
    const long long w = (long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    for (long long e = w * 32 + (threadIdx.x & 31); e < n; e += (long long)gridDim.x * blockDim.x)
        gauss_listed_pair(cand, kidx, pair, slowlist[e], false, crlist, ctl);
}

// The pairs gauss_slow_kernel left, with log_cr. Consecutive entries go to different CTAs: a couple of hundred of
// them in five warps of one SM waited for its FP64 pipe (500,000 10-D states: 17 us).
__global__ void __launch_bounds__(256) gauss_cr_kernel(const uint4 *cand, const unsigned short *kidx,
                                                       const unsigned *crlist, GaussChunk *ctl, double2 *pair)
{
    const long long n = ctl->slow_cr;
    for (long long e = (long long)threadIdx.x * gridDim.x + blockIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        gauss_listed_pair(cand, kidx, pair, crlist[e], true, nullptr, ctl);
}

// Exclusive scan of the per-CTA counts in place (one CTA of 1024 threads); the total goes to ctl.
__global__ void __launch_bounds__(1024) gauss_scan_kernel(long long *cnt, int nb, GaussChunk *ctl)
{
    __shared__ long long part[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long run = 0;
    for (int b0 = 0; b0 < nb; b0 += 1024)
    {
        const int b = b0 + (int)threadIdx.x;
        const long long v = b < nb ? cnt[b] : 0;
        long long x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o)
                x += y;
        }
        if (lane == 31)
            part[warp] = x;
        __syncthreads();
        if (warp == 0)
        {
            long long p = part[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const long long y = __shfl_up_sync(0xffffffffu, p, o);
                if (lane >= o)
                    p += y;
            }
            part[lane] = p;
        }
        __syncthreads();
        if (b < nb)
            cnt[b] = run + (warp ? part[warp - 1] : 0) + x - v;
        run += part[31];
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        ctl->accepted = run;
        ctl->consumed = -1;
    }
}

struct GaussArgs
{
    const double2 *pair;         // pairs of each CTA's accepted candidates (gauss_pairs_kernel)
    const unsigned short *kidx;  // their candidate indices within the CTA
    const long long *off;        // accepted candidates before each CTA
    int nb;                      // CTAs of the chunk
    int64_t need;                // pairs the call still needs
    int64_t v0;                  // value index of the chunk's first pair
    int64_t M;                   // values of the call
    double stddev;
    SpaceParams sp;
    StatesView mean;
    MutStatesView out;
    SamplerState *st;
    GaussChunk *ctl;
};

// Accepted candidate j of the chunk (in stream order) becomes pair j: values v0 + 2j and v0 + 2j + 1;
// the value past the call's end is cached. The words through the last needed candidate are the
// chunk's consumption.
__global__ void __launch_bounds__(256) gauss_emit_kernel(const __grid_constant__ GaussArgs a)
{
    const int b = blockIdx.x;
    const long long rank0 = a.off[b];
    if (rank0 >= a.need)
        return;  // the call's pairs all come from earlier candidates
    const long long next = b + 1 < a.nb ? a.off[b + 1] : a.ctl->accepted;
    const int np = (int)(min(next, (long long)a.need) - rank0);  // at most 1,024
    const int64_t base = (int64_t)b * kGaussPerCta;
#pragma unroll 1
    for (int q = threadIdx.x; q < np; q += 256)
    {
        const double2 g = a.pair[base + q];
        const int64_t j = rank0 + q, v = a.v0 + 2 * j;
        gauss_emit(a.sp, a.mean, a.stddev, a.out, v, g.x);
        if (v + 1 < a.M)
            gauss_emit(a.sp, a.mean, a.stddev, a.out, v + 1, g.y);
        else
        {
            a.st->saved = g.y;
            a.st->has_saved = 1;
        }
        if (j == a.need - 1)
            a.ctl->consumed = 4 * (base + a.kidx[base + q] + 1);
    }
}

// Commits the words the chunk used: K = ctl->consumed (or all W words when the chunk fell short).
// raw holds the rest of the generator's current block (r = 624 - pos words) and then whole blocks,
// untempered, so the generator after word K is the block holding word K - 1.
__global__ void __launch_bounds__(256) gauss_advance_kernel(SamplerState *st, const unsigned *raw, int64_t W,
                                                            const GaussChunk *ctl)
{
    const long long c = ctl->consumed;
    const int64_t K = c >= 0 ? c : W;
    const int64_t r = 624 - (int64_t)st->pos;
    __syncthreads();  // every thread has read pos
    if (K <= r)
    {
        if (threadIdx.x == 0)
            st->pos = (unsigned)(624 - r + K);
        return;
    }
    const int64_t start = r + 624 * ((K - r - 1) / 624);
    for (int i = threadIdx.x; i < 624; i += blockDim.x)
        st->mt[i] = raw[start + i];
    if (threadIdx.x == 0)
        st->pos = (unsigned)(K - start);
}

// The same commit when raw holds exactly the words after the sampler's next one (segmented form): the
// generator after word K is the window of the 624 words before it (position 624), taken from the old
// block for the part before raw[0].
__global__ void __launch_bounds__(256) gauss_advance_seg_kernel(SamplerState *st, const unsigned *raw, int64_t W,
                                                                const GaussChunk *ctl)
{
    __shared__ unsigned old[624];
    const long long c = ctl->consumed;
    const int64_t K = c >= 0 ? c : W;
    const int pos = (int)st->pos;
    for (int i = threadIdx.x; i < 624; i += blockDim.x)
        old[i] = st->mt[i];
    __syncthreads();  // every thread has read pos and the block
    const int64_t r = 624 - pos;
    if (K <= r)
    {
        if (threadIdx.x == 0)
            st->pos = (unsigned)(pos + K);
        return;
    }
    for (int i = threadIdx.x; i < 624; i += blockDim.x)
    {
        const int64_t m = K - 624 + i;  // word m of raw (m < 0: the old block's word pos + m)
        st->mt[i] = m < 0 ? old[pos + m] : raw[m];
    }
    if (threadIdx.x == 0)
        st->pos = 624u;
}

int64_t launch_sample_gaussian(const LaunchCfg &lc, SamplerState *st, bool has_saved, const SpaceParams &sp,
                               StatesView meanv, double stddev, int64_t n, MutStatesView out, unsigned *words,
                               int64_t cap_words, GaussChunk *ctl, long long *cnt, double2 *pair,
                               unsigned short *kidx, unsigned *slowlist, unsigned *jump_scratch,
                               const uint32_t *polys, int64_t L)
{
    const int64_t M = n * sp.dim;
    if (M == 0)
        return 0;
    int64_t v = 0;
    if (has_saved)
    {
        gauss_saved_kernel<<<1, 32, 0, lc.stream>>>(st, sp, meanv, stddev, out);
        note_launch();
        v = 1;
    }
    int64_t need = (M - v + 1) / 2, chunks = 0;
    const int64_t gmax = (cap_words - 624) / 4;
    while (need > 0)
    {
        // acceptance pi/4: the expected count plus 8 standard deviations of the candidates needed
        const double mu = (double)need / 0.7853981633974483;
        const int64_t G = std::max<int64_t>(1, std::min<int64_t>(gmax, (int64_t)std::ceil(mu + 8.0 * std::sqrt(mu) + 64.0)));
        const int nb = (int)((G + kGaussPerCta - 1) / kGaussPerCta);
        // segmented (jump-ahead) generation of the candidates' words when the chunk is large
        const bool seg = polys && 4 * G >= ((int64_t)1 << 18);
        if (seg)
            launch_raw_words_jump(lc, st, 4 * G, words, jump_scratch, polys, L);
        else
            mt_words_kernel<true><<<1, 256, 0, lc.stream>>>(st, 4 * G, words);
        cudaMemsetAsync(&ctl->slow, 0, 2 * sizeof(long long), lc.stream);  // slow and slow_cr
        unsigned *crlist = slowlist + gauss_pair_slots(cap_words);
        gauss_pairs_kernel<<<nb, 256, 0, lc.stream>>>((const uint4 *)words, G, cnt, pair, kidx, slowlist, ctl);
        gauss_slow_kernel<<<lc.sm_count * 8, 256, 0, lc.stream>>>((const uint4 *)words, kidx, slowlist, crlist, ctl,
                                                                  pair);
        gauss_cr_kernel<<<lc.sm_count, 256, 0, lc.stream>>>((const uint4 *)words, kidx, crlist, ctl, pair);
        gauss_scan_kernel<<<1, 1024, 0, lc.stream>>>(cnt, nb, ctl);
        GaussArgs a{pair, kidx, cnt, nb, need, v, M, stddev, sp, meanv, out, st, ctl};
        gauss_emit_kernel<<<nb, 256, 0, lc.stream>>>(a);
        if (seg)
            gauss_advance_seg_kernel<<<1, 256, 0, lc.stream>>>(st, words, 4 * G, ctl);
        else
            gauss_advance_kernel<<<1, 256, 0, lc.stream>>>(st, words, 4 * G, ctl);
        for (int i = 0; i < 7; ++i)
            note_launch();
        GaussChunk h{};
        if (cudaMemcpyAsync(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost, lc.stream) != cudaSuccess ||
            cudaStreamSynchronize(lc.stream) != cudaSuccess)
            return -1;
        const int64_t got = std::min<int64_t>(h.accepted, need);
        if (got <= 0)  // >= 64 candidates without one accepted: the stream is broken, not unlucky
            return -1;
        v += 2 * got;
        need -= got;
        ++chunks;
    }
    return chunks;
}

// FP32 FMA throughput probe: independent FMA chains, no memory traffic in the loop.
__global__ void __launch_bounds__(256) fma_peak_kernel(float *sink, int iters, float seed)
{
    float a0 = seed + threadIdx.x, a1 = a0 + 1.f, a2 = a0 + 2.f, a3 = a0 + 3.f, a4 = a0 + 4.f, a5 = a0 + 5.f,
          a6 = a0 + 6.f, a7 = a0 + 7.f;
    const float b = 0.999999f, c = 1e-7f;
    for (int i = 0; i < iters; ++i)
    {
#pragma unroll
        for (int j = 0; j < 16; ++j)
        {
            a0 = fmaf(a0, b, c);
            a1 = fmaf(a1, b, c);
            a2 = fmaf(a2, b, c);
            a3 = fmaf(a3, b, c);
            a4 = fmaf(a4, b, c);
            a5 = fmaf(a5, b, c);
            a6 = fmaf(a6, b, c);
            a7 = fmaf(a7, b, c);
        }
    }
    const float r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (r == 12345.678f)
        sink[0] = r;
}

__global__ void sincos32_kernel(const double *theta, int64_t n, float *c, float *s)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        sincos_ff(split_double(theta[i]), c[i], s[i]);
}

void launch_sincos32(const LaunchCfg &lc, const double *theta, int64_t n, float *c, float *s)
{
    if (n == 0)
        return;
    sincos32_kernel<<<(int)((n + 255) / 256), 256, 0, lc.stream>>>(theta, n, c, s);
    note_launch();
}

__global__ void __launch_bounds__(256) dfma_peak_kernel(double *sink, int iters, double seed)
{
    double a0 = seed + threadIdx.x, a1 = a0 + 1.0, a2 = a0 + 2.0, a3 = a0 + 3.0;
    const double b = 0.999999, c = 1e-7;
    for (int i = 0; i < iters; ++i)
    {
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            a0 = fma(a0, b, c);
            a1 = fma(a1, b, c);
            a2 = fma(a2, b, c);
            a3 = fma(a3, b, c);
        }
    }
    const double r = a0 + a1 + a2 + a3;
    if (r == 12345.678)
        sink[0] = r;
}

double measure_fp64_peak(const LaunchCfg &lc)
{
    double *sink = nullptr;
    cudaMalloc(&sink, 16);
    const int blocks = lc.sm_count * 8, iters = 256;
    dfma_peak_kernel<<<blocks, 256, 0, lc.stream>>>(sink, 8, 1.0);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, lc.stream);
    dfma_peak_kernel<<<blocks, 256, 0, lc.stream>>>(sink, iters, 1.0);
    cudaEventRecord(e1, lc.stream);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    note_launch();
    note_launch();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    return ms > 0.f ? 2.0 * 4 * 8 * (double)iters * blocks * 256 / (ms * 1e-3) : 0.0;
}

double measure_fp32_peak(const LaunchCfg &lc)
{
    float *sink = nullptr;
    cudaMalloc(&sink, 16);
    const int blocks = lc.sm_count * 8, iters = 4096;
    fma_peak_kernel<<<blocks, 256, 0, lc.stream>>>(sink, 64, 1.f);  // warm-up
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best = 0.0;
    for (int rep = 0; rep < 3; ++rep)
    {
        cudaEventRecord(e0, lc.stream);
        fma_peak_kernel<<<blocks, 256, 0, lc.stream>>>(sink, iters, 1.f);
        cudaEventRecord(e1, lc.stream);
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        const double flops = 2.0 * 8 * 16 * (double)iters * blocks * 256;
        if (ms > 0.f && flops / (ms * 1e-3) > best)
            best = flops / (ms * 1e-3);
    }
    note_launch();
    note_launch();
    note_launch();
    note_launch();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    return best;
}

__global__ void log_rn_kernel(const double *x, int64_t n, double *out)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = log_rn(x[i]);
}

void launch_log_rn(const LaunchCfg &lc, const double *x, int64_t n, double *out)
{
    if (n == 0)
        return;
    log_rn_kernel<<<(int)((n + 255) / 256), 256, 0, lc.stream>>>(x, n, out);
    note_launch();
}

}  // namespace gbo
