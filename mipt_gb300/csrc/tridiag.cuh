// Eigenvalues of real symmetric tridiagonal matrices by Sturm counts, one
// thread per eigenvalue, or several where SMs would be idle.
//
// Givens' bisection on the number of sign changes of the leading principal
// minors p_i(x) of T - x (p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}):
//   1. twenty bisections in FP32, good to a few 2^-22 of |T|, whose bracket
//      the FP64 search takes only as far as two FP64 counts confirm it;
//   2. in FP64, bisection until a bracket holds exactly one eigenvalue, then
//      regula falsi with the Illinois weighting (Dowell and Jarratt, 1971) on
//      p_d, whose sign change the bracket then holds.
// GB300 runs FP32 about 75 times as fast as FP64, an FP64 result takes 64
// clocks and a division 650, so the recurrence is kept free of divisions (one
// dependent FMA per step, the minors rescaled by powers of two) and the FP32
// start takes the place of most FP64 counts.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mg
{

// Squared off-diagonals are at least this times |T|^2: a zero minor is then
// followed by a non-zero one, and an eigenvalue moves by at most 1e-17 |T|. With
// |T| in [1/4, 1], as the caller scales it, 16 unscaled steps stay in range
// (between 1e-282 and 4^16). FP32 counts: 4 steps, 1e-7 |T|.
constexpr double kTinyE2 = 1e-34;
constexpr float kTinyE2f = 1e-14f;
constexpr int kSturmRescale = 16;
// Half-width added to the FP32 bracket, in units of |T|.
constexpr double kSturmSlack = 2e-6;

struct SturmValue
{
    int count;    // eigenvalues below x
    float mant;   // |p_d(x)| = mant * 2^expo
    int expo;
};

// de[i] = (diagonal i, squared off-diagonal between i - 1 and i; 0 for i = 0).
__device__ __forceinline__ SturmValue sturm_eval(const double2 *__restrict__ de, int d, double x)
{
    double pm = 0.0, p = 1.0;
    unsigned cnt = 0;
    int expo = 0;
    auto step = [&](int i) {
        const double2 t = de[i];
        const double u = t.y * pm;
        const double pn = fma(t.x - x, p, -u);
        cnt += static_cast<unsigned>(__double2hiint(pn) ^ __double2hiint(p)) >> 31;
        pm = p;
        p = pn;
    };
    auto rescale = [&]() {
        const int hp = (__double2hiint(p) >> 20) & 0x7ff, hm = (__double2hiint(pm) >> 20) & 0x7ff;
        int e = hp > hm ? hp : hm;
        e = e < 1 ? 1 : (e > 2045 ? 2045 : e);
        const double s = __hiloint2double((2046 - e) << 20, 0); // 2^(1023 - e)
        p *= s;
        pm *= s;
        expo += e - 1023;
    };
    int i = 0;
    for (; i + kSturmRescale <= d; i += kSturmRescale)
    {
#pragma unroll
        for (int u = 0; u < kSturmRescale; ++u) step(i + u);
        rescale();
    }
    for (; i < d; ++i) step(i);
    rescale();
    return SturmValue{static_cast<int>(cnt), fabsf(static_cast<float>(p)), expo};
}

// The same count in FP32; df holds the matrix over |T|, x is in those units.
__device__ __forceinline__ int sturm_count32(const float2 *__restrict__ df, int d, float x)
{
    float pm = 0.f, p = 1.f;
    unsigned cnt = 0;
    auto step = [&](int i) {
        const float2 t = df[i];
        const float u = t.y * pm;
        const float pn = fmaf(t.x - x, p, -u);
        cnt += static_cast<unsigned>(__float_as_int(pn) ^ __float_as_int(p)) >> 31;
        pm = p;
        p = pn;
    };
    int i = 0;
    for (; i + 4 <= d; i += 4)
    {
#pragma unroll
        for (int u = 0; u < 4; ++u) step(i + u);
        const int hp = (__float_as_int(p) >> 23) & 0xff, hm = (__float_as_int(pm) >> 23) & 0xff;
        int e = hp > hm ? hp : hm;
        e = e < 1 ? 1 : (e > 253 ? 253 : e);
        const float s = __int_as_float((254 - e) << 23); // 2^(127 - e)
        p *= s;
        pm *= s;
    }
    for (; i < d; ++i) step(i);
    return static_cast<int>(cnt);
}

// Squared off-diagonal's FP32 entry of df.
__device__ __forceinline__ float2 sturm_entry32(double2 de, double inv_norm, int i)
{
    const float e2 = static_cast<float>(de.y * inv_norm * inv_norm);
    return make_float2(static_cast<float>(de.x * inv_norm), i > 0 ? fmaxf(e2, kTinyE2f) : 0.f);
}

// Eigenvalue `index` (ascending) of the matrix, all of whose eigenvalues lie
// in (-bound, bound), norm being |T| (1/4 to 1); eigenvalues below `cutoff`
// (0 or more) may come back as any value below it.
__device__ __forceinline__ double sturm_eigenvalue(const double2 *__restrict__ de, const float2 *__restrict__ df,
                                                   int d, int index, double norm, double bound, double cutoff)
{
    const double tol = 1.1102230246251565e-16 * norm;
    double lo = -bound, hi = bound;
    SturmValue L{0, 1.f, 0}, H{d, 1.f, 0};
    bool know_l = false, know_h = false;
    int side = 0;
    // One FP64 count at x; isolated: the bracket held one eigenvalue.
    auto probe = [&](double x, bool isolated) {
        const SturmValue v = sturm_eval(de, d, x);
        if (v.count > index)
        {
            hi = x;
            H = v;
            know_h = true;
            if (isolated && side == 1) L.expo -= 1;
            side = 1;
        }
        else
        {
            lo = x;
            L = v;
            know_l = true;
            if (isolated && side == -1) H.expo -= 1;
            side = -1;
        }
    };
    float a = -1e-6f, b = 1.001f; // nothing below the (positive) cutoff is looked for
    for (int it = 0; it < 20; ++it)
    {
        const float x = 0.5f * (a + b);
        if (sturm_count32(df, d, x) > index)
            b = x;
        else
            a = x;
    }
    double guess[2] = {(static_cast<double>(a) - kSturmSlack) * norm, (static_cast<double>(b) + kSturmSlack) * norm};
    if (guess[0] < cutoff) guess[0] = cutoff;
    // First the two ends of the FP32 bracket, then the search.
    // Two regula falsi steps in a row have to leave a quarter of the bracket,
    // or a bisection follows (p_d grows like x^62 beside an eigenvalue when 62
    // others are near zero); after 64 steps only bisections. 64 + 56 of them
    // end any search.
    int tries = 0;
    double w_try = 0.0;
    // Geometric means, in FP32, of brackets that span much of the range.
    const double least = fmax(0.01 * cutoff, 1e-30);
    for (int it = -2; it < 160; ++it)
    {
        const double w = hi - lo;
        if (hi <= cutoff || !(w > tol)) break;
        double x = lo + 0.5 * w;
        bool isolated = false;
        if (it < 0)
        {
            x = guess[it + 2];
            if (!(x > lo && x < hi)) continue;
        }
        else
        {
            if (!(x > lo && x < hi)) break;
            isolated = know_l && know_h && H.count - L.count == 1;
            // Steps no smaller than this leave the bracket's ends representably.
            const double half = fmax(0.5 * tol, 2.3e-16 * fmax(fabs(lo), fabs(hi)));
            if (tries == 2 && w > 0.25 * w_try)
                tries = 0;
            else if (isolated && w > 4.0 * half && it < 64)
            {
                if (tries == 2) tries = 0;
                if (tries++ == 0) w_try = w;
                // |p(lo)| / (|p(lo)| + |p(hi)|) of the way; FP32 is enough for a guess.
                int de2 = H.expo - L.expo;
                de2 = de2 > 120 ? 120 : (de2 < -120 ? -120 : de2);
                const float r = H.mant / fmaxf(L.mant, 1e-30f) * exp2f(static_cast<float>(de2));
                const double y = lo + w * static_cast<double>(1.f / (1.f + r));
                x = y < lo + half ? lo + half : (y > hi - half ? hi - half : y);
            }
            else if (lo > least && hi > 16.0 * lo)
                x = static_cast<double>(sqrtf(static_cast<float>(lo)) * sqrtf(static_cast<float>(hi)));
        }
        probe(x, isolated);
    }
    return 0.5 * (lo + hi);
}

// The same by 2^gl neighbouring lanes: counts at 2^gl points of the bracket at
// once (multisection) narrow it 2^gl + 1 fold, so with 16 lanes nine FP64
// counts end a search, none of which depends on how p_d grows or on how many
// eigenvalues the bracket holds. Every lane of the warp calls this; a group
// without an eigenvalue to find (on = false) counts along.
__device__ __forceinline__ double sturm_eigenvalue_lanes(const double2 *__restrict__ de, const float2 *__restrict__ df,
                                                         int d, int index, double norm, double bound, double cutoff,
                                                         int gl, bool on)
{
    const int G = 1 << gl, lane = threadIdx.x & 31, sub = lane & (G - 1);
    const unsigned low = G == 32 ? 0xffffffffu : (1u << G) - 1u;
    // The first lane of the group whose count is above `index`; G if none.
    auto first_above = [&](bool above) {
        const unsigned m = (__ballot_sync(0xffffffffu, above) >> (lane - sub)) & low;
        return m ? __ffs(m) - 1 : G;
    };
    // As many rounds as narrow the FP32 bracket 2^20 fold.
    float a = -1e-6f, b = 1.001f; // nothing below the (positive) cutoff is looked for
    const float stepf = 1.f / static_cast<float>(G + 1);
    for (float left = 1 << 20; left > 1.f; left *= stepf)
    {
        const float w = (b - a) * stepf;
        const int f = first_above(sturm_count32(df, d, a + w * static_cast<float>(sub + 1)) > index);
        b = f == G ? b : a + w * static_cast<float>(f + 1);
        a = f == 0 ? a : a + w * static_cast<float>(f);
    }
    const double tol = 1.1102230246251565e-16 * norm;
    double lo = -bound, hi = bound;
    // First points over the FP32 bracket, its ends among them.
    double x0 = (static_cast<double>(a) - kSturmSlack) * norm;
    double dx = (static_cast<double>(b) + kSturmSlack) * norm;
    if (x0 < cutoff) x0 = cutoff;
    dx = dx > x0 ? (dx - x0) / static_cast<double>(G - 1) : 0.0;
    const double step = 1.0 / static_cast<double>(G + 1);
    for (int it = 0; it < 64; ++it)
    {
        if (!__any_sync(0xffffffffu, on)) break;
        const int f = first_above(sturm_eval(de, d, fma(dx, static_cast<double>(sub), x0)).count > index);
        const double nlo = f == 0 ? lo : fma(dx, static_cast<double>(f - 1), x0);
        const double nhi = f == G ? hi : fma(dx, static_cast<double>(f), x0);
        // Done at the tolerance, or where rounding keeps the bracket from narrowing.
        const double w = nhi - nlo;
        if (on)
        {
            on = !(nhi <= cutoff) && w > tol && (it == 0 || w < hi - lo);
            lo = nlo;
            hi = nhi;
        }
        dx = w * step;
        x0 = lo + dx;
    }
    return 0.5 * (lo + hi);
}

} // namespace mg
