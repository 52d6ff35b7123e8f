// The accumulate/clamp loop of Constraint (code/nans.cpp:1176-1230) without its clamps.
//
// The loop adds the same three increments every round (the velocities do not change inside it): ln to
// the normal sum sn, clamped at 0, and lt1, lt2 to the tangent sums, clamped to +-m with
// m = (float)(c2 * sn); only the last round's differences are used. From zero sums:
//
//   * ln <= 0: sn stays 0 and so does m; after two rounds every difference is +0.
//   * ln > 0: sn_k is the k-fold sum of ln, and m_k is about k c2 ln. An increment |lt| below
//     0.9999 c2 ln is never clamped: its sum is the k-fold sum of lt. One above 1.0001 c2 ln is clamped
//     in every round: its sum is +-m_k. With at most 100 rounds the sums' rounding errors are below
//     100 * 2^-24 of their values and m's below 103 * 2^-24, so neither comparison can come out
//     otherwise: unclamped, |st_k| <= 0.9999 k q (1 + 6e-6) < k q (1 - 7e-6) <= m_k for q = c2 ln;
//     clamped, m_(k-1) + 1.0001 q exceeds m_k <= (m_(k-1) + q)(1 + 4 2^-24) by more than the
//     2.4e-5 q that its error reaches.
//   * Increments between the two, NaNs and values outside the normal range are left to the loop.
//
// The k-fold sums are three independent chains of additions; the loop's round is ~50 instructions
// (123 cycles on one warp of a GB300). Plain IEEE single arithmetic, compiled for the device and for
// the host (the CPU check against the loop, tests/impulse_check.cpp).
#pragma once
#include "nans_fbound.cuh"

namespace nans
{

constexpr int kDirectRounds = 100;

NANS_FB_FN float friction_bound(const FBound &fb, double c2, float s)
{
    bool cert;
    const float m = fbound_mul(fb, s, &cert);
    return cert ? m : (float)(c2 * (double)s);
}

// The last round's differences of `iters` rounds from zero sums, where decided (true).
NANS_FB_FN bool impulse_direct(float ln, float lt1, float lt2, double c2, const FBound &fb, int iters, float &dn,
                               float &dt1, float &dt2)
{
    if (iters < 2 || iters > kDirectRounds || !fb.ok)
        return false;
    if (ln <= 0.0f)
    {
        dn = dt1 = dt2 = 0.0f;
        return lt1 == lt1 && lt2 == lt2;
    }
    const float q = fb.ch * ln;
    const float a1 = lt1 < 0.0f ? -lt1 : lt1, a2 = lt2 < 0.0f ? -lt2 : lt2;
    const float hi = 1.0001f * q, lo = 0.9999f * q;
    const bool cl1 = a1 > hi, cl2 = a2 > hi;
    if (!(ln > 1e-18f && ln < 1e18f && q > 1e-28f && q < 1e28f && (cl1 || a1 < lo) && (cl2 || a2 < lo)))
        return false;
    float sn = ln, u1 = lt1, u2 = lt2, on = 0.0f, o1 = 0.0f, o2 = 0.0f;
    for (int k = 1; k < iters; ++k)
    {
        on = sn;
        o1 = u1;
        o2 = u2;
        sn = sn + ln;
        u1 = u1 + lt1;
        u2 = u2 + lt2;
    }
    dn = sn - on;
    dt1 = u1 - o1;
    dt2 = u2 - o2;
    if (cl1 || cl2)
    {
        // both sums move by the bound's own difference (its sign is exact)
        const float d = friction_bound(fb, c2, sn) - friction_bound(fb, c2, on);
        if (cl1)
            dt1 = lt1 < 0.0f ? -d : d;
        if (cl2)
            dt2 = lt2 < 0.0f ? -d : d;
    }
    return true;
}

} // namespace nans
