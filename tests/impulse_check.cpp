// CPU check of the solver's loop without clamps (nans_projekat_gb300/csrc/nans_impulse.cuh) against
// the loop it stands for (code/nans.cpp:1176-1230, the friction bound in double), bit for bit:
// seeded increments over all magnitudes, increments within a few parts in 1e3 and 1e6 of the bound,
// zeros, infinities and NaNs; 2 to 100 rounds. Prints "ok <decided> <tried>" or the first mismatch.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "nans_impulse.cuh"

static unsigned bits(float x)
{
    unsigned u;
    std::memcpy(&u, &x, 4);
    return u;
}
static uint64_t state = 12345;
static uint64_t rnd()
{
    uint64_t z = (state += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
static double uni() { return (double)(rnd() >> 11) * (1.0 / 9007199254740992.0); }
static float any()
{
    unsigned u = (unsigned)rnd();
    float x;
    std::memcpy(&x, &u, 4);
    return x;
}
static float mag(double lo, double hi)
{
    const float x = (float)std::exp(std::log(lo) + (std::log(hi) - std::log(lo)) * uni());
    return rnd() & 1 ? x : -x;
}

static void loop(float ln, float lt1, float lt2, double c2, int iters, float *d)
{
    float s[3] = {0, 0, 0};
    d[0] = d[1] = d[2] = 0;
    const float inc[3] = {ln, lt1, lt2};
    for (int k = 0; k < iters; ++k)
    {
        float old = s[0];
        s[0] = s[0] + ln;
        if (s[0] < 0.0f)
            s[0] = 0.0f;
        d[0] = s[0] - old;
        const float m = (float)(c2 * (double)s[0]);
        for (int q = 1; q < 3; ++q)
        {
            old = s[q];
            s[q] = s[q] + inc[q];
            if (s[q] < -m)
                s[q] = -m;
            if (s[q] > m)
                s[q] = m;
            d[q] = s[q] - old;
        }
    }
}

int main()
{
    const float special[] = {0.0f, -0.0f, INFINITY, -INFINITY, NAN, 1e-45f, -1e-40f, 1e-30f, 3e38f};
    long long decided = 0, tried = 0;
    for (int c = 0; c < 400; ++c)
    {
        const float cf = c == 0 ? 0.5f : c == 1 ? 0.1f : c == 2 ? 1.0f : c == 3 ? 0.0f : std::fabs(mag(1e-4, 1e3));
        const double c2 = 1.4142135623730951 * (double)cf;
        const nans::FBound fb = nans::fbound_split(c2);
        for (int i = 0; i < 40000; ++i)
        {
            const int iters = i % 4 == 0 ? 70 : (i % 4 == 1 ? 2 + (int)(rnd() % 99) : 10);
            float ln = mag(1e-6, 1e4), lt[2];
            const int kind = (int)(rnd() % 8);
            if (kind == 0)
                ln = any();
            if (kind == 1)
                ln = special[rnd() % 9];
            for (int q = 0; q < 2; ++q)
            {
                const int k2 = (int)(rnd() % 8);
                if (k2 == 0)
                    lt[q] = any();
                else if (k2 == 1)
                    lt[q] = special[rnd() % 9];
                else if (k2 == 2)
                    lt[q] = mag(1e-9, 1e6);
                else
                {
                    // about the bound: within 3e-3, or within 3e-6 of one of the two limits
                    const double at = k2 == 3 ? 0.9999 : (k2 == 4 ? 1.0001 : 1.0);
                    const double r = at * (1.0 + (k2 <= 4 ? 3e-6 : 3e-3) * (2 * uni() - 1));
                    lt[q] = (float)(c2 * (double)ln * r) * (rnd() & 1 ? 1.0f : -1.0f);
                }
            }
            float d[3], e0 = 0, e1 = 0, e2 = 0;
            ++tried;
            if (!nans::impulse_direct(ln, lt[0], lt[1], c2, fb, iters, e0, e1, e2))
                continue;
            ++decided;
            loop(ln, lt[0], lt[1], c2, iters, d);
            if (bits(d[0]) != bits(e0) || bits(d[1]) != bits(e1) || bits(d[2]) != bits(e2))
            {
                std::printf("mismatch: ln %a lt %a %a cf %a iters %d: loop %a %a %a direct %a %a %a\n", ln, lt[0], lt[1],
                            cf, iters, d[0], d[1], d[2], e0, e1, e2);
                return 1;
            }
        }
    }
    std::printf("ok %lld %lld\n", decided, tried);
    return 0;
}
