/* The location's residuals in pairs of floats (h + l, about 46 bits) instead of doubles, with a bound of their
 * distance from the reference's double form, which says whether their float is certainly the reference's.
 * Host and device compile the same source, without contraction.
 *
 * Errors, with u = 2^-24 (a rounding's relative error), D the largest time difference from the cell's corner time t0,
 * B the largest time, M = max(1, |vpvs|) for a scaled phase and 1 for another:
 *   - a place f and 1 - f are within 3 u^2 of their doubles, the four weights of a row in sum within 23 u^2, the times
 *     interpolated at x and x + 1 within 130 u^2 D (weights; products, 23 u^2 D; sums of the low parts, 80 u^2 D), and
 *     A - b f, a mean of these two but for its own sums, within 300 u^2 D; a scaled phase has M times that;
 *   - obs - t0 is exact as a pair, and brings at most 10 u^2 |obs - t0| into the sums after it.  obs - t0 vpvs is exact as
 *     three floats; as a pair it is off by u^2 |t0 vpvs|, and the pair is brought to l <= u h at once: a low part of the
 *     size u |t0 vpvs| beside a small h would lose as much again in each sum that follows;
 *   - the reference's own double is within 14 2^-53 M B < 0.5 u^2 M B;
 *   - where a window leaves the grid (one that starts at the last plane) the place along z lies between 1 and 2, and
 *     all that the weights multiply grows with the sum W of their magnitudes, 1 in the grid and up to 3 outside.
 * The margin is M W (512 u^2 D + 2 u^2 B) + 16 u^2 |obs - t0|. */
#ifndef FD_PAIR_H
#define FD_PAIR_H

#include <math.h>

#ifdef __CUDACC__
#define FDP_FN static __device__ __forceinline__
#else
#define FDP_FN static inline
#endif

typedef struct {
    float h, l;
} fdp_ff;

/* a row of trials in one cell: the residual at place f is A - b f */
typedef struct
#ifdef __CUDACC__
    __align__(16)
#endif
{
    float ah, al, bh, bl;
} fdp_row;

FDP_FN fdp_ff fdp_pair(float h, float l)
{
    fdp_ff r;
    r.h = h;
    r.l = l;
    return r;
}
FDP_FN fdp_ff fdp_one_minus(fdp_ff f)
{
    const float h = 1.f - f.h;
    return fdp_pair(h, ((1.f - h) - f.h) - f.l);
}
FDP_FN fdp_ff fdp_mul(fdp_ff a, fdp_ff b)
{
    const float p = a.h * b.h;
    return fdp_pair(p, fmaf(a.h, b.h, -p) + fmaf(a.h, b.l, a.l * b.h));
}
FDP_FN fdp_ff fdp_add(fdp_ff a, fdp_ff b)
{
    const float h = a.h + b.h, v = h - a.h;
    return fdp_pair(h, ((a.h - (h - v)) + (b.h - v)) + (a.l + b.l));
}
FDP_FN fdp_ff fdp_neg(fdp_ff a) { return fdp_pair(-a.h, -a.l); }
/* a - b, exact */
FDP_FN fdp_ff fdp_diff(float a, float b) { return fdp_add(fdp_pair(a, 0.f), fdp_pair(-b, 0.f)); }
FDP_FN fdp_ff fdp_scale(fdp_ff a, float s)
{
    const float p = a.h * s;
    return fdp_pair(p, fmaf(a.l, s, fmaf(a.h, s, -p)));
}

/* the weights of a row at places fy, fz: (1-fy)(1-fz), fy(1-fz), (1-fy)fz, fy fz */
FDP_FN void fdp_weights(fdp_ff fy, fdp_ff fz, fdp_ff w[4])
{
    const fdp_ff gy = fdp_one_minus(fy), gz = fdp_one_minus(fz);
    w[0] = fdp_mul(gy, gz);
    w[1] = fdp_mul(fy, gz);
    w[2] = fdp_mul(gy, fz);
    w[3] = fdp_mul(fy, fz);
}

/* A and b of one phase from the times of the row's cell at t (x), t + nx (y), t + nxy (z), and the margin.  Times enter
 * as their differences from the corner's: they are exact and of a step's size, so the pairs' error is too. */
FDP_FN void fdp_coefficients(float obstime, int scaled, float vpvs, const float *t, int nx, int nxy, const fdp_ff w[4],
                             fdp_row *ab, float *m)
{
    const float t0 = t[0];
    float big = fabsf(t0), dmax = 0.f;
    fdp_ff v[2] = {{0.f, 0.f}, {0.f, 0.f}};
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 1; k < 8; k++) {
        const float tk = t[(k & 1) + (k & 2 ? nx : 0) + (k & 4 ? nxy : 0)];
        const fdp_ff d = fdp_diff(tk, t0);
        big = fmaxf(big, fabsf(tk));
        dmax = fmaxf(dmax, fabsf(d.h));
        v[k & 1] = fdp_add(v[k & 1], fdp_mul(w[k >> 1], d));
    }
    fdp_ff c = {t0, 0.f}, a = v[0], b = fdp_add(v[1], fdp_neg(v[0]));
    float mag = 1.f;
    if (scaled) {
        c = fdp_scale(c, vpvs);
        a = fdp_scale(a, vpvs);
        b = fdp_scale(b, vpvs);
        mag = fmaxf(1.f, fabsf(vpvs));
    }
    c = fdp_add(fdp_pair(obstime, 0.f), fdp_neg(c));
    c = fdp_diff(c.h, -c.l);
    const fdp_ff A = fdp_add(c, fdp_neg(a));
    ab->ah = A.h;
    ab->al = A.l;
    ab->bh = b.h;
    ab->bl = b.l;
    const float mw = mag * ((fabsf(w[0].h) + fabsf(w[1].h)) + (fabsf(w[2].h) + fabsf(w[3].h)));
    *m = mw * (1.8189894035458565e-12f * dmax + 7.105427357601002e-15f * big) + 5.684341886080802e-14f * fabsf(c.h);
}

/* The residual A - b f rounded to float, f = fh + fl: 1 and the reference's float if that is certain, that
 * is if A - b f - m and A - b f + m round to the same float; else the caller forms the residual in double. */
FDP_FN int fdp_residual(const fdp_row *ab, float m, float fh, float fl, float *res)
{
    const float p = ab->bh * fh, e = fmaf(ab->bl, fh, fmaf(ab->bh, fl, fmaf(ab->bh, fh, -p)));
    const float d = ab->ah - p, v = d - ab->ah;
    const float low = ((ab->ah - (d - v)) + (-p - v)) + (ab->al - e);
    const float up = d + (low + m);
    *res = up;
    return up == d + (low - m);
}

/* obstime - t vpvs of a node's time, rounded to float: 1 and the reference's float if that is certain (the reference
 * forms it in double and rounds once more).  With p + e the product and d + er the difference obstime - p, both exact as
 * pairs, the value is d + (er - e), exactly; in float er - e and the margin's sums lose less than 4 u^2 (|obstime| + |p|).
 * A tie of two floats is inside any margin, and with vpvs of few bits (7/4) every second time makes one.  But there er - e
 * is a float, so that d + (er - e) is one rounding of the exact value; and the reference's double is exact as well while
 * the operands lie within 2^4 and 2^24 of each other: all terms are multiples of 2^-48 |p| and of 2^-24 |obstime|. */
FDP_FN int fdp_scaled_residual(float obstime, float t, float vpvs, float *res)
{
    const float p = t * vpvs, e = fmaf(t, vpvs, -p);
    const float d = obstime - p, v = d - obstime, er = (obstime - (d - v)) + (-p - v);
    const float low = er - e, size = fabsf(obstime) + fabsf(p), m = 1.4210854715202004e-14f * size;
    const float up = d + (low + m);
    *res = up;
    if (up == d + (low - m)) return 1;
    const float w = low - er;
    *res = d + low;
    return (er - (low - w)) + (-e - w) == 0.f && fabsf(obstime) <= 16.f * fabsf(p) && fabsf(p) <= 16777216.f * fabsf(obstime);
}

#endif
