/* sin, cos and atan2 in fixed point, with a proof of each rounding: the result is the correctly rounded double, or
 * the call answers that it cannot tell (zero, tiny, huge or non-finite arguments; an exact value within about 2^-80
 * of a rounding boundary, one call in 2^26) and the caller takes the double-double functions of fd_trig.h, which
 * agree wherever this one answers.  Host and device compile the same source.
 *
 * Why: FP64 instructions issue once in 64 cycles per scheduler here and a double-double sine takes some 250 of
 * them; 64-bit integer products are four full-rate instructions.
 *
 * Method: unsigned 128-bit fixed point (fdx_u), a value v at scale s held as v 2^s.
 *  - sin, cos: x = k pi/128 + r exactly to 2^-111, |r| <= pi/256; 1 - cos r and sin r from their Taylor series with
 *    w = r^2, the leading terms in two words and the later ones, which are below 2^-21, in one word or half of one;
 *    then the addition theorem with a table of sin(j pi/128), j = 0..64.
 *  - atan2: of a = max(|x|, |y|) and b = the other, the angle is k pi/128 + atan t, t = (b C - a S) / (a C + b S) with
 *    C, S = cos, sin(k pi/128): the quotient from a reciprocal by two Newton steps and one remainder, atan t from
 *    its Taylor series; then the octant.
 *  - rounding: truncations and dropped terms add up to less than 2^-81.2 (sin, cos) and 2^-80.2 (atan2); a value is
 *    rounded if no midpoint of neighbouring doubles lies within twice that. */
#ifndef FD_TRIG_FX_H
#define FD_TRIG_FX_H

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define FDX_FN static __device__ __forceinline__
#define FDX_TABLE static __device__ const
#else
#define FDX_FN static inline
#define FDX_TABLE static const
#endif

typedef unsigned __int128 fdx_u;

/* sin(j pi/128) at scale 126 */
FDX_TABLE uint64_t fdx_sin_table[65][2] = {
    {0x0000000000000000ull, 0x0000000000000000ull},
    {0x0192155f7a3667dfull, 0x938a73db97fb419eull},
    {0x0323ecbe21bb027cull, 0xdda85e552cadf146ull},
    {0x04b54824b3867d73ull, 0x2fbbaba04a69e1aeull},
    {0x0645e9af0a6d0af8ull, 0x7639cb644a5dfb9cull},
    {0x07d59395aa5cc38dull, 0x1382394d72b6bc52ull},
    {0x0964083747309d11ull, 0x3000a89a11e07c20ull},
    {0x0af10a22459fe32aull, 0x63feef3bb58b1f11ull},
    {0x0c7c5c1e34d3055bull, 0x25cc8c00e4fccd85ull},
    {0x0e05c1353f27b17eull, 0x50ebc61ade6ca83dull},
    {0x0f8cfcbd90af8d57ull, 0xa4221dc4ba772599ull},
    {0x1111d262b1f67760ull, 0x93082adeaa668861ull},
    {0x1294062ed59f05a8ull, 0xb5c974ee7b4d7eeaull},
    {0x14135c9417660143ull, 0x25f12be894607981ull},
    {0x158f9a75ab1fdcfeull, 0x1023f2a7309dff08ull},
    {0x17088530fa459eaeull, 0xd3987de6ce8dbc77ull},
    {0x187de2a6aea962d1ull, 0xa6245854b3dfbb87ull},
    {0x19ef7943a8ed8a2dull, 0xb5025217b755ac5dull},
    {0x1b5d1009e15cc02bull, 0x66c5972e8305c606ull},
    {0x1cc66e9931c45e16ull, 0x850e59c37f8f5a3aull},
    {0x1e2b5d3806f63b1eull, 0x0d891d3c684161e4ull},
    {0x1f8ba4dbf89ab9fbull, 0x44f80f922252171aull},
    {0x20e70f3245ffdb2dull, 0x2ff5e5c5fca202b0ull},
    {0x223d66a836964508ull, 0x6e24b2a0d8763213ull},
    {0x238e76735cd190d9ull, 0x2ee933fb2ffd521aull},
    {0x24da0a99ba25bd51ull, 0x2c5e0864479c705cull},
    {0x261feff9c2e069c2ull, 0x0673b2116b21e972ull},
    {0x275ff45240a17278ull, 0xf8978e55258e2b9aull},
    {0x2899e64a123bac30ull, 0x0ed459fb8d6688d3ull},
    {0x29cd9577c7cbd227ull, 0x8527db9d664d1a29ull},
    {0x2afad26919d93f45ull, 0x46fb36a022706a53ull},
    {0x2c216eaa3a59bdb6ull, 0xb932b40357252f34ull},
    {0x2d413cccfe779921ull, 0x165f626cdd52afa8ull},
    {0x2e5a106fdfff2c86ull, 0xa77878ec8ae2fd37ull},
    {0x2f6bbe44d55f5dbcull, 0x2b214c83d4a35b57ull},
    {0x30761c17ff2edba4ull, 0x2f7c1c572e2c82f6ull},
    {0x317900d62a2e8169ull, 0xd0f689766499cc9bull},
    {0x3274449324c7f69eull, 0xa0cd4906f85a4c89ull},
    {0x3367c08fe70e8167ull, 0x88ebcc76dc5e692aull},
    {0x34534f408c4f03bbull, 0x5d13fa883a2afbe4ull},
    {0x3536cc521d434606ull, 0x7d8c3a2db6b20f9aull},
    {0x361214b02a03ff36ull, 0xc92e7f80198d5d29ull},
    {0x36e5068a32dc7b21ull, 0xcb066d8c94f690ffull},
    {0x37af8158df2a533eull, 0xd2c66a9c7fb0eb9bull},
    {0x387165e3017b61a4ull, 0x7d3a2a0dcbe31604ull},
    {0x392a96426823e9edull, 0x0489e16b99fd5457ull},
    {0x39daf5e8798ee5e1ull, 0x84944a54a7522a4cull},
    {0x3a8269a29b927358ull, 0x856b516d286d7a09ull},
    {0x3b20d79e651a8c51ull, 0x5f98408c6b075860ull},
    {0x3bb6276d998478c1ull, 0xe1be3083ed992c07ull},
    {0x3c424209ed0dc97full, 0x59c49f6cd6ca1cc5ull},
    {0x3cc511d891c223ddull, 0x29521af7115755a9ull},
    {0x3d3e82ad8c5bb4bbull, 0x058f171fc0edc631ull},
    {0x3dae81ced092c67aull, 0x0b1e47d67307ff09ull},
    {0x3e14fdf72461ae54ull, 0xb1eb71ad2622246full},
    {0x3e71e758c9cb118aull, 0x11412b823466ca60ull},
    {0x3ec52f9feeb96055ull, 0x885ca8d87f4a9c8cull},
    {0x3f0ec9f4e297526aull, 0xc959de3ff2d705daull},
    {0x3f4eaafe114a2d42ull, 0xfab9af6547076aefull},
    {0x3f84c8e1c33fa68full, 0x64334765676d9d3cull},
    {0x3fb11b47a24a4b3cull, 0x104e43bf71c9ba7cull},
    {0x3fd39b5a0310742aull, 0x43d9a18cfc6ae162ull},
    {0x3fec43c6f2dafbc7ull, 0x5087a3b6abd6514full},
    {0x3ffb10c1099a1976ull, 0x5595d548d9a585cdull},
    {0x4000000000000000ull, 0x0000000000000000ull},
};

FDX_FN uint64_t fdx_mulhi(uint64_t a, uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

FDX_FN int64_t fdx_mulhi_s(int64_t a, int64_t b)
{
#ifdef __CUDA_ARCH__
    return __mul64hi(a, b);
#else
    return (int64_t)(((__int128)a * b) >> 64);
#endif
}

FDX_FN uint32_t fdx_mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

FDX_FN int fdx_clz(uint64_t a)   /* a != 0 */
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)a);
#else
    return __builtin_clzll(a);
#endif
}

FDX_FN fdx_u fdx_make(uint64_t hi, uint64_t lo) { return ((fdx_u)hi << 64) | lo; }
FDX_FN uint64_t fdx_hi(fdx_u a) { return (uint64_t)(a >> 64); }
FDX_FN uint64_t fdx_lo(fdx_u a) { return (uint64_t)a; }

/* -a if neg */
FDX_FN fdx_u fdx_neg_if(fdx_u a, int neg) { return neg ? -a : a; }

FDX_FN fdx_u fdx_mul_ww(uint64_t a, uint64_t b) { return (fdx_u)a * b; }

/* floor(w a / 2^64), within 1 */
FDX_FN fdx_u fdx_mul_wu(uint64_t w, fdx_u a) { return fdx_mul_ww(w, fdx_hi(a)) + fdx_mulhi(w, fdx_lo(a)); }

/* a b / 2^128, within 3 */
FDX_FN fdx_u fdx_mul_uu(fdx_u a, fdx_u b)
{
    return fdx_mul_ww(fdx_hi(a), fdx_hi(b)) + fdx_mulhi(fdx_hi(a), fdx_lo(b)) + fdx_mulhi(fdx_lo(a), fdx_hi(b));
}

FDX_FN uint64_t fdx_bits(double v)
{
    uint64_t u;
    memcpy(&u, &v, sizeof u);
    return u;
}

/* (-1)^neg v 2^-scale rounded to double; 0 if a midpoint of doubles lies within 2^guard of v */
FDX_FN int fdx_round(fdx_u v, int neg, int scale, int guard, double *out)
{
    if (fdx_hi(v) == 0) return 0;
    const int lz = fdx_clz(fdx_hi(v));
    if (guard + lz >= 73) return 0;
    const fdx_u t = lz ? (v << lz) : v;
    const uint64_t rest = (fdx_hi(t) << 53) | (fdx_lo(t) >> 11);   /* below the last place of the result; half a place is 2^63 */
    const uint64_t near = (guard + lz > 11 ? 1ull << (guard + lz - 11) : 1ull) + 2;
    if (rest - (0x8000000000000000ull - near) <= 2 * near) return 0;
    const uint64_t u = ((uint64_t)(1023 + 127 - 1 - scale - lz) << 52) + (fdx_hi(t) >> 11) + (rest >> 63) + ((uint64_t)neg << 63);
    memcpy(out, &u, sizeof u);
    return 1;
}

/* sin x and cos x; 0 if one of them could not be proved */
FDX_FN int fdx_sincos(double x, double *s, double *c)
{
    const uint64_t u = fdx_bits(x);
    const int e = (int)((u >> 52) & 2047) - 1023;
    if (e < -30 || e > 3) return 0;
    const int xneg = (int)(u >> 63);
    const uint64_t m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    /* |x| at scale 120: m 2^(68 + e) */
    const int sh = 68 + e;
    const fdx_u X = sh >= 64 ? fdx_make(m << (sh - 64), 0) : fdx_make(m >> (64 - sh), m << sh);
    /* k = |x| 128/pi to the nearest: fdx_hi(X) at scale 56 times 128/pi at scale 57 */
    const unsigned k = (unsigned)((fdx_mulhi(fdx_hi(X), 0x517cc1b727220a95ull) + (1ull << 48)) >> 49);
    const fdx_u kp = fdx_make(0x0006487ed5110b46ull, 0x11a62633145c06e1ull) * k;
    fdx_u r = X - kp;
    const int rneg = (int)(fdx_hi(r) >> 63);
    r = fdx_neg_if(r, rneg);
    /* w = r^2 at scale 140, its first word wh at scale 76, w32 at scale 44 */
    const uint64_t rh = (fdx_hi(r) << 14) | (fdx_lo(r) >> 50), rl = fdx_lo(r) << 14;   /* scales 70 and 134 */
    const uint64_t cross = fdx_mulhi(rh, rl);
    const fdx_u W = fdx_mul_ww(rh, rh) + ((fdx_u)cross << 1);
    const uint64_t wh = fdx_hi(W);
    const uint32_t w32 = (uint32_t)(wh >> 32);
    /* 1 - cos r = w/2 - w^2 (1/4! - w (1/6! - w (1/8! - w/10!))) at scale 124 */
    const uint32_t u1 = 0xd00d00d0u - (fdx_mulhi32(0x93f27dbcu, w32) >> 18);
    const uint64_t u2 = 0xb60b60b60b60b60bull - (((uint64_t)w32 * u1) >> 18);
    const uint64_t u3 = 0xaaaaaaaaaaaaaaabull - (fdx_mulhi(wh, u2) >> 17);
    const uint64_t u4 = fdx_mulhi(fdx_mulhi(wh, wh), u3);   /* scale 92 */
    const fdx_u V = (W >> 17) - ((fdx_u)u4 << 32);
    /* sin |r| = r - r w (1/3! - w (1/5! - w (1/7! - w/9!))) at scale 124 */
    const uint32_t v1 = 0xd00d00d0u - (fdx_mulhi32(0xb8ef1d2bu, w32) >> 18);
    const uint64_t v2 = 0x8888888888888889ull - (((uint64_t)w32 * v1) >> 18);
    const uint64_t v3 = 0xaaaaaaaaaaaaaaabull - (fdx_mulhi(wh, v2) >> 16);
    const uint64_t rz = fdx_mulhi(rh, fdx_mulhi(wh, v3));   /* scale 84 */
    const fdx_u sr = (r << 4) - ((fdx_u)rz << 40);
    /* sin and cos of i pi/128 + r, i = k mod 64, at scale 122 */
    const int i = (int)(k & 63), q = (int)((k >> 6) & 3);
    const fdx_u A = fdx_make(fdx_sin_table[i][0], fdx_sin_table[i][1]);
    const fdx_u B = fdx_make(fdx_sin_table[64 - i][0], fdx_sin_table[64 - i][1]);
    fdx_u s0 = (A >> 4) - fdx_mul_uu(A, V);
    fdx_u c0 = (B >> 4) - fdx_mul_uu(B, V);
    const fdx_u bs = fdx_mul_uu(B, sr), as = fdx_mul_uu(A, sr);
    s0 += fdx_neg_if(bs, rneg);
    c0 += fdx_neg_if(as, !rneg);
    const int sneg = (int)(fdx_hi(s0) >> 63), cneg = (int)(fdx_hi(c0) >> 63);   /* below 0 by r */
    s0 = fdx_neg_if(s0, sneg);
    c0 = fdx_neg_if(c0, cneg);
    const int odd = q & 1;
    return fdx_round(odd ? c0 : s0, xneg ^ (q >> 1) ^ (odd ? cneg : sneg), 122, 42, s)
        & fdx_round(odd ? s0 : c0, (odd ^ (q >> 1)) ^ (odd ? sneg : cneg), 122, 42, c);
}

/* atan2(y, x); 0 if it could not be proved */
FDX_FN int fdx_atan2(double y, double x, double *out)
{
    const uint64_t uy = fdx_bits(y), ux = fdx_bits(x);
    const uint64_t my = uy & 0x7fffffffffffffffull, mx = ux & 0x7fffffffffffffffull;
    const int swap = my > mx;
    const uint64_t ua = swap ? my : mx, ub = swap ? mx : my;
    const int ea = (int)(ua >> 52), d = ea - (int)(ub >> 52);
    if (ea >= 2047 || ea < 64 || d > 24) return 0;
    /* a at scale 62 of its power of two, b at scale 126 */
    const uint64_t a = ((ua & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
    const uint64_t bm = ((ub & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
    const fdx_u b = d ? fdx_make(bm >> d, bm << (64 - d)) : fdx_make(bm, 0);
    const float t0 = (float)(uint32_t)(fdx_hi(b) >> 32) / (float)(uint32_t)(a >> 32);
    const int k = (int)(atanf(t0) * 40.743665f + 0.5f);
    const fdx_u S = fdx_make(fdx_sin_table[k][0], fdx_sin_table[k][1]);
    const fdx_u C = fdx_make(fdx_sin_table[64 - k][0], fdx_sin_table[64 - k][1]);
    /* numerator and denominator at scale 124; t <= tan(pi/256 + 2^-20) */
    fdx_u N = fdx_mul_uu(b, C) - fdx_mul_wu(a, S);
    const fdx_u D = fdx_mul_wu(a, C) + fdx_mul_uu(b, S);
    const int nneg = (int)(fdx_hi(N) >> 63);
    N = fdx_neg_if(N, nneg);
    /* y2 = 1/D at scale 62 within 2^-58 of it, from a float and two Newton steps on dh = D at scale 62 */
    const uint64_t dh = (fdx_hi(D) << 2) | (fdx_lo(D) >> 62);
    const uint64_t y0 = (uint64_t)(uint32_t)(1152921504606846976.0f / (float)(uint32_t)(dh >> 32)) << 32;
    const int64_t e0 = (int64_t)((1ull << 60) - fdx_mulhi(dh, y0));
    const uint64_t y1 = y0 + (uint64_t)fdx_mulhi_s((int64_t)y0, e0 * 16);
    const int64_t e1 = (int64_t)((1ull << 60) - fdx_mulhi(dh, y1));
    const uint64_t y2 = y1 + (uint64_t)fdx_mulhi_s((int64_t)y1, e1 * 16);
    /* t = q0 + remainder / D, at scale 123 */
    const uint64_t q0 = fdx_mulhi((fdx_hi(N) << 8) | (fdx_lo(N) >> 56), y2);   /* scales 68 + 62 - 64 */
    const fdx_u rem = (N << 2) - fdx_mul_wu(q0, D);     /* scale 126 */
    const int64_t rem2 = (int64_t)((fdx_hi(rem) << 62) | (fdx_lo(rem) >> 2));  /* scale 124 */
    const int64_t t1 = 2 * fdx_mulhi_s(rem2, (int64_t)y2);
    const fdx_u t = ((fdx_u)q0 << 57) + (fdx_u)(__int128)t1;
    /* atan t = t - t w (1/3 - w (1/5 - w (1/7 - w (1/9 - w (1/11 - w/13))))) */
    const uint64_t th = (fdx_hi(t) << 11) | (fdx_lo(t) >> 53);   /* scale 70 */
    const uint64_t wh = fdx_mulhi(th, th);
    const uint32_t w32 = (uint32_t)(wh >> 32);
    const uint32_t g1 = 0xba2e8ba3u - (fdx_mulhi32(0x9d89d89eu, w32) >> 12);
    const uint32_t g2 = 0xe38e38e4u - (fdx_mulhi32(g1, w32) >> 12);
    const uint64_t g3 = 0x9249249249249249ull - (((uint64_t)w32 * g2) >> 13);
    const uint64_t g4 = 0xcccccccccccccccdull - (fdx_mulhi(wh, g3) >> 12);
    const uint64_t g5 = 0xaaaaaaaaaaaaaaabull - (fdx_mulhi(wh, g4) >> 13);
    const uint64_t tz = fdx_mulhi(th, fdx_mulhi(wh, g5));   /* scale 83 */
    fdx_u v = t - ((fdx_u)tz << 40);
    v = fdx_make(0x003243f6a8885a30ull, 0x8d313198a2e03707ull) * (unsigned)k + fdx_neg_if(v, nneg);
    if (swap) v = fdx_make(0x0c90fdaa22168c23ull, 0x4c4c6628b80dc1cdull) - v;
    if (ux >> 63) v = fdx_make(0x1921fb54442d1846ull, 0x9898cc51701b839aull) - v;
    return fdx_round(v, (int)(uy >> 63), 123, 44, out);
}

#endif
