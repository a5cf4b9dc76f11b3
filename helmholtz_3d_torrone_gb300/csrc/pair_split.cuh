// pair_split.cuh -- the FP64 pair arithmetic on GB300's FP32 and integer
// pipes: every value is an unevaluated sum h + l of two FP32 numbers (48
// bits), or a 64-bit integer where cancellation would eat those bits.
//
// GB300 issues one FP64 instruction for about 70 FP32 ones, so a pair
// evaluated here (232 instructions) costs a tenth of the 38.5 FP64
// instructions of pair64.cuh.  What keeps the error small:
//
// * Coordinates are scaled by k and taken about the source tile's origin o:
//   s = x_s - o, a = x_t - o, A = -2a, all formed in FP64 and split into a
//   30-bit integer head (times a power of two) and an FP32 tail.  Then
//     |a - s|^2 - |a|^2 = |s|^2 + A.s      and      -2 (a - s).n = A.n + 2 s.n
//   are sums of three 64-bit integer products (IMAD.WIDE, exact) and six
//   FP32 products of heads with tails (2^-31 of the heads, so that their
//   rounding is below 2^-54).
// * rho comes from r^2 = h + l by one Newton step on the FP32 root g:
//   rho = g + (r^2 - g^2) / 2g, where h - g^2 is exact in one FMA.
// * Far from the tile the phase is taken about the tile's origin: with
//   rho_c = |a| the sum over the tile carries e^{i (rho - rho_c)}, and the
//   FP64 factor e^{i rho_c} is applied once per tile.  rho - rho_c =
//   (r^2 - |a|^2) / (rho + rho_c) keeps its relative accuracy, so the phase
//   error is 2^-48 of a phase of the tile's size (one to three radians), not
//   of k rho.
// * e^{i theta}: nearest of kSplitTable angles, the rest r (at most 3.9e-4)
//   reduced with a three-part step, and
//   cos = tc - (ts r + tc (r^2/2 - r^4/24)), sin = ts + tc (r - r^3/6) - ...
//   The heads of the table lie on the grid 2^-23, a multiple of the last
//   place of ts r, so Fast2Sum is exact whatever the magnitudes.  With 8192
//   entries r^2/2 < 7.4e-8 and its FP32 rounding stays below 2^-47.
// * Products drop only tail times tail; sums use TwoSum (Knuth) or, where
//   the order of magnitude is known, Fast2Sum (Dekker).
// Entries carry a relative error of about 2^-46.5, of random sign, against
// 2^-50 in pair64.cuh, whose sums of n entries one after another add an error
// that grows like sqrt(n): which of the two is the smaller in a product of a
// smooth density depends on n and k h (split_serves has the figures and the
// line).  A random or concentrated density gets the entries' own error: at
// n = 2,938 1.2e-15 against 2.4e-16.
#pragma once

#include <cstdint>

namespace hz {

constexpr int kSplitTable = 8192;  // (head, tail) of cos(2 pi j / 8192): 64 KB

struct FF {
    float h, l;
};

__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

__device__ __forceinline__ float rsqrt_seed(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float rcp_seed(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// s + e = a + b exactly (Knuth)
__device__ __forceinline__ FF two_sum(float a, float b)
{
    const float s = fadd(a, b), bb = fsub(s, a);
    return {s, fadd(fsub(a, fsub(s, bb)), fsub(b, bb))};
}

// the same for |a| >= |b|, or a a multiple of b's last place (Dekker)
__device__ __forceinline__ FF fast_two_sum(float a, float b)
{
    const float s = fadd(a, b);
    return {s, fsub(b, fsub(s, a))};
}

__device__ __forceinline__ FF ff_mul(FF a, FF b)
{
    const float p = fmul(a.h, b.h);
    return {p, ffma(a.l, b.h, ffma(a.h, b.l, ffma(a.h, b.h, -p)))};
}

__device__ __forceinline__ FF ff_neg(FF a) { return {-a.h, -a.l}; }

// FP32 head and tail of a double (48 bits).
__device__ __forceinline__ FF ff_of_double(double v)
{
    const float h = (float)v;
    return {h, (float)(v - (double)h)};
}

// W units (|W| < 2^62) plus the FP32 remainder e; sc32 = 2^32 units, sc8 =
// 2^8 units.  The caller adds 2^7 to W so that dropping its last 8 bits rounds.
__device__ __forceinline__ FF ff_of_int(long long W, float sc32, float sc8, float e)
{
    const int hi = (int)(W >> 32);
    const float f = __int2float_rn(hi);
    const int back = __float2int_rn(f);
    const int rem = (int)__funnelshift_l((unsigned)W, (unsigned)(hi - back), 24);
    return fast_two_sum(fmul(f, sc32), ffma(__int2float_rn(rem), sc8, e));
}

// rho = sqrt(r2) and y = 1 / rho, both normalised.
__device__ __forceinline__ void split_root(FF r2, FF &rho, FF &y)
{
    const float y0 = rsqrt_seed(r2.h);
    const float t = fmul(r2.h, y0);
    const float he = fmul(ffma(-t, y0, 1.0f), 0.5f);
    const float y1 = ffma(y0, he, y0);
    const float g = ffma(t, he, t);
    const float d = fadd(ffma(-g, g, r2.h), r2.l);
    rho = {g, fmul(d, fmul(y1, 0.5f))};
    const float e = ffma(-y1, rho.l, ffma(-y1, g, 1.0f));
    y = {y1, fmul(y1, ffma(e, e, e))};
}

// cos and sin of th; tab[j] = (head, tail) of cos(2 pi j / kSplitTable).
__device__ __forceinline__ void split_sincos(FF th, const float2 *tab, FF &c, FF &s)
{
    const float step1 = 0x1.921fb6p-11f, step2 = -0x1.777a5cp-36f, step3 = -0x1.ee59dap-61f;  // 2 pi / 8192
    const float jm = ffma(th.h, 1303.797294f, 12582912.0f);
    const int j = __float_as_int(jm);
    const float jf = fsub(jm, 12582912.0f);
    FF r = two_sum(ffma(-jf, step1, th.h), ffma(-jf, step2, th.l));
    r.l = ffma(-jf, step3, r.l);
    const float2 tc = tab[j & (kSplitTable - 1)];
    const float2 ts = tab[(j - kSplitTable / 4) & (kSplitTable - 1)];
    const float z = fmul(r.h, r.h);
    const float sl = ffma(fmul(r.h, z), -1.0f / 6.0f, r.l);                       // sin r - r.h
    const float cm = ffma(r.h, r.l, fmul(z, ffma(z, -1.0f / 24.0f, 0.5f)));       // 1 - cos r
    {
        const float p = fmul(ts.x, r.h);
        float l = ffma(ts.x, r.h, -p);
        l = ffma(ts.x, sl, l);
        l = ffma(ts.y, r.h, l);
        l = ffma(tc.x, cm, l);
        const FF q = fast_two_sum(tc.x, -p);
        c = {q.h, fsub(fadd(tc.y, q.l), l)};
    }
    {
        const float p = fmul(tc.x, r.h);
        float l = ffma(tc.x, r.h, -p);
        l = ffma(tc.x, sl, l);
        l = ffma(tc.y, r.h, l);
        l = ffma(-ts.x, cm, l);
        const FF q = fast_two_sum(ts.x, p);
        s = {q.h, fadd(fadd(ts.y, q.l), l)};
    }
}

// theta = rho - rho_c = w / (rho + rho_c)
__device__ __forceinline__ FF split_phase_offset(FF w, FF rho, FF rc)
{
    const FF d = two_sum(rho.h, rc.h);
    const float dl = fadd(d.l, fadd(rho.l, rc.l));
    const float z = rcp_seed(d.h);
    const float q = fmul(w.h, z);
    const float r = ffma(-q, dl, fadd(ffma(-q, d.h, w.h), w.l));
    return {q, fmul(r, z)};
}

// u = e^{i theta} (-y + i)
__device__ __forceinline__ void split_kernel(FF y, FF c, FF s, FF &ur, FF &ui)
{
    const FF yc = ff_mul(y, c), ys = ff_mul(y, s);
    const FF a = two_sum(-yc.h, -s.h);
    ur = {a.h, fsub(a.l, fadd(yc.l, s.l))};
    const FF b = two_sum(c.h, -ys.h);
    ui = {b.h, fadd(b.l, fsub(c.l, ys.l))};
}

// acc (h, l) += a b + sg c d (sg = +-1): products to 48 bits, head sums by
// TwoSum, tails summed at their own scale first.
template <int SG>
__device__ __forceinline__ void split_dot2(FF &acc, FF a, FF b, FF c, FF d)
{
    const FF p = ff_mul(a, b), q = ff_mul(c, d);
    const FF v = two_sum(p.h, SG > 0 ? q.h : -q.h);
    const float vl = fadd(v.l, SG > 0 ? fadd(p.l, q.l) : fsub(p.l, q.l));
    const FF t = two_sum(acc.h, v.h);
    acc = {t.h, fadd(acc.l, fadd(t.l, vl))};
}

}  // namespace hz
