// pair32.cuh -- the FP32 pair arithmetic of the single, batched and multi
// right-hand-side FP32 sweeps.
//
// SCALED records hold the coordinates times k (Rec32::lambda = k), so that
// rho below is k rho and the entry's factor is
//   e^{i rho} (-1/rho + i) / rho^2 (x_t - x_s).n   (k^2 on the densities).
// In a tile whose radius is at most kCentreRadius the phase is taken about the
// tile (tiles with near pairs too, in the single and batched sweeps, whose
// regularised pairs have sums of their own; not in the multi right-hand-side
// sweep, which has one sum for both): theta = rho - rc with rc = |x_t - o|, the FP32
// distance to the tile's origin, so |theta| is at most the radius, needs no
// range reduction before the SFU's sin and cos, and the tile's sum is turned
// once by e^{i rc} (Turn).  Any FP32 value near |x_t - o| serves as rc, as
// long as the turn belongs to that very value.  22 FP32 instructions and
// three SFU ones a pair, against 29 and three with the phase k rho reduced
// per pair, which wider tiles and the multi sweep's near tiles keep.
//
// Records with lambda = 1 (k below 2^-14, negative k, k tau below 2^-40:
// lambda32 in sweep_f32.cu) reduce k rho in revolutions with k/(2 pi) split
// into an FP32 head and tail.
#pragma once

#include <cstdint>

namespace hz {

constexpr float kCentreRadius = 6.0f;

// hi + lo += f without rounding loss (Knuth's TwoSum; FP32 only).
__device__ __forceinline__ void two_sum_acc(float &hi, float &lo, float f)
{
    const float s = hi + f;
    const float bp = s - hi;
    const float e = (hi - (s - bp)) + (f - bp);
    hi = s;
    lo += e;
}

struct Wave32 {
    float k, kh, kl;  // k and k/(2 pi) = kh + kl (lambda = 1 only)
};

// rc = |rel| and e^{i rc}.  The turn is common to the tile's sources, so its
// sine and cosine come from Taylor polynomials on [-pi/4, pi/4] (below 6e-8),
// not from the SFU (4e-7).  Keeping them to 48 bits changed no product's error
// and cost 2.5 % of the sweep.
struct Turn {
    float rc, c, s;
};

__device__ __forceinline__ Turn turn_of(const float3 rel)
{
    Turn t;
    t.rc = sqrtf(fmaf(rel.x, rel.x, fmaf(rel.y, rel.y, rel.z * rel.z)));
    const float n = fmaf(t.rc, 0.63661977236758134f, 12582912.f) - 12582912.f;
    const int q = (int)n;
    // less n pi/2, pi/2 = 1.5703125 (8 bits) + 4.838268e-4 (24 bits) + the rest
    float r = fmaf(-n, 1.5703125f, t.rc);
    r = fmaf(-n, 4.838267923332751e-4f, r);
    r = fmaf(-n, 2.563344151594519e-12f, r);
    const float z2 = r * r;
    const float sn = fmaf(r * z2, fmaf(z2, fmaf(z2, fmaf(z2, 1.f / 362880.f, -1.f / 5040.f), 1.f / 120.f), -1.f / 6.f), r);
    const float cs = fmaf(z2, fmaf(z2, fmaf(z2, fmaf(z2, fmaf(z2, -1.f / 3628800.f, 1.f / 40320.f), -1.f / 720.f), 1.f / 24.f), -0.5f), 1.f);
    const float a = (q & 1) ? cs : sn, b = (q & 1) ? sn : cs;
    t.s = (q & 2) ? -a : a;
    t.c = ((q + 1) & 2) ? -b : b;
    return t;
}

// (u1, u2) = (k sin + cos / rho, k cos - sin / rho) of the phase k rho - rc, and
// rr = 1 / rho^2 (k = 1 when SCALED).  SLOW: rc = 0 and the phase is reduced.
template <bool SCALED, bool SLOW>
__device__ __forceinline__ void kernel32(const Wave32 &w, float r2, float rc, float &u1, float &u2, float &rr)
{
    const float rinv = rsqrtf(r2);
    const float rho = r2 * rinv;
    float S, C;
    if (SCALED) {
        float th;
        if (SLOW) {
            // less the nearest multiple of 2 pi = 6.28125 + 0.00193... (n has at
            // most 10 bits, 6.28125 has 8: the first step is exact)
            const float n = fmaf(rho, 0.15915494309189535f, 12582912.f) - 12582912.f;
            th = fmaf(-n, 0.0019353071795864769f, fmaf(-n, 6.28125f, rho));
        } else {
            th = rho - rc;
        }
        __sincosf(th, &S, &C);
        u1 = fmaf(C, rinv, S);
        u2 = fmaf(-S, rinv, C);
    } else {
        // revolutions rho k/(2 pi) less the nearest integer (|rho kh| < 2^22:
        // add and remove 1.5 2^23), exact to ~2^-24 before the SFU
        const float n = fmaf(rho, w.kh, 12582912.f) - 12582912.f;
        const float f = fmaf(rho, w.kl, fmaf(rho, w.kh, -n));
        __sincosf(f * 6.28318530717958647692f, &S, &C);
        u1 = fmaf(C, rinv, w.k * S);
        u2 = fmaf(w.k, C, -S * rinv);
    }
    rr = rinv * rinv;
}

// re + i im times e^{i rc}, or e^{-i rc} for CONJ
template <bool CONJ>
__device__ __forceinline__ void turn_sum(const Turn &t, float &re, float &im)
{
    const float s = CONJ ? -t.s : t.s;
    const float r = fmaf(t.c, re, -s * im);
    im = fmaf(t.c, im, s * re);
    re = r;
}

// ---- two sources at a time: packed FP32 pairs (one issue slot for two) ----
typedef unsigned long long F2;

__device__ __forceinline__ F2 f2_pack(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(F2 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ F2 f2_rsqrt(F2 v)
{
    float a, b;
    f2_unpack(v, a, b);
    return f2_pack(rsqrtf(a), rsqrtf(b));
}
__device__ __forceinline__ void f2_sincos(F2 v, F2 &s, F2 &c)
{
    float a, b, sa, ca, sb, cb;
    f2_unpack(v, a, b);
    __sincosf(a, &sa, &ca);
    __sincosf(b, &sb, &cb);
    s = f2_pack(sa, sb);
    c = f2_pack(ca, cb);
}
__device__ __forceinline__ float f2_sum(F2 v)
{
    float a, b;
    f2_unpack(v, a, b);
    return a + b;
}

}  // namespace hz
