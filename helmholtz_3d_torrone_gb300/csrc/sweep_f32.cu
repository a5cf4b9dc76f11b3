// sweep_f32.cu -- FP32 matrix-free pair sweep (the bulk matvec of the
// mixed-precision solver): the same operator as sweep_f64.cu, evaluated on
// the FP32 and SFU pipes.
//
// Precision design:
//  * Sources are stored in a spatially blocked sweep order (8^3 node
//    blocks), so a tile of kTile32 consecutive sources is compact.  Each
//    tile has an FP64 origin o; sources hold FP32 offsets x_s - o.  Targets
//    and origins are held as FP32 head + tail pairs, and a target forms
//    x_t - o = (t_hi - o_hi) + (t_lo - o_lo): the head difference is rounded
//    to half an ulp of itself, so the offset of close pairs keeps FP32
//    relative precision with no FP64 instruction in the tile loop.
//  * Coordinates are stored times k, and the phase is taken about the source
//    tile's origin (pair32.cuh), except where a tile's radius is above 6 / k:
//    |k rho - k rho_c| is small, goes to the SFU's sin/cos without a range reduction, and the
//    tile's sum is turned by e^{i k rho_c} once.  Against the phase reduced per
//    pair the error to the FP64 product fell, 3.2e-7 -> 2.6e-7 of |K p| on the
//    64^3 torus (k = 15) and 3.4e-7 -> 3.1e-7 at 128^3 (k = 20).
//  * The near-field test rho <= tau is decided in FP64 (with the FP64
//    sweep's own arithmetic) whenever the FP32 rho^2 lies within 1e-4 of
//    tau^2, so FP32 and FP64 operators classify every pair alike.
//  * Per tile the contributions are summed in FP32; across tiles into FP32
//    head + tail pairs by TwoSum (about 48 significant bits).
//
// Throughput design: the kernel is bound by the FP32 and SFU pipes (22 FP32
// operations and three SFU ones a pair, 22 and 24 cycles of a partition), and
// GB300 runs FP64 at 1/64 of the FP32 rate, so the tile loop holds no FP64
// instruction.  Two sources at a time go through packed FP32 instructions
// (fma.f32x2), which do not raise the FP32 rate but halve its issue slots, so
// that the SFU's run beside them; a tile is staged as rows of 256 floats so
// that one 128-bit load gives two packed operands.  A source tile whose
// bounding sphere is farther than tau (with a 1e-3 margin) from the target
// tile's holds no near pair; a bit mask built once per tube in FP64 says
// which, and such tiles run the loop without near-field tests and phase
// reduction.  The factor k^2 sg/(4 pi) is folded into the densities (and
// divided out of the stored regularisation factors).  TMA bulk copies stage
// the tiles, double-buffered on mbarriers with bounded waits.  Block shape and
// targets per thread come from a small table of compiled variants; the
// autotuner times them on the operator's own data.
//
// One A p on GB300, first scalar with the phase reduced per pair, then packed
// and centred, then with units of equal cost and near tiles centred as well:
// n = 2,938 0.040 (packed) -> 0.037 ms, 9,765 0.149 -> 0.120, 19,532 0.603 ->
// 0.429 -> 0.383, 36,212 1.90 -> 1.31 -> 1.18, 145,272 28.5 -> 18.1 -> 17.7,
// 581,420 365 -> 257 -> 258 (1,307 Gpair/s).
#include "hz_internal.cuh"
#include "bulk_copy.cuh"
#include "pair32.cuh"

#include <cstring>
#include <type_traits>
#include <vector>

namespace hz {
namespace {

constexpr double kPi = 3.14159265358979323846264338328;

// Internal MODE bit: records scaled by k, phase centred on the source tile
// (pair32.cuh).
constexpr int SWEEP_SCALED = 4;

struct Args32 {
    int64_t n, npad, mwords;
    Wave32 wave;
    float tau2, guard_lo, guard_hi;  // (lambda tau)^2 and the tie band around it
    double tau;
    int scaled;  // lambda = k (batches: per operator)
    int sub;     // units of a tile
    const float4 *pos, *nrm;
    const float *soa;   // [tiles][kFixed][kTile32]: -x, -y, -z (tile-local), n, reg
    float *dens;        // [tiles][6][kTile32]: re, im, -im of w p and of pt
    const float4 *thi, *tlo, *ohi, *olo;
    const uint32_t *nearmask;
    const double4_32a *tpos;
    const int *perm;
    const double4_32a *pos64;  // tube order (for the near-field guard)
    const double *p_re, *p_im, *pt_re, *pt_im;
    double *q_re, *q_im, *qt_re, *qt_im;
    unsigned *err;
    // stream-K partition: CTA c takes the units [cta_begin(c), cta_begin(c + 1))
    // of the blocks x tiles x sub (target block, part of a source tile) ones
    const int64_t *cuts;   // units at equal costs (build_cuts32); NULL: a CTA takes a block
    unsigned *done;        // per target block: units whose sums lie in partial
    int nctas;
    double4_32a *partial;  // [P][2][slots per block]: (A re, A im, A^H re, A^H im)
};

constexpr int kFixed = kFixed32;  // staged floats per source besides the densities
template <int MODE>
constexpr int kDens = 3 * ((MODE & SWEEP_PAIR) == SWEEP_PAIR ? 2 : 1);
template <int MODE>
constexpr int kStage = (kFixed + kDens<MODE>) * kTile32;  // floats of a staged tile

// A tile counts `sub` units, and the FP32 sums over a unit are added to the
// cross-tile sums one by one, so products agree to the rounding of those sums
// (about 2^-48) wherever the units are cut: variants and grid sizes change
// their last bits.  Whole tiles are the cheapest (a unit's end costs 2 % of a half), but
// small tubes need parts for every CTA to have its share: n = 2,938 0.042 ms
// with tiles, 0.039 with halves, 0.037 with quarters; n = 9,765 0.123 and
// 0.120 with halves; n = 145,272 17.5 with tiles, 17.9 with halves.
constexpr int kRun32 = 64;  // sources of the smallest unit
int sub_of(int64_t ntiles) { return ntiles < 24 ? 4 : ntiles < 80 ? 2 : 1; }

// Relative cost of a tile: far, near tile (near-field test, its branch
// taken now and then), the target tile itself (taken for most sources).
constexpr int kCostFar = 16, kCostNear = 19, kCostSelf = 30;
constexpr int kCuts = 16384;  // equal-cost cuts kept per tube: 26 or more a CTA (608 CTAs)

// First unit of CTA c of P.  Cut by count, the CTAs with the near tiles set
// the time: 0.149 ms at n = 9,765 and 1.30 at n = 36,212, of which 0.03 and
// 0.2 were the others' waiting.
__device__ __forceinline__ int64_t cta_begin(const Args32 &a, int c)
{
    if (!a.cuts) return (int64_t)c * (a.npad / kTile32) * a.sub;
    return __ldg(a.cuts + (unsigned)c * (unsigned)kCuts / (unsigned)a.nctas);
}

// Largest c with cta_begin(c) <= u (all threads of a block take part).
template <class Begin>
__device__ __forceinline__ int cta_of_unit(int64_t u, int nctas, const Begin &begin)
{
    int count = 0;
    for (int c0 = 0; c0 < nctas; c0 += blockDim.x) {
        const int c = c0 + (int)threadIdx.x;
        count += __syncthreads_count(c < nctas && begin(c) <= u);
    }
    return count - 1;
}

// Densities of slot s, scale (w p, pt) in FP32, scale = lambda^2 sg / (4 pi).
__device__ __forceinline__ void store_dens(float *dens, int64_t s, int half, float re, float im)
{
    float *d = dens + (s / kTile32) * (6 * kTile32) + half * (3 * kTile32) + (s & (kTile32 - 1));
    d[0] = re;
    d[kTile32] = im;
    d[2 * kTile32] = -im;
}

__global__ void prep32_kernel(int64_t npad, const int *__restrict__ perm, const double4_32a *__restrict__ tpos,
                              const double *__restrict__ p_re, const double *__restrict__ p_im,
                              const double *__restrict__ pt_re, const double *__restrict__ pt_im, double scale,
                              float *__restrict__ dens, unsigned *__restrict__ done)
{
    if (blockIdx.x == 0)
        for (int64_t b = threadIdx.x; b < npad / kTile32; b += blockDim.x) done[b] = 0;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < npad; s += (int64_t)gridDim.x * blockDim.x) {
        const int c = perm[s];
        const double ws = (c >= 0) ? tpos[s].w * scale : 0.0;
        if (p_re) store_dens(dens, s, 0, c >= 0 ? (float)(ws * p_re[c]) : 0.f, c >= 0 ? (float)(ws * p_im[c]) : 0.f);
        if (pt_re)
            store_dens(dens, s, 1, c >= 0 ? (float)(scale * pt_re[c]) : 0.f, c >= 0 ? (float)(scale * pt_im[c]) : 0.f);
    }
}

// What a thread holds of its TG targets.
template <int TG>
struct Targets {
    float3 th[TG], tl[TG], tn[TG];  // position head and tail, normal
    float reg[TG];
};

// Cross-tile sums: FP32 head + tail (TwoSum), about 48 significant bits.
template <int TG>
struct Sums {
    float hAr[TG], lAr[TG], hAi[TG], lAi[TG], hHr[TG], lHr[TG], hHi[TG], lHi[TG];
};

// The FP64 decision rho <= tau of a pair whose FP32 rho^2 is close to tau^2.
__device__ __noinline__ bool near_exact(const Args32 &a, int64_t tslot, int64_t sslot)
{
    const int c = a.perm[sslot];
    if (c < 0) return false;
    const double4_32a q = a.pos64[c];
    const double4_32a tp = a.tpos[tslot];
    const double x1 = tp.x - q.x, x2 = tp.y - q.y, x3 = tp.z - q.z;
    return !(sqrt(x1 * x1 + x2 * x2 + x3 * x3) > a.tau);
}

__device__ __forceinline__ bool is_near(const Args32 &a, float r2, int64_t tslot, int64_t sslot)
{
    if (r2 > a.guard_lo && r2 < a.guard_hi) return near_exact(a, tslot, sslot);
    return r2 <= a.tau2;
}

// A unit of a tile against TG targets, scalar (records with lambda = 1).  Four
// sources' values come by one 128-bit load a row (a load a value: 13 to 21 %
// more time at n = 19,532).
template <int MODE, bool DIR, int NT, int TG, bool NEAR>
__device__ __forceinline__ void unit_scalar(const Args32 &a, const float *st, int j0, int j1,
                                            const float3 (&rel)[TG], const Targets<TG> &t, int64_t tslot0,
                                            int64_t sslot0, float (&fAr)[TG], float (&fAi)[TG], float (&fHr)[TG],
                                            float (&fHi)[TG])
{
    constexpr int ROWS = kFixed + kDens<MODE>, H0 = ROWS - 3;  // the last three rows: the densities of A^H
#pragma unroll
    for (int g = 0; g < TG; g++) fAr[g] = fAi[g] = fHr[g] = fHi[g] = 0.f;
#pragma unroll 1
    for (int j = j0; j < j1; j += 4) {
        float v[ROWS][4];
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const float4 x = *reinterpret_cast<const float4 *>(st + r * kTile32 + j);
            v[r][0] = x.x;
            v[r][1] = x.y;
            v[r][2] = x.z;
            v[r][3] = x.w;
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int g = 0; g < TG; g++) {
                const float dx = rel[g].x + v[0][q], dy = rel[g].y + v[1][q], dz = rel[g].z + v[2][q];
                const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                const bool near = NEAR && is_near(a, r2, tslot0 + (int64_t)g * NT, sslot0 + j + q);
                float u1, u2, rr;
                kernel32<false, true>(a.wave, r2, 0.f, u1, u2, rr);
                const float ps = fmaf(dx, v[3][q], fmaf(dy, v[4][q], dz * v[5][q]));        // (x_t - x_s).n_s
                const float pt = fmaf(dx, t.tn[g].x, fmaf(dy, t.tn[g].y, dz * t.tn[g].z));  // (x_t - x_s).n_t
                if (MODE & SWEEP_A) {
                    const float f = rr * (DIR ? ps : pt), dr = v[kFixed][q], di = v[kFixed + 1][q];
                    const float vr = near ? (DIR ? v[6][q] : t.reg[g]) : -u1 * f, vi = near ? 0.f : u2 * f;
                    fAr[g] = fmaf(vr, dr, fmaf(-vi, di, fAr[g]));
                    fAi[g] = fmaf(vr, di, fmaf(vi, dr, fAi[g]));
                }
                if (MODE & SWEEP_AH) {
                    const float f = rr * (DIR ? pt : ps), dr = v[H0][q], di = v[H0 + 1][q];
                    const float vr = near ? (DIR ? t.reg[g] : v[6][q]) : u1 * f, vi = near ? 0.f : u2 * f;
                    fHr[g] = fmaf(vr, dr, fmaf(-vi, di, fHr[g]));
                    fHi[g] = fmaf(vr, di, fmaf(vi, dr, fHi[g]));
                }
            }
    }
}

// How a tile is summed: phase centred, the same with the near-field test, or
// (tiles wider than kCentreRadius) phase reduced per pair and the test.
enum { TILE_FAR = 0, TILE_NEAR = 1, TILE_WIDE = 2 };

// A unit of a tile, two sources at a time in packed FP32.  With y = 1/rho,
// e^{i theta} = C + i S and q the projection over rho^2, A's entry times d is
// q (-(S e1 + C e2) + i (C e1 - S e2)), e1 = dr - y di, e2 = di + y dr (A^H:
// conj(d) and the real part's sign), so that no operand needs a negation (-im
// is staged).  Near pairs add their regularisation factor times d to sums of
// their own (they take no phase) and go on at rho^2 = 1e16, where the rest of
// the loop adds 1e-16 of the entry's scale.
template <int MODE, bool DIR, int NT, int TG, int KIND>
__device__ __forceinline__ void unit_packed(const Args32 &a, const float *st, int j0, int j1, const float3 (&rel)[TG],
                                            const Targets<TG> &t, const Turn (&turn)[TG], int64_t tslot0,
                                            int64_t sslot0, float (&fAr)[TG], float (&fAi)[TG], float (&fHr)[TG],
                                            float (&fHi)[TG])
{
    constexpr int T = kTile32;
    constexpr bool A = (MODE & SWEEP_A) != 0, H = (MODE & SWEEP_AH) != 0;
    constexpr bool SRC = (A && DIR) || (H && !DIR), TGT = (A && !DIR) || (H && DIR);
    F2 rx[TG], ry[TG], rz[TG], nrc[TG], tx[TG], ty[TG], tz[TG];
    F2 aR[TG], aI[TG], aJ[TG], hR[TG], hI[TG], hJ[TG];
#pragma unroll
    for (int g = 0; g < TG; g++) {
        rx[g] = f2_pack(rel[g].x, rel[g].x);
        ry[g] = f2_pack(rel[g].y, rel[g].y);
        rz[g] = f2_pack(rel[g].z, rel[g].z);
        if (KIND != TILE_WIDE) nrc[g] = f2_pack(-turn[g].rc, -turn[g].rc);
        if (TGT) {
            tx[g] = f2_pack(t.tn[g].x, t.tn[g].x);
            ty[g] = f2_pack(t.tn[g].y, t.tn[g].y);
            tz[g] = f2_pack(t.tn[g].z, t.tn[g].z);
        }
        aR[g] = aI[g] = aJ[g] = hR[g] = hI[g] = hJ[g] = 0;
        if (A) fAr[g] = fAi[g] = 0.f;
        if (H) fHr[g] = fHi[g] = 0.f;
    }
    auto at = [&](int row, int j) { return *reinterpret_cast<const ulonglong2 *>(st + row * T + j); };
    // A fixed inner count lets the compiler unroll: with the unit's length as
    // the bound the sweep was 3 % slower.
#pragma unroll 1
    for (int jb = j0; jb < j1; jb += kRun32) {
#pragma unroll 8
        for (int j = jb; j < jb + kRun32; j += 4) {
            const ulonglong2 X = at(0, j), Y = at(1, j), Z = at(2, j);
            ulonglong2 NX, NY, NZ, DR, DI, DN, ER, EI, EN;
            if (SRC) {
                NX = at(3, j);
                NY = at(4, j);
                NZ = at(5, j);
            }
            if (A) {
                DR = at(kFixed, j);
                DI = at(kFixed + 1, j);
                DN = at(kFixed + 2, j);
            }
            if (H) {
                ER = at(kFixed + kDens<MODE> - 3, j);
                EI = at(kFixed + kDens<MODE> - 2, j);
                EN = at(kFixed + kDens<MODE> - 1, j);
            }
            F2 DX[TG][2], DY[TG][2], DZ[TG][2], R2[TG][2];
            auto offsets = [&](int g, int h) {
                DX[g][h] = f2_add(rx[g], h ? X.y : X.x);
                DY[g][h] = f2_add(ry[g], h ? Y.y : Y.x);
                DZ[g][h] = f2_add(rz[g], h ? Z.y : Z.x);
                R2[g][h] = f2_fma(DX[g][h], DX[g][h], f2_fma(DY[g][h], DY[g][h], f2_mul(DZ[g][h], DZ[g][h])));
            };
#pragma unroll
            for (int g = 0; g < TG; g++) {
                if (KIND != TILE_FAR) {
                    offsets(g, 0);
                    offsets(g, 1);
                    float r[4];
                    f2_unpack(R2[g][0], r[0], r[1]);
                    f2_unpack(R2[g][1], r[2], r[3]);
                    if (fminf(fminf(r[0], r[1]), fminf(r[2], r[3])) < a.guard_hi) {
                        bool nr[4], tie = false;
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            nr[q] = r[q] <= a.tau2;
                            tie |= r[q] > a.guard_lo && r[q] < a.guard_hi;
                        }
                        if (tie) {
#pragma unroll
                            for (int q = 0; q < 4; q++)
                                nr[q] = is_near(a, r[q], tslot0 + (int64_t)g * NT, sslot0 + j + q);
                        }
                        const ulonglong2 RG = at(6, j);
                        float w[4];
                        f2_unpack(RG.x, w[0], w[1]);
                        f2_unpack(RG.y, w[2], w[3]);
                        auto add = [&](float own, bool src, const ulonglong2 &re, const ulonglong2 &im, float &fr,
                                       float &fi) {
                            float x[4], y[4];
                            f2_unpack(re.x, x[0], x[1]);
                            f2_unpack(re.y, x[2], x[3]);
                            f2_unpack(im.x, y[0], y[1]);
                            f2_unpack(im.y, y[2], y[3]);
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                const float v = nr[q] ? (src ? w[q] : own) : 0.f;
                                fr = fmaf(v, x[q], fr);
                                fi = fmaf(v, y[q], fi);
                            }
                        };
                        if (A) add(t.reg[g], DIR, DR, DI, fAr[g], fAi[g]);
                        if (H) add(t.reg[g], !DIR, ER, EI, fHr[g], fHi[g]);
#pragma unroll
                        for (int q = 0; q < 4; q++) r[q] = nr[q] ? 1e16f : r[q];
                        R2[g][0] = f2_pack(r[0], r[1]);
                        R2[g][1] = f2_pack(r[2], r[3]);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                auto of = [&](const ulonglong2 &v) { return h ? v.y : v.x; };
#pragma unroll
                for (int g = 0; g < TG; g++) {
                    if (KIND == TILE_FAR) offsets(g, h);
                    const F2 dx = DX[g][h], dy = DY[g][h], dz = DZ[g][h], r2 = R2[g][h];
                    const F2 y = f2_rsqrt(r2);
                    F2 S, C, th;
                    if (KIND == TILE_WIDE) {
                        // less the nearest multiple of 2 pi = 6.28125 + 0.00193...
                        const F2 rho = f2_mul(r2, y), M = f2_pack(12582912.f, 12582912.f);
                        const F2 n = f2_add(f2_fma(rho, f2_pack(0.15915494309189535f, 0.15915494309189535f), M),
                                            f2_pack(-12582912.f, -12582912.f));
                        th = f2_fma(n, f2_pack(-0.0019353071795864769f, -0.0019353071795864769f),
                                    f2_fma(n, f2_pack(-6.28125f, -6.28125f), rho));
                    } else {
                        th = f2_fma(r2, y, nrc[g]);
                    }
                    f2_sincos(th, S, C);
                    const F2 yy = f2_mul(y, y);
                    F2 ps, pt;
                    if (SRC) ps = f2_mul(yy, f2_fma(dx, of(NX), f2_fma(dy, of(NY), f2_mul(dz, of(NZ)))));
                    if (TGT) pt = f2_mul(yy, f2_fma(dx, tx[g], f2_fma(dy, ty[g], f2_mul(dz, tz[g]))));
                    F2 e1, e2, f1, f2;
                    if (A) {
                        const F2 q = DIR ? ps : pt;
                        e1 = f2_mul(q, f2_fma(y, of(DN), of(DR)));
                        e2 = f2_mul(q, f2_fma(y, of(DR), of(DI)));
                    }
                    if (H) {
                        const F2 q = DIR ? pt : ps;
                        f1 = f2_mul(q, f2_fma(y, of(EI), of(ER)));
                        f2 = f2_mul(q, f2_fma(y, of(ER), of(EN)));
                    }
                    if (A) {
                        aR[g] = f2_fma(S, e1, f2_fma(C, e2, aR[g]));
                        aI[g] = f2_fma(C, e1, aI[g]);
                        aJ[g] = f2_fma(S, e2, aJ[g]);
                    }
                    if (H) {
                        hR[g] = f2_fma(S, f1, f2_fma(C, f2, hR[g]));
                        hI[g] = f2_fma(C, f1, hI[g]);
                        hJ[g] = f2_fma(S, f2, hJ[g]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int g = 0; g < TG; g++) {
        if (A) {
            float re = -f2_sum(aR[g]), im = f2_sum(aI[g]) - f2_sum(aJ[g]);
            if (KIND != TILE_WIDE) turn_sum<false>(turn[g], re, im);
            fAr[g] += re;
            fAi[g] += im;
        }
        if (H) {
            float re = f2_sum(hR[g]), im = f2_sum(hI[g]) - f2_sum(hJ[g]);
            if (KIND != TILE_WIDE) turn_sum<true>(turn[g], re, im);
            fHr[g] += re;
            fHi[g] += im;
        }
    }
}

// The pairs of the block's targets with the units [q0, q1) of the staged
// source tile, added to sum.
template <int MODE, bool DIR, int NT, int TG>
__device__ __forceinline__ void tile_pairs(const Args32 &a, const float *st, int64_t tile, int q0, int q1, bool near,
                                           const float3 (&rel)[TG], const Turn (&turn)[TG], bool centred,
                                           const Targets<TG> &t, int64_t slot0, Sums<TG> &sum)
{
    const int64_t sslot0 = tile * kTile32;
    const int len = kTile32 / a.sub;
    auto units = [&](auto unit) {
#pragma unroll 1
        for (int q = q0; q < q1; q++) {
            float fAr[TG], fAi[TG], fHr[TG], fHi[TG];
            unit(q * len, q * len + len, fAr, fAi, fHr, fHi);
#pragma unroll
            for (int g = 0; g < TG; g++) {
                if (MODE & SWEEP_A) {
                    two_sum_acc(sum.hAr[g], sum.lAr[g], fAr[g]);
                    two_sum_acc(sum.hAi[g], sum.lAi[g], fAi[g]);
                }
                if (MODE & SWEEP_AH) {
                    two_sum_acc(sum.hHr[g], sum.lHr[g], fHr[g]);
                    two_sum_acc(sum.hHi[g], sum.lHi[g], fHi[g]);
                }
            }
        }
    };
    if (!(MODE & SWEEP_SCALED)) {
        units([&](int j0, int j1, float (&fAr)[TG], float (&fAi)[TG], float (&fHr)[TG], float (&fHi)[TG]) {
            if (near)
                unit_scalar<MODE, DIR, NT, TG, true>(a, st, j0, j1, rel, t, slot0, sslot0, fAr, fAi, fHr, fHi);
            else
                unit_scalar<MODE, DIR, NT, TG, false>(a, st, j0, j1, rel, t, slot0, sslot0, fAr, fAi, fHr, fHi);
        });
    } else if (!centred) {
        units([&](int j0, int j1, float (&fAr)[TG], float (&fAi)[TG], float (&fHr)[TG], float (&fHi)[TG]) {
            unit_packed<MODE, DIR, NT, TG, TILE_WIDE>(a, st, j0, j1, rel, t, turn, slot0, sslot0, fAr, fAi,
                                                            fHr, fHi);
        });
    } else if (near) {
        units([&](int j0, int j1, float (&fAr)[TG], float (&fAi)[TG], float (&fHr)[TG], float (&fHi)[TG]) {
            unit_packed<MODE, DIR, NT, TG, TILE_NEAR>(a, st, j0, j1, rel, t, turn, slot0, sslot0, fAr, fAi,
                                                            fHr, fHi);
        });
    } else {
        units([&](int j0, int j1, float (&fAr)[TG], float (&fAi)[TG], float (&fHr)[TG], float (&fHi)[TG]) {
            unit_packed<MODE, DIR, NT, TG, TILE_FAR>(a, st, j0, j1, rel, t, turn, slot0, sslot0, fAr, fAi,
                                                            fHr, fHi);
        });
    }
}

template <int NT, int TG>
__device__ __forceinline__ void load_targets(const Args32 &a, int64_t slot0, Targets<TG> &t, Sums<TG> &sum)
{
#pragma unroll
    for (int g = 0; g < TG; g++) {
        const int64_t s = slot0 + (int64_t)g * NT;
        const float4 h = a.thi[s], l = a.tlo[s], nn = a.nrm[s];
        t.th[g] = make_float3(h.x, h.y, h.z);
        t.tl[g] = make_float3(l.x, l.y, l.z);
        t.tn[g] = make_float3(nn.x, nn.y, nn.z);
        t.reg[g] = a.pos[s].w;
        sum.hAr[g] = sum.lAr[g] = sum.hAi[g] = sum.lAi[g] = 0.f;
        sum.hHr[g] = sum.lHr[g] = sum.hHi[g] = sum.lHi[g] = 0.f;
    }
}

// x_t - o of the targets (the head difference is rounded once, to half an ulp
// of itself) and the turns of a centred tile.
template <int MODE, int TG>
__device__ __forceinline__ bool tile_offsets(const Args32 &a, int64_t tile, const Targets<TG> &t,
                                             float3 (&rel)[TG], Turn (&turn)[TG])
{
    const float4 oh = a.ohi[tile], ol = a.olo[tile];
    const bool centred = (MODE & SWEEP_SCALED) && oh.w <= kCentreRadius;
#pragma unroll
    for (int g = 0; g < TG; g++) {
        rel[g] = make_float3((t.th[g].x - oh.x) + (t.tl[g].x - ol.x), (t.th[g].y - oh.y) + (t.tl[g].y - ol.y),
                             (t.th[g].z - oh.z) + (t.tl[g].z - ol.z));
        if (centred) turn[g] = turn_of(rel[g]);
    }
    return centred;
}

template <int MODE>
__device__ __forceinline__ void issue_tile(const Args32 &a, int64_t tile, float *st, uint64_t *bar)
{
    constexpr uint32_t fixed = kFixed * kTile32 * sizeof(float), dens = kDens<MODE> * kTile32 * sizeof(float);
    mbar_arrive_expect_tx(bar, fixed + dens);
    bulk_g2s(st, a.soa + tile * (kFixed * kTile32), fixed, bar);
    bulk_g2s(st + kFixed * kTile32, a.dens + tile * (6 * kTile32) + ((MODE & SWEEP_A) ? 0 : 3 * kTile32), dens, bar);
}

// Final value of one target slot: q = sum + p/2 (A), qt = w sum + pt/2 (A^H).
template <int MODE>
__device__ __forceinline__ void write_slot(const Args32 &a, int64_t s, double ar, double ai, double hr, double hi)
{
    const int c = a.perm[s];
    if (c < 0) return;
    if (MODE & SWEEP_A) {
        if (!isfinite(ar) || !isfinite(ai)) atomicOr(a.err, DEV_ERR_NONFINITE);
        a.q_re[c] = ar + 0.5 * a.p_re[c];
        a.q_im[c] = ai + 0.5 * a.p_im[c];
    }
    if (MODE & SWEEP_AH) {
        const double w = a.tpos[s].w;
        const double r = w * hr, i = w * hi;
        if (!isfinite(r) || !isfinite(i)) atomicOr(a.err, DEV_ERR_NONFINITE);
        a.qt_re[c] = r + 0.5 * a.pt_re[c];
        a.qt_im[c] = i + 0.5 * a.pt_im[c];
    }
}

// The pieces of a target block that the partition split between CTAs, summed
// in CTA order by whichever CTA finishes last: the caller has written `units`
// units' sums to partial; begin(c) is the partition, u0 the block's first unit,
// total its units, and write(slot, sums) stores a slot.
template <int SLOTS, class Begin, class Write>
__device__ __forceinline__ void finish_block(unsigned *done, unsigned units, unsigned total, int64_t u0, int nctas,
                                             const double4_32a *partial, const Begin &begin, const Write &write)
{
    __shared__ unsigned before;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) before = atomicAdd(done, units);
    __syncthreads();
    if (before + units != total) return;
    __threadfence();
    const int lo = cta_of_unit(u0, nctas, begin), hi = cta_of_unit(u0 + total - 1, nctas, begin);
    for (int k = threadIdx.x; k < SLOTS; k += blockDim.x) {
        double ar = 0.0, ai = 0.0, hr = 0.0, hi_ = 0.0;
#pragma unroll 4
        for (int c = lo; c <= hi; c++) {
            const int64_t b = begin(c);
            if (b == begin(c + 1)) continue;  // a CTA without units
            // a CTA's first block is its slot 0, its last one slot 1
            const double2 *v = reinterpret_cast<const double2 *>(partial + ((int64_t)c * 2 + (b < u0)) * SLOTS + k);
            const double2 x = __ldcg(v), y = __ldcg(v + 1);
            ar += x.x;
            ai += x.y;
            hr += y.x;
            hi_ += y.y;
        }
        write(k, ar, ai, hr, hi_);
    }
}

// Persistent stream-K sweep: every CTA walks its own contiguous range of
// (target block, part of a source tile) units, ranges of equal cost whatever
// the tube size.  A target block that lies wholly in one CTA's range is written
// out directly; the pieces of a block split between CTAs go to the partial
// buffer (slot 0: the CTA's first block, slot 1: its last), and the CTA that
// finishes a block adds them up (as a kernel of its own that took 10 us and a
// launch, mostly 64-bit divisions).
template <int MODE, bool DIR, int NT, int TG, int MINB>
__global__ void __launch_bounds__(NT, MINB) sweep32_kernel(Args32 a)
{
    constexpr int SLOTS = NT * TG;
    static_assert(SLOTS == kTile32, "one target tile per block: every shape then runs the same loops on a pair");
    __shared__ alignas(128) float stage[2][kStage<MODE>];
    __shared__ alignas(8) uint64_t bar[2];

    const int64_t ntiles = a.npad / kTile32, bu = ntiles * a.sub;
    const int64_t u_begin = cta_begin(a, blockIdx.x), u_end = cta_begin(a, blockIdx.x + 1);
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    __syncthreads();
    if (u_begin >= u_end) return;
    if (threadIdx.x == 0) issue_tile<MODE>(a, (u_begin % bu) / a.sub, stage[0], &bar[0]);
    int seg = 0;
    unsigned it = 0;
    for (int64_t u = u_begin; u < u_end;) {
        const int64_t blk = u / bu, u0 = blk * bu, seg_begin = u;
        const int64_t seg_end = (u_end < u0 + bu) ? u_end : u0 + bu;
        const int64_t slot0 = blk * SLOTS + threadIdx.x;
        Targets<TG> t;
        Sums<TG> sum;
        load_targets<NT, TG>(a, slot0, t, sum);
        const uint32_t *mrow = a.nearmask + blk * a.mwords;  // the near-tile mask of this target tile
        for (; u < seg_end; it++) {
            const int buf = (int)(it & 1);
            const int64_t tile = (u - u0) / a.sub;
            const int q0 = (int)((u - u0) % a.sub), q1 = (int)min((int64_t)a.sub, q0 + seg_end - u);
            u += q1 - q0;
            if (threadIdx.x == 0 && u < u_end)
                issue_tile<MODE>(a, tile + 1 < ntiles ? tile + 1 : 0, stage[buf ^ 1], &bar[buf ^ 1]);
            const bool near = (__ldg(mrow + (tile >> 5)) >> (tile & 31)) & 1u;
            float3 rel[TG];
            Turn turn[TG];
            const bool centred = tile_offsets<MODE, TG>(a, tile, t, rel, turn);
            const bool ok = mbar_wait_bounded(&bar[buf], (it >> 1) & 1, g_data_wait_limit);
            if (__syncthreads_or(!ok)) {
                if (threadIdx.x == 0) {
                    atomicOr(a.err, DEV_ERR_WAIT);
                    mbar_drain(&bar[buf], (it >> 1) & 1, &bar[buf ^ 1], ((it + 1) >> 1) & 1, u < u_end);
                }
                return;
            }
            tile_pairs<MODE, DIR, NT, TG>(a, stage[buf], tile, q0, q1, near, rel, turn, centred, t, slot0, sum);
            __syncthreads();
        }
        const bool whole = seg_end - seg_begin == bu;
#pragma unroll
        for (int g = 0; g < TG; g++) {
            const double ar = (double)sum.hAr[g] + (double)sum.lAr[g], ai = (double)sum.hAi[g] + (double)sum.lAi[g];
            const double hr = (double)sum.hHr[g] + (double)sum.lHr[g], hi = (double)sum.hHi[g] + (double)sum.lHi[g];
            if (whole) {
                write_slot<MODE>(a, slot0 + (int64_t)g * NT, ar, ai, hr, hi);
            } else {
                a.partial[((int64_t)blockIdx.x * 2 + seg) * SLOTS + threadIdx.x + g * NT] =
                    make_double4_32a(ar, ai, hr, hi);
            }
        }
        if (!whole)
            finish_block<SLOTS>(
                a.done + blk, (unsigned)(seg_end - seg_begin), (unsigned)bu, u0, a.nctas, a.partial,
                [&](int c) { return cta_begin(a, c); },
                [&](int k, double ar, double ai, double hr, double hi) {
                    write_slot<MODE>(a, blk * SLOTS + k, ar, ai, hr, hi);
                });
        seg = 1;
    }
}

// Cost of 32 source tiles of a target tile's row.
__device__ __forceinline__ int word_cost(const uint32_t *mrow, int64_t w, int64_t ntiles, int64_t self)
{
    const int tiles = (int)min((int64_t)32, ntiles - w * 32);
    return tiles * kCostFar + __popc(mrow[w]) * (kCostNear - kCostFar) +
           ((self >> 5) == w ? kCostSelf - kCostNear : 0);
}

// rows[t] = cost of target tile t's row
__global__ void __launch_bounds__(256) row_cost_kernel(int64_t ntiles, int64_t mwords, const uint32_t *__restrict__ mask,
                                                       int64_t *__restrict__ rows)
{
    const int64_t t = blockIdx.x * (int64_t)8 + (threadIdx.x >> 5);
    if (t >= ntiles) return;
    int64_t c = 0;
    for (int64_t w = threadIdx.x & 31; w < mwords; w += 32) c += word_cost(mask + t * mwords, w, ntiles, t);
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) rows[t] = c;
}

// rows: exclusive prefix sums, rows[ntiles] the total (one block)
__global__ void __launch_bounds__(1024) row_scan_kernel(int64_t ntiles, int64_t *__restrict__ rows)
{
    __shared__ int64_t part[32], carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t b = 0; b <= ntiles; b += 1024) {
        const int64_t t = b + threadIdx.x;
        const int64_t v = t < ntiles ? rows[t] : 0;
        int64_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) part[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int64_t p = part[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t y = __shfl_up_sync(0xffffffffu, p, o);
                if (lane >= o) p += y;
            }
            part[lane] = p;
        }
        __syncthreads();
        const int64_t base = carry + (warp ? part[warp - 1] : 0);
        if (t <= ntiles) rows[t] = base + x - v;
        __syncthreads();
        if (threadIdx.x == 0) carry += part[31];
        __syncthreads();
    }
}

// First lane whose inclusive sum of v exceeds r (the caller knows there is
// one), r less the sums before it.
__device__ __forceinline__ int lane_of(int v, int64_t &r)
{
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if ((int)(threadIdx.x & 31) >= o) x += y;
    }
    const int f = __ffs(__ballot_sync(0xffffffffu, x > r)) - 1;
    r -= __shfl_sync(0xffffffffu, x - v, f);
    return f;
}

// cuts[i]: the unit at cost i / kCuts of the total (one warp a cut)
__global__ void __launch_bounds__(256) cuts_kernel(int64_t ntiles, int64_t mwords, int sub,
                                                   const uint32_t *__restrict__ mask,
                                                   const int64_t *__restrict__ rows, int64_t *__restrict__ cuts)
{
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i > kCuts) return;
    const int64_t total = rows[ntiles], x = total / kCuts * i + total % kCuts * i / kCuts;
    if (i == kCuts) {
        if (lane == 0) cuts[i] = ntiles * ntiles * sub;
        return;
    }
    int64_t lo = 0;  // the last row with rows[lo] <= x
    for (int64_t len = ntiles; len > 1;) {
        const int64_t step = (len + 31) / 32, at = lane * step;
        const int k = __popc(__ballot_sync(0xffffffffu, at < len && rows[lo + (at < len ? at : 0)] <= x)) - 1;
        lo += k * step;
        len = min(step, len - k * step);
    }
    const uint32_t *mrow = mask + lo * mwords;
    int64_t r = x - rows[lo], w = 0;
    for (;; w += 32) {
        const int c = w + lane < mwords ? word_cost(mrow, w + lane, ntiles, lo) : 0;
        const int sum = __reduce_add_sync(0xffffffffu, c);
        if (r < sum) {
            w += lane_of(c, r);
            break;
        }
        r -= sum;
    }
    const int64_t t = w * 32 + lane;
    const int c = t >= ntiles ? 0 : t == lo ? kCostSelf : ((mrow[w] >> lane) & 1u) ? kCostNear : kCostFar;
    const int f = lane_of(c, r);
    if (lane == 0) {
        const int64_t tile = w * 32 + f;
        const int ct = tile == lo ? kCostSelf : ((mrow[w] >> f) & 1u) ? kCostNear : kCostFar;
        cuts[i] = (lo * ntiles + tile) * sub + (int)(r * sub / ct);
    }
}

// ------------------------------------------------------------ batches
// One operator of a batch: its sweep arguments (records, densities,
// constants) and its place in the batch's unit and block numbering.  The
// product vectors are columns of [R][stride] arrays passed to the launch.
struct BatchOp {
    Args32 a;
    int64_t unit0;   // first global unit
    int64_t cost0, cost;  // costs of the operators before it, and its own
    const int64_t *rows;  // its row costs (rows[ntiles]: the total)
    int64_t ntiles;
    int dir;
    int col;         // column of P and Q
    double scale;    // lambda^2 sg / (4 pi), folded into the densities
};

struct BatchVec {
    const double *p_re, *p_im;
    double *q_re, *q_im;
    int64_t stride;
    int64_t *begins;  // [nctas + 1] partition of the launch
};

// First unit of CTA c: the operators' cuts laid end to end by their costs.
__device__ __forceinline__ int64_t batch_begin(const BatchOp *ops, int nops, int nctas, int c)
{
    const int64_t total = ops[nops - 1].cost0 + ops[nops - 1].cost;
    const int64_t x = total / nctas * c + total % nctas * c / nctas;
    int o = 0;
    while (o + 1 < nops && x >= ops[o + 1].cost0) o++;
    const int64_t y = x - ops[o].cost0, n = ops[o].cost;
    return ops[o].unit0 + __ldg(ops[o].a.cuts + (y / n * kCuts + y % n * kCuts / n));
}

// dens of every operator from its column of P (blockIdx.y = operator), and the
// partition (found anew for every piece of a split block, six 64-bit divisions
// a time, it took 10 us of a batch of one and 40 of eight operators of six tiles)
__global__ void batch_prep_kernel(const BatchOp *__restrict__ ops, int nops, int64_t units, int nctas, BatchVec v)
{
    if (blockIdx.x == gridDim.x - 1 && blockIdx.y == 0)
        for (int c = threadIdx.x; c <= nctas; c += blockDim.x)
            v.begins[c] = c == nctas ? units : batch_begin(ops, nops, nctas, c);
    const BatchOp &o = ops[blockIdx.y];
    const double *pr = v.p_re + (int64_t)o.col * v.stride, *pi = v.p_im + (int64_t)o.col * v.stride;
    if (blockIdx.x == 0)
        for (int64_t b = threadIdx.x; b < o.ntiles; b += blockDim.x) o.a.done[b] = 0;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < o.a.npad;
         s += (int64_t)gridDim.x * blockDim.x) {
        const int c = o.a.perm[s];
        const double ws = (c >= 0) ? o.a.tpos[s].w * o.scale : 0.0;
        store_dens(o.a.dens, s, 0, c >= 0 ? (float)(ws * pr[c]) : 0.f, c >= 0 ? (float)(ws * pi[c]) : 0.f);
    }
}

__device__ __forceinline__ int batch_op_of_unit(const BatchOp *ops, int nops, int64_t u, int from)
{
    int o = from;
    while (o + 1 < nops && u >= ops[o + 1].unit0) o++;
    return o;
}

// cost0 and cost of the described operators (one thread)
__global__ void batch_cost_kernel(BatchOp *ops, int nops)
{
    int64_t c = 0;
    for (int o = 0; o < nops; o++) {
        ops[o].cost0 = c;
        ops[o].cost = ops[o].rows[ops[o].ntiles];
        c += ops[o].cost;
    }
}

__device__ __forceinline__ void batch_write(const Args32 &a, int64_t s, double ar, double ai, const double *p_re,
                                            const double *p_im, double *q_re, double *q_im)
{
    const int c = a.perm[s];
    if (c < 0) return;
    if (!isfinite(ar) || !isfinite(ai)) atomicOr(a.err, DEV_ERR_NONFINITE);
    q_re[c] = ar + 0.5 * p_re[c];
    q_im[c] = ai + 0.5 * p_im[c];
}

// The units of one segment (one target block of one operator) for the
// batched sweep: the same loops as sweep32_kernel with SWEEP_A.
template <int MODE, bool DIR, int NT, int TG>
__device__ __forceinline__ bool batch_tiles(const Args32 &a, const BatchOp *ops, int nops, int o, int64_t &u,
                                            int64_t u0, int64_t seg_end, int64_t u_end, unsigned &it, int64_t blk,
                                            int64_t slot0, const Targets<TG> &t, Sums<TG> &sum,
                                            float (*stage)[kStage<SWEEP_A>], uint64_t *bar)
{
    const uint32_t *mrow = a.nearmask + blk * a.mwords;
    const int shift = a.sub >> 1;  // log2 of 1, 2 or 4
    for (; u < seg_end; it++) {
        const int buf = (int)(it & 1);
        const int64_t tile = (u - u0) >> shift;
        const int q0 = (int)(u - u0) & (a.sub - 1), q1 = (int)min((int64_t)a.sub, q0 + seg_end - u);
        u += q1 - q0;
        if (threadIdx.x == 0 && u < u_end) {  // the next tile: of this block, else the first of the next one
            const bool same = tile + 1 < ops[o].ntiles;
            const int o2 = same ? o : batch_op_of_unit(ops, nops, u, o);
            issue_tile<SWEEP_A>(same ? a : ops[o2].a, same ? tile + 1 : 0, stage[buf ^ 1], &bar[buf ^ 1]);
        }
        const bool near = (__ldg(mrow + (tile >> 5)) >> (tile & 31)) & 1u;
        float3 rel[TG];
        Turn turn[TG];
        const bool centred = tile_offsets<MODE, TG>(a, tile, t, rel, turn);
        const bool ok = mbar_wait_bounded(&bar[buf], (it >> 1) & 1, g_data_wait_limit);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                atomicOr(a.err, DEV_ERR_WAIT);
                mbar_drain(&bar[buf], (it >> 1) & 1, &bar[buf ^ 1], ((it + 1) >> 1) & 1, u < u_end);
            }
            return false;
        }
        tile_pairs<MODE, DIR, NT, TG>(a, stage[buf], tile, q0, q1, near, rel, turn, centred, t, slot0, sum);
        __syncthreads();
    }
    return true;
}

// Q[r] = A_r P[r] for every operator r of a batch in one persistent launch:
// the stream-K partition of sweep32_kernel over the concatenated units, so
// operators of different sizes share the GPU without a tail per operator.
template <int NT, int TG, int MINB>
__global__ void __launch_bounds__(NT, MINB) sweep32_batch_kernel(const BatchOp *__restrict__ ops, int nops,
                                                                 int nctas, double4_32a *partial, BatchVec v)
{
    constexpr int SLOTS = NT * TG;
    __shared__ alignas(128) float stage[2][kStage<SWEEP_A>];
    __shared__ alignas(8) uint64_t bar[2];
    auto begin = [&](int c) { return __ldg(v.begins + c); };
    const int64_t u_begin = begin(blockIdx.x), u_end = begin(blockIdx.x + 1);
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    __syncthreads();
    if (u_begin >= u_end) return;
    int o = batch_op_of_unit(ops, nops, u_begin, 0);
    if (threadIdx.x == 0)
        issue_tile<SWEEP_A>(ops[o].a, (u_begin - ops[o].unit0) / ops[o].a.sub % ops[o].ntiles, stage[0], &bar[0]);
    int seg = 0;
    unsigned it = 0;
    for (int64_t u = u_begin; u < u_end;) {
        o = batch_op_of_unit(ops, nops, u, o);
        const Args32 a = ops[o].a;
        const int64_t ntiles = ops[o].ntiles, unit0 = ops[o].unit0, bu = ntiles * a.sub;
        const int64_t blk = (u - unit0) / bu, u0 = unit0 + blk * bu, seg_begin = u;
        const int64_t seg_end = (u_end < u0 + bu) ? u_end : u0 + bu;
        const bool whole = seg_end - seg_begin == bu;
        const int64_t slot0 = blk * SLOTS + threadIdx.x;
        Targets<TG> t;
        Sums<TG> sum;
        load_targets<NT, TG>(a, slot0, t, sum);
        auto walk = [&](auto mode, auto dir) {
            return batch_tiles<decltype(mode)::value, decltype(dir)::value, NT, TG>(
                a, ops, nops, o, u, u0, seg_end, u_end, it, blk, slot0, t, sum, stage, bar);
        };
        using Scaled = std::integral_constant<int, SWEEP_A | SWEEP_SCALED>;
        using Plain = std::integral_constant<int, SWEEP_A>;
        const bool ok = a.scaled ? (ops[o].dir ? walk(Scaled{}, std::true_type{}) : walk(Scaled{}, std::false_type{}))
                                 : (ops[o].dir ? walk(Plain{}, std::true_type{}) : walk(Plain{}, std::false_type{}));
        if (!ok) return;
        const int64_t off = (int64_t)ops[o].col * v.stride;
        const double *pr = v.p_re + off, *pi = v.p_im + off;
        double *qr = v.q_re + off, *qi = v.q_im + off;
#pragma unroll
        for (int g = 0; g < TG; g++) {
            const double ar = (double)sum.hAr[g] + (double)sum.lAr[g], ai = (double)sum.hAi[g] + (double)sum.lAi[g];
            if (whole)
                batch_write(a, slot0 + (int64_t)g * NT, ar, ai, pr, pi, qr, qi);
            else
                partial[((int64_t)blockIdx.x * 2 + seg) * SLOTS + threadIdx.x + g * NT] =
                    make_double4_32a(ar, ai, 0.0, 0.0);
        }
        if (!whole)
            finish_block<SLOTS>(a.done + blk, (unsigned)(seg_end - seg_begin), (unsigned)bu, u0, nctas, partial, begin,
                                [&](int k, double ar, double ai, double, double) {
                                    batch_write(a, blk * SLOTS + k, ar, ai, pr, pi, qr, qi);
                                });
        seg = 1;
    }
}

template <int NT, int TG, int MINB>
int64_t batch_resident_ctas()
{
    static int64_t cached = 0;
    if (cached == 0) {
        int dev = 0, sms = 152, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sweep32_batch_kernel<NT, TG, MINB>, NT, 0) !=
                cudaSuccess ||
            per < 1) {
            cudaGetLastError();
            per = MINB;
        }
        cached = (int64_t)per * sms;
    }
    return cached;
}

template <int NT, int TG, int MINB>
int launch_batch(const BatchOp *ops_dev, int nops, int64_t units, double4_32a *partial, size_t partial_bytes,
                 BatchVec v, int64_t max_npad, cudaStream_t s, cudaEvent_t ev0)
{
    constexpr int SLOTS = NT * TG;
    constexpr size_t piece = 2 * SLOTS * sizeof(double4_32a);
    int64_t p = batch_resident_ctas<NT, TG, MINB>();
    if (p > units) p = units;
    if (p * (piece + sizeof(int64_t)) + sizeof(int64_t) > partial_bytes)
        p = partial_bytes / (piece + sizeof(int64_t)) - 1;
    if (p < 1) {
        set_error("batched FP32 sweep: partial buffer too small");
        return HZ_ERR_STATE;
    }
    v.begins = reinterpret_cast<int64_t *>(partial + p * 2 * SLOTS);
    long long bx = (max_npad + 255) / 256;
    if (bx > 256) bx = 256;
    batch_prep_kernel<<<dim3((unsigned)bx, (unsigned)nops), 256, 0, s>>>(ops_dev, nops, units, (int)p, v);
    HZ_CHECK_LAUNCH();
    if (ev0) HZ_CHECK_CUDA(record_timing_event(ev0, s));
    sweep32_batch_kernel<NT, TG, MINB><<<(unsigned)p, NT, 0, s>>>(ops_dev, nops, (int)p, partial, v);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

// Resident CTAs of one sweep instantiation on this device (cached).
template <int MODE, bool DIR, int NT, int TG, int MINB>
int64_t resident_ctas()
{
    static int64_t cached = 0;
    if (cached == 0) {
        int dev = 0, sms = 152, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sweep32_kernel<MODE, DIR, NT, TG, MINB>, NT, 0) !=
                cudaSuccess ||
            per < 1) {
            cudaGetLastError();
            per = MINB;
        }
        cached = (int64_t)per * sms;
    }
    return cached;
}

// persistent: one CTA per resident slot (stream-K); otherwise one CTA per
// target block (the partition then never splits a block).
template <int MODE, bool DIR, int NT, int TG, int MINB>
int launch_streamk(Args32 a, bool persistent, size_t partial_bytes, cudaStream_t s)
{
    constexpr int SLOTS = NT * TG;
    const int64_t blocks = a.npad / SLOTS;
    int64_t p = blocks;
    if (persistent) {
        const int64_t units = blocks * (a.npad / kTile32) * a.sub;
        p = resident_ctas<MODE, DIR, NT, TG, MINB>();
        if (p > units) p = units;
        if ((size_t)p * 2 * SLOTS * sizeof(double4_32a) > partial_bytes)
            p = partial_bytes / (2 * SLOTS * sizeof(double4_32a));
    } else {
        a.cuts = nullptr;
    }
    if (p < 1) {
        set_error("FP32 sweep: stream-K partial buffer too small");
        return HZ_ERR_STATE;
    }
    a.nctas = (int)p;
    sweep32_kernel<MODE, DIR, NT, TG, MINB><<<(unsigned)p, NT, 0, s>>>(a);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

// Compiled variants: (block size, targets per thread, minimum resident
// blocks) x (persistent stream-K grid, or one CTA per target block).  Every
// shape covers the 256 slots of one target tile.  Below 24 tiles the persistent
// variants all run the first shape: a CTA has one or two units of 64 sources
// there, and two targets a thread or 80 registers only make it longer (n = 2,938:
// 39 us, the others 48 to 75).
constexpr int kShapes = 4;
template <int MODE, bool DIR>
int launch_cfg(int cfg, const Args32 &a, size_t pb, cudaStream_t s)
{
    const bool persistent = cfg < kShapes;
    const int shape = a.sub == 4 && persistent ? 0 : cfg % kShapes;
    switch (shape) {
    case 1: return launch_streamk<MODE, DIR, 128, 2, 4>(a, persistent, pb, s);
    case 2: return launch_streamk<MODE, DIR, 256, 1, 3>(a, persistent, pb, s);
    case 3: return launch_streamk<MODE, DIR, 128, 2, 3>(a, persistent, pb, s);
    default: return launch_streamk<MODE, DIR, 256, 1, 2>(a, persistent, pb, s);
    }
}

template <int MODE>
int launch32(int cfg, const Args32 &a, bool dir, size_t pb, cudaStream_t s)
{
    return dir ? launch_cfg<MODE, true>(cfg, a, pb, s) : launch_cfg<MODE, false>(cfg, a, pb, s);
}

}  // namespace

// The constants of an operator's FP32 records: k, k/(2 pi) split into a head
// with 12 significant bits and an FP32 tail, (lambda tau)^2 and its tie band.
Const32 constants32(const SweepConst &c, double lambda)
{
    Const32 r;
    r.scaled = lambda != 1.0 || c.wave == 1.0;
    r.k = (float)c.wave;
    const double kc = c.wave / (2.0 * kPi);
    int e;
    frexp(kc, &e);
    const double q = ldexp(1.0, e - 12);
    const double head = nearbyint(kc / q) * q;
    r.kh = (float)head;
    r.kl = (float)(kc - head);
    const double t2 = (lambda * c.tau) * (lambda * c.tau);
    r.tau2 = (float)t2;
    r.guard_lo = (float)(t2 * (1.0 - 1e-4));
    r.guard_hi = (float)(t2 * (1.0 + 1e-4));
    return r;
}

// Below k = 2^-14 (and for k <= 0) the coordinates stay unscaled, so that k^2 on
// the densities costs no more than 2^-28 of the FP32 range; below k tau = 2^-40 as
// well, so that (k rho)^2 and its inverse stay inside it whatever the unit of
// length.
double lambda32(double wave, double tau) { return wave >= 1.0 / 16384 && wave * tau >= 0x1p-40 ? wave : 1.0; }

double sweep32_reg_scale(int interior, double lambda)
{
    return ((interior == 1) ? -1.0 : 1.0) * (4.0 * kPi) / (lambda * lambda);
}

int sweep32_num_configs() { return 2 * kShapes; }

namespace {
template <int MODE, bool DIR, int NT, int TG, int MINB>
size_t partial_need()
{
    return (size_t)resident_ctas<MODE, DIR, NT, TG, MINB>() * 2 * NT * TG * sizeof(double4_32a);
}
template <int MODE, bool DIR>
size_t partial_need_all()
{
    size_t m = 0;
    const size_t v[kShapes] = {partial_need<MODE, DIR, 256, 1, 2>(), partial_need<MODE, DIR, 128, 2, 4>(),
                               partial_need<MODE, DIR, 256, 1, 3>(), partial_need<MODE, DIR, 128, 2, 3>()};
    for (size_t x : v) m = x > m ? x : m;
    return m;
}
}  // namespace

size_t sweep32_partial_bytes()
{
    constexpr int S = SWEEP_SCALED;
    const size_t v[12] = {partial_need_all<SWEEP_A, false>(),        partial_need_all<SWEEP_A, true>(),
                          partial_need_all<SWEEP_AH, false>(),       partial_need_all<SWEEP_AH, true>(),
                          partial_need_all<SWEEP_PAIR, false>(),     partial_need_all<SWEEP_PAIR, true>(),
                          partial_need_all<SWEEP_A | S, false>(),    partial_need_all<SWEEP_A | S, true>(),
                          partial_need_all<SWEEP_AH | S, false>(),   partial_need_all<SWEEP_AH | S, true>(),
                          partial_need_all<SWEEP_PAIR | S, false>(), partial_need_all<SWEEP_PAIR | S, true>()};
    size_t m = 0;
    for (size_t x : v) m = x > m ? x : m;
    return m;
}

static void set_constants(const SweepConst &c, double lambda, Args32 &a)
{
    const Const32 k = constants32(c, lambda);
    a.scaled = k.scaled;
    a.wave = {k.k, k.kh, k.kl};
    a.tau = c.tau;
    a.tau2 = k.tau2;
    a.guard_lo = k.guard_lo;
    a.guard_hi = k.guard_hi;
}

size_t cuts32_bytes(int64_t ntiles)
{
    return (size_t)(kCuts + 1 + ntiles + 1) * sizeof(int64_t) + (size_t)ntiles * sizeof(unsigned);
}

int build_cuts32(Rec32 &r, void *mem, cudaStream_t s)
{
    const int64_t ntiles = r.npad / kTile32;
    r.cuts = static_cast<int64_t *>(mem);
    r.rows = r.cuts + kCuts + 1;
    r.done = reinterpret_cast<unsigned *>(r.rows + ntiles + 1);
    row_cost_kernel<<<(unsigned)((ntiles + 7) / 8), 256, 0, s>>>(ntiles, r.mwords, r.nearmask, r.rows);
    HZ_CHECK_LAUNCH();
    row_scan_kernel<<<1, 1024, 0, s>>>(ntiles, r.rows);
    HZ_CHECK_LAUNCH();
    cuts_kernel<<<kCuts / 8 + 1, 256, 0, s>>>(ntiles, r.mwords, sub_of(ntiles), r.nearmask, r.rows,
                                                    r.cuts);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

// ---------------------------------------------------------------- batches
size_t batch32_desc_bytes(int R) { return (size_t)R * sizeof(BatchOp); }

int batch32_describe(const Batch32Item *items, int R, int cfg, void *desc_dev, int64_t &units, cudaStream_t s,
                     const int *cols)
{
    (void)cfg;
    std::vector<BatchOp> h(R);
    units = 0;
    for (int r = 0; r < R; r++) {
        const int col = cols ? cols[r] : r;
        const Batch32Item &it = items[col];
        BatchOp &b = h[r];
        memset(&b, 0, sizeof(b));
        b.col = col;
        Args32 &a = b.a;
        a.n = it.c.n;
        a.npad = it.r.npad;
        a.mwords = it.r.mwords;
        set_constants(it.c, it.r.lambda, a);
        a.pos = it.r.pos;
        a.soa = it.r.soa;
        a.nrm = it.r.nrm;
        a.dens = it.dens;
        a.thi = it.r.thi;
        a.tlo = it.r.tlo;
        a.ohi = it.r.ohi;
        a.olo = it.r.olo;
        a.nearmask = it.r.nearmask;
        a.tpos = it.r.tpos;
        a.perm = it.r.perm;
        a.pos64 = it.pos64;
        a.err = it.c.err;
        if (it.r.npad % kTile32 != 0 || it.r.npad == 0 || !it.r.cuts) {
            set_error("batched FP32 sweep: operator %d has %lld slots", col, (long long)it.r.npad);
            return HZ_ERR_STATE;
        }
        b.ntiles = it.r.npad / kTile32;
        b.unit0 = units;
        b.rows = it.r.rows;
        a.cuts = it.r.cuts;
        a.done = it.r.done;
        b.dir = it.c.dirichlet != 0;
        b.scale = 1.0 / sweep32_reg_scale(it.c.interior, it.r.lambda);
        a.sub = sub_of(b.ntiles);
        units += b.ntiles * b.ntiles * a.sub;
    }
    HZ_CHECK_CUDA(cudaMemcpyAsync(desc_dev, h.data(), R * sizeof(BatchOp), cudaMemcpyHostToDevice, s));
    if (R > 0) {
        batch_cost_kernel<<<1, 1, 0, s>>>(static_cast<BatchOp *>(desc_dev), R);
        HZ_CHECK_LAUNCH();
    }
    HZ_CHECK_CUDA(cudaStreamSynchronize(s));
    return HZ_OK;
}

size_t batch32_partial_bytes()
{
    const int64_t v[kShapes] = {batch_resident_ctas<256, 1, 2>(), batch_resident_ctas<128, 2, 4>(),
                                batch_resident_ctas<256, 1, 3>(), batch_resident_ctas<128, 2, 3>()};
    int64_t m = 0;
    for (int64_t x : v) m = x > m ? x : m;
    // the pieces of split blocks, and the partition
    return (size_t)m * (2 * 256 * sizeof(double4_32a) + sizeof(int64_t)) + sizeof(int64_t);
}

int sweep_f32_batch(int cfg, const void *desc_dev, int R, int ncols, int64_t units, double4_32a *partial, size_t partial_bytes, const double *p_re, const double *p_im,
                    double *q_re, double *q_im, int64_t stride, int64_t max_npad, cudaStream_t s, cudaEvent_t ev0,
                    cudaEvent_t ev1)
{
    // padded tails of the columns stay zero
    HZ_CHECK_CUDA(cudaMemsetAsync(q_re, 0, (size_t)ncols * stride * sizeof(double), s));
    HZ_CHECK_CUDA(cudaMemsetAsync(q_im, 0, (size_t)ncols * stride * sizeof(double), s));
    if (R <= 0 || units <= 0) return HZ_OK;
    const BatchOp *ops = static_cast<const BatchOp *>(desc_dev);
    BatchVec v{p_re, p_im, q_re, q_im, stride, nullptr};
    const size_t pb = partial_bytes;
    switch (cfg % kShapes) {
    case 1: HZ_TRY((launch_batch<128, 2, 4>(ops, R, units, partial, pb, v, max_npad, s, ev0))); break;
    case 2: HZ_TRY((launch_batch<256, 1, 3>(ops, R, units, partial, pb, v, max_npad, s, ev0))); break;
    case 3: HZ_TRY((launch_batch<128, 2, 3>(ops, R, units, partial, pb, v, max_npad, s, ev0))); break;
    default: HZ_TRY((launch_batch<256, 1, 2>(ops, R, units, partial, pb, v, max_npad, s, ev0))); break;
    }
    if (ev1) HZ_CHECK_CUDA(record_timing_event(ev1, s));
    return HZ_OK;
}

int sweep_f32(const SweepConst &c, const Rec32 &r, const double4_32a *pos64, int mode, const double *p_re,
              const double *p_im, const double *pt_re, const double *pt_im, double *q_re, double *q_im,
              double *qt_re, double *qt_im, float *dens, cudaStream_t s, cudaEvent_t ev0,
              cudaEvent_t ev1, int cfg)
{
    if (c.n <= 0) return HZ_OK;
    const bool useA = (mode & SWEEP_A) != 0, useH = (mode & SWEEP_AH) != 0;
    const double scale = 1.0 / sweep32_reg_scale(c.interior, r.lambda);
    {
        int dev = 0, sms = 152;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        long long b = (r.npad + 255) / 256;
        if (b > sms * 8) b = sms * 8;
        prep32_kernel<<<(unsigned)b, 256, 0, s>>>(r.npad, r.perm, r.tpos, useA ? p_re : nullptr,
                                                  useA ? p_im : nullptr, useH ? pt_re : nullptr,
                                                  useH ? pt_im : nullptr, scale, dens, r.done);
        HZ_CHECK_LAUNCH();
    }
    Args32 a;
    a.n = c.n;
    a.npad = r.npad;
    set_constants(c, r.lambda, a);
    a.mwords = r.mwords;
    a.thi = r.thi;
    a.tlo = r.tlo;
    a.ohi = r.ohi;
    a.olo = r.olo;
    a.nearmask = r.nearmask;
    a.pos = r.pos;
    a.soa = r.soa;
    a.nrm = r.nrm;
    a.dens = dens;
    a.tpos = r.tpos;
    a.perm = r.perm;
    a.pos64 = pos64;
    a.p_re = p_re; a.p_im = p_im; a.pt_re = pt_re; a.pt_im = pt_im;
    a.q_re = q_re; a.q_im = q_im; a.qt_re = qt_re; a.qt_im = qt_im;
    a.err = c.err;
    if (ev0) HZ_CHECK_CUDA(record_timing_event(ev0, s));
    a.partial = r.partial;
    a.cuts = r.cuts;
    a.done = r.done;
    a.sub = sub_of(r.npad / kTile32);
    const bool dir = c.dirichlet != 0;
    constexpr int S = SWEEP_SCALED;
    if (a.scaled) {
        if (mode == SWEEP_PAIR) HZ_TRY(launch32<SWEEP_PAIR | S>(cfg, a, dir, r.partial_bytes, s));
        else if (mode == SWEEP_A) HZ_TRY(launch32<SWEEP_A | S>(cfg, a, dir, r.partial_bytes, s));
        else HZ_TRY(launch32<SWEEP_AH | S>(cfg, a, dir, r.partial_bytes, s));
    } else {
        if (mode == SWEEP_PAIR) HZ_TRY(launch32<SWEEP_PAIR>(cfg, a, dir, r.partial_bytes, s));
        else if (mode == SWEEP_A) HZ_TRY(launch32<SWEEP_A>(cfg, a, dir, r.partial_bytes, s));
        else HZ_TRY(launch32<SWEEP_AH>(cfg, a, dir, r.partial_bytes, s));
    }
    if (ev1) HZ_CHECK_CUDA(record_timing_event(ev1, s));
    return HZ_OK;
}

HZ_DEFINE_WAIT_LIMIT_SETTER(set_wait_limit_f32)

}  // namespace hz
