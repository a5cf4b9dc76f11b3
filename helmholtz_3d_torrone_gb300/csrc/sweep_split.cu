// sweep_split.cu -- the FP64 products q = A p, qt = A^H pt (sweep_f64.cu) with
// every pair evaluated as pairs of FP32 numbers (pair_split.cuh).
//
// Bound by issue slots: 232 instructions a pair (A p; 326 for the fused pass) on
// 77 % of the cycles, the FMA pipe 63 % busy (n = 145,272: 159 ms, 132 Gpair/s),
// against the 38.5 FP64 instructions (about 2,600 FP32 slots) of sweep64_kernel.
//
// One thread owns one target of the blocked sweep order (Rec32::perm); a CTA
// of 256 threads walks a contiguous range of (target tile, half or quarter
// source tile) units, as sweep32_kernel does, so the chip is full from a few
// thousand points on.  Units of 128 or 64 sources (96 bytes of fixed record
// and 16 of density each) come by TMA bulk copies, double-buffered on mbarriers with
// bounded waits; the cosine table takes 64 KB of shared memory, which leaves
// room for two CTAs an SM.  Per target and source tile about 50 FP64
// instructions set up the offsets and the phase of the tile's origin; they and
// the FP64 sums (the 48-bit sums of 16 sources are added in FP64) run on the
// otherwise idle FP64 pipe.
#include "hz_internal.cuh"
#include "bulk_copy.cuh"
#include "pair_split.cuh"

namespace hz {
namespace {

constexpr double kPiS = 3.14159265358979323846264338328;
constexpr int kHalf = 128;       // sources per staged half tile
constexpr int kRun = 16;         // sources per 48-bit sum
constexpr int kRecs = 6;         // float4 of fixed record per source
constexpr int kExpBlocks = 152;  // blocks of the density maximum

// MODE bit beside SWEEP_A: the k-derivative of A's entries.
constexpr int SPLIT_DK = 8;

struct ArgsSplit {
    int64_t npad, units;
    int part;                   // sources per unit: 128 or 64 (launch_split)
    int64_t nctas;
    float tau2, ktau;
    double wave, tau;
    const float4 *rec;          // [kRecs][npad]
    const float4 *densA, *densH;
    const double4_32a *tile;    // scaled origin, scaled radius (at least k tau)
    const float2 *table;
    const double4_32a *tpos;    // unscaled position and weight per slot
    const double4_32a *nrm;     // tube order: (n, w)
    const int *perm;
    const int *expo;            // exponents of the density scales (A, A^H)
    const double *p_re, *p_im, *pt_re, *pt_im;
    double *q_re, *q_im, *qt_re, *qt_im;
    double4_32a *partial;       // [nctas][2][256]
    const double *dreg;         // SPLIT_DK: d reg / dk in tube order, times dreg_scale
    double dreg_scale;
    unsigned *err;
};

// float 2^e, -126 <= e <= 127
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }
__device__ __forceinline__ double pow2d(int e) { return __hiloint2double((e + 1023) << 20, 0); }
// smallest e with v < 2^e
__device__ __forceinline__ int exponent_above(float v) { return ((__float_as_int(v) >> 23) & 255) - 126; }

__global__ void split_table_kernel(float2 *tab)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < kSplitTable; j += gridDim.x * blockDim.x) {
        const double c = cospi((double)j / (kSplitTable / 2));
        const double h = rint(c * 8388608.0) / 8388608.0;  // the head on the grid 2^-23
        tab[j] = make_float2((float)h, (float)(c - h));
    }
}

__global__ void split_tile_kernel(int64_t ntiles, const double4_32a *__restrict__ origin, double wave, double ktau,
                                  double4_32a *__restrict__ tile)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= ntiles) return;
    const double4_32a o = origin[t];
    tile[t] = make_double4_32a(wave * o.x, wave * o.y, wave * o.z, fmax(wave * o.w * (1.0 + 1e-9), ktau));
}

__device__ __forceinline__ void split_coord(double v, double unit, double inv_unit, int &h, float &f, float &l)
{
    const double r = rint(v * inv_unit);
    h = (int)r;
    f = (float)v;
    l = (float)fma(-r, unit, v);
}

// Fixed source records (see the packing in load_source); reg2 = 2 reg / scale.
__global__ void __launch_bounds__(256) split_records_kernel(int64_t npad, const int *__restrict__ perm,
                                                            const double4_32a *__restrict__ tpos,
                                                            const double4_32a *__restrict__ pos,
                                                            const double4_32a *__restrict__ nrm,
                                                            const double4_32a *__restrict__ tile, double wave,
                                                            double reg_scale, float4 *__restrict__ rec)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= npad) return;
    const int c = perm[i];
    const double4_32a o = tile[i / kTile32];
    const int eS = exponent_above((float)(o.w * (1.0 + 1e-6)));
    const double uS = pow2d(eS - 30), iS = pow2d(30 - eS);
    double s[3] = {0, 0, 0}, n[3] = {0, 0, 0}, reg = 0;
    if (c >= 0) {
        const double4_32a x = tpos[i], m = nrm[c];
        s[0] = wave * x.x - o.x;
        s[1] = wave * x.y - o.y;
        s[2] = wave * x.z - o.z;
        n[0] = m.x;
        n[1] = m.y;
        n[2] = m.z;
        reg = pos[c].w * reg_scale;
    }
    int sh[3], nh[3];
    float sf[3], sl[3], nf[3], nl[3];
    for (int a = 0; a < 3; a++) {
        split_coord(s[a], uS, iS, sh[a], sf[a], sl[a]);
        split_coord(n[a], pow2d(-30), pow2d(30), nh[a], nf[a], nl[a]);
    }
    const double s2 = fma(s[2], s[2], fma(s[1], s[1], s[0] * s[0]));
    const double sn = fma(s[2], n[2], fma(s[1], n[1], s[0] * n[0]));
    const long long S2 = __double2ll_rn(s2 * iS * iS), SN = __double2ll_rn(2.0 * sn * iS * pow2d(30));
    const FF rg = ff_of_double(reg);
    auto f = [](int v) { return __int_as_float(v); };
    rec[0 * npad + i] = make_float4(f(sh[0]), f(sh[1]), f(sh[2]), f(nh[0]));
    rec[1 * npad + i] = make_float4(f(nh[1]), f(nh[2]), f((int)S2), f((int)(S2 >> 32)));
    rec[2 * npad + i] = make_float4(f((int)SN), f((int)(SN >> 32)), sf[0], sf[1]);
    rec[3 * npad + i] = make_float4(sf[2], sl[0], sl[1], sl[2]);
    rec[4 * npad + i] = make_float4(nf[0], nf[1], nf[2], nl[0]);
    rec[5 * npad + i] = make_float4(nl[1], nl[2], rg.h, rg.l);
}

// Largest exponent field of |w p| and |pt| per block (high words of doubles
// order like their values).
__global__ void __launch_bounds__(256) split_max_kernel(int64_t n, const double4_32a *__restrict__ nrm,
                                                        const double *__restrict__ p_re,
                                                        const double *__restrict__ p_im,
                                                        const double *__restrict__ pt_re,
                                                        const double *__restrict__ pt_im, int *__restrict__ part)
{
    int a = 0, b = 0;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
        if (p_re) {
            const double w = nrm[s].w;
            a = max(a, max(__double2hiint(w * p_re[s]) & 0x7fffffff, __double2hiint(w * p_im[s]) & 0x7fffffff));
        }
        if (pt_re) b = max(b, max(__double2hiint(pt_re[s]) & 0x7fffffff, __double2hiint(pt_im[s]) & 0x7fffffff));
    }
    a = __reduce_max_sync(0xffffffffu, a);
    b = __reduce_max_sync(0xffffffffu, b);
    __shared__ int sh[2][8];
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = a;
        sh[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        int v = 0;
        for (int w = 0; w < 8; w++) v = max(v, sh[threadIdx.x][w]);
        part[threadIdx.x * kExpBlocks + blockIdx.x] = v;
    }
}

// Densities scaled to at most 1 and split: -k^2 sg/(8 pi) w p for A (the
// entries carry -2 (x_t - x_s).n), +k^2 sg/(8 pi) pt for A^H.  The exponents
// taken out, the densities' and k^2's (k^2 sg/(8 pi) = scale 2^scale_exp), go to
// expo: what is left lies in the FP32 range whatever the unit of length.
__global__ void __launch_bounds__(256) split_dens_kernel(int64_t npad, const int *__restrict__ perm,
                                                         const double4_32a *__restrict__ tpos,
                                                         const double *__restrict__ p_re,
                                                         const double *__restrict__ p_im,
                                                         const double *__restrict__ pt_re,
                                                         const double *__restrict__ pt_im, double scale,
                                                         int scale_exp, const int *__restrict__ part,
                                                         int *__restrict__ expo, float4 *__restrict__ densA,
                                                         float4 *__restrict__ densH)
{
    __shared__ int ex[2];
    if (threadIdx.x < 64) {
        const int m = threadIdx.x >> 5;
        int v = 0;
        for (int b = threadIdx.x & 31; b < kExpBlocks; b += 32) v = max(v, part[m * kExpBlocks + b]);
        v = __reduce_max_sync(0xffffffffu, v);
        // values below 2^(e + 1); clamped so that 2^e and 2^-e are normal
        int e = (v >> 20) - 1022;
        e = max(-1000, min(1000, e));
        if ((threadIdx.x & 31) == 0) {
            ex[m] = e;
            if (blockIdx.x == 0) expo[m] = e + scale_exp;
        }
    }
    __syncthreads();
    const double fa = pow2d(-ex[0]), fh = pow2d(-ex[1]);
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < npad; s += (int64_t)gridDim.x * blockDim.x) {
        const int c = perm[s];
        if (p_re) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c >= 0) {
                const double w = tpos[s].w;
                const FF r = ff_of_double(-scale * ((w * p_re[c]) * fa)), i = ff_of_double(-scale * ((w * p_im[c]) * fa));
                v = make_float4(r.h, i.h, r.l, i.l);
            }
            densA[s] = v;
        }
        if (pt_re) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c >= 0) {
                const FF r = ff_of_double(scale * (pt_re[c] * fh)), i = ff_of_double(scale * (pt_im[c] * fh));
                v = make_float4(r.h, i.h, r.l, i.l);
            }
            densH[s] = v;
        }
    }
}

// What a thread holds of its target for one source tile.
struct Offsets {
    int h[3];           // A / 2^(eL - 30)
    float f[3], l[3];   // A and its tail
    FF a2, rc;          // |a|^2 and |a| (far tiles)
    long long a2i;      // |a|^2 in the close tiles' unit
    long long an;       // A.n_t in the unit 2^(eL - 60)
};

struct TargetNormal {
    int h[3];
    float f[3], l[3];  // 2 n and twice its tail
};

// Uniform constants of one (target tile, source tile) pair.
struct TileUnits {
    int shS;             // eL - eS: from the sources' unit to the pair's
    int shT;             // eL - eS - 1 (at least 0)
    int x;               // close tiles: extra shift that keeps r^2 below 2^62
    float w32, w8;       // 2^32 and 2^8 units of W
    float r32, r8;       // the same after the extra shift
    float lo, hi;        // close tiles: r^2 in [lo, hi] is formed again from the FP64 coordinates
    float n32, n8;       // 2^32 and 2^8 units of A.n
};

// The entries of one pair: A's (ar, ai) and A^H's before conjugation (hr, hi).
template <int MODE, bool DIR, bool CLOSE>
__device__ __forceinline__ void split_entry(const ArgsSplit &a, const float4 (*st)[kHalf], int j, const float2 *tab,
                                            const Offsets &t, const TargetNormal &tn, FF treg, const TileUnits &u,
                                            int64_t tslot, int64_t sslot, FF &ar, FF &ai, FF &hr, FF &hi)
{
    constexpr bool A = (MODE & SWEEP_A) != 0, H = (MODE & SWEEP_AH) != 0;
    constexpr bool SRC = (A && DIR) || (H && !DIR);  // (x_t - x_s).n_s wanted
    constexpr bool TGT = (A && !DIR) || (H && DIR);  // (x_t - x_s).n_t wanted
    constexpr bool DK = (MODE & SPLIT_DK) != 0;      // the factor is e^{i theta} y alone
    const float4 r0 = st[0][j], r1 = st[1][j], r2_ = st[2][j], r3 = st[3][j];
    const int s0 = __float_as_int(r0.x), s1 = __float_as_int(r0.y), s2 = __float_as_int(r0.z);
    long long W = ((((long long)__float_as_int(r1.w) << 32) | (unsigned)__float_as_int(r1.z)) >> u.shS) + 128;
    W += (long long)t.h[0] * s0;
    W += (long long)t.h[1] * s1;
    W += (long long)t.h[2] * s2;
    float e = fmul(t.f[0], r3.y);
    e = ffma(t.f[1], r3.z, e);
    e = ffma(t.f[2], r3.w, e);
    e = ffma(t.l[0], r2_.z, e);
    e = ffma(t.l[1], r2_.w, e);
    e = ffma(t.l[2], r3.x, e);
    FF r2, w;
    bool far = true;
    if (CLOSE) {
        r2 = ff_of_int((W >> u.x) + t.a2i, u.r32, u.r8, e);
        far = r2.h > a.tau2;
        if (r2.h >= u.lo && r2.h <= u.hi) {
            // decided as the reference does: rho^2 without fused operations
            const double4_32a p = a.tpos[tslot], q = a.tpos[sslot];
            const double dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
            const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            far = __dsqrt_rn(d2) > a.tau;
            r2 = ff_of_double(a.wave * (a.wave * d2));
        }
    } else {
        w = ff_of_int(W, u.w32, u.w8, e);
        const FF q = fast_two_sum(t.a2.h, w.h);
        r2 = {q.h, fadd(q.l, fadd(t.a2.l, w.l))};
    }
    FF rho, y, th, c, s, ur, ui;
    split_root(r2, rho, y);
    th = CLOSE ? rho : split_phase_offset(w, rho, t.rc);
    split_sincos(th, tab, c, s);
    FF y2;
    if (DK) {
        ur = c;
        ui = s;
        y2 = y;
    } else {
        split_kernel(y, c, s, ur, ui);
        y2 = ff_mul(y, y);
    }
    FF vsr, vsi, vtr, vti;
    if (SRC) {
        const float4 r4 = st[4][j], r5 = st[5][j];
        long long N = ((((long long)__float_as_int(r2_.y) << 32) | (unsigned)__float_as_int(r2_.x)) >> u.shS) + 128;
        N += (long long)t.h[0] * __float_as_int(r0.w);
        N += (long long)t.h[1] * __float_as_int(r1.x);
        N += (long long)t.h[2] * __float_as_int(r1.y);
        float g = fmul(t.f[0], r4.w);
        g = ffma(t.f[1], r5.x, g);
        g = ffma(t.f[2], r5.y, g);
        g = ffma(t.l[0], r4.x, g);
        g = ffma(t.l[1], r4.y, g);
        g = ffma(t.l[2], r4.z, g);
        const FF f = ff_mul(y2, ff_of_int(N, u.n32, u.n8, g));
        vsr = ff_mul(ur, f);
        vsi = ff_mul(ui, f);
    }
    if (TGT) {
        long long D = (long long)tn.h[0] * s0;
        D += (long long)tn.h[1] * s1;
        D += (long long)tn.h[2] * s2;
        float g = fmul(tn.f[0], r3.y);
        g = ffma(tn.f[1], r3.z, g);
        g = ffma(tn.f[2], r3.w, g);
        g = ffma(tn.l[0], r2_.z, g);
        g = ffma(tn.l[1], r2_.w, g);
        g = ffma(tn.l[2], r3.x, g);
        const FF f = ff_mul(y2, ff_of_int(t.an + (D >> u.shT), u.n32, u.n8, g));
        vtr = ff_mul(ur, f);
        vti = ff_mul(ui, f);
    }
    ar = DIR ? vsr : vtr;
    ai = DIR ? vsi : vti;
    hr = DIR ? vtr : vsr;
    hi = DIR ? vti : vsi;
    if (CLOSE && !far) {
        if (DK) {
            const int q = a.perm[DIR ? sslot : tslot];
            ar = ai = {0.f, 0.f};
            if (q >= 0) ar = ff_of_double(a.dreg[q] * a.dreg_scale);
            return;
        }
        const float4 r5 = st[5][j];
        const FF srg = {r5.z, r5.w};
        ar = ff_neg(DIR ? srg : treg);
        hr = DIR ? treg : srg;
        ai = hi = {0.f, 0.f};
    }
}

template <int MODE, bool DIR, bool CLOSE>
__device__ __forceinline__ void split_pair(const ArgsSplit &a, const float4 (*st)[kHalf], int j, const float2 *tab,
                                           const Offsets &t, const TargetNormal &tn, FF treg, const TileUnits &u,
                                           int64_t tslot, int64_t sslot, FF (&accA)[2], FF (&accH)[2])
{
    constexpr bool A = (MODE & SWEEP_A) != 0, H = (MODE & SWEEP_AH) != 0;
    FF ar, ai, hr, hi;
    split_entry<MODE, DIR, CLOSE>(a, st, j, tab, t, tn, treg, u, tslot, sslot, ar, ai, hr, hi);
    if (A) {
        const float4 d = st[kRecs][j];
        const FF dr = {d.x, d.z}, di = {d.y, d.w};
        split_dot2<-1>(accA[0], ar, dr, ai, di);
        split_dot2<1>(accA[1], ar, di, ai, dr);
    }
    if (H) {
        const float4 d = st[kRecs + (A ? 1 : 0)][j];
        const FF dr = {d.x, d.z}, di = {d.y, d.w};
        split_dot2<1>(accH[0], hr, dr, hi, di);
        split_dot2<-1>(accH[1], hr, di, hi, dr);
    }
}

template <int MODE, bool DIR, bool CLOSE>
__device__ __forceinline__ void split_part(const ArgsSplit &a, const float4 (*st)[kHalf], const float2 *tab,
                                           const Offsets &t, const TargetNormal &tn, FF treg, const TileUnits &u,
                                           int64_t tslot, int64_t sslot0, double (&dA)[2], double (&dH)[2])
{
#pragma unroll 1
    for (int j0 = 0; j0 < a.part; j0 += kRun) {
        FF accA[2] = {{0.f, 0.f}, {0.f, 0.f}}, accH[2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 1
        for (int j = j0; j < j0 + kRun; j++)
            split_pair<MODE, DIR, CLOSE>(a, st, j, tab, t, tn, treg, u, tslot, sslot0 + j, accA, accH);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (MODE & SWEEP_A) dA[q] += (double)accA[q].h + (double)accA[q].l;
            if (MODE & SWEEP_AH) dH[q] += (double)accH[q].h + (double)accH[q].l;
        }
    }
}

// e^{i x}, 0 <= x < 4000, from the split table
__device__ __forceinline__ void split_phase64(double x, const float2 *tab, double &cr, double &sr)
{
    const int m = __double2int_rn(x * (kSplitTable / (2.0 * kPiS)));
    double r = fma(-(double)m, 0.003067961575652589 / 4, x);  // the step to 31 bits, and the rest
    r = fma(-(double)m, 1.1869336926769907e-13 / 4, r);
    const float2 c = tab[m & (kSplitTable - 1)], s = tab[(m - kSplitTable / 4) & (kSplitTable - 1)];
    const double tc = (double)c.x + (double)c.y, ts = (double)s.x + (double)s.y;
    const double z = r * r, sn = fma(r * z, -1.0 / 6.0, r), cm = z * fma(z, -1.0 / 24.0, 0.5);
    cr = tc - fma(ts, sn, tc * cm);
    sr = ts + fma(tc, sn, -(ts * cm));
}

// Offsets of a thread's target (scaled position X, Y, Z in the tile with
// origin `to`) from source tile `tile`, the tile's units, and for a far tile
// the phase of its origin.
template <bool TGT>
__device__ __forceinline__ void set_tile(const ArgsSplit &a, int64_t tile, const double4_32a &to, double X, double Y,
                                         double Z, double nx, double ny, double nz, const float2 *tab, Offsets &t,
                                         TileUnits &un, bool &close, double &phr, double &phi)
{
    const float ox = (float)to.x, oy = (float)to.y, oz = (float)to.z, Rt = (float)to.w;
    const double4_32a o = a.tile[tile];
    const float Rs = (float)o.w;
    const float cx = ox - (float)o.x, cy = oy - (float)o.y, cz = oz - (float)o.z;
    const float ct = sqrtf(fmaf(cx, cx, fmaf(cy, cy, cz * cz)));
    close = ct - Rt < 2.5f * Rs + a.ktau + 1e-4f * (ct + Rt + fabsf(ox) + fabsf(oy) + fabsf(oz));
    const int eS = exponent_above((float)(o.w * (1.0 + 1e-6)));
    const int eL = max(eS + 1, exponent_above(2.0002f * (ct + Rt)));
    un.shS = eL - eS;
    un.shT = eL - eS - 1;
    un.x = max(0, eL - eS - 3);
    un.w32 = pow2f(eL + eS - 28);
    un.w8 = pow2f(eL + eS - 52);
    un.r32 = un.w32 * pow2f(un.x);
    un.r8 = un.w8 * pow2f(un.x);
    un.n32 = pow2f(eL - 28);
    un.n8 = pow2f(eL - 52);
    const double uL = pow2d(eL - 30), iL = pow2d(30 - eL);
    const double ax = -2.0 * (X - o.x), ay = -2.0 * (Y - o.y), az = -2.0 * (Z - o.z);
    const double A[3] = {ax, ay, az};
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double m = fma(A[i], iL, 6755399441055744.0);  // nearest integer in the low word
        t.h[i] = __double2loint(m);
        t.f[i] = (float)A[i];
        t.l[i] = (float)fma(-uL, m - 6755399441055744.0, A[i]);
    }
    const double a2 = 0.25 * fma(az, az, fma(ay, ay, ax * ax));
    if (close) {
        t.a2i = __double2ll_rn(a2 * pow2d(60 - eL - eS - un.x));
        // r^2 is off by less than 2^-52 of 2^(eL + eS + x) (typically a quarter of
        // that), whatever its size.  Below 2^-9 of that (rho below 1/8 to 1/16
        // of the tile's radius) it would be off by more than 2^-43 of itself and
        // is formed again, as it is next to tau^2: on the 64^3 sphere (tiles of
        // 10 h, tau = 2 h) a lane in 0.02 % of a warp's steps.  (From 2^-8 on,
        // 0.6 % of the steps: 3 to 9 % more time.)
        const float off = pow2f(eL + eS + un.x - 52);
        un.lo = a.tau2 - fmaxf(1e-6f * a.tau2, off);
        un.hi = fmaxf(a.tau2 + 1e-6f * a.tau2, pow2f(eL + eS + un.x - 9));
    } else {
        const double y0 = (double)rsqrt_seed((float)a2);
        const double e = fma(-(a2 * y0), y0, 1.0);
        const double y = fma(y0 * e, fma(e, 0.375, 0.5), y0);
        const double g = a2 * y;
        const double rc = fma(fma(-g, g, a2), 0.5 * y, g);
        t.a2 = ff_of_double(a2);
        t.rc = ff_of_double(rc);
        split_phase64(rc, tab, phr, phi);
    }
    if (TGT) t.an = __double2ll_rn(fma(az, nz, fma(ay, ny, ax * nx)) * pow2d(60 - eL)) + 128;
}

template <bool TGT>
__device__ __forceinline__ void load_target(const ArgsSplit &a, int64_t slot, double &X, double &Y, double &Z,
                                            double &nx, double &ny, double &nz, FF &treg, TargetNormal &tn)
{
    const double4_32a tp = a.tpos[slot];
    X = a.wave * tp.x;
    Y = a.wave * tp.y;
    Z = a.wave * tp.z;
    const float4 r5 = a.rec[5 * a.npad + slot];
    treg = {r5.z, r5.w};
    nx = ny = nz = 0.0;
    if (!TGT) return;
    const int c = a.perm[slot];
    if (c >= 0) {
        const double4_32a m = a.nrm[c];
        nx = m.x;
        ny = m.y;
        nz = m.z;
    }
    const float4 r0 = a.rec[slot], r1 = a.rec[a.npad + slot], r4 = a.rec[4 * a.npad + slot];
    tn.h[0] = __float_as_int(r0.w);
    tn.h[1] = __float_as_int(r1.x);
    tn.h[2] = __float_as_int(r1.y);
    tn.f[0] = 2.f * r4.x;
    tn.f[1] = 2.f * r4.y;
    tn.f[2] = 2.f * r4.z;
    tn.l[0] = 2.f * r4.w;
    tn.l[1] = 2.f * r5.x;
    tn.l[2] = 2.f * r5.y;
}

template <int MODE>
__device__ __forceinline__ void split_write(const ArgsSplit &a, int64_t s, double ar, double ai, double hr, double hi)
{
    const int c = a.perm[s];
    if (c < 0) return;
    if (MODE & SWEEP_A) {
        const double r = ldexp(ar, a.expo[0]), i = ldexp(ai, a.expo[0]);
        if (!(MODE & SPLIT_DK) && (!isfinite(r) || !isfinite(i))) atomicOr(a.err, DEV_ERR_NONFINITE);
        a.q_re[c] = (MODE & SPLIT_DK) ? r : r + 0.5 * a.p_re[c];
        a.q_im[c] = (MODE & SPLIT_DK) ? i : i + 0.5 * a.p_im[c];
    }
    if (MODE & SWEEP_AH) {
        const double w = a.tpos[s].w, r = ldexp(w * hr, a.expo[1]), i = ldexp(w * hi, a.expo[1]);
        if (!isfinite(r) || !isfinite(i)) atomicOr(a.err, DEV_ERR_NONFINITE);
        a.qt_re[c] = r + 0.5 * a.pt_re[c];
        a.qt_im[c] = i + 0.5 * a.pt_im[c];
    }
}

// float4 arrays of a staged half tile
template <int MODE>
constexpr int kSplitArrays = kRecs + (MODE == SWEEP_PAIR ? 2 : 1);

template <int MODE, bool DIR>
__global__ void __launch_bounds__(kTile32, 2) sweep_split_kernel(ArgsSplit a)
{
    constexpr int NA = kSplitArrays<MODE>;
    constexpr bool TGT = ((MODE & SWEEP_A) && !DIR) || ((MODE & SWEEP_AH) && DIR);
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ alignas(8) uint64_t bar[2];
    float2 *tab = reinterpret_cast<float2 *>(smem);
    float4(*stage)[kHalf] = reinterpret_cast<float4(*)[kHalf]>(smem + kSplitTable * sizeof(float2));
    const int64_t parts = a.npad / a.part;
    const int last = kTile32 / a.part - 1;  // parts of a tile less one: 1 or 3
    const int64_t u_begin = (int64_t)blockIdx.x * a.units / a.nctas;
    const int64_t u_end = ((int64_t)blockIdx.x + 1) * a.units / a.nctas;
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    for (int i = threadIdx.x; i < kSplitTable / 2; i += kTile32)
        reinterpret_cast<float4 *>(tab)[i] = __ldg(reinterpret_cast<const float4 *>(a.table) + i);
    __syncthreads();
    if (u_begin >= u_end) return;
    auto issue = [&](int64_t u, int buf) {
        const int64_t base = (u % parts) * a.part;
        const uint32_t bytes = a.part * (uint32_t)sizeof(float4);
        mbar_arrive_expect_tx(&bar[buf], NA * bytes);
#pragma unroll
        for (int r = 0; r < kRecs; r++) bulk_g2s(&stage[buf * NA + r][0], a.rec + r * a.npad + base, bytes, &bar[buf]);
        if (MODE & SWEEP_A) bulk_g2s(&stage[buf * NA + kRecs][0], a.densA + base, bytes, &bar[buf]);
        if (MODE & SWEEP_AH) bulk_g2s(&stage[buf * NA + NA - 1][0], a.densH + base, bytes, &bar[buf]);
    };
    if (threadIdx.x == 0) issue(u_begin, 0);
    int seg = 0;
    for (int64_t u = u_begin; u < u_end;) {
        const int64_t blk = u / parts;
        const int64_t seg_end = (u_end < (blk + 1) * parts) ? u_end : (blk + 1) * parts;
        const bool whole = (u == blk * parts) && (seg_end == (blk + 1) * parts);
        const int64_t slot = blk * kTile32 + threadIdx.x;
        const double4_32a to = a.tile[blk];
        double X, Y, Z, nx, ny, nz;
        FF treg;
        TargetNormal tn = {};
        load_target<TGT>(a, slot, X, Y, Z, nx, ny, nz, treg, tn);
        double q[4] = {0, 0, 0, 0};
        double dA[2] = {0, 0}, dH[2] = {0, 0};
        Offsets t = {};
        TileUnits un = {};
        bool close = false, fresh = true;
        double phr = 1.0, phi = 0.0;
        for (; u < seg_end; u++) {
            const int64_t it = u - u_begin;
            const int buf = (int)(it & 1);
            if (threadIdx.x == 0 && u + 1 < u_end) issue(u + 1, buf ^ 1);
            const int64_t part = u - blk * parts, tile = part >> (last == 1 ? 1 : 2);
            if (fresh || (part & last) == 0) {
                fresh = false;
                set_tile<TGT>(a, tile, to, X, Y, Z, nx, ny, nz, tab, t, un, close, phr, phi);
            }
            const bool ok = mbar_wait_bounded(&bar[buf], (uint32_t)((it >> 1) & 1), g_data_wait_limit);
            if (__syncthreads_or(!ok)) {
                if (threadIdx.x == 0) {
                    atomicOr(a.err, DEV_ERR_WAIT);
                    mbar_drain(&bar[buf], (uint32_t)((it >> 1) & 1), &bar[buf ^ 1], (uint32_t)(((it + 1) >> 1) & 1),
                               u + 1 < u_end);
                }
                return;
            }
            if (close)
                split_part<MODE, DIR, true>(a, stage + buf * NA, tab, t, tn, treg, un, slot, part * a.part, dA, dH);
            else
                split_part<MODE, DIR, false>(a, stage + buf * NA, tab, t, tn, treg, un, slot, part * a.part, dA, dH);
            if ((part & last) == last || u + 1 == seg_end) {
                if (close) {
                    q[0] += dA[0];
                    q[1] += dA[1];
                    q[2] += dH[0];
                    q[3] += dH[1];
                } else {
                    if (MODE & SWEEP_A) {
                        q[0] += fma(phr, dA[0], -(phi * dA[1]));
                        q[1] += fma(phr, dA[1], phi * dA[0]);
                    }
                    if (MODE & SWEEP_AH) {
                        q[2] += fma(phr, dH[0], phi * dH[1]);
                        q[3] += fma(phr, dH[1], -(phi * dH[0]));
                    }
                }
                dA[0] = dA[1] = dH[0] = dH[1] = 0.0;
            }
            __syncthreads();
        }
        if (whole)
            split_write<MODE>(a, slot, q[0], q[1], q[2], q[3]);
        else
            a.partial[((int64_t)blockIdx.x * 2 + seg) * kTile32 + threadIdx.x] =
                make_double4_32a(q[0], q[1], q[2], q[3]);
        seg = 1;
    }
}

// Adds up the pieces of target tiles split between CTAs, in a fixed order:
// four threads a slot take every fourth piece, then their sums are added.  (One
// thread a slot with a 64-bit division a piece took 22 us at n = 2,938, where
// a tile has 25 pieces.  The last CTA of a tile adding them up inside the sweep
// cost the fused pass registers: 4.32 -> 4.62 ms at n = 19,532.)
constexpr int kFixSlots = 64;
template <int MODE>
__global__ void __launch_bounds__(4 * kFixSlots) split_fixup_kernel(ArgsSplit a)
{
    __shared__ double4_32a part[3][kFixSlots];
    const int64_t blk = blockIdx.x, parts = a.npad / a.part;
    auto cta_of = [&](int64_t u) { return ((u + 1) * a.nctas - 1) / a.units; };
    const int64_t c_lo = cta_of(blk * parts), c_hi = cta_of((blk + 1) * parts - 1);
    if (c_lo == c_hi) return;
    const int g = threadIdx.x / kFixSlots, s = threadIdx.x % kFixSlots, slot = blockIdx.y * kFixSlots + s;
    // only the first CTA can have begun in an earlier tile (its slot 1)
    const int first = (c_lo * a.units / a.nctas) / parts == blk ? 0 : 1;
    double q[4] = {0, 0, 0, 0};
#pragma unroll 4
    for (int64_t c = c_lo + g; c <= c_hi; c += 4) {
        const double4_32a v = a.partial[(c * 2 + (c == c_lo ? first : 0)) * kTile32 + slot];
        q[0] += v.x;
        q[1] += v.y;
        q[2] += v.z;
        q[3] += v.w;
    }
    if (g > 0) part[g - 1][s] = make_double4_32a(q[0], q[1], q[2], q[3]);
    __syncthreads();
    if (g > 0) return;
    for (int w = 0; w < 3; w++) {
        const double4_32a v = part[w][s];
        q[0] += v.x;
        q[1] += v.y;
        q[2] += v.z;
        q[3] += v.w;
    }
    split_write<MODE>(a, blk * kTile32 + slot, q[0], q[1], q[2], q[3]);
}

// ------------------------------------------------- several right-hand sides
// Q = A P for blocks of RB = 4, 8 or 16 columns: the entry of a pair is formed
// once (about 165 slots) and each column adds 50.  Wider blocks hold 4 RB FP32
// sums a thread and keep their FP64 sums in shared memory, which leaves one CTA
// an SM; their columns' independent chains fill the pipe instead of warps.
constexpr int kColsMax = 16;
template <int RB>
constexpr int kColsCtas = RB <= 4 ? 2 : 1;
template <int RB>
constexpr size_t kColsSmem = kSplitTable * sizeof(float2) + 2 * (kRecs + RB) * kHalf * sizeof(float4) +
                             (RB <= 4 ? 0 : 2 * RB * kTile32 * sizeof(double));

struct ColsArgs {
    int nr;
    int64_t n, splits;
    const double *p_re, *p_im;  // [nr][n]
    double *q_re, *q_im;
    double2 *partial;           // [splits][RB][npad], splits > 1
};

// Exponents and split densities of column blockIdx.y (see split_max_kernel).
__global__ void __launch_bounds__(256) cols_max_kernel(int64_t n, const double4_32a *__restrict__ nrm,
                                                       const double *__restrict__ p_re,
                                                       const double *__restrict__ p_im, int *__restrict__ part)
{
    const double *pr = p_re + blockIdx.y * n, *pi = p_im + blockIdx.y * n;
    int a = 0;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
        const double w = nrm[s].w;
        a = max(a, max(__double2hiint(w * pr[s]) & 0x7fffffff, __double2hiint(w * pi[s]) & 0x7fffffff));
    }
    a = __reduce_max_sync(0xffffffffu, a);
    __shared__ int sh[8];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) a = max(a, sh[w]);
        part[blockIdx.y * kExpBlocks + blockIdx.x] = a;
    }
}

__global__ void __launch_bounds__(256) cols_dens_kernel(int64_t n, int64_t npad, int nr,
                                                        const int *__restrict__ perm,
                                                        const double4_32a *__restrict__ tpos,
                                                        const double *__restrict__ p_re,
                                                        const double *__restrict__ p_im, double scale,
                                                        int scale_exp, const int *__restrict__ part,
                                                        int *__restrict__ expo, float4 *__restrict__ dens)
{
    const int r = blockIdx.y;
    __shared__ int ex;
    if (threadIdx.x < 32) {
        int v = 0;
        if (r < nr)
            for (int b = threadIdx.x; b < kExpBlocks; b += 32) v = max(v, part[r * kExpBlocks + b]);
        v = __reduce_max_sync(0xffffffffu, v);
        if (threadIdx.x == 0) {
            ex = max(-1000, min(1000, (v >> 20) - 1022));
            if (blockIdx.x == 0) expo[r] = ex + scale_exp;
        }
    }
    __syncthreads();
    const double f = pow2d(-ex);
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < npad; s += (int64_t)gridDim.x * blockDim.x) {
        const int c = perm[s];
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c >= 0 && r < nr) {
            const double w = tpos[s].w;
            const FF x = ff_of_double(-scale * ((w * p_re[r * n + c]) * f)), y = ff_of_double(-scale * ((w * p_im[r * n + c]) * f));
            v = make_float4(x.h, y.h, x.l, y.l);
        }
        dens[r * npad + s] = v;
    }
}

// q[i] is column sum i: q + i when it lies in registers, strided in shared
// memory otherwise.
template <int RB, bool DIR, bool CLOSE>
__device__ __forceinline__ void cols_half(const ArgsSplit &a, const float4 (*st)[kHalf], const float2 *tab,
                                          const Offsets &t, const TargetNormal &tn, FF treg, const TileUnits &u,
                                          int64_t tslot, int64_t sslot0, double phr, double phi, double *q)
{
    constexpr int STEP = RB <= 4 ? 1 : kTile32;
#pragma unroll 1
    for (int j0 = 0; j0 < kHalf; j0 += kRun) {
        FF acc[2 * RB];
#pragma unroll
        for (int r = 0; r < 2 * RB; r++) acc[r] = {0.f, 0.f};
#pragma unroll 1
        for (int j = j0; j < j0 + kRun; j++) {
            FF ar, ai, hr, hi;
            split_entry<SWEEP_A, DIR, CLOSE>(a, st, j, tab, t, tn, treg, u, tslot, sslot0 + j, ar, ai, hr, hi);
#pragma unroll
            for (int r = 0; r < RB; r++) {
                const float4 d = st[kRecs + r][j];
                const FF dr = {d.x, d.z}, di = {d.y, d.w};
                split_dot2<-1>(acc[2 * r], ar, dr, ai, di);
                split_dot2<1>(acc[2 * r + 1], ar, di, ai, dr);
            }
        }
#pragma unroll
        for (int r = 0; r < RB; r++) {
            const double x = (double)acc[2 * r].h + (double)acc[2 * r].l;
            const double y = (double)acc[2 * r + 1].h + (double)acc[2 * r + 1].l;
            double &u0 = q[2 * r * STEP], &u1 = q[(2 * r + 1) * STEP];
            if (CLOSE) {
                u0 += x;
                u1 += y;
            } else {
                u0 = fma(phr, x, fma(-phi, y, u0));
                u1 = fma(phr, y, fma(phi, x, u1));
            }
        }
    }
}

// CTA (target tile, share of the source tiles); with several shares the
// sums go to partial and cols_reduce_kernel adds them up.
template <int RB, bool DIR>
__global__ void __launch_bounds__(kTile32, kColsCtas<RB>) cols_kernel(ArgsSplit a, ColsArgs m)
{
    constexpr int NA = kRecs + RB, STEP = RB <= 4 ? 1 : kTile32;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ alignas(8) uint64_t bar[2];
    float2 *tab = reinterpret_cast<float2 *>(smem);
    float4(*stage)[kHalf] = reinterpret_cast<float4(*)[kHalf]>(smem + kSplitTable * sizeof(float2));
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    for (int i = threadIdx.x; i < kSplitTable / 2; i += kTile32)
        reinterpret_cast<float4 *>(tab)[i] = __ldg(reinterpret_cast<const float4 *>(a.table) + i);
    __syncthreads();
    const int64_t tiles = a.npad / kTile32, blk = blockIdx.x, slot = blk * kTile32 + threadIdx.x;
    const int64_t h_begin = 2 * ((int64_t)blockIdx.y * tiles / m.splits);
    const int64_t h_end = 2 * (((int64_t)blockIdx.y + 1) * tiles / m.splits);
    auto issue = [&](int64_t h, int buf) {
        const uint32_t bytes = kHalf * sizeof(float4);
        mbar_arrive_expect_tx(&bar[buf], NA * bytes);
#pragma unroll
        for (int r = 0; r < kRecs; r++) bulk_g2s(&stage[buf * NA + r][0], a.rec + r * a.npad + h * kHalf, bytes, &bar[buf]);
#pragma unroll
        for (int r = 0; r < RB; r++)
            bulk_g2s(&stage[buf * NA + kRecs + r][0], a.densA + r * a.npad + h * kHalf, bytes, &bar[buf]);
    };
    if (threadIdx.x == 0 && h_begin < h_end) issue(h_begin, 0);
    const double4_32a to = a.tile[blk];
    double X, Y, Z, nx, ny, nz, phr = 1.0, phi = 0.0;
    FF treg;
    TargetNormal tn = {};
    load_target<!DIR>(a, slot, X, Y, Z, nx, ny, nz, treg, tn);
    double qr[RB <= 4 ? 2 * RB : 1];
    double *q = RB <= 4 ? qr
                        : reinterpret_cast<double *>(smem + kSplitTable * sizeof(float2) +
                                                     2 * NA * kHalf * sizeof(float4)) + threadIdx.x;
#pragma unroll
    for (int r = 0; r < 2 * RB; r++) q[r * STEP] = 0.0;
    Offsets t = {};
    TileUnits un = {};
    bool close = false;
    for (int64_t h = h_begin; h < h_end; h++) {
        const int64_t it = h - h_begin;
        const int buf = (int)(it & 1);
        if (threadIdx.x == 0 && h + 1 < h_end) issue(h + 1, buf ^ 1);
        if (!(h & 1)) set_tile<!DIR>(a, h >> 1, to, X, Y, Z, nx, ny, nz, tab, t, un, close, phr, phi);
        const bool ok = mbar_wait_bounded(&bar[buf], (uint32_t)((it >> 1) & 1), g_data_wait_limit);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                atomicOr(a.err, DEV_ERR_WAIT);
                mbar_drain(&bar[buf], (uint32_t)((it >> 1) & 1), &bar[buf ^ 1], (uint32_t)(((it + 1) >> 1) & 1),
                           h + 1 < h_end);
            }
            return;
        }
        if (close)
            cols_half<RB, DIR, true>(a, stage + buf * NA, tab, t, tn, treg, un, slot, h * kHalf, phr, phi, q);
        else
            cols_half<RB, DIR, false>(a, stage + buf * NA, tab, t, tn, treg, un, slot, h * kHalf, phr, phi, q);
        __syncthreads();
    }
    if (m.splits > 1) {
#pragma unroll
        for (int r = 0; r < RB; r++)
            m.partial[((int64_t)blockIdx.y * RB + r) * a.npad + slot] =
                make_double2(q[2 * r * STEP], q[(2 * r + 1) * STEP]);
        return;
    }
    const int c = a.perm[slot];
    if (c < 0) return;
#pragma unroll
    for (int r = 0; r < RB; r++) {
        if (r >= m.nr) break;
        const double x = ldexp(q[2 * r * STEP], a.expo[r]), y = ldexp(q[(2 * r + 1) * STEP], a.expo[r]);
        if (!isfinite(x) || !isfinite(y)) atomicOr(a.err, DEV_ERR_NONFINITE);
        m.q_re[r * m.n + c] = x + 0.5 * m.p_re[r * m.n + c];
        m.q_im[r * m.n + c] = y + 0.5 * m.p_im[r * m.n + c];
    }
}

template <int RB>
__global__ void __launch_bounds__(256) cols_reduce_kernel(ArgsSplit a, ColsArgs m)
{
    const int r = blockIdx.y;
    const int64_t slot = blockIdx.x * (int64_t)256 + threadIdx.x;
    if (slot >= a.npad) return;
    const int c = a.perm[slot];
    if (c < 0) return;
    double x = 0, y = 0;
    for (int64_t s = 0; s < m.splits; s++) {
        const double2 v = m.partial[(s * RB + r) * a.npad + slot];
        x += v.x;
        y += v.y;
    }
    x = ldexp(x, a.expo[r]);
    y = ldexp(y, a.expo[r]);
    if (!isfinite(x) || !isfinite(y)) atomicOr(a.err, DEV_ERR_NONFINITE);
    m.q_re[r * m.n + c] = x + 0.5 * m.p_re[r * m.n + c];
    m.q_im[r * m.n + c] = y + 0.5 * m.p_im[r * m.n + c];
}

// Shares of the source tiles: about three rounds of resident CTAs, so that the
// last one is short, and at least four tiles each (the set-up of a CTA copies
// the 64 KB table).
int64_t cols_splits(int64_t tiles, int ctas)
{
    int64_t s = (3 * (int64_t)ctas + tiles - 1) / tiles;
    if (s > tiles / 4) s = tiles / 4;
    return s < 1 ? 1 : s;
}

template <int RB>
size_t cols_bytes(int64_t npad, int64_t &splits)
{
    splits = cols_splits(npad / kTile32, kColsCtas<RB> * sm_count());
    // densities, partial sums, block maxima and exponents
    return (size_t)npad * RB * (sizeof(float4) + (size_t)(splits > 1 ? splits : 0) * sizeof(double2)) +
           (RB * kExpBlocks + RB) * sizeof(int);
}

ArgsSplit split_args(const SweepConst &c, const RecSplit &v, const double4_32a *nrm);

template <int RB>
int launch_cols(const SweepConst &c, const RecSplit &v, const double4_32a *nrm, int nr, const double *p_re,
                const double *p_im, double *q_re, double *q_im, void *scratch, cudaStream_t s)
{
    const int64_t tiles = v.npad / kTile32;
    const int sms = sm_count();
    ColsArgs m;
    m.nr = nr;
    m.n = c.n;
    cols_bytes<RB>(v.npad, m.splits);
    m.p_re = p_re;
    m.p_im = p_im;
    m.q_re = q_re;
    m.q_im = q_im;
    float4 *dens = static_cast<float4 *>(scratch);
    m.partial = reinterpret_cast<double2 *>(dens + (int64_t)RB * v.npad);
    int *expo = reinterpret_cast<int *>(m.partial + (m.splits > 1 ? m.splits : 0) * RB * v.npad), *part = expo + RB;
    cols_max_kernel<<<dim3(kExpBlocks, (unsigned)nr), 256, 0, s>>>(c.n, nrm, p_re, p_im, part);
    HZ_CHECK_LAUNCH();
    int64_t b = (v.npad + 255) / 256;
    if (b > 2 * sms) b = 2 * sms;
    const double sg = (c.interior == 1) ? -1.0 : 1.0;
    int es;
    const double scale = frexp(sg * c.wave * c.wave / (8.0 * kPiS), &es);
    cols_dens_kernel<<<dim3((unsigned)b, RB), 256, 0, s>>>(c.n, v.npad, nr, v.perm, v.tpos, p_re, p_im, scale, es,
                                                           part, expo, dens);
    HZ_CHECK_LAUNCH();
    ArgsSplit a = split_args(c, v, nrm);
    a.densA = dens;
    a.expo = expo;
    auto kernel = c.dirichlet ? cols_kernel<RB, true> : cols_kernel<RB, false>;
    HZ_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kColsSmem<RB>));
    kernel<<<dim3((unsigned)tiles, (unsigned)m.splits), kTile32, kColsSmem<RB>, s>>>(a, m);
    HZ_CHECK_LAUNCH();
    if (m.splits > 1) {
        cols_reduce_kernel<RB><<<dim3((unsigned)tiles, (unsigned)nr), 256, 0, s>>>(a, m);
        HZ_CHECK_LAUNCH();
    }
    return HZ_OK;
}

template <int MODE, bool DIR>
int launch_split(ArgsSplit a, size_t partial_bytes, cudaStream_t s)
{
    constexpr size_t smem = kSplitTable * sizeof(float2) + 2 * kSplitArrays<MODE> * kHalf * sizeof(float4);
    HZ_CHECK_CUDA(cudaFuncSetAttribute(sweep_split_kernel<MODE, DIR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem));
    const int64_t tiles = a.npad / kTile32;
    int64_t p = 2 * (int64_t)sm_count();
    const int64_t room = (int64_t)(partial_bytes / (2 * kTile32 * sizeof(double4_32a)));
    if (p > room) p = room;
    // Units of 128 sources, or of 64 where that takes a tenth off the fullest
    // CTA's share (n = 3,168: 392 units on 304 CTAs, 0.171 -> 0.138 ms; a unit's
    // end costs 2 % of 64 sources, so elsewhere 128).
    auto share = [&](int64_t part) { return (tiles * (a.npad / part) + p - 1) / p * part; };
    a.part = p > 0 && 11 * share(64) < 10 * share(kHalf) ? 64 : kHalf;
    a.units = tiles * (a.npad / a.part);
    if (p > a.units) p = a.units;
    if (p < 1) {
        set_error("split FP64 sweep: partial buffer too small");
        return HZ_ERR_STATE;
    }
    a.nctas = p;
    sweep_split_kernel<MODE, DIR><<<(unsigned)p, kTile32, smem, s>>>(a);
    HZ_CHECK_LAUNCH();
    split_fixup_kernel<MODE><<<dim3((unsigned)tiles, kTile32 / kFixSlots), 4 * kFixSlots, 0, s>>>(a);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

}  // namespace

size_t split_record_bytes(int64_t npad)
{
    // records, densities, tiles, table, maxima and exponents
    return (size_t)npad * (kRecs + 2) * sizeof(float4) + (size_t)(npad / kTile32) * sizeof(double4_32a) +
           kSplitTable * sizeof(float2) + (2 * kExpBlocks + 8) * sizeof(int);
}

RecSplit split_record_views(void *mem, const Rec32 &r)
{
    RecSplit v;
    v.npad = r.npad;
    v.rec = static_cast<float4 *>(mem);
    v.dens = v.rec + kRecs * r.npad;
    v.tile = reinterpret_cast<double4_32a *>(v.dens + 2 * r.npad);
    v.table = reinterpret_cast<float2 *>(v.tile + r.npad / kTile32);
    v.expo = reinterpret_cast<int *>(v.table + kSplitTable);
    v.perm = r.perm;
    v.tpos = r.tpos;
    v.partial = r.partial;
    v.partial_bytes = r.partial_bytes;
    return v;
}

// Where the split sweep serves.
// * k rho < 4000: there the table reduction of the origin phases ends (as the
//   FP64 sweep's).
// * (k h)^2 <= n^(1/2) / 308 (Dirichlet; k h <= 0.42 at n = 2,938, 0.56 at 9,352, 0.79
//   at 36,212) or n^(3/4) / 3480 (Neumann; 0.34, 0.52, 0.8), and k h <= 0.8: the
//   phases, and with them the entries' error, grow with k h, the FP64 sweep's error
//   with its sequential sum over n.  Error of smooth densities, root mean square,
//   as a part of the FP64 sweep's, Dirichlet / Neumann: n = 2,938 at k h = 0.30
//   0.71 / 0.83, 0.42 0.91 / 1.03; 3,427 at 0.23 0.73 / 0.81, 0.43 0.91 / 1.35; 3,906 at 0.17
//   0.66 / 0.83, 0.41 0.92 / 1.12; 4,465 at 0.27 0.64 / 0.77, 0.46 0.95 / 0.98; 6,338 at 0.46
//   0.70 / 0.70; 9,352 at 0.51 0.85 / 0.90, 0.56 0.90 / 1.16; 24,643 at 0.71 0.90 / 0.91; 36,212
//   at 0.78 0.76 / 0.80.
// * n >= 2800 and k h n^2 >= 2.4e6 (k h >= 0.28 at n = 2,938, 0.12 at 4,465, 0.03 at
//   9,352): at low k the near pairs' projections, off by 2^-51 of the tile's
//   radius, are the error, and a sum over few points costs FP64 instructions
//   little.  The same part for the worse of A and A^H, Neumann: n = 2,511 at
//   k h = 0.05 2.18, 0.36 1.21; 2,938 at 0.05 1.99, 0.11 1.28, 0.22 0.91; 3,427 at 0.10 1.18,
//   0.16 1.16, 0.23 0.84; 4,465 at 0.04 1.28, 0.10 1.08, 0.17 0.86; 6,338 at 0.03 0.89; 9,352
//   at 0.03 0.84; 57,290 at 0.01 0.35.  The FP64 sweep takes milliseconds there, the
//   split one 0.1.
// * k tau >= 2^-28 keeps 1/(k rho)^2 below 2^56 and the units of a close tile's
//   r^2, 2^-53 of (k tau)^2, inside the FP32 range.
// * tau >= h: the projection (x_t - x_s).n carries an error of 2^-51 of the
//   tile's radius (10 to 30 h), which is 2^-46 of the nearest far pairs' entries
//   at rho = h and would grow as 1 / rho below (the FP64 sweep keeps that at k
//   below 1, where it subtracts the unscaled coordinates).
bool split_serves(int64_t n, double wave, double H, double tau, double extent, bool dirichlet)
{
    const double kh = wave * H, m = (double)n;
    const double most = dirichlet ? sqrt(m) / 308.0 : sqrt(m * sqrt(m)) / 3480.0;
    return n >= 2800 && kh * m * m >= 2.4e6 && kh <= 0.8 && kh * kh <= most && wave > 1e-100 && wave < 1e100 &&
           wave * tau >= 0x1p-28 && tau >= H && wave * extent < 4000.0;
}

int build_split_records(const SweepConst &c, const RecSplit &v, const Rec32 &r, const double4_32a *pos,
                        const double4_32a *nrm, cudaStream_t s)
{
    const int64_t tiles = r.npad / kTile32;
    split_table_kernel<<<32, 256, 0, s>>>(v.table);
    HZ_CHECK_LAUNCH();
    split_tile_kernel<<<(unsigned)((tiles + 255) / 256), 256, 0, s>>>(tiles, r.origin, c.wave, c.wave * c.tau, v.tile);
    HZ_CHECK_LAUNCH();
    const double sg = (c.interior == 1) ? -1.0 : 1.0;
    split_records_kernel<<<(unsigned)((r.npad + 255) / 256), 256, 0, s>>>(
        r.npad, r.perm, r.tpos, pos, nrm, v.tile, c.wave, 2.0 * sg * (4.0 * kPiS) / (c.wave * c.wave), v.rec);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

namespace {

// Densities of one product: scale as in split_dens_kernel.
int split_densities(const SweepConst &c, const RecSplit &v, const double4_32a *nrm, const double *pr, const double *pi,
                    const double *tr, const double *ti, double scale, cudaStream_t s)
{
    int *part = v.expo + 8;  // kExpBlocks maxima each
    split_max_kernel<<<kExpBlocks, 256, 0, s>>>(c.n, nrm, pr, pi, tr, ti, part);
    HZ_CHECK_LAUNCH();
    int64_t b = (v.npad + 255) / 256;
    const int64_t cap = 8 * (int64_t)sm_count();
    if (b > cap) b = cap;
    int es;
    scale = frexp(scale, &es);
    split_dens_kernel<<<(unsigned)b, 256, 0, s>>>(v.npad, v.perm, v.tpos, pr, pi, tr, ti, scale, es, part, v.expo,
                                                  v.dens, v.dens + v.npad);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

ArgsSplit split_args(const SweepConst &c, const RecSplit &v, const double4_32a *nrm)
{
    ArgsSplit a = {};
    a.npad = v.npad;
    a.wave = c.wave;
    a.tau = c.tau;
    a.ktau = (float)(c.wave * c.tau);
    a.tau2 = (float)((c.wave * c.tau) * (c.wave * c.tau));
    a.rec = v.rec;
    a.densA = v.dens;
    a.densH = v.dens + v.npad;
    a.tile = v.tile;
    a.table = v.table;
    a.tpos = v.tpos;
    a.nrm = nrm;
    a.perm = v.perm;
    a.expo = v.expo;
    a.partial = v.partial;
    a.err = c.err;
    return a;
}

}  // namespace

int sweep_split(const SweepConst &c, const RecSplit &v, const double4_32a *nrm, int mode, const double *p_re,
                const double *p_im, const double *pt_re, const double *pt_im, double *q_re, double *q_im,
                double *qt_re, double *qt_im, cudaStream_t s, cudaEvent_t ev0, cudaEvent_t ev1)
{
    const bool useA = (mode & SWEEP_A) != 0, useH = (mode & SWEEP_AH) != 0;
    const double sg = (c.interior == 1) ? -1.0 : 1.0;
    HZ_TRY(split_densities(c, v, nrm, useA ? p_re : nullptr, useA ? p_im : nullptr, useH ? pt_re : nullptr,
                           useH ? pt_im : nullptr, sg * c.wave * c.wave / (8.0 * kPiS), s));
    ArgsSplit a = split_args(c, v, nrm);
    a.p_re = p_re; a.p_im = p_im; a.pt_re = pt_re; a.pt_im = pt_im;
    a.q_re = q_re; a.q_im = q_im; a.qt_re = qt_re; a.qt_im = qt_im;
    if (ev0) HZ_CHECK_CUDA(record_timing_event(ev0, s));
    const bool dir = c.dirichlet != 0;
    const size_t pb = v.partial_bytes;
    if (mode == SWEEP_PAIR)
        HZ_TRY((dir ? launch_split<SWEEP_PAIR, true>(a, pb, s) : launch_split<SWEEP_PAIR, false>(a, pb, s)));
    else if (mode == SWEEP_A)
        HZ_TRY((dir ? launch_split<SWEEP_A, true>(a, pb, s) : launch_split<SWEEP_A, false>(a, pb, s)));
    else
        HZ_TRY((dir ? launch_split<SWEEP_AH, true>(a, pb, s) : launch_split<SWEEP_AH, false>(a, pb, s)));
    if (ev1) HZ_CHECK_CUDA(record_timing_event(ev1, s));
    return HZ_OK;
}

// q = (dA/dk) p: far entries -(k / 4 pi) e^{i k rho} (x_t - x_s).n / rho w_s sg,
// near ones w_s dreg (FP64 sincos per pair, one target a thread: 26.2 ms at
// n = 9,542; here 0.9).
int sweep_split_dk(const SweepConst &c, const RecSplit &v, const double4_32a *nrm, const double *dreg,
                   const double *p_re, const double *p_im, double *q_re, double *q_im, cudaStream_t s)
{
    const double sg = (c.interior == 1) ? -1.0 : 1.0;
    HZ_TRY(split_densities(c, v, nrm, p_re, p_im, nullptr, nullptr, -sg * c.wave / (8.0 * kPiS), s));
    ArgsSplit a = split_args(c, v, nrm);
    a.dreg = dreg;
    a.dreg_scale = sg * 8.0 * kPiS / c.wave;
    a.p_re = p_re; a.p_im = p_im; a.q_re = q_re; a.q_im = q_im;
    constexpr int M = SWEEP_A | SPLIT_DK;
    return c.dirichlet ? launch_split<M, true>(a, v.partial_bytes, s) : launch_split<M, false>(a, v.partial_bytes, s);
}

size_t split_cols_scratch_bytes(int64_t npad, int nr)
{
    int64_t splits;
    return nr <= 4 ? cols_bytes<4>(npad, splits) : nr <= 8 ? cols_bytes<8>(npad, splits) : cols_bytes<16>(npad, splits);
}

// One pass over nr <= 16 columns ([nr][n]); scratch of split_cols_scratch_bytes.
int sweep_split_cols(const SweepConst &c, const RecSplit &v, const double4_32a *nrm, int nr, const double *p_re,
                     const double *p_im, double *q_re, double *q_im, void *scratch, cudaStream_t s)
{
    static_assert(kColsMax == 16, "the multi right-hand-side sweep's FP64 block");
    if (nr <= 4) return launch_cols<4>(c, v, nrm, nr, p_re, p_im, q_re, q_im, scratch, s);
    if (nr <= 8) return launch_cols<8>(c, v, nrm, nr, p_re, p_im, q_re, q_im, scratch, s);
    return launch_cols<16>(c, v, nrm, nr, p_re, p_im, q_re, q_im, scratch, s);
}

HZ_DEFINE_WAIT_LIMIT_SETTER(set_wait_limit_split)

}  // namespace hz
