// sweep_multi.cu -- multi-right-hand-side pair sweeps: Q = A P for a block of
// RB density vectors with one kernel evaluation per point pair.
//
// Every pair's kernel value (distance, phase, sin/cos, projection) is
// computed once and multiplied into RB densities.  The FP32 pass follows
// sweep_f32.cu (pair32.cuh, the near-tile mask, head/tail target offsets and
// TwoSum cross-tile sums, no FP64 instruction in the tile loop); its densities
// lie in rows of two columns, (re, re, im, im), so that a column pair costs
// four packed FMAs.  The FP64 pass is sweep_split.cu's where that serves, else
// the kernel below with the arithmetic of pair64.cuh.
//
// A pass on GB300 (torus), before and now: FP32, 16 columns, n = 27,508 5.76 ->
// 3.20 ms, n = 145,272 102 -> 74; 8 columns 3.94 -> 1.89 and 56.6 -> 44; 32
// columns 9.33 -> 5.80 and 177 -> 147.  FP64, 16 columns, 259 -> 38.8 and
// 5,455 -> 1,036; 8 columns 169 -> 21.9 and 3,558 -> 589.
#include "hz_internal.cuh"
#include "pair64.cuh"
#include "pair32.cuh"
#include "bulk_copy.cuh"
#include "krylov_multi.cuh"

namespace hz {
namespace {

constexpr double kPi = 3.14159265358979323846264338328;
// right-hand sides per kernel pass: a pass over RB columns evaluates each
// pair once and spends 4 FMAs per column on it
constexpr int kRBMax32 = 32;
constexpr int kRBMax64 = 16;

// ------------------------------------------------------------------ FP32
constexpr int kHalf32 = 128;  // sources per staged half tile

struct ArgsM32 {
    int64_t n, npad, mwords, splits;
    int nr;  // right-hand sides in this pass (<= RB)
    Wave32 wave;
    float tau2, guard_lo, guard_hi;
    double tau;
    const float4 *pos, *nrm;
    const float4 *dens;  // [RB/2][npad]: (re_{2q}, re_{2q+1}, im_{2q}, im_{2q+1})
    const float4 *thi, *tlo, *ohi, *olo;
    const uint32_t *nearmask;
    const double4_32a *tpos, *pos64;
    const int *perm;
    const double *p_re, *p_im;  // [nr][n] (diagonal term)
    double *q_re, *q_im;        // [nr][n]
    float4 *sums;               // [splits][RB][npad]: re and im, head + tail each
    unsigned *err;
};

template <int RB>
__global__ void prepm32_kernel(int64_t n, int64_t npad, int nr, const int *__restrict__ perm,
                               const double4_32a *__restrict__ tpos, const double *__restrict__ p_re,
                               const double *__restrict__ p_im, double scale, float4 *__restrict__ dens)
{
    const int q = blockIdx.y, r0 = 2 * q, r1 = 2 * q + 1;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < npad; s += (int64_t)gridDim.x * blockDim.x) {
        const int c = perm[s];
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c >= 0) {
            const double ws = tpos[s].w * scale;
            if (r0 < nr) {
                v.x = (float)(ws * p_re[(int64_t)r0 * n + c]);
                v.z = (float)(ws * p_im[(int64_t)r0 * n + c]);
            }
            if (r1 < nr) {
                v.y = (float)(ws * p_re[(int64_t)r1 * n + c]);
                v.w = (float)(ws * p_im[(int64_t)r1 * n + c]);
            }
        }
        dens[(int64_t)q * npad + s] = v;
    }
}

// One source: its entries for the thread's kTgM targets, multiplied into RB
// columns two at a time.
constexpr int kTgM = 2;
constexpr int kNT32m = kTile32 / kTgM;  // threads of a CTA, which owns one target tile

template <int RB, bool DIR, bool SCALED, bool SLOW>
__device__ __forceinline__ void pairm32(const ArgsM32 &a, const float4 *st, int j, const float3 (&rel)[kTgM],
                                        const float3 (&tn)[kTgM], const float (&treg)[kTgM], const Turn (&turn)[kTgM],
                                        int64_t tslot, int64_t src_slot, F2 (&accR)[kTgM][RB / 2],
                                        F2 (&accI)[kTgM][RB / 2])
{
    const float4 s_p = st[j], s_n = st[kHalf32 + j];
    F2 VR[kTgM], VI[kTgM], NV[kTgM];
#pragma unroll
    for (int g = 0; g < kTgM; g++) {
        const float dx = rel[g].x - s_p.x, dy = rel[g].y - s_p.y, dz = rel[g].z - s_p.z;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        bool near = false;
        if (SLOW) {
            near = r2 <= a.tau2;
            if (r2 > a.guard_lo && r2 < a.guard_hi) {
                const int c = a.perm[src_slot];
                if (c >= 0) {
                    const double4_32a q = a.pos64[c];
                    const double4_32a tp = a.tpos[tslot + g * kNT32m];
                    const double x1 = tp.x - q.x, x2 = tp.y - q.y, x3 = tp.z - q.z;
                    near = !(sqrt(x1 * x1 + x2 * x2 + x3 * x3) > a.tau);
                }
            }
        }
        float u1, u2, rr;
        kernel32<SCALED, SLOW>(a.wave, r2, SLOW ? 0.f : turn[g].rc, u1, u2, rr);
        const float pA = DIR ? fmaf(dx, s_n.x, fmaf(dy, s_n.y, dz * s_n.z))
                             : fmaf(dx, tn[g].x, fmaf(dy, tn[g].y, dz * tn[g].z));
        const float f = rr * pA;
        float vr = -u1 * f, vi = u2 * f;
        if (SLOW && near) {
            vr = DIR ? s_p.w : treg[g];
            vi = 0.f;
        }
        VR[g] = f2_pack(vr, vr);
        VI[g] = f2_pack(vi, vi);
        NV[g] = f2_pack(-vi, -vi);
    }
#pragma unroll
    for (int q = 0; q < RB / 2; q++) {
        const ulonglong2 d = *reinterpret_cast<const ulonglong2 *>(st + (2 + q) * kHalf32 + j);
#pragma unroll
        for (int g = 0; g < kTgM; g++) {
            accR[g][q] = f2_fma(VR[g], d.x, f2_fma(NV[g], d.y, accR[g][q]));
            accI[g][q] = f2_fma(VR[g], d.y, f2_fma(VI[g], d.x, accI[g][q]));
        }
    }
}

// Two targets a thread halve the loads of the staged densities (a 128-bit
// broadcast load takes four of an SM's cycles, and one a pair for every two
// columns bound the one-target form).  The cross-tile sums (FP32 head + tail)
// live in global memory, read and written once a tile from L2: in registers
// they left one CTA of eight warps an SM (16 columns, n = 27,750: 5.8 ms), in
// shared memory two of four (3.7 ms).
template <int RB>
constexpr size_t smem_m32 = 2 * (2 + RB / 2) * kHalf32 * sizeof(float4);
template <int RB>
constexpr int kCtas32m = RB <= 8 ? 4 : RB <= 16 ? 3 : 2;

template <int RB, bool DIR, bool SCALED>
__global__ void __launch_bounds__(kNT32m, kCtas32m<RB>) sweepm32_kernel(ArgsM32 a)
{
    constexpr int NA = 2 + RB / 2;
    extern __shared__ __align__(128) float4 smem32[];
    __shared__ alignas(8) uint64_t bar[2];
    float4 *stage[2] = {smem32, smem32 + NA * kHalf32};
    const int64_t blk = blockIdx.x, slot = blk * kTile32 + threadIdx.x;
    float3 th[kTgM], tl[kTgM], tn[kTgM], rel[kTgM];
    float treg[kTgM];
#pragma unroll
    for (int g = 0; g < kTgM; g++) {
        const float4 h = a.thi[slot + g * kNT32m], l = a.tlo[slot + g * kNT32m], m = a.nrm[slot + g * kNT32m];
        th[g] = make_float3(h.x, h.y, h.z);
        tl[g] = make_float3(l.x, l.y, l.z);
        tn[g] = make_float3(m.x, m.y, m.z);
        treg[g] = a.pos[slot + g * kNT32m].w;
    }
    const uint32_t *mrow = a.nearmask + blk * a.mwords;  // near-tile mask row
    const int64_t tiles = a.npad / kTile32;
    const int64_t h_begin = 2 * ((int64_t)blockIdx.y * tiles / a.splits);
    const int64_t h_end = 2 * (((int64_t)blockIdx.y + 1) * tiles / a.splits);
    float4 *sum = a.sums + (int64_t)blockIdx.y * RB * a.npad + slot;
    bool first = true;
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    __syncthreads();
    auto issue = [&](int64_t h, int buf) {
        const int64_t base = h * kHalf32;
        const uint32_t bytes = kHalf32 * sizeof(float4);
        mbar_arrive_expect_tx(&bar[buf], NA * bytes);
        bulk_g2s(stage[buf], a.pos + base, bytes, &bar[buf]);
        bulk_g2s(stage[buf] + kHalf32, a.nrm + base, bytes, &bar[buf]);
#pragma unroll
        for (int q = 0; q < RB / 2; q++)
            bulk_g2s(stage[buf] + (2 + q) * kHalf32, a.dens + q * a.npad + base, bytes, &bar[buf]);
    };
    if (threadIdx.x == 0 && h_begin < h_end) issue(h_begin, 0);
    F2 accR[kTgM][RB / 2], accI[kTgM][RB / 2];
    Turn turn[kTgM];
#pragma unroll
    for (int g = 0; g < kTgM; g++) {
#pragma unroll
        for (int q = 0; q < RB / 2; q++) accR[g][q] = accI[g][q] = 0;
        rel[g] = make_float3(0.f, 0.f, 0.f);
        turn[g] = {};
    }
    bool slow = false;
    for (int64_t h = h_begin; h < h_end; h++) {
        const int64_t it = h - h_begin, tile = h >> 1;
        const int buf = (int)(it & 1);
        if (threadIdx.x == 0 && h + 1 < h_end) issue(h + 1, buf ^ 1);
        if (!(h & 1)) {
            const float4 oh = a.ohi[tile], ol = a.olo[tile];
            slow = ((__ldg(mrow + (tile >> 5)) >> (tile & 31)) & 1u) || (SCALED && oh.w > kCentreRadius);
#pragma unroll
            for (int g = 0; g < kTgM; g++) {
                rel[g] = make_float3((th[g].x - oh.x) + (tl[g].x - ol.x), (th[g].y - oh.y) + (tl[g].y - ol.y),
                                     (th[g].z - oh.z) + (tl[g].z - ol.z));
                if (SCALED && !slow) turn[g] = turn_of(rel[g]);
            }
        }
        const bool ok = mbar_wait_bounded(&bar[buf], (uint32_t)((it >> 1) & 1), g_data_wait_limit);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                atomicOr(a.err, DEV_ERR_WAIT);
                mbar_drain(&bar[buf], (uint32_t)((it >> 1) & 1), &bar[buf ^ 1], (uint32_t)(((it + 1) >> 1) & 1),
                           h + 1 < h_end);
            }
            return;
        }
        const float4 *st = stage[buf];
        const int64_t base = h * kHalf32;
        if (slow) {
            for (int j = 0; j < kHalf32; j++)
                pairm32<RB, DIR, SCALED, true>(a, st, j, rel, tn, treg, turn, slot, base + j, accR, accI);
        } else {
            for (int j = 0; j < kHalf32; j++)
                pairm32<RB, DIR, SCALED, false>(a, st, j, rel, tn, treg, turn, slot, base + j, accR, accI);
        }
        if (h & 1) {
#pragma unroll
            for (int g = 0; g < kTgM; g++)
#pragma unroll
                for (int q = 0; q < RB / 2; q++) {
                    float re[2], im[2];
                    f2_unpack(accR[g][q], re[0], re[1]);
                    f2_unpack(accI[g][q], im[0], im[1]);
                    accR[g][q] = accI[g][q] = 0;
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        if (SCALED && !slow) turn_sum<false>(turn[g], re[e], im[e]);
                        float4 *at = sum + (int64_t)(2 * q + e) * a.npad + g * kNT32m;
                        float4 x = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *at;
                        two_sum_acc(x.x, x.y, re[e]);
                        two_sum_acc(x.z, x.w, im[e]);
                        *at = x;
                    }
                }
            first = false;
        }
        __syncthreads();
    }
}

// Adds up the shares of the source tiles in order, and the diagonal term.
template <int RB>
__global__ void __launch_bounds__(256) reducem32_kernel(ArgsM32 a)
{
    const int r = blockIdx.y;
    const int64_t slot = blockIdx.x * (int64_t)256 + threadIdx.x;
    if (slot >= a.npad) return;
    const int c = a.perm[slot];
    if (c < 0) return;
    double vr = 0, vi = 0;
    for (int64_t s = 0; s < a.splits; s++) {
        const float4 v = a.sums[(s * RB + r) * a.npad + slot];
        vr += (double)v.x + (double)v.y;
        vi += (double)v.z + (double)v.w;
    }
    if (!isfinite(vr) || !isfinite(vi)) atomicOr(a.err, DEV_ERR_NONFINITE);
    a.q_re[(int64_t)r * a.n + c] = vr + 0.5 * a.p_re[(int64_t)r * a.n + c];
    a.q_im[(int64_t)r * a.n + c] = vi + 0.5 * a.p_im[(int64_t)r * a.n + c];
}

// ------------------------------------------------------------------ FP64
constexpr int kT64m = 128;  // sources per tile = threads per block

struct ArgsM64 {
    int64_t n;
    int nr;
    double wave, tau, tau2, sg;
    float kscale;     // k * 2048 / (2 pi), the phase table index in FP32
    long long tau2b;  // bit pattern of tau^2
    const double4_32a *pos, *nrm;
    const double4_32a *dens;  // [RB/2][n]: (w p_{2q}, w p_{2q+1})
    const double *p_re, *p_im;
    double *q_re, *q_im;
    unsigned *err;
};

template <int RB>
__global__ void prepm64_kernel(int64_t n, int nr, const double4_32a *__restrict__ nrm, const double *__restrict__ p_re,
                               const double *__restrict__ p_im, double4_32a *__restrict__ dens)
{
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
        const double w = nrm[s].w;
#pragma unroll
        for (int q = 0; q < RB / 2; q++) {
            const int r0 = 2 * q, r1 = 2 * q + 1;
            double4_32a v = make_double4_32a(0, 0, 0, 0);
            if (r0 < nr) {
                v.x = w * p_re[(int64_t)r0 * n + s];
                v.y = w * p_im[(int64_t)r0 * n + s];
            }
            if (r1 < nr) {
                v.z = w * p_re[(int64_t)r1 * n + s];
                v.w = w * p_im[(int64_t)r1 * n + s];
            }
            dens[(int64_t)q * n + s] = v;
        }
    }
}

template <int RB>
constexpr size_t smem_m64() { return 2 * (2 + RB / 2) * kT64m * sizeof(double4_32a); }

template <int RB, bool DIR>
__global__ void __launch_bounds__(kT64m) sweepm64_kernel(ArgsM64 a)
{
    constexpr int T = kT64m;
    extern __shared__ __align__(128) double4_32a smem64[];
    __shared__ alignas(8) uint64_t bar[2];
    __shared__ alignas(16) double2 tab[kPhaseTable];
    fill_phase_table(tab);
    double4_32a *sp[2] = {smem64, smem64 + (2 + RB / 2) * T};
    const double c4 = 1. / (4. * kPi);
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = t < a.n;
    double4_32a tp = make_double4_32a(0, 0, 0, 0), tn = make_double4_32a(0, 0, 0, 0);
    if (valid) {
        tp = a.pos[t];
        tn = a.nrm[t];
    }
    double acc[2 * RB];
#pragma unroll
    for (int i = 0; i < 2 * RB; i++) acc[i] = 0.0;
    const int64_t ntiles = (a.n + T - 1) / T;
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    __syncthreads();
    auto issue = [&](int64_t tile, int buf) {
        const int64_t base = tile * T;
        const int64_t cnt = (a.n - base < T) ? (a.n - base) : T;
        const uint32_t bytes = (uint32_t)(cnt * sizeof(double4_32a));
        mbar_arrive_expect_tx(&bar[buf], (2 + RB / 2) * bytes);
        bulk_g2s(sp[buf], a.pos + base, bytes, &bar[buf]);
        bulk_g2s(sp[buf] + T, a.nrm + base, bytes, &bar[buf]);
#pragma unroll
        for (int q = 0; q < RB / 2; q++) bulk_g2s(sp[buf] + (2 + q) * T, a.dens + q * a.n + base, bytes, &bar[buf]);
    };
    if (threadIdx.x == 0 && ntiles > 0) issue(0, 0);
    for (int64_t tile = 0; tile < ntiles; tile++) {
        const int buf = (int)(tile & 1);
        if (threadIdx.x == 0 && tile + 1 < ntiles) issue(tile + 1, buf ^ 1);
        const bool ok = mbar_wait_bounded(&bar[buf], (uint32_t)((tile >> 1) & 1), g_data_wait_limit);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                atomicOr(a.err, DEV_ERR_WAIT);
                mbar_drain(&bar[buf], (uint32_t)((tile >> 1) & 1), &bar[buf ^ 1], (uint32_t)(((tile + 1) >> 1) & 1),
                           tile + 1 < ntiles);
            }
            return;
        }
        const int64_t base = tile * T;
        const int cnt = (int)((a.n - base < T) ? (a.n - base) : T);
        const double4_32a *P = sp[buf], *Nn = sp[buf] + T, *D = sp[buf] + 2 * T;
        if (valid) {
            for (int j = 0; j < cnt; j++) {
                const double4_32a s_p = P[j], s_n = Nn[j];
                const double xmy1 = tp.x - s_p.x, xmy2 = tp.y - s_p.y, xmy3 = tp.z - s_p.z;
                const double r2 = fma(xmy3, xmy3, fma(xmy2, xmy2, xmy1 * xmy1));
                // near-field test as in sweep_f64.cu: bit patterns, the
                // reference's arithmetic within 8192 ulps of tau^2
                const long long rb = __double_as_longlong(r2);
                bool far = rb > a.tau2b;
                if ((unsigned long long)(rb - a.tau2b + 8192) <= 16384ull) {
                    const double r2ref = __dadd_rn(__dadd_rn(__dmul_rn(xmy1, xmy1), __dmul_rn(xmy2, xmy2)),
                                                   __dmul_rn(xmy3, xmy3));
                    far = __dsqrt_rn(r2ref) > a.tau;
                }
                double vr, vi;
                if (far) {
                    double ur, ui, y2;
                    far_factor64<false>(r2, a.wave, a.kscale, tab, ur, ui, y2);
                    const double in = DIR ? fma(xmy3, s_n.z, fma(xmy2, s_n.y, xmy1 * s_n.x))
                                          : fma(xmy3, tn.z, fma(xmy2, tn.y, xmy1 * tn.x));
                    const double f = (a.sg * c4) * (in * y2);
                    vr = ur * f;
                    vi = ui * f;
                } else {
                    vr = DIR ? s_p.w : tp.w;
                    vi = 0.0;
                }
#pragma unroll
                for (int q = 0; q < RB / 2; q++) {
                    const double4_32a d = D[q * T + j];
                    acc[4 * q + 0] += vr * d.x - vi * d.y;
                    acc[4 * q + 1] += vr * d.y + vi * d.x;
                    acc[4 * q + 2] += vr * d.z - vi * d.w;
                    acc[4 * q + 3] += vr * d.w + vi * d.z;
                }
            }
        }
        __syncthreads();
    }
    if (!valid) return;
#pragma unroll
    for (int r = 0; r < RB; r++) {
        if (r >= a.nr) break;
        const double vr = acc[2 * r], vi = acc[2 * r + 1];
        if (!isfinite(vr) || !isfinite(vi)) atomicOr(a.err, DEV_ERR_NONFINITE);
        a.q_re[(int64_t)r * a.n + t] = vr + 0.5 * a.p_re[(int64_t)r * a.n + t];
        a.q_im[(int64_t)r * a.n + t] = vi + 0.5 * a.p_im[(int64_t)r * a.n + t];
    }
}

int blocks_for(int64_t work)
{
    long long b = (work + 255) / 256;
    if (b > 4096) b = 4096;
    return (int)(b < 1 ? 1 : b);
}

// Block of the next pass for `left` remaining columns: the smallest compiled
// block that holds them all, else the largest.  FP32, 17 to 24 columns: 16 and
// then 8 (74 + 44 ms at n = 145,272, one pass of 32 147 ms).
int pass_block(int precision, int left)
{
    const int top = (precision == HZ_PREC_F64) ? kRBMax64 : kRBMax32;
    if (top == kRBMax32 && left > 16 && left <= 24) return 16;
    for (int rb = 8; rb < top; rb *= 2)
        if (left <= rb) return rb;
    return top;
}

template <int RB>
int launch_m64(const SweepConst &c, const Rec64 &r64, int nr, const double *pr, const double *pi, double *qr,
               double *qi, void *scratch, cudaStream_t s)
{
    constexpr int smem = (int)smem_m64<RB>();
    if (!(c.wave * c.extent <= kMaxPhase64)) {
        set_error("FP64 multi-RHS sweep: k * domain diagonal = %g exceeds the phase reduction's range (%g)",
                  c.wave * c.extent, kMaxPhase64);
        return HZ_ERR_ARG;
    }
    HZ_CHECK_CUDA(cudaFuncSetAttribute(sweepm64_kernel<RB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    HZ_CHECK_CUDA(cudaFuncSetAttribute(sweepm64_kernel<RB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    double4_32a *dens = static_cast<double4_32a *>(scratch);
    prepm64_kernel<RB><<<blocks_for(c.n), 256, 0, s>>>(c.n, nr, r64.nrm, pr, pi, dens);
    HZ_CHECK_LAUNCH();
    ArgsM64 a;
    a.n = c.n;
    a.nr = nr;
    a.wave = c.wave;
    a.tau = c.tau;
    a.tau2 = c.tau * c.tau;
    a.tau2b = __builtin_bit_cast(long long, a.tau2);
    a.kscale = (float)(c.wave * (kPhaseTable / (2.0 * kPi)));
    a.sg = (c.interior == 1) ? -1.0 : 1.0;
    a.pos = r64.pos;
    a.nrm = r64.nrm;
    a.dens = dens;
    a.p_re = pr;
    a.p_im = pi;
    a.q_re = qr;
    a.q_im = qi;
    a.err = c.err;
    const unsigned blocks = (unsigned)((c.n + kT64m - 1) / kT64m);
    if (c.dirichlet) sweepm64_kernel<RB, true><<<blocks, kT64m, smem, s>>>(a);
    else sweepm64_kernel<RB, false><<<blocks, kT64m, smem, s>>>(a);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

// Shares of the source tiles of the FP32 pass: one when the target tiles fill
// the chip six times over, else enough for about four rounds of resident CTAs
// (short last round), of at least two tiles each.
template <int RB>
int64_t splits_m32(int64_t npad)
{
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t tiles = npad / kTile32, ctas = (int64_t)kCtas32m<RB> * sms;
    if (tiles >= 6 * ctas) return 1;
    int64_t s = (4 * ctas + tiles - 1) / tiles;
    if (s > tiles / 2) s = tiles / 2;
    return s < 1 ? 1 : s;
}

template <int RB>
size_t bytes_m32(int64_t npad)
{
    const int64_t sp = splits_m32<RB>(npad);
    return (size_t)npad * (RB / 2 + sp * RB) * sizeof(float4);
}

template <int RB>
int launch_m32(const SweepConst &c, const Rec32 &r32, const Rec64 &r64, int nr, const double *pr, const double *pi,
               double *qr, double *qi, void *scratch, cudaStream_t s)
{
    const Const32 k32 = constants32(c, r32.lambda);
    auto kernel = k32.scaled ? (c.dirichlet ? sweepm32_kernel<RB, true, true> : sweepm32_kernel<RB, false, true>)
                             : (c.dirichlet ? sweepm32_kernel<RB, true, false> : sweepm32_kernel<RB, false, false>);
    HZ_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_m32<RB>));
    float4 *dens = static_cast<float4 *>(scratch);
    const double scale = 1.0 / sweep32_reg_scale(c.interior, r32.lambda);
    prepm32_kernel<RB><<<dim3((unsigned)(r32.npad / 256), RB / 2), 256, 0, s>>>(c.n, r32.npad, nr, r32.perm, r32.tpos,
                                                                               pr, pi, scale, dens);
    HZ_CHECK_LAUNCH();
    ArgsM32 a;
    a.n = c.n;
    a.npad = r32.npad;
    a.splits = splits_m32<RB>(r32.npad);
    a.sums = dens + (int64_t)(RB / 2) * r32.npad;
    a.nr = nr;
    a.wave = {k32.k, k32.kh, k32.kl};
    a.tau = c.tau;
    a.mwords = r32.mwords;
    a.tau2 = k32.tau2;
    a.guard_lo = k32.guard_lo;
    a.guard_hi = k32.guard_hi;
    a.pos = r32.pos;
    a.nrm = r32.nrm;
    a.dens = dens;
    a.thi = r32.thi;
    a.tlo = r32.tlo;
    a.ohi = r32.ohi;
    a.olo = r32.olo;
    a.nearmask = r32.nearmask;
    a.tpos = r32.tpos;
    a.pos64 = r64.pos;
    a.perm = r32.perm;
    a.p_re = pr;
    a.p_im = pi;
    a.q_re = qr;
    a.q_im = qi;
    a.err = c.err;
    const unsigned tiles = (unsigned)(r32.npad / kTile32);
    kernel<<<dim3(tiles, (unsigned)a.splits), kNT32m, smem_m32<RB>, s>>>(a);
    HZ_CHECK_LAUNCH();
    reducem32_kernel<RB><<<dim3(tiles, (unsigned)nr), 256, 0, s>>>(a);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

}  // namespace

long long multi_rhs_passes(int precision, int nrhs)
{
    long long p = 0;
    for (int r0 = 0; r0 < nrhs; r0 += pass_block(precision, nrhs - r0)) p++;
    return p;
}

size_t multi_rhs_scratch_bytes(int precision, int nrhs, int64_t n, const Rec32 &r32, const Rec64 &r64)
{
    size_t most = 0;
    for (int r0 = 0; r0 < nrhs;) {
        const int rb = pass_block(precision, nrhs - r0), nr = (nrhs - r0 < rb) ? (nrhs - r0) : rb;
        size_t b;
        if (precision != HZ_PREC_F64)
            b = rb == 8 ? bytes_m32<8>(r32.npad) : rb == 16 ? bytes_m32<16>(r32.npad) : bytes_m32<32>(r32.npad);
        else if (r64.split)
            b = split_cols_scratch_bytes(r32.npad, nr);
        else
            b = (size_t)(rb / 2) * (size_t)n * sizeof(double4_32a);
        if (b > most) most = b;
        r0 += nr;
    }
    return most;
}

int sweep_multi(const SweepConst &c, const Rec32 &r32, const Rec64 &r64, int precision, int nrhs,
                const double *p_re, const double *p_im, double *q_re, double *q_im, void *scratch,
                cudaStream_t s)
{
    if (c.n <= 0 || nrhs <= 0) return HZ_OK;
    for (int r0 = 0; r0 < nrhs;) {
        const int rb = pass_block(precision, nrhs - r0);
        const int nr = (nrhs - r0 < rb) ? (nrhs - r0) : rb;
        const double *pr = p_re + (int64_t)r0 * c.n, *pi = p_im + (int64_t)r0 * c.n;
        double *qr = q_re + (int64_t)r0 * c.n, *qi = q_im + (int64_t)r0 * c.n;
        if (precision == HZ_PREC_F64) {
            if (r64.split) HZ_TRY(sweep_split_cols(c, *r64.split, r64.nrm, nr, pr, pi, qr, qi, scratch, s));
            else if (rb == 8) HZ_TRY(launch_m64<8>(c, r64, nr, pr, pi, qr, qi, scratch, s));
            else HZ_TRY(launch_m64<16>(c, r64, nr, pr, pi, qr, qi, scratch, s));
        } else {
            if (rb == 8) HZ_TRY(launch_m32<8>(c, r32, r64, nr, pr, pi, qr, qi, scratch, s));
            else if (rb == 16) HZ_TRY(launch_m32<16>(c, r32, r64, nr, pr, pi, qr, qi, scratch, s));
            else HZ_TRY(launch_m32<32>(c, r32, r64, nr, pr, pi, qr, qi, scratch, s));
        }
        r0 += nr;
    }
    return HZ_OK;
}

HZ_DEFINE_WAIT_LIMIT_SETTER(set_wait_limit_multi)

}  // namespace hz
