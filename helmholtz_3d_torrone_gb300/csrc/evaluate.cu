// evaluate.cu -- off-surface field at receivers, boundary data at the tube
// points, and the dense complex matvec behind the CompBiCG drop-in.
#include <limits>

#include "hz_internal.cuh"
#include "pair64.cuh"

namespace hz {
namespace {

constexpr int kEvalThreads = 256;

// One pair of the field in plain FP64: any distance, k and infinities.
template <bool SINGLE>
__device__ __noinline__ bool field_pair(double x, double y, double z, double nx, double ny, double nz, double wave,
                                        double tau, double &re, double &im)
{
    const double rho = sqrt(x * x + y * y + z * z);
    if (!(rho > tau)) return false;
    double S, C;
    sincos(wave * rho, &S, &C);
    if (SINGLE) {
        re = C / rho;
        im = S / rho;
    } else {
        const double in = (x * nx + y * ny + z * nz) / (rho * rho);
        re = -(wave * S + C / rho) * in;
        im = (wave * C - S / rho) * in;
    }
    return true;
}

// A block sums the field at R receivers: sources strided over the block, FP64,
// reduced in a fixed order.  Single layer: NeumannTest (large3Dexample2.c:1810-1824),
//   u += (-Phi) sigma w with -Phi = (cos(k r) + i sin(k r)) / (-4 pi r);
// double layer: the Dirichlet matrix's kernel (:4471-4497) off the surface,
//   u += sg (ct1 + i ct2) ((x - x_p).n_p) sigma w.
// Pairs with r <= tau are skipped, as in the reference.
//
// Bound by the FP64 pipe (1.65 lanes a clock an SM): sincos, sqrt and the
// division are 67 FP64 instructions a pair; far_factor64 on (k r)^2 is 39, and
// two a source for w sigma are shared by the R receivers.  Coordinates are
// subtracted unscaled, so neither the factor nor the test r <= tau depends on
// how far from the origin the box lies.  The 32 KB phase table is filled once a
// block, so the blocks stay and take receivers in turn.  The table serves
// k r < 4000; pairs beyond, within 1e-12 of tau, and NaN go through field_pair.
// The split FP32 arithmetic of the products would be 8 times as fast, but
// its entries carry 2^-46.5 where these carry 2^-52: a field was off by
// 2.2e-15 instead of 5e-16.  9,216 receivers of a sphere's tube at 48^3:
// 13.3 -> 8.3 ms.
template <bool SINGLE, int R>
__global__ void __launch_bounds__(kEvalThreads, 2)
    eval_kernel(int64_t n, const double4_32a *__restrict__ pos, const double4_32a *__restrict__ nrm,
                const double *__restrict__ s_re, const double *__restrict__ s_im, int64_t m,
                const double *__restrict__ rx, double wave, double k2, double tau, double near_lo, double near_hi,
                double plain, double scale, double *u_re, double *u_im)
{
    const float kscale = (float)(kPhaseTable / (2 * 3.14159265358979323846));
    __shared__ alignas(16) double2 tab[kPhaseTable];
    __shared__ double sh[2 * R][kEvalThreads / 32];
    fill_phase_table_folded(tab);
    for (int64_t r0 = blockIdx.x * (int64_t)R; r0 < m; r0 += gridDim.x * (int64_t)R) {
        __syncthreads();
        double X[R][3], ur[R], ui[R];
#pragma unroll
        for (int g = 0; g < R; g++) {
            const int64_t r = min(r0 + g, m - 1);
            for (int a = 0; a < 3; a++) X[g][a] = rx[3 * r + a];
            ur[g] = ui[g] = 0.0;
        }
        for (int64_t c = threadIdx.x; c < n; c += kEvalThreads) {
            const double4_32a p = pos[c], q = nrm[c];
            const double d0 = q.w * s_re[c], d1 = q.w * s_im[c];
#pragma unroll
            for (int g = 0; g < R; g++) {
                const double x = X[g][0] - p.x, y = X[g][1] - p.y, z = X[g][2] - p.z;
                const double r2 = fma(z, z, fma(y, y, x * x)), kr2 = k2 * r2;
                double vr, vi;
                if (r2 > near_hi && kr2 < 1.6e7) {
                    if (SINGLE) {
                        double y;
                        far_wave64(kr2, kscale, tab, vr, vi, y);
                        vr *= y;
                        vi *= y;
                    } else {
                        double y2;
                        far_factor64<true>(kr2, 1.0, kscale, tab, vr, vi, y2);
                        const double f = fma(z, q.z, fma(y, q.y, x * q.x)) * y2;
                        vr *= f;
                        vi *= f;
                    }
                } else if (r2 <= near_lo) {
                    continue;
                } else {
                    if (!field_pair<SINGLE>(x, y, z, q.x, q.y, q.z, wave, tau, vr, vi)) continue;
                    vr *= plain;
                    vi *= plain;
                }
                ur[g] = fma(-vi, d1, fma(vr, d0, ur[g]));
                ui[g] = fma(vi, d0, fma(vr, d1, ui[g]));
            }
        }
#pragma unroll
        for (int g = 0; g < R; g++)
            for (int o = 16; o > 0; o >>= 1) {
                ur[g] += __shfl_down_sync(0xffffffffu, ur[g], o);
                ui[g] += __shfl_down_sync(0xffffffffu, ui[g], o);
            }
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int g = 0; g < R; g++) {
                sh[2 * g][threadIdx.x >> 5] = ur[g];
                sh[2 * g + 1][threadIdx.x >> 5] = ui[g];
            }
        __syncthreads();
        if (threadIdx.x < 2 * R && r0 + threadIdx.x / 2 < m) {
            double a = 0.0;
            for (int w = 0; w < kEvalThreads / 32; w++) a += sh[threadIdx.x][w];
            ((threadIdx.x & 1) ? u_im : u_re)[r0 + threadIdx.x / 2] = scale * a;
        }
    }
}

// The phase table holds for receivers in general position; k = 0, a negative k,
// one so small that (k tau)^2 leaves the FP32 range and one whose cube leaves the
// FP64 range take field_pair alone.
template <bool SINGLE, int R>
int eval_blocks(int64_t n, const double4_32a *pos, const double4_32a *nrm, const double *s_re, const double *s_im,
                int64_t m, const double *rx, double wave, double tau, double sg, double *u_re, double *u_im,
                cudaStream_t s)
{
    const double kt = wave * tau, inf = std::numeric_limits<double>::infinity();
    const bool table = wave > 1e-100 && wave < 1e100 && kt * kt > 1e-30 && kt < 4000.0;
    // the table's pairs are the fields' over k (single layer) and k^3
    const double f = !table ? 1.0 : SINGLE ? wave : wave * wave * wave, c = (SINGLE ? -1.0 : sg) / (4.0 * 3.14159265358979323846264338328);
    int64_t b = (m + R - 1) / R;
    const int64_t cap = 2 * (int64_t)sm_count();
    if (b > cap) b = cap;
    eval_kernel<SINGLE, R><<<(unsigned)b, kEvalThreads, 0, s>>>(
        n, pos, nrm, s_re, s_im, m, rx, wave, wave * wave, tau, table ? tau * tau * (1 - 1e-12) : -1.0,
        table ? tau * tau * (1 + 1e-12) : inf, 1.0 / f, c * f, u_re, u_im);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

// Boundary data at projected points (see HZ_RHS_*).
__global__ void rhs_kernel(int64_t n, const double4_32a *__restrict__ pos, const double4_32a *__restrict__ nrm, double sx,
                           double sy, double sz, double W, int kind, double *b_re, double *b_im)
{
    const double PI = 3.14159265358979323846264338328;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        const double4_32a p = pos[c], q = nrm[c];
        const double dx = p.x - sx, dy = p.y - sy, dz = p.z - sz;
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        double S, C;
        sincos(W * r, &S, &C);
        double re, im;
        if (kind == HZ_RHS_POINT_DIRICHLET) {
            re = C / (4. * PI * r);
            im = S / (4. * PI * r);
        } else if (kind == HZ_RHS_POINT_NEUMANN) {
            const double dn = -(dx * q.x + dy * q.y + dz * q.z) / r;
            const double gr = (-C - W * r * S) / (4. * PI * r * r);
            const double gi = (W * r * C - S) / (4. * PI * r * r);
            re = gr * dn;
            im = gi * dn;
        } else if (kind == HZ_RHS_MONOPOLE_NEUMANN) {
            re = (S / r) + (C / (W * r * r));
            im = (S / (W * r * r)) - (C / r);
        } else {
            re = -1.0 * C / (W * r);
            im = -1.0 * S / (W * r);
        }
        b_re[c] = re;
        b_im[c] = im;
    }
}

// Receivers on a plane and a mask from the trilinearly interpolated
// distance grid (1 = keep, 0 = inside or within mask of the surface).
__global__ void slice_points_kernel(int axis, double c, int n2, double lo, double h2, double mask, int N, double H,
                                    double int_l, const double *__restrict__ d, double *rx, unsigned char *keep)
{
    const int64_t total = (int64_t)n2 * n2;
    const long long S = N + 1;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int a = (int)(q / n2), b = (int)(q % n2);
        const double u = lo + a * h2, v = lo + b * h2;
        double x, y, z;
        if (axis == 0) { x = c; y = u; z = v; }
        else if (axis == 1) { x = u; y = c; z = v; }
        else { x = u; y = v; z = c; }
        rx[3 * q] = x;
        rx[3 * q + 1] = y;
        rx[3 * q + 2] = z;
        int i = (int)floor((y - int_l) / H), j = (int)floor((x - int_l) / H), k = (int)floor((z - int_l) / H);
        unsigned char kp = 1;
        if (i >= 0 && j >= 0 && k >= 0 && i < N && j < N && k < N) {
            const double ly = (y - int_l) / H - i, lx = (x - int_l) / H - j, lz = (z - int_l) / H - k;
            const long long o = ((long long)i * S + j) * S + k;
            double acc = 0.0;
            for (int di = 0; di < 2; di++)
                for (int dj = 0; dj < 2; dj++)
                    for (int dk = 0; dk < 2; dk++) {
                        const double wgt = (di ? ly : 1 - ly) * (dj ? lx : 1 - lx) * (dk ? lz : 1 - lz);
                        acc += wgt * d[o + di * S * S + dj * S + dk];
                    }
            if (acc > -mask) kp = 0;
        }
        keep[q] = kp;
    }
}

__global__ void apply_mask_kernel(int64_t m, const unsigned char *__restrict__ keep, double *u_re, double *u_im)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < m; q += (int64_t)gridDim.x * blockDim.x)
        if (!keep[q]) {
            u_re[q] = 0.0;
            u_im[q] = 0.0;
        }
}

// Incident plane waves u = e^{ik d.x} at the projected points, one column
// [ndir][n] per direction: Dirichlet data (kind 0) or its derivative along
// the outward normal -n (kind 1).
__global__ void plane_wave_kernel(int64_t n, const double4_32a *__restrict__ pos, const double4_32a *__restrict__ nrm,
                                  int ndir, const double *__restrict__ dirs, double W, int kind, double *b_re,
                                  double *b_im)
{
    const int r = blockIdx.y;
    const double dx = dirs[3 * r], dy = dirs[3 * r + 1], dz = dirs[3 * r + 2];
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        const double4_32a p = pos[c];
        double S, C;
        sincos(W * (dx * p.x + dy * p.y + dz * p.z), &S, &C);
        double re = C, im = S;
        if (kind == HZ_RHS_POINT_NEUMANN) {
            const double4_32a q = nrm[c];
            const double dn = -(dx * q.x + dy * q.y + dz * q.z);  // d . n_out
            re = -W * dn * S;                                     // i k (d.n_out) e^{ik d.x}
            im = W * dn * C;
        }
        b_re[(int64_t)r * n + c] = re;
        b_im[(int64_t)r * n + c] = im;
    }
}

// Dense complex products on a row-major n x n matrix (real and imaginary
// parts), large3Dexample2.c:3262-3309: q = A p and qt = A^H pt in one pass
// over A.  A block owns kDenseRows rows; each warp walks its rows with
// coalesced column loads, and A^H contributions for the block's rows are
// written to partial[row_block][col] and reduced in a second, ordered pass.
constexpr int kDenseRows = 32;

__global__ void dense_rows_kernel(int64_t n, const double *__restrict__ are, const double *__restrict__ aim,
                                  const double *__restrict__ p_re, const double *__restrict__ p_im,
                                  const double *__restrict__ pt_re, const double *__restrict__ pt_im,
                                  double *__restrict__ q_re, double *__restrict__ q_im,
                                  double *__restrict__ part_re, double *__restrict__ part_im, int do_a, int do_adj)
{
    const int64_t r0 = (int64_t)blockIdx.x * kDenseRows;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nwarps = blockDim.x >> 5;
    // A p: one warp per row
    for (int rr = warp; do_a && rr < kDenseRows; rr += nwarps) {
        const int64_t row = r0 + rr;
        if (row >= n) break;
        const double *ar = are + row * n, *ai = aim + row * n;
        double sr = 0.0, si = 0.0;
        for (int64_t k = lane; k < n; k += 32) {
            const double a = ar[k], b = ai[k];
            sr += (a * p_re[k] - b * p_im[k]);
            si += (a * p_im[k] + b * p_re[k]);
        }
        for (int o = 16; o > 0; o >>= 1) {
            sr += __shfl_down_sync(0xffffffffu, sr, o);
            si += __shfl_down_sync(0xffffffffu, si, o);
        }
        if (lane == 0) {
            q_re[row] = sr;
            q_im[row] = si;
        }
    }
    if (!do_adj) return;
    // A^H pt partials: column k accumulates conj(A[row][k]) pt[row] over the block's rows
    for (int64_t k = threadIdx.x; k < n; k += blockDim.x) {
        double sr = 0.0, si = 0.0;
        for (int rr = 0; rr < kDenseRows; rr++) {
            const int64_t row = r0 + rr;
            if (row >= n) break;
            const double a = are[row * n + k], b = aim[row * n + k];
            sr += (a * pt_re[row] + b * pt_im[row]);
            si += (a * pt_im[row] - b * pt_re[row]);
        }
        part_re[(int64_t)blockIdx.x * n + k] = sr;
        part_im[(int64_t)blockIdx.x * n + k] = si;
    }
}

__global__ void dense_adj_reduce_kernel(int64_t n, int64_t nblk, const double *__restrict__ part_re,
                                        const double *__restrict__ part_im, double *qt_re, double *qt_im)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        double sr = 0.0, si = 0.0;
        for (int64_t b = 0; b < nblk; b++) {
            sr += part_re[b * n + k];
            si += part_im[b * n + k];
        }
        qt_re[k] = sr;
        qt_im[k] = si;
    }
}

}  // namespace

int launch_eval(int64_t n, const double4_32a *pos, const double4_32a *nrm, const double *s_re, const double *s_im,
                int64_t m, const double *rx, double wave, double tau, int interior, int layer, double *u_re,
                double *u_im, cudaStream_t s)
{
    if (m <= 0) return HZ_OK;
    if (m > 0x7fffffffLL) {
        set_error("hz_eval: too many receivers");
        return HZ_ERR_ARG;
    }
    const double sg = interior == 1 ? -1.0 : 1.0;
    // four receivers a block when that still leaves every SM its two blocks
    const bool wide = m >= 8 * (int64_t)sm_count();
    auto f = layer == HZ_SINGLE_LAYER ? (wide ? eval_blocks<true, 4> : eval_blocks<true, 1>)
                                      : (wide ? eval_blocks<false, 4> : eval_blocks<false, 1>);
    return f(n, pos, nrm, s_re, s_im, m, rx, wave, tau, sg, u_re, u_im, s);
}

int launch_rhs(int64_t n, const double4_32a *pos, const double4_32a *nrm, const double *src, double wave, int kind,
               double *b_re, double *b_im, cudaStream_t s)
{
    if (n <= 0) return HZ_OK;
    long long b = (n + 255) / 256;
    if (b > 4096) b = 4096;
    rhs_kernel<<<(unsigned)b, 256, 0, s>>>(n, pos, nrm, src[0], src[1], src[2], wave, kind, b_re, b_im);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

int launch_plane_waves(int64_t n, const double4_32a *pos, const double4_32a *nrm, int ndir, const double *dirs,
                       double wave, int kind, double *b_re, double *b_im, cudaStream_t s)
{
    if (n <= 0) return HZ_OK;
    long long b = (n + 255) / 256;
    if (b > 256) b = 256;
    plane_wave_kernel<<<dim3((unsigned)b, (unsigned)ndir), 256, 0, s>>>(n, pos, nrm, ndir, dirs, wave, kind, b_re, b_im);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

int launch_slice(int axis, double c, int n2, double lo, double h2, double mask, int N, double H, double int_l,
                 const double *d, double *rx, unsigned char *keep, cudaStream_t s)
{
    const int64_t total = (int64_t)n2 * n2;
    long long b = (total + 255) / 256;
    if (b > 4096) b = 4096;
    slice_points_kernel<<<(unsigned)b, 256, 0, s>>>(axis, c, n2, lo, h2, mask, N, H, int_l, d, rx, keep);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

int launch_mask(int64_t m, const unsigned char *keep, double *u_re, double *u_im, cudaStream_t s)
{
    long long b = (m + 255) / 256;
    if (b > 4096) b = 4096;
    apply_mask_kernel<<<(unsigned)b, 256, 0, s>>>(m, keep, u_re, u_im);
    HZ_CHECK_LAUNCH();
    return HZ_OK;
}

size_t dense_partial_elems(int64_t n) { return (size_t)((n + kDenseRows - 1) / kDenseRows) * (size_t)n; }

int launch_dense(int64_t n, const double *are, const double *aim, const double *p_re, const double *p_im,
                 const double *pt_re, const double *pt_im, double *q_re, double *q_im, double *qt_re,
                 double *qt_im, double *part_re, double *part_im, cudaStream_t s)
{
    const int64_t nblk = (n + kDenseRows - 1) / kDenseRows;
    const int do_adj = (pt_re != nullptr), do_a = (p_re != nullptr);
    dense_rows_kernel<<<(unsigned)nblk, 256, 0, s>>>(n, are, aim, p_re, p_im, pt_re, pt_im, q_re, q_im, part_re,
                                                      part_im, do_a, do_adj);
    HZ_CHECK_LAUNCH();
    if (do_adj) {
        long long b = (n + 255) / 256;
        if (b > 4096) b = 4096;
        dense_adj_reduce_kernel<<<(unsigned)b, 256, 0, s>>>(n, nblk, part_re, part_im, qt_re, qt_im);
        HZ_CHECK_LAUNCH();
    }
    return HZ_OK;
}

}  // namespace hz
