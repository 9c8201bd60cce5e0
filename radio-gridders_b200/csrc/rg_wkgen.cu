// The w-kernel generator behind the C ABI: oversampled tap tables from a
// PSWF-tapered w-screen, in the layout the gridders index
// (kern_by_w[plane].data[(yf*ov + xf)*S*S + y*S + x], src/reference/grid.c:53-56).
//
// The reference has no generator of its own: its kernels come from the
// crocodile scripts as HDF5 files (README.md:25-26, loaded by
// src/common/hdf5.c:1362-1509).  This one is written from the mathematics:
//
//   s_w(l, m)  = A(l) A(m) exp(+2 pi i w (1 - sqrt(1 - l^2 - m^2)))
//                on an M x M screen, l = theta (i - M/2) / M,
//   K_w(p, q)  = 1/M^2 sum_ij s_w(l_i, m_j) exp(-2 pi i (p l_i + q m_j) / theta),
//   tap[plane][yf][xf][ty][tx] = K_w(tx - S/2 - xf/ov, ty - S/2 - yf/ov),
//
// A(x) = psi_0(c, 2x/theta), the zeroth prolate spheroidal wave function
// normalised to psi_0(0) = 1.  psi_0 is evaluated from its expansion in
// normalised Legendre polynomials, whose coefficients are the eigenvector of
// the smallest eigenvalue of a symmetric tridiagonal matrix (Bouwkamp 1947;
// Xiao, Rokhlin & Yarvin 2001); the eigenvalue is found by Sturm-sequence
// bisection and the eigenvector by inverse iteration (Wilkinson, The
// Algebraic Eigenvalue Problem, ch. 5 and 9).  The screen and the two
// non-uniform DFT sums run on the device in FP64, folded by the screen's
// symmetry into real matrix products.
#include <algorithm>
#include <cmath>
#include <vector>

#include "rg_internal.h"

namespace rg {
namespace {

// Tridiagonal matrix of the operator (1 - x^2) d2/dx2 - 2x d/dx - c^2 x^2 in
// the normalised even-degree Legendre basis sqrt(k + 1/2) P_k, k = 0, 2, ...
void pswf_matrix(double c, int nterms, std::vector<double> &d, std::vector<double> &e)
{
    d.resize(nterms);
    e.resize(nterms > 0 ? nterms - 1 : 0);
    const double c2 = c * c;
    for (int j = 0; j < nterms; j++) {
        const double k = 2.0 * j;
        d[j] = k * (k + 1) + c2 * (2 * k * (k + 1) - 1) / ((2 * k + 3) * (2 * k - 1));
        if (j + 1 < nterms) e[j] = c2 * (k + 1) * (k + 2) / ((2 * k + 3) * std::sqrt((2 * k + 1) * (2 * k + 5)));
    }
}

// Eigenvalues of the tridiagonal matrix below x (Sturm sequence of the LDL^T
// pivots).
int sturm_count(const std::vector<double> &d, const std::vector<double> &e, double x)
{
    int count = 0;
    double q = d[0] - x;
    if (q < 0) count++;
    for (size_t i = 1; i < d.size(); i++) {
        const double qq = q != 0.0 ? q : 1e-300;
        q = d[i] - x - e[i - 1] * e[i - 1] / qq;
        if (q < 0) count++;
    }
    return count;
}

// Solve (T - sigma I) y = b for tridiagonal T: elimination with partial pivoting,
// which fills one diagonal above the two.
void shifted_solve(const std::vector<double> &d, const std::vector<double> &e, double sigma,
                   const std::vector<double> &b, std::vector<double> &y)
{
    const int n = (int)d.size();
    std::vector<double> p0(n), p1(n, 0.0), p2(n, 0.0), r(b);
    for (int i = 0; i < n; i++) {
        p0[i] = d[i] - sigma;
        if (i + 1 < n) p1[i] = e[i];
    }
    for (int i = 0; i + 1 < n; i++) {
        double below = e[i];  // row i + 1: below, p0, p1 at columns i, i + 1, i + 2
        if (std::fabs(below) > std::fabs(p0[i])) {
            std::swap(below, p0[i]);
            std::swap(p0[i + 1], p1[i]);
            std::swap(p1[i + 1], p2[i]);
            std::swap(r[i], r[i + 1]);
        }
        if (p0[i] == 0.0) p0[i] = 1e-300;  // exactly singular: any scaled eigenvector will do
        const double f = below / p0[i];
        p0[i + 1] -= f * p1[i];
        p1[i + 1] -= f * p2[i];
        r[i + 1] -= f * r[i];
    }
    if (p0[n - 1] == 0.0) p0[n - 1] = 1e-300;
    y.assign(n, 0.0);
    for (int i = n - 1; i >= 0; i--) {
        double s = r[i];
        if (i + 1 < n) s -= p1[i] * y[i + 1];
        if (i + 2 < n) s -= p2[i] * y[i + 2];
        y[i] = s / p0[i];
    }
}

// Expansion coefficients of psi_0(c, .) (unnormalised, any sign).
std::vector<double> pswf_coefficients(double c)
{
    const int nterms = (int)(2 * c + 40);
    std::vector<double> d, e;
    pswf_matrix(c, nterms, d, e);
    // Gershgorin interval, then bisection for the smallest eigenvalue
    double lo = d[0], hi = d[0];
    for (int i = 0; i < nterms; i++) {
        const double r = (i > 0 ? std::fabs(e[i - 1]) : 0.0) + (i + 1 < nterms ? std::fabs(e[i]) : 0.0);
        lo = std::fmin(lo, d[i] - r);
        hi = std::fmax(hi, d[i] + r);
    }
    // to 1e-9 of the interval's scale: the next eigenvalue is about 4c away, so each
    // inverse iteration gains seven digits or more and six are plenty
    for (int it = 0; it < 200 && hi - lo > 1e-9 * std::fmax(1.0, std::fabs(lo) + std::fabs(hi)); it++) {
        const double mid = 0.5 * (lo + hi);
        if (sturm_count(d, e, mid) >= 1) hi = mid;
        else lo = mid;
    }
    const double lambda = 0.5 * (lo + hi);
    std::vector<double> x(nterms, 1.0), y;
    for (int it = 0; it < 6; it++) {
        shifted_solve(d, e, lambda, x, y);
        double nrm = 0.0;
        for (double v : y) nrm += v * v;
        nrm = std::sqrt(nrm);
        for (int i = 0; i < nterms; i++) x[i] = y[i] / nrm;
    }
    return x;
}

// psi_0(c, x) / psi_0(c, 0) from the coefficients at n points, by the Legendre
// recurrence, a block of points a degree at a time (the divisions go side by
// side). Nothing is allocated by n, and out may be x.
void pswf_values(const std::vector<double> &coef, const double *x, int64_t n, double *out)
{
    constexpr int B = 512;  // four arrays of 4 KB
    const int degrees = 2 * (int)coef.size() - 2;
    std::vector<double> scaled(coef.size());
    for (size_t j = 0; j < coef.size(); j++) scaled[j] = coef[j] * std::sqrt(2.0 * (double)j + 0.5);
    double at0 = scaled[0], q_prev = 1.0, q_cur = 0.0;  // the sum at x = 0; P_0 and P_1 there
    for (int deg = 1; deg < degrees; deg++) {
        const double q_next = (-(double)deg * q_prev) / (deg + 1);
        q_prev = q_cur;
        q_cur = q_next;
        if (deg % 2) at0 += scaled[(deg + 1) / 2] * q_cur;
    }
    double xb[B], p_prev[B], p_cur[B], sum[B];
    for (int64_t b = 0; b < n; b += B) {
        const int cnt = (int)std::min<int64_t>(B, n - b);
        for (int i = 0; i < cnt; i++) {
            xb[i] = p_cur[i] = x[b + i];
            p_prev[i] = 1.0;
            sum[i] = scaled[0];
        }
        for (int deg = 1; deg < degrees; deg++) {
            for (int i = 0; i < cnt; i++) {
                const double p_next = ((2 * deg + 1) * xb[i] * p_cur[i] - deg * p_prev[i]) / (deg + 1);
                p_prev[i] = p_cur[i];
                p_cur[i] = p_next;
            }
            if (deg % 2) {  // p_cur is the even degree deg + 1
                const double c = scaled[(deg + 1) / 2];
                for (int i = 0; i < cnt; i++) sum[i] += c * p_cur[i];
            }
        }
        for (int i = 0; i < cnt; i++) out[b + i] = sum[i] / at0;
    }
}

// The sums, folded. The screen is even in l and in m, so with i' = i - M/2 a
// row's sum over i' = -M/2 .. M/2 - 1 is
//   T(q) = s(0) + sum_{0 < i' < M/2} s(i') 2 cos(2 pi off_q i' / M) + s(-M/2) exp(pi i off_q),
// real factors but for the unpaired edge, which takes two real columns of its
// own: both sums are real matrix products of depth K = M/2 + 2 with one factor
// matrix cq[k][q] = {1, 2 cos(2 pi off_q k / M), .., cos(pi off_q), sin(pi off_q)},
// over M/2 + 2 rows j' in place of M. Off q = f*S + t (sub-cell shift f, tap t):
// off_q = t - S/2 - f/ov.
//
// The products run on the FP64 tensor pipe (mma m8n8k4, 37 TFLOP/s measured, the
// rate of the FP64 multiply-add pipe, with an eighth of its instructions and
// operand reads): 64 x 64 tiles, K in shared memory 68 deep (all of the default
// screen's 66), one 32 x 32 block a warp. 401 planes of 16 x 16 taps, 8 x
// oversampled (2.6 GFLOP): 38 + 80 us, two thirds of that pipe's rate; copies and
// stores by running pointers and offsets in place of an index for each element
// took them there from 41 + 93 us, at half the instructions. Persistent CTAs
// with the factors resident and the other operand double-buffered (two CTAs an
// SM) take 43 + 84, four or five CTAs an SM with shallower tiles 37..38 +
// 78..85. The call: 4831 -> 180 us (the sums as plain loops took 3387 and 1152).

// a[k][row], row = (plane K + j') 2 + part: the screen's rows as the left
// factor. k < M/2: s(i' = k); k = M/2, M/2 + 1: the edge i' = -M/2 times the
// edge factors' real and imaginary parts. The rows j' run the same way, the
// edge row twice, so the second product takes them as they come.
// A thread takes one pixel of 8 planes, whose root and taper they share: 13 us
// for 401 planes of 65 x 65 pixels, 20..24 us with an element a thread (bound by
// instructions issued, 346 -> 135 an element).
constexpr int kScreenPlanes = 8;

__global__ void wscreen_kernel(const double *__restrict__ w_planes, int planes, const double *__restrict__ taper,
                               int M, double theta, double2 *__restrict__ a)
{
    const int h = M / 2, J = h + 1, k = blockIdx.y;
    const int64_t pairs = (int64_t)planes * (h + 2);
    const unsigned groups = (planes + kScreenPlanes - 1) / kScreenPlanes, total = groups * J;  // below 2^25
    for (unsigned n = blockIdx.x * blockDim.x + threadIdx.x; n < total; n += gridDim.x * blockDim.x) {
        const int j = n % J;
        const int ic = k < h ? k : -h, jc = j < h ? j : -h;
        const double l = theta * (double)ic / M, m = theta * (double)jc / M;
        const double one_minus_n = 1.0 - sqrt(1.0 - (l * l + m * m));
        const double t = taper[ic + h] * taper[jc + h];
        for (int p = n / J; p < planes; p += groups) {
            double sn, cs;
            sincospi(2.0 * w_planes[p] * one_minus_n, &sn, &cs);
            const double re = t * cs, im = t * sn;
            double2 *at = a + (int64_t)k * pairs + (int64_t)p * (h + 2) + j;
            at[0] = make_double2(re, im);
            if (k == h) at[pairs] = make_double2(-im, re);
            if (j == h) {
                at[1] = make_double2(-im, re);
                if (k == h) at[pairs + 1] = make_double2(-re, -im);
            }
        }
    }
}

__global__ void wkgen_factors_kernel(int S, int ov, int M, double *__restrict__ cq)
{
    const int Q = ov * S, h = M / 2, total = Q * (h + 2);
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < total; n += gridDim.x * blockDim.x) {
        const int q = n % Q, k = n / Q;
        const double off = (double)(q % S - S / 2) - (double)(q / S) / ov;
        cq[n] = k == 0 ? 1.0 : k < h ? 2.0 * cospi(2.0 * off * (double)k / M) : k == h ? cospi(off) : sinpi(off);
    }
}

constexpr int kGemmTile = 64, kGemmDepth = 68;
constexpr int kGemmStride = kGemmTile + 4;  // 4 mod 16 doubles: a fragment's 4 k x 8 rows fall on distinct banks
constexpr int kGemmThreads = 128;

__device__ __forceinline__ void mma_f64(double2 &c, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c.x), "+d"(c.y)
                 : "d"(a), "d"(b));
}

// 16 bytes to shared memory, or zeros where bytes is 0
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
                 "l"(gmem), "r"(bytes)
                 : "memory");
}

// A lane's two neighbouring columns of an operand: element of depth k at
// p[k * stride], and nothing where the columns lie past the edge (p then
// points at the operand's first columns and is not read).
struct Operand {
    const double *p;
    int64_t stride;
    int bytes;
    __device__ Operand(const double *base, int64_t off, int64_t stride_, bool on)
        : p(base + (on ? off : 0)), stride(stride_), bytes(on ? 16 : 0)
    {
    }
};

// One warp's 32 x 32 block of a 64 x 64 tile: rows row0 + 8 i, columns col(j) +
// 0..7; c[i][j] holds row lane / 4, columns 2 (lane % 4) and the next. A warp
// copies one depth of both operands at a time.
template <class Col>
__device__ __forceinline__ void gemm_tile(double2 (&c)[4][4], double *sa, double *sb, int K, Operand a, Operand b,
                                          int row0, Col col)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int W = kGemmThreads / 32;
    a.p += warp * a.stride, b.p += warp * b.stride;
    for (int k0 = 0; k0 < K; k0 += kGemmDepth) {
        const int live = min(kGemmDepth, K - k0), depth = (live + 3) & ~3;
        __syncthreads();
        double *da = sa + warp * kGemmStride + 2 * lane, *db = sb + warp * kGemmStride + 2 * lane;
        int k = warp;
#pragma unroll 4
        for (; k < live; k += W) {
            cp_async16(da, a.p, a.bytes);
            cp_async16(db, b.p, b.bytes);
            a.p += W * a.stride, b.p += W * b.stride;
            da += W * kGemmStride, db += W * kGemmStride;
        }
        if (k < depth) {  // less than W depths of zeros
            *(double2 *)da = make_double2(0.0, 0.0);
            *(double2 *)db = make_double2(0.0, 0.0);
        }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const double *pa = sa + (lane & 3) * kGemmStride + row0 + (lane >> 2);
        const double *pb = sb + (lane & 3) * kGemmStride + (lane >> 2);
        for (int k = 0; k < depth; k += 4) {
            double fa[4], fb[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                fa[i] = pa[k * kGemmStride + 8 * i];
                fb[i] = pb[k * kGemmStride + col(i)];
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma_f64(c[i][j], fa[i], fb[j]);
        }
    }
}

// T[row][qx] = sum_k a[k][row] cq[k][qx]
__global__ void __launch_bounds__(kGemmThreads) wkgen_rows_kernel(const double *__restrict__ a,
                                                                  const double *__restrict__ cq, int64_t rows, int K,
                                                                  int Q, double *__restrict__ T)
{
    extern __shared__ double gemm_sm[];
    const int64_t r0 = (int64_t)blockIdx.x * kGemmTile;
    const int q0 = blockIdx.y * kGemmTile;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = (warp >> 1) * 32, col0 = (warp & 1) * 32;
    double2 c[4][4] = {};
    gemm_tile(
        c, gemm_sm, gemm_sm + kGemmDepth * kGemmStride, K,
        Operand(a, r0 + 2 * lane, rows, r0 + 2 * lane < rows), Operand(cq, q0 + 2 * lane, Q, q0 + 2 * lane < Q), row0,
        [&](int j) { return col0 + 8 * j; });
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int64_t r = r0 + row0 + 8 * i + (lane >> 2);
            const int q = q0 + col0 + 8 * j + 2 * (lane & 3);
            if (r < rows && q < Q) {  // Q is even
                *(double2 *)(T + r * Q + q) = c[i][j];
            }
        }
}

// data[plane][yf][xf][ty][tx] = 1/M^2 sum_k cq[k][qy] T[plane][k][part][qx],
// qy = yf*S + ty, qx = xf*S + tx: 64 qy x 32 qx a tile, the imaginary parts
// beside the real ones.
__global__ void __launch_bounds__(kGemmThreads) wkgen_cols_kernel(const double *__restrict__ T,
                                                                  const double *__restrict__ cq, int M, int S, int ov,
                                                                  double2 *__restrict__ out)
{
    extern __shared__ double gemm_sm[];
    const int Q = ov * S, h = M / 2, ytiles = (Q + kGemmTile - 1) / kGemmTile;
    const int p = blockIdx.x / ytiles, y0 = (blockIdx.x % ytiles) * kGemmTile, x0 = blockIdx.y * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = (warp >> 1) * 32, col0 = (warp & 1) * 16;
    const double *Tp = T + (int64_t)p * (h + 2) * 2 * Q;
    double2 c[4][4] = {};
    const int bx = x0 + (2 * lane & 31);
    gemm_tile(
        c, gemm_sm, gemm_sm + kGemmDepth * kGemmStride, h + 2,
        Operand(cq, y0 + 2 * lane, Q, y0 + 2 * lane < Q), Operand(Tp, (lane >> 4) * Q + bx, 2 * Q, bx < Q), row0,
        [&](int j) { return col0 + 8 * (j & 1) + 32 * (j >> 1); });
    const double inv = 1.0 / ((double)M * M);
    double2 *o = out + (int64_t)p * Q * Q;
    int ox[2];  // S is even: a lane's two taps are neighbours
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int qx = x0 + col0 + 8 * j + 2 * (lane & 3), xf = qx / S;
        ox[j] = qx < Q ? xf * S * S + qx - xf * S : -1;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int qy = y0 + row0 + 8 * i + (lane >> 2), yf = qy / S;
        const int64_t oy = (int64_t)yf * Q * S + (qy - yf * S) * S;
#pragma unroll
        for (int j = 0; j < 2; j++)
            if (qy < Q && ox[j] >= 0) {
                o[oy + ox[j]] = make_double2(c[i][j].x * inv, c[i][j + 2].x * inv);
                o[oy + ox[j] + 1] = make_double2(c[i][j].y * inv, c[i][j + 2].y * inv);
            }
    }
}

}  // namespace
}  // namespace rg

using namespace rg;

extern "C" {

rg_status rg_pswf0(double c, const double *x, int64_t n, double *out)
{
    if (n < 0 || (n > 0 && (!x || !out))) return fail(RG_ERR_INVALID_ARGUMENT, "x and out must be non-NULL");
    if (!(c > 0.0) || !std::isfinite(c) || c > 1000.0) return fail(RG_ERR_INVALID_ARGUMENT, "c must be in (0, 1000]");
    const std::vector<double> coef = pswf_coefficients(c);
    for (int64_t k = 0; k < n; k++)
        if (!(std::fabs(x[k]) <= 1.0)) return fail(RG_ERR_INVALID_ARGUMENT, "x must lie in [-1, 1]");
    pswf_values(coef, x, n, out);
    return RG_OK;
}

rg_status rg_wkern_generate(rg_context *ctx, double theta, const double *w_planes, int plane_count, int size,
                            int oversampling, double c, int screen_pixels, double *data_out)
{
    if (!ctx || !w_planes || !data_out) return fail(RG_ERR_INVALID_ARGUMENT, "ctx, w_planes and data_out must be non-NULL");
    if (!(theta > 0.0) || !(theta < 2.0)) return fail(RG_ERR_INVALID_ARGUMENT, "theta must be in (0, 2)");
    if (plane_count < 1 || plane_count > 65536) return fail(RG_ERR_INVALID_ARGUMENT, "plane_count must be in [1, 65536]");
    if (size < 2 || size > 64 || size % 2) return fail(RG_ERR_INVALID_ARGUMENT, "size must be even, in [2, 64]");
    if (oversampling < 1 || oversampling > 128) return fail(RG_ERR_INVALID_ARGUMENT, "oversampling must be in [1, 128]");
    const int M = screen_pixels > 0 ? screen_pixels : 128;
    if (M < 4 || M > 4096 || M % 2) return fail(RG_ERR_INVALID_ARGUMENT, "screen_pixels must be even, in [4, 4096]");
    const double cc = c > 0.0 ? c : M_PI * (size - 2) / 2.0;
    if (!std::isfinite(cc) || cc > 1000.0) return fail(RG_ERR_INVALID_ARGUMENT, "c must be finite and <= 1000");
    for (int p = 0; p < plane_count; p++)
        if (!std::isfinite(w_planes[p])) return fail(RG_ERR_INVALID_ARGUMENT, "w planes must be finite");
    // the screen must stay inside the unit circle: (theta/2)^2 * 2 < 1
    RG_CUDA(cudaSetDevice(ctx->device));
    begin_call(ctx);
    const std::vector<double> coef = pswf_coefficients(cc);
    // the taper is even, bit for bit: half of it computed, the rest mirrored
    std::vector<double> taper(M), half(M / 2 + 1), at(M / 2 + 1);
    for (int i = 0; i <= M / 2; i++) at[i] = 2.0 * (double)i / M;
    pswf_values(coef, at.data(), M / 2 + 1, half.data());
    for (int i = 0; i < M; i++) taper[i] = half[i < M / 2 ? M / 2 - i : i - M / 2];
    const int S = size, ov = oversampling, Q = ov * S;
    const int64_t ntaps = (int64_t)plane_count * Q * Q;
    const int J = M / 2 + 1, K = M / 2 + 2;
    const int64_t rows = (int64_t)plane_count * K * 2;
    void *d_w, *d_taper, *d_s, *d_cq, *d_T;
    RG_CHECK(scratch(ctx, "wkgen_w", sizeof(double) * plane_count, &d_w));
    RG_CHECK(scratch(ctx, "wkgen_taper", sizeof(double) * M, &d_taper));
    RG_CHECK(scratch(ctx, "wkgen_screen", sizeof(double) * (size_t)rows * K, &d_s));
    RG_CHECK(scratch(ctx, "wkgen_factors", sizeof(double) * (size_t)Q * K, &d_cq));
    RG_CHECK(scratch(ctx, "wkgen_rows", sizeof(double) * (size_t)rows * Q, &d_T));
    OutView ov_out;
    RG_CHECK(out_view(ctx, data_out, sizeof(double2) * (size_t)ntaps, "wkgen_out", false, &ov_out));
    RG_CUDA(cudaMemcpyAsync(d_w, w_planes, sizeof(double) * plane_count, cudaMemcpyHostToDevice, ctx->stream));
    RG_CUDA(cudaMemcpyAsync(d_taper, taper.data(), sizeof(double) * M, cudaMemcpyHostToDevice, ctx->stream));
    auto blocks = [](int64_t n) { return (unsigned)std::min<int64_t>((n + 255) / 256, 148 * 32); };
    const int groups = (plane_count + kScreenPlanes - 1) / kScreenPlanes;
    wscreen_kernel<<<dim3(blocks((int64_t)groups * J), J), 256, 0, ctx->stream>>>(
        (const double *)d_w, plane_count, (const double *)d_taper, M, theta, (double2 *)d_s);
    wkgen_factors_kernel<<<blocks((int64_t)Q * K), 256, 0, ctx->stream>>>(S, ov, M, (double *)d_cq);
    const int smem = 2 * kGemmDepth * kGemmStride * (int)sizeof(double);
    cudaFuncSetAttribute(wkgen_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(wkgen_cols_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const unsigned tiles = (unsigned)((Q + kGemmTile - 1) / kGemmTile);
    wkgen_rows_kernel<<<dim3((unsigned)((rows + kGemmTile - 1) / kGemmTile), tiles), kGemmThreads, smem, ctx->stream>>>(
        (const double *)d_s, (const double *)d_cq, rows, K, Q, (double *)d_T);
    wkgen_cols_kernel<<<dim3((unsigned)plane_count * tiles, (unsigned)((Q + 31) / 32)), kGemmThreads, smem,
                        ctx->stream>>>((const double *)d_T, (const double *)d_cq, M, S, ov, (double2 *)ov_out.dev);
    ctx->launches += 4;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "w-kernel generator launch");
    RG_CHECK(finish_out(ctx, ov_out));
    RG_CUDA(cudaStreamSynchronize(ctx->stream));
    return RG_OK;
}

}  // extern "C"
