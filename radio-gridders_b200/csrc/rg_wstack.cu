// W-stacking predict (degridding): model visibilities of point sources from
// w-stacked FFTs of the sky and a separable 3-D de-convolution — the
// reference's wstack_predict (src/wstack/predict.cpp:396-562) and its CUDA
// version wstack_predict_cu_3D (src/wstack/predict.cu:808-1081), FP64.
//
//   1. sources snapped to the image grid (N = floor(theta lambda) pixels of
//      1/lambda) inside a grid padded to G = N round(0.5/x0) pixels, each
//      divided by the grid correction corr_lm(du l) corr_lm(du m) corr_n(dw n)
//      (predict.cpp:187-245);
//   2. plane p = quadrant-swapped FFT (sign -1) of the swapped sky times the
//      Fresnel pattern exp(2 pi i dw (1 - sqrt(1 - l^2 - m^2))) raised to
//      p - floor(planes/2) (predict.cpp:466-491: the reference steps the sky by
//      one more power per plane; here each plane's power is formed from the
//      exact phase, planes*dw*ph reduced modulo one turn in FP64);
//   3. per visibility, sum over support_w x support_uv^2 taps of the stack
//      weighted by conv_w x conv_uv x conv_uv at the visibility's sub-cell
//      offsets (src/wstack/wstack_common.h:423-484).
//
// Two ways to step 3, with the same results to FP64 rounding:
//   through the stack (many sources): the rows that hold sources are
//     transformed, then every column of every plane into the stack in HBM
//     (planes x G^2 x 16 bytes), then one warp per visibility gathers its taps;
//   direct (few sources): a tap of the stack is a sum of one phasor per source,
//     separable in u, v and w, so a visibility is a sum over the sources of
//     three short sums of its kernel weights times the source's phasor powers.
//     No stack is made. wstack_use_direct has the rule.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "k_fft64.cuh"

namespace rg {
namespace {

// A quantised, grid-corrected source: its row and column in the swapped
// (fft-shifted) G x G sky, its place in the list of used rows, its pixel in the
// unpadded N x N image (for the Fresnel phase) and its value.
struct SkyEntry {
    int row, col, slot, x, y, pad;
    double val;
};

__device__ __forceinline__ double fresnel_turns(const SkyEntry &s, int N, double theta, double dw)
{
    const double l = theta * ((double)s.x - N / 2) / N;
    const double m = theta * ((double)s.y - N / 2) / N;
    return dw * (1.0 - sqrt(1.0 - l * l - m * m));
}

// exp(2 pi i k ph), the product reduced modulo one turn
__device__ __forceinline__ double2 fresnel_power(double ph, int k)
{
    const double turns = (double)k * ph;
    double sn, cs;
    sincospi(2.0 * (turns - rint(turns)), &sn, &cs);  // one turn removed exactly
    return make_double2(cs, sn);
}

// rows[p][slot][col]: plane p of the used rows, value * exp(2 pi i (t0 + p) ph)
__global__ void wstack_scatter_kernel(const SkyEntry *__restrict__ sky, int nsrc, int planes, int t0, int N, int G,
                                      int nrows, double theta, double dw, double2 *__restrict__ rows)
{
    const int64_t total = (int64_t)nsrc * planes;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x) {
        const SkyEntry e = sky[k % nsrc];
        const int p = (int)(k / nsrc);
        const double2 z = fresnel_power(fresnel_turns(e, N, theta, dw), t0 + p);
        rows[((int64_t)p * nrows + e.slot) * G + e.col] = make_double2(e.val * z.x, e.val * z.y);
    }
}

// Columns of the stack from the used rows' transforms (slot_of_row: -1 for a
// row without sources), stored at their shifted places.
struct LdSkyCol {
    const double2 *rows;
    const int *slot_of_row;
    int G, nrows;
    __device__ double2 operator()(int arr, int line, int n) const
    {
        const int slot = __ldg(slot_of_row + n);
        return slot < 0 ? make_double2(0.0, 0.0) : rows[((int64_t)arr * nrows + slot) * G + line];
    }
};
struct StStackCol {
    double2 *stack;
    int G;
    __device__ void operator()(int arr, int line, int n, double2 v) const
    {
        const int y = n < G / 2 ? n + G / 2 : n - G / 2, x = line < G / 2 ? line + G / 2 : line - G / 2;
        stack[((int64_t)arr * G + y) * G + x] = v;
    }
};

// The geometry and kernel tables of the de-convolution.
struct DegridGeom {
    double du, dw;
    int N, G, planes, suv, ovuv, sw, ovw;
    const double *conv_uv, *conv_w;
};

// A visibility's first tap (column, row, plane) and the rows of the kernel
// tables at its sub-cell offsets (src/wstack/wstack_common.h:423-484);
// otherwise the error bit.
struct DegridCell {
    int x, y, p;
    const double *gu, *gv, *gw;
};
__device__ __forceinline__ unsigned degrid_cell(const DegridGeom &g, double uu, double vv, double ww, DegridCell &c)
{
    if (!isfinite(uu) || !isfinite(vv) || !isfinite(ww)) return DERR_NONFINITE;
    const double cu = ceil(uu / g.du), cv = ceil(vv / g.du), cw = ceil(ww / g.dw);
    if (fabs(cu) > 1e9 || fabs(cv) > 1e9 || fabs(cw) > 1e9) return DERR_GRID_RANGE;  // far outside any stack
    const double flu = uu - cu * g.du, flv = vv - cv * g.du, flw = ww - cw * g.dw;
    const int ovu = (int)floor(fabs(flu) / g.du * g.ovuv);
    const int ovv = (int)floor(fabs(flv) / g.du * g.ovuv);
    const int ovw = (int)floor(fabs(flw) / g.dw * g.ovw);
    const int64_t x = (int64_t)cu + g.N - g.suv / 2, y = (int64_t)cv + g.N - g.suv / 2;
    const int64_t p = (int64_t)cw + g.planes / 2 - g.sw / 2;
    if (x < 0 || x + g.suv > g.G || y < 0 || y + g.suv > g.G || p < 0 || p + g.sw > g.planes || ovu >= g.ovuv ||
        ovv >= g.ovuv || ovw >= g.ovw)
        return DERR_GRID_RANGE;
    c.x = (int)x;
    c.y = (int)y;
    c.p = (int)p;
    c.gu = g.conv_uv + (int64_t)g.suv * ovu;
    c.gv = g.conv_uv + (int64_t)g.suv * ovv;
    c.gw = g.conv_w + (int64_t)g.sw * ovw;
    return 0;
}

// One warp per visibility: lanes over the support_uv^2 (u, v) taps, planes in
// turn, then a warp sum.
__global__ void wstack_degrid_kernel(const double2 *__restrict__ stack, const double *__restrict__ u,
                                     const double *__restrict__ v, const double *__restrict__ w, int64_t nvis,
                                     DegridGeom g, double2 *__restrict__ out, unsigned *err)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < nvis; i += warps) {
        DegridCell c;
        const unsigned e = degrid_cell(g, u[i], v[i], w[i], c);
        if (e) {
            if (lane == 0) {
                out[i] = make_double2(0.0, 0.0);
                atomicOr(err, e);
            }
            continue;
        }
        double2 acc = make_double2(0.0, 0.0);
        for (int a = 0; a < g.sw; a++) {
            const double gw = c.gw[a];
            const double2 *plane = stack + (int64_t)(c.p + a) * g.G * g.G;
            for (int t = lane; t < g.suv * g.suv; t += 32) {
                const int ty = t / g.suv, tx = t % g.suv;
                const double k = gw * c.gv[ty] * c.gu[tx];
                const double2 z = plane[(int64_t)(c.y + ty) * g.G + c.x + tx];
                acc.x = fma(z.x, k, acc.x);
                acc.y = fma(z.y, k, acc.y);
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
        }
        if (lane == 0) out[i] = acc;
    }
}

// Per source: the powers of its u, v and w phasors that a footprint's taps
// step through, pw[s][SU | SU | SW] (u, v: exp(-2 pi i t col / G) from the root
// table, w: exp(2 pi i a ph)), and its value times its phase on every plane,
// base[s][p].
template <int SU, int SW>
__global__ void wstack_source_kernel(const SkyEntry *__restrict__ sky, int nsrc, int planes, int t0, int N, int G,
                                     double theta, double dw, const double2 *__restrict__ roots,
                                     double2 *__restrict__ pw, double2 *__restrict__ base)
{
    const int s = blockIdx.x;
    const SkyEntry e = sky[s];
    const double ph = fresnel_turns(e, N, theta, dw);
    for (int k = threadIdx.x; k < 2 * SU + SW + planes; k += blockDim.x) {
        if (k < 2 * SU) {
            const int t = k % SU;
            pw[(int64_t)s * (2 * SU + SW) + k] = roots[(t * (k < SU ? e.col : e.row)) % G];
        } else if (k < 2 * SU + SW) {
            pw[(int64_t)s * (2 * SU + SW) + k] = fresnel_power(ph, k - 2 * SU);
        } else {
            const int p = k - 2 * SU - SW;
            const double2 z = fresnel_power(ph, t0 + p);
            base[(int64_t)s * planes + p] = make_double2(e.val * z.x, e.val * z.y);
        }
    }
}

__device__ __forceinline__ double2 zmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// Direct predict: V visibilities a thread, the sources in turn, their powers
// staged through shared memory. Supports below SU and SW have zero weights.
// Bound by the FP64 pipe (2 (2 SU + SW) + 18 multiply-adds a source and
// visibility) and, close behind, by shared memory, whose broadcast reads two
// visibilities a thread share. 50 sources and 200,000 visibilities
// (supports 8, 8, 6; G = 2048, 15 planes): 88 us with its set-up, the FP64
// pipe busy for half of its cycles (782 CTAs in two rounds of 444; 400 sources
// run at 0.53 of its rate); the whole call 5450 -> 138 us.
constexpr int kDirectThreads = 128, kDirectSources = 32;

template <int SU, int SW, int V>
__global__ void __launch_bounds__(kDirectThreads) wstack_direct_kernel(
    const double *__restrict__ u, const double *__restrict__ v, const double *__restrict__ w, int64_t nvis,
    DegridGeom g, const SkyEntry *__restrict__ sky, int nsrc, const double2 *__restrict__ pw,
    const double2 *__restrict__ base, const double2 *__restrict__ roots, unsigned magic, double2 *__restrict__ out,
    unsigned *err)
{
    constexpr int P = 2 * SU + SW;
    __shared__ double2 sp[kDirectSources][P];
    __shared__ int2 spos[kDirectSources];
    double gu[V][SU], gv[V][SU], gw[V][SW];
    unsigned x0[V], y0[V];
    int p0[V];
    double2 acc[V];
    const int64_t first = (int64_t)blockIdx.x * (kDirectThreads * V) + threadIdx.x;
    unsigned bad = 0, refused = 0;  // refused: the visibilities with no taps in the stack
    for (int q = 0; q < V; q++) {
        const int64_t i = first + q * kDirectThreads;
        DegridCell c;
        const unsigned e = i < nvis ? degrid_cell(g, u[i], v[i], w[i], c) : DERR_GRID_RANGE;
        const bool ok = e == 0;
        if (i < nvis) bad |= e;
        if (!ok) refused |= 1u << q;
#pragma unroll
        for (int t = 0; t < SU; t++) {
            gu[q][t] = ok && t < g.suv ? c.gu[t] : 0.0;
            gv[q][t] = ok && t < g.suv ? c.gv[t] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < SW; t++) gw[q][t] = ok && t < g.sw ? c.gw[t] : 0.0;
        // frequency indices of the first tap in the unshifted transform
        x0[q] = ok ? (c.x + g.G / 2) % g.G : 0;
        y0[q] = ok ? (c.y + g.G / 2) % g.G : 0;
        p0[q] = ok ? c.p : 0;
        acc[q] = make_double2(0.0, 0.0);
    }
    if (bad) atomicOr(err, bad);
    for (int s0 = 0; s0 < nsrc; s0 += kDirectSources) {
        const int cnt = min(kDirectSources, nsrc - s0);
        __syncthreads();
        for (int k = threadIdx.x; k < cnt * P; k += kDirectThreads) sp[0][k] = pw[(int64_t)s0 * P + k];
        for (int k = threadIdx.x; k < cnt; k += kDirectThreads) spos[k] = make_int2(sky[s0 + k].col, sky[s0 + k].row);
        __syncthreads();
        for (int s = 0; s < cnt; s++) {
            const int2 pos = spos[s];
            double2 b[V], r[V], su[V], sv[V], sz[V];
#pragma unroll
            for (int q = 0; q < V; q++) {
                // exp(-2 pi i (x0 col + y0 row) / G), the index (below 2^25) modulo G
                unsigned k = x0[q] * pos.x + y0[q] * pos.y;
                k -= __umulhi(k, magic) * (unsigned)g.G;
                k = min(k, k - (unsigned)g.G);  // the estimate is at most one low
                r[q] = __ldg(roots + k);
                b[q] = __ldg(base + (int64_t)(s0 + s) * g.planes + p0[q]);
                su[q] = sv[q] = sz[q] = make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int t = 0; t < SU; t++) {
                const double2 a = sp[s][t], c = sp[s][SU + t];
#pragma unroll
                for (int q = 0; q < V; q++) {
                    su[q] = make_double2(fma(gu[q][t], a.x, su[q].x), fma(gu[q][t], a.y, su[q].y));
                    sv[q] = make_double2(fma(gv[q][t], c.x, sv[q].x), fma(gv[q][t], c.y, sv[q].y));
                }
            }
#pragma unroll
            for (int t = 0; t < SW; t++) {
                const double2 a = sp[s][2 * SU + t];
#pragma unroll
                for (int q = 0; q < V; q++)
                    sz[q] = make_double2(fma(gw[q][t], a.x, sz[q].x), fma(gw[q][t], a.y, sz[q].y));
            }
#pragma unroll
            for (int q = 0; q < V; q++) {
                const double2 z = zmul(zmul(zmul(su[q], sv[q]), sz[q]), r[q]);
                acc[q].x = fma(z.x, b[q].x, fma(-z.y, b[q].y, acc[q].x));
                acc[q].y = fma(z.x, b[q].y, fma(z.y, b[q].x, acc[q].y));
            }
        }
    }
    for (int q = 0; q < V; q++) {
        const int64_t i = first + q * kDirectThreads;
        // zero also where a source's value is infinite and the sum is not a number
        if (i < nvis) out[i] = refused >> q & 1 ? make_double2(0.0, 0.0) : acc[q];
    }
}

template <int SU, int SW, int V>
void launch_direct(rg_context *ctx, const double *u, const double *v, const double *w, int64_t nvis, const DegridGeom &g,
                   const SkyEntry *sky, int nsrc, int t0, double theta, const double2 *roots, double2 *pw,
                   double2 *base, double2 *out, unsigned *err)
{
    if (nsrc > 0)
        wstack_source_kernel<SU, SW><<<nsrc, 64, 0, ctx->stream>>>(sky, nsrc, g.planes, t0, g.N, g.G, theta, g.dw,
                                                                   roots, pw, base);
    const unsigned magic = (unsigned)((1ull << 32) / (unsigned)g.G);
    const int64_t blocks = (nvis + kDirectThreads * V - 1) / (kDirectThreads * V);
    wstack_direct_kernel<SU, SW, V><<<(unsigned)blocks, kDirectThreads, 0, ctx->stream>>>(
        u, v, w, nvis, g, sky, nsrc, pw, base, roots, magic, out, err);
}

rg_status check_sepkern(const rg_sepkern *k, const char *name)
{
    if (!k || !k->data) return fail(RG_ERR_INVALID_ARGUMENT, std::string(name) + " is NULL");
    if (k->size < 1 || k->oversampling < 1 || (int64_t)k->size * k->oversampling > (1 << 26))
        return fail(RG_ERR_INVALID_ARGUMENT, std::string(name) + ": bad size or oversampling");
    return RG_OK;
}

// A table the host reads: the caller's memory, or a copy of it in `hold` when
// it lies on the device.
rg_status host_table(const rg_sepkern *k, std::vector<double> &hold, const double **out)
{
    *out = k->data;
    if (!is_device_pointer(k->data)) return RG_OK;
    hold.resize((size_t)k->size * k->oversampling);
    RG_CUDA(cudaMemcpy(hold.data(), k->data, sizeof(double) * hold.size(), cudaMemcpyDefault));
    *out = hold.data();
    return RG_OK;
}

// Direct or through the stack, whichever the measured rates make shorter.
// Direct: 0.103 ps a source, visibility and multiply-add (512 us for 400
// sources x 200,000 visibilities at supports 8, 8, 6), but 0.37 us a source at
// least, the time of one CTA's step, when the visibilities are too few to fill
// the device. Stack: 23 ps a cell and plane (1444 us for 15 planes of 2048 x
// 2048 cells), 106 ps where G needs Bluestein's algorithm (6747 us at 2060), and
// 5 ps a tap (383 us for 200,000 x 384). 50 sources and 200,000 visibilities:
// 88 us against 1.8 ms; 20,000 sources: 26 ms against 1.8 ms.
bool wstack_use_direct(int64_t nvis, int nsrc, int planes, int G, int suv, int sw)
{
    if (suv > 16 || sw > 16) return false;
    const bool wide = suv > 8 || sw > 8;
    const double fma = 2.0 * (wide ? 48 : 16 + (sw <= 6 ? 6 : 8)) + 18;
    const double direct = nsrc * std::max((double)nvis * fma * 0.103e-12, 0.37e-6);
    const double cell = fft64_smooth(G) ? 23e-12 : 106e-12;
    const double stack = (double)planes * G * G * cell + (double)nvis * suv * suv * sw * 5e-12;
    return direct <= stack;
}

}  // namespace
}  // namespace rg

using namespace rg;

extern "C" rg_status rg_wstack_predict(rg_context *ctx, double theta, double lambda, const double *points,
                                       int npoints, const double *u, const double *v, const double *w,
                                       int64_t nvis, double du, double dw, double x0, const rg_sepkern *conv_uv,
                                       const rg_sepkern *conv_w, const rg_sepkern *corr_lm,
                                       const rg_sepkern *corr_n, double *vis_out)
{
    if (!ctx || (npoints > 0 && !points) || (nvis > 0 && (!u || !v || !w || !vis_out)))
        return fail(RG_ERR_INVALID_ARGUMENT, "NULL argument");
    if (npoints < 0 || nvis < 0) return fail(RG_ERR_INVALID_ARGUMENT, "negative counts");
    if (!(theta > 0.0 && theta < 1.0) || !(lambda > 0.0) || !std::isfinite(lambda))
        return fail(RG_ERR_INVALID_ARGUMENT, "theta must be in (0, 1) and lambda > 0");
    if (!(du > 0.0) || !(dw > 0.0) || !std::isfinite(du) || !std::isfinite(dw))
        return fail(RG_ERR_INVALID_ARGUMENT, "du and dw must be finite and > 0");
    RG_CHECK(check_sepkern(conv_uv, "conv_uv"));
    RG_CHECK(check_sepkern(conv_w, "conv_w"));
    RG_CHECK(check_sepkern(corr_lm, "corr_lm"));
    RG_CHECK(check_sepkern(corr_n, "corr_n"));
    // the padded grid: the reference's round(0.5 / x0) (predict.cpp:410)
    if (!(x0 > 0.0 && x0 < 0.5)) return fail(RG_ERR_INVALID_ARGUMENT, "x0 must be in (0, 0.5)");
    const double x0ih = std::round(0.5 / x0);
    if (std::fabs(0.5 / x0 - x0ih) > 1e-9)
        return fail(RG_ERR_UNSUPPORTED, "0.5 / x0 must be an integer (the padding factor)");
    const int N = (int)std::floor(theta * lambda);
    const int G = (int)(x0ih * N);
    if (N < 2 || N % 2) return fail(RG_ERR_UNSUPPORTED, "floor(theta * lambda) must be even and >= 2");
    if (!fft64_any_supported(G)) return fail(RG_ERR_UNSUPPORTED, "the padded grid must be at most 4096 pixels");
    const int suv = conv_uv->size, sw = conv_w->size;
    const double max_w = std::sin(theta / 2) * std::sqrt(2.0 * ((double)N * N));
    const int planes = (int)std::ceil(max_w / dw) + sw + 1;  // predict.cpp:420-421
    const int t0 = -planes / 2;                               // predict.cpp:472
    const size_t g2 = (size_t)G * G;
    if ((double)g2 * planes * 16.0 * 2.2 > 120e9) return fail(RG_ERR_UNSUPPORTED, "w stack too large");
    RG_CUDA(cudaSetDevice(ctx->device));
    begin_call(ctx);

    // the quantised, grid-corrected sky (predict.cpp:187-245), summed per
    // pixel in source order, at its fft-shifted position
    std::vector<double> pts((size_t)2 * npoints), lm_hold, nn_hold;
    if (npoints > 0) RG_CUDA(cudaMemcpy(pts.data(), points, sizeof(double) * pts.size(), cudaMemcpyDefault));
    const double *lm, *nn;
    RG_CHECK(host_table(corr_lm, lm_hold, &lm));
    RG_CHECK(host_table(corr_n, nn_hold, &nn));
    const int lm_t = corr_lm->size * corr_lm->oversampling, n_t = corr_n->size * corr_n->oversampling;
    const double lm_step = 1.0 / (double)lm_t, n_step = 1.0 / (double)n_t;
    const int gd = (G - N) / 2;
    std::vector<SkyEntry> sky;
    std::unordered_map<int64_t, int> at;  // pixel -> entry
    for (int i = 0; i < npoints; i++) {
        const double l = pts[2 * i], m = pts[2 * i + 1];
        if (!std::isfinite(l) || !std::isfinite(m)) return fail(RG_ERR_INVALID_ARGUMENT, "non-finite source position");
        const int lc = (int)std::floor((l / theta + 0.5) * (double)N);
        const int mc = (int)std::floor((m / theta + 0.5) * (double)N);
        if (lc < 0 || lc >= N || mc < 0 || mc >= N)
            return fail(RG_ERR_INVALID_ARGUMENT, "a source lies outside the image (|l|, |m| < theta / 2)");
        const double lq = (double)lc / lambda - theta / 2;
        const double mq = (double)mc / lambda - theta / 2;
        const double n = std::sqrt(1.0 - lq * lq - mq * mq) - 1.0;
        const int aau = (int)std::floor((du * lq) / lm_step) + lm_t / 2;
        const int aav = (int)std::floor((du * mq) / lm_step) + lm_t / 2;
        const int aaw = (int)std::floor((dw * n) / n_step) + n_t / 2;
        if (aau < 0 || aau >= lm_t || aav < 0 || aav >= lm_t || aaw < 0 || aaw >= n_t)
            return fail(RG_ERR_INVALID_ARGUMENT, "a source lies outside the grid-correction tables");
        double a = 1.0;
        a *= lm[aau];
        a *= lm[aav];
        a *= nn[aaw];
        const int col = (gd + lc + G / 2) % G, row = (gd + mc + G / 2) % G;
        const auto known = at.emplace((int64_t)row * G + col, (int)sky.size());
        if (known.second) sky.push_back({row, col, 0, lc, mc, 0, 1.0 / a});
        else sky[known.first->second].val += 1.0 / a;
    }
    const int nsrc = (int)sky.size();
    void *d_sky;
    RG_CHECK(scratch(ctx, "wstack_sky", sizeof(SkyEntry) * (size_t)(nsrc + 1), &d_sky));
    const void *tuv, *tw;
    RG_CHECK(stage_in(ctx, conv_uv->data, sizeof(double) * (size_t)suv * conv_uv->oversampling, "wstack_conv_uv", &tuv));
    RG_CHECK(stage_in(ctx, conv_w->data, sizeof(double) * (size_t)sw * conv_w->oversampling, "wstack_conv_w", &tw));
    const void *du_p, *dv_p, *dw_p;
    RG_CHECK(stage_in(ctx, u, sizeof(double) * (size_t)nvis, "in_u", &du_p));
    RG_CHECK(stage_in(ctx, v, sizeof(double) * (size_t)nvis, "in_v", &dv_p));
    RG_CHECK(stage_in(ctx, w, sizeof(double) * (size_t)nvis, "in_w", &dw_p));
    OutView ov;
    RG_CHECK(out_view(ctx, vis_out, sizeof(double2) * (size_t)nvis, "wstack_vis", false, &ov));
    Diag d;
    RG_CHECK(diag_begin(ctx, &d));

    const DegridGeom geom{du, dw, N, G, planes, suv, conv_uv->oversampling, sw, conv_w->oversampling,
                          (const double *)tuv, (const double *)tw};
    const double *pu = (const double *)du_p, *pv = (const double *)dv_p, *pw = (const double *)dw_p;
    double2 *vis = (double2 *)ov.dev;
    cudaStream_t st = ctx->stream;
    if (nvis > 0 && wstack_use_direct(nvis, nsrc, planes, G, suv, sw)) {
        const double2 *roots;
        RG_CHECK(roots64(ctx, G, &roots));
        void *powers, *base;
        RG_CHECK(scratch(ctx, "wstack_powers", sizeof(double2) * (size_t)(nsrc + 1) * 48, &powers));
        RG_CHECK(scratch(ctx, "wstack_base", sizeof(double2) * (size_t)(nsrc + 1) * planes, &base));
        if (nsrc > 0)
            RG_CUDA(cudaMemcpyAsync(d_sky, sky.data(), sizeof(SkyEntry) * nsrc, cudaMemcpyHostToDevice, st));
        begin_stage(ctx, "wstack_direct");
        auto direct = [&](auto launch) {
            launch(ctx, pu, pv, pw, nvis, geom, (const SkyEntry *)d_sky, nsrc, t0, theta, roots, (double2 *)powers,
                   (double2 *)base, vis, d.err);
        };
        if (suv <= 8 && sw <= 6) direct(launch_direct<8, 6, 2>);
        else if (suv <= 8 && sw <= 8) direct(launch_direct<8, 8, 2>);
        else direct(launch_direct<16, 16, 1>);
        ctx->launches += 2;
        end_stage(ctx);
    } else if (nvis > 0) {
        Fft64Plan plan;
        RG_CHECK(fft64_plan(ctx, G, &plan));
        std::vector<int> slot_of_row((size_t)G, -1);
        int nrows = 0;
        for (SkyEntry &s : sky) {
            if (slot_of_row[s.row] < 0) slot_of_row[s.row] = nrows++;
            s.slot = slot_of_row[s.row];
        }
        void *stack, *rows, *d_slots;
        RG_CHECK(scratch(ctx, "wstack_planes", sizeof(double2) * g2 * planes, &stack));
        RG_CHECK(scratch(ctx, "wstack_rows", sizeof(double2) * (size_t)planes * (nrows + 1) * G, &rows));
        RG_CHECK(scratch(ctx, "wstack_slots", sizeof(int) * (size_t)G, &d_slots));
        RG_CUDA(cudaMemcpyAsync(d_slots, slot_of_row.data(), sizeof(int) * G, cudaMemcpyHostToDevice, st));
        begin_stage(ctx, "wstack_fft");
        if (nsrc > 0) {
            RG_CUDA(cudaMemcpyAsync(d_sky, sky.data(), sizeof(SkyEntry) * nsrc, cudaMemcpyHostToDevice, st));
            RG_CUDA(cudaMemsetAsync(rows, 0, sizeof(double2) * (size_t)planes * nrows * G, st));
            const int64_t tot = (int64_t)nsrc * planes;
            wstack_scatter_kernel<<<(unsigned)std::min<int64_t>((tot + 255) / 256, 4096), 256, 0, st>>>(
                (const SkyEntry *)d_sky, nsrc, planes, t0, N, G, nrows, theta, dw, (double2 *)rows);
            launch_fft64_rows(st, (double2 *)rows, plan, planes * nrows, -1);
            ctx->launches += 2;
        }
        launch_fft64_lines<true>(st, plan, planes, G, -1,
                                 LdSkyCol{(const double2 *)rows, (const int *)d_slots, G, nrows},
                                 StStackCol{(double2 *)stack, G});
        end_stage(ctx);
        begin_stage(ctx, "wstack_degrid");
        const int64_t blocks = std::min<int64_t>((nvis + 7) / 8, (int64_t)ctx->sm_count * 16);
        wstack_degrid_kernel<<<(unsigned)blocks, 256, 0, st>>>((const double2 *)stack, pu, pv, pw, nvis, geom, vis,
                                                               d.err);
        ctx->launches += 2;
        end_stage(ctx);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "W-stacking predict launch");
    RG_CHECK(finish_out(ctx, ov));
    RG_CHECK(diag_end(ctx, d, nullptr));
    collect_timings(ctx);
    ctx->stats[0] = nvis;
    ctx->stats[3] = planes;
    ctx->stats[5] = ctx->launches;
    return RG_OK;
}
