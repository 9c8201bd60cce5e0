// Direct Fourier transform imager.
//
//   image[y][x] = factor * sum_k Re(V_k exp(-2 pi i phi_k(x, y)))
//   phi = u l + v m + w (1 - n),  l = theta (x - N/2)/N, m = theta (y - N/2)/N
//
// the phase convention of the reference's calculate_dft_sum_flat
// (src/dft/dft_cuda.cu:15-39), with l taken from the column and u, v, w in
// wavelengths (its defects, src/dft/dft_cuda.cu:55-57 and :98-112, removed).
//
// A CTA owns a 32 x 32 pixel tile; each thread four pixels of one column.
// Rows [row0, row0 + nrows) only (a rank's share of a row-partitioned image):
// tiles start at row0, so a share that starts on a multiple of 32 computes its
// rows exactly as the whole image does.
// Visibilities are staged through shared memory 256 at a time.  Precision
// modes (the precision study):
//   FP64_REDUCED: per (tile, visibility) the phase at the tile centre phi0 is
//     formed and reduced modulo 1 in FP64 and folded into the visibility
//     (V' = V exp(-2 pi i phi0)); per pixel only the small increment
//     delta = u dl + v dm + w (n0 - n) is formed in FP32, reduced modulo 1, and
//     fed to the hardware sin/cos.  Partial sums are FP32 per batch of 256,
//     accumulated in FP64.
//   FP32_NAIVE: phi formed in FP32 from FP32 u, v, w, l, m, n, reduced in FP32.
//   FP64: phi, reduction and sin/cos all FP64, per pixel and visibility only
//     where the tiles below do not apply or the visibilities are few.
//
// FP64 by tiles. Over a 32 x 32 tile the phase is separable but for a small
// rest: with g(l, m) = 1 - n and the tile's centre (l0, m0),
//   u l + v m + w g = [u l + w g(l, m0)] + [v m + w (g(l0, m) - g(l0, m0))] + w r(l, m),
// so with one phasor a visibility and column (times V: C) and one a visibility
// and row (B), the sum over visibilities of V exp(-2 pi i phi) is
//   sum_j (-2 pi i r)^j / j! sum_k w_k^j C_k(x) B_k(y):
// J real matrix products, summed into per-pixel moments and combined with the
// powers of r at the end. |r| <= hl hm max |l m| / n^3 over the tile, and J is the
// smallest count whose first term left out is below 1e-16. J = 4 at 500 x 500,
// theta 0.1, |w| <= 600.
#include <algorithm>
#include <cmath>

#include "rg_internal.h"

namespace rg {

constexpr int TILE = 32, DFT_BATCH = 256, PIX = 4;

// The largest |w|, as bits (non-negative doubles order as integers); infinity
// where any input is not finite. bits starts at zero.
__global__ void dft_range_kernel(const double *__restrict__ u, const double *__restrict__ v,
                                 const double *__restrict__ w, const double2 *__restrict__ vis, int64_t n,
                                 unsigned long long *__restrict__ bits)
{
    double m = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double2 z = vis[i];
        const bool ok = isfinite(u[i]) && isfinite(v[i]) && isfinite(w[i]) && isfinite(z.x) && isfinite(z.y);
        m = ok ? fmax(m, fabs(w[i])) : INFINITY;
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(bits, (unsigned long long)__double_as_longlong(m));
}

__device__ __forceinline__ double pixel_lm(int x, int N, double theta) { return theta * (double)(x - N / 2) / N; }

// Moments the tile at (x0, y0) needs; 0 where it goes pixel by pixel: more than
// kDftMoments, a pixel at or beyond the horizon, or inputs not finite.
constexpr int kDftMoments = 8;
__device__ __forceinline__ int dft_moments(int x0, int y0, int N, double theta, double wmax)
{
    const double hl = theta * (TILE / 2) / N;
    const double lm = fmax(fabs(pixel_lm(x0, N, theta)), fabs(pixel_lm(x0 + TILE, N, theta)));
    const double mm = fmax(fabs(pixel_lm(y0, N, theta)), fabs(pixel_lm(y0 + TILE, N, theta)));
    const double nn = 1.0 - lm * lm - mm * mm;
    if (!(nn > 0.01)) return 0;
    const double eps = 2.0 * M_PI * wmax * hl * hl * lm * mm / (nn * sqrt(nn));
    if (!(eps < 1.0)) return 0;
    double term = eps;
    for (int j = 1; j <= kDftMoments; j++) {
        if (term <= 1e-16) return j;
        term *= eps / (j + 1);
    }
    return 0;
}

template <int MODE>
__global__ void __launch_bounds__(256) dft_kernel(const double *__restrict__ u,
                                                  const double *__restrict__ v,
                                                  const double *__restrict__ w,
                                                  const double2 *__restrict__ vis, int64_t nvis,
                                                  double *__restrict__ image, int N, double theta,
                                                  double factor, int row0, int nrows,
                                                  const double *__restrict__ wmax)
{
    // FP64: the tiles that the moments do not cover (wmax nullptr: all), one share
    // of the visibilities a CTA as the moments have, so a few such tiles do not
    // leave the device idle
    int64_t k0 = 0, k1 = nvis;
    if (MODE == RG_DFT_FP64) {
        if (wmax && dft_moments(blockIdx.x * TILE, row0 + blockIdx.y * TILE, N, theta, *wmax) > 0) return;
        const int64_t share = (nvis + gridDim.z - 1) / gridDim.z;
        k0 = blockIdx.z * share;
        k1 = min(nvis, k0 + share);
        image += (int64_t)blockIdx.z * nrows * N;
    }
    // FP32 modes: (u, v, w, Re V) as one 16-byte entry and Im V beside it, so a
    // visibility is two shared-memory loads in the inner loop
    __shared__ float4 s4[DFT_BATCH];
    __shared__ float si[DFT_BATCH];
    __shared__ double du[DFT_BATCH], dv[DFT_BATCH], dw[DFT_BATCH], dr[DFT_BATCH], di[DFT_BATCH];
    const int tx = threadIdx.x % TILE, ty = threadIdx.x / TILE;  // ty in [0, 8)
    const int x0 = blockIdx.x * TILE, y0 = row0 + blockIdx.y * TILE;
    const int cx = x0 + TILE / 2, cy = y0 + TILE / 2;
    const double l0 = theta * (double)(cx - N / 2) / N;
    const double m0 = theta * (double)(cy - N / 2) / N;
    const double n0 = sqrt(1.0 - l0 * l0 - m0 * m0);

    const int x = x0 + tx;
    const double l = theta * (double)(x - N / 2) / N;
    double lp[PIX], mp[PIX], one_minus_n[PIX];
    float dl, dm[PIX], dn[PIX];
    dl = (float)(l - l0);
#pragma unroll
    for (int p = 0; p < PIX; p++) {
        const int y = y0 + ty + 8 * p;
        lp[p] = l;
        mp[p] = theta * (double)(y - N / 2) / N;
        const double nn = sqrt(1.0 - l * l - mp[p] * mp[p]);
        one_minus_n[p] = 1.0 - nn;
        dm[p] = (float)(mp[p] - m0);
        dn[p] = (float)(n0 - nn);
    }
    double acc[PIX] = {0.0, 0.0, 0.0, 0.0};

    for (int64_t b0 = k0; b0 < k1; b0 += DFT_BATCH) {
        const int cnt = (int)(k1 - b0 < DFT_BATCH ? k1 - b0 : DFT_BATCH);
        __syncthreads();
        if ((int)threadIdx.x < cnt) {
            const int64_t k = b0 + threadIdx.x;
            const double uu = u[k], vv = v[k], ww = w[k];
            const double2 z = vis[k];
            if (MODE == RG_DFT_FP64_REDUCED) {
                double ph = uu * l0 + vv * m0 + ww * (1.0 - n0);
                ph -= rint(ph);
                double s, c;
                sincospi(2.0 * ph, &s, &c);
                // V' = V exp(-2 pi i phi0)
                s4[threadIdx.x] = make_float4((float)uu, (float)vv, (float)ww, (float)(z.x * c + z.y * s));
                si[threadIdx.x] = (float)(z.y * c - z.x * s);
            } else if (MODE == RG_DFT_FP32_NAIVE) {
                s4[threadIdx.x] = make_float4((float)uu, (float)vv, (float)ww, (float)z.x);
                si[threadIdx.x] = (float)z.y;
            } else {
                du[threadIdx.x] = uu;
                dv[threadIdx.x] = vv;
                dw[threadIdx.x] = ww;
                dr[threadIdx.x] = z.x;
                di[threadIdx.x] = z.y;
            }
        }
        __syncthreads();
        if (MODE == RG_DFT_FP64) {
            double part[PIX] = {0.0, 0.0, 0.0, 0.0};
            for (int j = 0; j < cnt; j++) {
#pragma unroll
                for (int p = 0; p < PIX; p++) {
                    double ph = du[j] * lp[p] + dv[j] * mp[p] + dw[j] * one_minus_n[p];
                    ph -= rint(ph);
                    double s, c;
                    sincospi(2.0 * ph, &s, &c);
                    part[p] += dr[j] * c + di[j] * s;
                }
            }
#pragma unroll
            for (int p = 0; p < PIX; p++) acc[p] += part[p];
        } else {
            float part[PIX] = {0.f, 0.f, 0.f, 0.f};
            float fl[PIX], fm[PIX], fn[PIX];
#pragma unroll
            for (int p = 0; p < PIX; p++) {
                if (MODE == RG_DFT_FP32_NAIVE) {
                    fl[p] = (float)lp[p];
                    fm[p] = (float)mp[p];
                    fn[p] = (float)one_minus_n[p];
                } else {
                    fl[p] = dl;
                    fm[p] = dm[p];
                    fn[p] = dn[p];
                }
            }
#pragma unroll 4
            for (int j = 0; j < cnt; j++) {
                const float4 e = s4[j];
                const float uj = e.x, vj = e.y, wj = e.z, rj = e.w, ij = si[j];
#pragma unroll
                for (int p = 0; p < PIX; p++) {
                    float d = fmaf(uj, fl[p], fmaf(vj, fm[p], wj * fn[p]));
                    // nearest integer by the 1.5 * 2^23 shift (|d| < 2^22 turns):
                    // two adds on the FMA pipe instead of a rounding instruction
                    d -= (d + 12582912.f) - 12582912.f;
                    float s, c;
                    __sincosf(6.283185307179586f * d, &s, &c);
                    part[p] = fmaf(rj, c, fmaf(ij, s, part[p]));
                }
            }
#pragma unroll
            for (int p = 0; p < PIX; p++) acc[p] += (double)part[p];
        }
    }
#pragma unroll
    for (int p = 0; p < PIX; p++) {
        const int y = y0 + ty + 8 * p;
        if (x < N && y < row0 + nrows) image[(int64_t)(y - row0) * N + x] = factor * acc[p];
    }
}

// exp(-2 pi i t) for a phase t in turns, |t| <= 1/2: the nearest of 64 tabulated phasors
// times the Taylor series of the rest (|x| <= pi / 64: the first terms left out
// are below 1e-17).
__device__ __forceinline__ double2 phasor(double t, const double2 *table)
{
    const double k = rint(t * 64.0);
    const double x = (t - k * (1.0 / 64.0)) * (2.0 * M_PI), x2 = x * x;
    const double2 a = table[(int)k & 63];
    const double s = x * fma(x2, fma(x2, fma(x2, fma(x2, 1.0 / 362880.0, -1.0 / 5040.0), 1.0 / 120.0), -1.0 / 6.0), 1.0);
    const double c = fma(x2, fma(x2, fma(x2, fma(x2, 1.0 / 40320.0, -1.0 / 720.0), 1.0 / 24.0), -0.5), 1.0);
    return make_double2(fma(a.x, c, a.y * s), fma(a.y, c, -a.x * s));  // a (c - i s)
}

// a b + c modulo one turn, in about [-1/2, 1/2]: whole turns leave the product
// before c is added, and what its rounding lost comes back, so a phase of
// hundreds of turns keeps the precision of its fraction.
__device__ __forceinline__ double turns(double a, double b, double c)
{
    const double p = a * b;
    const double t = (p - rint(p)) + (fma(a, b, -p) + c);
    return t - rint(t);
}

// One tile and one share of the visibilities (blockIdx.z of gridDim.z): four
// warps, each 8 columns x 32 rows of every moment, on the FP64 tensor pipe (mma
// m8n8k4: the depth is two visibilities' real and imaginary parts). 32
// visibilities at a time: phasors of both sides into shared memory, then the
// products; the weights w^j are put on the left fragment in registers. Tiles of
// MIN..MAX moments only. part: [share][row][column], times scale.
// Bound by the FP64 pipe: 2 J + about 2 multiply-adds a pixel and visibility,
// where reduction and sincospi took about 59. 500 x 500 pixels, 20,000
// visibilities: 15.9 -> 3.5 ms, the products at 0.66 of the pipe's rate and the
// phasors 0.16 of its cycles.
constexpr int kDftVis = 32, kDftStrideB = TILE + 4;  // 4 mod 16: a fragment's 4 k x 8 rows on distinct banks

template <int MIN, int MAX>
__global__ void __launch_bounds__(128) dft_moments_kernel(const double *__restrict__ u, const double *__restrict__ v,
                                                          const double *__restrict__ w,
                                                          const double2 *__restrict__ vis, int64_t nvis,
                                                          double *__restrict__ part, int N, double theta,
                                                          double scale, int row0, int nrows,
                                                          const double *__restrict__ wmax_p)
{
    __shared__ double2 sC[kDftVis][TILE];
    __shared__ double sB[2 * kDftVis][kDftStrideB];
    __shared__ double sw[kDftVis], su[kDftVis], sv[kDftVis], sws[kDftVis];
    __shared__ double2 sz[kDftVis], table[64];
    const int x0 = blockIdx.x * TILE, y0 = row0 + blockIdx.y * TILE;
    const double wmax = *wmax_p;
    const int J = dft_moments(x0, y0, N, theta, wmax);
    if (J < MIN || J > MAX) return;
    const double wscale = wmax > 0.0 ? 1.0 / wmax : 0.0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    if (tid < 64) {
        double s, c;
        sincospi(tid / 32.0, &s, &c);
        table[tid] = make_double2(c, -s);
    }
    auto one_minus_n = [&](double l, double m) { return 1.0 - sqrt(1.0 - l * l - m * m); };
    const double l0 = pixel_lm(x0 + TILE / 2, N, theta), m0 = pixel_lm(y0 + TILE / 2, N, theta);
    const double g0 = one_minus_n(l0, m0);
    // this thread's column and row when phasors are made
    const double lx = pixel_lm(x0 + lane, N, theta), my = pixel_lm(y0 + lane, N, theta);
    const double gx = one_minus_n(lx, m0), gy = one_minus_n(l0, my) - g0;
    double2 acc[MAX][4];
#pragma unroll
    for (int j = 0; j < MAX; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[j][i] = make_double2(0.0, 0.0);
    const int64_t share = (nvis + gridDim.z - 1) / gridDim.z;
    const int64_t k0 = blockIdx.z * share, k1 = min(nvis, k0 + share);
    for (int64_t b = k0; b < k1; b += kDftVis) {
        const int cnt = (int)min((int64_t)kDftVis, k1 - b);
        __syncthreads();
        if (tid < kDftVis) {
            const bool on = tid < cnt;
            su[tid] = on ? u[b + tid] : 0.0;
            sv[tid] = on ? v[b + tid] : 0.0;
            sw[tid] = on ? w[b + tid] : 0.0;
            sws[tid] = sw[tid] * wscale;
            sz[tid] = on ? vis[b + tid] : make_double2(0.0, 0.0);
        }
        __syncthreads();
#pragma unroll 2
        for (int k = warp; k < kDftVis; k += 4) {
            const double ww = sw[k];
            const double2 z = sz[k];
            const double2 a = phasor(turns(su[k], lx, ww * gx), table);
            sC[k][lane] = make_double2(fma(z.x, a.x, -z.y * a.y), fma(z.x, a.y, z.y * a.x));
            const double2 c = phasor(turns(sv[k], my, ww * gy), table);
            sB[2 * k][lane] = c.x;
            sB[2 * k + 1][lane] = c.y;
        }
        __syncthreads();
        for (int k = 0; k < cnt; k += 2) {
            const double2 z = sC[k + (t >> 1)][8 * warp + g];
            const double ws = sws[k + (t >> 1)];
            // rows of (re, -im) for the real part of the product, (im, re) for the imaginary
            double even = t & 1 ? -z.y : z.x, odd = t & 1 ? z.x : z.y;
            double fb[4];
#pragma unroll
            for (int i = 0; i < 4; i++) fb[i] = sB[2 * k + t][8 * i + g];
            odd *= ws;
            const double w2 = ws * ws;
#pragma unroll
            for (int j = 0; j < MAX; j++) {
                if (j < MIN || j < J) {
                    const double fa = j & 1 ? odd : even;
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                                     : "+d"(acc[j][i].x), "+d"(acc[j][i].y)
                                     : "d"(fa), "d"(fb[i]));
                    if (j & 1) odd *= w2;
                    else even *= w2;
                }
            }
        }
    }
    // combine: the term of moment j is (-i q)^j / j! with q = 2 pi r wmax
    const int x = x0 + 8 * warp + g;
    const double l = pixel_lm(x, N, theta), gl = one_minus_n(l, m0);
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int y = y0 + 8 * i + 2 * t + h;
            if (x >= N || y >= row0 + nrows) continue;
            const double m = pixel_lm(y, N, theta);
            const double q = 2.0 * M_PI * wmax * ((one_minus_n(l, m) - gl) - (one_minus_n(l0, m) - g0));
            double sum = 0.0, f = 1.0;
#pragma unroll
            for (int j = 0; j < MAX; j++) {
                if (j > 0) f *= q / j;
                const double mom = h ? acc[j][i].y : acc[j][i].x;
                // Re((-i)^j (re + i im)): re, im, -re, -im
                sum = fma(j & 2 ? -f : f, mom, sum);
            }
            part[((int64_t)blockIdx.z * nrows + (y - row0)) * N + x] = scale * sum;
        }
}

// image = factor * the sum of the shares, in order
__global__ void dft_shares_kernel(const double *__restrict__ part, int shares, double *__restrict__ image, int N,
                                  double factor, int nrows)
{
    const int x = blockIdx.x * TILE + threadIdx.x % TILE;
    if (x >= N) return;
    for (int y = blockIdx.y * TILE + threadIdx.x / TILE; y < min(nrows, (int)(blockIdx.y + 1) * TILE); y += 8) {
        double s = 0.0;
        for (int k = 0; k < shares; k++) s += part[((int64_t)k * nrows + y) * N + x];
        image[(int64_t)y * N + x] = factor * s;
    }
}

// Tiles of the whole image: the rules below go by it, so a band of rows is summed
// as the image's rows are.
static int64_t dft64_tiles(int grid_size)
{
    const int64_t side = (grid_size + TILE - 1) / TILE;
    return side * side;
}

// Shares the visibilities are split into: six rounds of four resident CTAs an SM
// over the tiles, for a short tail (three rounds: 3.64 against 3.48 ms at
// 500 x 500), at least 512 visibilities each. Below 1024 visibilities that is one
// share, whose tiles go through them one after another: one round there, at
// least 32 each. 64 x 64, 400 visibilities: 143 -> 68 us; 380 x 380, 400: 104 ->
// 90; the same on larger calls would cost (100 x 100, 5000: 184 -> 229 us).
int dft64_shares(int grid_size, int64_t n, int sm_count)
{
    const int64_t tiles = dft64_tiles(grid_size);
    int64_t s = ((int64_t)sm_count * 24 + tiles - 1) / tiles;
    if (s > n / 512) s = n / 512;
    if (n < 1024) s = std::min<int64_t>((int64_t)sm_count * 4 / tiles, n / 32);
    return s < 1 ? 1 : (int)(s > 64 ? 64 : s);
}

// FP64, pixel by pixel for the whole image, where the visibilities are too few to
// pay for the moments' launches, 20 us: a tile takes 0.47 us a visibility so,
// about half of that by moments (8 x 8 pixels, 1 visibility: 24 against 43 us;
// 16 x 16, 64: 53 against 73; 200 x 200, 64 and 96: 53 and 65 against 53 and 49;
// 500 x 500, 10: 29 against 41). Up to 16 tiles, at most 128 pixels a side, the
// line lies higher, such tiles needing more moments (128 x 128, 96: 68 against 74).
static bool dft64_by_pixel(int grid_size, int64_t n, int sm_count)
{
    const int64_t tiles = dft64_tiles(grid_size);
    return tiles <= 16 ? n <= 96 : n * std::max<int64_t>(tiles, sm_count) <= (int64_t)64 * sm_count;
}

void launch_dft(cudaStream_t s, const double *u, const double *v, const double *w,
                const double2 *vis, int64_t n, double *image, int grid_size, double theta,
                int precision, double factor, int sm_count, int row0, int nrows, double *work)
{
    if (nrows < 0) {
        row0 = 0;
        nrows = grid_size;
    }
    if (nrows == 0) return;
    dim3 grd((grid_size + TILE - 1) / TILE, (nrows + TILE - 1) / TILE);
    switch (precision) {
        case RG_DFT_FP32_NAIVE:
            dft_kernel<RG_DFT_FP32_NAIVE><<<grd, 256, 0, s>>>(u, v, w, vis, n, image, grid_size, theta, factor, row0,
                                                                 nrows, nullptr);
            break;
        case RG_DFT_FP64: {
            if (dft64_by_pixel(grid_size, n, sm_count)) {
                dft_kernel<RG_DFT_FP64><<<grd, 256, 0, s>>>(u, v, w, vis, n, image, grid_size, theta, factor, row0,
                                                            nrows, nullptr);
                break;
            }
            const int shares = dft64_shares(grid_size, n, sm_count);
            double *wmax = work, *part = shares > 1 ? work + 2 : image;
            const double scale = shares > 1 ? 1.0 : factor;  // one share: the image itself
            cudaMemsetAsync(wmax, 0, sizeof(double), s);
            if (n > 0)
                dft_range_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 592), 256, 0, s>>>(
                    u, v, w, vis, n, (unsigned long long *)wmax);
            const dim3 tiles(grd.x, grd.y, shares);
            dft_moments_kernel<1, 4><<<tiles, 128, 0, s>>>(u, v, w, vis, n, part, grid_size, theta, scale, row0, nrows,
                                                           wmax);
            dft_moments_kernel<5, kDftMoments><<<tiles, 128, 0, s>>>(u, v, w, vis, n, part, grid_size, theta, scale,
                                                                    row0, nrows, wmax);
            dft_kernel<RG_DFT_FP64><<<tiles, 256, 0, s>>>(u, v, w, vis, n, part, grid_size, theta, scale, row0, nrows,
                                                          wmax);
            if (shares > 1) dft_shares_kernel<<<grd, 256, 0, s>>>(part, shares, image, grid_size, factor, nrows);
            break;
        }
        default:
            dft_kernel<RG_DFT_FP64_REDUCED><<<grd, 256, 0, s>>>(u, v, w, vis, n, image, grid_size, theta, factor, row0,
                                                                 nrows, nullptr);
            break;
    }
}

}  // namespace rg
