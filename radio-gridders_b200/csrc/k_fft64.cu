// Plans and launches of the FP64 transforms (k_fft64.cuh): in-place 2-D
// transforms and the dirty image's two passes.
//
// Both passes are bound by memory and by the latency of one CTA's
// load - transform - store sequence, with the FP64 pipe behind them
// (5 n^2 log2 n^2 operations: 0.7 GFLOP at n = 2500). One image of a 2500 x 2500
// grid, with the caller's copy of the grid: 300 us, against 4522 us as
// hermitian, shift, radix-2 Bluestein rows, transpose, rows, transpose, shift
// and real part, each a pass of its own. The rows take 77 us (114 with all of
// them transformed, 193 with 16 points a thread and 11 warps an SM, strided
// twiddles and addresses formed point by point) and the columns 159 (227).
#include <algorithm>
#include <string>

#include "k_fft64.cuh"

namespace rg {

bool fft64_any_supported(int n) { return n >= 2 && n <= 4096; }

bool fft64_smooth(int n)
{
    for (int r : {2, 3, 5, 7})
        while (n % r == 0) n /= r;
    return n == 1;
}

// Splits L into stages; false if it has a prime factor above 7. Odd radices
// first: their first stage stores with an odd stride, free of bank conflicts.
// Powers of two as 8s (16s where a thread has the registers: wide) with one 4 or
// 2 for the rest, or 4s in place of an 8 and a 2.
static bool fft64_stages(int L, bool wide, Fft64Plan *p)
{
    int n = L, lg = 0;
    p->nst = 0;
    for (int r : {7, 5, 3})
        while (n % r == 0) {
            n /= r;
            p->radix[p->nst++] = r;
        }
    while (n % 2 == 0) {
        n /= 2;
        lg++;
    }
    if (n != 1) return false;
    while (lg > 0) {
        int e = std::min(lg, 3);
        if (wide) e = lg == 5 || lg == 6 || lg == 9 ? 3 : std::min(lg, 4);
        else if (lg == 4) e = 2;
        p->radix[p->nst++] = 1 << e;
        lg -= e;
    }
    p->L = L;
    p->pad = (L & (L - 1)) == 0 && L >= 256;
    int64_t ns = 1;
    for (int k = 0; k < p->nst; k++) {
        p->magic[k] = ns > 1 ? (unsigned)(((1ull << 32) + ns - 1) / ns) : 0u;
        ns *= p->radix[k];
    }
    return true;
}

// tw[k] = exp(-2 pi i k / L)
__global__ void fft64_twiddle_kernel(double2 *__restrict__ tw, int L)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= L) return;
    double s, c;
    sincospi(-2.0 * (double)k / (double)L, &s, &c);
    tw[k] = make_double2(c, s);
}

// One stage's twiddles: tw[i - 1][k] = exp(-2 pi i i k / (R Ns)), i < R, k < Ns.
__global__ void fft64_stage_twiddle_kernel(double2 *__restrict__ tw, int R, int Ns)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= (R - 1) * Ns) return;
    const int i = n / Ns + 1, k = n % Ns;
    double s, c;
    sincospi(-2.0 * (double)(i * k) / (double)(R * Ns), &s, &c);
    tw[n] = make_double2(c, s);
}

// chirp[m] = exp(-pi i m^2 / n), the phase reduced exactly (m^2 mod 2n in
// integers), and the filter before its transform: conj(chirp) wrapped to
// length L (it is even in m), zero between.
__global__ void fft64_chirp_kernel(double2 *__restrict__ chirp, double2 *__restrict__ wrapped, int n, int L)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= L) return;
    const int d = m < n ? m : L - m;
    double2 v = make_double2(0.0, 0.0);
    if (d < n) {
        const long long q = ((long long)d * d) % (2LL * n);
        double s, c;
        sincospi(-(double)q / (double)n, &s, &c);
        v = make_double2(c, -s);
        if (m < n) chirp[m] = make_double2(c, s);
    }
    wrapped[m] = v;
}

struct LdRows {
    const double2 *d;
    int64_t ld;
    __device__ double2 operator()(int, int line, int n) const { return d[line * ld + n]; }
};
struct StRows {
    double2 *d;
    int64_t ld;
    __device__ void operator()(int, int line, int n, double2 v) const { d[line * ld + n] = v; }
};
struct LdCols {
    const double2 *d;
    int64_t ld, array;
    __device__ double2 operator()(int arr, int line, int n) const { return d[arr * array + n * ld + line]; }
};
struct StCols {
    double2 *d;
    int64_t ld, array;
    __device__ void operator()(int arr, int line, int n, double2 v) const { d[arr * array + n * ld + line] = v; }
};

void launch_fft64_rows(cudaStream_t s, double2 *data, const Fft64Plan &p, int rows, int sign)
{
    launch_fft64_lines<false>(s, p, 1, rows, sign, LdRows{data, p.n}, StRows{data, p.n});
}

rg_status roots64(rg_context *ctx, int n, const double2 **out)
{
    const std::string name = "roots64_" + std::to_string(n);
    const auto known = ctx->scratch.find(name);
    const bool fresh = known == ctx->scratch.end() || !known->second.ptr;
    void *mem;
    RG_CHECK(scratch(ctx, name.c_str(), sizeof(double2) * (size_t)n, &mem));
    if (fresh) {
        fft64_twiddle_kernel<<<(n + 127) / 128, 128, 0, ctx->stream>>>((double2 *)mem, n);
        // a launch that failed shows here alone: the stream has nothing to report
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);  // a later call may be on another stream
        if (e != cudaSuccess) {
            cudaFree(mem);
            ctx->scratch.erase(name);
            return cuda_fail(e, "table of roots");
        }
    }
    *out = (const double2 *)mem;
    return RG_OK;
}

rg_status fft64_plan(rg_context *ctx, int n, Fft64Plan *out)
{
    auto it = ctx->fft64_plans.find(n);
    if (it != ctx->fft64_plans.end()) {
        *out = it->second;
        return RG_OK;
    }
    Fft64Plan p;
    p.n = n;
    const bool direct = fft64_stages(n, false, &p);
    if (!direct) {
        // the cheapest convolution length: points times passes over them, of
        // those whose stages fit one CTA's threads
        Fft64Plan best;
        int64_t cost = INT64_MAX;
        for (int L = 2 * n - 1; L <= 8192; L++) {
            Fft64Plan c;
            if (!fft64_stages(L, true, &c) || fft64_threads<16>(c, 0) > 512) continue;
            if ((int64_t)L * (c.nst + 1) < cost) {
                cost = (int64_t)L * (c.nst + 1);
                best = c;
            }
        }
        p = best;
        p.n = n;
    }
    p.scale = 1.0 / (double)p.L;
    void *tw;
    RG_CHECK(scratch(ctx, ("fft64_" + std::to_string(n)).c_str(), sizeof(double2) * (size_t)p.L, &tw));
    p.tw = (const double2 *)tw;
    double2 *at = (double2 *)tw;
    for (int k = 0, ns = 1; k < p.nst; ns *= p.radix[k++]) {
        const int cnt = (p.radix[k] - 1) * ns;
        if (k > 0) fft64_stage_twiddle_kernel<<<(cnt + 127) / 128, 128, 0, ctx->stream>>>(at, p.radix[k], ns);
        at += cnt;
    }
    if (!direct) {
        void *mem;
        RG_CHECK(scratch(ctx, ("chirp64_" + std::to_string(n)).c_str(), sizeof(double2) * (size_t)(p.L + n), &mem));
        double2 *filter = (double2 *)mem, *chirp = filter + p.L;
        fft64_chirp_kernel<<<(p.L + 127) / 128, 128, 0, ctx->stream>>>(chirp, filter, n, p.L);
        Fft64Plan q = p;  // the L-point transform of the filter
        q.n = p.L;
        launch_fft64_rows(ctx->stream, filter, q, 1, -1);
        p.filter = filter;
        p.chirp = chirp;
    }
    RG_CUDA(cudaGetLastError());
    RG_CUDA(cudaStreamSynchronize(ctx->stream));  // a later call may be on another stream
    ctx->fft64_plans[n] = p;
    *out = p;
    return RG_OK;
}

void launch_fft64_2d(cudaStream_t s, double2 *data, int batch, const Fft64Plan &py, const Fft64Plan &px, int sign)
{
    const int ny = py.n, nx = px.n;
    const int64_t array = (int64_t)ny * nx;
    // a launch counts its lines and CTAs in 32 bits: at most 2^30 lines each
    // (2^31 rows of 2 points are 69 GB, which fits the device)
    const int step = (1 << 30) / std::max(ny, nx);
    for (int64_t at = 0; at < batch; at += step) {
        const int cnt = (int)std::min<int64_t>(step, batch - at);
        double2 *d = data + at * array;
        launch_fft64_rows(s, d, px, cnt * ny, sign);
        launch_fft64_lines<true>(s, py, cnt, nx, sign, LdCols{d, nx, array}, StCols{d, nx, array});
    }
}

// Rows of the dirty image: row y of the hermitian sum h (src/reference/grid.c:
// 639-662: linear index i >= N + 1 pairs with N^2 + N - i; row 0 and element
// (1, 0) are left as they are) with its columns shifted (grid.c:665-680),
// f_y[n] = h(y, n + N/2 mod N). Only rows 0..N/2 are transformed: away from column 0,
// h(N - y, N - x) = conj(h(y, x)), so with d_y = conj(h(N - y, 0)) - h(y, 0), which the
// thread that reads column 0 leaves in delta,
//   X_(N-y)[k] = conj(X_y[k] + (-1)^k d_y).
struct LdImageRow {
    const double2 *g;
    double2 *delta;
    int N;
    __device__ double2 sum(int64_t i) const
    {
        const double2 a = g[i];
        if (i < N + 1) return a;
        const double2 b = g[(int64_t)N * N + N - i];
        return make_double2(a.x + b.x, a.y - b.y);
    }
    __device__ double2 operator()(int, int y, int n) const
    {
        const int x = n < N / 2 ? n + N / 2 : n - N / 2;
        const double2 h = sum((int64_t)y * N + x);
        if (x == 0 && y > 0 && y < N / 2) {
            const double2 m = sum((int64_t)(N - y) * N);
            delta[y] = make_double2(m.x - h.x, -m.y - h.y);
        }
        return h;
    }
};
// Columns of all rows, in shifted order, from the transformed half.
struct LdImageCol {
    const double2 *rows, *delta;
    int N;
    __device__ double2 operator()(int, int k, int n) const
    {
        const int y = n < N / 2 ? n + N / 2 : n - N / 2;
        if (y <= N / 2) return rows[(int64_t)y * N + k];
        const double2 v = rows[(int64_t)(N - y) * N + k], d = __ldg(delta + N - y);
        return k & 1 ? make_double2(v.x - d.x, d.y - v.y) : make_double2(v.x + d.x, -v.y - d.y);
    }
};
// Columns: the transformed grid and the image at their shifted places.
struct StImageCol {
    double2 *g;
    double *img;
    const double *taper;
    int N;
    __device__ void operator()(int, int line, int n, double2 v) const
    {
        const int y = n < N / 2 ? n + N / 2 : n - N / 2, x = line < N / 2 ? line + N / 2 : line - N / 2;
        const int64_t i = (int64_t)y * N + x;
        g[i] = v;
        img[i] = taper ? v.x / (__ldg(taper + y) * __ldg(taper + x)) : v.x;
    }
};

void launch_image_from_grid(cudaStream_t s, double2 *grid, double2 *tmp, double *image, const double *taper,
                            const Fft64Plan &p)
{
    const int N = p.n;
    double2 *delta = tmp + (int64_t)(N / 2 + 1) * N;
    launch_fft64_lines<false>(s, p, 1, N / 2 + 1, -1, LdImageRow{grid, delta, N}, StRows{tmp, N});
    launch_fft64_lines<true>(s, p, 1, N, -1, LdImageCol{tmp, delta, N}, StImageCol{grid, image, taper, N});
}

}  // namespace rg
