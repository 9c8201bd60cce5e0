// FP64 transforms of any length up to 4096: the line kernel and its pieces.
//
// A CTA transforms `lines` of L points, held in shared memory: mixed-radix
// Stockham stages (radices 2, 3, 4, 5, 7, 8 and 16), each stage's butterflies
// in registers. The first stage reads its points through a load functor and
// the last writes through a store functor, so reordering (shift, hermitian
// sum, taper) is done on the way and a 2-D transform is two passes over
// memory: rows, then groups of adjacent columns. A stage reads all its points
// into registers before any is written, so one copy in shared memory is enough
// (8192 points fit a CTA).
//
// Lengths with a prime factor above 7 go through Bluestein's chirp-z algorithm
// (Bluestein 1970; Rabiner, Schafer & Rader 1969): with c[m] = exp(-pi i m^2 / n),
//   X[k] = c[k] sum_j (x[j] c[j]) conj(c[k - j]),
// a cyclic convolution of length L >= 2n - 1 done as two L-point transforms in
// the same kernel. The reference transforms any even grid size with FFTW
// (src/reference/main.c:269-294), and grid.out's grid size is
// floor(lambda * theta).
#pragma once

#include <utility>

#include "rg_internal.h"

namespace rg {

__device__ __forceinline__ double2 cmul64(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cadd64(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub64(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 swap64(double2 a) { return make_double2(a.y, a.x); }

// Forward transforms of R points in registers, natural order in and out.
template <int R>
struct Dft64;

template <>
struct Dft64<2> {
    static __device__ __forceinline__ void run(double2 *a)
    {
        const double2 x = a[0], y = a[1];
        a[0] = cadd64(x, y);
        a[1] = csub64(x, y);
    }
};

// a, b, c, d -> transform in order (the arguments are references)
__device__ __forceinline__ void dft4(double2 &a, double2 &b, double2 &c, double2 &d)
{
    const double2 s0 = cadd64(a, c), d0 = csub64(a, c), s1 = cadd64(b, d), d1 = csub64(b, d);
    a = cadd64(s0, s1);
    c = csub64(s0, s1);
    b = make_double2(d0.x + d1.y, d0.y - d1.x);  // d0 - i d1
    d = make_double2(d0.x - d1.y, d0.y + d1.x);
}

template <>
struct Dft64<4> {
    static __device__ __forceinline__ void run(double2 *a) { dft4(a[0], a[1], a[2], a[3]); }
};

template <>
struct Dft64<3> {
    static __device__ __forceinline__ void run(double2 *a)
    {
        constexpr double s = 0.86602540378443864676;
        const double2 p = cadd64(a[1], a[2]), m = csub64(a[1], a[2]);
        const double2 c = make_double2(fma(-0.5, p.x, a[0].x), fma(-0.5, p.y, a[0].y));
        a[0] = cadd64(a[0], p);
        a[1] = make_double2(fma(s, m.y, c.x), fma(-s, m.x, c.y));
        a[2] = make_double2(fma(-s, m.y, c.x), fma(s, m.x, c.y));
    }
};

template <>
struct Dft64<5> {
    static __device__ __forceinline__ void run(double2 *a)
    {
        constexpr double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
        constexpr double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
        const double2 p1 = cadd64(a[1], a[4]), m1 = csub64(a[1], a[4]);
        const double2 p2 = cadd64(a[2], a[3]), m2 = csub64(a[2], a[3]);
        const double2 x = a[0];
        const double2 u = make_double2(fma(c1, p1.x, fma(c2, p2.x, x.x)), fma(c1, p1.y, fma(c2, p2.y, x.y)));
        const double2 v = make_double2(fma(c2, p1.x, fma(c1, p2.x, x.x)), fma(c2, p1.y, fma(c1, p2.y, x.y)));
        const double2 q = make_double2(fma(s1, m1.x, s2 * m2.x), fma(s1, m1.y, s2 * m2.y));
        const double2 r = make_double2(fma(s2, m1.x, -s1 * m2.x), fma(s2, m1.y, -s1 * m2.y));
        a[0] = cadd64(x, cadd64(p1, p2));
        a[1] = make_double2(u.x + q.y, u.y - q.x);  // u - i q
        a[4] = make_double2(u.x - q.y, u.y + q.x);
        a[2] = make_double2(v.x + r.y, v.y - r.x);
        a[3] = make_double2(v.x - r.y, v.y + r.x);
    }
};

template <>
struct Dft64<7> {
    static __device__ __forceinline__ void run(double2 *a)
    {
        constexpr double c[3] = {0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
        constexpr double s[3] = {0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
        double2 p[3], m[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            p[j] = cadd64(a[j + 1], a[6 - j]);
            m[j] = csub64(a[j + 1], a[6 - j]);
        }
        const double2 x = a[0];
        a[0] = cadd64(cadd64(x, p[0]), cadd64(p[1], p[2]));
#pragma unroll
        for (int k = 1; k <= 3; k++) {
            double2 u = x, q = make_double2(0.0, 0.0);
#pragma unroll
            for (int j = 1; j <= 3; j++) {
                const int e = (j * k) % 7;  // angle 2 pi e / 7, e in 1..6
                const double cc = c[(e <= 3 ? e : 7 - e) - 1], ss = e <= 3 ? s[e - 1] : -s[6 - e];
                u = make_double2(fma(cc, p[j - 1].x, u.x), fma(cc, p[j - 1].y, u.y));
                q = make_double2(fma(ss, m[j - 1].x, q.x), fma(ss, m[j - 1].y, q.y));
            }
            a[k] = make_double2(u.x + q.y, u.y - q.x);
            a[7 - k] = make_double2(u.x - q.y, u.y + q.x);
        }
    }
};

template <>
struct Dft64<8> {
    static __device__ __forceinline__ void run(double2 *a)
    {
        constexpr double h = 0.70710678118654752440;
        dft4(a[0], a[2], a[4], a[6]);
        dft4(a[1], a[3], a[5], a[7]);
        // odd half times exp(-2 pi i k / 8), k = 0..3
        const double2 o1 = make_double2(h * (a[3].x + a[3].y), h * (a[3].y - a[3].x));
        const double2 o2 = make_double2(a[5].y, -a[5].x);
        const double2 o3 = make_double2(h * (a[7].y - a[7].x), -h * (a[7].x + a[7].y));
        const double2 e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6], o0 = a[1];
        a[0] = cadd64(e0, o0);
        a[4] = csub64(e0, o0);
        a[1] = cadd64(e1, o1);
        a[5] = csub64(e1, o1);
        a[2] = cadd64(e2, o2);
        a[6] = csub64(e2, o2);
        a[3] = cadd64(e3, o3);
        a[7] = csub64(e3, o3);
    }
};

template <>
struct Dft64<16> {
    static __device__ __forceinline__ void run(double2 *a)
    {
        constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, h = 0.70710678118654752440;
        // exp(-2 pi i e / 16)
        constexpr double wc[10] = {1.0, c1, h, s1, 0.0, -s1, -h, -c1, -1.0, -c1};
        constexpr double ws[10] = {0.0, -s1, -h, -c1, -1.0, -c1, -h, -s1, 0.0, s1};
#pragma unroll
        for (int n = 0; n < 4; n++) dft4(a[n], a[4 + n], a[8 + n], a[12 + n]);
#pragma unroll
        for (int n = 1; n < 4; n++)
#pragma unroll
            for (int k = 1; k < 4; k++) {
                double2 &z = a[4 * k + n];
                if (n * k == 4) z = make_double2(z.y, -z.x);
                else z = cmul64(z, make_double2(wc[n * k], ws[n * k]));
            }
#pragma unroll
        for (int k = 0; k < 4; k++) dft4(a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3]);
        // a[4 k1 + k2] = X[k1 + 4 k2]: transpose the 4 x 4
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int n = k + 1; n < 4; n++) {
                const double2 t = a[4 * k + n];
                a[4 * k + n] = a[4 * n + k];
                a[4 * n + k] = t;
            }
    }
};

// f(0), f(1), ..., f(N - 1) with the index a compile-time constant: the arrays it
// indexes stay in registers.
template <class F, int... I>
__device__ __forceinline__ void static_for_seq(F f, std::integer_sequence<int, I...>)
{
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F f)
{
    static_for_seq(f, std::make_integer_sequence<int, N>{});
}

// Butterflies of radix r a thread holds at once, for about PTS points in registers.
template <int PTS>
__host__ __device__ constexpr int fft64_per(int r)
{
    return PTS / r > 1 ? PTS / r : 1;
}

// Threads of a CTA at most: 10 points a thread leave registers for 20 warps on an
// SM, 16 points for 16.
__host__ __device__ constexpr int fft64_max_threads(int pts) { return pts > 10 ? 512 : 640; }

// Shared memory of a CTA: point n of line t at n + t L, or for columns
// interleaved at n 2^lgT + t. With an odd first radix (every length that is not
// a power of two) a stage's strided stores spread over the banks by themselves;
// a power of two takes one spare element after every 16 (pad). Either way the
// R points of a butterfly lie at one stride from its first.
struct Fft64Work {
    double2 *sm;
    int L, lgT;
    bool pad;
};

// One Stockham stage of radix R: sub-transforms of length Ns become R Ns long.
// tw: the stage's twiddles exp(-2 pi i i k / (R Ns)) at [i - 1][k], k < Ns.
// from_in: points come from in(t, n); to_out: results go to out(t, n, v).
// filter: a result in shared memory is multiplied by filter[n] and its parts
// exchanged (the inverse transform follows as a forward one).
template <int R, int PTS, bool COL, class In, class Out>
__device__ __forceinline__ void fft64_stage(const Fft64Work &w, const double2 *__restrict__ tw, int Ns,
                                            unsigned magic, bool from_in, bool to_out,
                                            const double2 *__restrict__ filter, In in, Out out)
{
    constexpr int PER = fft64_per<PTS>(R);
    // opaque to the compiler, which would otherwise compute every radix's
    // addresses ahead of the stage loop and spill them
    int L = w.L;
    asm volatile("" : "+r"(L));
    const int nj = L / R, items = nj << w.lgT, lg = COL ? w.lgT : 0;
    const int ld = nj << lg, lds = ld + (w.pad ? ld >> 4 : 0);  // a butterfly's stride when read
    double2 a[PER][R];
    int line[PER], first[PER], block[PER];  // a butterfly's line, its j and j / Ns * Ns
    // a thread past the last butterfly repeats it and stores nothing: the
    // registers are written on every path, so none live from stage to stage
    static_for<PER>([&](auto q) {
        const int it = min((int)(threadIdx.x + q * blockDim.x), items - 1);
        const int t = COL ? it & ((1 << w.lgT) - 1) : w.lgT ? it / nj : 0;
        const int j = COL ? it >> w.lgT : it - t * nj;
        line[q] = t;
        first[q] = j;
        block[q] = Ns > 1 ? (int)__umulhi((unsigned)j, magic) * Ns : j;
    });
    if (from_in) {
        static_for<PER>([&](auto q) { static_for<R>([&](auto i) { a[q][i] = in(line[q], first[q] + i * nj); }); });
    } else {
        static_for<PER>([&](auto q) {
            const int n = COL ? (first[q] << lg) + line[q] : first[q] + line[q] * L;
            const double2 *src = w.sm + n + (w.pad ? n >> 4 : 0);
            static_for<R>([&](auto i) { a[q][i] = src[i * lds]; });
            if (Ns > 1) {
                const double2 *wk = tw + (first[q] - block[q]);
                static_for<R - 1>([&](auto i) { a[q][i + 1] = cmul64(a[q][i + 1], __ldg(wk + i * Ns)); });
            }
        });
    }
    static_for<PER>([&](auto q) { Dft64<R>::run(a[q]); });
    if (!to_out) __syncthreads();  // every read of this stage is done
    static_for<PER>([&](auto q) {
        if ((int)(threadIdx.x + q * blockDim.x) < items) {
            const int d0 = block[q] * R + (first[q] - block[q]);
            if (to_out) {
                static_for<R>([&](auto i) { out(line[q], d0 + i * Ns, a[q][i]); });
            } else {
                if (filter)
                    static_for<R>([&](auto i) { a[q][i] = swap64(cmul64(a[q][i], __ldg(filter + d0 + i * Ns))); });
                const int n = COL ? (d0 << lg) + line[q] : d0 + line[q] * L, step = Ns << lg;
                double2 *dst = w.sm + n;
                if (w.pad) {
                    // n's place in its 16 is below step, or step is a multiple of 16
                    dst += n >> 4;
                    static_for<R>([&](auto i) { dst[i * step + ((i * step) >> 4)] = a[q][i]; });
                } else {
                    static_for<R>([&](auto i) { dst[i * step] = a[q][i]; });
                }
            }
        }
    });
    if (!to_out) __syncthreads();
}

template <int PTS, bool COL, class In, class Out>
__device__ __forceinline__ void fft64_transform(const Fft64Work &w, const Fft64Plan &p, bool first_in, bool last_out,
                                                const double2 *filter, In in, Out out)
{
    int Ns = 1;
    const double2 *tw = p.tw;
#pragma unroll 1
    for (int s = 0; s < p.nst; s++) {
        const bool fi = first_in && s == 0, last = s + 1 == p.nst, lo = last_out && last;
        const double2 *f = last ? filter : nullptr;
        const unsigned mg = p.magic[s];
        const int r = p.radix[s];
        switch (r) {
            case 16:
                if constexpr (PTS >= 16) fft64_stage<16, PTS, COL>(w, tw, Ns, mg, fi, lo, f, in, out);
                break;
            case 8: fft64_stage<8, PTS, COL>(w, tw, Ns, mg, fi, lo, f, in, out); break;
            case 7: fft64_stage<7, PTS, COL>(w, tw, Ns, mg, fi, lo, f, in, out); break;
            case 5: fft64_stage<5, PTS, COL>(w, tw, Ns, mg, fi, lo, f, in, out); break;
            case 4: fft64_stage<4, PTS, COL>(w, tw, Ns, mg, fi, lo, f, in, out); break;
            case 3: fft64_stage<3, PTS, COL>(w, tw, Ns, mg, fi, lo, f, in, out); break;
            default: fft64_stage<2, PTS, COL>(w, tw, Ns, mg, fi, lo, f, in, out); break;
        }
        tw += (r - 1) * Ns;
        Ns *= r;
    }
}

// CTA = 2^lgT lines of one array (`lines` lines an array, `groups` CTAs an
// array). ld(array, line, n) and st(array, line, n, v) move the points; swap:
// the backward transform (parts exchanged on the way in and out).
template <int PTS, bool COL, bool BLUESTEIN, class Ld, class St>
__global__ void __launch_bounds__(fft64_max_threads(PTS)) fft64_lines_kernel(Fft64Plan p, int lines, int groups, int lgT, bool swap, Ld ld,
                                                          St st)
{
    extern __shared__ double2 fft64_sm[];
    const int arr = blockIdx.x / groups, line0 = (blockIdx.x % groups) << lgT;
    const Fft64Work w{fft64_sm, p.L, lgT, p.pad};
    auto in = [&](int t, int n) -> double2 {
        double2 v = make_double2(0.0, 0.0);
        if (line0 + t < lines && (!BLUESTEIN || n < p.n)) {
            v = ld(arr, line0 + t, n);
            if (swap) v = swap64(v);
            if (BLUESTEIN) v = cmul64(v, __ldg(p.chirp + n));
        }
        return v;
    };
    auto out = [&](int t, int n, double2 v) {
        if (line0 + t >= lines || (BLUESTEIN && n >= p.n)) return;
        if (BLUESTEIN) {
            v = cmul64(swap64(v), __ldg(p.chirp + n));
            v = make_double2(v.x * p.scale, v.y * p.scale);
        }
        st(arr, line0 + t, n, swap ? swap64(v) : v);
    };
    if (BLUESTEIN) {
        fft64_transform<PTS, COL>(w, p, true, false, p.filter, in, out);
        fft64_transform<PTS, COL>(w, p, false, true, nullptr, in, out);
    } else {
        fft64_transform<PTS, COL>(w, p, true, true, nullptr, in, out);
    }
}

// Threads for 2^lgT lines: enough for every stage's butterflies at once.
template <int PTS>
int fft64_threads(const Fft64Plan &p, int lgT)
{
    int threads = 32;
    for (int k = 0; k < p.nst; k++) {
        const int items = (p.L / p.radix[k]) << lgT, per = fft64_per<PTS>(p.radix[k]);
        threads = threads > (items + per - 1) / per ? threads : (items + per - 1) / per;
    }
    return (threads + 31) & ~31;
}

// Lines a CTA takes: up to 8192 points (2048 for rows, whose lines need no
// neighbour) and 8 columns (128-byte pieces of a row), fewer while the launch
// would leave an SM (of 148) without two CTAs. Two columns at least where they fit, so a
// 32-byte sector is read once.
inline int fft64_lines_lg(const Fft64Plan &p, bool col, int64_t lines)
{
    auto fits = [&](int lg) { return (p.L << lg) <= (col ? 8192 : 2048) && fft64_threads<16>(p, lg) <= 512; };
    int lg = 0;
    while (lg < (col ? 3 : 2) && fits(lg + 1) && (lines >> (lg + 1)) >= 2 * 148) lg++;
    if (col && lg == 0 && lines > 1 && fits(1)) lg = 1;
    return lg;
}

template <bool COL, class Ld, class St>
void launch_fft64_lines(cudaStream_t s, const Fft64Plan &p, int batch, int lines, int sign, Ld ld, St st)
{
    if (batch < 1 || lines < 1) return;
    const int lgT = fft64_lines_lg(p, COL, (int64_t)batch * lines);
    const int groups = (lines + (1 << lgT) - 1) >> lgT;
    const int pts = p.L << lgT;
    const size_t smem = p.nst < 2 && !p.chirp ? 0 : sizeof(double2) * (size_t)(pts + (p.pad ? pts / 16 : 0));
    auto go = [&](auto kernel, int threads) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kernel<<<(unsigned)batch * groups, threads, smem, s>>>(p, lines, groups, lgT, sign > 0, ld, st);
    };
    // 10 points a thread for more warps on an SM; 16 where that would need too
    // many threads and for the convolution lengths' radix 16
    bool wide = false;
    for (int k = 0; k < p.nst; k++) wide = wide || p.radix[k] > 8;
    const int few = fft64_threads<10>(p, lgT);
    if (p.chirp) go(fft64_lines_kernel<16, COL, true, Ld, St>, fft64_threads<16>(p, lgT));
    else if (!wide && few <= fft64_max_threads(10)) go(fft64_lines_kernel<10, COL, false, Ld, St>, few);
    else go(fft64_lines_kernel<16, COL, false, Ld, St>, fft64_threads<16>(p, lgT));
}

}  // namespace rg
