"""The FP64 transforms' host code (no GPU): compiled as it is, against a fake CUDA
runtime that records launches and fails them on request. A failed launch is
reported by cudaGetLastError alone; the stream's synchronisation succeeds."""
import ctypes as ct
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.realpath(__file__)))
PKG = os.path.join(REPO, "radio-gridders_b200")

FAKE = r"""
#include <atomic>
#include <cstdlib>
#include "rg_internal.h"

static int fail_from = -1, launches = 0;
static cudaError_t last = cudaSuccess;

// A recorded launch of a line kernel: which kernel, its blocks, its lines an
// array, its blocks an array and the first element it reads.
struct Line {
    int64_t kernel, blocks, lines, groups, at;
};
static Line *record = nullptr;
static unsigned blocks_x = 0;

extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
char __cudaInitModule(void **) { return 1; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3, size_t, struct CUstream_st *) { blocks_x = g.x; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st)
{
    *g = dim3(1); *b = dim3(1); *s = 0; *(void **)st = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t, cudaStream_t)
{
    if (record)
        record[launches] = Line{(int64_t)f, blocks_x, *(int *)args[1], *(int *)args[2], *(int64_t *)args[5]};
    if (launches++ >= fail_from && fail_from >= 0) return last = cudaErrorLaunchOutOfResources;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError(void) { return last; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
}

namespace rg {
rg_status cuda_fail(cudaError_t, const char *) { return RG_ERR_CUDA; }
rg_status scratch(rg_context *ctx, const char *name, size_t bytes, void **out)
{
    Buffer &b = ctx->scratch[name];
    if (!b.ptr) b = Buffer{std::malloc(bytes), bytes};
    *out = b.ptr;
    return RG_OK;
}
}  // namespace rg

// Status of a table asked for while launches fail from the nth on, then of the
// same table while they work, then the launches of that second call.
extern "C" void probe(int plan, int n, int nth, int *out)
{
    rg_context ctx;
    auto ask = [&]() -> int {
        rg::Fft64Plan p;
        const double2 *roots = nullptr;
        return plan ? rg::fft64_plan(&ctx, n, &p) : rg::roots64(&ctx, n, &roots);
    };
    launches = 0;
    fail_from = nth;
    out[0] = ask();
    launches = 0;
    fail_from = 1 << 30;
    out[1] = ask();
    out[2] = launches;
    launches = 0;
    out[3] = ask();
    out[4] = launches;
}

// The launches of a transform of batch ny x nx arrays at address 0.
extern "C" int lines(int batch, int ny, int nx, Line *out)
{
    rg_context ctx;
    rg::Fft64Plan py, px;
    fail_from = -1;
    if (rg::fft64_plan(&ctx, ny, &py) != RG_OK || rg::fft64_plan(&ctx, nx, &px) != RG_OK) return -1;
    launches = 0;
    record = out;
    rg::launch_fft64_2d(nullptr, nullptr, batch, py, px, -1);
    record = nullptr;
    return launches;
}
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    obj = os.path.join(PKG, "_build", "k_fft64.o")
    subprocess.run(["make", "-s", "-C", PKG, obj], check=True)
    d = tmp_path_factory.mktemp("fake")
    (d / "fake.cpp").write_text(FAKE)
    so = str(d / "fake.so")
    # bound within the file: another library of the process may hold the real runtime
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include", "-I",
                    os.path.join(PKG, "csrc"), "-o", so, str(d / "fake.cpp"), obj], check=True)
    return ct.CDLL(so)


# the table of roots; a plan of stages (twiddle launches) and one of Bluestein's
# algorithm (chirp and filter after them), each failing at its first launch and
# the second plan at its last too
@pytest.mark.parametrize("plan,n,nth", [(False, 512, 0), (True, 512, 0), (True, 1030, 0), (True, 1030, 4)])
def test_a_failed_launch_leaves_no_table(fake, plan, n, nth):
    out = (ct.c_int * 5)()
    fake.probe(int(plan), n, nth, out)
    first, again, made, known, none = out
    assert first != 0
    assert again == 0 and made > nth
    assert known == 0 and none == 0


class Line(ct.Structure):
    _fields_ = [(f, ct.c_int64) for f in ("kernel", "blocks", "lines", "groups", "at")]


# one array, a few, and batches whose rows number 2^31 and more, or just fewer
@pytest.mark.parametrize("batch,ny,nx", [(1, 64, 64), (3, 5, 7), (1 << 30, 2, 2), ((1 << 30) - 1, 2, 3),
                                         ((1 << 31) - 1, 2, 2), (600000, 4096, 2), (600000, 2, 4096)])
def test_every_row_and_column_of_a_batch_is_launched(fake, batch, ny, nx):
    rec = (Line * 64)()
    n = fake.lines(batch, ny, nx, rec)
    assert 2 <= n <= 64 and n % 2 == 0
    rows = cols = 0  # arrays launched so far
    for k in range(n):
        r = rec[k]
        assert 0 < r.blocks < 1 << 31 and 0 < r.groups <= r.blocks and r.blocks % r.groups == 0
        if r.kernel == rec[0].kernel:  # rows: the arrays' rows as lines of one array
            assert r.blocks == r.groups and r.lines % ny == 0 and r.at == 16 * nx * ny * rows
            rows += r.lines // ny
        else:
            assert r.lines == nx and r.at == 16 * nx * ny * cols and rows >= cols + r.blocks // r.groups
            cols += r.blocks // r.groups
    assert rows == batch and cols == batch
