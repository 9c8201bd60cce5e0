"""The FP64 transforms' tables after a failed launch (no GPU): the compiled host
code against a fake CUDA runtime whose launches fail on request. A failed launch
is reported by cudaGetLastError alone; the stream's synchronisation succeeds."""
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

extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
char __cudaInitModule(void **) { return 1; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st)
{
    *g = dim3(1); *b = dim3(1); *s = 0; *(void **)st = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t)
{
    if (fail_from >= 0 && launches++ >= fail_from) return last = cudaErrorLaunchOutOfResources;
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
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    obj = os.path.join(PKG, "_build", "k_fft64.o")
    subprocess.run(["make", "-s", "-C", PKG, obj], check=True)
    d = tmp_path_factory.mktemp("fake")
    (d / "fake.cpp").write_text(FAKE)
    so = str(d / "fake.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-I", os.path.join(PKG, "csrc"),
                    "-o", so, str(d / "fake.cpp"), obj], check=True)
    fn = ct.CDLL(so).probe

    def run(plan, n, nth):
        out = (ct.c_int * 5)()
        fn(int(plan), n, nth, out)
        return list(out)
    return run


# the table of roots; a plan of stages (twiddle launches) and one of Bluestein's
# algorithm (chirp and filter after them), each failing at its first launch and
# the second plan at its last too
@pytest.mark.parametrize("plan,n,nth", [(False, 512, 0), (True, 512, 0), (True, 1030, 0), (True, 1030, 4)])
def test_a_failed_launch_leaves_no_table(probe, plan, n, nth):
    first, again, made, known, none = probe(plan, n, nth)
    assert first != 0
    assert again == 0 and made > nth
    assert known == 0 and none == 0
