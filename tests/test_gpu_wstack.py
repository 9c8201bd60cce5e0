"""W-stacking predict on the device (rg_wstack_predict) against the oracle's
restatement of the reference's wstack_predict (src/wstack/predict.cpp:
396-562) with the same kernels: FP64 on both sides, so the visibilities
agree to rounding; and against the direct sum over the quantised sky."""
import functools
import types

import numpy as np
import pytest

from test_wstack_oracle import case, numpy_predict

pytestmark = pytest.mark.gpu


def _run(ctx, c, **kw):
    return ctx.wstack_predict(c["theta"], c["lam"], c["points"], c["u"], c["v"], c["w"], c["du"], c["dw"], c["x0"],
                              c["conv_uv"], c["conv_w"], c["corr_lm"], c["corr_n"], **kw)


@pytest.mark.parametrize("lam,nv,npts,sw", [(2560.0, 3000, 10, 6), (5120.0, 20000, 25, 4), (2500.0, 777, 3, 6)])
def test_predict_matches_oracle(ctx, sim, oracle, lam, nv, npts, sw):
    c = case(sim, seed=int(lam) + nv, lam=lam, nv=nv, npts=npts, sw=sw)
    got = _run(ctx, c)
    ref = oracle.wstack_predict(c["theta"], c["lam"], c["points"], c["u"], c["v"], c["w"], c["du"], c["dw"],
                                c["x0"], c["conv_uv"], c["conv_w"], c["corr_lm"], c["corr_n"])
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-11
    dft = oracle.predict_dft_quantized(c["theta"], c["lam"], c["points"], c["u"], c["v"], c["w"])
    assert np.linalg.norm(got - dft) / np.linalg.norm(dft) < 2e-3


# few sources go directly, many (and supports above 16) through the stack: one
# visibility or source, part-filled threads, every support class of the direct
# path, a stack side that needs Bluestein's algorithm (412)
@pytest.mark.parametrize("lam,nv,npts,suv,sw", [(1280.0, 1, 1, 8, 6), (1280.0, 257, 33, 8, 6), (1280.0, 500, 7, 6, 8),
                                                (1280.0, 300, 65, 12, 4), (1280.0, 129, 5, 16, 16),
                                                (1280.0, 200, 3, 18, 4), (1280.0, 30, 3000, 8, 6),
                                                (2060.0, 50, 2000, 8, 4)])
def test_predict_direct_and_stack_match_oracle(ctx, sim, oracle, lam, nv, npts, suv, sw):
    c = case(sim, seed=nv + npts, lam=lam, nv=nv, npts=npts, suv=suv, sw=sw)
    got = _run(ctx, c)
    ref = oracle.wstack_predict(c["theta"], c["lam"], c["points"], c["u"], c["v"], c["w"], c["du"], c["dw"],
                                c["x0"], c["conv_uv"], c["conv_w"], c["corr_lm"], c["corr_n"])
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-11


def test_predict_device_buffers_and_errors(rg, ctx, sim):
    torch = pytest.importorskip("torch")
    c = case(sim, seed=5, nv=500)
    host = _run(ctx, c)
    dev = torch.device("cuda", 0)
    d = dict(c)
    for k in ("u", "v", "w"):
        d[k] = torch.from_numpy(c[k]).to(dev)
    out = torch.zeros(500, dtype=torch.complex128, device=dev)
    _run(ctx, d, out=out)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), host)
    bad = dict(c)
    bad["u"] = c["u"] * 10.0  # taps far outside the stack
    with pytest.raises(rg.RGError):
        _run(ctx, bad)
    bad = dict(c)
    bad["points"] = np.array([[0.9 * c["theta"], 0.0]])  # outside the image
    with pytest.raises(rg.RGError):
        _run(ctx, bad)


# a few sources go directly, 3000 through the stack
@pytest.mark.parametrize("nv,npts", [(200, 3), (30, 3000)])
def test_refused_visibility_is_zero_beside_an_infinite_source(rg, ctx, sim, nv, npts):
    """A grid correction of zero makes every source infinite; the visibilities
    whose taps leave the stack, and those that are not finite, come back as zero
    with the error all the same, and only those."""
    c = case(sim, seed=3, lam=1280.0, nv=nv, npts=npts)
    c["corr_n"] = np.zeros_like(c["corr_n"])
    c["u"][nv // 2] *= 1e6
    c["w"][nv - 1] = np.nan
    out = np.full(nv, 7.0 + 7.0j)
    with pytest.raises(rg.RGError):
        _run(ctx, c, out=out)
    zero = np.zeros(nv, bool)
    zero[[nv // 2, nv - 1]] = True
    assert np.all(out[zero] == 0) and not np.isfinite(out[~zero]).any()


@pytest.fixture(scope="module")
def tables(sim):
    """The separable kernels, each made once (seconds)."""
    return types.SimpleNamespace(sepkern_pswf=functools.lru_cache(None)(sim.sepkern_pswf))


# Each way by name, far from where the rule changes over (a factor of three or
# more in the times it compares). Direct: every class of supports, 32 sources
# several times over with a remainder. Stack: many sources, or supports beyond the
# direct kernel's 16; powers of two, and lengths for Bluestein's algorithm, up to
# the largest stack.
@pytest.mark.parametrize("way,lam,nv,npts,suv,sw,dw", [
    ("direct", 5120.0, 300, 70, 12, 4, 50.0), ("direct", 5120.0, 100, 130, 8, 6, 50.0),
    ("direct", 5120.0, 257, 64, 8, 8, 50.0), ("direct", 5120.0, 100, 33, 12, 12, 50.0),
    ("stack", 5120.0, 200, 3000, 8, 6, 50.0), ("stack", 10240.0, 100, 40, 18, 4, 30.0),
    ("stack", 10300.0, 100, 40, 18, 4, 30.0), ("stack", 20480.0, 50, 20, 18, 4, 60.0),
    ("stack", 20420.0, 50, 20, 18, 4, 60.0)])
def test_predict_ways_match_numpy(rg, tables, way, lam, nv, npts, suv, sw, dw):
    c = case(tables, seed=nv + npts, lam=lam, nv=nv, npts=npts, suv=suv, sw=sw, dw=dw)
    ctx = rg.Context(0)  # its own: the largest stack's memory goes with it
    ctx.set_profiling(True)
    got = _run(ctx, c)
    stages = [s for s, _ in ctx.last_timings()]
    ctx.close()
    assert stages == (["wstack_direct"] if way == "direct" else ["wstack_fft", "wstack_degrid"])
    ref = numpy_predict(c)
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-11
