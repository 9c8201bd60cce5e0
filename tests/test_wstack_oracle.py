"""The W-stacking predict oracle (the C restatement of the reference's
wstack_predict, src/wstack/predict.cpp:396-562) against the direct sum over
the quantised sky it approximates (predict_visibility_quantized_vec,
src/wstack/predict.cpp:89-129), with the project's PSWF separable kernels
(simulate.sepkern_pswf).  CPU only.

The reference's own predict cannot be built here (it needs libhdf5, FFTW's
guru interface and its HDF5 kernel files), so its parity is pinned by this
property — a predict equal to the DFT of the same sky within the kernel's
accuracy — and the GPU predict is checked against this oracle."""
import numpy as np
import pytest


def case(sim, seed=0, theta=0.1, lam=2560.0, nv=2000, npts=10, dw=50.0, suv=8, sw=6):
    import oracle
    rng = np.random.default_rng(seed)
    n = int(np.floor(theta * lam))
    du = 1.0 / (2.0 * theta)
    pts = rng.uniform(-0.45 * theta, 0.45 * theta, (npts, 2))
    planes = oracle.wstack_planes(theta, lam, dw, sw)
    lim_u = (n - suv // 2 - 2) * du
    wl = (planes // 2 - sw // 2 - 1) * dw
    u, v = rng.uniform(-lim_u, lim_u, (2, nv))
    w = rng.uniform(-wl, wl, nv)
    cu, ku = sim.sepkern_pswf(suv, 1024, 0.25, corr_oversampling=1024)
    cw, kw = sim.sepkern_pswf(sw, 1024, 0.25, corr_oversampling=1024)
    return dict(theta=theta, lam=lam, points=pts, u=u, v=v, w=w, du=du, dw=dw, x0=0.25, conv_uv=cu, conv_w=cw,
                corr_lm=ku, corr_n=kw)


def test_oracle_predict_matches_quantised_dft(sim, oracle):
    c = case(sim)
    got = oracle.wstack_predict(c["theta"], c["lam"], c["points"], c["u"], c["v"], c["w"], c["du"], c["dw"],
                                c["x0"], c["conv_uv"], c["conv_w"], c["corr_lm"], c["corr_n"])
    ref = oracle.predict_dft_quantized(c["theta"], c["lam"], c["points"], c["u"], c["v"], c["w"])
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 2e-3


def test_oracle_predict_is_linear_in_the_sky(sim, oracle):
    """Two source lists predicted together equal the sum of each alone."""
    c = case(sim, seed=1, npts=6)
    args = (c["u"], c["v"], c["w"], c["du"], c["dw"], c["x0"], c["conv_uv"], c["conv_w"], c["corr_lm"], c["corr_n"])
    a = oracle.wstack_predict(c["theta"], c["lam"], c["points"][:3], *args)
    b = oracle.wstack_predict(c["theta"], c["lam"], c["points"][3:], *args)
    ab = oracle.wstack_predict(c["theta"], c["lam"], c["points"], *args)
    assert np.linalg.norm(ab - (a + b)) / np.linalg.norm(ab) < 1e-12


def numpy_predict(c):
    """The same predict with numpy's FFT, a plane at a time, for stacks too large
    (or of lengths too slow) for the oracle."""
    theta, lam, du, dw = c["theta"], c["lam"], c["du"], c["dw"]
    n = int(np.floor(theta * lam))
    g, (ovuv, suv), (ovw, sw) = 2 * n, c["conv_uv"].shape, c["conv_w"].shape
    planes = int(np.ceil(np.sin(theta / 2) * np.sqrt(2.0 * n * n) / dw)) + sw + 1
    lm, nn = c["corr_lm"].ravel(), c["corr_n"].ravel()
    cell = np.floor((c["points"] / theta + 0.5) * n).astype(int)  # column, row in the unpadded image
    q = cell / lam - theta / 2
    at = np.floor(du * q * lm.size).astype(int) + lm.size // 2
    an = np.floor(dw * (np.sqrt(1.0 - (q * q).sum(1)) - 1.0) * nn.size).astype(int) + nn.size // 2
    val = 1.0 / (lm[at[:, 0]] * lm[at[:, 1]] * nn[an])
    l, m = theta * (cell - n // 2).T / n
    ph = dw * (1.0 - np.sqrt(1.0 - l * l - m * m))
    pos = ((g - n) // 2 + cell + g // 2) % g

    def taps(x, step, table):
        cl = np.ceil(x / step)
        ov = np.floor(np.abs(x - cl * step) / step * table.shape[0]).astype(int)
        return cl.astype(int) - table.shape[1] // 2, table[ov]

    (x0, gu), (y0, gv), (p0, gw) = (taps(c["u"], du, c["conv_uv"]), taps(c["v"], du, c["conv_uv"]),
                                    taps(c["w"], dw, c["conv_w"]))
    cols, rows = x0[:, None] + n + np.arange(suv), y0[:, None] + n + np.arange(suv)
    out = np.zeros(len(c["u"]), complex)
    for p in range(planes):
        a = p - planes // 2 - p0  # the plane's place among a visibility's taps
        on = np.flatnonzero((a >= 0) & (a < sw))
        if not on.size:
            continue
        sky = np.zeros((g, g), complex)
        np.add.at(sky, (pos[:, 1], pos[:, 0]), val * np.exp(2j * np.pi * ((p - planes // 2) * ph)))
        stack = np.fft.fftshift(np.fft.fft2(sky))
        near = stack[rows[on][:, :, None], cols[on][:, None, :]]
        out[on] += gw[on, a[on]] * np.einsum("ky,kx,kyx->k", gv[on], gu[on], near)
    return out


def test_numpy_predict_is_the_oracles(sim, oracle):
    c = case(sim, seed=2, lam=1280.0, nv=60, npts=40)
    ref = oracle.wstack_predict(c["theta"], c["lam"], c["points"], c["u"], c["v"], c["w"], c["du"], c["dw"], c["x0"],
                                c["conv_uv"], c["conv_w"], c["corr_lm"], c["corr_n"])
    assert np.linalg.norm(numpy_predict(c) - ref) / np.linalg.norm(ref) < 1e-12
