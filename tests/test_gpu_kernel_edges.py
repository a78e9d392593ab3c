"""Kernels at the sizes where they can go wrong (tile edges, remainders, the smallest and
largest of a range), against FP64 numpy/scipy of the same definition."""
import math

import numpy as np
import pytest

from oracle import bluebild as bb

pytestmark = pytest.mark.gpu


def _rel_l2(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300)


def _points(rng, n, umax, wmax, images):
    u, v = rng.uniform(-umax, umax, (2, n))
    w = rng.uniform(-wmax, wmax, n) if wmax else np.zeros(n)
    c = rng.standard_normal((n, images)) + 1j * rng.standard_normal((n, images))
    return np.stack([u, v, w], 1).astype(np.float32), c.astype(np.complex64)


def _check_nufft(ctx, lmn, uvw, c, tol, bound):
    import bipp_b200 as bipp

    plan = bipp.NufftSynthesis(ctx, bipp.NufftSynthesisOptions().set_tolerance(tol), lmn, c.shape[1], uvw.shape[0])
    plan.add(uvw, c)
    l64, uvw64 = lmn.astype(np.float64), uvw.astype(np.float64)
    pix = np.random.default_rng(3).choice(lmn.shape[0], min(lmn.shape[0], 3000), replace=False)
    for i in range(c.shape[1]):
        ref = bb.nuft_sum(1.0, c[:, i].astype(np.complex128), uvw64[:, 0], uvw64[:, 1], uvw64[:, 2], l64[pix, 0],
                          l64[pix, 1], l64[pix, 2])
        assert _rel_l2(plan.get_image(i)[pix], ref) <= bound, i
    plan.close()


@pytest.mark.parametrize("images", [3, 4])
@pytest.mark.parametrize("tol", [1e-3, 1e-5, 1e-7])
def test_spread_more_than_eight_channels(ctx, images, tol):
    """9 and 12 channels (3 and 4 images with their first-order lattice channels): two
    tensor-core spreading launches. Bound as for up to 8 channels: 20 tolerances, at least 2e-6."""
    from bipp_b200 import simulate as sim

    rng = np.random.default_rng(21)
    lmn = sim.make_lmn_grid(45, math.radians(12.0)).astype(np.float32)
    uvw, c = _points(rng, 900, 4000.0, 200.0, images)
    _check_nufft(ctx, lmn, uvw, c, tol, max(20 * tol, 2e-6))


@pytest.mark.parametrize("px", [585, 1755, 2926, 4096])
def test_fft_lines_with_factor_1024(ctx, px):
    """Image widths whose fine grid is 1024 times 1, 3, 5 or 7 (radices .., 16, 16, 4)."""
    rng = np.random.default_rng(22)
    na = 9
    a, b = np.meshgrid(np.arange(na), np.arange(px), indexing="ij")
    for transposed in (False, True):
        l = (b.reshape(-1) - px / 2 + 0.5) * (0.2 / px)
        m = (a.reshape(-1) - na / 2 + 0.25) * (0.02 / na)
        if transposed:
            l, m = (l.reshape(na, px).T.reshape(-1), m.reshape(na, px).T.reshape(-1))
        lmn = np.stack([l, m, np.sqrt(1 - l * l - m * m)], 1).astype(np.float32)
        uvw, c = _points(rng, 500, 500.0, 20.0, 1)
        _check_nufft(ctx, lmn, uvw, c, 1e-6, 2e-5)


@pytest.mark.parametrize("tol", [1e-2, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("wmax", [0.0, 30.0, 333.0, 2500.0])
def test_w_planes(ctx, wmax, tol):
    """No w extent at all, and extents whose planes end at different places of a tile layer."""
    from bipp_b200 import simulate as sim

    rng = np.random.default_rng(23)
    lmn = sim.make_lmn_grid(33, math.radians(16.0)).astype(np.float32)
    uvw, c = _points(rng, 400, 1500.0, wmax, 1)
    _check_nufft(ctx, lmn, uvw, c, tol, 20 * tol)


@pytest.mark.parametrize("n_in,n_out", [(1, 1), (255, 257), (256, 256), (257, 300), (9000, 65)])
@pytest.mark.parametrize("double", [False, True])
def test_direct_sum_sizes(ctx, n_in, n_out, double):
    """FP32: sine and cosine within 2^-20 each and the FP32 result, so 2e-6 of the summed
    magnitudes. FP64: phases below 2e3 rounded to 2^-52 of that, 1e-11 of them."""
    import bipp_b200 as bipp

    rng = np.random.default_rng(n_in + n_out)
    rt, ct = (np.float64, np.complex128) if double else (np.float32, np.complex64)
    u = rng.uniform(-900, 900, (3, n_in)).astype(rt)
    x = rng.uniform(-1, 1, (3, n_out)).astype(rt)
    v = (rng.standard_normal(n_in) + 1j * rng.standard_normal(n_in)).astype(ct)
    out = bipp.nuft_sum(rt(1.25), v, u[0], u[1], u[2], x[0], x[1], x[2], ctx=ctx)
    ref = (np.exp(1j * 1.25 * (x.astype(np.float64).T @ u.astype(np.float64))) @ v.astype(np.complex128)).real
    assert np.abs(out - ref).max() <= (1e-11 if double else 2e-6) * np.abs(v).sum()


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e30])
def test_direct_sum_out_of_range(ctx, bad):
    """A non-finite input coordinate or value reaches every output as NaN; a huge finite one
    stays finite; a non-finite pixel only its own output."""
    import bipp_b200 as bipp

    rng = np.random.default_rng(7)
    base = [rng.uniform(-1, 1, 300).astype(np.float32) for _ in range(3)]
    pix = [rng.uniform(-1, 1, 40).astype(np.float32) for _ in range(3)]
    val = np.ones(300, np.complex64)
    u = base[0].copy()
    u[17] = bad
    out = bipp.nuft_sum(np.float32(1.0), val, u, base[1], base[2], *pix, ctx=ctx)
    assert np.isfinite(out).all() if bad == 1e30 else np.isnan(out).all()
    if bad != 1e30:
        v = val.copy()
        v[3] = bad
        assert not np.isfinite(bipp.nuft_sum(np.float32(1.0), v, *base, *pix, ctx=ctx)).any()
        x = pix[0].copy()
        x[5] = bad
        out = bipp.nuft_sum(np.float32(1.0), val, *base, x, pix[1], pix[2], ctx=ctx)
        assert np.isnan(out[5]) and np.isfinite(np.delete(out, 5)).all()


def _steps(rng, b, n, dtype):
    """b Hermitian visibility matrices of n antennas (sources plus noise) and positions with
    every pair at least half a wavelength apart."""
    side = int(math.ceil(math.sqrt(n)))
    grid = np.stack(np.meshgrid(np.arange(side), np.arange(side)), -1).reshape(-1, 2)[:n] * 3.0
    xyz = np.zeros((b, n, 3))
    xyz[:, :, :2] = grid + rng.uniform(-0.9, 0.9, (b, n, 2))
    q = 8
    dirs = rng.standard_normal((b, q, 3)) * 0.1
    a = np.exp(1j * np.pi * np.einsum("bqc,bnc->bnq", dirs, xyz))
    noise = rng.standard_normal((b, n, n)) + 1j * rng.standard_normal((b, n, n))
    s = np.einsum("bnq,q,bmq->bnm", a, rng.uniform(1, 20, q), a.conj()) + 0.05 * (noise + noise.conj().transpose(0, 2, 1))
    return s.astype(dtype), xyz


@pytest.mark.parametrize("n,b", [(1, 3), (2, 1), (31, 2), (33, 5), (63, 1), (64, 2), (65, 2), (96, 1), (127, 3), (129, 1),
                                 (200, 2), (257, 1), (321, 1), (513, 1), (40, 400), (130, 40)])
@pytest.mark.parametrize("precision", ["single", "double"])
def test_eigh_gram_sizes(ctx, n, b, precision):
    """Sizes around the tiles and panels of the Cholesky factor, inverse, tridiagonalisation
    and eigenpairs, alone and in batches. Eigenvalues against scipy's FP64 solver on the same
    inputs, and eigenvectors that reconstruct S: normwise 64 eps sqrt(n) for FP64 and 32 eps
    sqrt(n) for FP32 (a backward stable solver stays below n eps)."""
    import scipy.linalg

    import bipp_b200 as bipp

    rng = np.random.default_rng(1000 * n + b)
    dbl = precision == "double"
    s, xyz = _steps(rng, b, n, np.complex128 if dbl else np.complex64)
    wl = np.full(b, 2.0)
    v, d, nred, _ = bipp.eigh_gram_batched(wl, s, xyz, ctx=ctx, precision=precision)
    assert (nred == n).all()
    eps = np.finfo(np.float64 if dbl else np.float32).eps
    tol = (64 if dbl else 32) * eps * math.sqrt(n)
    for k in sorted(set([0, b // 2, b - 1])):
        x = xyz[k] if dbl else xyz[k].astype(np.float32).astype(np.float64)
        g = np.sinc(np.linalg.norm(x[:, None] - x[None], axis=2))
        s64 = np.tril(s[k]).astype(np.complex128)
        s64 = s64 + np.tril(s64, -1).conj().T
        np.fill_diagonal(s64, s64.diagonal().real)
        ref = scipy.linalg.eigh(s64, g, eigvals_only=True)
        scale = np.abs(ref).max()
        cond = np.linalg.cond(g)
        assert np.abs(d[k] - ref).max() <= tol * scale * max(1.0, math.sqrt(cond)), k
        vk = v[k].astype(np.complex128)
        assert np.linalg.norm(g @ (vk * d[k]) @ vk.conj().T @ g - s64) <= tol * n * cond * scale, k


@pytest.mark.parametrize("n,b", [(896, 223), (897, 185), (897, 186)])
def test_eigenvalues_of_many_large_matrices(ctx, n, b):
    """Batches around the sizes from which a matrix takes one CTA of the panel kernel; most
    antennas are flagged (zero rows). FP32 eigenvalues against scipy's FP64 solver, 32 eps
    sqrt(kept) normwise as above."""
    import scipy.linalg

    import bipp_b200 as bipp

    rng = np.random.default_rng(n + b)
    kept = 45
    s0, x0 = _steps(rng, 3, kept, np.complex64)
    s = np.zeros((b, n, n), dtype=np.complex64)
    xyz = np.zeros((b, n, 3))
    xyz[:, :, 2] = 10.0 + np.arange(n)
    at = np.sort(rng.choice(n, kept, replace=False))
    for k in range(b):
        s[k][np.ix_(at, at)] = s0[k % 3]
        xyz[k, at] = x0[k % 3]
    _, d, nred, _ = bipp.eigh_gram_batched(np.full(b, 2.0), s, xyz, ctx=ctx)
    assert (nred == kept).all()
    tol = 32 * np.finfo(np.float32).eps * math.sqrt(kept)
    for k in (0, 1, b - 1):
        x = x0[k % 3].astype(np.float32).astype(np.float64)
        g = np.sinc(np.linalg.norm(x[:, None] - x[None], axis=2))
        s64 = np.tril(s0[k % 3]).astype(np.complex128)
        s64 = s64 + np.tril(s64, -1).conj().T
        np.fill_diagonal(s64, s64.diagonal().real)
        ref = scipy.linalg.eigh(s64, g, eigvals_only=True)
        bound = tol * np.abs(ref).max() * max(1.0, math.sqrt(np.linalg.cond(g)))
        assert np.abs(d[k][:kept] - ref).max() <= bound, k


@pytest.mark.parametrize("px", [11, 26, 41, 63, 114, 200, 274, 343, 514, 900, 1200])
def test_fft_lines_with_several_odd_factors(ctx, px):
    """Image widths whose fine grids have more than one odd factor (among them 48, 144, 240,
    432, 1575 -> 1600, 2100 -> 2160 cells) or are small, along either axis of the image."""
    rng = np.random.default_rng(24)
    na = 20
    a, b = np.meshgrid(np.arange(na), np.arange(px), indexing="ij")
    for transposed in (False, True):
        l = (b.reshape(-1) - px / 2 + 0.5) * (0.2 / px)
        m = (a.reshape(-1) - na / 2 + 0.25) * (0.03 / na)
        if transposed:
            l, m = (l.reshape(na, px).T.reshape(-1), m.reshape(na, px).T.reshape(-1))
        lmn = np.stack([l, m, np.sqrt(1 - l * l - m * m)], 1).astype(np.float32)
        uvw, c = _points(rng, 500, 400.0, 20.0, 1)
        _check_nufft(ctx, lmn, uvw, c, 1e-6, 2e-5)


@pytest.mark.parametrize("n", [24, 40, 130, 300])
@pytest.mark.parametrize("power", [-60, -300, -505, -514, -517, -519, -522, -600])
def test_nearly_decoupled_tridiagonal(ctx, n, power):
    """Tridiagonal FP64 matrices whose couplings are tiny, so that eigenvalues meet diagonal
    entries exactly and products of pivots pass the smallest numbers. The eigenvalues are the
    diagonal to a rounding of the norm each way (4 eps), the eigenvectors unit vectors to 64
    eps (the couplings, below 2^-60, over gaps of 1 / 2 n, are far less)."""
    import bipp_b200 as bipp

    d0 = 0.5 + (np.arange(n) * 7 % n + 0.25) / (2.0 * n) if n % 7 else 0.5 + np.arange(n) / (2.0 * n)
    e = np.full(n - 1, 2.0 ** power)
    s = np.diag(d0) + np.diag(e, -1) + np.diag(e, 1)
    v, d, nred, _ = bipp.eigh(2.0, s.astype(np.complex128), np.eye(n), ctx=ctx, full=True)
    eps = np.finfo(np.float64).eps
    order = np.argsort(d0)
    assert nred == n
    assert np.abs(d - d0[order]).max() <= 4 * eps
    assert np.abs(np.abs(v[order, :]) - np.eye(n)).max() <= 64 * eps


@pytest.mark.parametrize("n", [100, 301, 512])
@pytest.mark.parametrize("top", [3.0, 4.0, 8.0, 100.0])
def test_eigenvalue_width(ctx, n, top):
    """Eigenvalues of the second difference matrix, 2 cos(pi k / (n + 1)), beside one decoupled
    entry that sets the norm, in FP64. Bisection ends at a width of half a rounding of the
    norm, so the error is uniform within eps / 4 of it: 0.144 eps in the mean square, and 0.2
    eps allowed with the counts' own roundings (ending at a whole one gives up to 0.289)."""
    import bipp_b200 as bipp

    ld = np.longdouble
    exact = np.sort(2 * np.cos(np.arange(1, n + 1).astype(ld) * (4 * np.arctan(ld(1))) / (n + 1)))
    s = np.zeros((n + 1, n + 1), dtype=np.complex128)
    s[np.arange(1, n), np.arange(n - 1)] = 1.0
    s[np.arange(n - 1), np.arange(1, n)] = 1.0
    s[n, n] = top
    _, d, nred, _ = bipp.eigh(2.0, s, np.eye(n + 1), ctx=ctx, full=True)
    assert nred == n + 1
    err = (d[:n].astype(ld) - exact)[np.abs(exact) <= top / 2]
    assert np.sqrt(np.mean(err ** 2)) <= 0.2 * np.finfo(np.float64).eps * top


@pytest.mark.parametrize("umax", [10.0, 900.0, 3e4])
def test_direct_sum_double_phases(ctx, umax):
    """FP64 direct sums against 80-bit ones: no further off than the plain FP64 form of the
    phase, alpha x rounded and every product and sum of it, which rounds more often than the
    kernel's multiply-adds; 1.1 for the sampling of 600 outputs of 2000 terms."""
    import bipp_b200 as bipp

    ld = np.longdouble
    twopi = 8 * np.arctan(ld(1))
    got, plain = [], []
    for seed in range(12):
        rng = np.random.default_rng(seed)
        u, x = rng.uniform(-umax, umax, (3, 2000)), rng.uniform(-1, 1, (3, 50))
        v = rng.standard_normal(2000) + 1j * rng.standard_normal(2000)
        alpha = 1.25 * (1 + 0.3 * rng.random())

        def total(phase):
            phase = phase.astype(ld)
            phase = phase - twopi * np.round(phase / twopi)
            return (np.cos(phase) * v.real - np.sin(phase) * v.imag).sum(1)

        ref = total(ld(alpha) * (x.astype(ld).T @ u.astype(ld)))
        xa = (alpha * x).T
        p = xa[:, 0, None] * u[0] + xa[:, 1, None] * u[1] + xa[:, 2, None] * u[2]
        out = bipp.nuft_sum(alpha, v, u[0], u[1], u[2], x[0], x[1], x[2], ctx=ctx)
        # the sum itself rounds too, in FP64 on either side: a real and an imaginary product per
        # term, added in turn
        both = np.stack([np.cos(p) * v.real, -np.sin(p) * v.imag], 2).reshape(len(p), -1)
        plain.append((total(p) - ref) + (both.cumsum(1)[:, -1] - both.astype(ld).sum(1)))
        got.append(out - ref)
    assert np.sqrt(np.mean(np.square(got))) <= 1.1 * np.sqrt(np.mean(np.square(plain)))


def _both_spreaders(ctx, monkeypatch, lmn, uvw, c, tol):
    """Images of more than 8 channels by default and with the shared-memory atomics."""
    import bipp_b200 as bipp

    out = []
    for warp in (False, True):
        if warp:
            monkeypatch.setenv("BIPP_B200_SPREAD", "warp")
        plan = bipp.NufftSynthesis(ctx, bipp.NufftSynthesisOptions().set_tolerance(tol), lmn, c.shape[1], uvw.shape[0])
        plan.add(uvw, c)
        out.append(np.stack([plan.get_image(i) for i in range(c.shape[1])]).astype(np.float64))
        plan.close()
    return out


@pytest.mark.parametrize("images,tol", [(3, 1e-5), (4, 1e-4), (4, 1e-5)])
@pytest.mark.parametrize("values", ["sky", "noise", "heavy"])
def test_more_than_eight_channels_keep_single_precision(ctx, monkeypatch, images, tol, values):
    """9 and 12 channels on the tensor cores against the spreader with FP32 products and sums,
    whose transform they share, so that only operands and sums differ: dropped products of
    2^-22, FP32 additions on either side, 1e-6 (2^-20) in all. Heavy tiles of short baselines,
    point sources whose values add up in phase, and values that span four decades."""
    from bipp_b200 import simulate as sim

    rng = np.random.default_rng(31)
    n = 20000
    lmn = sim.make_lmn_grid(64, math.radians(12.0)).astype(np.float32)
    r, a = np.exp(rng.uniform(np.log(20), np.log(4000), n)), rng.uniform(0, 2 * np.pi, n)
    uvw = np.stack([r * np.cos(a), r * np.sin(a), rng.uniform(-200, 200, n)], 1).astype(np.float32)
    c = rng.standard_normal((n, images)) + 1j * rng.standard_normal((n, images))
    if values == "sky":
        lm = rng.uniform(-0.1, 0.1, (12, 2))
        at = np.concatenate([lm, np.sqrt(1 - (lm ** 2).sum(1))[:, None]], 1)
        c = np.exp(-1j * uvw.astype(np.float64) @ at.T) @ np.exp(rng.uniform(-4, 2, (12, images)))
    elif values == "heavy":
        c[20:] *= 1e-4
    tc, warp = _both_spreaders(ctx, monkeypatch, lmn, uvw, c.astype(np.complex64), tol)
    for i in range(images):
        assert _rel_l2(tc[i], warp[i]) <= 1e-6, i
    assert not np.array_equal(tc, warp)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 17, 32, 33, 48, 49, 2049, 5000])
def test_more_than_eight_channels_point_counts(ctx, monkeypatch, n):
    """Points of one place of the grid, so that its tiles get exactly n: phases that are not
    full, one or two accumulators in use, tiles spread in parts. Bound as above, of the terms'
    mean square (the same phase at every point lets an image's terms cancel)."""
    from bipp_b200 import simulate as sim

    rng = np.random.default_rng(n)
    lmn = sim.make_lmn_grid(40, math.radians(12.0)).astype(np.float32)
    uvw = (np.array([1234.0, -777.0, 111.0]) + rng.uniform(-0.5, 0.5, (n, 3))).astype(np.float32)
    c = (rng.standard_normal((n, 4)) + 1j * rng.standard_normal((n, 4))).astype(np.complex64)
    tc, warp = _both_spreaders(ctx, monkeypatch, lmn, uvw, c, 1e-5)
    size = np.linalg.norm(c, axis=0) * math.sqrt(lmn.shape[0] / 2)
    for i in range(4):
        assert np.linalg.norm(tc[i] - warp[i]) <= 1e-6 * size[i], i
