"""Eigenvectors of the generalised eigensolver, checked one by one against the matrices they
belong to: G-orthonormality and the residual of every pair."""
import ctypes as C
import math

import numpy as np
import pytest
import scipy.linalg

gpu = pytest.mark.gpu


def _failures(s, g, x, d, eps):
    """Pairs of S x = d G x (columns of x, ascending d) outside their bounds, as text.

    With L L^H = G and y = L^H x the solver works on C = L^-1 S L^-H in precision eps: its
    orthogonal transformations and products leave errors of eps sqrt(n) normwise, taken 32
    times. Orthonormality X^H G X = Y^H Y: the rounded L^-1 and the last product act on
    columns of length ||L|| ||L^-1|| = sqrt(cond G); eigenvectors of the tridiagonal matrix,
    found in FP64 from eigenvalues good to a rounding of the norm, are orthogonal to that
    over their gap (and re-orthogonalised below gaps of 1e-10; the bound of 1e-5 holds for gaps
    about there, and pairs below a tenth of that get none). Residual in the same frame,
    L^-1 (S x - d G x) = C y - d y: relative to ||S|| ||G^-1||, the size of the terms of C."""
    n = s.shape[0]
    tol = 32 * eps * math.sqrt(n)
    g = np.asarray(g, dtype=np.complex128)
    low = np.linalg.cholesky(g)
    y = low.conj().T @ x
    gap = np.abs(d[:, None] - d[None])
    gap64 = np.minimum(8 * np.finfo(np.float64).eps * np.abs(d).max() / np.maximum(gap, 1e-300), 1e-5)
    gap64[gap < 1e-11 * np.abs(d).max()] = 0.0
    orth = np.abs(y.conj().T @ y - np.eye(x.shape[1]))
    bad = ["orthonormality %.2e at %s" % (orth[i, j], (i, j))
           for i, j in zip(*np.nonzero(~(orth <= tol * math.sqrt(np.linalg.cond(g)) + gap64)))]
    size = np.linalg.norm(s, 2) * np.linalg.norm(np.linalg.inv(g), 2)
    res = np.linalg.norm(scipy.linalg.solve_triangular(low, s @ x - (g @ x) * d, lower=True), axis=0) / size
    bad += ["residual %.2e of %d" % (res[i], i) for i in np.nonzero(~(res <= tol))[0]]
    return bad


def _antennas(rng, n):
    """Positions with every pair at least half a wavelength (of 2) apart."""
    side = int(math.ceil(math.sqrt(n)))
    grid = np.stack(np.meshgrid(np.arange(side), np.arange(side)), -1).reshape(-1, 2)[:n] * 3.0
    xyz = np.zeros((n, 3))
    xyz[:, :2] = grid + rng.uniform(-0.9, 0.9, (n, 2))
    return xyz


def _sources(rng, xyz):
    """Visibilities of 8 sources and noise, Hermitian."""
    a = np.exp(1j * np.pi * xyz @ (rng.standard_normal((8, 3)) * 0.1).T)
    noise = rng.standard_normal((len(xyz),) * 2) + 1j * rng.standard_normal((len(xyz),) * 2)
    return (a * rng.uniform(1, 20, 8)) @ a.conj().T + 0.05 * (noise + noise.conj().T)


def _gram(xyz):
    return np.sinc(np.linalg.norm(xyz[:, None] - xyz[None], axis=2))


def _hermitian(s):
    s = np.tril(s).astype(np.complex128)
    s = s + np.tril(s, -1).conj().T
    np.fill_diagonal(s, s.diagonal().real)
    return s


@pytest.mark.parametrize("n", [2, 40, 129, 321])
@pytest.mark.parametrize("eps", [np.finfo(np.float32).eps, np.finfo(np.float64).eps])
def test_checks_see_wrong_vectors(n, eps):
    """The checks pass for scipy's solution rounded to the precision and see a zero, a
    repeated, a turned and an unnormalised eigenvector, of noise and of sources alike."""
    rng = np.random.default_rng(n)
    xyz = _antennas(rng, n)
    s, g = _hermitian(_sources(rng, xyz)), _gram(xyz)
    d, x = scipy.linalg.eigh(s, g)
    if eps > 1e-10:
        d, x = d.astype(np.float32).astype(np.float64), x.astype(np.complex64).astype(np.complex128)
    assert not _failures(s, g, x, d, eps)
    for i in (0, n // 2, n - 1):
        for change in ("zero", "repeat", "turn", "scale"):
            z = x.copy()
            z[:, i] = {"zero": 0 * x[:, i], "repeat": x[:, i - 1], "turn": x[:, i] + 0.02 * x[:, i - 1],
                       "scale": 1.02 * x[:, i]}[change]
            assert _failures(s, g, z, d, eps), (i, change)


@gpu
@pytest.mark.parametrize("n,b", [(2, 3), (31, 2), (64, 2), (65, 1), (96, 40), (97, 3), (129, 1), (200, 2), (257, 1),
                                 (300, 20), (321, 1), (513, 1), (130, 160)])
@pytest.mark.parametrize("precision", ["single", "double"])
def test_eigenvectors_of_batches(ctx, n, b, precision):
    """W = I: single matrices on clusters of CTAs, batches on one CTA each."""
    import bipp_b200 as bipp

    dbl = precision == "double"
    rng = np.random.default_rng(100 * n + b)
    x0 = np.stack([_antennas(rng, n) for _ in range(min(b, 3))])
    s0 = np.stack([_sources(rng, x) for x in x0]).astype(np.complex128 if dbl else np.complex64)
    at = np.arange(b) % len(x0)
    v, d, nred, _ = bipp.eigh_gram_batched(np.full(b, 2.0), s0[at], x0[at], ctx=ctx, precision=precision)
    assert (nred == n).all()
    for k in sorted({0, b // 2, b - 1}):
        x = x0[at[k]] if dbl else x0[at[k]].astype(np.float32).astype(np.float64)
        bad = _failures(_hermitian(s0[at[k]]), _gram(x), v[k].astype(np.complex128), d[k].astype(np.float64),
                        np.finfo(np.float64 if dbl else np.float32).eps)
        assert not bad, (k, len(bad), bad[:4])


@gpu
@pytest.mark.parametrize("beams", [1, 2, 31, 63, 64, 65, 130])
@pytest.mark.parametrize("flagged", [0, 1, 7])
@pytest.mark.parametrize("double", [False, True])
def test_beamformed_eigenvectors(ctx, beams, flagged, double):
    """Orthonormal complex beams of more antennas than beams, some of them flagged: the
    complex factor and inverse at and beside the 64 rows of its one-launch form."""
    import bipp_b200 as bipp

    if flagged >= beams:
        pytest.skip("no beam left")
    rng = np.random.default_rng(10 * beams + flagged)
    rt, ct = (np.float64, np.complex128) if double else (np.float32, np.complex64)
    n = beams + 20
    xyz = _antennas(rng, n).astype(rt)
    w = np.linalg.qr(rng.standard_normal((n, beams)) + 1j * rng.standard_normal((n, beams)))[0].astype(ct)
    s = _sources(rng, xyz.astype(np.float64))
    s = (w.conj().T @ s @ w).astype(ct)
    off = rng.choice(beams, flagged, replace=False)
    s[off] = 0
    s[:, off] = 0
    keep = np.setdiff1d(np.arange(beams), off)
    v, d, nred, _ = bipp.eigh_gram_full(rt(2.0), s, w, xyz, ctx=ctx)
    assert nred == len(keep)
    wk = w[:, keep].astype(np.complex128)
    g = wk.conj().T @ _gram(xyz.astype(np.float64)) @ wk
    g = 0.5 * (g + g.conj().T)
    sk = _hermitian(s[np.ix_(keep, keep)])
    x = np.linalg.lstsq(wk, v[:, :nred].astype(np.complex128), rcond=None)[0]
    eps = np.finfo(rt).eps
    ref = scipy.linalg.eigh(sk, g, eigvals_only=True)
    size = np.linalg.norm(sk, 2) * np.linalg.norm(np.linalg.inv(g), 2)
    assert np.abs(d[:nred] - ref).max() <= 32 * eps * math.sqrt(nred) * size
    assert not d[nred:].any() and not v[:, nred:].any()
    bad = _failures(sk, g, x, d[:nred].astype(np.float64), eps)
    assert not bad, (len(bad), bad[:4])


@gpu
@pytest.mark.parametrize("double", [False, True])
def test_batched_column_major_entries(ctx, double):
    """bipp_eigh_gram_batched_s/_d take the matrices column-major, the _rows_ forms row-major:
    the same results bit for bit, with flagged antennas and over two chunks of steps."""
    import bipp_b200 as bipp
    from bipp_b200._lib import check

    rng = np.random.default_rng(5)
    b, n = 300, 33
    rt, ct = (np.float64, np.complex128) if double else (np.float32, np.complex64)
    xyz = np.stack([_antennas(rng, n) for _ in range(b)]).astype(rt)
    s = np.stack([_sources(rng, x.astype(np.float64)) for x in xyz]).astype(ct)
    for k in range(0, b, 3):
        off = rng.choice(n, 1 + k % 5, replace=False)
        s[k][off] = 0
        s[k][:, off] = 0
    wl = np.full(b, 2.0, dtype=rt)
    v, d, nred, scale = bipp.eigh_gram_batched(wl, s, xyz, ctx=ctx, precision="double" if double else "single")
    fn = ctx._lib.bipp_eigh_gram_batched_d if double else ctx._lib.bipp_eigh_gram_batched_s
    columns, pos = np.ascontiguousarray(s.transpose(0, 2, 1)), np.ascontiguousarray(xyz.transpose(0, 2, 1))
    v2, d2 = np.empty((b, n, n), dtype=ct), np.empty((b, n), dtype=rt)
    nred2, scale2 = np.empty(b, dtype=np.uint64), np.empty(b, dtype=rt)
    check(fn(ctx.handle, b, n, *(a.ctypes.data_as(C.c_void_p) for a in (wl, columns, pos, d2, v2, nred2, scale2))))
    assert np.array_equal(nred, nred2) and len(set(nred2.tolist())) > 3
    assert np.array_equal(scale, scale2) and np.array_equal(d, d2)
    assert np.array_equal(v, v2.transpose(0, 2, 1))


def _degenerate(kind, n):
    """Hermitian matrices with equal, nearly equal or vanishing eigenvalues."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    four = np.repeat([1.0, 2.0, 3.0, 4.0], n // 4 + 1)[:n]
    if kind == "identity":
        return 2.5 * np.eye(n) + 0j
    if kind == "diagonal":
        return np.diag(four) + 0j
    if kind == "clusters":
        q = np.linalg.qr(x)[0]
        return (q * four) @ q.conj().T
    if kind == "two stations":
        return np.kron(np.eye(2), x[:n // 2, :n // 2] + x[:n // 2, :n // 2].conj().T)
    if kind == "pairs":   # Wilkinson's: eigenvalues in pairs that agree to all digits
        return np.diag(np.abs(np.arange(n) - n // 2) + 0.01) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1) + 0j
    if kind == "floor":   # most eigenvalues at a thousandth of the largest
        q = np.linalg.qr(x)[0]
        return (q * 10.0 ** np.linspace(0, -30, n)) @ q.conj().T + 1e-3 * np.eye(n)
    rank = {"ones": 0, "rank 3": 3, "half rank": n // 2}[kind]
    return x[:, :rank] @ x[:, :rank].conj().T if rank else np.ones((n, n)) + 0j


@gpu
@pytest.mark.parametrize("kind", ["identity", "diagonal", "clusters", "two stations", "pairs", "floor", "ones", "rank 3",
                                  "half rank"])
@pytest.mark.parametrize("n", [2, 6, 40, 96, 130, 258])
@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("gram", [False, True])
def test_equal_eigenvalues(ctx, kind, n, double, gram):
    """Equal eigenvalues get orthonormal eigenvectors of their space, as LAPACK's ?hegv gives."""
    import bipp_b200 as bipp

    rt, ct = (np.float64, np.complex128) if double else (np.float32, np.complex64)
    s = _hermitian(_degenerate(kind, n).astype(ct))
    xyz = _antennas(np.random.default_rng(1), n).astype(rt)
    eye = np.eye(n, dtype=ct)
    if gram:
        g = _gram(xyz.astype(np.float64))
        v, d, nred, _ = bipp.eigh_gram_full(rt(2.0), s.astype(ct), eye, xyz, ctx=ctx)
    else:
        g = np.eye(n)
        v, d, nred, _ = bipp.eigh(rt(2.0), s.astype(ct), eye, ctx=ctx, full=True)
    assert nred == n
    eps = np.finfo(rt).eps
    ref = scipy.linalg.eigh(s, g, eigvals_only=True)
    size = np.linalg.norm(s, 2) * np.linalg.norm(np.linalg.inv(g), 2)
    assert np.abs(d - ref).max() <= 32 * eps * math.sqrt(n) * size
    bad = _failures(s, g, v.astype(np.complex128), d.astype(np.float64), eps)
    assert not bad, (len(bad), bad[:4])


@gpu
@pytest.mark.parametrize("kind", ["two stations", "ones", "rank 3", "half rank"])
def test_equal_eigenvalues_in_a_batch(ctx, kind):
    """Beside matrices without any, over two chunks, and in a range of the spectrum."""
    import bipp_b200 as bipp

    rng = np.random.default_rng(3)
    b, n = 260, 24
    xyz = np.stack([_antennas(rng, n)] * b).astype(np.float32)
    s = np.stack([_sources(rng, xyz[0].astype(np.float64)) for _ in range(4)] * (b // 4)).astype(np.complex64)
    with_equal = [0, 5, 131, 259]
    s[with_equal] = _degenerate(kind, n)
    g = _gram(xyz[0].astype(np.float64))
    v, d, nred, _ = bipp.eigh_gram_batched(np.full(b, 2.0), s, xyz, ctx=ctx)
    for k in with_equal + [1, 258]:
        bad = _failures(_hermitian(s[k]), g, v[k].astype(np.complex128), d[k].astype(np.float64), np.finfo(np.float32).eps)
        assert nred[k] == n and not bad, (k, len(bad), bad[:4])


@gpu
@pytest.mark.parametrize("n", [130, 500, 700, 1030])
def test_reduction_of_an_exact_low_rank_matrix(ctx, n):
    """All ones in FP32: what is left of the matrix shrinks by a rounding per column, and its
    squares underflow after three (1030 rows: the panel kernel, 130 and more the clusters)."""
    import bipp_b200 as bipp

    s = np.ones((n, n), np.complex64)
    v, d, nred, _ = bipp.eigh(np.float32(2.0), s, np.eye(n, dtype=np.complex64), ctx=ctx, full=True)
    bad = _failures(s.astype(np.complex128), np.eye(n), v.astype(np.complex128), d.astype(np.float64),
                    np.finfo(np.float32).eps)
    assert nred == n and not bad, (len(bad), bad[:4])
