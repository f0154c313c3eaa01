"""Operands that fixed point does not suit: the digit kernels' results stand only
where their error is that of FP64 sums, the rest is formed by the DMMA kernels.

These tests call the library's internal launchers, since through the entry
points the inversion's own rounding hides what a contraction loses on a screened
interaction of small entries.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEMM = "_ZN2qx14gemm_nt_digitsEP6qx_ctxPKdiiS3_iiiPdi"
P0 = "_ZN2qx15launch_eps_fp64EP6qx_ctxPKdiiiS3_iPdimi"
CONTRACT = "_ZN2qx25launch_pair_contract_fp64EP6qx_ctxPKdiiiS3_imiPdi"


@pytest.fixture(scope="module")
def env():
    import torch
    from quasix_b200 import _native
    ctx = _native.Context()
    yield torch, ctx
    ctx.close()


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _pad(a, ld):
    out = np.zeros(a.shape[:-1] + (ld,))
    out[..., :a.shape[-1]] = a
    return out


def contract(env, b, wl):
    """v[w][p] = 2 sum_n b[p][n] sum_k<=n wl[w][n][k] b[p][k]"""
    torch, ctx = env
    (P, K), nw = b.shape, wl.shape[0]
    ld = (K + 7) // 8 * 8
    tb, tw = (torch.from_numpy(_pad(x, ld)).cuda() for x in (b, wl))
    v = torch.full((nw, P), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    getattr(ctx.lib, CONTRACT)(ctx.handle, _ptr(tb), C.c_int(ld), C.c_int(P), C.c_int(K), _ptr(tw), C.c_int(ld),
                               C.c_size_t(K * ld), C.c_int(nw), _ptr(v), C.c_int(P))
    torch.cuda.synchronize()
    return v.cpu().numpy()


def contract_exact(b, wl):
    """In extended precision (64-bit mantissa)."""
    bl, w = b.astype(np.longdouble), wl.astype(np.longdouble)
    return np.stack([2 * (bl * (bl @ np.tril(x).T)).sum(1) for x in w])


def definite(rng, K, g, nw):
    """Half-lower forms of -M M^T scaled by g on both sides."""
    out = []
    for _ in range(nw):
        m = rng.normal(size=(K, K))
        w = -(m @ m.T) / K * np.outer(g, g)
        out.append(np.tril(w, -1) + np.diag(np.diag(w)) / 2)
    return np.stack(out)


@pytest.mark.parametrize("K,P,decades", [(161, 5, 0), (300, 64, 4), (300, 65, 6), (420, 130, 8), (180, 300, -4)])
def test_contraction_of_opposite_grading(env, K, P, decades):
    """Entries of b up where those of W' are down (and alike, negative), one pair
    in three flat.  v = -|M^T g b|^2 has no cancellation beyond its sums': random
    partial sums of K terms round at up to 2^-53 |v| each, K / 4 of them in C and
    K / 4 in v, with 6 standard deviations 6 sqrt(K / 2) 2^-53 |v|; digits that
    stand add their own four (24 with the same allowance)."""
    rng = np.random.default_rng(K + P)
    g = 10.0 ** (-abs(decades) * rng.uniform(size=K))
    wl = definite(rng, K, g, 3)
    b = rng.normal(size=(P, K))
    graded = np.arange(P) % 3 > 0
    b[graded] *= g if decades < 0 else 1 / g
    got, ref = contract(env, b, wl), contract_exact(b, wl)
    err = np.abs((got - ref) / ref).astype(float) * 2.0 ** 53
    assert err.max() < 6 * np.sqrt(K / 2) + 24
    # Not finite in one pair: that pair only.
    b[3, 7] = np.inf
    again = contract(env, b, wl)
    assert not np.isfinite(again[:, 3]).any()
    keep = np.arange(P) != 3
    assert (np.abs((again - ref) / ref).astype(float)[:, keep] * 2.0 ** 53).max() < 6 * np.sqrt(K / 2) + 24


@pytest.mark.parametrize("K,big", [(200, 0.0), (200, 1e3), (500, 1e3), (500, 1e6)])
def test_contraction_of_indefinite_matrices(env, K, big):
    """Wigner matrices, and `big` in one direction: the digits stand up to the rounding
    of FP64 partial sums, of which N |b r| 2^-53 is the estimate (k_gw_f64.cu); six
    deviations of either, or of the K / 2 roundings of v's own sums."""
    rng = np.random.default_rng(K)
    u, b = rng.normal(size=K) / np.sqrt(K), rng.normal(size=(130, K))
    w = rng.normal(size=(2, K, K)) / np.sqrt(K)
    w = w + w.transpose(0, 2, 1) - big * np.outer(u, u)
    wl = np.stack([np.tril(x, -1) + np.diag(np.diag(x)) / 2 for x in w])
    got, ref = contract(env, b, wl), contract_exact(b, wl)
    for k in range(2):
        c = b * (b @ wl[k].T)
        mag = sum(2 * np.abs(c[:, q:q + 64].sum(1)) for q in range(0, K, 64))
        nbr = np.linalg.norm(b, axis=1) * np.sqrt((b * b) @ (wl[k] ** 2).sum(1))
        assert (np.abs(got[k] - ref[k]).astype(float) <= 2.0 ** -53 * 6 * (nbr + np.sqrt(K / 2) * mag)).all()


def test_contraction_of_zeros(env):
    rng = np.random.default_rng(1)
    wl = definite(rng, 200, np.ones(200), 2)
    b = rng.normal(size=(70, 200))
    b[5] = 0.0
    wl[1] = 0.0
    wl[0, 9] = 0.0
    got, ref = contract(env, b, wl), contract_exact(b, wl)
    assert (got[:, 5] == 0).all() and (got[1] == 0).all()
    err = np.abs(got[0] - ref[0])[np.arange(70) != 5] / np.abs(ref[0])[np.arange(70) != 5]
    assert err.astype(float).max() * 2.0 ** 53 < 6 * np.sqrt(100) + 24


def p0(env, b, chi):
    """eps[w] = I + b diag(chi[w]) b^T"""
    torch, ctx = env
    (N, K), nw = b.shape, chi.shape[0]
    ldk, ldn = (K + 7) // 8 * 8, (N + 7) // 8 * 8
    tb, tc = (torch.from_numpy(_pad(x, ldk)).cuda() for x in (b, chi))
    eps = torch.zeros((nw, N, ldn), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    getattr(ctx.lib, P0)(ctx.handle, _ptr(tb), C.c_int(ldk), C.c_int(N), C.c_int(K), _ptr(tc), C.c_int(nw), _ptr(eps),
                         C.c_int(ldn), C.c_size_t(N * ldn), C.c_int(1))
    torch.cuda.synchronize()
    return eps.cpu().numpy()[:, :, :N]


@pytest.mark.parametrize("N,K,rows", [(256, 1023, "normal"), (256, 1024, "normal"), (300, 1100, "normal"),
                                      (511, 1031, "normal"), (257, 1030, "opposite"), (320, 1040, "some opposite"),
                                      (300, 1024, "outliers"), (256, 1025, "zeros")])
def test_p0_of_rough_rows(env, N, K, rows):
    """Rows of B graded over four decades, half of them up where the others are
    down; large single entries; empty rows.  In 2^-53 of the root-sum-square of an
    element's terms: FP64 sums err by 0.3 sqrt(K) (k_digits.cu), two rows that stand
    for their digits by rho rho' / 10 <= 0.63 sqrt(K), 5.5 such deviations among 10^5
    elements; and where the terms have one sign (the diagonal) the K partial sums
    round by up to half an ulp of the value each, sqrt(K) of them in the rms, and
    once to store."""
    rng = np.random.default_rng(N + K)
    b = 3.0 * rng.normal(size=(N, K))
    d = rng.uniform(0.4, 4.0, K)
    chi = np.stack([4 / d, 4 * d / (d * d + 1.0)])
    g = 10.0 ** (-4 * rng.uniform(size=K))
    if rows == "opposite":
        b *= np.where(np.arange(N)[:, None] % 2 == 0, g, 1e-4 / g)
    if rows == "some opposite":
        b[100:103] *= g
        b[257:260] *= 1e-4 / g
    if rows == "outliers":
        b[::5, 7] = 1e6
        b[3::5, 900] = 1e7
    if rows == "zeros":
        b[[0, 100, 255]] = 0.0
    got = p0(env, b, chi)
    bl = b.astype(np.longdouble)
    for w, c in enumerate(chi):
        ref = (bl * c) @ bl.T + np.eye(N)
        rss = np.sqrt((b * b * c * c) @ (b * b).T)
        err = np.abs(got[w] - ref).astype(float)
        bound = 2.0 ** -53 * (3.5 * np.sqrt(K) * rss + (1 + np.sqrt(K)) * np.abs(ref).astype(float))
        assert (err - bound).max() <= 0
        assert np.array_equal(got[w], got[w].T)
    b[7, 11] = np.nan
    bad = ~np.isfinite(p0(env, b, chi))
    assert bad[:, 7].all() and bad[:, :, 7].all() and bad.sum() == 2 * (2 * N - 1)


def test_p0_of_residue_weights(env):
    """Real shifts up to 0.9 of the smallest transition, the transitions over a factor
    of 12: weights within a factor of 64.  The bound of test_p0_of_rough_rows."""
    rng = np.random.default_rng(8)
    N, K = 300, 1400
    b, d = 3.0 * rng.normal(size=(N, K)), rng.uniform(0.35, 4.2, K)
    d[0], d[1] = 0.35, 4.2
    chi = np.stack([4 * d / (d * d - (f * 0.35) ** 2) for f in (0.5, 0.8, 0.9)])
    got, bl = p0(env, b, chi), b.astype(np.longdouble)
    for w, c in enumerate(chi):
        ref = (bl * c) @ bl.T + np.eye(N)
        rss = np.sqrt((b * b * c * c) @ (b * b).T)
        bound = 2.0 ** -53 * (3.5 * np.sqrt(K) * rss + (1 + np.sqrt(K)) * np.abs(ref).astype(float))
        assert (np.abs(got[w] - ref).astype(float) - bound).max() <= 0


@pytest.mark.parametrize("M,N,K,rows", [(256, 256, 161, "normal"), (300, 259, 170, "some opposite"),
                                        (257, 400, 301, "opposite"), (500, 256, 700, "outliers"),
                                        (256, 321, 200, "zeros")])
def test_product_of_rough_rows(env, M, N, K, rows):
    """C = A B^T with the rows of test_p0_of_rough_rows; tiles that stand for their
    digits err by up to sqrt(K) (5.5 such deviations)."""
    torch, ctx = env
    rng = np.random.default_rng(M + K)
    a, b = rng.normal(size=(M, K)), rng.normal(size=(N, K))
    g = 10.0 ** (-4 * rng.uniform(size=K))
    if rows == "opposite":
        a, b = a * g, b * 1e-4 / g
    if rows == "some opposite":
        a[100:103] *= g
        b[257:] *= 1e-4 / g
    if rows == "outliers":
        a[::70, 7] = 1e6
        b[3, 90] = 1e7
    if rows == "zeros":
        a[[0, 100, 255]] = 0.0
        b[320] = 0.0
    ld, ldc = (K + 7) // 8 * 8, N + 3
    ta, tb = (torch.from_numpy(_pad(x, ld)).cuda() for x in (a, b))
    c = torch.full((M, ldc), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    f = getattr(ctx.lib, GEMM)
    f.restype = C.c_bool
    assert f(ctx.handle, _ptr(ta), C.c_int(M), C.c_int(ld), _ptr(tb), C.c_int(N), C.c_int(ld), C.c_int(K), _ptr(c),
             C.c_int(ldc))
    torch.cuda.synchronize()
    got = c.cpu().numpy()
    assert (got[:, N:] == 7.0).all()
    ref = a.astype(np.longdouble) @ b.astype(np.longdouble).T
    rss = np.sqrt((a * a) @ (b * b).T)
    bound = 2.0 ** -53 * (5.5 * np.sqrt(K) * rss + (1 + np.sqrt(K)) * np.abs(ref).astype(float))
    assert (np.abs(got[:, :N] - ref).astype(float) - bound).max() <= 0
