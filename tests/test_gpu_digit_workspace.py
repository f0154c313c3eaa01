"""The digit operands' workspace: chunks of frequencies, pairs and rows (ragged last
ones) give the same bits as one launch, a limit holds, and what does not fit it
runs on the FP64 tensor pipe."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_digit_checks import GEMM, _pad, _ptr, contract, contract_exact, definite, env, p0  # noqa: F401

pytestmark = pytest.mark.gpu


def product(env, a, b):
    torch, ctx = env
    (M, K), N = a.shape, b.shape[0]
    ld = (K + 7) // 8 * 8
    ta, tb = (torch.from_numpy(_pad(x, ld)).cuda() for x in (a, b))
    c = torch.zeros((M, N), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    f = getattr(ctx.lib, GEMM)
    f.restype = C.c_bool
    taken = f(ctx.handle, _ptr(ta), C.c_int(M), C.c_int(ld), _ptr(tb), C.c_int(N), C.c_int(ld), C.c_int(K), _ptr(c),
              C.c_int(N))
    torch.cuda.synchronize()
    return c.cpu().numpy() if taken else None


@pytest.fixture
def limited(env):  # noqa: F811
    yield lambda n: env[1].set_digit_workspace(n)
    env[1].set_digit_workspace(0)


def test_p0_in_chunks(env, limited):  # noqa: F811
    """4, 4 and 2 of 10 frequencies of 2.3 MB in 3/8 of 25 MB."""
    rng = np.random.default_rng(1)
    b = rng.normal(size=(300, 1100))
    b[7] *= 10.0 ** (-4 * rng.uniform(size=1100))
    chi = rng.uniform(0.2, 2.0, (10, 1100))
    one = p0(env, b, chi)
    limited(25 << 20)
    assert np.array_equal(p0(env, b, chi), one)
    limited(5 << 20)  # not one frequency
    dmma = p0(env, b, chi)
    assert np.abs(dmma - one).max() < 1e-12 * np.abs(one).max()
    assert not np.array_equal(dmma, one)


def test_contraction_in_chunks(env, limited):  # noqa: F811
    """512, 512 and 276 of 1300 pairs, 3, 3 and 1 of 7 frequencies of 0.64 MB in 3/8 of 5.5 MB."""
    rng = np.random.default_rng(2)
    wl, b = definite(rng, 300, np.ones(300), 7), rng.normal(size=(1300, 300))
    g = 10.0 ** (-3 * rng.uniform(size=300))
    wl[2] *= np.outer(g, g)
    b[600] /= g
    one = contract(env, b, wl)
    limited(11 << 19)
    assert np.array_equal(contract(env, b, wl), one)
    limited(1 << 20)
    dmma = contract(env, b, wl)
    assert np.abs(dmma / one - 1).max() < 1e-13
    assert not np.array_equal(dmma, one)


def test_product_in_chunks(env, limited):  # noqa: F811
    """256, 256 and 188 of 700 rows of A, 512 and 388 of 900 of B, 1456 bytes each."""
    rng = np.random.default_rng(3)
    a, b = rng.normal(size=(700, 200)), rng.normal(size=(900, 200))
    a[300, 5] = 1e5
    one = product(env, a, b)
    assert np.abs(one - a @ b.T).max() < 1e-12 * np.abs(one).max()
    limited(2 << 20)
    assert np.array_equal(product(env, a, b), one)
    limited(1 << 19)
    assert product(env, a, b) is None


def test_more_frequencies_than_one_group(env):  # noqa: F811
    """Groups of 7 frequencies (8.5 MB of digits each in 60 MB), the last of 5: its
    padding items are skipped alike by loads, MMAs and epilogue."""
    rng = np.random.default_rng(4)
    K, P, nw = 1100, 290, 19
    w = definite(rng, K, np.ones(K), 1)[0]
    scale = np.linspace(0.3, 2.0, nw)
    b = rng.normal(size=(P, K))
    got = contract(env, b, scale[:, None, None] * w)
    ref = contract_exact(b[::37], w[None])[0]
    err = np.abs(got[:, ::37] / (scale[:, None] * ref) - 1).astype(float)
    assert err.max() < 2.0 ** -53 * (6 * np.sqrt(K / 2) + 24)


def test_limit_holds(env):  # noqa: F811
    import torch
    from quasix_b200 import _native
    rng = np.random.default_rng(5)
    wl, b = definite(rng, 420, np.ones(420), 12), rng.normal(size=(6000, 420))
    bov, chi = rng.normal(size=(420, 3000)), rng.uniform(0.2, 2.0, (12, 3000))
    for limit in (0, 48 << 20):  # (the first leaves torch's own blocks cached)
        ctx = _native.Context()
        ctx.set_digit_workspace(limit)
        before = torch.cuda.mem_get_info()[0]
        contract((torch, ctx), b, wl)
        p0((torch, ctx), bov, chi)
        used = before - torch.cuda.mem_get_info()[0]
        ctx.close()
    # (four slots and the status words in the allocator's granules of 2 MB)
    assert used <= (48 << 20) + 5 * (2 << 20)


def test_operands_make_room(env):  # noqa: F811
    """A workspace that fits the device only without the digit operands of an earlier
    call: 120 MB and more of them are held, 90 MB are free, and the rho response of
    40 frequencies at naux 690 takes 150 MB."""
    import torch
    from quasix_b200 import _native
    rng = np.random.default_rng(6)
    nocc, nvir, naux, nf = 2, 40, 690, 40
    e = np.concatenate([np.linspace(-1.0, -0.5, nocc), np.linspace(0.1, 2.0, nvir)])
    lov = rng.normal(size=(naux, nocc, nvir)) * 0.05
    freqs = np.linspace(0.0, 2.0, nf)
    out = np.zeros((nf, naux, naux))
    ctx = _native.Context()
    call = lambda n: ctx.check(ctx.lib.qx_get_rho_response(ctx.handle, n, freqs.ctypes.data, e.ctypes.data, lov.ctypes.data,
                                                           naux, nocc, nvir, 0, out.ctypes.data))
    call(1)
    p0((torch, ctx), rng.normal(size=(690, 4000)), rng.uniform(0.2, 2.0, (8, 4000)))
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - (90 << 20), dtype=torch.uint8, device="cuda")
    try:
        call(nf)
    finally:
        del hog
        torch.cuda.empty_cache()
        ctx.close()
    b = lov.reshape(naux, -1)
    d = (e[:nocc, None] - e[None, nocc:]).reshape(-1)
    ref = 4.0 * (b * (d / (freqs[-1] ** 2 + d * d))) @ b.T
    assert np.abs(out[-1] - ref).max() < 1e-12 * np.abs(ref).max()


def test_bad_context():
    from quasix_b200 import _native
    assert _native.load().qx_ctx_set_digit_workspace(None, 0) != 0
