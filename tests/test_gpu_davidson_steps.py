"""The device steps of a Davidson solve (Rayleigh-Ritz in shared memory, the
subspace extension, the contracted direct kernel) at the edges of their sizes,
against dense diagonalisation or the oracle's Davidson."""
import numpy as np
import pytest

from oracle import qx_oracle as O
from quasix_b200.synth import make_system

pytestmark = pytest.mark.gpu


def spectrum(kind, n):
    rng = np.random.default_rng(n)
    if kind == "dense":
        a = rng.standard_normal((n, n))
        return 0.5 * (a + a.T)
    if kind == "integers":  # Sturm points fall on diagonal entries
        return np.diag(np.arange(n) - (n - 1) / 2.0)
    if kind == "repeated":
        q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        h = (q * (np.arange(n) // 3)) @ q.T
        return 0.5 * (h + h.T)
    return np.zeros((n, n))


@pytest.mark.parametrize("kind", ["dense", "integers", "repeated", "zero"])
@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17])
def test_ritz_spectra(kind, n):
    """n <= n_roots: all eigenvalues of the matrix, to a backward error of a few n eps |H|."""
    import quasix_b200 as q
    h = spectrum(kind, n)
    got = q.davidson_bse(lambda x: h @ x, np.diag(h).copy(), q.DavidsonConfig(n_roots=n))
    tol = 8 * n * 2.2e-16 * max(np.linalg.norm(h, 2), 1e-300)
    assert np.abs(got["eigenvalues"] - np.linalg.eigvalsh(h)).max() <= tol
    if kind == "dense":
        v = got["eigenvectors"]
        assert np.linalg.norm(h @ v - v * got["eigenvalues"], axis=0).max() <= 4 * tol


@pytest.mark.parametrize("n,roots,space", [(63, 2, 20), (64, 5, 30), (300, 1, 145), (300, 5, 144), (300, 5, 160),
                                           (300, 16, 100), (300, 17, 100), (9600, 3, 30), (200000, 3, 24)])
def test_subspace_steps(n, roots, space):
    """One block to all SMs, staged and unstaged rows, small and large subspaces, restarts."""
    import quasix_b200 as q
    rng = np.random.default_rng(n + space)
    gaps = np.sort(rng.uniform(0.3, 3.0, n))
    gaps[:roots] = 0.2 + 0.01 * np.arange(roots)
    u = rng.standard_normal((n, 4)) * 0.4 / np.sqrt(n)
    op = lambda x: gaps[:, None] * x + u @ (u.T @ x)
    cfg = dict(n_roots=roots, max_iter=300, max_space=space, tol_residual=1e-9)
    got = q.davidson_bse(op, gaps, q.DavidsonConfig(**cfg))
    ref = O.davidson_bse(op, gaps, O.DavidsonConfig(**cfg))
    assert got["all_converged"] and all(ref["converged"])
    assert np.abs(got["eigenvalues"] - ref["eigenvalues"]).max() < 1e-9
    v = got["eigenvectors"]
    assert np.linalg.norm(op(v) - v * got["eigenvalues"], axis=0).max() < 1e-8


@pytest.mark.parametrize("nocc,nvir,roots", [(8, 64, 1), (8, 71, 5), (7, 81, 7)])
def test_contracted_direct_kernel(nocc, nvir, roots):
    """Dimension >= 512: the solve applies the contracted direct kernel; odd row
    counts and more vectors than one pass takes."""
    import quasix_b200 as q
    naux = 90
    s = make_system(nocc, nvir, naux, seed=nocc, pi_norm=2.0)
    dia, dij, dab = O.bse_blocks(s.lpq, nocc)
    w0 = O.bse_w0(s.lpq, s.mo_energy, nocc)
    delta = (s.mo_energy[None, nocc:] - s.mo_energy[:nocc, None]).reshape(-1)
    k = q.BSETDAKernel(nocc, nvir, naux, delta, dia, dij, dab, w0)
    got = k.solve_davidson_with_config(q.DavidsonConfig(n_roots=roots, max_iter=300, tol_residual=1e-8))
    k.close()
    h = O.bse_apply_tda(np.eye(nocc * nvir), delta, dia, dij, dab, w0, nocc, nvir)
    assert got["all_converged"]
    assert np.abs(got["eigenvalues"] - np.linalg.eigvalsh(0.5 * (h + h.T))[:roots]).max() < 1e-9
    v = got["eigenvectors"]
    assert np.linalg.norm(h @ v - v * got["eigenvalues"], axis=0).max() < 2e-8


@pytest.mark.parametrize("nocc,nvir,naux,nvec", [(17, 40, 170, 3), (17, 41, 161, 10), (16, 33, 260, 11), (8, 70, 90, 4),
                                                 (15, 36, 200, 2), (20, 357, 48, 21)])
def test_contracted_apply(nocc, nvir, naux, nvec):
    """Blocks of vectors before and after the contracted direct kernel is formed
    (with and without digits), against the factored oracle."""
    import quasix_b200 as q
    rng = np.random.default_rng(nvec)
    dia, dij, dab = (rng.standard_normal(sh) * 0.05
                     for sh in ((nocc * nvir, naux), (nocc * nocc, naux), (nvir * nvir, naux)))
    w0 = np.eye(naux) + 0.01 * rng.standard_normal((naux, naux))
    w0 = 0.5 * (w0 + w0.T)
    delta = rng.uniform(0.3, 3.0, nocc * nvir)
    k = q.BSETDAKernel(nocc, nvir, naux, delta, dia, dij, dab, w0)
    x = rng.standard_normal((nocc * nvir, nvec))
    ref = O.bse_apply_tda(x, delta, dia, dij, dab, w0, nocc, nvir)
    for _ in range(4):  # factored at first, contracted when that has cost as much
        got = k.apply_hamiltonian_batch(x)
        assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()
    one = k.apply_hamiltonian_batch(np.ascontiguousarray(x[:, :1]))
    k.close()
    assert np.abs(one - ref[:, :1]).max() < 1e-12 * np.abs(ref).max()
