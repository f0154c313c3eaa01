"""A call on a BSE kernel object depends on its arguments, not on the calls before
it: the contracted direct kernel belongs to one solve (dimension 1024 and up)."""
import numpy as np
import pytest

from oracle import qx_oracle as O

pytestmark = pytest.mark.gpu


def _kernel(nocc, nvir, naux, seed):
    import quasix_b200 as q
    rng = np.random.default_rng(seed)
    dia, dij, dab = (rng.standard_normal(sh) * 0.1 / np.sqrt(naux)
                     for sh in ((nocc * nvir, naux), (nocc, nocc, naux), (nvir, nvir, naux)))
    dij = (dij + dij.transpose(1, 0, 2)).reshape(-1, naux)
    dab = (dab + dab.transpose(1, 0, 2)).reshape(-1, naux)
    w0 = np.eye(naux)
    delta = rng.uniform(0.3, 3.0, nocc * nvir)
    ref = lambda x: O.bse_apply_tda(x, delta, dia, dij, dab, w0, nocc, nvir)
    return q.BSETDAKernel(nocc, nvir, naux, delta, dia, dij, dab, w0), ref


def test_apply_is_the_same_before_and_after():
    """More vectors than forming the contracted kernel costs, and a solve, between two
    applications to the same block: the same bits, and no memory kept."""
    import torch
    import quasix_b200 as q
    k, ref = _kernel(16, 81, 200, 1)
    x = np.random.default_rng(2).standard_normal((16 * 81, 7))
    first = k.apply_hamiltonian_batch(x)
    assert np.abs(first - ref(x)).max() < 1e-12 * np.abs(first).max()
    for _ in range(4):
        assert np.array_equal(k.apply_hamiltonian_batch(x), first)
    cfg = q.DavidsonConfig(n_roots=3, max_iter=300, tol_residual=1e-8)
    one = k.solve_davidson_with_config(cfg)
    free = torch.cuda.mem_get_info()[0]
    assert np.array_equal(k.apply_hamiltonian_batch(x), first)
    two = k.solve_davidson_with_config(cfg)
    assert torch.cuda.mem_get_info()[0] >= free  # (nov^2 doubles are 13 MB)
    k.close()
    assert np.array_equal(one["eigenvalues"], two["eigenvalues"])
    assert np.array_equal(one["eigenvectors"], two["eigenvectors"])


@pytest.mark.parametrize("nocc,nvir,naux,roots", [(16, 64, 161, 1), (17, 61, 170, 5), (13, 81, 90, 12), (8, 357, 48, 11)])
def test_solve_with_contracted_kernel(nocc, nvir, naux, roots):
    """With and without digits, odd row counts, more vectors than one pass takes."""
    import quasix_b200 as q
    k, ref = _kernel(nocc, nvir, naux, roots)
    got = k.solve_davidson_with_config(q.DavidsonConfig(n_roots=roots, max_iter=400, max_space=120, tol_residual=1e-8))
    k.close()
    h = ref(np.eye(nocc * nvir))
    assert got["all_converged"]
    assert np.abs(got["eigenvalues"] - np.linalg.eigvalsh(0.5 * (h + h.T))[:roots]).max() < 1e-9
    v = got["eigenvectors"]
    assert np.linalg.norm(h @ v - v * got["eigenvalues"], axis=0).max() < 2e-8
