"""The FP64 contractions on the integer tensor pipe (csrc/k_digits.cu) at the
edges of their tiles (256 rows, 128 columns, 128 of K), of their K ranges
(16384) and of the rules that choose them (P0: naux >= 256 and nov >= 1024;
contraction: naux > 160).

P0: the digits' worst error per element is below 16 K 2^-56 of the rows'
bounds (see test_digit_model.py); with normal entries 1e-13 of max |Pi| holds
with room.  Sigma: 1e-10 Ha, the bar of the plain path.
"""
import numpy as np
import pytest

from oracle import qx_oracle as O
from quasix_b200.synth import make_system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def q():
    import quasix_b200
    return quasix_b200


def _case(nocc, nvir, naux, seed):
    rng = np.random.default_rng(seed)
    e = np.concatenate([np.sort(rng.uniform(-1.2, -0.3, nocc)), np.sort(rng.uniform(0.05, 3.0, nvir))])
    return e, rng.normal(0.0, 0.05, (naux, nocc, nvir))


@pytest.mark.parametrize("nocc,nvir,naux", [(16, 64, 256), (16, 64, 255), (11, 93, 256), (25, 41, 257), (16, 71, 385),
                                            (20, 64, 511), (128, 128, 256), (113, 145, 260), (130, 253, 300)])
def test_p0_at_tile_edges(q, nocc, nvir, naux):
    e, lov = _case(nocc, nvir, naux, naux)
    freqs = [0.0, 0.4, 30.0]
    got = q.get_rho_response_batch(freqs, e, lov)
    b = lov.reshape(naux, -1)
    d = (e[:nocc, None] - e[None, nocc:]).reshape(-1)
    for k, f in enumerate(freqs):
        ref = 4.0 * (b * (d / (f * f + d * d))) @ b.T
        assert np.abs(got[k] - ref).max() < 1e-13 * np.abs(ref).max()
        if naux >= 256 and nocc * nvir >= 1024:  # the digit kernel stores the lower triangle and its mirror
            assert np.array_equal(got[k], got[k].T)


@pytest.mark.parametrize("scale", [1e-140, 1e140])
def test_p0_scale(q, scale):
    e, lov = _case(16, 64, 256, 1)
    got = q.get_rho_response_batch([0.3], e, lov * scale)[0] + 0.0
    ref = q.get_rho_response_batch([0.3], e, lov)[0]
    # Pi = I - (I - Pi): the identity swallows a tiny Pi and vanishes in a huge one.
    ref = ref * scale * scale
    assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max() + 2.3e-16


def test_p0_graded_weights_take_the_general_path(q):
    """A smallest transition 1/100 of the largest: parity as for any other energies."""
    e, lov = _case(16, 64, 256, 2)
    e[15], e[16] = -0.01, 0.01
    got = q.get_rho_response_batch([0.0, 0.02], e, lov)
    for k, f in enumerate([0.0, 0.02]):
        ref = O.get_rho_response(f, e, lov)
        assert np.abs(got[k] - ref).max() < 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("nocc,nvir,naux,orbs", [(6, 30, 160, None), (6, 30, 161, None), (6, 30, 168, [5, 6]),
                                                 (7, 25, 255, None), (7, 30, 257, [0, 6, 7, 36]), (4, 19, 390, None),
                                                 (5, 18, 511, [4])])
def test_sigma_at_tile_edges(q, nocc, nvir, naux, orbs):
    s = make_system(nocc, nvir, naux, seed=naux, pi_norm=2.0)
    orbs = list(range(nocc + nvir)) if orbs is None else orbs
    got, _ = q.get_sigma_diag(s.mo_energy, s.lpq, orbs, nocc, nw=9)
    ref, _ = O.get_sigma_diag(s.mo_energy, s.lpq, orbs, nocc, nw=9)
    assert np.abs(got - ref).max() < 1e-10


def test_sigma_over_many_frequencies(q):
    """More frequencies than one L2 group of the contraction's item order."""
    s = make_system(9, 35, 200, seed=4, pi_norm=3.0)
    got, _ = q.get_sigma_diag(s.mo_energy, s.lpq, [8, 9], 9, nw=70)
    ref, _ = O.get_sigma_diag(s.mo_energy, s.lpq, [8, 9], 9, nw=70)
    assert np.abs(got - ref).max() < 1e-10


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_tensor_is_reported(q, bad):
    s = make_system(6, 30, 200, seed=5, pi_norm=2.0)
    lpq = s.lpq.copy()
    lpq[3, 5, 6] = lpq[3, 6, 5] = bad
    with pytest.raises(RuntimeError):
        q.get_sigma_diag(s.mo_energy, lpq, [5, 6], 6, nw=8)


@pytest.mark.parametrize("nocc,nvir,naux", [(8, 31, 161), (8, 32, 161), (9, 43, 260)])
def test_adjoint_at_tile_edges(q, nocc, nvir, naux):
    """The adjoint's product over all frequencies (from naux 161 and dimension 256 on)."""
    s = make_system(nocc, nvir, naux, seed=naux, pi_norm=2.0)
    tg, nw = [nocc - 1, nocc], 9
    vxc = np.diag(O.compute_exchange(np.ascontiguousarray(s.lpq[:, :, :nocc].transpose(1, 2, 0))))
    r = q.g0w0_cd(s.mo_energy, s.lpq, nocc, tg, nw=nw, vxc=vxc, tol=1e-13, max_iter=100)
    lam = np.array([1.0, 0.7])
    ge, gl, _ = q.g0w0_cd_grad(s.mo_energy, s.lpq, nocc, tg, r["qp_energies"], lam, nw=nw)
    oe, ol = O.g0w0_cd_grad(s.mo_energy, s.lpq, nocc, tg, r["qp_energies"], lam, nw)
    assert np.abs(ge - oe).max() < 1e-10 * np.abs(oe).max()
    assert np.abs(gl - ol).max() < 1e-10 * np.abs(ol).max()
