"""The device functional at the edges of its 32-bin tiles, in both matrix layouts."""
import numpy as np
import pytest

from ermod_openacc_b200 import slvfe as SF

pytestmark = pytest.mark.gpu


def _data(sizes, seed):
    """Species of `sizes` bins each, their correlation matrix of correlated multinomial counts (every
    row sums to the molecule number, as engstore's do), and a solution distribution with an empty core."""
    rng = np.random.default_rng(seed)
    crd, spec, mean, rho, cols = [], [], [], [], []
    for p, n in enumerate(sizes):
        c = np.concatenate([np.linspace(-4.0, -0.03, n // 2), np.linspace(0.03, 25.0, n - n // 2)])
        q = rng.uniform(0.5, 2.0, n) * np.exp(rng.normal(0.0, 0.4, (60, 1)) * np.tanh(c / 3.0))
        number = 100.0 * (p + 1)
        q *= number / q.sum(axis=1, keepdims=True)
        r = q.mean(axis=0) * np.exp(-0.3 * np.tanh(c / 3.0))
        r[-max(1, n // 10):] = 0.0
        crd.append(c); spec.append(np.full(n, p + 1)); mean.append(q.mean(axis=0)); cols.append(q)
        rho.append(r * number / r.sum())
    chi = np.concatenate(cols, axis=1).T @ np.concatenate(cols, axis=1) / 60
    spec = np.concatenate(spec)
    for p, m in enumerate(mean):
        at = np.nonzero(spec == p + 1)[0]
        chi[np.ix_(at, at)] *= 1.0 - 1.0 / (100.0 * (p + 1))
        chi[at, at] += m
    return np.concatenate(rho), np.concatenate(mean), chi, np.concatenate(crd), spec


@pytest.mark.parametrize("sizes,group", [((20,), 1), ((31,), 1), ((32,), 1), ((33,), 1), ((64, 40), 1), ((47, 50), 1),
                                         ((300, 33, 150), 1), ((300, 90), 3), ((1100, 297), 1)])
def test_solve_at_tile_edges(engine_lib, sizes, group):
    """One tile less a bin, a tile, a tile and one, species that start inside a tile, merged bins and
    the size of the default mesh, against the host's FP64 functional.  Both solve a system whose
    condition number is below 1e5 here, so solutions agree to 1e5 x n x 2^-53 < 2e-8 relative;
    the functional is second order in that."""
    rho, rho0, chi, crd, spec = _data(sizes, sum(sizes))
    av = [-1.0 - p for p in range(len(sizes))]
    want = SF.delta_mu(rho, rho0, chi, crd, spec, 300.0, av, group=group)
    for layout in (np.ascontiguousarray, np.asfortranarray):
        info = {}
        got = SF.delta_mu_gpu(rho, rho0, layout(chi), crd, spec, 300.0, av, group=group, info=info)
        np.testing.assert_allclose(got[0], want[0], rtol=2e-8)
        assert not info["used_evd"]


def test_layouts_differ_only_by_transposition(engine_lib):
    """A matrix that is not symmetric (the Cholesky solve rejects it, the eigen-decomposition takes
    it): the two layouts are read as the same matrix."""
    rho, rho0, chi, crd, spec = _data((90, 37), 3)
    chi = chi * (1.0 + 1e-4 * np.random.default_rng(1).normal(size=chi.shape))
    a = SF.delta_mu_gpu(rho, rho0, np.ascontiguousarray(chi), crd, spec, 300.0, [-1.0, -2.0])
    b = SF.delta_mu_gpu(rho, rho0, np.asfortranarray(chi), crd, spec, 300.0, [-1.0, -2.0])
    assert np.array_equal(a[0], b[0])
