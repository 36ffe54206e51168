"""The point-by-point kernels behind the operators: the divergence's cc sum with
components of any size, the potential step's orbital groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = np.array([0.1, 0.12, 0.09])


@pytest.mark.parametrize('scale', [(1.0, 1.0, 1.0), (0.0, 1.0, 1.0), (1.0, 0.0, -1.0), (1.0, -1.0, 0.0),
                                   (1e-100, 1e-90, 1e-95), (1e90, 1e80, 1e95), (1e-310, 1.0, 1e-310)])
@pytest.mark.parametrize('n', [[17, 18, 19], [33, 20, 18]])
def test_divergence_cc_of_any_scale(pkg, O, n, scale):
    """cc against the oracle, relative to its largest value (1e-13, as every FP64-level operator)."""
    N = int(np.prod(n))
    u = (np.random.default_rng(N).uniform(-1.0, 1.0, (3, N)) * np.array(scale)[:, None]).ravel()
    with pkg.mode(pkg.MODE_FP64):
        du, cc = pkg.Poisson().div_u_i(2, n, u, 16, H, cc=True)
    do, co = np.zeros(N), np.zeros(N)
    assert O.call('oracle_div_u_i', 2, *n, u, do, 16, H, co) == 0
    assert np.abs(du - do).max() <= 1e-13 * np.abs(do).max()
    assert np.abs(cc - co).max() <= 1e-13 * np.abs(co).max()


@pytest.mark.parametrize('norb', [1, 2, 3, 4, 6, 33])
def test_potential_step_orbital_groups(pkg, norb):
    """Energies of norb orbitals in one call: the bits of one call each (groups of four share a
    reduction whose additions pair the same lanes)."""
    n, bc, a = [5, 6, 7], [2, 2, 2], [-0.5 / 0.4 ** 2] * 3
    nsig, nreal, _ = pkg.hamiltonian_sizes(n, bc)
    r = np.random.default_rng(norb)
    psig, pot = r.standard_normal(norb * nsig), r.uniform(0.1, 1.0, nreal)
    h, en = pkg.hamiltonian_narr(n, bc, a, norb, psig, pot)
    for j in range(norb):
        hj, ek, ep = pkg.hamiltonian(n, bc, a, psig[j * nsig:(j + 1) * nsig].copy(), pot)
        assert ep == en[j, 3]
        assert np.array_equal(hj, h[j * nsig:(j + 1) * nsig])
