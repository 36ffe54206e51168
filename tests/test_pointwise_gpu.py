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


@pytest.mark.parametrize('mode', ['fp64', 'tc_exact'])
@pytest.mark.parametrize('op', ['d_s0s0_1d_sym8_md', 'd_s0s0_1d_sym8_d1', 'd_s0s1_1d_sym8', 'd_s1s0_1d_sym8'])
def test_arrays_of_lines_are_one_array(pkg, op, mode):
    """Contiguous sweeps over several arrays, padded leading dimensions included: the bits of one
    call per array.  FP64 sweeps also at the sizes around the smaller chunks (8 positions)."""
    wav = op in ('d_s0s1_1d_sym8', 'd_s1s0_1d_sym8')
    m, taps = (2, 8) if wav else (1, 29 if op.endswith('d1') else 16)
    with pkg.mode(pkg.MODE_FP64 if mode == 'fp64' else pkg.MODE_TC_EXACT):
        K = pkg.Kernel(op)
        for n, rows, narr, bc, pad in ((7, 1, 5, 0, 0), (9, 3, 40, 1, 2), (65, 2, 3, -1, 1), (8, 4, 130, 2, 0)):
            nx, ny = n + (taps - 1) * (bc == -1) + pad, n + (taps - 1) * (bc == 1) + pad
            sx, sy = nx * rows * m * m, ny * rows * m * m
            r = np.random.default_rng(n)
            x, y = r.uniform(-1, 1, narr * sx), r.uniform(-1, 1, narr * sy)
            one = y.copy()
            tail = (0.7, 1.5) if wav else (0.7, -0.3, 1.5)
            K.run(2, 0, [n, rows], bc, [nx, rows], [ny, rows], narr, x, y, *tail)
            for j in range(narr):
                yj = one[j * sy:(j + 1) * sy].copy()
                K.run(2, 0, [n, rows], bc, [nx, rows], [ny, rows], 1, x[j * sx:(j + 1) * sx].copy(), yj, *tail)
                assert np.array_equal(y[j * sy:(j + 1) * sy], yj), (n, bc, j)


@pytest.mark.parametrize('n', [[32, 32, 32], [40, 36, 50], [20, 70, 33]])
def test_sweeps_of_a_plan_in_order(pkg, n):
    """Sweeps start while the kernel before them ends: repeated calls on changing inputs, without
    a synchronisation in between and on two streams, and as a replayed capture, give the bits of
    calls that are each waited for."""
    import torch
    N, narr = int(np.prod(n)), 2
    g = torch.Generator(device='cuda').manual_seed(N)
    xs = [torch.randn(N * narr, dtype=torch.float64, device='cuda', generator=g) * 10.0 ** (3 * k) for k in range(6)]
    new = lambda: torch.full((N * narr,), float('nan'), dtype=torch.float64, device='cuda')  # noqa: E731
    mf, kin = pkg.Kernel('d_sfrf_ld_narr'), pkg.Kernel('d_kin_narr')
    w1, w2 = [new() for _ in range(2)], [new() for _ in range(2)]

    def step(x, y, z, s, k):
        mf.run_dev(3, n, [0] * 3, n, n, narr, x, y, w1[k], w2[k], stream=s)
        kin.run_dev(3, n, [2] * 3, narr, y, z, w1[k], w2[k], [-0.5, -0.6, -0.7], 0.0, 0.0, stream=s)

    with pkg.mode(pkg.MODE_TC_EXACT):
        ref = []
        for x in xs:
            y, z = new(), new()
            step(x, y, z, None, 0)
            torch.cuda.synchronize()
            ref.append((y, z))
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        out = [(new(), new()) for _ in xs]
        torch.cuda.synchronize()
        for i, x in enumerate(xs):
            step(x, *out[i], streams[i % 2], i % 2)
        torch.cuda.synchronize()
        for (y, z), (ry, rz) in zip(out, ref):
            assert torch.equal(y, ry) and torch.equal(z, rz)
        x, y, z = new(), new(), new()
        s = streams[0]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s, capture_error_mode='relaxed'):   # scratch is allocated
            step(x, y, z, s, 0)
        for xi, (ry, rz) in zip(xs, ref):
            x.copy_(xi)
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, ry) and torch.equal(z, rz)
        pkg.check()
