"""A batch keeps its configuration when a new one is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [[24, 33, 40], [27, 24, 31]]


@pytest.mark.parametrize('graph', [False, True])
@pytest.mark.parametrize('mode', ['MODE_FP64', 'MODE_TC_EXACT'])
def test_refused_configuration_leaves_the_old_one(pkg, mode, graph):
    """An order that is no permutation (either operator) is refused; get_config and the next run
    are what they were before, and a later valid configuration takes effect."""
    import torch
    n = sum(int(np.prod(d)) for d in DIMS)
    g = torch.Generator(device='cuda').manual_seed(n)
    x = torch.randn(n, dtype=torch.float64, device='cuda', generator=g)
    stream = torch.cuda.Stream() if graph else None
    with pkg.mode(getattr(pkg, mode)):
        B = pkg.Batch(DIMS, mf_bc=[2, 2, 2], kin_bc=[2, 0, 2], kin_a=[-0.5, -0.6, -0.7])
        new = lambda: torch.full((n,), float('nan'), dtype=torch.float64, device='cuda')  # noqa: E731
        y, z = new(), new()
        torch.cuda.synchronize()
        B.run(x, y, z, stream=stream)
        torch.cuda.synchronize()
        ref = y.clone(), z.clone()
        was = [B.get_config(op) for op in (pkg.BATCH_OP_MF, pkg.BATCH_OP_KIN)]
        engine = pkg.ENGINE_FP64_Q64 if mode == 'MODE_FP64' else pkg.ENGINE_TC
        for op, order in ((pkg.BATCH_OP_KIN, [0, 0, 2]), (pkg.BATCH_OP_KIN, [-1, 0, 0]), (pkg.BATCH_OP_MF, [0, 1, 3])):
            with pytest.raises(pkg.LibconvError):
                B.set_config(op, engine, order)
            assert [B.get_config(o) for o in (pkg.BATCH_OP_MF, pkg.BATCH_OP_KIN)] == was
            y.fill_(float('nan'))
            z.fill_(float('nan'))
            torch.cuda.synchronize()
            B.run(x, y, z, stream=stream)
            torch.cuda.synchronize()
            assert torch.equal(y, ref[0]) and torch.equal(z, ref[1])
        B.set_config(pkg.BATCH_OP_KIN, engine, [2, 0, 1])
        assert B.get_config(pkg.BATCH_OP_KIN)[1] == [2, 0, 1]
        z.fill_(float('nan'))
        torch.cuda.synchronize()
        B.run(x, y, z, stream=stream)
        torch.cuda.synchronize()
        assert float((z - ref[1]).abs().max()) <= 1e-13 * float(ref[1].abs().max())
        B.close()
        pkg.check()


# grids whose third axis is cut into segments by the shared exponent pass (few grids), segments
# that do not divide it, more segments than a grid has planes, and many grids (no segments)
@pytest.mark.parametrize('dims', [[[72, 72, 72]], [[40, 33, 125], [9, 64, 17]], [[24, 70, 8], [33, 20, 130], [64, 64, 3]],
                                  [[25 + g % 9, 30 - g % 7, 24 + g % 5] for g in range(40)]])
def test_shared_exponents_of_a_batch(pkg, O, dims):
    """Kinetic sweeps of a batch give the bits of one call per grid: the same line exponents."""
    import torch
    a, bc = [-0.5, -0.6, -0.7], [2, 0, 2]
    n = [int(np.prod(d)) for d in dims]
    r = np.random.default_rng(sum(n))
    xs = [r.uniform(-1, 1, d[::-1]) * 2.0 ** r.integers(-40, 40, (d[2], 1, 1)) * 2.0 ** r.integers(-9, 9, (d[1], 1)) for d in dims]
    with pkg.mode(pkg.MODE_TC_EXACT):
        B = pkg.Batch(dims, kin_bc=bc, kin_a=a)
        B.set_config(pkg.BATCH_OP_KIN, pkg.ENGINE_TC, [0, 1, 2])
        x = torch.from_numpy(np.concatenate([v.ravel() for v in xs])).cuda()
        y = torch.full_like(x, float('nan'))
        for _ in range(2):                       # the second run finds the exponents of the first
            B.run(x, None, y)
        torch.cuda.synchronize()
        y, off = y.cpu().numpy(), np.concatenate([[0], np.cumsum(n)])
        for g, d in enumerate(dims):
            yg, w = np.zeros(n[g]), np.zeros(n[g])
            pkg.Kernel('d_kin').run(3, d, bc, xs[g].ravel(), yg, w, w, a, 0.0, 0.0)
            assert np.array_equal(y[off[g]:off[g + 1]], yg), g
        B.close()
        pkg.check()
