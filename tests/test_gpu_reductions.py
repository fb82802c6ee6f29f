"""Reductions over the bins and the nodes (energies, momenta, rho, Gauss
residual) where their walks end: fewer particles than a block, one row, z rows
that are not a multiple of four nodes, tiles dealt out to many blocks, tiny and
large tiles (rho's two ways to round a contribution), an empty species.

Against numpy in FP64 from the exported state.  rho, G and the momenta to 1e-12
relative L2 (fixed-point rho: 2^-51 of a particle's charge at most; FP64 sums
of at most 1e5 terms: 1e-11 x 1e-2 cancellation), energies to 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "px", "py", "pz")


@pytest.mark.parametrize("cells,ppc", [((3, 3, 3), 1), ((8, 4, 8), 7), ((8, 4, 8), 300), ((17, 5, 11), 9), ((5, 9, 130), 2)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_reductions_match_numpy(pkg, oracle_mod, cells, ppc, precision):
    h = (0.1, 0.11, 0.09)
    L = tuple(c * v for c, v in zip(cells, h))
    table = pkg.configs.species_table(ppc)
    shape = tuple(c + 2 for c in cells)
    rng = np.random.default_rng(4)
    with pkg.PicSimulation(cells, L, 0.01, table, precision=precision) as sim:
        for i in (0, 2):  # species 1 stays empty
            a = pkg.host_species(cells, L, i, ppc, (0.1, 0.0, -0.05), 0.3, 9)
            sim.load_particles(i, *a)
        F = {}
        for f in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz"):
            sim.set_field(f, rng.standard_normal(int(np.prod(shape))))
            F[f] = sim.get_field(f).reshape(shape)
        parts = [sim.particles(i) for i in range(3)]
        rho = sim.charge_density()
        G = sim.gauss_residual()
        mom, en, ref = sim.momentum(), sim.energy(), sim.energy_reference()
        check = sim.gauss_check(set_baseline=True)
    x = [np.concatenate([p[k] for p in parts]) for k in "xyz"]
    m = np.concatenate([np.full(p["x"].size, table[i][1]) for i, p in enumerate(parts)])
    want = oracle_mod.charge_density(*x, m, cells, h)
    assert np.linalg.norm(rho - want) <= 1e-12 * np.linalg.norm(want)
    wantG = oracle_mod.gauss_residual(F["Ex"], F["Ey"], F["Ez"], rho, cells, h)
    assert np.linalg.norm(G - wantG) <= 1e-12 * np.linalg.norm(wantG)
    inner = (slice(1, -1),) * 3
    g = wantG.reshape(shape)[inner]
    np.testing.assert_allclose(check, [0.0, np.abs(rho.reshape(shape)[inner]).max(), 0.0, np.abs(g).max()], rtol=1e-12)
    kin = 0.0
    for i, p in enumerate(parts):
        M = table[i][1] / table[i][0]
        P = np.stack([p[k] for k in KEYS[3:]], 1)
        np.testing.assert_allclose(mom[i], M * P.sum(0), rtol=1e-12, atol=1e-14 * abs(M) * np.abs(P).sum())
        p2 = (P * P).sum(1)
        kin += M * (p2 / (np.sqrt(1.0 + p2) + 1.0)).sum()
    e = 0.5 * sum((F[f][inner] ** 2).sum() for f in ("Ex", "Ey", "Ez"))
    b = 0.5 * sum((F[f][inner] ** 2).sum() for f in ("Hx", "Hy", "Hz"))
    np.testing.assert_allclose(en, [e, b, kin, e + b + kin], rtol=1e-12)
    np.testing.assert_allclose(ref, sum((F[f] ** 2).sum() for f in ("Ex", "Ey", "Ez")), rtol=1e-12)


@pytest.mark.parametrize("tile,precision", [((1, 1, 4), "fp64"), ((1, 1, 4), "fp32"), ((4, 4, 8), "fp64"), ((8, 8, 8), "fp64"),
                                            ((8, 8, 8), "fp32"), ((10, 8, 12), "fp64")])
def test_rho_boxes_per_block(pkg, oracle_mod, tile, precision):
    # 8, 8, 4 and 2 boxes fit (the FP32 push takes no tile as large as the
    # last); ragged tiles, both ways to round a contribution
    cells, ppc, h = (21, 9, 25), 40, (0.1, 0.1, 0.1)
    L = tuple(c * v for c, v in zip(cells, h))
    table = pkg.configs.species_table(ppc)
    with pkg.PicSimulation(cells, L, 0.01, table, precision=precision, tile=tile) as sim:
        for i in range(3):
            sim.init_species(i, ppc, (0.1, 0.0, -0.05), 0.3, 9 + i)
        parts = [sim.particles(i) for i in range(3)]
        rho = sim.charge_density()
    x = [np.concatenate([p[k] for p in parts]) for k in "xyz"]
    m = np.concatenate([np.full(p["x"].size, table[i][1]) for i, p in enumerate(parts)])
    # the neutral sum cancels: against the sum of |charge| each node receives
    want = oracle_mod.charge_density(*x, m, cells, h)
    scale = oracle_mod.charge_density(*x, np.abs(m), cells, h)
    assert np.linalg.norm(rho - want) <= 1e-12 * np.linalg.norm(scale)
