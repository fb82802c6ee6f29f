"""The adjoint kernels sum lambda_E and lambda_H in fixed point, in a quantum that
follows the adjoints of a batch of 256 particles.

Scaling: with q/m times 2^k, the charge weight and the fields times 2^-k every
force and so every position and momentum keeps its bits, the loss and its gradient
scale by 2^-2k exactly, and the adjoints of the field values by 2^-k.  FP64 for k of
both signs up to 300, far outside a float's range; FP32 within it.  1e-9 and 1e-4
relative L2: only the order of the FP64 sums differs (the tolerances of the other
gradient tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,k", [("fp64", 300), ("fp64", 140), ("fp64", -140), ("fp64", -300), ("fp32", 20),
                                         ("fp32", -20)])
def test_gradient_scales_with_the_fields(pkg, precision, k):
    cells, h, got = (16, 8, 8), 0.1, []
    for e in (0, k):
        table = [(q_m * 2.0 ** e, m * 2.0 ** -e, sort) for q_m, m, sort in pkg.configs.species_table(4)]
        with pkg.PicSimulation(cells, tuple(c * h for c in cells), 0.05, table, precision=precision) as sim:
            for s, sp in enumerate(pkg.configs.SPECIES_BEAM_PLASMA):
                sim.init_species(s, 4, drift=sp["drift"], vth=0.1, seed=3 + s)
            rng = np.random.default_rng(2)
            for f in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz"):
                sim.set_field(f, 0.1 * 2.0 ** -e * rng.standard_normal(sim.shape))
            sim.forward(6, 3)
            got.append(sim.backward(field="Ex", window=4, species=1))
    a, b = got
    assert b["loss"] * 2.0 ** (2 * k) == pytest.approx(a["loss"], rel=1e-9 if precision == "fp64" else 1e-4)
    d = b["d_p0"] * 2.0 ** (2 * k)
    assert np.linalg.norm(a["d_p0"]) > 0
    assert np.linalg.norm(d - a["d_p0"]) / np.linalg.norm(a["d_p0"]) < (1e-9 if precision == "fp64" else 1e-4)


# 256 particles per cell and chunks of 8 cells of a row: a batch is a cell
H, TAU, PPC, CELLS = 0.1, 0.05, 256, (32, 16, 32)


def spiked(pkg, precision, spike, tile=None, k=0):
    """d_p0 of a cold plasma's particles in the order of their positions, and those:
    fields of 1e-7 and 1 at one node (q/m, charge weights and fields scaled by k as above)"""
    table = [(-1.0 * 2.0 ** k, -25.0 / TAU ** 2 / PPC * 2.0 ** -k, 0)]
    with pkg.PicSimulation(CELLS, tuple(c * H for c in CELLS), TAU, table, precision=precision, tile=tile) as sim:
        sim.init_species(0, PPC, seed=7)
        rng = np.random.default_rng(1)
        for f in ("Ex", "Ey", "Ez"):
            a = 1e-7 * rng.standard_normal(sim.shape)
            if f == "Ex":
                a[tuple(c + 1 for c in spike)] = 1.0
            sim.set_field(f, a * 2.0 ** -k)
        p0 = sim.particles(0)
        x = np.stack([p0[q] for q in "xyz"], 1)
        sim.forward(2, 2)
        g = sim.backward(field="Ex", window=2, species=0)
    order = np.lexsort(x.T)
    return g["d_p0"][order], x[order]


@pytest.mark.parametrize("precision,tx", [("fp64", 8), ("fp32", 6)])
@pytest.mark.parametrize("first", [False, True])
def test_large_adjoints_beside_small_ones(pkg, precision, tx, first):
    """One node whose field is 1e7 times the others' makes the adjoints of the
    particles around it that much larger: those of particles a few cells away, in
    other batches of the same chunk, must come out as from tiles of 4 cells, where
    they are in another chunk.  FP64 1e-10 relative L2: the current of particles
    at v ~ 2.5e-9 rounded to 2^-70 of the light-speed bound, 4e-12, times a coupling
    of 25 to the fields; lambda's own rounding, 2^-45 of a batch's largest at most, is
    far below.  FP32 1e-4, as the other gradient tests.  In a quantum of the large
    adjoints, 2^-51 and 2^-31 of 1e7 times the others, the error would be 1e-7 and 0.1."""
    i, l, k = tx, 4, 8  # the first row of a tile
    spike = (i, l, k if first else k + 7)
    rows, x = spiked(pkg, precision, spike)
    alone, y = spiked(pkg, precision, spike, (1, 1, 4))
    assert np.array_equal(x, y)
    c = np.floor(x / H).astype(int)
    away = (c[:, 0] == i) & (c[:, 1] == l) & (c[:, 2] >= (k + 5 if first else k)) & (c[:, 2] < (k + 8 if first else k + 3))
    near = np.all(c == spike, axis=1)
    assert away.sum() > 100 and np.abs(alone[near]).max() > 1e5 * np.abs(alone[away]).max() > 0
    err = np.linalg.norm(rows[away] - alone[away]) / np.linalg.norm(alone[away])
    assert err < (1e-10 if precision == "fp64" else 1e-4)


@pytest.mark.parametrize("precision,tx,top", [("fp64", 8, 1024), ("fp32", 6, 128)])
def test_adjoints_that_overflow_do_not_come_out_finite(pkg, precision, tx, top):
    """Scaled so that products of the large adjoints with the fields (2^-3k) overflow
    and the others' do not: a particle's gradient is either not finite or the
    unscaled run's, scaled (1e-9 and 1e-4 of the largest)."""
    spike = (tx, 4, 8)
    base, x = spiked(pkg, precision, spike)
    k = -int(np.ceil((top + 10 - np.log2(np.abs(base).max())) / 3))
    with np.errstate(all="ignore"):
        got, y = spiked(pkg, precision, spike, k=k)
        assert np.array_equal(x, y)
        ok = np.isfinite(got).all(1)
        assert 0.9 < ok.mean() < 1.0
        err = np.abs(got[ok] * 2.0 ** (2 * k) - base[ok]).max()
    assert err < (1e-9 if precision == "fp64" else 1e-4) * np.abs(base).max()
