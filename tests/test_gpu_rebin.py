"""Bins under heavy migration: more departures from a tile in one step than the
first part of its hole list holds (kHoleMax = 1024), with one and with several
CTAs per tile, and bins rebuilt because arrivals did not fit.

FP64: identical per-cell counts and every field within 1e-12 relative L2 of
the CPU oracle, the bar of the other parity tests.  FP32: every particle is
still there once, and a particle's bits survive the rebuild of its bin: the
sorted particle table after a step that rebuilds bins equals that of a run
whose bins have room (the current sums differ in the order of FP64 additions
only, so momenta agree to FP32 rounding: 1e-6)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, TAU = 0.1, 0.05
KEYS = ("x", "y", "z", "px", "py", "pz")


def plasma(pkg, cells, ppc, drift, vth, seed=5):
    L = tuple(c * H for c in cells)
    return L, pkg.host_species(cells, L, 0, ppc, drift, vth, seed)


# A beam through thin tiles: 2x8x8 cells, about 22 of the 100 particles of each
# of the 64 cells of a face leave per step (the oracle, like the reference,
# takes at most 50 per cell).  160 tiles: one CTA each; 8: several.
@pytest.mark.parametrize("cells", [(40, 16, 32), (8, 8, 16)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_departures_past_the_first_list(pkg, oracle_mod, cells, precision):
    ppc = 100
    L, a = plasma(pkg, cells, ppc, (0.5, 0.0, 0.0), 0.02)
    m = 0.01 / ppc
    orc = oracle_mod.OracleSim(cells, L, TAU, threads=8)
    orc.add_particles(0, *a, m, 1.0)
    with pkg.PicSimulation(cells, L, TAU, [(1.0, m, 0)], precision=precision, tile=(2, 8, 8),
                           outbox_fraction=0.5) as sim:
        n = sim.load_particles(0, *a)
        assert n == a[0].size
        slots, tiles = sim.layout()["slots"], sim.layout()["tiles"]
        for nt in range(2):
            sim.step(nt)
            assert orc.step() == 0
            assert sim.counters()[0] > 1024 * tiles  # on average more than the first list holds
        assert sim.layout()["slots"] == slots        # no bin was rebuilt
        assert sim.num_particles(0) == n
        if precision == "fp64":
            assert np.array_equal(sim.cell_counts(), orc.cell_counts())
        tol = 1e-12 if precision == "fp64" else 1e-3
        for f in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz", "Jx", "Jy", "Jz"):
            want = orc.get_field(f)
            assert np.linalg.norm(sim.get_field(f) - want) <= tol * np.linalg.norm(want), f


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_rebuilt_bins_keep_every_particle(pkg, precision):
    cells, ppc = (12, 8, 16), 40
    L, a = plasma(pkg, cells, ppc, (0.0, 0.0, 0.0), 0.6)
    cold = pkg.host_species(cells, L, 1, 5, (0.0, 0.0, 0.0), 0.0, 6)
    shape = tuple(c + 2 for c in cells)
    firsts = [(i * shape[1] + l) * shape[2] + k for i in range(0, 12, 4) for l in range(0, 8, 4) for k in range(0, 16, 4)]
    tables = []
    for slack in (1e-9, 2.0):  # no room at all; room for anything
        with pkg.PicSimulation(cells, L, TAU, [(1.0, 1e-4, 0), (-1.0, -1e-4, 1)], precision=precision, tile=(4, 4, 4),
                               capacity_slack=slack, capacity_pad=0, outbox_fraction=0.5) as sim:
            sim.load_particles(0, *a)
            sim.load_particles(1, *cold)
            offsets = [[sim.cell_particles(s, c)["bin_offset"] for c in firsts] for s in range(2)]
            sim.step(0)
            after = [[sim.cell_particles(s, c)["bin_offset"] for c in firsts] for s in range(2)]
            assert (after[0] != offsets[0]) == (slack < 1.0)  # the hot species' bins were rebuilt
            assert after[1] == offsets[1]                     # the cold one's never
            p = [sim.particles(i) for i in range(2)]
            assert [q["x"].size for q in p] == [a[0].size, cold[0].size]
            tables.append([np.stack([q[k] for k in KEYS], 1)[np.lexsort((q["z"], q["y"], q["x"], q["cell"]))] for q in p])
            sim.step(1)
            assert sim.num_particles() == a[0].size + cold[0].size
    tol = 1e-12 if precision == "fp64" else 1e-6
    for got, want in zip(*tables):
        np.testing.assert_allclose(got, want, rtol=0, atol=tol)
