"""Pushes whose tiles are shared out to several CTAs (few tiles) against the
CPU oracle (FP64) and against the FP64 form (FP32).

Cases: a bin of less than one 256-particle block per CTA, bins that end just
before, on and after a block, a species without particles, one tile for the
whole grid, tiles cut short by the grid, and departures from every slice.
Tolerances: FP64 1e-12 relative L2 and identical per-cell counts, as for one
CTA per tile (only the order of the FP64 current sums differs); FP32 against
FP64 1e-3 relative L2 over 3 steps, the bound of the other FP32 parity tests,
and no particle lost."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, TAU = 0.1, 0.02
KEYS = ("x", "y", "z", "px", "py", "pz")


def species(pkg, cells, ppc, empty):
    L = tuple(c * H for c in cells)
    out = []
    for i, s in enumerate(pkg.configs.SPECIES_BEAM_PLASMA):
        a = pkg.host_species(cells, L, i, 0 if i == empty else ppc, s["drift"], max(s["vth"], 0.05), 3)
        out.append(a)
    return out


@pytest.mark.parametrize("cells,ppc,empty", [
    ((3, 3, 4), 1, None),        # 36 particles per species: less than one block
    ((8, 4, 8), 1, None),        # 256: exactly one block, one tile
    ((8, 4, 8), 2, 1),           # two blocks, the middle species empty
    ((8, 4, 8), 41, 0),          # 10496 per species: 41 blocks, first species empty
    ((11, 5, 9), 7, None),       # tiles cut short on every axis
    ((19, 4, 4), 13, 2),         # a partial last block, last species empty
])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_sliced_push_matches_oracle(pkg, oracle_mod, cells, ppc, empty, precision):
    L = tuple(c * H for c in cells)
    table = pkg.configs.species_table(ppc)
    parts = species(pkg, cells, ppc, empty)
    orc = oracle_mod.OracleSim(cells, L, TAU)
    with pkg.PicSimulation(cells, L, TAU, table, precision=precision) as sim:
        for i, a in enumerate(parts):
            assert sim.load_particles(i, *a) == a[0].size
            if a[0].size:
                orc.add_particles(i, *a, table[i][1], table[i][0])
        n = [sim.num_particles(i) for i in range(3)]
        for nt in range(3):
            sim.step(nt)
            assert orc.step() == 0
            if precision == "fp64":
                assert np.array_equal(sim.cell_counts(), orc.cell_counts())
        assert [sim.num_particles(i) for i in range(3)] == n
        tol = 1e-12 if precision == "fp64" else 1e-3
        for f in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz", "Jx", "Jy", "Jz"):
            want = orc.get_field(f)
            assert np.linalg.norm(sim.get_field(f) - want) <= tol * np.linalg.norm(want), f
        # every bin holds each particle once and nothing else
        got = np.concatenate([np.stack([sim.particles(i)[k] for k in KEYS], 1) for i in range(3) if n[i]])
        assert len(np.unique(got, axis=0)) == sum(n)
        if sim.layout()["tiles"] > 1:  # a box of one tile wraps inside it
            assert sim.counters()[0] > 0


# FP64 push with and without the shared-memory copy of the next particle and the
# second tile current (8x8x8 has room for it, the others have not): the
# copy is left out where it would cost a CTA per SM (8x6x8 cells) or does not
# fit (16x9x8), kept otherwise (16x8x8, one CTA per SM)
@pytest.mark.parametrize("tile", [(8, 6, 8), (16, 9, 8), (16, 8, 8), (8, 8, 8)])
def test_plain_push_tiles_of_every_staging(pkg, oracle_mod, tile):
    cells, ppc = (20, 13, 17), 6
    L = tuple(c * H for c in cells)
    table = pkg.configs.species_table(ppc)
    orc = oracle_mod.OracleSim(cells, L, TAU)
    with pkg.PicSimulation(cells, L, TAU, table, tile=tile) as sim:
        for i, a in enumerate(species(pkg, cells, ppc, None)):
            sim.load_particles(i, *a)
            orc.add_particles(i, *a, table[i][1], table[i][0])
        for nt in range(3):
            sim.step(nt)
            assert orc.step() == 0
            assert np.array_equal(sim.cell_counts(), orc.cell_counts())
        for f in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz", "Jx", "Jy", "Jz"):
            want = orc.get_field(f)
            assert np.linalg.norm(sim.get_field(f) - want) <= 1e-12 * np.linalg.norm(want), f
