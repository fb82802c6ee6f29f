"""A rebin asks first for bins with room for more arrivals, then for what the counts
need: near the limit of 2^23 slots in a tile (FP64) the first is refused and the
step goes on with the second, without an error in the handle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, CELLS, TILE = 0.1, (16, 4, 8), (8, 4, 8)
STAY, MOVE = 5_900_000, 1_000_000


def test_step_whose_first_layout_is_refused(pkg):
    L = tuple(c * H for c in CELLS)
    rng = np.random.default_rng(1)
    x = rng.uniform(0.0, 1.0, (STAY + MOVE, 3)) * (0.78, L[1], L[2])
    x[STAY:, 0] = 0.8 + 1e-3 * rng.uniform(0.1, 1.0, MOVE)  # beyond the boundary of the tiles, on their way back
    px = np.zeros(STAY + MOVE)
    px[STAY:] = -0.2
    with pkg.PicSimulation(CELLS, L, 0.02, [(-1.0, -1e-9, 0)], tile=TILE, capacity_slack=0.1, outbox_fraction=0.5) as sim:
        zero = np.zeros(STAY + MOVE)
        assert sim.load_particles(0, *x.T.copy(), px, zero, zero) == STAY + MOVE
        sim.run(1)
        assert sim.lib.pic_last_status(sim.h) == 0
        assert sim.lib.pic_last_error_string(sim.h) == b""
        assert sim.num_particles(0) == STAY + MOVE
        sim.run(2)
        assert sim.num_particles(0) == STAY + MOVE
