"""A field that is not finite shows in the Gauss check's maxima, whether one node
or every node of it is: no maximum over |G - G0| or |G| passes a NaN over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", ["one", "all"])
@pytest.mark.parametrize("cells", [(5, 9, 130), (6, 4, 8)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_gauss_check_reports_a_nan(pkg, precision, cells, nodes):
    with pkg.PicSimulation(cells, tuple(0.1 * c for c in cells), 0.01, pkg.configs.species_table(2),
                           precision=precision) as sim:
        for s in range(3):
            sim.init_species(s, 2, seed=s)
        a = np.zeros(sim.shape)
        sim.set_field("Ex", a)
        base = sim.gauss_check(set_baseline=True)
        assert np.isfinite(base).all() and base[0] == 0.0
        a[(slice(None),) * 3 if nodes == "all" else (3, 2, cells[2] // 2)] = np.nan
        sim.set_field("Ex", a)
        now = sim.gauss_check()
        assert np.isnan(now[0]) and np.isnan(now[2])
        assert now[1] == pytest.approx(base[1], rel=1e-12) and now[3] == pytest.approx(base[3], rel=1e-12)  # rho's atomics
        again = sim.gauss_check(set_baseline=True)
        assert np.isnan(again[[0, 2, 3]]).all() and again[1] == pytest.approx(base[1], rel=1e-12)
