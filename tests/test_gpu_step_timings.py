"""pic_step_timings after a step that failed: the last step that succeeded, read
before the failure or not, and PIC_ERR_STATE where there was none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("steps,read", [(0, False), (1, False), (1, True), (2, False), (3, True)])
def test_timings_after_a_failed_step(pkg, precision, steps, read):
    with pkg.PicSimulation((8, 4, 8), (0.8, 0.4, 0.8), 0.02, pkg.configs.species_table(8), precision=precision) as sim:
        for s in range(3):
            sim.init_species(s, 8, vth=0.02, seed=s)
        sim.run(steps)
        before = sim.timings() if read else None
        sim.perturb_momenta(1, np.full((sim.num_particles(1), 3), np.nan), 1.0)
        for _ in range(2):
            with pytest.raises(pkg.PicError):
                sim.step()
            if not steps:
                t = np.zeros(5, np.float32)
                assert pkg._capi.PIC_ERR[sim.lib.pic_step_timings(sim.h, t.ctypes.data_as(pkg._capi.F))] == "PIC_ERR_STATE"
                continue
            t = sim.timings()
            assert (t >= 0).all() and t[1] > 0 and 0 < t[4] < 1e3
            if read:
                assert np.array_equal(t, before)
