"""The differentiable run of a plasma whose particles spread over many cells: its
particle kernels go on without the windows of shared memory that serve particles
which stay near each other.

The gradient of a run that changes over on its way (the forward from step 16 on, the
reverse from the step that the counts tell) is that of other chunks, which change over
elsewhere: 1e-9 (FP64) and 1e-4 (FP32) relative L2, as the other gradient tests.  The
device time of the hot run is at most 3.5 times that of a cold one (forward and
backward, measured 1.8 and 2.6; with windows throughout 4.6 and 6.4): positions spread
over the box read and add all over the field arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, TAU = 0.1, 0.05


def make(pkg, cells, ppc, vth, precision, **kw):
    sim = pkg.PicSimulation(cells, tuple(c * H for c in cells), TAU, pkg.configs.species_table(ppc), precision=precision,
                            capacity_slack=1.0, outbox_fraction=0.5, **kw)
    for s in range(3):
        sim.init_species(s, ppc, vth=vth, seed=3 + s)
    return sim


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("every,sub", [(24, 24), (10, 3)])
def test_gradient_of_a_run_that_spreads(pkg, precision, every, sub):
    cells, ppc, steps = (24, 16, 20), 8, 24
    got = []
    for kw in ({}, dict(tile=(2, 2, 4))):
        with make(pkg, cells, ppc, 0.4, precision, **kw) as sim:
            p0 = sim.particles(1)
            sim.forward(steps, every, sub)
            g = sim.backward(field="Ex", window=3, species=1)
            order = np.lexsort([p0[k] for k in ("px", "py", "pz", "x", "y", "z")])
            got.append((g["d_p0"][order], sim.get_field("Ex")))
    with make(pkg, cells, ppc, 0.4, precision) as sim:
        sim.run(steps)
        want = sim.get_field("Ex")
    tol = 1e-12 if precision == "fp64" else 1e-4
    for g in got:
        assert np.linalg.norm(g[1] - want) < tol * np.linalg.norm(want)
    assert np.linalg.norm(got[0][0]) > 0
    assert np.linalg.norm(got[1][0] - got[0][0]) < (1e-9 if precision == "fp64" else 1e-4) * np.linalg.norm(got[0][0])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_time_of_a_run_that_spreads(pkg, precision):
    t = {}
    for vth in (0.001, 0.3):
        best = None
        for _ in range(3):
            with make(pkg, (64, 32, 32), 16, vth, precision) as sim:
                sim.forward(60, 10)
                sim.backward(field="Ex", window=1, species=1, want_p0=False)
                ms = sim.adjoint_timings().astype(float)
                best = ms if best is None else np.minimum(best, ms)
        t[vth] = best
    assert (t[0.3] < 3.5 * t[0.001]).all(), t
