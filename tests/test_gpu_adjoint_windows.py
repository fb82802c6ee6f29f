"""The differentiable run's particle kernels keep a chunk's neighbourhood in
shared memory and treat particles outside it through global memory.  A hot
plasma (several cells of drift apart within the run, both sides of the periodic
boundaries) takes both ways in every chunk; the tiling decides which particle
takes which, so the gradient must not depend on it.  Sizes: chunks of one
particle and of more than 256, a species that is empty, a box smaller than a
window; chunks of more than 1024 with windows of the fixed strides (the last
case, against chunks of 1000 with the others).

Forward against pic_run: 1e-12 relative L2 (only the order of FP64 sums
differs); FP32 1e-4, as the other FP32 forward test.  Gradients between two
tilings: FP64 1e-9, FP32 1e-4 relative L2 (the tolerances of the test of the
checkpoint intervals)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, TAU, STEPS = 0.1, 0.05, 20
KEYS = ("x", "y", "z", "px", "py", "pz")


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def make(pkg, cells, ppc, vth, precision, **kw):
    sim = pkg.PicSimulation(cells, tuple(c * H for c in cells), TAU, pkg.configs.species_table(max(ppc, 1)),
                            precision=precision, capacity_slack=1.0, outbox_fraction=0.5, **kw)
    for s, sp in enumerate(pkg.configs.SPECIES_BEAM_PLASMA):
        sim.init_species(s, 0 if (s == 0 and ppc < 2) else ppc, drift=sp["drift"], vth=vth if s else 0.0, seed=3 + s)
    return sim


@pytest.mark.parametrize("cells,ppc,vth", [((24, 16, 20), 6, 0.3), ((5, 4, 4), 1, 0.4), ((16, 6, 8), 90, 0.2),
                                           ((16, 8, 16), 250, 0.02)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_gradient_does_not_depend_on_the_tiling(pkg, cells, ppc, vth, precision):
    loss = dict(field="Ex", window=7, species=1, drift=(0.0, 0.0, 0.0), vth=vth)
    got = []
    for kw in ({}, dict(tile=(2, 2, 4))):
        with make(pkg, cells, ppc, vth, precision, **kw) as sim:
            p0 = sim.particles(1)
            sim.forward(STEPS, 8)
            g = sim.backward(**loss)
            order = np.lexsort([p0[k] for k in KEYS])
            got.append((g["d_p0"][order], g["d_drift"], g["d_vth"], sim.get_field("Ex"), sim.get_field("Jy"),
                        sim.get_field("Hz"), sim.get_field("Qx") if precision == "fp64" else None))
    with make(pkg, cells, ppc, vth, precision) as sim:
        sim.run(STEPS)
        tol = 1e-12 if precision == "fp64" else 1e-4
        assert rel(got[0][3], sim.get_field("Ex")) < tol and rel(got[1][3], sim.get_field("Ex")) < tol
        assert rel(got[0][4], sim.get_field("Jy")) < tol
        assert rel(got[0][5], sim.get_field("Hz")) < tol
        if precision == "fp64":
            assert rel(got[0][6], sim.get_field("Qx")) < tol
    tol = 1e-9 if precision == "fp64" else 1e-4
    assert np.linalg.norm(got[0][0]) > 0
    assert rel(got[1][0], got[0][0]) < tol
    assert rel(got[1][1], got[0][1]) < tol and abs(got[1][2] - got[0][2]) < tol * abs(got[0][2])


def test_kept_buffers_serve_runs_of_other_shapes(pkg):
    """One handle through runs of growing and shrinking length, one and two
    checkpoint levels, with and without a record, other particle numbers and a
    release in between: each gives the gradient of a fresh handle (1e-9, the
    order of FP64 sums)."""
    loss = dict(field="Ex", window=3, species=2, drift=(0.2, 0.0, 0.0), vth=0.002)

    def start(sim, ppc):
        for s, sp in enumerate(pkg.configs.SPECIES_BEAM_PLASMA):
            sim.init_species(s, ppc, drift=sp["drift"], vth=max(sp["vth"], 0.02), seed=3 + s)
        for f in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz"):
            sim.set_field(f, np.zeros(int(np.prod(sim.shape))))

    def fresh():
        cells = (16, 8, 8)
        return pkg.PicSimulation(cells, tuple(c * H for c in cells), 0.02, pkg.configs.species_table(4))

    with fresh() as kept:
        for ppc, steps, every, sub, record in ((4, 9, 4, None, False), (4, 20, 6, 2, False), (12, 5, 5, None, True),
                                               (4, 20, 20, None, False), (1, 4, 2, None, False)):
            start(kept, ppc)
            kept.branch_record(record)
            kept.forward(steps, every, sub)
            g = kept.backward(**loss)
            with fresh() as sim:
                start(sim, ppc)
                sim.forward(steps, every, sub)
                w = sim.backward(**loss)
            assert rel(g["d_p0"], w["d_p0"]) < 1e-9 and rel(g["d_drift"], w["d_drift"]) < 1e-9
            assert g["loss"] == pytest.approx(w["loss"], rel=1e-12)
            if steps == 5:
                kept.adjoint_free()
