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
