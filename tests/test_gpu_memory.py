"""Calls on a device with no memory left but what the handle itself holds unused:
buffers kept from an earlier differentiable run go back to the device when a call
needs them, so the call succeeds as it does on a handle that keeps none."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CELLS, PPC = (64, 64, 64), 8
MB = 1 << 20


@contextlib.contextmanager
def device_filled(leave):
    """holds all free device memory but about `leave` bytes"""
    import torch
    torch.cuda.empty_cache()
    held = []
    try:
        while True:
            free = torch.cuda.mem_get_info()[0] - leave
            if free < 4 * MB:
                break
            try:
                held.append(torch.empty(free // (2 * MB) * 2 * MB, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                leave += 2 * MB
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def make(pkg, ppc=PPC):
    sim = pkg.PicSimulation(CELLS, tuple(0.1 * c for c in CELLS), 0.02, [(-1.0, -1.0 / PPC, 0)])
    sim.init_species(0, ppc, vth=0.05, seed=5)
    return sim


def call(sim, name):
    if name == "particles":
        return np.sort(sim.particles(0)["x"])  # the order within a bin is any
    if name == "perturb":
        sim.perturb_momenta(0, np.ones((sim.num_particles(0), 3)), 1e-6)
        return sim.momentum()
    return sim.charge_density()


@pytest.mark.parametrize("name", ["particles", "perturb", "rho"])
def test_kept_adjoint_buffers_are_given_back(pkg, name):
    with make(pkg) as other:
        other.forward(1, 1)
        want = call(other, name)  # and every kernel is loaded
    with make(pkg) as sim:
        if name == "perturb":
            sim.momentum()
        sim.forward(4, 4)
        sim.backward(field="Ex", window=1, species=0, want_p0=False)
        sim.init_species(0, PPC, vth=0.05, seed=5)
        for f in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz"):
            sim.set_field(f, np.zeros(sim.shape))
        sim.forward(1, 1)  # keeps the reverse run's buffers, unused
        with device_filled(MB):
            got = call(sim, name)
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)  # FP64 sums in any order


def test_backward_after_one_that_found_no_memory(pkg):
    """The first pic_backward gets the segment states and not the particle adjoints;
    the next, with memory, gives the gradient of a fresh handle (1e-9, the order of
    FP64 sums)."""
    loss = dict(field="Ex", window=2, species=0)

    def run(fill):
        with make(pkg) as sim:
            order = np.lexsort([sim.particles(0)[k] for k in ("px", "y", "x")])
            sim.forward(4, 4)
            if fill:
                n = sim.num_particles(0)
                with device_filled(5 * 52 * n + 64 * MB + 24 * n):  # states and fields, half of the adjoints
                    with pytest.raises(pkg.PicError, match="particle adjoints|field"):
                        sim.backward(**loss)
            return sim.backward(**loss)["d_p0"][order]

    want, got = run(False), run(True)
    assert np.linalg.norm(want) > 0
    assert np.linalg.norm(got - want) < 1e-9 * np.linalg.norm(want)
