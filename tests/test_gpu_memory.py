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


@pytest.mark.parametrize("kind", ["species", "adjoint"])
def test_a_smaller_run_holds_no_more_than_a_fresh_one(pkg, kind):
    """After a run 1.8 times as large: at most 65 MB more per kept buffer of hundreds of
    MB (one species' arrays; the adjoint's state, checkpoints, segment states and
    adjoints), where up to twice the need was held."""
    import torch

    def used(first):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        with make(pkg, 20 if kind == "species" else PPC) as sim:
            if kind == "species":
                if first:
                    sim.init_species(0, 36, vth=0.05, seed=5)
                sim.init_species(0, 20, vth=0.05, seed=5)
            else:
                if first:
                    sim.forward(9, 1)
                sim.forward(5, 1)
            return before - torch.cuda.mem_get_info()[0]

    used(True)  # what the process keeps anyway
    fresh, after = used(False), used(True)
    assert after - fresh <= (1 if kind == "species" else 4) * 65 * MB + 4 * MB
