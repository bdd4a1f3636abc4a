"""Uploads are ordered before the kernels that read them.

A context's kernels run on a stream that does not wait for the legacy one, and
a copy from pageable memory on the legacy stream may return before the data has
arrived.  So no kernel may be launched on a context's stream while such a copy
can be under way: block-CSR offsets that had not arrived would send the kernels
that write through them out of range."""
import numpy as np
import pytest

import fake_runtime


@pytest.fixture(scope="module")
def fake():
    return fake_runtime.runtime(sms=2)  # a few hundred rows are more than a single-pass launch holds


@pytest.mark.parametrize("nv", [7, 700, 5003])
def test_stand_alone_solver(fake, nv):
    fake.reset()
    fake.cipc.pcg_bsr(*fake_runtime.ring_system(nv))
    assert fake.events("launch", "pcg")
    assert bool(fake.events("launch", "packTilesKernel")) == (nv > 512)
    assert not fake.events("unordered")


@pytest.mark.parametrize("precond", ["jacobi", "fsai", "learned"])
def test_contexts(fake, precond):
    fake.reset()
    sim = fake.cipc.Simulator(fake.cipc.scene_two_cubes(5), precond=precond)
    sim.set("x", sim.get("x"))
    sim.assemble()
    sim.solve()
    sim.step_bounds(np.zeros((sim.nv, 3)))
    sim.collision_sets()
    sim.intersected()
    sim.close()
    assert len(fake.events("launch", "packTilesKernel")) == (1 if precond == "jacobi" else 3)
    assert not fake.events("unordered")
