"""Device memory of the streaming PCG."""
import numpy as np
import pytest

import fake_runtime


def test_first_solve_of_a_context():
    """Tiles and gathered vectors are allocated once, at the size the mesh fixes,
    and the vectors of the kernels over block-CSR rows not at all."""
    fake = fake_runtime.runtime(sms=2)
    fake.reset()
    sim = fake.cipc.Simulator(fake.cipc.scene_two_cubes(5))
    sim.assemble()
    rows = np.diff(sim.export_bsr()["rowPtr"])
    fake.reset()
    sim.solve()
    got = [int(e.split()[1]) for e in fake.events("malloc")]
    steps = sum(-(-int(rows[t:t + 8].max()) // 4) for t in range(0, sim.nv, 8))
    for exact in (32 * 4 * steps, 288 * 8 * steps, 16 * 8 * sim.nv):
        assert exact in got
    assert 2 * 8 * (6 * 3 * sim.nv + 6) not in got
    sim.close()


@pytest.mark.parametrize("nv", [700, 30011, 60011])
def test_stand_alone_solver_allocates_once(nv):
    """One allocation holds all but a few words, and it is given back."""
    fake = fake_runtime.runtime()
    fake.reset()
    fake.cipc.pcg_bsr(*fake_runtime.ring_system(nv))
    big = [n for n in (int(e.split()[1]) for e in fake.events("malloc")) if n > 1 << 16]
    assert len(big) == 1
    assert fake.L.fake_live() == 0
