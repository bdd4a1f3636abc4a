"""A call that ran out of device memory reports it and leaves the context
usable: what it had begun is not taken for done by the next call."""
import pytest

import fake_runtime


@pytest.mark.parametrize("first,failing,again", [(100, 1000, 100), (100, 1000, 150), (64, 129, 1)])
def test_buffer_whose_growth_failed(first, failing, again):
    assert fake_runtime.runtime().L.buffer_recovers(first, failing, again) == 1


@pytest.mark.parametrize("precond", ["jacobi", "fsai"])
def test_tiles_of_a_solve_that_failed_are_laid_out_again(precond):
    """Whichever allocation of a context's first streaming solve fails, the next
    solve writes the columns of every tile set that has none yet."""
    fake = fake_runtime.runtime(sms=2)
    sets = 1 if precond == "jacobi" else 3
    failures = 0
    for nth in range(1, 100):
        fake.reset()
        sim = fake.cipc.Simulator(fake.cipc.scene_two_cubes(5), precond=precond)
        sim.assemble()
        fake.reset()
        fake.L.fake_fail_malloc(nth)
        try:
            sim.solve()
            break  # fewer allocations than this
        except fake.cipc.CipcError:
            failures += 1
        fake.L.fake_fail_malloc(0)
        sim.solve()
        assert len(fake.events("launch", "columns 1")) == sets, nth
        sim.close()
    fake.L.fake_fail_malloc(0)
    assert failures > 10
