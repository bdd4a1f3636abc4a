"""The dynamic shared memory limit of a kernel belongs to the process, and
contexts may be used from several threads: a limit that follows the system at
hand could be lowered by another thread between its setting and the launch,
which is then refused.  No call may lower it."""
import fake_runtime


def test_smaller_systems_leave_the_limit_alone():
    fake = fake_runtime.runtime()
    fake.reset()
    for nv in (120011, 60011, 18001, 9001):  # the first two in tiles, the others in one pass
        fake.cipc.pcg_bsr(*fake_runtime.ring_system(nv))
    launches = fake.events("launch", "pcgStreamKernel") + fake.events("launch", "pcgPipelinedKernel")
    assert len({e.split(" smem ")[1] for e in launches}) >= 4
    assert not fake.events("lowered") and not fake.events("refused")
