"""Which PCG kernel a system goes to."""
import numpy as np
import pytest

import fake_runtime

KERNELS = ("pcgPipelinedKernel", "pcgStreamKernel", "pcgPersistentKernel", "pcgRowsKernel")


@pytest.fixture(scope="module")
def fake():
    return fake_runtime.runtime()


def launched(fake):
    """The last solve's kernel, with its mangled arguments, and its grid."""
    launch = [e for e in fake.events("launch") if any(k in e for k in KERNELS)][-1]
    return launch.split()[1], int(launch.split(" grid ")[1].split()[0])


def tangle(fake, nv, tets, seed=3):
    """A context of tetrahedra between any of nv points: every row is wide."""
    rng = np.random.default_rng(seed)
    scene = fake.cipc.scene_two_cubes(1)
    x = rng.random((nv, 3))
    t = np.array([rng.choice(nv, 4, replace=False) for _ in range(tets)], np.int32)
    e = x[t[:, 1:]] - x[t[:, :1]]
    flip = np.linalg.det(e) < 0
    t[flip, 2:] = t[flip, 2:][:, ::-1]
    scene.update(x=x, tets=t, btype=np.zeros(nv, np.int32))
    return fake.cipc.Simulator(scene, precond="fsai")


@pytest.mark.parametrize("nv,tets,rows", [(443, 500, 64), (443, 2000, 16), (443, 8000, 8)])
def test_factor_of_wide_rows_stays_in_one_pass(fake, nv, tets, rows):
    """Where 64 rows and their factor do not fit a block, fewer do: the factor is
    then read in FP32, which the streaming kernel's tiles would round to FP16."""
    sim = tangle(fake, nv, tets)
    sim.assemble()
    fake.reset()
    sim.solve()
    name, grid = launched(fake)
    sim.close()
    assert "pcgPipelinedKernelIddLb1E" in name
    assert grid == -(-nv // rows)


def test_rows_that_fit_no_block_stream(fake):
    fake.reset()
    fake.cipc.pcg_bsr(*fake_runtime.ring_system(9001, range(1, 31)))
    assert "pcgStreamKernel" in launched(fake)[0]


@pytest.mark.parametrize("nv,rows", [(1, 64), (443, 64), (4736, 64), (4737, 33), (9001, 61), (9473, 65), (18944, 128)])
def test_rows_per_block(fake, nv, rows):
    """64 rows a block while an even spread over the 148 SMs has at most 32."""
    fake.reset()
    fake.cipc.pcg_bsr(*fake_runtime.ring_system(nv))
    name, grid = launched(fake)
    assert "pcgPipelinedKernel" in name
    assert grid == -(-nv // rows)


@pytest.mark.parametrize("every,degree,tiles", [
    (8, 0, True), (8, 12, True), (8, 24, True), (2, 30, True), (1, 200, True), (400, 200, True),
    (8, 60, False), (2, 200, False), (8, 200, False), (16, 100, False), (32, 100, False)])
def test_padding_of_tiles(fake, every, degree, tiles):
    """Where the rows of a tile differ so much that most of its slots would be
    empty, and they are many or in long chains, the block-CSR rows are read as
    they are, and no tiles are stored."""
    system = fake_runtime.hub_system(40011, every, degree)
    fake.reset()
    fake.cipc.pcg_bsr(*system)
    assert ("pcgStreamKernel" if tiles else "pcgRowsKernel") in launched(fake)[0]
    assert len(fake.events("launch", "packTilesKernel")) == int(tiles)
