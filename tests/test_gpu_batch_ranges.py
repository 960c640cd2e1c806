"""Reading one scene of a batch: the kernels go over the scene's range of
storage, which moves when scenes leave and join.  Every read is compared bit
for bit with the same scene stepped alone in a batch of its own, before and
after the substep that drops a removed scene, and for a scene that has not
been stepped yet.
"""
import numpy as np
import pytest

from slosh_b200 import scenes
from slosh_b200._lib import SLOSH_E_OVERFLOW, SloshError
from slosh_b200.batch import MpmBatch

pytestmark = pytest.mark.gpu


def _batch():
    return MpmBatch(3, max_particles=1 << 16, grid_capacity=1 << 13, max_scenes=8, max_bodies=32)


def test_reads_follow_scenes_that_leave_and_join(cuda_lib):
    scs = [scenes.random_scene_3d(n, m, 1 / 64, seed=i) for i, (n, m) in
           enumerate([(4001, "fluid"), (5003, "sand"), (4507, "elastic"), (6007, "fluid")])]
    b, alone = _batch(), [_batch() for _ in scs]
    slots, solo, steps = {}, {}, {}

    def join(i):
        slots[i], solo[i], steps[i] = b.add(scs[i]), alone[i].add(scs[i]), 0

    def check():
        for i, slot in slots.items():
            assert b.positions(slot).tobytes() == alone[i].positions(solo[i]).tobytes(), i
            assert b.download_particles(slot).tobytes() == alone[i].download_particles(solo[i]).tobytes(), i
            assert b.timestep_bound(slot) == alone[i].timestep_bound(solo[i]), i

    def step(n):
        b.step(n)
        for i in slots:
            alone[i].step(n)

    for i in range(3):
        join(i)
    check()
    step(3)
    check()
    b.remove_scene(slots.pop(1))  # still in storage until the next substep
    check()
    join(3)  # behind the scene that leaves
    check()
    step(2)
    check()
    join(1)
    step(1)
    check()
    for x in [b, *alone]:
        x.close()


def test_timestep_bound_after_an_unreported_overflow(cuda_lib):
    """More blocks than the pool's grid holds: particles are lost, and the
    scenes behind move down in storage.  The bound counts every particle left
    to its scene, whether or not the overflow was reported yet."""
    nothing = 4.294967e-3  # of a scene without particles
    survived = False
    for _ in range(10):  # which blocks find room differs from run to run
        b = MpmBatch(3, max_particles=1 << 17, grid_capacity=128, max_scenes=16, max_bodies=32)
        b.add(scenes.random_scene_3d(60000, "fluid", 1 / 64, seed=1))
        slots = [b.add(scenes.random_scene_3d(600, "fluid", 1 / 64, seed=2 + i)) for i in range(8)]
        b.step(1)
        before = [b.timestep_bound(s) for s in slots]
        with pytest.raises(SloshError) as e:
            b.sync()
        assert e.value.code == SLOSH_E_OVERFLOW
        after = [b.timestep_bound(s) for s in slots]
        b.close()
        assert before == after
        survived = survived or min(after) < 0.9 * nothing
    assert survived, "a small scene kept particles"
