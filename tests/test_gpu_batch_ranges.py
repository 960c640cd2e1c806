"""Reading one scene of a batch: the kernels go over the scene's range of
storage, which moves when scenes leave and join.  Every read is compared bit
for bit with the same scene stepped alone in a batch of its own, before and
after the substep that drops a removed scene, and for a scene that has not
been stepped yet.
"""
import numpy as np
import pytest

from slosh_b200 import scenes
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
