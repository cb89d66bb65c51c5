"""Calls of lbgpu_batch_step between other calls: that they return before their work ends, and that members' own
steps between them are seen."""
import pytest

import lbgpu
from helpers import same

pytestmark = pytest.mark.gpu


def singles(lat, n):
    for _ in range(n):
        lat.step(1)


@pytest.mark.parametrize("precision", ["f16r", "bf16r"])
def test_rounding_keys_follow_members_that_step_alone(precision):
    """A stochastically rounded member counts its collisions wherever it steps, also where its own steps leave
    its buffers in place, or its state is set again."""
    def run(batched):
        lat = lbgpu.Lattice(33, 40, lbgpu.storage_form(precision)[0], "pull")
        lbgpu.configure_storage(lat, precision, 0.03, 7)
        lat.setup_cylinder(8, 20, 4, 0.03, 30.0, lbgpu.WALL_REGULARIZED, lbgpu.OUTLET_CONST)
        with lbgpu.Batch(lbgpu.storage_form(precision)[0]) as b:
            b.add(lat)
            go = b.step if batched else (lambda n: singles(lat, n))
            go(7)
            lat.step(16)
            go(46)
            b.synchronize()
            first = lat.populations()
            go(1)
            lat.set_populations(first, first)
            go(22)
            b.synchronize()
            out = (first, lat.populations())
        lat.close()
        return out

    for got, exp in zip(run(True), run(False)):
        assert same(got, exp)
@pytest.mark.parametrize("storage,scheme", [("f32", "pull"), ("f32", "aa"), ("f16b", "pull")])
def test_batch_steps_do_not_wait(storage, scheme):
    """Even counts return while the GPU still works, whatever their remainder."""
    import torch

    base = lbgpu.storage_form(storage)[0]
    lats = []
    for _ in range(8):
        lat = lbgpu.Lattice(2048, 1024, base, scheme)
        lbgpu.configure_storage(lat, storage, 0.03)
        lat.setup_cylinder(400, 500, 100, 0.03, 60.0, lbgpu.WALL_BOUNCEBACK, lbgpu.OUTLET_CONST)
        lats.append(lat)
    with lbgpu.Batch(base) as b:
        for lat in lats:
            b.add(lat)
        b.step(41)
        b.step(2)
        stream = torch.cuda.ExternalStream(lats[0].stream)
        for n in (110, 114, 112):
            b.synchronize()
            stream.synchronize()
            b.step(n)
            assert not stream.query(), n
        b.synchronize()
    for lat in lats:
        lat.close()


def test_the_tuner_leaves_alone_what_its_settings_do_not_reach():
    """Pull members that take two steps a launch: one timing, no setting changed; the class of an AA member beside
    them, and odd counts, are tuned."""
    lats = [lbgpu.Lattice(40, 30, "f32", "pull"), lbgpu.Lattice(300, 90, "f32", "pull"), lbgpu.Lattice(300, 90, "f32", "aa")]
    for lat in lats:
        lat.setup_cylinder(9, 12, 3, 0.03, 30.0, lbgpu.WALL_BOUNCEBACK, lbgpu.OUTLET_CONST)
    small, large = lbgpu.size_class(40 * 30), lbgpu.size_class(300 * 90)
    with lbgpu.Batch("f32") as b:
        b.add(lats[0])
        slot = b.add(lats[1])
        b.set_shape(small, 32)
        b.threads = 256
        best = b.autotune(4)
        assert lats[0].steps_done == lats[1].steps_done == 5
        assert (b.shape(small), b.threads) == ((32, 1), 256)
        assert [k for k, ms in enumerate(best) if ms > 0] == sorted({small, large})
        b.remove(slot)
        b.add(lats[2])
        best = b.autotune(4)
        # the launch forms, three widths and four or five strip lengths of the large class, and one for the other class
        done = lats[0].steps_done
        assert done - 5 in (5 * (6 + 3 + 4 + 1), 5 * (6 + 3 + 5 + 1)) and b.shape(small) == (32, 1)
        assert best[small] > 0 and best[large] > 0
        b.autotune(3)
        assert lats[0].steps_done >= done + 4 * (6 + 2 * (3 + 4))
    for lat in lats:
        lat.close()


@pytest.mark.parametrize("precision,ly,launches", [("f64", 4, 10), ("f64", 5, 5), ("f32", 3, 10), ("f32", 4, 5), ("f16", 3, 5)])
def test_batches_of_members_of_few_rows(precision, ly, launches):
    """They step one at a time where tiles hold little but halo, and as alone either way."""
    def make():
        lat = lbgpu.Lattice(700, ly, precision, "pull")
        lat.setup_cylinder(300, 90, 1, 0.03, 0.6, lbgpu.WALL_BOUNCEBACK, lbgpu.OUTLET_CONST)
        return lat

    lats, ref = [make(), make()], make()
    with lbgpu.Batch(precision) as b:
        for lat in lats:
            b.add(lat)
        b.step(3)
        b.step(10)
        assert b.last_launches == launches
        b.synchronize()
        singles(ref, 13)
        for lat in lats:
            assert same(lat.populations(), ref.populations())
    for one in lats + [ref]:
        one.close()
