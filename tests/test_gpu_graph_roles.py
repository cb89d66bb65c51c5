"""Graphs that a caller captures on a lattice's stream, between ordinary calls of many steps.

A captured graph holds the buffers and side-store slots of its capture.  An even number of steps has to leave
them in place from then on, however many launches the steps take, so that the graph can be replayed
at any such point.
"""
import numpy as np
import pytest

import lbgpu
from helpers import same

pytestmark = pytest.mark.gpu


class Captured:
    """What `work` does on the lattice's stream, replayed there."""

    def __init__(self, lat, work):
        import torch

        torch.zeros(1, device="cuda")
        self.stream = torch.cuda.ExternalStream(lat.stream)
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph, stream=self.stream, capture_error_mode="thread_local"):
            work()

    def replay(self):
        import torch

        with torch.cuda.stream(self.stream):
            self.graph.replay()


def channel(lx, ly, storage, steps):
    lat = lbgpu.Lattice(lx, ly, lbgpu.storage_form(storage)[0], "pull")
    lbgpu.configure_storage(lat, storage, 0.03, 5)
    lat.setup_cylinder(lx // 5 + 1, ly // 2 + 1, ly // 10 + 1, 0.03, 60.0, lbgpu.WALL_REGULARIZED, lbgpu.OUTLET_CONST)
    for n in steps:
        lat.step(n)
    return lat


def singles(lat, n):
    for _ in range(n):
        lat.step(1)


# shapes of eight, four and two steps a launch; rounding to nearest, with and without a row shift
@pytest.mark.parametrize("storage,lx,ly", [("f64", 150, 41), ("f64", 401, 160), ("f32", 150, 41), ("f32", 700, 200),
                                           ("f16", 150, 41), ("f16", 1030, 130), ("f16s", 150, 41), ("bf16b", 401, 161),
                                           ("f32", 1030, 700), ("f16s", 2100, 1500)])
@pytest.mark.parametrize("before", [[5], [9, 2], [1, 8, 8]])
def test_replays_between_calls_of_many_steps(storage, lx, ly, before):
    with channel(lx, ly, storage, before) as lat, channel(lx, ly, storage, before) as ref:
        graph = Captured(lat, lambda: lat.step(4))
        total = 0
        for n in (0, 2, 8, 30, 4, 14):
            lat.step(n)
            graph.replay()
            total += n + 4
        lat.synchronize()
        singles(ref, total)
        assert same(lat.populations(), ref.populations())
        del graph


@pytest.mark.parametrize("storage", ["f64", "f16s"])
def test_replays_after_the_state_is_set_again(storage):
    """New populations, or the channel set up again, and as many steps as before the capture."""
    with channel(150, 41, storage, [9]) as lat, channel(150, 41, storage, [9]) as ref:
        graph = Captured(lat, lambda: lat.step(4))
        start = ref.populations()
        for again in range(2):
            for one in (lat, ref):
                if again:
                    one.setup_cylinder(31, 21, 5, 0.03, 60.0, lbgpu.WALL_REGULARIZED, lbgpu.OUTLET_CONST)
                else:
                    one.set_populations(start, 0.5 * start)
            lat.step(9)
            graph.replay()
            graph.replay()
            lat.synchronize()
            singles(ref, 17)
            assert same(lat.populations(), ref.populations())
        del graph


def test_a_captured_accumulation_reads_the_state_of_its_replay():
    with channel(150, 41, "f64", [5]) as lat, channel(150, 41, "f64", [5]) as ref:
        for one in (lat, ref):
            one.velocity_accumulate()
            one.velocity_reset()
        graph = Captured(lat, lat.velocity_accumulate)
        for _ in range(3):
            lat.step(10)
            graph.replay()
            singles(ref, 10)
            ref.velocity_accumulate()
        ux, uy, samples = lat.velocity_average()      # one sample by the host's count: the sum
        ex, ey, k = ref.velocity_average()
        assert (samples, k) == (1, 3)
        assert np.allclose(ux, 3 * ex, rtol=1e-14, atol=1e-16) and np.allclose(uy, 3 * ey, rtol=1e-14, atol=1e-16)
        del graph


@pytest.mark.parametrize("storage", ["f64", "f16"])
def test_a_member_s_graph_between_batch_calls(storage):
    sizes = [(150, 41), (70, 33)]
    lats = [channel(lx, ly, storage, [5]) for lx, ly in sizes]
    refs = [channel(lx, ly, storage, [5]) for lx, ly in sizes]
    with lbgpu.Batch(storage) as b:
        for lat in lats:
            b.add(lat)
        graph = Captured(lats[0], lambda: lats[0].step(2))
        for n in (2, 6, 4, 22, 40):
            b.step(n)
            graph.replay()
            singles(refs[0], n + 2)
            singles(refs[1], n)
        b.synchronize()
        lats[0].synchronize()
        for lat, ref in zip(lats, refs):
            assert same(lat.populations(), ref.populations())
        del graph
    for one in lats + refs:
        one.close()


@pytest.mark.parametrize("steps", [10, 30])
def test_a_captured_batch_step(steps):
    with channel(150, 41, "f32", [5]) as lat, channel(150, 41, "f32", [5]) as ref, lbgpu.Batch("f32") as b:
        b.add(lat)
        b.step(6)
        b.synchronize()
        graph = Captured(lat, lambda: b.step(steps))
        graph.replay()
        b.step(2)
        lat.step(8)
        graph.replay()
        lat.synchronize()
        singles(ref, 6 + 2 * steps + 2 + 8)
        assert same(lat.populations(), ref.populations())
        del graph


def test_a_captured_batch_step_that_would_wait_is_refused():
    with channel(150, 41, "f32", [5]) as lat, channel(150, 41, "f32", [5]) as ref, lbgpu.Batch("f32") as b:
        b.add(lat)

        def refused():
            with pytest.raises(lbgpu.LbError):
                b.step(4)                       # the batch has not stepped yet
        Captured(lat, refused)
        b.step(6)

        def odd():
            with pytest.raises(lbgpu.LbError):
                b.step(3)
        Captured(lat, odd)
        b.step(3)
        b.synchronize()
        singles(ref, 9)
        assert same(lat.populations(), ref.populations())
