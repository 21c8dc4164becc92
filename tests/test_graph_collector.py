"""Graph captures and Python's cyclic collector: a collection inside a capture may free another graph, which
invalidates the capture, so the collector is held off while one runs; and a dropped trainer's graph goes with
the trainer, not with a later collection."""

import gc
import threading
import weakref

import pytest
import torch


def test_the_collector_is_held_for_the_outermost_capture_and_put_back():
    from voxneus_b200._lib import collector_held

    inside, leave = threading.Event(), threading.Event()

    def other():  # a capture on another thread that ends later
        with collector_held():
            inside.set()
            leave.wait(10)

    assert gc.isenabled()
    t = threading.Thread(target=other)
    with collector_held():
        assert not gc.isenabled()
        t.start()
        assert inside.wait(10)
    assert not gc.isenabled()
    leave.set()
    t.join()
    assert gc.isenabled()
    with pytest.raises(ValueError), collector_held():
        raise ValueError
    assert gc.isenabled()
    gc.disable()
    try:
        with collector_held():
            pass
        assert not gc.isenabled()  # a caller that runs without it still does
    finally:
        gc.enable()


def _step(seed):
    from voxneus_b200.models import VoxNeuS
    from voxneus_b200.rendering import RaySampler
    from voxneus_b200.training import FusedTrainer

    dev = torch.device("cuda", 0)
    torch.manual_seed(seed)
    m = VoxNeuS(grid_res=24, hash_log2_size=10, occupancy_res=8).to(dev)
    o = torch.nn.functional.normalize(torch.randn(128, 3, device=dev), dim=-1) * 3.0
    d = torch.nn.functional.normalize(-o + 0.2 * torch.randn(128, 3, device=dev), dim=-1)
    tr = FusedTrainer(m, RaySampler(16, 16, perturb=True), band_voxels=3.0, cuda_graph=True)
    for i in range(4):
        out = tr.step(o, d, torch.rand(128, 3, device=dev), step=i)
    assert tr.graph() is not None and bool(torch.isfinite(out["loss_rgb"]))
    return tr


@pytest.mark.gpu
def test_a_dropped_graph_waiting_for_the_collector_does_not_break_a_capture(monkeypatch):
    """A trainer that only the collector frees is garbage when the next one captures its step, and the objects made
    inside the capture are more than the collector's threshold."""
    from voxneus_b200 import training

    inner, keep = training.FusedTrainer._render_backward, gc.get_threshold()

    def busy(self, *a, **k):
        if torch.cuda.is_current_stream_capturing():
            gc.set_threshold(50, 1, 1)
            kept = [[i] for i in range(5000)]
            assert kept
        return inner(self, *a, **k)

    gc.collect()
    gc.set_threshold(10 ** 9)
    try:
        ring = [_step(0)]
        gone = weakref.ref(ring[0])
        ring.append(ring)
        del ring
        assert gone() is not None
        monkeypatch.setattr(training.FusedTrainer, "_render_backward", busy)
        _step(1)
    finally:
        gc.set_threshold(*keep)
    torch.cuda.synchronize()


@pytest.mark.gpu
def test_a_dropped_trainer_frees_its_graph():
    gc.collect()
    tr = _step(0)
    gone = [weakref.ref(tr), weakref.ref(tr.graph())]
    gc.disable()
    try:
        del tr
        assert [r() for r in gone] == [None, None]
    finally:
        gc.enable()
