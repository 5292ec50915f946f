"""Kernels that give up waiting say so in status words on the device; the host reads them where it has waited anyway, if such a kernel ran
since.  A replayed step runs the kernels of its capture without passing through their Python wrappers."""
from types import SimpleNamespace

import pytest
import torch

from iian_b200 import ops
from iian_b200.engine.runner import ModelRunner, _GraphSlot
from iian_b200.ops.cuda_backend import CudaKernels, KernelError


def replayed(monkeypatch, reports, code):
    """A decode step replayed from a slot whose kernels do or do not report, and whose replay leaves ``code`` in the status words."""
    status = torch.zeros(2, dtype=torch.int32)
    monkeypatch.setattr(CudaKernels, "_tc_status", {torch.device("cpu"): status})
    monkeypatch.setattr(CudaKernels, "_tc_used", False)
    monkeypatch.setattr(ops, "kernels", lambda: CudaKernels())
    slot = _GraphSlot()
    slot.logits, slot.reports = torch.zeros(1, 4), reports
    slot.graph = SimpleNamespace(replay=lambda: status.copy_(torch.tensor([code, 7], dtype=torch.int32)))
    runner = ModelRunner.__new__(ModelRunner)
    runner.max_num_seqs, runner._graphs, runner.launches, runner.native = 8, {(1, 256): slot}, 0, None
    runner.build_decode_context = lambda entries, s: SimpleNamespace(upload_bytes=0)
    runner._step_graph([SimpleNamespace(start=5)])
    return runner, status


def test_a_replayed_kernel_that_gave_up_is_reported(monkeypatch):
    runner, status = replayed(monkeypatch, True, 3)
    with pytest.raises(KernelError, match="gave up"):
        runner.check_device_status()
    assert status.tolist() == [0, 0]
    runner.check_device_status()                    # said once
    runner._step_graph([SimpleNamespace(start=5)])  # and again when the next replay gives up
    with pytest.raises(KernelError, match="gave up"):
        runner.check_device_status()


def test_replays_without_such_kernels_read_nothing(monkeypatch):
    runner, status = replayed(monkeypatch, False, 3)
    runner.check_device_status()
    assert status.tolist() == [3, 7]


@pytest.mark.parametrize("before", [False, True])
@pytest.mark.parametrize("ran", [False, True])
def test_what_ran_within_a_capture_is_told_from_what_ran_before(monkeypatch, before, ran):
    monkeypatch.setattr(CudaKernels, "_tc_used", before)
    k = CudaKernels()
    with k.status_use() as seen:
        assert not CudaKernels._tc_used
        if ran:
            CudaKernels._tc_used = True
    assert seen.reports == ran and CudaKernels._tc_used == (before or ran)
