"""A batch's table is written on the default stream: on another stream, the work that was queued
before (and may still use the memory the batch's workspace was given) has to be done by then."""
import pytest
import torch


class _Tensor:
    """As much of a CUDA image as BatchPlan looks at."""

    shape, dtype, device, is_cuda = (8, 8), torch.uint8, torch.device("cpu"), True

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return 4096

    def stride(self, dim):
        return 8

    def element_size(self):
        return 1


@pytest.mark.parametrize("handle", [0, 1, 0x7F00])
def test_prepare_waits_for_the_current_stream(monkeypatch, handle):
    import nsgb

    log = []

    class Stream:
        cuda_stream = handle

        def synchronize(self):
            log.append("wait")

    class Lib:
        nsgb_batch_workspace_size = staticmethod(nsgb.lib.nsgb_batch_workspace_size)

        @staticmethod
        def nsgb_batch_prepare(*args):
            log.append("prepare")
            return 0

    monkeypatch.setattr(nsgb, "lib", Lib)
    monkeypatch.setattr(nsgb, "_check_image", lambda t, name: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream())
    nsgb.BatchPlan([_Tensor()], [_Tensor()], with_outputs=False)
    assert log == (["wait", "prepare"] if handle else ["prepare"])
