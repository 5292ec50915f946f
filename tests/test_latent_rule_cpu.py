"""Which kernel a step's attention over a cached latent goes to: short keys in many row tiles stay on mma.sync."""
import pytest

from iian_b200.ops.cuda_backend import CudaKernels


@pytest.mark.parametrize("seqs,new,cached,heads,rank,tc", [
    (16, 30, 0, 32, 512, False), (60, 20, 0, 128, 512, False), (16, 60, 0, 128, 512, False), (100, 20, 30, 16, 512, False),
    (16, 30, 0, 128, 256, False), (200, 2, 100, 16, 512, False),
    (4, 100, 0, 128, 512, True), (16, 60, 0, 32, 256, True), (20, 20, 100, 128, 512, True), (1, 1000, 0, 16, 512, True),
    (64, 1, 1000, 32, 512, True), (48, 1, 2000, 16, 512, False), (200, 2, 100, 32, 512, True)])
def test_rule(monkeypatch, seqs, new, cached, heads, rank, tc):
    monkeypatch.setattr(CudaKernels, "sm_count", classmethod(lambda cls, device=None: 148))
    parts = CudaKernels().latent_attention_tc_parts(seqs * new, seqs, new, heads, rank, cached + new, None)
    assert (parts > 0) == tc
