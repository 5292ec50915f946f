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


@pytest.mark.parametrize("rank,heads,bucket,contexts,window,line", [
    # a graph's sequences and bucket of contexts: what it meets may be half of that
    (512, 16, (48, 4096), None, None, False), (512, 16, (64, 4096), None, None, False), (512, 16, (128, 4096), None, None, True),
    (512, 16, (64, 8192), None, None, True), (256, 16, (48, 4096), None, None, False), (256, 16, (64, 4096), None, None, True),
    (512, 16, (128, 4096), None, 1000, False),
    # an eager step's real contexts
    (512, 16, None, [2100] * 44, None, False), (512, 16, None, [8000] * 24, None, False), (512, 16, None, [3000] * 48, None, False),
    (512, 16, None, [800 + 68 * i for i in range(48)], None, True), (512, 16, None, [4000] * 64, None, True), (512, 5, None, [4000] * 64, None, True),
    (256, 16, None, [4000] * 48, None, True), (512, 16, None, [4000] * 64, 900, False), (512, 16, None, [90] * 3, None, False),
    (512, 17, None, [4000] * 64, None, False), (128, 16, None, [4000] * 64, None, False)])
def test_rule_of_decoded_tokens_with_keys_as_rows(monkeypatch, rank, heads, bucket, contexts, window, line):
    monkeypatch.setattr(CudaKernels, "sm_count", classmethod(lambda cls, device=None: 148))
    seqs, longest = bucket or (len(contexts), max(contexts))
    pays = lambda new: CudaKernels().latent_line_pays(seqs, new, heads, rank, longest, window, contexts or ())
    assert pays(1) == line and not pays(2)
