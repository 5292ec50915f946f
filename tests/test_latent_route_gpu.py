"""A Galodra model whose attention takes the tcgen05 kernel over the cached latent, through the step function: a long prompt, the mixed step
behind it, and decoded tokens of 32 heads eagerly and out of a captured graph; against the plain implementation, and against the same steps on
the kernel it is chosen over."""
import os

import pytest
import torch

import plain_galodra as plain
from galodra_cases import dense, layer, mixer
from helpers import first_bad, max_error, random_tokens, replay_and_collect

pytestmark = pytest.mark.gpu

CONFIG = {"architecture": "Galodra", "vocab": 131, "width": 256, "norm": {"eps": 1e-6}, "postln_alpha": 2.0, "layers": [
    layer(mixer(32, 32, 64, 32, 256, None, 64), dense(128)), layer(mixer(32, 32, 64, 32, 256, 700, 64), dense(128))]}


@pytest.fixture(scope="module")
def case(tmp_path_factory):
    from iian_b200.config.registry import get_architecture
    from iian_b200.weights.random_init import write_model_folder
    d = os.path.join(str(tmp_path_factory.mktemp("latent")), "galodra")
    arch = get_architecture("Galodra")
    write_model_folder(d, arch, arch.load_config(CONFIG), seed=21, store_dtype=torch.bfloat16, std=0.08, norm_jitter=0.3)
    reqs = {f"r{i}": random_tokens(CONFIG["vocab"], 1104 if i == 0 else 9 + i, 60 + i) for i in range(16)}
    cfg, w = plain.load_folder(d)
    return d, reqs, {rid: plain.forward(cfg, w, t) for rid, t in reqs.items()}


def steps(reqs):
    """900 tokens of the long prompt; the rest of it but four beside the short ones; four decoded tokens of all."""
    portion = lambda rid, a, b: {"id": rid, "tokens": reqs[rid][a:b], "want": list(range(b - a))}
    out = [[portion("r0", 0, 900)], [portion(rid, 900 if rid == "r0" else 0, len(t) - 4) for rid, t in reqs.items()]]
    out += [[portion(rid, len(t) - k, len(t) - k + 1) for rid, t in reqs.items()] for k in (4, 3, 2, 1)]
    return [{"step": i, "entries": e, "end": list(reqs) if i == len(out) - 1 else []} for i, e in enumerate(out)]


@pytest.mark.parametrize("graphs", [False, True])
def test_steps_on_tcgen05(case, graphs, monkeypatch):
    from iian_b200.engine.replay import TraceReplayer
    from iian_b200.ops import cuda_backend
    d, reqs, want = case
    got = []
    for tc in (True, False):
        monkeypatch.setattr(cuda_backend.CudaKernels, "LATENT_TC", tc)
        before = cuda_backend.LAUNCHES_BY_ENTRY.get("latent_attention_tc", 0)
        rp = TraceReplayer.from_folder(d, "bfloat16", 2048, 16, 16)
        rp.runner.cuda_graphs = graphs
        got.append(replay_and_collect(rp, steps(reqs)))
        rp.runner.check_device_status()
        assert rp.runner.num_graphs == (1 if graphs else 0)
        # two layers of the prompt and of the mixed step; of decoded tokens the layer without a window, at a graph's warm-up and capture, where
        # the bucket's context decides (eagerly 16 tokens of 32 heads behind 1,104 are too few)
        assert cuda_backend.LAUNCHES_BY_ENTRY.get("latent_attention_tc", 0) - before == (0 if not tc else 6 if graphs else 4)
    scale = max(w.abs().max().item() for w in want.values())
    for g in got:                                # the bound of the other whole-model tests of this design in bfloat16
        assert len(g) == sum(len(t) for t in reqs.values())
        bad = first_bad(g, want, 3e-2 * scale)
        assert bad is None, f"first wrong logits at {bad}; worst {max_error(g, want)}"


LINE = {**CONFIG, "layers": [layer(mixer(16, 32, 64, 32, 256, None, 64), dense(128)), layer(mixer(16, 32, 64, 32, 512, 700, 64), dense(128))]}


@pytest.fixture(scope="module")
def line_case(tmp_path_factory):
    from iian_b200.config.registry import get_architecture
    from iian_b200.weights.random_init import write_model_folder
    d = os.path.join(str(tmp_path_factory.mktemp("line")), "galodra")
    arch = get_architecture("Galodra")
    write_model_folder(d, arch, arch.load_config(LINE), seed=22, store_dtype=torch.bfloat16, std=0.08, norm_jitter=0.3)
    reqs = {f"r{i}": random_tokens(LINE["vocab"], (1104, 1900)[i] if i < 2 else 9 + 17 * i, 80 + i) for i in range(14)}
    cfg, w = plain.load_folder(d)
    return d, reqs, {rid: plain.forward(cfg, w, t) for rid, t in reqs.items()}


@pytest.mark.parametrize("graphs", [False, True])
def test_decoded_tokens_with_keys_as_rows(line_case, graphs, monkeypatch):
    """14 requests, then 13 without the longest: one graph for 16 and contexts of 1,025 to 2,048, replayed with padding and two sets of lengths."""
    from iian_b200.engine.replay import TraceReplayer
    from iian_b200.ops import cuda_backend
    d, reqs, want = line_case
    portion = lambda rid, a, b: {"id": rid, "tokens": reqs[rid][a:b], "want": list(range(b - a))}
    todo = [{"step": i, "entries": [portion(rid, 0, len(t) - 4)], "end": []} for i, (rid, t) in enumerate(reqs.items())]
    for k in (4, 3, 2, 1):
        todo.append({"step": len(todo), "entries": [portion(rid, len(t) - k, len(t) - k + 1) for rid, t in reqs.items() if rid != "r1" or k > 2],
                     "end": ["r1"] if k == 3 else [r for r in reqs if r != "r1"] if k == 1 else []})
    scale = max(w.abs().max().item() for w in want.values())
    for line in (True, False):
        monkeypatch.setattr(cuda_backend.CudaKernels, "latent_line_pays", lambda self, s, new, *rest, line=line: line and new == 1)
        before = cuda_backend.LAUNCHES_BY_ENTRY.get("latent_line", 0)
        rp = TraceReplayer.from_folder(d, "bfloat16", 8192, 16, 16)
        rp.runner.cuda_graphs = graphs
        got = replay_and_collect(rp, todo)
        rp.runner.check_device_status()
        assert rp.runner.num_graphs == (1 if graphs else 0)
        # two layers, in each of four steps or at a graph's warm-up and capture
        assert cuda_backend.LAUNCHES_BY_ENTRY.get("latent_line", 0) - before == (0 if not line else 4 if graphs else 8)
        assert len(got) == sum(len(t) for t in reqs.values()) - 2
        bad = first_bad(got, want, 3e-2 * scale)             # as above
        assert bad is None, f"first wrong logits at {bad}; worst {max_error(got, want)}"
