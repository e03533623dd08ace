"""Prompts of requests beside the rest of a program: other threads' CUDA work, calls outside inference mode, memory."""
import threading

import pytest
import torch

from bitmtp_b200 import fast_generate, generate, native, synthetic
from bitmtp_b200.fast_runtime import GraphAtlas

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
SIGMA = 256
ATLASES = {"ar": (8, (1,), ("ar",)), "d4": (4, (1, 4, 5, 6, 7, 8, 9), ("ar", "draft", "verify"))}


def _served(kind, seed=1):
    block, widths, roles = ATLASES[kind]
    cfg = synthetic.make_config(synthetic.TINY, block_size=block)
    model = generate.model_from_state(generate.args_from_config(cfg), synthetic.make_state(cfg, seed=seed), DEV)
    model.prepare_merged_weights(max_positions=SIGMA + max(widths))
    atlas = GraphAtlas(model, model.args, DEV, segment_ladder=(SIGMA,), m_set=widths, roles=roles, capture_verbose=False)
    return cfg, model, atlas


def _request(kind, cfg, model, atlas, seq):
    policy = fast_generate.fast_ar_generate if kind == "ar" else fast_generate.fast_speculative_generate
    return policy(model, atlas, synthetic.random_prompt(seq, cfg["vocab_size"], seed=seq), max_gen_len=6, eos_ids=())[0].tolist()


@pytest.mark.parametrize("kind", list(ATLASES))
def test_requests_of_an_atlas_without_slab_graphs_capture_nothing(kind, monkeypatch):
    """The third prompt of a length is launched like the first, also by a program that captured that shape itself."""
    cfg, model, atlas = _served(kind)
    ids = synthetic.random_prompt(40, cfg["vocab_size"], seed=40)[0].to(DEV)
    want = _request(kind, cfg, model, atlas, 40)
    for _ in range(3):
        atlas.prefill(ids, SIGMA)

    def refuse(*args, **kwargs):
        raise AssertionError("a request began a capture")
    monkeypatch.setattr(torch.cuda, "graph", refuse)
    monkeypatch.setattr(torch.cuda.CUDAGraph, "capture_begin", refuse)
    for seq in (40, 57, 57, 57):
        tokens = _request(kind, cfg, model, atlas, seq)
        assert seq != 40 or tokens == want


@pytest.mark.parametrize("kind", list(ATLASES))
@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
def test_prefill_follows_a_request(kind, mode):
    """Requests run in inference mode; a prompt outside it finds what they left usable, and leaves it so."""
    cfg, model, atlas = _served(kind)
    want = _request(kind, cfg, model, atlas, 30)
    ids = synthetic.random_prompt(30, cfg["vocab_size"], seed=30)[0].to(DEV)
    with mode():
        logits = atlas.prefill(ids, SIGMA)
    assert int(logits.argmax()) == want[0]
    assert _request(kind, cfg, model, atlas, 30) == want


@pytest.mark.parametrize("kind", list(ATLASES))
def test_threads_serve_their_own_models(kind):
    """Two threads, each with a model, an atlas and a stream of its own, prompts whose lengths come back; a third that
    allocates, copies to the host and synchronises."""
    served = [_served(kind, seed) for seed in (1, 2)]
    lengths = range(20, 50, 3)
    want = [[_request(kind, *s, seq) for seq in lengths] for s in served]
    failures, stop = [], threading.Event()

    def guarded(body):
        def run():
            try:
                with torch.cuda.stream(torch.cuda.Stream()):
                    body()
            except Exception as e:                       # noqa: BLE001 - whatever it is, the test reports it
                failures.append(repr(e)[:300])
        return threading.Thread(target=run, daemon=True)

    def serve(i):
        for _ in range(3):
            for seq, tokens in zip(lengths, want[i]):
                assert _request(kind, *served[i], seq) == tokens, seq

    def other_work():
        n = 0
        while not stop.is_set():
            n += 1
            torch.ones(1000 + 7919 * n % 1000000, device=DEV).sum().item()
            torch.cuda.synchronize()

    other = guarded(other_work)
    threads = [guarded(lambda i=i: serve(i)) for i in (0, 1)]
    for t in (other, *threads):
        t.start()
    for t in threads:
        t.join(120)
    stop.set()
    other.join(30)
    assert not failures and not any(t.is_alive() for t in (other, *threads))
    assert native.lib().bm_device_error() == 0


def test_prompt_lengths_share_one_workspace(monkeypatch):
    """Prompts of many lengths hold no more memory than the longest one and the longest of one pass, and a prompt of a new
    length leaves the captured passes of the others alone."""
    sigma = 1400
    cfg = synthetic.make_config(dict(synthetic.TINY, n_heads=16, n_kv_heads=8, dim=512, ffn_dim=512), block_size=8)
    model = generate.model_from_state(generate.args_from_config(cfg), synthetic.make_state(cfg, seed=1), DEV)
    model.prepare_merged_weights(max_positions=sigma + 1)
    atlas = GraphAtlas(model, model.args, DEV, segment_ladder=(sigma,), m_set=(1,), roles=("ar",), capture_verbose=False)

    def prefill(seq):
        logits = atlas.prefill(synthetic.random_prompt(seq, cfg["vocab_size"], seed=seq)[0].to(DEV), sigma).clone()
        torch.cuda.synchronize()
        return logits

    want = {seq: prefill(seq) for seq in (300, 1279, sigma)}
    held = torch.cuda.memory_allocated(DEV)
    for seq in range(320, sigma, 60):
        prefill(seq)
    assert torch.cuda.memory_allocated(DEV) <= held
    for seq in (300, 300, 1395):
        prefill(seq)

    def refuse(*args, **kwargs):
        raise AssertionError("a pass was captured again")
    monkeypatch.setattr(torch.cuda, "graph", refuse)
    prefill(301)
    for _ in range(2):
        assert torch.equal(prefill(300).view(torch.int32), want[300].view(torch.int32))
    assert native.lib().bm_device_error() == 0


def test_a_pass_captured_by_the_caller_leaves_nothing_behind():
    """The first prompt of a model under the caller's own capture: its buffers belong to that graph, and prompts before its
    first replay, after it and beside it come out the same."""
    cfg, model, atlas = _served("ar")
    ids = synthetic.random_prompt(40, cfg["vocab_size"], seed=40)[0].to(DEV)
    _request("ar", cfg, model, atlas, 9)                        # loads what the head needs; too short for a pass
    with torch.no_grad():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = atlas.prefill(ids, SIGMA)
        got = [atlas.prefill(ids, SIGMA).clone() for _ in range(3)]
        graph.replay()
        got += [captured.clone(), atlas.prefill(ids, SIGMA).clone()]
        graph.replay()
        got.append(captured.clone())
        cache = model.forward_sdlm_prefill(token_values=ids, cache=[None] * model.args.n_layers)
    torch.cuda.synchronize()
    assert native.lib().bm_device_error() == 0
    for logits in got:
        assert torch.equal(logits.view(torch.int32), cache[-1:].view(torch.int32))
