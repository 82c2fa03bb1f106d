"""The layers' launch sequence from C++ (engine/host_step.py) for steps of up to 1,023 tokens: bit for bit the Python runner's, with
both prompt attentions; and what its first step may not cost."""
import pytest
import torch

import tiny
from spissa_b200 import Engine
from spissa_b200.csrc import lib as K
from spissa_b200.engine import host_step, pack_step

pytestmark = pytest.mark.gpu
# gate and up rows in blocks of 128, head sizes 64 and 128
MODELS = {64: (dict(tiny.TINY_E, intermediate_size=384, max_position_embeddings=4096), tiny.TINY_E_INIT),
          128: (dict(tiny.TINY_F, max_position_embeddings=4096), tiny.TINY_F_INIT)}


@pytest.fixture(scope="module")
def folders(tmp_path_factory):
    return {hd: str(tiny.make_folder(cfg, init, tmp_path_factory.mktemp(f"host_{hd}"))) for hd, (cfg, init) in MODELS.items()}


@pytest.mark.parametrize("hd", [64, 128])
def test_steps_of_up_to_1023_tokens_equal_the_python_runner(folders, hd):
    V = MODELS[hd][0]["vocab_size"]
    steps = [[129], [255], [256], [300, 129, 1], [64, 400, 63], [1023]]
    outs = {}
    for host in (True, False):
        engine = Engine.from_folder(folders[hd], dtype="bfloat16", max_tokens=64 * 40)
        engine.model.host_steps = host
        rows, fused = [], 0
        for i, counts in enumerate(steps):
            slots = [engine.acquire() for _ in counts]
            seqs = [tiny.random_prompt(V, n + 290, 100 * i + n) for n in counts]
            for cut in (lambda q, n: q[:n], lambda q, n: q[n:n + 30], lambda q, n: q[n + 30:]):          # the last: 260 more of each
                parts = [cut(q, n) for q, n in zip(seqs, counts)]
                fused += sum(map(len, parts)) > 1023
                rows.append(engine.step([(s, p, [0, len(p) - 1]) for s, p in zip(slots, parts)]).cpu())
            for s in slots:
                engine.release(s)
        engine.cache.check()
        if host:
            assert engine.model._host_step.runs == 3 * len(steps) and fused == 0
            s = engine.acquire()
            engine.step([(s, tiny.random_prompt(V, 1024, 7), [1023])])                                   # beyond: from Python
            assert engine.model._host_step.runs == 3 * len(steps) and engine.model._fused_prefill.runs == 1
        else:
            assert not engine.model._host_step and engine.model._fused_prefill.runs == 3 * len(steps)
        outs[host] = rows
    for a, b in zip(outs[True], outs[False]):
        assert torch.isfinite(a).all() and torch.equal(a, b)


def first_step(engine, n):
    dev = torch.device("cuda:0")
    slot = engine.acquire()
    pages = engine.cache.reserve([(slot, n)])
    return pages, pack_step([(slot, tiny.random_prompt(100, n, n), [n - 1])], [0], pages.tables, dev)


def test_the_first_step_does_not_wait_for_the_device(folders):
    engine = Engine.from_folder(folders[64], dtype="bfloat16", max_tokens=64 * 8)
    pages, step = first_step(engine, 200)
    torch.cuda.synchronize()
    torch.cuda.set_sync_debug_mode("error")
    try:
        assert engine.model._host_runner(step, engine.cache)                    # the layers' records
    finally:
        torch.cuda.set_sync_debug_mode("default")
    tables = {r.inv_freq for r in engine.model._host_step.layers}
    assert len(tables) == 1                                                     # equal frequency tables are one


def test_records_of_another_cache_are_made_anew(folders):
    one, two = (Engine.from_folder(folders[64], dtype="bfloat16", max_tokens=64 * 8) for _ in range(2))
    _, step = first_step(one, 100)
    runner = one.model._host_step or (one.model._host_runner(step, one.cache) and one.model._host_step)
    pools = [r.k_pool for r in runner.layers]
    assert runner.takes(step, two.cache) and [r.k_pool for r in runner.layers] != pools
    assert runner.takes(step, one.cache) and [r.k_pool for r in runner.layers] == pools
    assert runner.cache() is one.cache                                          # the cache itself, not a number that another may get


def test_short_steps_ask_for_no_attention_of_long_ones(folders, monkeypatch):
    asked, load = [], K.load
    monkeypatch.setattr(K, "load", lambda m, *a, **k: (asked.append(m), load(m, *a, **k))[1])
    monkeypatch.setattr(host_step, "_bound", 0)
    engine = Engine.from_folder(folders[64], dtype="bfloat16", max_tokens=64 * 16)
    s = engine.acquire()
    engine.step([(s, tiny.random_prompt(777, 255, 1), [254])])
    assert engine.model._host_step.runs == 1 and "flash_tc" not in asked
    engine.step([(s, tiny.random_prompt(777, 256, 2), [255])])
    assert engine.model._host_step.runs == 2 and "flash_tc" in asked


@pytest.mark.parametrize("hd", [64, 128])
def test_norm_weights_at_any_address(folders, hd):
    """Weights that a program hands over as parts of one buffer, at odd places."""
    import json
    from pathlib import Path

    from spissa_b200 import LlamaConfig
    cfg = LlamaConfig.from_dict(json.loads((Path(folders[hd]) / "config.json").read_text()))
    H = MODELS[hd][0]["hidden_size"]
    g = torch.Generator(device="cuda:0").manual_seed(1)

    def tensors():
        probe = Engine.from_folder(folders[hd], dtype="bfloat16", max_tokens=64)
        return {w.name: torch.empty(w.shape, device="cuda:0").normal_(0, 0.02, generator=g).bfloat16() for w in probe.model.weight_specs()}
    plain = tensors()
    odd = {}
    for name, t in plain.items():
        if t.dim() == 1:
            room = torch.empty(H + 1, dtype=t.dtype, device=t.device)
            room[1:] = t
            t = room[1:]
            assert t.data_ptr() % 4 == 2
        odd[name] = t
    rows = []
    for weights in (plain, odd):
        engine = Engine(cfg, weights, "bfloat16", 64 * 8, 2, "cuda:0")
        s = engine.acquire()
        rows.append([engine.step([(s, tiny.random_prompt(500, n, n), [n - 1])]).cpu() for n in (40, 200, 1)])
    assert all(torch.isfinite(a).all() and torch.equal(a, b) for a, b in zip(*rows))
