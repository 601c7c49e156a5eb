"""Steps that are not pure decoding replay a CUDA graph of their exact shape from the second time
the shape is seen: the first run is eager, the second captures, the rest replay. The logits must
not care which of the three a step was, nor whose requests, contents and pages it carries."""

import numpy as np
import pytest
import torch

from plain_reference import plain_config, plain_forward
from tiny_configs import TINY, random_ids, tiny_config, tiny_tensors

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def make(dtype, **core_options):
    from matricxon_b200.engine.core import EngineCore, model_from_tensors

    store = torch.bfloat16 if dtype == "bfloat16" else torch.float32
    tensors = tiny_tensors("B", store)
    model = model_from_tensors(tiny_config("B"), tensors, dtype=dtype, device=DEV)
    core = EngineCore(model, max_cache_tokens=1024, max_requests=8, poison_cache=True, **core_options)
    return core, plain_config(TINY["B"][0]), {k: v.float() for k, v in tensors.items()}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_repeated_mixed_shape_is_captured_and_replayed(dtype):
    from matricxon_b200.engine.step import StepEntry

    core, cfg, weights = make(dtype)
    runner, cache = core.runner, core.cache
    vocab = cfg["vocab"]
    sequences = {"d1": random_ids(40, vocab, 1), "d2": random_ids(55, vocab, 2), "p": random_ids(83, vocab, 3)}
    reference = {rid: plain_forward(cfg, weights, ids, dtype=torch.float32).numpy() for rid, ids in sequences.items()}
    for rid in sequences:
        cache.add_request(rid)
    runner.run([StepEntry("d1", sequences["d1"][:20]), StepEntry("d2", sequences["d2"][:30])])
    done = {"d1": 20, "d2": 30, "p": 0}
    got = {rid: {} for rid in sequences}
    modes = []
    for turn in range(8):                       # the same shape eight times: 1 + 1 + 10 tokens
        entries = [StepEntry("d1", sequences["d1"][done["d1"]:done["d1"] + 1], [0]),
                   StepEntry("d2", sequences["d2"][done["d2"]:done["d2"] + 1], [0]),
                   StepEntry("p", sequences["p"][done["p"]:done["p"] + 10], [9, 0])]
        graphs_before = len(runner._shape_graphs)
        logits = runner.run(entries).clone()
        modes.append(len(runner._shape_graphs) - graphs_before)
        got["d1"][done["d1"]] = logits[0]
        got["d2"][done["d2"]] = logits[1]
        got["p"][done["p"] + 9] = logits[2]
        got["p"][done["p"]] = logits[3]
        done["d1"] += 1
        done["d2"] += 1
        done["p"] += 10
    runner.check_status()
    assert modes == [0, 1, 0, 0, 0, 0, 0, 0]            # eager, captured, then replayed
    assert len(runner._shape_graphs) == 1 and not runner._graphs
    for rid, rows in got.items():
        for position, row in rows.items():
            ref = reference[rid][position]
            limit = 2e-5 if dtype == "float32" else 0.03 * float(np.abs(reference[rid]).max())
            assert np.abs(row.cpu().numpy() - ref).max() <= limit, (rid, position)
    # other requests, other pages, the same shape: the graph serves them too
    for rid in sequences:
        cache.free_request(rid)
    fresh = {"x": random_ids(30, vocab, 4), "y": random_ids(30, vocab, 5), "z": random_ids(30, vocab, 6)}
    for rid in fresh:
        cache.add_request(rid)
    runner.run([StepEntry("x", fresh["x"][:12]), StepEntry("y", fresh["y"][:7])])
    logits = runner.run([StepEntry("x", fresh["x"][12:13], [0]), StepEntry("y", fresh["y"][7:8], [0]),
                         StepEntry("z", fresh["z"][:10], [9, 0])]).clone()
    runner.check_status()
    assert len(runner._shape_graphs) == 1
    for row, (rid, position) in zip(logits, (("x", 12), ("y", 7), ("z", 9), ("z", 0))):
        ref = plain_forward(cfg, weights, fresh[rid], dtype=torch.float32).numpy()
        limit = 2e-5 if dtype == "float32" else 0.03 * float(np.abs(ref).max())
        assert np.abs(row.cpu().numpy() - ref[position]).max() <= limit, (rid, position)


def test_graphs_of_shapes_are_bounded_and_the_oldest_goes():
    from matricxon_b200.engine.step import StepEntry

    core, cfg, weights = make("float32")
    runner, cache = core.runner, core.cache
    runner.max_shape_graphs = 2
    ids = random_ids(400, cfg["vocab"], 7)
    reference = plain_forward(cfg, weights, ids[:200], dtype=torch.float32).numpy()
    for size in (5, 6, 7, 5):                     # three shapes, two slots; 5 comes back after it went
        cache.add_request("r")
        done = 0
        for _ in range(4):
            logits = runner.run([StepEntry("r", ids[done:done + size], [size - 1])])
            assert np.abs(logits[0].cpu().numpy() - reference[done + size - 1]).max() <= 2e-5
            done += size
        cache.free_request("r")
        assert len(runner._shape_graphs) <= 2
    runner.check_status()
    assert [key[0][0] for key in runner._shape_graphs] == [7, 5]


def large(kind, dtype):
    """(core that captures, core that does not, vocabulary): layers wide enough for the kernels of real sizes (heads of 128 on
    tcgen05, products with the tokens as columns, recurrences over groups and chunks), so that a captured step chains them."""
    from matricxon_b200.engine.core import EngineCore, model_from_tensors

    store = torch.float32 if dtype == "float32" else torch.bfloat16
    if kind == "starcoder2":
        from test_gpu_real_sizes import COMMON, make_material

        raw = dict(COMMON, hidden_size=1024, num_attention_heads=8, num_key_value_heads=2, intermediate_size=8192,
                   vocab_size=2048, rope_theta=10000.0, tie_word_embeddings=False, sliding_window=400)
        config, tensors, _, _ = make_material(raw)
        vocab = 2048
    else:
        import palelix_configs as p

        raw = p.model(1024, 512, [
            p.parallel((8, 2, 128, 128, 0.08, (64, 10000.0)), (8, 8, 128, 128, 4), 1.0, 1.0, mlp=p.dense(8192)),
            p.lightning(8, 128, 128, [1 - 2.0 ** (-5 - i / 3) for i in range(8)], mlp=p.dense(8192)),
            p.delta(8, 4, 128, 128, 4, mlp=p.dense(8192))])
        tensors = p.draw(raw, 5, store)
        config, vocab = p.config_of(raw, tensors), 512
    cores = []
    for use_graphs in (True, False):
        model = model_from_tensors(config, {k: v.to(store) for k, v in tensors.items()}, dtype=dtype, device=DEV)
        cores.append(EngineCore(model, max_cache_tokens=8192, max_requests=8, poison_cache=True, use_graphs=use_graphs))
    return *cores, vocab


@pytest.mark.parametrize("kind,dtype", [("starcoder2", "bfloat16"), ("starcoder2", "float32"), ("palelix", "bfloat16")])
def test_captured_mixed_steps_chain_the_kernels_of_real_sizes(kind, dtype, monkeypatch):
    """Three decoding requests beside portions of 300 tokens: eager, captured and replayed steps, which start each kernel while
    the one before it drains (the two attention kernels at a time), give the logits of steps that do not."""
    from matricxon_b200.engine.step import StepEntry
    from matricxon_b200.ops import kernels

    captured, eager, vocab = large(kind, dtype)
    called = {}
    for name in ("gemm_columns", "gemm_columns_in_parts", "gemm_f32_split", "paged_attention_tc"):
        def counted(*args, _call=getattr(kernels, name), _name=name, **options):
            called.setdefault(_name, []).append(options.get("beside"))
            return _call(*args, **options)
        monkeypatch.setattr(kernels, name, counted)
    lengths = {"a": 20, "b": 333, "c": 700}
    ids = {rid: random_ids(n + 20, vocab, n) for rid, n in lengths.items()}
    prompt = random_ids(300 * 5, vocab, 9)

    def run(core, turns):
        for rid, n in lengths.items():
            core.cache.add_request(rid)
            core.runner.run([StepEntry(rid, ids[rid][:n])])
        core.cache.add_request("p")
        logits = []
        for turn in range(turns):
            entries = [StepEntry(rid, [ids[rid][n + turn]], [0]) for rid, n in lengths.items()]
            entries.append(StepEntry("p", prompt[300 * turn:300 * (turn + 1)], [299]))
            logits.append(core.runner.run(entries).clone())
        core.runner.check_status()
        for rid in (*lengths, "p"):
            core.cache.free_request(rid)
        return torch.stack(logits)

    want = run(eager, 5)
    called.clear()
    got = run(captured, 5)                              # eager, captured, three replays
    assert len(captured.runner._shape_graphs) == 1 and not eager.runner._shape_graphs
    if dtype == "float32":
        assert len(called["gemm_f32_split"]) > 0
    elif kind == "starcoder2":
        assert True in called["paged_attention_tc"] and len(called["gemm_columns"]) > 0
    # the same kernels on the same numbers: bit for bit
    assert bool(got.isfinite().all()) and torch.equal(got, want)
    again = run(captured, 5)                            # replays only, on other pages
    if dtype == "float32":                              # a captured prompt of 20 tokens shares its keys out as for the longest
        assert float((again - want).abs().max()) <= 2e-5
    else:
        assert torch.equal(again, want)
