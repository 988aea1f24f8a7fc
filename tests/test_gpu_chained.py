"""Decode steps whose launches overlap their predecessors give the bits of the serial ones, eager and as a graph, and the choice stays in its scope."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _steps(model, kv_dtype, chained, graph, monkeypatch):
    from mary_b200.runtime.batch import BatchMeta
    from mary_b200.runtime.kv_cache import PagedKVCache
    monkeypatch.setattr(type(model), "CHAIN_MAX_ROWS", 64 if chained else 0)
    g = torch.Generator(device="cuda").manual_seed(1)
    spec = model.kv_spec()
    cache = PagedKVCache(spec["num_layers"], 64, 16, spec["kv_heads"], spec["head_dim"], dtype=torch.bfloat16, device="cuda", kv_dtype=kv_dtype)
    for l in range(spec["num_layers"]):
        for t in (cache.k[l], cache.v[l]):
            if kv_dtype:
                t.codes, t.sz = t.quantize(torch.randn(t.shape, device="cuda", generator=g))
            else:
                t.copy_(torch.randn(t.shape, device="cuda", generator=g))
    kv = [100, 37, 260]
    table = np.random.default_rng(0).permutation(64)[:60].reshape(3, 20).astype(np.int32)
    meta = BatchMeta.build([1, 1, 1], kv, table, 16, "cuda")
    ids = torch.randint(0, 4096, (3,), device="cuda", dtype=torch.int32, generator=g)
    with torch.no_grad():
        outs = [model(ids, meta, cache).clone() for _ in range(3)]
        if graph:
            torch.cuda.synchronize()
            gr = torch.cuda.CUDAGraph()
            with torch.cuda.graph(gr):
                out = model(ids, meta, cache)
            for _ in range(3):
                gr.replay()
            outs.append(out)
    torch.cuda.synchronize()
    return outs


@pytest.mark.parametrize("kv_dtype", [None, "int8"])
def test_chained_decode_equals_serial(kv_dtype, monkeypatch):
    from mary_b200.models.gemma4 import Gemma4Model, Gemma4TextConfig
    from mary_b200.models.gemma4.weights import init_random_
    from mary_b200.ops import cuda as K
    cfg = Gemma4TextConfig(hidden_size=1024, num_hidden_layers=6, num_attention_heads=8, num_key_value_heads=4, head_dim=128,
                           intermediate_size=4096, vocab_size=4096, sliding_window=64)
    model = Gemma4Model(cfg, dtype=torch.bfloat16, device="cuda")
    init_random_(model, 0)
    want = _steps(model, kv_dtype, False, False, monkeypatch)
    for graph in (False, True):
        for got in _steps(model, kv_dtype, True, graph, monkeypatch):
            assert torch.equal(got, want[0])
    assert all(torch.equal(w, want[0]) for w in want) and K.last_status() == 0


def test_scope_is_the_threads_own():
    from mary_b200.ops import cuda as K
    seen = []
    with K.chained:
        with K.chained:
            pass
        t = threading.Thread(target=lambda: seen.append(K.lib().mary_pdl_scope(-1)))
        t.start()
        t.join()
        assert K.lib().mary_pdl_scope(1) == 1
    assert seen == [-1] and K.lib().mary_pdl_scope(-1) == -1
