"""The engine where the attention cuts its KV range and leaves its result quantised (caches of 1024 cells and more), eagerly and in a graph:
logits bit-identical to the separate quantiser's, greedy tokens those of the graph composed from the oracle's ops, rows within the 3e-2 that a few
int8 rounding flips explain (test_gpu_model.py)."""
import numpy as np
import pytest

from llama_ref import OracleLlama, tiny_model

pytestmark = pytest.mark.gpu


def _config(d_model, n_head, n_kv_head):
    from cactus_b200.engine import LlamaConfig
    return LlamaConfig(n_layer=2, d_model=d_model, n_head=n_head, n_kv_head=n_kv_head, d_ff=2 * d_model, vocab=320)


def _ubatches(rng, vocab):
    """27 prompt tokens of three sequences, 7 and 3 and 1 tokens that continue them, as (tokens, pos, seq, slots)."""
    lens, head = [9, 4, 14], 27
    out = [(np.concatenate([np.arange(n) for n in lens]), np.concatenate([np.full(n, s) for s, n in enumerate(lens)]))]
    for counts in ((3, 1, 3), (1, 1, 1), (0, 0, 1)):
        out.append((np.concatenate([lens[s] + np.arange(n) for s, n in enumerate(counts)]), np.concatenate([np.full(n, s) for s, n in enumerate(counts)])))
        lens = [a + b for a, b in zip(lens, counts)]
    at = 0
    for pos, seq in out:
        yield rng.integers(0, vocab, len(pos)), pos.astype(np.int64), seq.astype(np.int64), at + np.arange(len(pos))
        at += len(pos)
    assert head == len(out[0][0])


# a cluster of 2; more splits than a cluster has CTAs, which the combine pass adds; H D = 576, which no quantised output takes; heads of 128
@pytest.mark.parametrize("d_model,n_head,n_kv_head,n_cells,quantises", [(256, 4, 2, 1024, True), (256, 4, 2, 8192, True), (576, 9, 3, 1024, False), (512, 4, 1, 2048, True)])
@pytest.mark.parametrize("use_graphs", [False, True])
def test_quantising_attention_in_the_engine(oracle, d_model, n_head, n_kv_head, n_cells, quantises, use_graphs):
    from cactus_b200.engine import LlamaEngine, LlamaWeights
    cfg = _config(d_model, n_head, n_kv_head)
    arrays = tiny_model(oracle, cfg)
    engines = [LlamaEngine(LlamaWeights.from_numpy(cfg, arrays), n_cells, max_tokens=32, use_graphs=use_graphs) for _ in range(2)]
    assert engines[0].fa_quant_max_tokens == (32 if quantises else 0)
    engines[1].fa_quant_max_tokens = 0
    ref = OracleLlama(oracle, cfg, arrays, n_cells, acc_mode=1)
    for ubatch in _ubatches(np.random.default_rng(1), cfg.vocab):
        got, ids = (a.copy() for a in engines[0].decode(*ubatch))
        assert np.array_equal(got, engines[1].decode(*ubatch)[0])
        want = ref.decode(*ubatch)
        assert np.array_equal(ids, want.argmax(-1))
        assert (np.abs(got - want).max(axis=1) / np.abs(want).max()).max() < 3e-2


def test_where_the_query_tiled_kernel_is_considered(oracle):
    """From 128 tokens on the query-tiled kernel may take a prompt, which needs the attention's result in f32."""
    from cactus_b200.engine import LlamaEngine, LlamaWeights
    cfg = _config(256, 4, 2)
    arrays = tiny_model(oracle, cfg)
    engines = [LlamaEngine(LlamaWeights.from_numpy(cfg, arrays), 1024, max_tokens=128, use_graphs=False) for _ in range(2)]
    assert engines[0].fa_quant_max_tokens == 127
    engines[1].fa_quant_max_tokens = 0
    tokens = np.random.default_rng(2).integers(0, cfg.vocab, 128)
    for T in (127, 128):
        args = (tokens[:T], np.arange(T), np.zeros(T, np.int64), np.arange(T))
        assert np.array_equal(engines[0].decode(*args)[0], engines[1].decode(*args)[0])
        for e in engines:
            e.clear()
