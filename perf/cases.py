"""Performance cases: the work a user has this framework do, through its public entry points.

Three kinds of case:

* ``mul_mat``   -- ``ops.mul_mat(weight, x)``: one quantised product, as a host that drives single ops calls it;
* ``attention`` -- ``ops.flash_attn_ext(q, k, v, mask, scale)``: one attention op over the unified f16 KV cache;
* ``step``      -- ``LlamaEngine.decode(tokens, pos, seq, slots)``: one whole ubatch (decode tokens, a prompt, or both).

A case names sizes only; weights, activations, caches and token ids come from the seed.  Sequence lengths are part of the
case (drawn from its ``ragged`` number), so that the work of a case does not depend on the seed.
"""
from __future__ import annotations

import numpy as np
import torch

from cactus_b200 import ops
from cactus_b200.engine import LLAMA_3_8B, LLAMA_32_1B, LlamaEngine, LlamaWeights, random_blocks

ARCH = {"1b": LLAMA_32_1B, "8b": LLAMA_3_8B}
WTYPE = {"q4_0": ops.Q4_0, "q8_0": ops.Q8_0}
BLOCK = {"q4_0": 18, "q8_0": 34}


def _mul_mat(wtype, K, M, N, **kw):
    return dict(kind="mul_mat", wtype=wtype, K=K, M=M, N=N, **kw)


def _attention(D, H, Hkv, seqs, lo, hi, q_max, tokens_max, cells, ragged, **kw):
    return dict(kind="attention", D=D, H=H, Hkv=Hkv, seqs=seqs, lo=lo, hi=hi, q_max=q_max, tokens_max=tokens_max, cells=cells, ragged=ragged, **kw)


def _step(arch, seqs, lo, hi, prompt, cells, ragged, **kw):
    return dict(kind="step", arch=arch, seqs=seqs, lo=lo, hi=hi, prompt=prompt, cells=cells, ragged=ragged, **kw)


def listed():
    return [
        # a projection of the 4096-wide model for one token, for a handful, and for a full ubatch of prompt tokens
        _mul_mat("q4_0", 4096, 4096, 1, name="mul_mat_q4_4096_n1"),
        _mul_mat("q4_0", 4096, 4096, 8, name="mul_mat_q4_4096_n8"),
        _mul_mat("q4_0", 4096, 4096, 512, name="mul_mat_q4_4096_n512"),
        # the down projection for the odd number of tokens that a ragged ubatch has
        _mul_mat("q4_0", 14336, 4096, 77, name="mul_mat_q4_down_n77"),
        # the Q8_0 output head of the 1B model for one token
        _mul_mat("q8_0", 2048, 128256, 1, name="mul_mat_q8_head_n1"),
        # attention of a decode ubatch: one token of each of 64 ragged sequences in a 65536-cell cache
        _attention(128, 32, 8, 64, 16, 2048, 1, 64, 65536, 0, name="attention_decode_64seq"),
        # attention of a mixed ubatch: 16 ragged sequences with 1-256 query tokens each in an 8192-cell cache
        _attention(128, 32, 8, 16, 64, 4096, 256, 512, 8192, 0, name="attention_ubatch_16seq"),
        # a single user's chat on the 1B model: one token per step, logits back on the host
        _step("1b", 1, 640, 640, 0, 1024, 0, name="decode_1b_1seq"),
        # a few users on the 8B model
        _step("8b", 7, 16, 2048, 0, 16384, 1, name="decode_8b_7seq"),
        # continuous batching at its full width, all sequences decoding
        _step("8b", 64, 16, 2048, 0, 65536, 0, name="decode_8b_64seq"),
        # the prompt of a chat: 512 tokens of one sequence
        _step("1b", 0, 0, 0, 512, 1024, 0, name="prompt_1b_512"),
        # continuous batching while a new prompt comes in: 48 sequences decode, 464 tokens of the prompt fill the ubatch
        _step("8b", 48, 16, 2048, 464, 65536, 2, name="mixed_8b_512"),
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["mul_mat", "mul_mat", "attention", "step", "step"])
    if kind == "mul_mat":
        wtype = rng.choice(["q4_0", "q4_0", "q8_0"])
        K = 32 * _log_int(rng, 8, 448)
        M = _log_int(rng, 256, 32768)
        return _mul_mat(wtype, K, M, _log_int(rng, 1, 512))
    if kind == "attention":
        seqs = _log_int(rng, 1, 64)
        q_max = rng.choice([1, 1, _log_int(rng, 2, 256)])
        return _attention(rng.choice([64, 128]), rng.choice([16, 32]), 8, seqs, 16, _log_int(rng, 128, 4096), q_max, 512,
                          min(65536, 256 * max(4, _log_int(rng, 4, 256))), rng.randrange(1 << 20))
    arch = rng.choice(["1b", "8b"])
    if rng.random() < 0.6:      # all sequences decode
        return _step(arch, _log_int(rng, 1, 64), 16, _log_int(rng, 64, 2048), 0, 65536 if arch == "8b" else 16384, rng.randrange(1 << 20))
    seqs = rng.choice([0, _log_int(rng, 1, 48)])
    return _step(arch, seqs, 16, _log_int(rng, 64, 2048), _log_int(rng, 16, 464), 65536 if arch == "8b" else 16384, rng.randrange(1 << 20))


# ---- sequences in the unified cache ----------------------------------------------------------------------------------
def _lengths(seqs, lo, hi, room, ragged):
    """Cached tokens of each sequence, uniform in [lo, hi], scaled down where they do not fit the room."""
    if seqs == 0:
        return np.zeros(0, np.int64)
    lens = np.random.default_rng([7, ragged]).integers(lo, hi + 1, seqs)
    lens = np.maximum(1, np.floor(lens * min(1.0, room / lens.sum())).astype(np.int64))
    while lens.sum() > room:
        lens[np.argmax(lens)] -= 1
    return lens


def _layout(lens, cells):
    """Position and sequence of every cell: sequence after sequence, each a contiguous run."""
    cell_pos, cell_seq = np.full(cells, -1, np.int32), np.full(cells, -1, np.int32)
    head = 0
    for s, n in enumerate(lens):
        cell_pos[head:head + n] = np.arange(n)
        cell_seq[head:head + n] = s
        head += n
    return cell_pos, cell_seq, int(head)


def _attention_tokens(case):
    """Contexts, and query tokens per sequence: the last ones of each context, whose K/V are in the cache already."""
    ctx = _lengths(case["seqs"], case["lo"], case["hi"], case["cells"], case["ragged"])
    nq = np.random.default_rng([8, case["ragged"]]).integers(1, case["q_max"] + 1, case["seqs"])
    nq = np.minimum(nq, ctx)
    nq = np.maximum(1, np.floor(nq * min(1.0, case["tokens_max"] / nq.sum())).astype(np.int64))
    return ctx, nq


def _pairs(ctx, nq):
    """(query token, attended cell) pairs of causal attention."""
    return int((ctx * nq - nq * (nq - 1) // 2).sum())


def _step_tokens(case):
    """Cached lengths of the decoding sequences; then one token each, then the prompt's tokens as a new sequence."""
    lens = _lengths(case["seqs"], case["lo"], case["hi"], case["cells"] - 2 * case["seqs"] - case["prompt"], case["ragged"])
    S, P = case["seqs"], case["prompt"]
    pos = np.concatenate([lens, np.arange(P)]).astype(np.int32)
    seq = np.concatenate([np.arange(S), np.full(P, S)]).astype(np.int32)
    return lens, pos, seq


# ---- weights ----------------------------------------------------------------------------------------------------------
def _weights(cfg, gen):
    """Random weights at the scales a trained model has: the embedding sets the residual stream and a layer adds little to
    it (its two output projections are small), so that the stream carries a token through all layers.  With equal scales
    everywhere the logits would be chaotic: a last-bit difference in the first layer decides them."""
    w = LlamaWeights(cfg)
    t, d = w.tensors, cfg.d_model

    def make(wtype, K, M, std):
        return ops.QWeight.from_blocks(wtype, K, M, random_blocks(wtype, M, K, gen, std=std))
    t["token_embd.weight"] = make(cfg.head_type, d, cfg.vocab, 2.0)
    t["output.weight"] = make(cfg.head_type, d, cfg.vocab, 0.02)
    t["output_norm.weight"] = torch.ones(d, device="cuda")
    names = {"wq": "attn_q", "wk": "attn_k", "wv": "attn_v", "wo": "attn_output", "gate": "ffn_gate", "up": "ffn_up", "down": "ffn_down"}
    small = 0.02 / (2 * cfg.n_layer) ** 0.5
    for il in range(cfg.n_layer):
        for short, K, M in cfg.mul_mat_shapes():
            t[f"blk.{il}.{names[short]}.weight"] = make(cfg.layer_type, K, M, small if short in ("wo", "down") else 0.02)
        for norm in ("attn_norm", "ffn_norm"):
            t[f"blk.{il}.{norm}.weight"] = 1.0 + 0.1 * torch.randn(d, device="cuda", generator=gen)
    return w


# ---- prepare ---------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "mul_mat":
        wt, K, M = WTYPE[case["wtype"]], case["K"], case["M"]
        w = ops.QWeight.from_blocks(wt, K, M, random_blocks(wt, M, K, gen))
        return {"case": case, "w": w, "x": torch.randn((case["N"], K), device="cuda", generator=gen)}
    if case["kind"] == "attention":
        ctx, nq = _attention_tokens(case)
        total = int(ctx.sum())
        n_kv = (total + 255) // 256 * 256
        cell_pos, cell_seq, _ = _layout(ctx, n_kv)
        tok_pos = np.concatenate([np.arange(c - n, c) for c, n in zip(ctx, nq)])
        tok_seq = np.repeat(np.arange(case["seqs"]), nq)
        Nq = len(tok_pos)
        cp, cs, tp, ts = (torch.from_numpy(a.astype(np.int32)).cuda() for a in (cell_pos, cell_seq, tok_pos, tok_seq))
        mask = torch.full(((Nq + 63) // 64 * 64, n_kv), float("-inf"), dtype=torch.float16, device="cuda")
        mask[:Nq][(cs[None] == ts[:, None]) & (cp[None] <= tp[:, None])] = 0
        kv = [torch.randn((n_kv, case["Hkv"], case["D"]), device="cuda", generator=gen).half() for _ in range(2)]
        q = torch.randn((Nq, case["H"], case["D"]), device="cuda", generator=gen)
        return {"case": case, "q": q, "k": kv[0], "v": kv[1], "mask": mask, "scale": float(case["D"]) ** -0.5}
    cfg = ARCH[case["arch"]]
    lens, pos, seq = _step_tokens(case)
    T = len(pos)
    # decode steps replay a CUDA graph per token count (the engine's default); prompt ubatches come in every size and run directly
    eng = LlamaEngine(_weights(cfg, gen), case["cells"], max_tokens=T, use_graphs=case["prompt"] == 0)
    cell_pos, cell_seq, head = _layout(lens, case["cells"])
    eng.cell_pos.copy_(torch.from_numpy(cell_pos))
    eng.cell_seq.copy_(torch.from_numpy(cell_seq))
    for c in eng.k_cache + eng.v_cache:     # what the sequences' earlier ubatches left in the cache
        c[:head] = torch.randn((head, c.shape[1]), device="cuda", generator=gen).half()
    rng = np.random.default_rng(seed)
    return {"case": case, "eng": eng, "tokens": rng.integers(0, cfg.vocab, T).astype(np.int32), "pos": pos, "seq": seq,
            "slots": np.arange(head, head + T, dtype=np.int32)}


# ---- run -------------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["case"]["kind"]
    if kind == "mul_mat":
        return ops.mul_mat(state["w"], state["x"])
    if kind == "attention":
        return ops.flash_attn_ext(state["q"], state["k"], state["v"], state["mask"], state["scale"])
    eng = state["eng"]
    if state["case"]["prompt"] == 0:        # decode: the logits of every token come back for the sampler
        logits, _ = eng.decode(state["tokens"], state["pos"], state["seq"], state["slots"])
    else:                                   # prompt tokens: greedy ids come back, the logits stay where they are
        eng.decode(state["tokens"], state["pos"], state["seq"], state["slots"], want_logits=False)
        logits = eng.logits
    # the greedy ids are the argmax of these logits (ties of random logits would not compare); the last layer's cache
    # carries what all layers did to the new tokens
    return {"logits": logits, "k": eng.k_cache[-1], "v": eng.v_cache[-1]}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "mul_mat":
        K, M, N = case["K"], case["M"], case["N"]
        return {"bytes": M * (K // 32) * BLOCK[case["wtype"]] + 4 * N * K + 4 * N * M, "flops": 2 * M * K * N}
    if case["kind"] == "attention":
        ctx, nq = _attention_tokens(case)
        Nq, total, D, H = int(nq.sum()), int(ctx.sum()), case["D"], case["H"]
        n_kv = (total + 255) // 256 * 256
        return {"bytes": 4 * total * case["Hkv"] * D + 8 * Nq * H * D + 2 * Nq * n_kv, "flops": 4 * H * D * _pairs(ctx, nq)}
    cfg = ARCH[case["arch"]]
    lens, pos, _ = _step_tokens(case)
    T, kvd = len(pos), cfg.n_kv_head * cfg.head_dim
    params = sum(K * M for _, K, M in cfg.mul_mat_shapes()) * cfg.n_layer + cfg.vocab * cfg.d_model
    cells = int((lens + 1).sum()) + case["prompt"]
    pairs = int((pos.astype(np.int64) + 1).sum())
    emb = T * (cfg.d_model // 32) * {ops.Q4_0: 18, ops.Q8_0: 34}[cfg.head_type]
    return {"bytes": cfg.weight_bytes_per_step() + 4 * cells * kvd * cfg.n_layer + emb + 4 * T * cfg.vocab,
            "flops": 2 * params * T + 4 * cfg.n_head * cfg.head_dim * pairs * cfg.n_layer}


def tolerance(case):
    if case["kind"] == "mul_mat":       # exact integer dots, f32 scales and sums in another order
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "attention":     # f16 inputs, f32 softmax and sums
        return {"rel": 1e-5, "max": 1e-3}
    # every product re-quantises its input to 8 bits: a last-bit difference of an f32 sum moves a value by one of 127 steps,
    # and 16 or 32 layers of such steps end about one quantisation error (1.5e-2) apart
    return {"rel": 2.5e-2, "max": 0.25}
