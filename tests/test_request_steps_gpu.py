"""Steps of several requests: long prompts side by side in one attention launch and in automatic segments, and tokens drawn by a cluster of
blocks from a vocabulary that every block has a part of."""
import ctypes

import numpy as np
import pytest

import decoder_models as dm
from oracle import budurax, lutelorn

pytestmark = pytest.mark.gpu

TOL = 3e-2      # of the logits' scale per row: bf16 models, the bound of the other decoder tests
LENGTHS = (33, 256, 257, 700, 40, 600, 64, 513, 300, 35)     # ten neighbours: eight in the first attention launch, one to three blocks of rows each


@pytest.mark.parametrize("kind", ["capped", "uncapped", "mamba"])
def test_ten_prompts_of_unequal_lengths(tmp_path, kind):
    """Every row of every request, some of them behind an earlier portion, with the segment length left to the model (256 tokens here: three segments of
    the longest)."""
    if kind == "mamba":
        c = dm.config([dm.mamba(), dm.latent(), dm.mamba(ff=None)])
        w, forward = dm.weights(c, 3), budurax.forward
    else:
        c = dm.lutelorn([dm.lightning(), dm.attention(softcap=8.0 if kind == "capped" else None), dm.lightning(ff=None)])
        w, forward = dm.lutelorn_weights(c, 3), lutelorn.forward
    rng = np.random.default_rng(4)
    texts = [rng.integers(0, c["vocab"], n) for n in LENGTHS]
    want = [forward(c, w, t) for t in texts]
    model = dm.load(tmp_path, c, w, "bfloat16")
    for before in ((0,) * len(texts), (0, 5, 0, 190, 0, 44, 31, 0, 43, 2)):
        seqs = [model.open(len(t)) for t in texts]
        early = [(q, t[:n]) for q, t, n in zip(seqs, texts, before) if n]
        if early:
            model.step(early, [0])
        rest = [(q, t[n:]) for q, t, n in zip(seqs, texts, before)]
        got = model.step(rest, range(sum(len(t) for _, t in rest)))
        assert dm.close(got, np.concatenate([full[n:] for full, n in zip(want, before)]), TOL), (kind, before)
        for q in seqs:
            model.close(q)
    model.close_model()


def _stepped(model, prompts, follow, steps):
    """(logits that each token was chosen from, what opened them) with the given tokens fed one step at a time."""
    seqs = [model.open(len(p) + steps + 1) for p in prompts]
    at = np.cumsum([len(p) for p in prompts]) - 1
    first = model.step(list(zip(seqs, prompts)), [int(a) for a in at])
    return seqs, first, [model.step([(q, [int(t)]) for q, t in zip(seqs, row)], range(len(seqs))) for row in follow]


@pytest.mark.parametrize("heads", ["random", "repeated", "tail"])
def test_tokens_from_a_large_vocabulary(tmp_path, heads):
    """40003 logits: each of the eight blocks that share a row has pieces of it, the last piece is ragged.  Winners anywhere; equal logits in every block's
    pieces (the first must win); all logits equal but the last three."""
    vocab, steps = 40003, 24
    c = dm.lutelorn([dm.lightning(ff=None)], width=64, vocab=vocab)
    w = dm.lutelorn_weights(c, 9)
    if heads == "repeated":
        w["head"] = w["head"][np.arange(vocab) % 5000]
    if heads == "tail":
        w["head"][:vocab - 3] = 0.0
    prompts = [np.random.default_rng(i).integers(0, vocab, n) for i, n in enumerate((5, 1, 9))]
    model = dm.load(tmp_path, c, w, "bfloat16")
    seqs, first, _ = _stepped(model, prompts, [], steps)
    start = first.argmax(-1)
    tokens = model.generate(seqs, start, steps)
    for q in seqs:
        model.close(q)
    seqs, _, logits = _stepped(model, prompts, np.concatenate([start[None], tokens[:-1]]), steps)
    assert np.array_equal(np.stack(logits).argmax(-1), tokens)       # numpy's argmax is the first of equals
    if heads == "random":
        assert len(set((tokens // 2048 % 8).reshape(-1))) == 8       # every block won
    elif heads == "repeated":
        assert tokens.max() < 5000
    else:
        assert set(tokens.reshape(-1)) <= {0, vocab - 3, vocab - 2, vocab - 1} and tokens.max() >= vocab - 3
    model.close_model()


def test_draws_from_a_large_vocabulary_follow_the_rule_of_one_block(tmp_path):
    """At a temperature, each token of the device loop is what sample_rows (one block per row) draws from the same logits with the same seed."""
    import torch
    import gpt_b200
    from gpt_b200 import decoder
    vocab, steps, seed, temperature = 40003, 12, 77, 1.3
    c = dm.lutelorn([dm.lightning(ff=None)], width=64, vocab=vocab)
    model = dm.load(tmp_path, c, dm.lutelorn_weights(c, 9), "bfloat16")
    prompts = [np.random.default_rng(i).integers(0, vocab, n) for i, n in enumerate((5, 1, 9))]
    seqs, first, _ = _stepped(model, prompts, [], steps)
    start = first.argmax(-1)
    tokens = model.generate(seqs, start, steps, temperature=temperature, seed=seed)
    for q in seqs:
        model.close(q)
    _, _, logits = _stepped(model, prompts, np.concatenate([start[None], tokens[:-1]]), steps)
    lib, be = decoder.load_library(), gpt_b200.Backend(0)
    out = torch.empty(len(prompts), device="cuda", dtype=torch.int32)
    for i, rows in enumerate(logits):
        rows = torch.as_tensor(np.asarray(rows), device="cuda").contiguous()
        assert lib.gptb200_sample_rows(be.handle, ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(rows.data_ptr()), len(prompts), vocab, vocab, temperature, seed, i) == 0
        be.synchronize()
        assert out.tolist() == list(tokens[i]), i
    assert len(set((tokens // 2048 % 8).reshape(-1))) >= 6
    be.close()
    model.close_model()
