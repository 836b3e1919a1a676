"""Generation steps of the GPT-2 model as one launch: against a float64 forward pass over the whole text."""
import math

import pytest

pytestmark = pytest.mark.gpu


def _shapes(c):
    L, D, H = c["num_layers"], c["d_model"], c["d_ffn"]
    return [("wte", (c["vocab_size_padded"], D)), ("wpe", (c["max_seq_len"], D)), ("ln1_w", (L, D)), ("ln1_b", (L, D)), ("qkv_w", (L, D, 3 * D)), ("qkv_b", (L, 3 * D)),
            ("proj_w", (L, D, D)), ("proj_b", (L, D)), ("ln2_w", (L, D)), ("ln2_b", (L, D)), ("up_w", (L, D, H)), ("up_b", (L, H)), ("down_w", (L, H, D)), ("down_b", (L, D)),
            ("lnf_w", (D,)), ("lnf_b", (D,))]


def _forward(torch, c, flat, tokens):
    w, at = {}, 0
    for name, shape in _shapes(c):
        n = math.prod(shape)
        w[name] = flat[at:at + n].view(shape)
        at += n
    B, T = tokens.shape
    D, H = c["d_model"], c["num_heads"]
    norm = lambda x, g, b: torch.nn.functional.layer_norm(x, (D,), g, b, 1e-5)
    x = w["wte"][tokens.long()] + w["wpe"][:T]
    mask = torch.ones(T, T, device="cuda", dtype=torch.bool).tril()
    for i in range(c["num_layers"]):
        q, k, v = (norm(x, w["ln1_w"][i], w["ln1_b"][i]) @ w["qkv_w"][i] + w["qkv_b"][i]).view(B, T, 3, H, D // H).permute(2, 0, 3, 1, 4)
        p = torch.softmax((q @ k.transpose(-1, -2) * (D // H) ** -0.5).masked_fill(~mask, -math.inf), -1)
        x = x + (p @ v).transpose(1, 2).reshape(B, T, D) @ w["proj_w"][i] + w["proj_b"][i]
        u = norm(x, w["ln2_w"][i], w["ln2_b"][i]) @ w["up_w"][i] + w["up_b"][i]
        x = x + torch.nn.functional.gelu(u, approximate="tanh") @ w["down_w"][i] + w["down_b"][i]
    return norm(x, w["lnf_w"], w["lnf_b"]) @ w["wte"].t()


GPT2 = dict(d_model=768, num_heads=12, d_ffn=3072, vocab_size_padded=1000)
SIZES = {
    "gpt2": GPT2,
    "head8": dict(d_model=64, num_heads=8, d_ffn=308, vocab_size_padded=332),           # ragged column groups and slices
    "head128": dict(d_model=384, num_heads=3, d_ffn=1284, vocab_size_padded=64),
    "wide": dict(d_model=1600, num_heads=25, d_ffn=6400, vocab_size_padded=260),         # up to three items per block, five heads per slice
    "medium": dict(d_model=1024, num_heads=16, d_ffn=4096, vocab_size_padded=516),       # two heads per slice, slices of more than 256 rows
    "large": dict(d_model=1280, num_heads=20, d_ffn=5120, vocab_size_padded=516),        # two items per block, three heads per slice
}


@pytest.mark.parametrize("size,batch,layers,prompt,steps", [
    ("gpt2", 1, 2, 60, 12), ("gpt2", 2, 2, 125, 8), ("gpt2", 1, 12, 1, 6), ("head8", 1, 3, 7, 40), ("head8", 2, 1, 31, 3), ("head128", 2, 2, 5, 70),
    ("wide", 1, 2, 130, 4), ("wide", 2, 1, 9, 3), ("head128", 1, 1, 1, 1),
    ("gpt2", 3, 2, 61, 6), ("gpt2", 8, 3, 9, 4), ("gpt2", 9, 1, 33, 3), ("gpt2", 16, 1, 5, 3), ("gpt2", 17, 2, 130, 4), ("gpt2", 32, 1, 3, 3), ("gpt2", 33, 1, 64, 3), ("gpt2", 64, 2, 70, 5),
    ("head8", 5, 2, 3, 30), ("head8", 40, 1, 17, 3), ("head128", 12, 2, 6, 5), ("wide", 4, 1, 20, 3), ("wide", 50, 1, 8, 3), ("gpt2", 65, 1, 5, 2)])
def test_generation_step_matches_the_whole_forward_pass(size, batch, layers, prompt, steps):
    """Logits of every step within 1e-5 of their scale (fp32 sums of up to 6400 terms, layer after layer; the same bound as for the
    operator-by-operator step)."""
    import torch
    import gpt_b200
    c = dict(max_seq_len=prompt + steps + 1, num_layers=layers, **SIZES[size])
    c["vocab_size"] = c["vocab_size_padded"] - 3
    gen = torch.Generator(device="cuda").manual_seed(batch + prompt)
    model = gpt_b200.Model(c, 0, torch.cuda.current_stream().cuda_stream, gpt_b200.MODE_3XTF32, use_grad=False)
    flat = torch.cat([(torch.randn(*shape, device="cuda", generator=gen) * 0.05 + (1.0 if name in ("ln1_w", "ln2_w", "lnf_w") else 0.0)).reshape(-1) for name, shape in _shapes(c)])
    assert flat.numel() == model.num_params
    model.load_weights(flat.cpu().numpy())
    text = torch.randint(0, c["vocab_size"], (batch, prompt + steps), device="cuda", dtype=torch.int32, generator=gen)
    want = _forward(torch, c, flat.double(), text)[:, prompt:]
    for _ in range(2):      # a second text in the same buffers
        model.generate_begin(text[:, :prompt].contiguous(), batch, prompt, prompt + steps)
        out = torch.full((steps, batch, c["vocab_size_padded"]), float("nan"), device="cuda")
        for i in range(steps):
            model.generate_step(text[:, prompt + i].contiguous(), out[i])
        torch.cuda.synchronize()
        got = out.transpose(0, 1).double()
        assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())
    assert model.generate_position == prompt + steps
    model.close()


@pytest.mark.parametrize("batch,prompt,steps", [(1, 8, 40), (2, 8, 24), (5, 8, 16), (12, 5, 12), (64, 2, 6)])
def test_one_launch_is_as_exact_as_the_operators(batch, prompt, steps):
    """GPT-2 124M's layers: the logits' error against 64 bits is no larger than that of the step that runs operator by operator (option
    skinny_rows) on the same cache, texts and weights; both are fixed, so there is nothing to allow for."""
    import torch
    import gpt_b200
    c = dict(max_seq_len=64, num_layers=12, vocab_size=2000, **dict(GPT2, vocab_size_padded=2000))
    gen = torch.Generator(device="cuda").manual_seed(batch)
    parts = []
    for name, shape in _shapes(c):
        t = torch.randn(*shape, device="cuda", generator=gen) * (0.004 if name in ("proj_w", "down_w") else 0.02)
        parts.append((t + (1.0 if name in ("ln1_w", "ln2_w", "lnf_w") else 0.0)).reshape(-1))
    flat = torch.cat(parts)
    text = torch.randint(0, c["vocab_size"], (batch, prompt + steps), device="cuda", dtype=torch.int32, generator=gen)
    want = _forward(torch, c, flat.double(), text)[:, prompt:].transpose(0, 1)
    errors = []
    for operators in (False, True):
        model = gpt_b200.Model(c, 0, torch.cuda.current_stream().cuda_stream, gpt_b200.MODE_3XTF32, use_grad=False)
        model.load_weights(flat.cpu().numpy())
        if operators:
            model.set_option("skinny_rows", 64)
        model.generate_begin(text[:, :prompt].contiguous(), batch, prompt, prompt + steps)
        out = torch.empty(steps, batch, c["vocab_size_padded"], device="cuda")
        before = model.launch_count()
        for i in range(steps):
            model.generate_step(text[:, prompt + i].contiguous(), out[i])
        assert (model.launch_count() - before > 2 * steps) == operators
        torch.cuda.synchronize()
        errors.append(float((out.double() - want).norm() / want.norm()))
        model.close()
    assert errors[0] <= errors[1], errors


def test_a_grid_barrier_that_nothing_reaches_ends_and_is_reported():
    """The wait gives up after its limit, for the whole block and in every later launch; the context stays usable."""
    import torch
    import gpt_b200
    b = gpt_b200.Backend(0)
    assert b.lib.gptb200_selftest_grid_barrier(b.handle, 0) == 1 and b.lib.gptb200_selftest_grid_barrier(None, 10) == 1
    for polls in (1, 1000):
        assert b.lib.gptb200_selftest_grid_barrier(b.handle, polls) == 0
        with pytest.raises(gpt_b200.GptB200Error) as e:
            b.synchronize()
        assert e.value.status == 4 and "device status 110" in str(e.value)
    b.synchronize()
    b.close()


def _generated(torch, c, batch, text, prompt, prepare=lambda model: None, between=lambda model, i: None, graph=False):
    """(logits of the steps, launches of each) of a text in a new model, and the float64 logits."""
    import gpt_b200
    steps = text.shape[1] - prompt
    gen = torch.Generator(device="cuda").manual_seed(7)
    flat = torch.cat([(torch.randn(*shape, device="cuda", generator=gen) * 0.05 + (1.0 if name in ("ln1_w", "ln2_w", "lnf_w") else 0.0)).reshape(-1) for name, shape in _shapes(c)])
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        model = gpt_b200.Model(c, 0, stream.cuda_stream, gpt_b200.MODE_3XTF32, use_grad=False)
        model.load_weights(flat.cpu().numpy())
        prepare(model)
        model.generate_begin(text[:, :prompt].contiguous(), batch, prompt, prompt + steps)
        out, launches = torch.full((steps, batch, c["vocab_size_padded"]), float("nan"), device="cuda"), []
        token, logits, captured = torch.empty(batch, device="cuda", dtype=torch.int32), torch.empty(batch, c["vocab_size_padded"], device="cuda"), None
        for i in range(steps):
            between(model, i)
            token.copy_(text[:, prompt + i])
            before = model.launch_count()
            if captured:
                captured.replay()
            else:
                model.generate_step(token, logits)
                if graph and i == 0:     # the steps after the first are replays of the second's capture
                    captured = torch.cuda.CUDAGraph()
                    before = model.launch_count()
                    with torch.cuda.graph(captured, stream=stream):
                        model.generate_step(token, logits)
            launches.append(model.launch_count() - before)
            out[i].copy_(logits)
        stream.synchronize()
        model.synchronize()
        del captured
        model.close()
    return out.transpose(0, 1).double(), launches, _forward(torch, c, flat.double(), text)[:, prompt:]


def _case(torch, size, batch, layers, prompt, steps):
    c = dict(max_seq_len=prompt + steps + 1, num_layers=layers, **SIZES[size])
    c["vocab_size"] = c["vocab_size_padded"] - 3
    return c, torch.randint(0, c["vocab_size"], (batch, prompt + steps), device="cuda", dtype=torch.int32, generator=torch.Generator(device="cuda").manual_seed(batch + prompt))


FEW, ROWS = 1, 2     # launches of a step: the kernel of one or two rows; the other with the un-embedding


@pytest.mark.parametrize("size,batch,prompt,steps,kernel", [
    ("medium", 1, 70, 3, FEW), ("medium", 2, 130, 3, FEW), ("large", 1, 33, 3, FEW), ("large", 2, 150, 2, FEW), ("wide", 1, 60, 3, FEW),
    ("medium", 2, 401, 2, ROWS), ("large", 2, 256, 2, ROWS), ("medium", 12, 9, 3, ROWS), ("large", 64, 5, 2, ROWS)])
def test_widths_beyond_768(size, batch, prompt, steps, kernel):
    """Several items per block, several heads per slice, slices of more than one body of weights: 1e-5 of the logits' scale, as above."""
    import torch
    c, text = _case(torch, size, batch, 2, prompt, steps)
    got, launches, want = _generated(torch, c, batch, text, prompt)
    assert launches == [kernel] * steps
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())


def test_the_kernel_changes_with_the_position():
    """From the kernel of one or two rows to the operators and on to the other kernel, over one cache."""
    import torch
    c, text = _case(torch, "large", 2, 1, 198, 61)
    got, launches, want = _generated(torch, c, 2, text, 198)
    assert launches[:3] == [FEW] * 3 and all(n > ROWS for n in launches[3:58]) and launches[58:] == [ROWS] * 3
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())


@pytest.mark.parametrize("size,batch,prompt,steps,kernel", [("gpt2", 1, 20, 8, FEW), ("medium", 2, 20, 5, FEW), ("gpt2", 8, 20, 6, ROWS), ("gpt2", 64, 3, 5, ROWS), ("gpt2", 3, 20, 6, 0)])
def test_a_captured_step_is_replayed_at_every_position(size, batch, prompt, steps, kernel):
    """The position and the barriers' counters live on the device: one capture serves all steps after the first.  Three rows over a short cache are
    captured operator by operator."""
    import torch
    c, text = _case(torch, size, batch, 2, prompt, steps)
    got, launches, want = _generated(torch, c, batch, text, prompt, graph=True)
    assert (launches[0] == kernel or (kernel == 0 and launches[0] > ROWS)) and launches[1:] == [0] * (steps - 1)
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())


@pytest.mark.parametrize("size,batch,sms,kernel", [("gpt2", 1, 100, FEW), ("head128", 2, 89, FEW), ("gpt2", 20, 90, ROWS), ("gpt2", 1, 60, 0), ("gpt2", 9, 16, 0)])
def test_steps_on_part_of_the_sms(size, batch, sms, kernel):
    """Option max_sms: more items per block on fewer blocks, operators where too few are left."""
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines are drawn for 148 SMs")
    c, text = _case(torch, size, batch, 2, 11, 4)
    got, launches, want = _generated(torch, c, batch, text, 11, prepare=lambda model: model.set_option("max_sms", sms))
    assert launches == [kernel] * 4 if kernel else min(launches) > ROWS
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())


@pytest.mark.parametrize("batch", [1, 8])
def test_the_form_may_change_between_steps(batch):
    """Options are read at every step: one launch, operators, one launch over the same cache, and fewer SMs than planned for."""
    import torch
    c, text = _case(torch, "gpt2", batch, 2, 15, 7)
    changes = {2: ("skinny", 0), 4: ("skinny", 1), 5: ("max_sms", 120)}
    got, launches, want = _generated(torch, c, batch, text, 15, between=lambda model, i: i in changes and model.set_option(*changes[i]))
    one = FEW if batch <= 2 else ROWS
    assert launches[:2] == [one] * 2 and min(launches[2:4]) > ROWS and launches[4:] == [one] * 3
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())


@pytest.mark.parametrize("name,index", [("wte", (5, 7)), ("up_w", (0, 3, 9)), ("qkv_w", (0, 11, 100))])
def test_infinite_weights_give_what_the_operators_give(name, index):
    """One infinite weight: which logits are infinite and which are NaN is the same with products in three bf16 parts as with fp32 FMAs.  (Inside the layers an infinite
    value meets a norm or a softmax in every form; an infinite embedding also reaches the un-embedding as a weight.)"""
    import torch
    import gpt_b200
    batch, prompt, steps = 12, 5, 4
    c = dict(max_seq_len=64, num_layers=2, vocab_size=600, **dict(GPT2, vocab_size_padded=600))
    gen = torch.Generator(device="cuda").manual_seed(3)
    parts = []
    for n, shape in _shapes(c):
        t = torch.randn(*shape, device="cuda", generator=gen) * 0.02 + (1.0 if n in ("ln1_w", "ln2_w", "lnf_w") else 0.0)
        if n == name:
            t[index] = float("inf")
        parts.append(t.reshape(-1))
    text = torch.randint(6, 600, (batch, prompt + steps), device="cuda", dtype=torch.int32, generator=gen)
    text[3, prompt + 1] = 5
    got = []
    for operators in (False, True):
        model = gpt_b200.Model(c, 0, torch.cuda.current_stream().cuda_stream, gpt_b200.MODE_TF32, use_grad=False)
        model.load_weights(torch.cat(parts).cpu().numpy())
        if operators:
            model.set_option("skinny_rows", 64)
            model.set_option("skinny_tensor", 0)
        model.generate_begin(text[:, :prompt].contiguous(), batch, prompt, prompt + steps)
        out = torch.empty(steps, batch, 600, device="cuda")
        for i in range(steps):
            model.generate_step(text[:, prompt + i].contiguous(), out[i])
        torch.cuda.synchronize()
        got.append(out)
        model.close()
    new, old = got
    assert torch.equal(new.isnan(), old.isnan()) and torch.equal(new.isposinf(), old.isposinf()) and torch.equal(new.isneginf(), old.isneginf())
    assert not old.isfinite().all() and (name != "wte" or old.isposinf().any())
