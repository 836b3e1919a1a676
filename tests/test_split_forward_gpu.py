"""Forward products that are split over k: bias and GELU ride the reduction.  And products of 9 to 64 rows in three bf16 parts."""
import pytest

pytestmark = pytest.mark.gpu


def _problem(torch, m, k, n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x, w = torch.randn(m, k, device="cuda", generator=gen), torch.randn(k, n, device="cuda", generator=gen) * k ** -0.5
    b = torch.randn(n + 1, device="cuda", generator=gen)[1:]      # not 16-byte aligned
    return x, w, b, x.double() @ w.double() + b.double()


@pytest.mark.parametrize("m,k,n", [(65, 3072, 768), (200, 1540, 132), (500, 2052, 260), (70, 512, 772), (300, 3072, 768), (1000, 3072, 768), (1540, 3072, 768)])
@pytest.mark.parametrize("mode,tol", [(0, 1e-5), (1, 2e-3)])
def test_epilogue_behind_split_k(m, k, n, mode, tol):
    """Several parts, the last one shorter, ragged rows and columns; tolerances of the modes.  A first call may be inside a capture and gives the same bits there."""
    import torch
    import gpt_b200
    x, w, b, want = _problem(torch, m, k, n, m + k + n)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    for captured in (False, True):
        with torch.cuda.stream(stream):
            be = gpt_b200.Backend(0, stream.cuda_stream, mode)
            y, act = torch.full((m + 1, n), 7.0, device="cuda"), torch.full((m + 1, n), 7.0, device="cuda")
            stream.synchronize()
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=stream):
                    be.device_linear_activation_fused_forward(y, act, x, w, b, True, 1, m, k, n)
                graph.replay()
            else:
                be.device_linear_activation_fused_forward(y, act, x, w, b, True, 1, m, k, n)
            be.synchronize()
            assert float((y[:m].double() - want).abs().max()) <= tol * float(want.abs().max())
            assert float((act[:m].double() - torch.nn.functional.gelu(want, approximate="tanh")).abs().max()) <= tol * float(want.abs().max())
            assert (y[m] == 7).all() and (act[m] == 7).all()
            if captured:
                assert torch.equal(y, eager[0]) and torch.equal(act, eager[1])
                del graph
            eager = y, act
            be.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_scratch_of_a_captured_call_outlives_its_growth(mode):
    """Scratch that grows inside a capture, between the calls of one graph, and after it: the graph still owns the memory that it writes."""
    import torch
    import gpt_b200
    m, k, n, big, huge = 300, 3072, 768, (100, 768, 50304), (128, 768, 50304)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    need = lambda m, k, n, *form: gpt_b200.plan_layer(sms, mode, m, n, k, *form)["scratch_kib"]
    assert 0 < need(m, k, n, False, True, True) < need(*big, False, False) < need(*huge, False, False)
    x, w, b, _ = _problem(torch, m, k, n, mode)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        be = gpt_b200.Backend(0, stream.cuda_stream, mode)
        y, act, want = (torch.empty(m, n, device="cuda") for _ in range(3))
        h, wte, logits = torch.randn(*huge[:2], device="cuda"), torch.randn(huge[2], huge[1], device="cuda"), torch.zeros(huge[0], huge[2], device="cuda")
        call = lambda: be.device_linear_activation_fused_forward(y, act, x, w, b, True, 1, m, k, n)
        large = lambda size: be.device_unembedding_forward(logits, h, wte, 1, *size)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            call()                # no scratch yet
            large(big)            # more than there is
            call()
        large(huge)
        exact, tol = h.double() @ wte.double().t(), 1e-5 if mode == 0 else 2e-3
        be.synchronize()
        assert float((logits.double() - exact).abs().max()) <= tol * float(exact.abs().max())
        call()
        want.copy_(y)
        stream.synchronize()
        fill = [torch.full((4 << 20,), float("nan"), device="cuda") for _ in range(16)]     # takes what was freed
        y.zero_()
        logits.zero_()
        graph.replay()
        be.synchronize()
        assert torch.equal(y, want) and all(t.isnan().all() for t in fill)
        assert float((logits[:big[0]].double() - exact[:big[0]]).abs().max()) <= tol * float(exact.abs().max())
        del graph
        be.close()


@pytest.mark.parametrize("m", [9, 16, 17, 33, 64])
@pytest.mark.parametrize("k,n", [(768, 2304), (1028, 1284), (36, 132), (3072, 768), (772, 19204)])
def test_rows_in_three_parts(m, k, n):
    """Ragged steps of 16 k, shares of k in clusters, several column tiles per block, both layouts of the weights.  At most seven truncating additions (2^-23 of
    the lesser products' sum each) before fp32 sums of k / 16 terms: below 5e-7 of the result's size, and no worse than the fp32 FMA kernel."""
    import torch
    import gpt_b200
    if m > 16 and k * n < 512 * 512:
        pytest.skip("another kernel's size")
    x, w, b, want = _problem(torch, m, k, n, m * 3 + k + n)
    wt = w.t().contiguous()
    be = gpt_b200.Backend(0, torch.cuda.current_stream().cuda_stream, 0)
    errors = {}
    for tensor in (1, 0):
        be.set_option("skinny_tensor", tensor)
        y, act, z = (torch.full((m + 1, n), 7.0, device="cuda") for _ in range(3))
        be.device_linear_activation_fused_forward(y, act, x, w, b, True, 1, m, k, n)
        be.device_unembedding_forward(z, x, wt, 1, m, k, n)
        be.synchronize()
        assert (y[m] == 7).all() and (act[m] == 7).all() and (z[m] == 7).all()
        plain, gelu = want - b.double(), torch.nn.functional.gelu(want, approximate="tanh")
        errors[tensor] = [float((got[:m].double() - ref).norm() / ref.norm()) for got, ref in ((y, want), (act, gelu), (z, plain))]
    for new, old in zip(errors[1], errors[0]):
        assert new <= 5e-7 and new <= old, errors
    be.close()


@pytest.mark.parametrize("m", [16, 32, 64])
def test_one_product_per_element(m):
    """Sums of a single product, as in a row that is zero but for one k: 2^-24 of it for the fp32 addition of the two accumulators' values, seven truncations
    (2^-23 each) of the lesser products, which are below 2^-6 of it, and 2^-30 for the one product that is left out: below 1.3 x 2^-24."""
    import torch
    import gpt_b200
    k, n = 772, 2308
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.zeros(m, k, device="cuda")
    x[torch.arange(m, device="cuda"), torch.arange(m, device="cuda") * 12] = 1.0 + torch.rand(m, device="cuda", generator=gen)
    x[0, 0] = 1.0077059                                # with 1.007767 the lesser products are as large as they get
    w = 1.0 + torch.rand(k, n, device="cuda", generator=gen)
    w[0, 0] = 1.007767
    want = x.double() @ w.double()
    be = gpt_b200.Backend(0, torch.cuda.current_stream().cuda_stream, 0)
    y, z = torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda")
    be.device_linear_activation_fused_forward(y, None, x, w, torch.zeros(n, device="cuda"), False, 1, m, k, n)
    be.device_unembedding_forward(z, x, w.t().contiguous(), 1, m, k, n)
    be.synchronize()
    for got in (y, z):
        assert float(((got.double() - want) / want).abs().max()) <= 1.3 * 2.0 ** -24
    be.close()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("m,k,n", [(9, 772, 2308), (16, 36, 132), (32, 768, 768), (64, 260, 19204)])
def test_infinite_operands_of_some_rows(m, k, n, mode):
    """Infinities, NaN and overflow in x, w and the last k give what fp32 FMAs give: the same infinite and NaN outputs, and the others as ever."""
    import torch
    import gpt_b200
    if m > 16 and k * n < 512 * 512:
        pytest.skip("another kernel's size")
    x, w, b, _ = _problem(torch, m, k, n, m + k + n)
    inf = float("inf")
    x[1, 5], x[2, k - 1], x[m - 1, 0] = inf, -inf, float("nan")
    x[4, 7], x[4, 8] = inf, -inf
    x[5, 3], w[3, 10] = 3e38, 3e38                     # overflows
    w[9, 2], w[k - 1, n - 1], w[11, 6] = -inf, inf, 0.0
    x[6, 11], x[6, 9] = inf, 0.0                       # inf x 0 at column 6, 0 x -inf at column 2
    be = gpt_b200.Backend(0, torch.cuda.current_stream().cuda_stream, mode)
    got = []
    for tensor in (1, 0):
        be.set_option("skinny_tensor", tensor)
        y, act, z = (torch.full((m + 1, n), 7.0, device="cuda") for _ in range(3))
        be.device_linear_activation_fused_forward(y, act, x, w, b, True, 1, m, k, n)
        be.device_unembedding_forward(z, x, w.t().contiguous(), 1, m, k, n)
        be.synchronize()
        got.append((y, act, z))
    for new, old in zip(*got):
        assert torch.equal(new.isnan(), old.isnan()) and torch.equal(new.isposinf(), old.isposinf()) and torch.equal(new.isneginf(), old.isneginf())
        assert old.isposinf().any() and old.isfinite().all(1).any()
        ok = old.abs() < 100                           # all but those of the overflowing row and column
        assert int(ok.sum()) > old.numel() // 3 and float((new[ok] - old[ok]).abs().max()) <= 2e-6 * float(old[ok].abs().max())
    be.close()


@pytest.mark.parametrize("m,k,n", [(600, 768, 3072), (1540, 768, 2304), (1000, 260, 1028), (2050, 3072, 768)])
@pytest.mark.parametrize("mode,tol", [(0, 1e-5), (1, 2e-3)])
def test_one_wave_of_tiles_backward(m, k, n, mode, tol):
    """Weight and input gradients as one wave of one-CTA tiles, whole and in parts of k: added to what is there, tolerances of the modes."""
    import torch
    import gpt_b200
    x, w, b, _ = _problem(torch, m, k, n, m + n)
    gy = torch.randn(m, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(m))
    be = gpt_b200.Backend(0, torch.cuda.current_stream().cuda_stream, mode)
    gx, gw, gb = torch.full((m + 1, k), 7.0, device="cuda"), torch.full_like(w, 3.0), torch.full((n,), 5.0, device="cuda")
    be.device_linear_backward(gx, gw, gb, gy, x, w, 1, m, k, n)
    be.synchronize()
    for got, want in ((gx[:m], gy.double() @ w.double().t()), (gw, x.double().t() @ gy.double() + 3.0), (gb, gy.double().sum(0) + 5.0)):
        assert float((got.double() - want).abs().max()) <= tol * float(want.abs().max())
    assert (gx[m] == 7).all()
    be.close()


@pytest.mark.parametrize("m", [9, 64])
def test_weights_written_just_before_the_call(m):
    """Option decode_early_launch = 1 covers the per-warp kernels only: products of 9 to 64 rows see weights that the launch before them wrote."""
    import torch
    import gpt_b200
    k, n = 768, 19200
    be = gpt_b200.Backend(0, torch.cuda.current_stream().cuda_stream, 0)
    be.set_option("decode_early_launch", 1)
    x, pre = torch.randn(m, k, device="cuda"), torch.full((n, k), 20.0, device="cuda")      # where the derivative of GELU is one
    w, z, out = torch.empty(n, k, device="cuda"), torch.empty(m, n, device="cuda"), torch.empty(m, k, device="cuda")
    grad = torch.randn(m, n, device="cuda")
    for seed in range(4):
        source = torch.randn(n, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))
        w.fill_(100.0)
        torch.cuda.synchronize()
        be.device_activation_backward(w, source, pre, 1, n, k)
        be.device_unembedding_forward(z, x, w, 1, m, k, n)
        be.synchronize()
        assert float((z.double() - x.double() @ source.double().t()).norm() / z.double().norm()) <= 1e-6
        w.fill_(100.0)
        torch.cuda.synchronize()
        be.device_activation_backward(w, source, pre, 1, n, k)
        be.linear_backward_input(out, grad, w.view(k, n), m, k, n)
        be.synchronize()
        want = grad.double() @ source.view(k, n).double().t()
        assert float((out.double() - want).norm() / want.norm()) <= 1e-6
    be.close()


@pytest.mark.parametrize("option,value", [("max_sms", 20), ("max_sms", 1), ("skinny_cluster", 1), ("skinny_cluster", 4)])
def test_rows_on_part_of_the_machine(option, value):
    import torch
    import gpt_b200
    be = gpt_b200.Backend(0, torch.cuda.current_stream().cuda_stream, 0)
    be.set_option(option, value)
    for m, k, n in ((12, 772, 772), (64, 260, 5124)):
        x, w, b, want = _problem(torch, m, k, n, m)
        y, z = torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda")
        be.device_linear_activation_fused_forward(y, None, x, w, b, False, 1, m, k, n)
        be.device_unembedding_forward(z, x, w.t().contiguous(), 1, m, k, n)
        be.synchronize()
        for got, ref in ((y, want), (z, want - b.double())):
            assert float((got.double() - ref).norm() / ref.norm()) <= 5e-7
    be.close()


@pytest.mark.parametrize("m,k,n,which", [(600, 768, 3072, "y gx gw"), (1540, 3072, 768, "y gw"), (2048, 768, 2304, "gx gw"), (3000, 3072, 768, "y gw")])
def test_one_wave_of_tf32_tiles_keeps_its_chains_short(m, k, n, which):
    """Operands that TF32 holds exactly, all positive: a chain of 32 truncating additions (at most 2^-23 of the partial sum each) before the fp32 sums, 16 on average over
    a growing sum, and 1e-6 for those: below 3e-6 of the result.  Chains of a whole k of 3072 are off by 2.2e-5.  The products that one wave of tiles takes."""
    import torch
    import gpt_b200
    gen = torch.Generator(device="cuda").manual_seed(m)
    exact = lambda *shape: (torch.rand(*shape, device="cuda", generator=gen).view(torch.int32) & -8192).view(torch.float32)
    x, w, gy = exact(m, k), exact(k, n), exact(m, n)
    be = gpt_b200.Backend(0, torch.cuda.current_stream().cuda_stream, 1)
    y, gx, gw, gb = torch.empty(m, n, device="cuda"), torch.empty(m, k, device="cuda"), torch.zeros(k, n, device="cuda"), torch.zeros(n, device="cuda")
    be.device_linear_activation_fused_forward(y, None, x, w, torch.zeros(n, device="cuda"), False, 1, m, k, n)
    be.device_linear_backward(gx, gw, gb, gy, x, w, 1, m, k, n)
    be.synchronize()
    for name, got, want in (("y", y, x.double() @ w.double()), ("gx", gx, gy.double() @ w.double().t()), ("gw", gw, x.double().t() @ gy.double())):
        if name in which.split():
            assert float((got.double() - want).norm() / want.norm()) <= 3e-6, name
    be.close()
