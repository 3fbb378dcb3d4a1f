"""W4A16 products with up to 17 tokens at the sizes where the launch rules change: strips shared by clusters of every size, groups
that leave warps without work, both sides of the line to the tensor-core kernel, against 64-bit sums."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

# (output features, input features): clusters of 1, 2, 3, 4, 7 and 8 CTAs on a strip, and a strip count that fills no cluster evenly
SHAPES = [(8192, 1024), (7104, 4096), (4096, 4096), (4096, 11008), (3520, 8192), (2048, 8192), (1280, 8192), (32, 8192), (64, 128)]


@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("silu", [False, True])
def test_strips_shared_by_clusters(n, k, silu):
    from lmdeploy_b200 import turbomind as tm
    from perf import cases
    if silu and n % 64:
        pytest.skip("pairs of columns come in blocks of 64")
    w = cases._linear(cases._gen(5, n), n, k)
    exact = cases._exact_weight(cases._gen(5, n), n, k)
    op = tm.LlamaLinear(0)
    for tokens in (1, 2, 8, 9, 12, 16, 17):
        x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(tokens)).half()
        n_out = n // 2 if silu else n
        buf = torch.full((tokens + 1, n_out), 777.0, dtype=torch.float16, device="cuda")
        op.forward(buf[:tokens], x, tokens, w, op.kFusedSiluFfn if silu else op.kGemm)
        op.gemm_s4_f16_.handle.check_device_status(torch.cuda.current_stream().cuda_stream)
        assert bool((buf[tokens] == 777.0).all())
        y, size = x.double() @ exact, x.double().abs() @ exact.abs()
        # one rounding of the result, and weights that are not rounded to fp16 where the products are summed per group
        slack = y.abs() * 2.0 ** -11 + size * (2.0 ** -11 + k * 2.0 ** -24) + 1e-7
        if silu:
            gate, up = y[:, 0::2], y[:, 1::2]
            y = torch.nn.functional.silu(gate) * up
            # gate and up are rounded to fp16 first (again 2^-11); |silu'| <= 1.1
            slack = 2 * (1.1 * slack[:, 0::2] * up.abs() + torch.nn.functional.silu(gate).abs() * slack[:, 1::2]) + y.abs() * 2.0 ** -11 + 1e-6
        over = ((buf[:tokens].double() - y).abs() / slack).max().item()
        assert over <= 1.0, f"{n} x {k}, {tokens} tokens: {over:.2f} of the bound"


# rings of three groups beside the sums of a large cluster, strips for which clusters of eight or seven do not all find room
@pytest.mark.parametrize("n,k", [(1280, 28672), (1312, 32768), (1760, 8192), (1760, 28672), (2016, 4096)])
@pytest.mark.parametrize("tokens", [1, 8, 12])
def test_long_strips_shared_by_clusters(n, k, tokens):
    from lmdeploy_b200 import turbomind as tm
    from perf import cases
    w = cases._linear(cases._gen(5, n), n, k)
    exact = cases._exact_weight(cases._gen(5, n), n, k)
    op = tm.LlamaLinear(0)
    x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(tokens)).half()
    out = torch.empty(tokens, n, dtype=torch.float16, device="cuda")
    op.forward(out, x, tokens, w, op.kGemm)
    op.gemm_s4_f16_.handle.check_device_status(torch.cuda.current_stream().cuda_stream)
    y, size = x.double() @ exact, x.double().abs() @ exact.abs()
    over = ((out.double() - y).abs() / (y.abs() * 2.0 ** -11 + size * (2.0 ** -11 + k * 2.0 ** -24) + 1e-7)).max().item()
    assert over <= 1.0, f"{over:.2f} of the bound"


def test_the_line_between_the_kernels_can_be_drawn_and_taken_back():
    """gemm_tc_min_n: the two kernels round differently, so a product's bits tell which one ran."""
    from lmdeploy_b200 import lib as l, turbomind as tm
    from perf import cases
    n, k, tokens = 11008, 4096, 16
    w = cases._linear(cases._gen(5, n), n, k)
    x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).half()
    op = tm.LlamaLinear(0)
    op.gemm_s4_f16_.handle = h = l.Handle(0)

    def product():
        out = torch.empty(tokens, n, dtype=torch.float16, device="cuda")
        op.forward(out, x, tokens, w, op.kGemm)
        h.check_device_status(torch.cuda.current_stream().cuda_stream)
        return out

    by_size = product()
    h.set_option("gemm_tc_min_n", 17)
    drawn = product()
    h.set_option("gemm_tc_min_n", -1)
    assert not torch.equal(by_size, drawn) and torch.equal(by_size, product())
    with pytest.raises(l.TmError):
        h.set_option("gemm_tc_min_n", 0)
    h.close()


@pytest.mark.parametrize("batch", [1, 2, 8, 9, 13])
def test_folded_norm_with_few_sequences(batch):
    """Residual add + RMSNorm folded into the GEMMs around it, by the column-owner kernel and by either kernel on either side, against
    norm kernels of their own: the bounds of the driver's test with 24 sequences, and the same bits from run to run."""
    import numpy as np
    from tests.test_gpu_llama import CFG, build
    model, _, _ = build(True, max_batch=16)
    steps, rng = 4, np.random.default_rng(batch)
    forced = np.full((steps, batch), -1, np.int32)
    forced[0] = rng.integers(0, CFG["vocab_size"], batch)
    runs, stream = [], torch.cuda.Stream()
    with torch.cuda.stream(stream):
        for fold in (1, 0, 1):
            model.handle.set_option("fold_norm", fold)
            st, logits = model.new_state(batch, steps, np.zeros(batch, np.int32), forced, keep_logits=True), []
            for _ in range(steps):
                model.decode(st, 1, use_graph=True, stream=stream.cuda_stream)
                stream.synchronize()
                logits.append(st.logits.cpu().numpy().copy())
            model.check_status(stream.cuda_stream)
            runs.append((np.stack(logits), model.last_launches()))
    model.close()
    (a, launches), (b, separate), (again, _) = runs
    assert separate - launches == 2 * CFG["num_layer"] - 1
    err = np.abs(a - b)
    assert err.max() <= 3e-2 and err.mean() / np.abs(b).mean() <= 5e-3, (err.max(), err.mean() / np.abs(b).mean())
    assert np.array_equal(a, again)


# column tiles that end inside a box of the weight, one and many groups, both classes of token tiles and their edges
@pytest.mark.parametrize("n,k", [(32, 128), (288, 384), (288, 4224), (4128, 1024), (38016, 256)])
@pytest.mark.parametrize("tokens", [17, 63, 64, 65, 127, 129])
@pytest.mark.parametrize("silu", [False, True])
def test_tensor_core_tiles_at_their_edges(n, k, tokens, silu):
    from lmdeploy_b200 import turbomind as tm
    from perf import cases
    if silu:
        n = n // 64 * 64 or 64
    w = cases._linear(cases._gen(5, n), n, k)
    exact = cases._exact_weight(cases._gen(5, n), n, k)
    op = tm.LlamaLinear(0)
    x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(tokens)).half()
    buf = torch.full((tokens + 1, n // 2 if silu else n), 777.0, dtype=torch.float16, device="cuda")
    op.forward(buf[:tokens], x, tokens, w, op.kFusedSiluFfn if silu else op.kGemm)
    op.gemm_s4_f16_.handle.check_device_status(torch.cuda.current_stream().cuda_stream)
    assert bool((buf[tokens] == 777.0).all())
    y, size = x.double() @ exact, x.double().abs() @ exact.abs()
    slack = y.abs() * 2.0 ** -11 + size * k * 2.0 ** -24 + 1e-7  # one rounding of the result, fp32 sums
    if silu:  # gate and up are rounded to fp16 first; |silu'| <= 1.1
        gate, up = y[:, 0::2], y[:, 1::2]
        y = torch.nn.functional.silu(gate) * up
        slack = 2 * (1.1 * slack[:, 0::2] * up.abs() + torch.nn.functional.silu(gate).abs() * slack[:, 1::2]) + y.abs() * 2.0 ** -11 + 1e-6
    over = ((buf[:tokens].double() - y).abs() / slack).max().item()
    assert over <= 1.0, f"{over:.2f} of the bound"


@pytest.mark.parametrize("n,k,tokens", [(4096, 4096, 1), (4096, 11008, 8), (22016, 4096, 4), (12288, 4096, 40), (22016, 4096, 300)])
def test_a_weight_written_by_the_kernel_ahead(n, k, tokens):
    """The packed weight, its scales and the tokens that copies just ahead of a direct call write are the ones it multiplies (copies let
    nothing start early; a kernel that does is in test_gpu_direct_calls.py)."""
    from lmdeploy_b200 import turbomind as tm
    from perf import cases
    sides = [cases._linear(cases._gen(s, n), n, k) for s in (1, 2)]
    xs = [torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(s)).half() for s in (1, 2)]
    op = tm.LlamaLinear(0)
    want = []
    for w, x in zip(sides, xs):
        want.append(torch.empty(tokens, n, dtype=torch.float16, device="cuda"))
        op.forward(want[-1], x, tokens, w, op.kGemm)
    live = tm.LlamaDenseWeight(k, n, sides[0].kernel.clone(), tm.WeightType.kINT4, None, sides[0].scales_and_zeros.clone(), 128)
    x, outs = xs[0].clone(), torch.zeros(16, tokens, n, dtype=torch.float16, device="cuda")
    for i in range(16):
        x.copy_(xs[i % 2])
        live.scales_and_zeros.copy_(sides[i % 2].scales_and_zeros)
        live.kernel.copy_(sides[i % 2].kernel)
        op.forward(outs[i], x, tokens, live, op.kGemm)
    for i in range(16):
        assert torch.equal(outs[i], want[i % 2]), i


@pytest.mark.parametrize("tokens", [1, 200])
def test_a_dense_weight_written_by_the_kernel_ahead(tokens):
    from lmdeploy_b200 import lib as l
    n, k, h = 4096, 4096, l.default_handle(0)
    ws, x = [torch.randn(n, k, device="cuda").bfloat16() for _ in range(2)], torch.randn(tokens, k, device="cuda").bfloat16()
    live, outs = torch.empty_like(ws[0]), torch.zeros(8, tokens, n, dtype=torch.bfloat16, device="cuda")
    for i in range(8):
        live.copy_(ws[i % 2])
        l.check(l.lib.tm_gemm_dense(h.ptr, outs[i].data_ptr(), n, 0, x.data_ptr(), k, live.data_ptr(), k, tokens, n, k, l.TM_DTYPE_BF16,
                                    torch.cuda.current_stream().cuda_stream), "tm_gemm_dense")
    for i in range(2, 8):
        assert torch.equal(outs[i], outs[i % 2])
    assert not torch.equal(outs[0], outs[1])
