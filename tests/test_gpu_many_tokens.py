"""Products with many tokens: the dense kernel and the W4A16 GEMM that expands its weight first (both with few columns and many
tokens; the bf16 pairs of CTAs are in test_gpu_dense_pairs.py), at the edges of their tiles, against 64-bit sums of the same operands."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _check(got, want, scale, k, digits, what):
    # one rounding of the result to `digits` binary digits, and fp32 sums of k products whose absolute values add up to `scale`
    bound = want.abs() * 2.0 ** -digits + scale * (k * 2.0 ** -24) + 1e-7
    over = ((got.double() - want).abs() / bound).max().item()
    assert over <= 1.0, f"{what}: {over:.2f} of the bound"


@pytest.mark.parametrize("tokens", [65, 128, 255, 256, 257, 2049])
@pytest.mark.parametrize("n_out,k,ld", [(128, 64, 128), (384, 200, 392), (1000, 136, 1000), (2080, 512, 2083)])
def test_dense_pairs(tokens, n_out, k, ld):
    """Odd column tiles, k that ends inside a block, tokens around a tile's end, rows that 16-byte stores cannot reach; both output
    types (weights this small stay with single CTAs).  Nothing beyond a row's n_out columns is written."""
    from lmdeploy_b200 import lib as l
    g = torch.Generator(device="cuda").manual_seed(tokens + n_out)
    x = torch.randn(tokens, k, device="cuda", generator=g).bfloat16()
    w = torch.randn(n_out, k, device="cuda", generator=g).bfloat16()
    want, scale = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    h = l.default_handle(0)
    for f32 in (0, 1):
        out = torch.full((tokens, ld), 7.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
        l.check(l.lib.tm_gemm_dense(h.ptr, out.data_ptr(), ld, f32, x.data_ptr(), k, w.data_ptr(), k, tokens, n_out, k, l.TM_DTYPE_BF16,
                                    _stream()), "tm_gemm_dense")
        h.check_device_status(torch.cuda.current_stream().cuda_stream)
        _check(out[:, :n_out], want, scale, k, 24 if f32 else 8, (tokens, n_out, k, f32))
        assert bool((out[:, n_out:] == 7.0).all())


@pytest.mark.parametrize("n,k,silu,tokens", [(4128, 2048, False, 6000), (4160, 4096, True, 6001), (4160, 4096, True, 8193), (20512, 4096, False, 8192)])
def test_expanded_weight(n, k, silu, tokens, monkeypatch):
    """Sizes that the launch rule sends through expanded rows (the scratch of a handle of its own: one piece, or several where the
    weight does not fit), feature counts that fill no tile of a pair."""
    from lmdeploy_b200 import lib as l
    from perf import cases
    monkeypatch.setenv("TM_B200_GEMM_SCRATCH_MB", "64")
    h = l.Handle(0)
    w = cases._linear(cases._gen(3, n), n, k)
    exact = cases._exact_weight(cases._gen(3, n), n, k)
    x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)).half()
    out = torch.empty(tokens, n // 2 if silu else n, dtype=torch.float16, device="cuda")
    launches = h.launch_count()
    l.check(l.lib.tm_gemm_s4_f16(h.ptr, out.data_ptr(), w.kernel.data_ptr(), x.data_ptr(), w.scales_and_zeros.data_ptr(), n, tokens, k, 128,
                                 int(silu), None, 0, _stream()), "tm_gemm_s4_f16")
    h.check_device_status(torch.cuda.current_stream().cuda_stream)
    pieces = -(-n * k * 2 // (64 << 20))
    assert h.launch_count() - launches == 2 * pieces
    y, scale = x.double() @ exact, x.double().abs() @ exact.abs()
    if not silu:
        _check(out, y, scale, k, 11, (n, k, tokens))
        return
    # gate and up are rounded to fp16 first; |silu'| <= 1.1
    slack = y.abs() * 2.0 ** -11 + scale * (k * 2.0 ** -24)
    gate, up = y[:, 0::2], y[:, 1::2]
    want = torch.nn.functional.silu(gate) * up
    bound = want.abs() * 2.0 ** -10 + 1.1 * slack[:, 0::2] * up.abs() + torch.nn.functional.silu(gate).abs() * slack[:, 1::2] + 1e-5
    over = ((out.double() - want).abs() / bound).max().item()
    assert over <= 1.0, f"{over:.2f} of the bound"


@pytest.mark.parametrize("n,k,tokens", [(57344, 1024, 17), (57344, 1024, 128), (40960, 2048, 100), (22016, 4096, 200)])
def test_units_cut_evenly(n, k, tokens):
    """At least as many column tiles as SMs, cut all the same: runs over several tiles, of which the first and the last are shared."""
    from lmdeploy_b200 import lib as l
    from perf import cases
    h = l.default_handle(0)
    w = cases._linear(cases._gen(4, n), n, k)
    exact = cases._exact_weight(cases._gen(4, n), n, k)
    x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)).half()
    out = torch.empty(tokens, n, dtype=torch.float16, device="cuda")
    for _ in range(2):
        l.check(l.lib.tm_gemm_s4_f16(h.ptr, out.data_ptr(), w.kernel.data_ptr(), x.data_ptr(), w.scales_and_zeros.data_ptr(), n, tokens, k, 128,
                                     0, None, 0, _stream()), "tm_gemm_s4_f16")
    h.check_device_status(torch.cuda.current_stream().cuda_stream)
    _check(out, x.double() @ exact, x.double().abs() @ exact.abs(), k, 11, (n, k, tokens))


@pytest.mark.parametrize("n,k,tokens", [(57344, 1024, 17), (22016, 4096, 200)])
def test_units_cut_evenly_wait_for_nobody(n, k, tokens):
    """A product that has a tile for every SM does not need its CTAs to run together: a bound of one cycle on the wait for a split
    tile's other CTAs changes nothing."""
    from lmdeploy_b200 import lib as l
    from perf import cases
    h = l.Handle(0)
    w = cases._linear(cases._gen(4, n), n, k)
    x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)).half()
    out = []
    for bound in (0, 1, 1, 1):
        h.set_option("gemm_wait_cycles", bound)
        launches = h.launch_count()
        out.append(torch.empty(tokens, n, dtype=torch.float16, device="cuda"))
        l.check(l.lib.tm_gemm_s4_f16(h.ptr, out[-1].data_ptr(), w.kernel.data_ptr(), x.data_ptr(), w.scales_and_zeros.data_ptr(), n, tokens, k, 128,
                                     0, None, 0, _stream()), "tm_gemm_s4_f16")
        h.check_device_status(torch.cuda.current_stream().cuda_stream)
        assert h.launch_count() - launches == 1 and torch.equal(out[-1], out[0])
    h.close()


def test_the_bound_on_split_tiles_is_not_the_dense_pipelines():
    """gemm_wait_cycles bounds the wait for a split tile's other CTAs: an expanded weight's product has none."""
    from lmdeploy_b200 import lib as l
    from perf import cases
    n, k, tokens = 4128, 2048, 6000
    h = l.Handle(0)
    w = cases._linear(cases._gen(4, n), n, k)
    x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)).half()
    out = []
    for bound in (0, 1):
        h.set_option("gemm_wait_cycles", bound)
        out.append(torch.empty(tokens, n, dtype=torch.float16, device="cuda"))
        launches = h.launch_count()
        l.check(l.lib.tm_gemm_s4_f16(h.ptr, out[-1].data_ptr(), w.kernel.data_ptr(), x.data_ptr(), w.scales_and_zeros.data_ptr(), n, tokens, k, 128,
                                     0, None, 0, _stream()), "tm_gemm_s4_f16")
        h.check_device_status(torch.cuda.current_stream().cuda_stream)
        assert h.launch_count() - launches == 2
    assert torch.equal(out[0], out[1])
    h.close()


def _enqueue(h, out, w, x, stream):
    from lmdeploy_b200 import lib as l
    n, k = w.output_dims, w.input_dims
    l.check(l.lib.tm_gemm_s4_f16(h.ptr, out.data_ptr(), w.kernel.data_ptr(), x.data_ptr(), w.scales_and_zeros.data_ptr(), n, x.shape[0], k, 128,
                                 0, None, 0, C.c_void_p(stream.cuda_stream)), "tm_gemm_s4_f16")


def test_expanded_weights_as_dependent_launches():
    """A chain of products, each with a weight of its own in the same scratch, launched with and without programmatic serialisation."""
    from lmdeploy_b200 import lib as l
    from perf import cases
    n, tokens = 4096, 6001
    h, st = l.Handle(0), torch.cuda.current_stream()
    ws = [cases._linear(cases._gen(4, i), n, n) for i in range(4)]
    x = torch.randn(tokens, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)).half()
    ends = []
    for pdl in (0, 1, 1):
        h.set_option("pdl_direct", pdl)
        y, launches = [x] + [torch.empty(tokens, n, dtype=torch.float16, device="cuda") for _ in range(len(ws))], h.launch_count()
        for _ in range(3):
            for w, a, b in zip(ws, y, y[1:]):
                _enqueue(h, b, w, a, st)
        assert h.launch_count() - launches == 3 * 2 * len(ws)
        h.check_device_status(st.cuda_stream)
        ends.append(y)
    assert all(torch.equal(a, b) for e in ends[1:] for a, b in zip(e, ends[0]))
    assert bool(torch.isfinite(ends[0][1]).all())
    h.close()


def test_streams_that_share_a_handle():
    """Products that keep an expanded weight or parts of tiles in the handle's scratch, on two streams at once: the same bits as one
    after the other."""
    from lmdeploy_b200 import lib as l
    from perf import cases
    h = l.Handle(0)
    g = torch.Generator(device="cuda").manual_seed(1)
    jobs = []  # (weight, activations): expanded, cut evenly, cut, split by the small-token kernel
    for i, (n, k, tokens) in enumerate([(4096, 4096, 6001), (57344, 1024, 17), (4096, 4096, 40), (22016, 4096, 4), (8192, 4096, 2048)]):
        jobs.append((cases._linear(cases._gen(6, i), n, k), torch.randn(tokens, k, device="cuda", generator=g).half()))
    new = lambda: [torch.empty(x.shape[0], w.output_dims, dtype=torch.float16, device="cuda") for w, x in jobs]  # noqa: E731
    one = torch.cuda.current_stream()
    want = new()
    for out, (w, x) in zip(want, jobs):
        _enqueue(h, out, w, x, one)
    h.check_device_status(one.cuda_stream)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[new() for _ in range(6)] for _ in streams]
    torch.cuda.synchronize()
    for r in range(6):
        for i in range(len(jobs)):
            for s, st in enumerate(streams):
                j = (i + 2 * s) % len(jobs)
                _enqueue(h, got[s][r][j], *jobs[j], st)
    for st in streams:
        h.check_device_status(st.cuda_stream)
    for s in range(2):
        for r in range(6):
            for j, out in enumerate(got[s][r]):
                assert torch.equal(out, want[j]), (s, r, j)
    h.close()


@pytest.mark.parametrize("n,k,tokens", [(4096, 4096, 6001), (57344, 1024, 17)])
def test_captured_products_make_do_without_scratch(n, k, tokens):
    """A caller's graph may run beside other work of the handle: products that fill the device are captured as whole tiles."""
    from lmdeploy_b200 import lib as l
    from perf import cases
    h, st = l.Handle(0), torch.cuda.Stream()
    w, exact = cases._linear(cases._gen(4, n), n, k), cases._exact_weight(cases._gen(4, n), n, k)
    x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)).half()
    out = torch.empty(tokens, n, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        launches, graph = h.launch_count(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            _enqueue(h, out, w, x, st)
        assert h.launch_count() - launches == 1
        for _ in range(2):
            out.zero_()
            graph.replay()
        h.check_device_status(st.cuda_stream)
    _check(out, x.double() @ exact, x.double().abs() @ exact.abs(), k, 11, (n, k, tokens))
    h.close()
