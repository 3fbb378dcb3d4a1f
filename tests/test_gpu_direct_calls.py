"""GPU: direct calls are dependent launches that wait for the kernel ahead before they read anything, weights included.  The kernel ahead
here lets its dependents start at once, waits (some 100 us, bounded) and only then writes every operand."""
import ctypes as C
import os
import shutil
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
CYCLES, BLOCKS = 200000, 24


@pytest.fixture(scope="module")
def late(tmp_path_factory):
    """late(dst, src, ...): one launch per pair, the first of which the call behind does not overlap any more; the operand that is to
    be watched goes last"""
    so = str(tmp_path_factory.mktemp("late") / "liblate.so")
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                        os.path.join(ROOT, "tests", "native", "late_writer.cu"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    lib = C.CDLL(so)
    lib.late_copy_launch.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int, C.c_int, C.c_void_p]

    def write(*pairs):
        for dst, src in pairs:
            assert dst.is_contiguous() and src.is_contiguous() and dst.nbytes == src.nbytes and dst.nbytes % 16 == 0
            assert lib.late_copy_launch(dst.data_ptr(), src.data_ptr(), dst.nbytes, BLOCKS, CYCLES, torch.cuda.current_stream().cuda_stream) == 0
    return write


def _turns(late, call, live, sides):
    """`call()` -> its output, behind writers of the two sets of operands in turn, each operand last once; the same bits as behind nothing"""
    want = []
    for side in sides:
        for dst, src in zip(live, side):
            dst.copy_(src)
        torch.cuda.synchronize()
        want.append(call())
        torch.cuda.synchronize()
    assert not torch.equal(*want)
    for turn in range(2 * len(live)):
        pairs = list(zip(live, sides[turn % 2]))
        last = turn // 2
        late(*(pairs[:last] + pairs[last + 1:] + [pairs[last]]))
        got = call()
        assert torch.equal(got, want[turn % 2]), (turn, last)


# column owner (alone, in clusters), stream-K (by its size, by the option), tensor cores (up to 64 tokens, more, tiles cut for balance), expanded
@pytest.mark.parametrize("n,k,tokens,cols", [(4096, 4096, 1, 1), (22016, 4096, 1, 1), (4096, 11008, 8, 1), (8192, 1024, 16, 1), (22016, 4096, 4, 1),
                                             (22016, 4096, 8, 1), (4096, 4096, 1, 0), (1280, 8192, 8, 0), (12288, 4096, 40, 1), (4096, 11008, 16, 1),
                                             (57344, 1024, 21, 1), (22016, 4096, 300, 1), (4160, 4096, 6001, 1)])
def test_w4a16(late, n, k, tokens, cols):
    from lmdeploy_b200 import lib as l
    from perf import cases
    h = l.Handle(0)
    h.set_option("gemv_cols", cols)
    sides = []
    for s in (1, 2):
        w = cases._linear(cases._gen(s, n), n, k)
        x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(s)).half()
        sides.append((x, w.scales_and_zeros, w.kernel))
    live = [torch.empty_like(t) for t in sides[0]]

    def call():
        out = torch.empty(tokens, n, dtype=torch.float16, device="cuda")
        l.check(l.lib.tm_gemm_s4_f16(h.ptr, out.data_ptr(), live[2].data_ptr(), live[0].data_ptr(), live[1].data_ptr(), n, tokens, k, 128, 0, None, 0,
                                     torch.cuda.current_stream().cuda_stream), "tm_gemm_s4_f16")
        return out
    _turns(late, call, live, sides)
    h.check_device_status(torch.cuda.current_stream().cuda_stream)
    h.close()


@pytest.mark.parametrize("n,k,tokens,workspace", [(57344, 1024, 8, True), (22016, 4096, 16, True), (22016, 4096, 64, True), (1280, 8192, 8, False)])
def test_w4a16_with_a_workspace_or_none(late, n, k, tokens, workspace):
    """The caller's workspace (also with 9 to 16 tokens, which the stream-K kernel takes then), and the variant without a handle"""
    from lmdeploy_b200 import lib as l
    from perf import cases
    h = l.default_handle(0)
    sides = []
    for s in (1, 2):
        w = cases._linear(cases._gen(s, n), n, k)
        x = torch.randn(tokens, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(s)).half()
        sides.append((x, w.scales_and_zeros, w.kernel))
    live = [torch.empty_like(t) for t in sides[0]]
    room = l.lib.tm_gemm_s4_f16_workspace_bytes(n, tokens, k)
    ws = torch.zeros(room, dtype=torch.uint8, device="cuda")

    def call():
        out, s = torch.empty(tokens, n, dtype=torch.float16, device="cuda"), torch.cuda.current_stream().cuda_stream
        ops = (out.data_ptr(), live[2].data_ptr(), live[0].data_ptr(), live[1].data_ptr(), n, tokens, k, 128, 0)
        if workspace:
            l.check(l.lib.tm_gemm_s4_f16(h.ptr, *ops, ws.data_ptr(), room, s), "tm_gemm_s4_f16")
        else:
            l.check(l.lib.tm_gemm_s4_f16_noalloc(*ops, s), "tm_gemm_s4_f16_noalloc")
        return out
    _turns(late, call, live, sides)


@pytest.mark.parametrize("tokens,dtype", [(1, "bfloat16"), (64, "bfloat16"), (600, "bfloat16"), (5, "float32")])
def test_dense(late, tokens, dtype):
    from lmdeploy_b200 import lib as l
    n, k, h, td = 4096, 2048, l.default_handle(0), getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    sides = [tuple(torch.randn(*s, device="cuda", generator=g).to(td) for s in ((tokens, k), (n, k))) for _ in range(2)]
    live = [torch.empty_like(t) for t in sides[0]]

    def call():
        out = torch.empty(tokens, n, dtype=td, device="cuda")
        l.check(l.lib.tm_gemm_dense(h.ptr, out.data_ptr(), n, 0, live[0].data_ptr(), k, live[1].data_ptr(), k, tokens, n, k,
                                    int(dtype == "float32"), torch.cuda.current_stream().cuda_stream), "tm_gemm_dense")
        return out
    _turns(late, call, live, sides)


@pytest.mark.parametrize("tokens,dtype", [(4, "bfloat16"), (200, "bfloat16"), (4, "float32")])
def test_mixture_of_experts(late, tokens, dtype):
    from lmdeploy_b200 import lib as l
    experts, width, ff, h, td = 16, 256, 128, l.default_handle(0), getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    draw = lambda t, *s: torch.randn(*s, device="cuda", generator=g).to(t)  # noqa: E731
    sides = [(draw(td, tokens, width), draw(td, tokens, width), draw(torch.float32, tokens, experts), draw(torch.float32, tokens, width),
              draw(torch.float32, width), draw(torch.float32, experts), draw(torch.float32, width), draw(td, experts, width, ff) * ff ** -0.5,
              draw(td, experts, 2 * ff, width) * width ** -0.5) for _ in range(2)]
    live = [torch.empty_like(t) for t in sides[0]]
    p = l.TmMoeParams()
    p.tokens, p.width, p.ff, p.experts, p.identity, p.top, p.groups, p.keep = tokens, width, ff, experts, 0, 4, 1, 1
    p.limit, p.slope, p.mult, p.norm_eps, p.logits_ld, p.input_ld, p.gate_ld, p.dtype = 7.0, 1.702, 0.7, 1e-3, experts, width, width, int(dtype == "float32")
    p.input, p.gate, p.logits, p.x, p.gate_bias, p.correction, p.norm_weight, p.w_down, p.w_experts = (t.data_ptr() for t in live)

    def call():
        out = torch.empty(tokens, width, dtype=td, device="cuda")
        p.norm_out = out.data_ptr()
        l.check(l.lib.tm_moe(h.ptr, C.byref(p), torch.cuda.current_stream().cuda_stream), "tm_moe")
        return out
    _turns(late, call, live, sides)
