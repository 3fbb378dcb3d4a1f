"""GPU: the norm kernels where a row's pieces per thread change, against 64-bit sums of the same halves."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 2048, 4088, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("m", [1, 3, 700])
def test_norms(n, m):
    from lmdeploy_b200 import lib as l
    g = torch.Generator(device="cuda").manual_seed(n + m)
    x, r = (torch.randn(m, n, device="cuda", generator=g).half() for _ in range(2))
    w = (1 + 0.1 * torch.randn(n, device="cuda", generator=g)).half()
    s, out = torch.cuda.current_stream().cuda_stream, torch.empty_like(x)
    norm = lambda v, base: v * torch.rsqrt((base * base).mean(1, keepdim=True) + 1e-6) * w.double()
    l.check(l.lib.tm_rmsnorm(out.data_ptr(), x.data_ptr(), w.data_ptr(), 1e-6, m, n, s), "norm")
    want = norm(x.double(), x.double())
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -10.5 + 2.0 ** -24).all()  # one rounding, and the fp32 factor's
    sums, added, res = r.double() + x.double(), (r.float() + x.float()).half(), r.clone()
    l.check(l.lib.tm_add_residual_rmsnorm(res.data_ptr(), x.data_ptr(), None, w.data_ptr(), 1e-6, m, n, s), "add and norm")
    assert torch.equal(res, added)
    want = norm(res.double(), sums)
    assert ((x.double() - want).abs() <= want.abs() * 2.0 ** -10.5 + 2.0 ** -24).all()
