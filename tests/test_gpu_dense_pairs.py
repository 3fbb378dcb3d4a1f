"""The bf16 dense product where pairs of CTAs take its tiles, with the epilogues of the config-driven decoders, against 64-bit
sums of the same operands.  Every size is one that the plan gives to pairs, and the test says so."""
import ctypes as C
import os
import shutil
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
ULP = 2.0 ** -24
GUARD = 7.0


@pytest.fixture(scope="module")
def dense(tmp_path_factory):
    from lmdeploy_b200 import build
    so = str(tmp_path_factory.mktemp("dense") / "libdense.so")
    flags = [f for f in build.NVCC_FLAGS if f not in ("-lineinfo",)]
    r = subprocess.run([NVCC] + flags + ["-Xcompiler", "-fvisibility=default", "-w", "-shared", os.path.join(ROOT, "tests", "native", "dense_epilogues.cu"),
                                         "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    lib = C.CDLL(so)
    lib.call_new.restype = C.c_void_p
    h = C.c_void_p()
    assert lib.tm_create(C.byref(h), 0) == 0
    yield lib, h
    lib.tm_destroy(h)


def _p(t):
    return C.c_void_p(0 if t is None else t.data_ptr())


class _Product:
    """x [tokens, k] (and x2 from column x2_from on) times w [n, k], its exact value and the bound of fp32 sums of it"""

    def __init__(self, dense, tokens, n, k, x2_from=0):
        self.lib, self.h = dense
        g = torch.Generator(device="cuda").manual_seed(tokens + n + k)
        draw = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
        self.draw, self.tokens, self.n = draw, tokens, n
        self.x, self.w = draw(tokens, k).bfloat16(), (draw(n, k) / k ** 0.5).bfloat16()
        self.x2 = draw(tokens, k).bfloat16() if x2_from else None
        wd = self.w.double()
        self.y, size = self.x.double() @ wd.T, self.x.double().abs() @ wd.abs().T
        if x2_from:
            self.y[:, x2_from:] = self.x2.double() @ wd[x2_from:].T
            size[:, x2_from:] = self.x2.double().abs() @ wd[x2_from:].abs().T
        self.err = size * (k * ULP)
        self.c = C.c_void_p(self.lib.call_new())
        self.lib.set_operands(self.c, _p(self.x), _p(self.x2), x2_from, k, _p(self.w), k, tokens, n, k)

    def run(self, route=3):
        assert self.lib.route(self.c, self.lib.sm_count(self.h)) == route, "the plan gives this size to pairs no more: choose another"
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert self.lib.run(self.h, self.c, st) == 0
        word = C.c_uint(0)
        assert self.lib.tm_check_device_status(self.h, st, C.byref(word)) == 0, hex(word.value)
        self.lib.call_free(self.c)


def _within(got, want, bound, what):
    over = ((got.double() - want).abs() / (bound + 1e-30)).max().item()
    assert over <= 1.0, f"{what}: {over:.2f} of the bound"


# columns: 19, 17 and 39 tiles (the last one of 72 columns), 40 tiles (the last one of 8); tokens of one tile, of several, ragged ones
@pytest.mark.parametrize("tokens,n,k", [(160, 2432, 4864), (600, 2176, 512), (257, 4936, 1000), (300, 5000, 512)])
@pytest.mark.parametrize("gated", [False, True])
def test_residual_and_row_sums(dense, tokens, n, k, gated):
    """Residual, its cast and its sums of squares per tile of columns; nothing is written behind the last tile's sums (a pair's
    second CTA has no tile where their number is odd)."""
    q = _Product(dense, tokens, n, k)
    before = q.draw(tokens, n)
    tiles, stride = -(-n // 128), (tokens + 7) // 8 * 8
    residual, cast = before.clone(), torch.full((tokens, n + 8), GUARD, device="cuda", dtype=torch.bfloat16)
    sums = torch.full((tiles + 2, stride), GUARD, device="cuda")
    gate = q.draw(tokens, n).bfloat16() if gated else None
    bias = q.draw(n) if gated else None
    mult = 0.5 if gated else 1.0
    q.lib.set_residual(q.c, _p(residual), n, _p(cast), n + 8, _p(sums), stride, _p(gate), n, _p(bias), C.c_float(mult))
    q.run()
    y, err = q.y, q.err
    if gated:
        a = gate.double() + bias.double()
        f = mult * torch.sigmoid(a)
        # __expf: 2 + 1.2 |a| ulps; the sum, the quotient and its product a few more
        err, y = f * err + (f * y).abs() * ((8 + 1.2 * a.abs()) * 2 * ULP), f * y
    want = before.double() + y
    err = err + want.abs() * ULP
    _within(residual, want, err, "residual")
    _within(cast[:, :n], want, err + want.abs() * 2.0 ** -8, "cast")
    assert bool((cast[:, n:] == GUARD).all())
    pad = lambda v: torch.nn.functional.pad(v, (0, tiles * 128 - n)).view(tokens, tiles, 128).sum(-1).T  # noqa: E731
    _within(sums[:tiles, :tokens], pad(want ** 2), pad(2 * want.abs() * err + err ** 2) + pad(want ** 2) * (32 * ULP), "sums of squares")
    assert bool((sums[tiles:] == GUARD).all()), "written behind the last tile's sums"
    assert bool((sums[:tiles, tokens:] == GUARD).all())


def _input(q, split, tanh, f32_from=0):
    """kInput: columns below `split` (some through tanh, some in fp32), gated ones behind; checks all of them"""
    n, tokens = q.n, q.tokens
    out, act = (torch.full((tokens, w + 8), GUARD, device="cuda", dtype=torch.bfloat16) for w in (split, (n - split) // 2))
    q.lib.set_input(q.c, _p(out), split + 8, tanh[0], tanh[1], split, _p(act), act.shape[1])
    f32 = torch.full((tokens, split - f32_from + 3), GUARD, device="cuda")
    if f32_from:
        q.lib.set_f32_columns(q.c, _p(f32), f32_from, f32.shape[1])

    def check():
        y, err = q.y, q.err
        want = y[:, :split].clone()
        want[:, tanh[0]:tanh[1]] = torch.tanh(want[:, tanh[0]:tanh[1]])
        stored = f32_from or split
        # |tanh'| <= 1, tanhf is within two ulps
        _within(out[:, :stored], want[:, :stored], err[:, :stored] + want[:, :stored].abs() * (2.0 ** -8 + 4 * ULP), "stored columns")
        assert bool((out[:, stored:] == GUARD).all())
        if f32_from:
            _within(f32[:, :split - f32_from], y[:, f32_from:split], err[:, f32_from:split] + y[:, f32_from:split].abs() * ULP, "fp32 columns")
            assert bool((f32[:, split - f32_from:] == GUARD).all())
        gate, up, eg, eu = y[:, split::2], y[:, split + 1::2], err[:, split::2], err[:, split + 1::2]
        gelu = torch.nn.functional.gelu(gate, approximate="tanh")
        # |gelu'| <= 1.13; __expf's argument u is off by a few ulps and it by 2 + 1.2 |u| more: |gelu| (8 + 4 |u|) ulps
        u = 1.5957691216057308 * (gate + 0.044715 * gate ** 3)
        bound = 1.13 * eg * up.abs() + gelu.abs() * eu + 1.13 * eg * eu + (gelu * up).abs() * (2.0 ** -8 + (8 + 4 * u.abs()) * 2 * ULP)
        _within(act[:, :(n - split) // 2], gelu * up, bound + 1e-30, "gated columns")
        assert bool((act[:, (n - split) // 2:] == GUARD).all())
    return check


@pytest.mark.parametrize("tokens,n,split,tanh,f32_from,route", [(200, 9216, 1024, (100, 300), 500, 3), (40, 1024, 512, (70, 400), 300, 2)])
def test_fp32_columns_that_begin_inside_a_warps(dense, tokens, n, split, tanh, f32_from, route):
    q = _Product(dense, tokens, n, 4096)
    check = _input(q, split, tanh, f32_from)
    q.run(route)
    check()


# 79 tiles with the gated columns ending inside the last one, a tile's k that ends inside a block, ragged tokens
@pytest.mark.parametrize("tokens,n,k,split,tanh", [(300, 9344, 4096, 5120, (1000, 1100)), (257, 10056, 1000, 256, (0, 0)), (129, 9216, 512, 9088, (0, 9088))])
def test_input_projection(dense, tokens, n, k, split, tanh):
    """Columns through tanh, gated columns, and rows that are scaled by their norm (sums of squares in several parts)."""
    q = _Product(dense, tokens, n, k)
    parts, stride = 3, tokens + 5
    ssq, gain = q.draw(parts, stride).abs() * k / parts, q.draw(1).abs() + 0.5
    q.lib.set_scale(q.c, _p(ssq), parts, stride, C.c_float(1.0 / k), C.c_float(1e-5), _p(gain))
    s = gain.double() / torch.sqrt(ssq.double()[:, :tokens].sum(0) / k + 1e-5)
    q.y *= s[:, None]
    q.err = q.err * s[:, None] + q.y.abs() * (8 * ULP)  # sums, quotient and root in fp32
    check = _input(q, split, tanh)
    q.run()
    check()


@pytest.mark.parametrize("tokens,n,k,x2_from,f32_from", [(300, 9377, 1024, 5120, 9344), (600, 2210, 512, 1024, 2177)])
@pytest.mark.parametrize("ld", [0, 3])
def test_second_operand_and_fp32_columns(dense, tokens, n, k, x2_from, f32_from, ld):
    """Columns that multiply a second operand, the last of them in fp32; rows that 16-byte stores reach, and not."""
    q = _Product(dense, tokens, n, k, x2_from)
    width = (f32_from + 7) // 8 * 8 + ld
    out, f32 = torch.full((tokens, width), GUARD, device="cuda", dtype=torch.bfloat16), torch.full((tokens, n - f32_from + 1), GUARD, device="cuda")
    q.lib.set_store(q.c, _p(out), width)
    q.lib.set_f32_columns(q.c, _p(f32), f32_from, f32.shape[1])
    q.run()
    _within(out[:, :f32_from], q.y[:, :f32_from], q.err[:, :f32_from] + q.y[:, :f32_from].abs() * 2.0 ** -8, "stored columns")
    assert bool((out[:, f32_from:] == GUARD).all())
    _within(f32[:, :-1], q.y[:, f32_from:], q.err[:, f32_from:] + q.y[:, f32_from:].abs() * ULP, "fp32 columns")
    assert bool((f32[:, -1] == GUARD).all())


# one tile of columns and a last one of 8, tokens of several bands of tiles and a last tile of one token
@pytest.mark.parametrize("tokens,n,k,ld", [(257, 5000, 512, 5000), (2049, 5000, 1000, 5003), (513, 9608, 4096, 9608), (97, 9600, 584, 9600)])
def test_stored_rows(dense, tokens, n, k, ld):
    q = _Product(dense, tokens, n, k)
    out = torch.full((tokens + 1, ld), GUARD, device="cuda", dtype=torch.bfloat16)
    q.lib.set_store(q.c, _p(out), ld)
    q.run()
    _within(out[:tokens, :n], q.y, q.err + q.y.abs() * 2.0 ** -8, "rows")
    assert bool((out[:, n:] == GUARD).all()) and bool((out[tokens] == GUARD).all())
