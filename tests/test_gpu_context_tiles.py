"""GPU: the context attention where its key tiles begin and end (one tile, two, three, a last one with one key), fp16 and int8 cache,
against 64-bit softmax over the same values."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("new,history", [([1], [0]), ([63, 64], [0, 0]), ([65, 128], [0, 1]), ([129, 1], [63, 64]), ([200, 7], [0, 190])])
def test_tiles(int8, new, history):
    from lmdeploy_b200 import lib as l
    H, G, B, S = 4, 2, len(new), 400
    g = torch.Generator(device="cuda").manual_seed(sum(new) + sum(history))
    scale, longest, T = 4.0 / 127, max(new), sum(new)
    rows = [torch.randn(B, G, S, 128, device="cuda", generator=g) for _ in range(2)]
    cache = [(r / scale).round().clamp(-128, 127).to(torch.int8) if int8 else r.half() for r in rows]
    q = torch.randn(B, H, longest, 128, device="cuda", generator=g).half()
    out = torch.full((T + 1, H * 128), 777.0, dtype=torch.float16, device="cuda")
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    ptrs = [torch.tensor([c[b].data_ptr() for b in range(B)], dtype=torch.int64, device="cuda") for c in cache]
    cu, ctx = ints([sum(new[:b]) for b in range(B + 1)]), ints([n + h for n, h in zip(new, history)])
    a = l.TmContextAttentionParams()
    a.attn_out, a.query, a.key_cache, a.val_cache = out.data_ptr(), q.data_ptr(), ptrs[0].data_ptr(), ptrs[1].data_ptr()
    a.cu_seqlens, a.context_lengths, a.cache_layer_offset = cu.data_ptr(), ctx.data_ptr(), 0
    a.batch_size, a.head_num, a.kv_head_num, a.size_per_head = B, H, G, 128
    a.max_q_len, a.max_seq_len, a.quant_policy, a.kv_scale = longest, S, 4 if int8 else 0, (C.c_float * 4)(scale, 0.0, scale, 0.0)
    l.check(l.lib.tm_context_attention(C.byref(a), torch.cuda.current_stream().cuda_stream), "tm_context_attention")
    k, v = ((c.float() * scale).half().double() if int8 else c.double() for c in cache)
    for b in range(B):
        n, h = new[b], history[b]
        kb, vb = (x[b, :, :h + n].repeat_interleave(H // G, 0) for x in (k, v))
        s = q[b, :, :n].double() @ kb.transpose(1, 2) * 128 ** -0.5
        s.masked_fill_(torch.arange(h + n, device="cuda")[None, :] > torch.arange(h, h + n, device="cuda")[:, None], float("-inf"))
        want = (torch.softmax(s, -1) @ vb).transpose(0, 1).reshape(n, -1)
        got = out[sum(new[:b]):sum(new[:b]) + n].double()
        # probabilities and outputs are rounded to fp16 (2^-11 each, the first over values of size 4)
        assert ((got - want).abs() <= want.abs() * 2.0 ** -10 + 4 * 2.0 ** -11).all()
        assert ((got - want).norm() / want.norm()).item() <= 2.0 ** -10
    assert bool((out[T] == 777.0).all())
