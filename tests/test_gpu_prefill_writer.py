"""GPU: the prefill driver writes keys and values straight to their cache rows; the same bits as the two public writers leave there one
after the other, for ragged batches behind cached tokens, and nothing outside the new rows.  From 2048 tokens on a CTA takes four of
them: the same bits again."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("int8", [True, False])
@pytest.mark.parametrize("new,history", [([1], [0]), ([7, 0, 33], [5, 9, 0]), ([16, 17, 1, 24], [40, 0, 63, 8]),
                                         ([700, 811, 1, 538], [9, 0, 899, 100]), ([900, 900, 247, 1], [0, 0, 1, 3])])
def test_rows_match_the_public_writers(int8, new, history, monkeypatch):
    from lmdeploy_b200 import lib as l, turbomind as tm
    from tests.test_gpu_llama import CFG, build
    monkeypatch.setitem(CFG, "session_len", 64 if sum(new) < 2047 else 960)
    model, _, _ = build(int8, max_batch=4)
    B, S, H, G, hid = len(new), CFG["session_len"], CFG["head_num"], CFG["kv_head_num"], CFG["head_num"] * 128
    rng, dev = np.random.default_rng(sum(new)), "cuda"
    tokens = [rng.integers(0, CFG["vocab_size"], n).tolist() for n in new]
    st = model.new_state(B, 1)
    for c in (st.k_cache, st.v_cache):
        c.copy_(torch.randint(-100, 100, c.shape, device=dev).to(c.dtype))
    before = [c.clone() for c in (st.k_cache, st.v_cache)]
    st.lengths.copy_(torch.tensor(history, dtype=torch.int32, device=dev))
    model.prefill(st, tokens)
    model.check_status(torch.cuda.current_stream().cuda_stream)
    # layer 0 by hand
    (attn, _, qkv, *_), T, longest = model._layers[0], sum(new), max(new)
    x = model._globals[0][torch.tensor([i for t in tokens for i in t], device=dev)]
    h, y = torch.empty_like(x), torch.empty(T, (H + 2 * G) * 128, dtype=torch.float16, device=dev)
    s = torch.cuda.current_stream().cuda_stream
    l.check(l.lib.tm_rmsnorm(h.data_ptr(), x.data_ptr(), attn.data_ptr(), CFG["norm_eps"], T, hid, s), "norm")
    tm.LlamaLinear(0).forward(y, h, T, qkv, tm.LlamaLinear.kGemm)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    pad = ints([b * longest - sum(new[:b]) for b in range(B) for _ in range(new[b])])
    q = torch.empty(B, H, longest, 128, dtype=torch.float16, device=dev)
    k, v = (torch.empty(B, G, longest, 128, dtype=torch.float16, device=dev) for _ in range(2))
    length, hist = ints(new), ints(history)
    l.check(l.lib.tm_add_fused_qkv_bias_transpose(q.data_ptr(), k.data_ptr(), v.data_ptr(), y.data_ptr(), None, pad.data_ptr(), hist.data_ptr(),
                                                  length.data_ptr(), B, longest, T, H, G, 128, 128, CFG["rope_theta"], S, 0, 0, s), "qkv")
    ptrs = [torch.tensor([c[b].data_ptr() for b in range(B)], dtype=torch.int64, device=dev) for c in before]
    scale = (l.C.c_float * 4)(*model._layers[0][-1])
    l.check(l.lib.tm_extend_kv_cache(ptrs[0].data_ptr(), ptrs[1].data_ptr(), 0, k.data_ptr(), v.data_ptr(), B, length.data_ptr(), longest,
                                     hist.data_ptr(), S, 128, G, s, 4 if int8 else 0, scale), "extend")
    for got, want in zip((st.k_cache, st.v_cache), before):
        assert torch.equal(got[:, 0], want[:, 0])
        for b in range(B):  # the other layers: new rows only
            rows = torch.ones(S, dtype=torch.bool, device=dev)
            rows[history[b]:history[b] + new[b]] = False
            assert torch.equal(got[b, 1:, :, rows], want[b, 1:, :, rows])
    model.close()


@pytest.mark.parametrize("heads,kv_heads", [(5, 1), (8, 8)])
@pytest.mark.parametrize("lengths,history", [([1024, 1024], [7, 0]), ([1021, 0, 3, 1025], [0, 5, 900, 31]), ([1300, 750, 1], [3000, 0, 64])])
@pytest.mark.parametrize("bias,rot,ntk,logn", [(True, 128, 0, 0), (False, 64, 1, 1)])
def test_four_tokens_a_block(heads, kv_heads, lengths, history, bias, rot, ntk, logn):
    """One call for all sequences against one call for each, which are too short for it; rows behind a sequence's end stay."""
    from lmdeploy_b200 import lib as l
    S, T, n, dev = max(lengths), sum(lengths), (heads + 2 * kv_heads) * 128, "cuda"
    g = torch.Generator(device=dev).manual_seed(T + heads)
    y = torch.randn(T, n, device=dev, generator=g).half()
    b = torch.randn(n, device=dev, generator=g).half() if bias else None
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    s = torch.cuda.current_stream().cuda_stream

    def write(out, rows, lens, hist):
        pad = ints([i * S - sum(lens[:i]) for i, k in enumerate(lens) for _ in range(k)])
        le, hi = ints(lens), ints(hist)
        l.check(l.lib.tm_add_fused_qkv_bias_transpose(*(o.data_ptr() for o in out), rows.data_ptr(), b.data_ptr() if bias else None, pad.data_ptr(),
                                                      hi.data_ptr(), le.data_ptr(), len(lens), S, rows.shape[0], heads, kv_heads, 128, rot, 10000.0,
                                                      1024, ntk, logn, s), "qkv")
        torch.cuda.synchronize()

    new = lambda: [torch.full((len(lengths), h, S, 128), 7.0, dtype=torch.float16, device=dev) for h in (heads, kv_heads, kv_heads)]
    got, want = new(), new()
    write(got, y, lengths, history)
    at = 0
    for i, k in enumerate(lengths):
        if k:
            write([o[i:i + 1] for o in want], y[at:at + k], [k], [history[i]])
        at += k
    for a, c in zip(got, want):
        assert torch.equal(a, c)
