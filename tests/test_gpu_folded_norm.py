"""GPU: the decode step with residual add and RMSNorm folded into the GEMMs on either side, at the projections' real sizes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _hidden(s, fold, repeats):
    """The normed hidden rows of one step from an empty cache, `repeats` times over, and the step's launches.  A captured step if folded."""
    out, batch = [], s.case["batch"]
    s.model.handle.set_option("fold_norm", fold)
    forced = np.array([[t[0] for t in s.tokens]], np.int32)
    with torch.cuda.stream(s.stream):
        st = s.model.new_state(batch, 1, forced_ids=forced, keep_hidden=True)
        for _ in range(repeats):
            st.lengths.zero_()
            st.step.zero_()
            s.model.decode(st, 1, use_graph=bool(fold), stream=s.stream.cuda_stream)
            out.append(st.hidden.clone())
        s.model.check_status(s.stream.cuda_stream)
    s.stream.synchronize()
    return out, s.model.last_launches()


# The tensor-core kernel's producers, among them those whose last unit lies in the first stage of the activation ring: 8192 x 28672 with up
# to 64 tokens, 4096 x 4096 and 4096 x 11008 with more.
@pytest.mark.parametrize("size,batch", [("70b", 17), ("70b", 21), ("70b", 64), ("7b", 65), ("7b", 128)])
def test_every_element_as_with_norm_kernels(size, batch):
    from perf import cases
    s = cases._Llama(dict(kind="decode", size=size, layers=2, batch=batch, shortest=8, longest=8, int8=False), batch)
    (want,), separate = _hidden(s, 0, 1)
    got, launches = _hidden(s, 1, 40)
    s.model.close()
    assert separate - launches == 3
    for g in got[1:]:
        assert torch.equal(g, got[0])
    # Rows of rms 1.  The fold moves the rounding of the normed rows (2^-11 of a value) in front of four products, each a sum of thousands
    # of such errors, and of what is rounded behind them: 2^-10.4 on average, eight times that for the largest of a million.  An
    # activation that a product takes for zero in 64 of its inputs costs an output 4 % of its size.
    err, size_of = (got[0].double() - want.double()).abs(), want.double().abs()
    assert (err <= 2.0 ** -7 + size_of * 2.0 ** -8).all() and err.mean() <= 2.0 ** -10, (err.max().item(), err.mean().item())


def _scaled(gen, n, k, factor, columns=slice(None)):
    """A weight whose chosen columns are `factor` times as large, in the library's layout and as numbers"""
    from perf import cases
    state = gen.get_state()
    w = cases._linear(gen, n, k)
    gen.set_state(state)
    q, z, s = cases._weight(gen, n, k)
    s = s.clone()
    s[:, columns] = (s[:, columns].float() * factor).half()
    sz = w.scales_and_zeros
    sz[:, columns, 1] = (sz[:, columns, 1].float() * factor).half()
    assert torch.equal(sz[..., 1], s)
    return w, ((q.view(-1, 128, n).half() - z[:, None].half()) * s[:, None]).view(k, n).double()


class _Rows:
    """Two layers of the 7B shape over one token per sequence and an empty cache (attention passes the values through), with a residual
    stream of a given rms from the embedding on; the normed hidden rows in 64 bits."""

    def __init__(self, batch, rms, seed, weight=1.0, jump=1.0):
        from lmdeploy_b200 import llama
        cfg = llama.LLAMA2_7B
        hid, inter, layers, vocab = cfg.hidden, cfg.inter_size, 2, 1000
        self.model = llama.LlamaModel(llama.LlamaConfig(cfg.head_num, cfg.kv_head_num, inter, layers, vocab, quant_policy=0), batch, 8, 0)
        g = torch.Generator(device="cuda").manual_seed(seed)
        draw = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
        emb, head = (draw(vocab, hid) * rms).half(), (draw(vocab, hid) * 0.02).half()
        norms = [((1 + 0.1 * draw(hid)) * weight).half() for _ in range(2 * layers)] + [(1 + 0.1 * draw(hid)).half()]
        values, halves = slice(2 * hid, 3 * hid), slice(1, None, 2)  # the value columns; the up columns of (gate, up) pairs
        norm = lambda v, w: v / torch.sqrt((v * v).mean(-1, keepdim=True) + cfg.norm_eps) * w.double()  # noqa: E731
        self.ids, self.stream, self.batch = torch.randint(0, vocab, (batch,), generator=g, device="cuda"), torch.cuda.Stream(), batch
        x = emb[self.ids].double()
        self.keep = []
        for i in range(layers):
            # what a half layer adds is as large as the rows, behind the first feed forward `jump` times as large
            size = rms * jump if i else rms
            per, per_ffn = (size / (1.6 * weight)) ** 0.5, (rms * jump / 1.6) ** 0.5 / weight
            (wq, eq), (wo, eo) = _scaled(g, 3 * hid, hid, per, values), _scaled(g, hid, hid, per)
            (wu, eu), (wd, ed) = _scaled(g, 2 * inter, hid, per_ffn, halves), _scaled(g, hid, inter, per_ffn)
            self.model.set_layer(i, norms[2 * i], norms[2 * i + 1], wq, wo, wu, wd)
            self.keep += [wq, wo, wu, wd]
            x = x + (norm(x, norms[2 * i]) @ eq)[:, values] @ eo
            y = norm(x, norms[2 * i + 1]) @ eu
            x = x + (torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]) @ ed
        self.model.set_globals(emb, norms[-1], head)
        self.keep += [emb, head] + norms
        self.want = norm(x, norms[-1])

    def hidden(self, fold):
        self.model.handle.set_option("fold_norm", fold)
        forced = self.ids.cpu().numpy()[None].astype(np.int32)
        with torch.cuda.stream(self.stream):
            st = self.model.new_state(self.batch, 1, forced_ids=forced, keep_hidden=True)
            self.model.decode(st, 1, use_graph=False, stream=self.stream.cuda_stream)
            self.model.check_status(self.stream.cuda_stream)
        self.stream.synchronize()
        return st.hidden.clone()

    def error(self, fold):
        """The largest error of a row, relative to it"""
        return ((self.hidden(fold).double() - self.want).norm(dim=1) / self.want.norm(dim=1)).max().item()


@pytest.mark.parametrize("rms", [5e-4, 2e-3, 0.02, 1.0, 50.0])
@pytest.mark.parametrize("batch", [1, 8, 24])
def test_rows_of_any_size(batch, rms):
    """Against 64 bits, no further off than with norm kernels of their own (the roundings are as many, in other places)."""
    s = _Rows(batch, rms, batch)
    folded, separate = s.error(1), s.error(0)
    s.model.close()
    assert separate < 0.01 and folded <= 1.1 * separate + 2.0 ** -14, (folded, separate)


@pytest.mark.parametrize("rms,weight,jump", [(600.0, 30.0, 1.0), (1500.0, 16.0, 1.0), (0.02, 1e-3, 1.0), (0.02, 1.0, 500.0), (1.0, 0.05, 200.0)])
@pytest.mark.parametrize("batch", [1, 8, 24])
def test_rows_and_weights_whose_product_leaves_the_range(batch, rms, weight, jump):
    """A residual times a norm weight beyond 65504 or among subnormal numbers, and rows that grow by orders of magnitude at once."""
    s = _Rows(batch, rms, batch, weight, jump)
    folded, separate = s.error(1), s.error(0)
    s.model.close()
    assert separate < 0.01 and folded <= 1.1 * separate + 2.0 ** -14, (folded, separate)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("batch", [2, 20])
def test_a_row_that_is_not_finite_stays_alone(batch, value):
    """An embedding with such a value makes its own row NaN and leaves the others' bits as they were."""
    s = _Rows(batch, 1.0, batch)
    emb = s.keep[-7]
    assert emb.shape == (1000, 4096)
    clean = s.hidden(1)
    bad = s.ids == s.ids[0]
    emb[s.ids[0], 5] = value
    torch.cuda.synchronize()
    spoilt, separate = s.hidden(1), s.hidden(0)
    s.model.close()
    assert spoilt[bad].isnan().all() and separate[bad].isnan().all()
    assert torch.equal(spoilt[~bad], clean[~bad])
