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
