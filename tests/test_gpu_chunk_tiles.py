"""GPU: prefill of the chunk attention where its key tiles begin and end (one tile, two, a last one that is nearly empty, chunks that
begin inside a tile), against 64-bit sums of the same values; and what a bad key may reach."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(case, seed, spoil=None):
    from perf import cases
    state = cases.prepare(case, seed)
    if spoil is not None:
        state["keep"][0][spoil, cases.HEADS * cases.D:(cases.HEADS + cases.KV_HEADS) * cases.D] = float("nan")
    out = cases.run(state)["out"].float()
    state["handle"].check_device_status(torch.cuda.current_stream().cuda_stream)
    return out


@pytest.mark.parametrize("tokens", [1, 63, 64, 65, 128, 129, 193, 257, 600])
@pytest.mark.parametrize("batch,chunk", [(1, 512), (2, 100), (1, 64)])
def test_tiles(tokens, batch, chunk):
    from perf import cases
    case = dict(kind="chunk", batch=batch, tokens=tokens, chunk=chunk)
    out, want = _run(case, tokens), cases.exact(case, tokens)["out"]
    # mixed weights and outputs are rounded to bf16 (2^-9 each), weights to fp16 (2^-12) and mixed with a half matrix (2^-12)
    assert ((out.double() - want).norm() / want.norm()).item() <= 2.0 ** -9 * 2


@pytest.mark.parametrize("spoil", [1, 64, 150])
def test_a_key_that_is_not_a_number_reaches_later_queries_of_its_chunk_only(spoil):
    case = dict(kind="chunk", batch=1, tokens=300, chunk=130)
    out, clean = _run(case, 4, spoil), _run(case, 4)
    end = (spoil // 130 + 1) * 130
    assert torch.equal(out[:spoil], clean[:spoil]) and torch.equal(out[end:], clean[end:])
    assert bool(out[spoil:end].isnan().all())
