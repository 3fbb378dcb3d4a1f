"""Decode step of the window attention over the numbers of splits that the launch rule picks (one, a few, remainders of the
merge's batches of eight), rings that wrap inside and between blocks of sixteen keys, against 64-bit attention."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 3, 7, 16, 37])
@pytest.mark.parametrize("history,window,pool", [(1, 1024, 0), (15, 1024, 16), (129, 2048, 16), (1001, 1024, 0), (2047, 2048, 16), (2063, 2048, 16), (6001, 1024, 16)])
def test_splits(batch, history, window, pool):
    from perf import cases
    case = dict(kind="window", batch=batch, history=history, window=window, pool=pool, softcap=0.0 if batch % 2 else 30.0)
    state = cases.prepare(case, 3)
    got = cases.run(state).double()
    state["handle"].check_device_status(torch.cuda.current_stream().cuda_stream)
    want = cases._exact_window(case, 3)
    # weights and outputs are rounded to bf16 (2^-9 each); means of N(0, 1) values: the error is relative to the largest value
    # of a row, 2^-9 (weights, worst case all to one side) + 2^-9, and 2^-8 of a score of at most 8 in the exponent
    bound = want.abs() * 2.0 ** -8 + want.abs().amax(1, keepdim=True) * 2.0 ** -5
    over = ((got - want).abs() / bound).max().item()
    assert over <= 1.0, f"{over:.2f} of the bound"
