"""Sampled tokens into the next step's inputs and the history."""
import pytest
import torch

from gpu_util import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,keep_lp", [(1, True), (128, True), (129, False), (300, True)])
def test_feed_back(rows, keep_lp):
    C, S, cap = native(), 320, 7
    g = torch.Generator(device="cuda").manual_seed(rows)
    new = lambda hi, *s: torch.randint(0, hi, s, device="cuda", dtype=torch.int32, generator=g)
    tokens, last, history = new(1000, S), new(1000, S), new(1000, S, cap)
    index = new(cap + 3, S).long()  # also behind the last position
    lp, hist_lp = torch.randn(S, device="cuda", generator=g), torch.randn(S, cap, device="cuda", generator=g)
    want = [t.clone() for t in (last, index, history, hist_lp)]
    for r in range(rows):
        at = min(int(index[r]), cap - 1)
        want[0][r] = want[2][r, at] = tokens[r]
        if keep_lp:
            want[3][r, at] = lp[r]
        want[1][r] += 1
    C.feed_back(tokens, lp if keep_lp else None, rows, last, index, history, hist_lp if keep_lp else None)
    assert all(torch.equal(a, b) for a, b in zip((last, index, history, hist_lp), want))
