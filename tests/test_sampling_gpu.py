"""The choice of a token at the sizes where its kernel changes: rows shorter than a block's share, the edges of a warp's and a
block's stretch, the lengths where a thread keeps 8, 20 or no tokens in registers; and rows of ties, masks and infinities."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def outside(row, temperature, top_p, u, token):
    """How far the draw lies outside the token's stretch of the kept mass (in 64 bits), as a share of that mass."""
    e = torch.exp((row.double() - row.double().max()) / temperature)
    if top_p < 1.0:
        ranked = torch.sort(e, descending=True).values
        e[e < ranked[int((torch.cumsum(ranked, 0) >= top_p * e.sum()).nonzero()[0])]] = 0.0
    cdf = torch.cumsum(e, 0)
    goal = u * float(cdf[-1])
    return max(float(cdf[token] - e[token]) - goal, goal - float(cdf[token]), 0.0) / float(cdf[-1])


@pytest.mark.parametrize("V", [1, 2, 31, 257, 8191, 8193, 65536, 65537, 163840, 163841, 200003])
def test_every_length_of_a_row(V):
    from blackwellllm_b200.kernels import ops
    from blackwellllm_b200.sampling.params import uniform
    g = torch.Generator().manual_seed(V)
    temps, tops = [0.6, 1.0, 0.6, 2.0, 0.0], [0.9, 1.0, 0.5, 0.999, 0.9]
    logits = torch.randn(5, V + 3, generator=g) * 3
    us = [uniform(V, i) for i in range(5)]
    u = torch.tensor(us)
    rows = logits.to(DEV)[:, 1:V + 1]          # rows that begin off a 16-byte boundary, further apart than they are long
    got = ops.sample(rows, torch.tensor(temps).to(DEV), torch.tensor(tops).to(DEV), u.to(DEV)).tolist()
    for r in range(4):
        # a weight's float32 exponent is off by up to 2^-22 of (max - x) / T < 60, so its weight by 1.5e-5; the sums are exact:
        # a draw may fall beside its token's stretch of the kept mass by that much
        assert outside(logits[r, 1:V + 1], temps[r], tops[r], us[r], got[r]) <= 2e-5, (r, V)
    assert ops.sample(rows, None, None, None).tolist() == rows.argmax(dim=1).tolist()
    repeat = ops.sample(rows.repeat(9, 1), torch.tensor(temps * 9).to(DEV), torch.tensor(tops * 9).to(DEV), u.repeat(9).to(DEV))
    assert repeat.tolist() == got * 9                 # whatever else is in the batch


@pytest.mark.parametrize("V", [50, 30000, 170000])
def test_ties_masks_and_rows_without_a_weight(V):
    from blackwellllm_b200.kernels import ops
    inf = math.inf
    rows = torch.full((8, V), -inf)
    rows[0, V - 1] = 1.0                              # one token left by a mask
    rows[1, [3, V // 2, V - 2]] = 2.0                 # ties: the nucleus keeps all of them
    rows[2, [3, V // 2, V - 2]] = 2.0
    rows[3] = 0.0                                     # all alike
    rows[4, 7] = torch.finfo(torch.float32).min       # masks of the type's lowest value
    rows[4, 9] = 5.0
    rows[5, :] = torch.finfo(torch.float32).min
    rows[6] = 1.0
    rows[6, 5] = inf                                  # no weight is above 0: the last of the first tokens
    rows[7] = -inf                                    # no weight is a number
    t = torch.full((8,), 0.6)
    p = torch.full((8,), 0.4)
    u = torch.tensor([0.99, 0.0, 0.999, 0.5, 0.3, 0.25, 0.5, 0.5])
    got = ops.sample(rows.to(DEV), t.to(DEV), p.to(DEV), u.to(DEV)).tolist()
    first = -(-V // 1024)                             # a thousandth of the row
    assert got[:3] == [V - 1, 3, V - 2]
    assert got[3] == int(0.5 * V) and got[4] == 9 and got[5] == int(0.25 * V)
    assert got[6] == (first - 1 if first - 1 != 5 else 4) and got[7] == -1
    # top_p <= 0 keeps the most probable token; the smallest and the largest uniform number fall inside the row
    ramp = torch.arange(V, dtype=torch.float32).repeat(3, 1) / V
    got = ops.sample(ramp.to(DEV), torch.ones(3, device=DEV), torch.tensor([0.0, 1.0, 1.0], device=DEV),
                     torch.tensor([0.7, 0.0, 1.0], device=DEV)).tolist()
    assert got == [V - 1, 0, V - 1]
    # a token that is no number has no weight, and the nucleus is then the whole row
    rows = torch.zeros(2, V)
    rows[:, 4] = math.nan
    got = ops.sample(rows.to(DEV), torch.ones(2, device=DEV), torch.tensor([0.01, 1.0], device=DEV),
                     torch.tensor([0.9999, 0.9999], device=DEV)).tolist()
    assert all(abs(i - 0.9999 * V) <= 0.0001 * V + 2 for i in got)


# rows short enough for one block, and numbers of rows from which one block a row is the faster form, beside the same rows a few at a
# time on clusters: masses are whole numbers, so both forms choose the same tokens
@pytest.mark.parametrize("R,V", [(3, 31), (40, 300), (5, 8192), (5, 8193), (45, 16001), (70, 32000), (140, 60000), (260, 128256), (105, 170001)])
def test_rows_choose_the_same_token_in_every_form(R, V):
    from blackwellllm_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(R, V, device="cuda", generator=g) * 2
    x[0], x[1, V // 2:] = 1.0, float("-inf")
    x[2, V - 1] = 30.0
    u, one = torch.rand(R, device="cuda", generator=g), torch.ones(R, device="cuda")
    for args in ((None, None, None), (0.6 * one, None, u), (0.9 * one, 0.9 * one, u), (torch.where(u < 0.5, 0.0, 1.0), 0.3 * one, u)):
        whole = ops.sample(x, *args)
        for at in range(0, R, 9):
            assert torch.equal(ops.sample(x[at:at + 9], *(a[at:at + 9] if a is not None else None for a in args)), whole[at:at + 9])
    # greedy rows of masks and of no numbers alone, and the lowest index of a tie
    x[0], x[1], x[2] = float("-inf"), float("nan"), 3.0
    x[0, V - 1], x[2, V // 3], x[2, V // 2] = -1e30, 4.0, 4.0
    for part in (x, x[:3]):
        assert ops.sample(part, None, None, None)[:3].tolist() == [V - 1, 0, V // 3]


@pytest.mark.parametrize("R,V", [(3, 300), (3, 40000), (3, 152064), (20, 152064), (3, 170000)])
@pytest.mark.parametrize("spread", [0.05, 1.0, 3.0, 12.0])
def test_nuclei_of_one_token_to_most_of_the_row(R, V, spread):
    """Found among a few listed tokens, in one warp or in a block, or from the histograms of the whole row; parameters on the device
    and with the launch alike."""
    from blackwellllm_b200.kernels import ops
    g = torch.Generator().manual_seed(V + R)
    rows = (torch.randn(R, V, generator=g) * spread).to(DEV)
    values = torch.stack([torch.full((R,), 0.8), torch.full((R,), 0.95), torch.rand(R, generator=g)])
    got = ops.sample(rows, *values.numpy())
    assert torch.equal(got, ops.sample(rows, *values.to(DEV)))
    for r in range(min(R, 3)):
        assert outside(rows[r].cpu(), 0.8, 0.95, float(values[2, r]), int(got[r])) <= 2e-5      # (as above)
