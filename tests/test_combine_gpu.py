"""The parts of a split forward merged in batches: numbers of parts at the edges of the batches and of the warp."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs", [2, 3, 4, 5, 8, 9, 12, 13, 16, 31, 32, 33, 37, 40])
@pytest.mark.parametrize("D", [32, 64, 128])
def test_runs(D, runs):
    import flash_b200 as fb
    B, H, Hk, M, N = 1, 8, 2, 3, 40 * 128 - 5
    g = torch.Generator(device="cuda").manual_seed(runs + D)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda").half() for h, n in ((H, M), (Hk, N), (Hk, N)))
    k[:, :, 1000:1400] *= 6  # maxima far apart between the runs
    o = fb.attention_in_runs(q, k, v, runs, True)
    s = q.double() @ k.double().repeat_interleave(H // Hk, 1).transpose(2, 3) / D ** 0.5
    s = s.masked_fill(torch.arange(N, device="cuda")[None] > torch.arange(M, device="cuda")[:, None] + N - M, -torch.inf)
    want = s.softmax(3) @ v.double().repeat_interleave(H // Hk, 1)
    # P and the result are rounded to 11 bits
    assert float((o.double() - want).norm()) <= 4 * 2.0 ** -11 * float(want.norm())
    if runs > 8:  # a score of +inf spoils its row, whichever part has it
        k2 = k.clone()
        k2[0, 0, 700], k2[0, 1, N - 9] = torch.inf, torch.inf
        q2 = q.abs()
        one, many = fb.attention_in_runs(q2, k2, v, 1, True), fb.attention_in_runs(q2, k2, v, runs, True)
        assert torch.equal(torch.isnan(one), torch.isnan(many)) and bool(torch.isnan(one).any())
    fb.check_status()
