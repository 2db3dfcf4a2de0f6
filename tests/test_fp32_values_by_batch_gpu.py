"""fp32 blocks of 16 and of 32 rows: a NaN or an infinity that the causal mask hides from 16 rows leaves them alone in both, and which rows it
reaches does not depend on what a sequence is batched with."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["k", "v", "q", "do"])
@pytest.mark.parametrize("gap", [0, 40])
@pytest.mark.parametrize("D", [16, 64, 128])
def test_same_rows_alone_and_in_a_batch(D, gap, where, value):
    import flash_b200 as fb
    B, H, M = 60, 4, 192  # 1440 blocks of 32 rows: more than any rule gives 16
    N = M + gap
    g = torch.Generator(device="cuda").manual_seed(gap + D)
    t = {n: torch.randn(B, H, l, D, generator=g, device="cuda") for n, l in (("q", M), ("k", N), ("v", N), ("do", M))}

    def step(b):
        x = [t[n][:b].clone().requires_grad_() for n in ("q", "k", "v")]
        o = fb.attention(*x, True)
        return o.detach(), *torch.autograd.grad(o, x, t["do"][:b])

    clean = step(B)
    rows = (3, 17, 84, 100, 175)  # both halves of blocks, of tiles of 64
    for h, i in zip((0, 1, 2, 3, 0), rows):
        t[where][::7, h, i + (gap if where in "kv" else 0)] = value
    many, one = step(B), step(1)
    fb.check_status()
    for a, b in zip(many, one):
        assert torch.equal(torch.isnan(a[:1]), torch.isnan(b)) and torch.equal(a[:1].nan_to_num(), b.nan_to_num())
    # head 1 holds one value only, at row 17 (key 17 + gap): the 16 rows (or keys) before, or behind, its block of 16 do not see it
    if where in "kv":
        assert all(torch.equal(many[x][:, 1, :16], clean[x][:, 1, :16]) for x in (0, 1))
        assert not bool(torch.isfinite(many[0][0, 1, 17:]).all(1).any()) or where == "k"
    else:
        first = (17 + gap) // 16 * 16 + 16
        assert all(torch.equal(many[x][:, 1, first:], clean[x][:, 1, first:]) for x in (2, 3))
    # sequences without such a value
    assert all(torch.equal(a[1:7], c[1:7]) for a, c in zip(many, clean))
