"""A NaN or an infinity in a key that the ids hide from a row does not reach the row's result, however the forward works the mask out: blocks of
one document, of a few (in order or scattered), and of many, with and without the causal bound."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def documents(kind, L, g):
    if kind == "one a block":
        return torch.arange(L, device="cuda") // 128 % 3
    if kind == "in order":
        return torch.arange(L, device="cuda") // 37
    return torch.randint(0, {"a few": 3, "many": 90}[kind], (L,), generator=g, device="cuda")


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("kind", ["one a block", "in order", "a few", "many"])
@pytest.mark.parametrize("D", [32, 64, 128])
def test_key_behind_the_ids(D, kind, causal, value, monkeypatch):
    import flash_b200 as fb
    from flash_b200 import ops
    monkeypatch.setattr(ops, "GROUP_QUERIES", False)
    B, H, L = 2, 2, 600
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(B, H, L, D, generator=g, device="cuda").bfloat16() for _ in range(3))
    docs = documents(kind, L, g)
    ids = -1 - docs
    ids[::50] = 5  # rows that attend everywhere; as keys they are in nobody's document
    eq = ids.expand(B, H, L)
    clean = fb.attention(q, k, v, causal, None, eq, eq, 1)
    i = torch.arange(L, device="cuda")
    for j in (3, 130, 301, 599):
        bad = k.clone()
        bad[:, :, j] = value
        o = fb.attention(q, bad, v, causal, None, eq, eq, 1)
        sees = (ids >= 0) | (ids == ids[j])
        if causal:
            sees = sees & (i >= j)
        assert bool(sees.any()) and bool((~sees).any())
        assert torch.equal(o[:, :, ~sees], clean[:, :, ~sees])
        # a score of NaN gives zeros, one of +inf NaN; one of -inf leaves the key out
        assert value != value or not bool((o[:, :, sees] == clean[:, :, sees]).all())
        assert value == value or bool((o[:, :, sees] == 0).all())
    fb.check_status()
