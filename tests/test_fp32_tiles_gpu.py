"""fp32 kernels at the edges of their 32-row CTAs and 64-column tiles, every head dim, with ids that leave whole tiles
unvisited, against plain attention in 64 bits (1e-4, the fp32 tests' bound)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "odd base"])
@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("M,N,causal,mode,per_head", [
    (1, 63, True, 0, False), (31, 64, True, 0, False), (33, 65, True, 1, False), (64, 64, False, 1, True),
    (127, 129, True, 1, True), (130, 700, True, 1, False), (513, 513, True, 1, True), (200, 77, False, 0, False)])
def test_tile_edges(M, N, causal, mode, per_head, D, offset):
    import flash_b200 as fb
    B, H, Hk = 2, 4, 2
    g = torch.Generator(device="cuda").manual_seed(M + N + D)

    def rows(h, n):  # with an odd base the rows are only 4-byte aligned
        x = torch.randn(B * h * n * D + offset, generator=g, device="cuda")[offset:].view(B, h, n, D)
        return x.detach().requires_grad_()

    q, k, v, do = rows(H, M), rows(Hk, N), rows(Hk, N), rows(H, M).detach()
    eq = ek = None
    keep = torch.ones(B, H, M, N, dtype=torch.bool, device="cuda")
    if mode == 1:
        heads = H if per_head else 1
        # documents of 50 to 180 tokens, so that tiles of 64 between them are skipped, and a few ids that see everything
        ends = torch.cumsum(torch.randint(50, 180, (B, heads, 20), generator=g, device="cuda"), 2)
        ek = -1 - (torch.arange(N, device="cuda")[:, None] >= ends[:, :, None, :]).sum(3)
        ek[torch.rand(ek.shape, generator=g, device="cuda") < 0.02] = 3
        eq = ek[..., torch.arange(M, device="cuda") + N - M] if N >= M else ek[..., torch.randint(0, N, (M,), generator=g, device="cuda")]
        eq, ek = eq.expand(B, H, M), ek.expand(B, H, N)
        keep &= (eq[..., None] >= 0) | (eq[..., None] == ek[..., None, :])
    if causal:
        keep &= torch.ones(M, N, dtype=torch.bool, device="cuda").tril(N - M)
    o = fb.attention(q, k, v, causal, None, eq, ek, mode)
    o.backward(do)
    fb.check_status()
    qe, ke, ve = [t.detach().double().requires_grad_() for t in (q, k, v)]
    s = (qe @ ke.repeat_interleave(2, 1).transpose(2, 3) / D ** 0.5).masked_fill(~keep, -torch.inf)
    oe = torch.softmax(s, 3) @ ve.repeat_interleave(2, 1)
    oe.backward(do.double())
    for what, got, want in (("o", o, oe), ("dq", q.grad, qe.grad), ("dk", k.grad, ke.grad), ("dv", v.grad, ve.grad)):
        assert (got.double() - want).abs().max().item() < 1e-4, what


@pytest.mark.parametrize("D", [16, 64, 128])
@pytest.mark.parametrize("G,sees", [(2, (0, 1)), (2, (1, 0)), (4, (0, 1, 1, 1)), (4, (1, 0, 0, 1)), (4, (1, 1, 1, 0)), (4, (0, 0, 0, 0))])
def test_heads_of_a_group_that_see_nothing_of_a_key_block(G, sees, D, monkeypatch):
    """Ids per head: some heads of a group have no query in the document that fills the first and the third block of
    keys, so dK / dV finds no tile for them there and goes straight on to the next head."""
    import flash_b200 as fb
    monkeypatch.setattr(fb.ops, "GROUP_QUERIES", False)  # the caller's order of queries, so that every block is mixed
    B, Hk, M, N = 2, 3, 1500, 500
    H = G * Hk
    g = torch.Generator(device="cuda").manual_seed(G + D)
    q, k, v, do = [torch.randn(B, h, n, D, generator=g, device="cuda") for h, n in ((H, M), (Hk, N), (Hk, N), (H, M))]
    ek = (-1 - torch.arange(N, device="cuda") // 128 % 2).expand(B, H, N)
    eq = -2 + torch.randint(0, 2, (B, H, M), generator=g, device="cuda")
    for h in range(H):
        if not sees[h % G]:
            eq[:, h] = -2
    keep = eq[..., None] == ek[..., None, :]
    for t in (q, k, v):
        t.requires_grad_()
    o = fb.attention(q, k, v, False, None, eq, ek, 1)
    o.backward(do)
    fb.check_status()
    qe, ke, ve = [t.detach().double().requires_grad_() for t in (q, k, v)]
    s = (qe @ ke.repeat_interleave(G, 1).transpose(2, 3) / D ** 0.5).masked_fill(~keep, -torch.inf)
    oe = torch.softmax(s, 3) @ ve.repeat_interleave(G, 1)
    oe.backward(do.double())
    for what, got, want in (("o", o, oe), ("dq", q.grad, qe.grad), ("dk", k.grad, ke.grad), ("dv", v.grad, ve.grad)):
        assert (got.double() - want).abs().max().item() < 1e-4, what


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["k", "v", "q", "do"])
@pytest.mark.parametrize("gap", [0, 64])
def test_values_that_the_causal_mask_hides_from_a_whole_block_of_rows(gap, where, value):
    """A NaN or an infinity in a key that no query of a block of 32 may see (or in a query that sees no key of a block)
    leaves that block's results alone, although a tile of 64 columns holds it."""
    import flash_b200 as fb
    B, H, M, D = 1, 2, 192, 64
    N = M + gap
    g = torch.Generator(device="cuda").manual_seed(gap)
    t = {n: torch.randn(B, H, l, D, generator=g, device="cuda") for n, l in (("q", M), ("k", N), ("v", N), ("do", M))}
    for n in ("q", "k", "v"):
        t[n].requires_grad_()

    def step():
        o = fb.attention(t["q"], t["k"], t["v"], True)
        return (o.detach(), *torch.autograd.grad(o, (t["q"], t["k"], t["v"]), t["do"]))

    clean = step()
    with torch.no_grad():
        # key 100 + gap is in the second half of a tile that queries 64..95 work on, query 70 in the first half of one
        # that keys 96 + gap.. work on
        t[where][0, 1, 100 + gap if where in "kv" else 70] = value
    o, dq, dk, dv = step()
    fb.check_status()
    if where in "kv":
        assert torch.equal(o[:, :, :96], clean[0][:, :, :96]) and torch.equal(dq[:, :, :96], clean[1][:, :, :96])
    else:
        rows = slice(96 + gap, None)
        assert torch.equal(dk[:, :, rows], clean[2][:, :, rows]) and torch.equal(dv[:, :, rows], clean[3][:, :, rows])


@pytest.mark.parametrize("D", [16, 128])
def test_blocks_without_a_visible_tile(D):
    """Many CTAs that load their rows and find nothing to do, between others that do: zeros, and the others undisturbed."""
    import flash_b200 as fb
    B, H, L = 8, 8, 1024
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v, do = [torch.randn(B, H, L, D, generator=g, device="cuda").requires_grad_() for _ in range(4)]
    ek = (-1 - torch.arange(L, device="cuda") // 256).expand(B, H, L)
    blind = torch.arange(L, device="cuda") // 128 % 2 == 1  # every other block of queries is in no document
    eq = torch.where(blind, torch.full_like(ek, -9), ek)

    def step():
        o = fb.attention(q, k, v, True, None, eq, ek, 1)
        return (o, *torch.autograd.grad(o, (q, k, v), do))

    o, dq, dk, dv = step()
    fb.check_status()
    assert bool((o[:, :, blind] == 0).all()) and bool((dq[:, :, blind] == 0).all())
    qe, ke, ve = [t[:2].detach().double().requires_grad_() for t in (q, k, v)]
    keep = ((eq[:2, :, :, None] == ek[:2, :, None]) & torch.ones(L, L, dtype=torch.bool, device="cuda").tril())[:, :, ~blind]
    s = (qe[:, :, ~blind] @ ke.transpose(2, 3) / D ** 0.5).masked_fill(~keep, -torch.inf)
    oe = torch.softmax(s, 3) @ ve
    want = torch.autograd.grad(oe, (qe, ke, ve), do[:2, :, ~blind].double())
    for got, x in ((o[:2, :, ~blind], oe), (dq[:2], want[0]), (dk[:2], want[1]), (dv[:2], want[2])):
        assert (got.double() - x).abs().max().item() < 1e-4
    for a, b in zip((o, dq, dk, dv), step()):
        assert torch.equal(a, b)
