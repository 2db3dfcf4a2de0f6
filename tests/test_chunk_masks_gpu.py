"""The backward kernels' 32-column masks: chunks with one, a few and more than six distinct ids, ids per head, key and
query tails, positions that attend everywhere, against plain attention in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("M,N,causal,ndoc,run,per_head", [
    (300, 300, True, 3, 1, False),     # scattered ids, few distinct
    (300, 300, True, 40, 1, True),     # scattered, more than six distinct in every chunk
    (513, 641, True, 25, 5, False),    # short runs: six and seven distinct codes in a chunk
    (257, 257, True, 9, 32, True),     # runs of a chunk's length
    (120, 500, False, 12, 4, False)])  # not causal, too few queries to be grouped
def test_backward_chunk_masks(M, N, causal, ndoc, run, per_head, D):
    import flash_b200 as fb
    B, H, Hk = 2, 4, 2
    g = torch.Generator(device="cuda").manual_seed(N + ndoc)
    q, k, v, do = [torch.randn(B, h, n, D, generator=g, device="cuda").bfloat16() for h, n in ((H, M), (Hk, N), (Hk, N), (H, M))]
    ek = -1 - torch.randint(0, ndoc, (B, H if per_head else 1, N // run + 1), generator=g, device="cuda").repeat_interleave(run, 2)[..., :N]
    ek[torch.rand(ek.shape, generator=g, device="cuda") < 0.03] = 5
    eq, ek = ek[..., N - M:].expand(B, H, M), ek.expand(B, H, N)
    keep = (eq[..., None] >= 0) | (eq[..., None] == ek[..., None, :])
    if causal:
        keep = keep & torch.ones(M, N, dtype=torch.bool, device="cuda").tril(N - M)
    for t in (q, k, v):
        t.requires_grad_()
    o = fb.attention(q, k, v, causal, None, eq, ek, 1)
    o.backward(do)
    fb.check_status()
    qe, ke, ve = [t.detach().double().requires_grad_() for t in (q, k, v)]
    s = (qe @ ke.repeat_interleave(2, 1).transpose(2, 3) / D ** 0.5).masked_fill(~keep, -torch.inf)
    oe = torch.softmax(s, 3) @ ve.repeat_interleave(2, 1)
    oe.backward(do.double())
    for what, got, want in (("o", o, oe), ("dq", q.grad, qe.grad), ("dk", k.grad, ke.grad), ("dv", v.grad, ve.grad)):
        # Rounded to bf16 on the way (2^-9 of the value each): P or dS, O (which enters dS through delta whatever the
        # size of the row's own gradient, hence the tensor's mean row beside the row's norm) and the result; twice that
        # for the sums. A mask bit that is wrong adds or drops a key of the at most few dozen that a row sees.
        want = want.detach()
        norm = want.norm(dim=3)
        bound = 6 * 2.0 ** -9 * (norm + norm.square().mean().sqrt())
        err = (got.detach().double() - want).norm(dim=3)
        assert bool((err <= bound).all()), (what, (err / bound).max().item())
