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


@pytest.mark.parametrize("M,N,causal,ndoc,run,per_head,D", [
    (300, 300, True, 5, 1, False, 64),     # five codes a chunk, six with an id that attends everywhere: some blocks either way
    (300, 300, True, 40, 1, True, 128),    # up to 32 codes
    (1000, 1300, True, 30, 10, False, 64),
    (120, 500, False, 6, 1, True, 128)])
def test_walk_and_compare_give_the_same_bits(M, N, causal, ndoc, run, per_head, D, monkeypatch):
    """The plan's flag of a block with many distinct codes decides how the backward compares its codes, and nothing else."""
    import flash_b200 as fb
    from flash_b200 import ops
    B, H, Hk = 2, 4, 2
    g = torch.Generator(device="cuda").manual_seed(N + ndoc)
    q, k, v, do = [torch.randn(B, h, n, D, generator=g, device="cuda").bfloat16() for h, n in ((H, M), (Hk, N), (Hk, N), (H, M))]
    ek = -1 - torch.randint(0, ndoc, (B, H if per_head else 1, N // run + 1), generator=g, device="cuda").repeat_interleave(run, 2)[..., :N]
    ek[torch.rand(ek.shape, generator=g, device="cuda") < 0.03] = 5
    eq, ek = ek[..., N - M:].expand(B, H, M), ek.expand(B, H, N)
    for t in (q, k, v):
        t.requires_grad_()
    build, flags = ops.build_plan, []

    def build_with(many):
        def made(*args):
            plan = build(*args)
            rows, nq, nk = B * (H if per_head else 1), -(-M // 128), -(-N // 128)
            up = lambda n: -(-n // 128) * 128
            at = rows * 128 * (nq + nk) + 4 * up(rows * nq) + 4 * up(rows * nk)  # codes, min / max, ranges
            qf, kf = plan[at:at + rows * nq], plan[at + up(rows * nq):at + up(rows * nq) + rows * nk]
            flags.extend((qf.clone(), kf.clone()))
            for f in (qf, kf):
                if many is not None:
                    f.copy_(f & 1 | (2 if many else 0))
            return plan
        return made

    results = []
    for many in (None, False, True):
        monkeypatch.setattr(ops, "build_plan", build_with(many))
        results.append(torch.autograd.grad(fb.attention(q, k, v, causal, None, eq, ek, 1), (q, k, v), do))
    fb.check_status()
    # the flags are the rule's: more than five distinct codes in 32 rows (padding of the last block included)
    codes = torch.nn.functional.pad(torch.where(eq >= 0, torch.full_like(eq, 1 << 40), eq)[:, :H if per_head else 1], (0, -M % 128), value=1 << 40)
    chunks = codes.reshape(-1, 32).sort(1).values
    want = ((chunks.diff(dim=1) != 0).sum(1) + 1 > 5).view(-1, 4).any(1)
    assert torch.equal((flags[0] & 2) != 0, want.view(-1))
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))
