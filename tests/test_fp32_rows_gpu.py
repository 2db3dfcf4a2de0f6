"""fp32 kernels: blocks of 16 rows in small calls, of 32 in large ones; a sequence's bits do not depend on which."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def exact(q, k, v, do, causal, eq, ek):
    q, k, v = (x.detach().double().requires_grad_() for x in (q, k, v))
    M, N, G = q.shape[2], k.shape[2], q.shape[1] // k.shape[1]
    s = q @ k.repeat_interleave(G, 1).transpose(2, 3) / q.shape[3] ** 0.5
    i, j = torch.arange(M, device="cuda")[:, None], torch.arange(N, device="cuda")[None]
    keep = torch.ones(M, N, dtype=torch.bool, device="cuda")
    if causal:
        keep = keep & (j <= i + max(0, N - M))
    if eq is not None:
        keep = keep & ((eq[..., None] >= 0) | (eq[..., None] == ek[..., None, :]))
    s = s.masked_fill(~keep, -torch.inf)
    p = (s - s.amax(3, keepdim=True).clamp(min=-1e300)).exp()
    o = (p / p.sum(3, keepdim=True).clamp(min=1e-300)) @ v.repeat_interleave(G, 1)
    return (o.detach(), *torch.autograd.grad(o, (q, k, v), do.double()))


@pytest.mark.parametrize("M,N", [(1, 1), (15, 15), (16, 17), (33, 64), (65, 130), (113, 129)])
@pytest.mark.parametrize("D", [16, 32, 64, 128])
def test_rows_of_a_block(D, M, N):
    import flash_b200 as fb
    H, Hk = 16, 8
    B = max(2, 700 // (H * ((M + 31) // 32)))  # more blocks of 32 rows than any rule gives 16
    g = torch.Generator(device="cuda").manual_seed(M + D)
    q, k, v, do = (torch.randn(B, h, n, D, generator=g, device="cuda") for h, n in ((H, M), (Hk, N), (Hk, N), (H, M)))
    ek = -1 - torch.randint(0, 3, (B, 1, N), generator=g, device="cuda")
    ek[torch.rand(ek.shape, generator=g, device="cuda") < 0.1] = 4
    eq, ek = ek[..., N - M:].expand(B, H, M), ek.expand(B, H, N)

    def step(b, ids):
        x = [t[:b].clone().requires_grad_() for t in (q, k, v)]
        o = fb.attention(*x, True, None, *((eq[:b], ek[:b], 1) if ids else (None, None, 0)))
        return o.detach(), *torch.autograd.grad(o, x, do[:b])

    for ids in (False, True):
        many, one = step(B, ids), step(1, ids)
        assert all(torch.equal(a[:1], b) for a, b in zip(many, one))
        # Sums of up to N + D terms (dK, dV: M rows of two heads) in fp32, a few behind each other. dS is a difference of two numbers as
        # large as |dO| |V|, which may all but cancel: the bound goes by what a term can be, or by the sum where that is larger.
        dp = float((do.norm(dim=3).amax() * v.norm(dim=3).amax())) / D ** 0.5
        terms = (v.abs().amax(), dp * k.abs().amax(), dp * q.abs().amax(), do.abs().amax())
        for got, want, term in zip(many, exact(q, k, v, do, True, *((eq, ek) if ids else (None, None))), terms):
            bound = 2.0 ** -24 * 8 * (max(M, N) + D) ** 0.5 * want.abs().amax(dim=(2, 3), keepdim=True).clamp(min=float(term))
            assert bool(((got.double() - want).abs() <= bound).all())
    fb.check_status()
