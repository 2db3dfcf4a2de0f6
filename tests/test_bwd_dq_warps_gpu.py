"""dQ with sixteen compute warps (ids, no causal mask, head dims up to 64) against the kernel with eight: ids that mask nothing, the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(1, 1), (100, 300), (128, 128), (129, 127), (300, 1000), (700, 129)])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_same_bits(dtype, D, M, N):
    import flash_b200 as fb
    B, H, Hk = 2, 4, 2
    g = torch.Generator(device="cuda").manual_seed(M + N + D)
    q, k, v, do = (torch.randn(B, h, n, D, generator=g, device="cuda").to(dtype) for h, n in ((H, M), (Hk, N), (Hk, N), (H, M)))
    eq, ek = torch.full((B, H, M), -3, device="cuda"), torch.full((B, H, N), -3, device="cuda")

    def step(ids):
        x = [t.clone().requires_grad_() for t in (q, k, v)]
        o = fb.attention(*x, False, None, *((eq, ek, 1) if ids else (None, None, 0)))
        return o.detach(), *torch.autograd.grad(o, x, do)

    assert all(torch.equal(a, b) for a, b in zip(step(True), step(False)))
    # two documents, the second one's queries and keys behind the first's: each is a call of its own
    if M > 1:
        m, n = M // 2, N // 2
        eq[..., m:], ek[..., n:] = -4, -4
        whole = step(True)
        for lo, hi, a, b in ((0, m, 0, n), (m, M, n, N)):
            x = [t.clone().requires_grad_() for t in (q[:, :, lo:hi], k[:, :, a:b], v[:, :, a:b])]
            o = fb.attention(*x, False)
            part = (o.detach(), *torch.autograd.grad(o, x, do[:, :, lo:hi]))
            for w, p in zip((whole[0][:, :, lo:hi], whole[1][:, :, lo:hi], whole[2][:, :, a:b], whole[3][:, :, a:b]), part):
                # P and dS are rounded to the type on either side, by other maxima
                eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
                assert float((w.double() - p.double()).norm()) <= 4 * eps * float(p.double().norm())
    fb.check_status()
