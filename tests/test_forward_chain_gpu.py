"""The forward's chain of tiles: three score buffers, one accumulator, a reference maximum handed from tile to tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(q, k, v, causal, keep=None):
    """(o, sum p |v|) in 64 bits; a row without keys gives zeros."""
    (B, H, M, D), N = q.shape, k.shape[2]
    s = q.double() @ k.double().transpose(2, 3) / D ** 0.5
    mask = torch.ones(M, N, dtype=torch.bool, device=q.device)
    if causal:
        mask = mask.tril(N - M)
    mask = mask if keep is None else mask & keep
    s = s.masked_fill(~mask, -torch.inf)
    p = (s - s.amax(3, keepdim=True).clamp(min=-1e300)).exp()
    p = p / p.sum(3, keepdim=True).clamp(min=1e-300)
    return p @ v.double(), p @ v.double().abs()


def check(o, ref, absolute, scale):
    # P is rounded to the inputs' type (half a unit in the last place of each entry), and so is the result; the scores
    # are sums in fp32 of products of at most `scale`, and exp2 turns their absolute error into a relative one of P
    unit = torch.finfo(o.dtype).eps / 2
    bound = unit * (absolute + ref.abs()) * 1.01 + scale * 2.0 ** -20 * absolute + 1e-6
    err = (o.double() - ref).abs()
    assert bool((err <= bound).all()), (err - bound).max().item()


@pytest.mark.parametrize("D", [16, 64, 128])
@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 7, 10])
@pytest.mark.parametrize("growing", [False, True], ids=["flat", "growing"])
def test_tiles_and_moving_maximum(tiles, D, growing):
    """`growing`: every tile's scores exceed the last one's by more than the slack of the lazy rescale in half of the
    rows, and fall in the others, so that each tile of one group moves the maximum that the other group goes on from."""
    import flash_b200 as fb
    B, H, M, N = 2, 40, 256, tiles * 128 - 5  # more items than SMs, whose tiles start at even and odd places of the ring
    g = torch.Generator(device="cuda").manual_seed(tiles * D)
    q, k, v = (torch.randn(B, H, n, D, generator=g, device="cuda") for n in (M, N, N))
    if growing:
        ramp = torch.arange(N, device="cuda") // 128 * 12.0
        q[..., 0] = torch.where(torch.arange(M, device="cuda") % 2 == 0, 1.0, -1.0) * D ** 0.5
        k[..., 0] = ramp
    q, k, v = (x.bfloat16() for x in (q, k, v))
    o = fb.attention(q, k, v)
    check(o, *reference(q, k, v, False), scale=16.0 + (12.0 * tiles if growing else 0))
    assert torch.equal(o, fb.attention(q, k, v))


@pytest.mark.parametrize("D", [64, 128])
def test_items_without_tiles_between_others(D):
    """Blocks whose ids no key carries, in between blocks with one to six tiles."""
    import flash_b200 as fb
    B, H, N = 2, 64, 1500
    g = torch.Generator(device="cuda").manual_seed(D)
    ids = -1 - torch.arange(N, device="cuda") // 170
    eq = ids.clone()
    eq[256:512] = -1000
    eq[1280:1408] = -1001
    q, k, v = (torch.randn(B, H, N, D, generator=g, device="cuda").half() for _ in range(3))
    o = fb.attention(q, k, v, True, None, eq.expand(B, H, N), ids.expand(B, H, N), fb.SCORE_FUNC_MODE1_DOC)
    ref, absolute = reference(q, k, v, True, eq[:, None] == ids[None, :])
    check(o, ref, absolute, 16.0)
    assert not o[:, :, 256:512].any() and not o[:, :, 1280:1408].any()
