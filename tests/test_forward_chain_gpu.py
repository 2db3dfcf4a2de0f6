"""The forward's two chains of tiles: an accumulator and a running maximum each, merged at the end of an item."""
import os
import subprocess
import sys

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
    rows, and fall in the others, so that each tile moves its chain's maximum."""
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


def growing_inputs(B, H, Hk, M, N, D, dtype, seed):
    """Scores that rise from tile to tile by more than the slack of the lazy rescale in half of the rows and fall in the
    others, twice over, so that both chains rescale, too, when they have come down."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda") for h, n in ((H, M), (Hk, N), (Hk, N)))
    q[..., 0] = torch.where(torch.arange(M, device="cuda") % 2 == 0, 1.0, -1.0) * D ** 0.5
    k[..., 0] = torch.arange(N, device="cuda") // 128 % 4 * 12.0
    return [x.to(dtype) for x in (q, k, v)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("form", ["full", "causal", "ids"])
@pytest.mark.parametrize("tiles", [1, 3, 6])
def test_many_items_a_cta_while_the_maximum_moves(tiles, form, D, dtype):
    """Six items a CTA on 148 SMs: the item slots, the accumulators and the barriers of both are used again several times,
    by items of an even, an odd and (ids, causal) a varying number of tiles."""
    import flash_b200 as fb
    B, H, M, N = 4, 112, 256, tiles * 128 - (0 if tiles == 1 else 5)
    M = min(M, N)
    H = H * 256 // (-(-M // 128) * 128)
    q, k, v = growing_inputs(B, H, H, M, N, D, dtype, tiles * D)
    keep, args = None, (form != "full",)
    if form == "ids":
        ek = -1 - torch.arange(N, device="cuda") // 170
        eq = ek[N - M:].clone()
        eq[::50] = 3  # attends to all
        keep = (eq[:, None] >= 0) | (eq[:, None] == ek)
        args = (True, None, eq.expand(B, H, M), ek.expand(B, H, N), fb.SCORE_FUNC_MODE1_DOC)
    o = fb.attention(q, k, v, *args)
    for b in range(B):
        check(o[b:b + 1], *reference(q[b:b + 1], k[b:b + 1], v[b:b + 1], form != "full", keep), scale=16.0 + 48.0)
    assert torch.equal(o, fb.attention(q, k, v, *args))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("runs", [1, 3])
def test_many_packed_items_while_the_maximum_moves(runs, D):
    import flash_b200 as fb
    B, H, Hk, M, N = 100, 32, 8, 16, 1400
    q, k, v = growing_inputs(B, H, Hk, M, N, D, torch.bfloat16, D)
    o = fb.attention_in_runs(q, k, v, runs, True)
    for b in range(0, B, 20):
        part = slice(b, b + 20)
        ke, ve = (x[part].repeat_interleave(H // Hk, 1) for x in (k, v))
        check(o[part], *reference(q[part], ke, ve, True), scale=16.0 + 48.0)


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


@pytest.mark.parametrize("tiles", [2, 5, 6])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_both_chains_have_a_maximum_of_their_own(dtype, D, tiles):
    """Each row sees one key in each of the last two tiles. Relative to their own chain's maximum both are an exact 1 in P,
    whatever their scores are, so that P's rounding (2^-9 or 2^-12 of each) is not in the result, of which the values leave
    little: what is left is the rounding of the result, and 2^-18 for scores and exponentials in fp32 (a score of 12 and
    its multiple by log2(e) to 2^-21 each, the exponential to 2^-22, twice the value of one)."""
    import flash_b200 as fb
    B, H, M, N = 2, 80, 256, tiles * 128
    q, k, v = (torch.zeros(B, H, n, D, device="cuda") for n in (M, N, N))
    q[..., 0] = 1 + torch.arange(M, device="cuda") % 128 / 64
    k[..., 0] = -200.0
    first, second = N - 256 + 37, N - 128 + 90
    k[:, :, first, 0], k[:, :, second, 0] = 3.0, 2.3125
    v[:, :, first], v[:, :, second] = 1.0, -2.0
    q, k, v = (x.to(dtype) for x in (q, k, v))
    o = fb.attention(q, k, v, False, 1.0)
    w = (0.6875 * q[..., :1].double()).exp()  # the first key's weight over the second's
    ref = ((w - 2.0) / (w + 1.0)).expand(B, H, M, D)
    unit = torch.finfo(dtype).eps / 2
    err = (o.double() - ref).abs()
    assert bool((err <= unit * ref.abs() * 1.01 + 2.0 ** -18).all()), err.max().item()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_values_behind_the_mask_of_a_whole_chain(value, D):
    """A row with no key in a chain's tiles does not see what their values are, by the causal mask and by ids."""
    import flash_b200 as fb
    H = 4
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(1, H, n, D, generator=g, device="cuda").bfloat16() for n in (128, 192, 192))
    v[:, :, 150] = value  # row i sees the keys up to i + 64: the first 64 rows have none in the second tile
    o = fb.attention(q, k, v, True)
    ref, absolute = reference(q[:, :, :64], k[:, :, :128], v[:, :, :128], True)
    check(o[:, :, :64], ref, absolute, 16.0)
    assert not torch.isfinite(o[:, :, 86:]).any()
    q, k, v = (torch.randn(1, H, 256, D, generator=g, device="cuda").bfloat16() for _ in range(3))
    ids = torch.where(torch.arange(256, device="cuda") < 100, -1, -2).expand(1, H, 256)
    v[:, :, 200] = value  # the first 100 rows share their block with others that do have keys in the second tile
    o = fb.attention(q, k, v, False, None, ids, ids, fb.SCORE_FUNC_MODE1_DOC)
    check(o[:, :, :100], *reference(q[:, :, :100], k[:, :, :100], v[:, :, :100], False), 16.0)
    assert not torch.isfinite(o[:, :, 100:]).any()


@pytest.mark.parametrize("D", [64, 128])
def test_a_row_whose_score_overflows_is_nan(D):
    import flash_b200 as fb
    q, k, v = (torch.randn(1, 4, 512, D, generator=torch.Generator(device="cuda").manual_seed(i), device="cuda").bfloat16() for i in range(3))
    q[..., 0] = 4.0
    k[:, :, 300] = 0.0
    k[:, :, 300, 0] = 3e38  # a score of +inf for the rows that see this key
    o = fb.attention(q, k, v, True)
    assert bool(torch.isfinite(o[:, :, :300]).all()) and bool(torch.isnan(o[:, :, 300:]).all())


def test_an_item_may_last_longer_than_the_limit_of_a_wait(repo_root):
    """An item of 1024 tiles takes over a million clocks, five times the limit set here, and no wait within it more than a
    twentieth of the limit: the epilogue group, which waits for the whole item, goes by its tiles."""
    code = """
import torch, flash_b200 as fb
q = torch.randn(1, 2, 128, 64, device="cuda").bfloat16()
k, v = (torch.randn(1, 2, 131072, 64, device="cuda").bfloat16() for _ in range(2))
o = fb.attention_in_runs(q, k, v, 1)
fb.check_status()
assert bool(torch.isfinite(o).all())
"""
    path = os.path.join(repo_root, "triton-flash-attention-with-flexible-masks_b200")
    env = dict(os.environ, FA_B200_WAIT_LIMIT_CLOCKS="200000", PYTHONPATH=path + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
