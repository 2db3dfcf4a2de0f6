"""Forward calls without ids that are short of work: query heads of a group packed into one tile, keys cut into
runs that are merged afterwards. Against plain attention in 64 bits, with a bound that scales with the result: the long
calls' outputs and gradients are a few hundredths of the inputs."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [  # B, H, Hk, M, N, D, causal
    (1, 8, 2, 1, 128, 64, True),      # one token, one tile of keys
    (2, 8, 1, 1, 4500, 128, True),    # a group of 8, ragged keys, split
    (1, 64, 8, 1, 700, 32, False),
    (16, 32, 8, 1, 1000, 128, True),  # packed, not split
    (1, 6, 2, 50, 3000, 64, True),    # a group of 3 in tiles of 2 heads: the second tile is half empty
    (1, 16, 4, 32, 9000, 128, True),  # a full tile of packed rows
    (1, 12, 4, 64, 64, 128, True),    # two heads a tile, diagonal inside it
    (1, 8, 8, 65, 5000, 64, True),    # no packing, split
    (1, 4, 4, 300, 7777, 128, True),  # three query blocks a head, split
    (1, 4, 4, 1000, 4096, 16, False),
    (1, 2, 1, 3, 40000, 128, True),
]


@pytest.fixture(scope="module")
def fb():
    import flash_b200
    return flash_b200


def _exact(q, k, v, causal):
    G, M, N = q.shape[1] // k.shape[1], q.shape[2], k.shape[2]
    q, k, v = q.double(), k.double().repeat_interleave(G, 1), v.double().repeat_interleave(G, 1)
    s = q @ k.transpose(2, 3) / q.shape[3] ** 0.5
    if causal:
        s = s.masked_fill(torch.ones(M, N, dtype=torch.bool, device=q.device).triu(N - M + 1), -torch.inf)
    return torch.softmax(s, 3) @ v, torch.logsumexp(s, 3) / torch.log(torch.tensor(2.0, device=q.device, dtype=torch.float64))


def _close(got, want, what):
    """Row by row, by norm. Rounded to 16 bits on the way, u of a value each: P or dS, O (which enters dS through delta
    whatever the size of the row's own gradient, hence the tensor's mean row beside the row's norm) and the result; the
    roundings of a row's D columns and N keys are independent, and 8 is over twice the sum of the three at four standard
    deviations of rows this long. A tile of 128 keys that is lost or counted twice is sqrt(128 / N) of an output's norm: at
    least 0.056 here, where the bound is 16 u = 0.031 in bf16."""
    u = 2.0 ** -9 if got.dtype == torch.bfloat16 else 2.0 ** -12
    norm = want.norm(dim=-1)
    bound = 8 * u * (norm + norm.square().mean().sqrt())
    err = (got.double() - want).norm(dim=-1)
    assert bool((err <= bound).all()), (what, (err / bound).max().item())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(str(int(x)) for x in c))
def test_short_forward(fb, case, dtype):
    B, H, Hk, M, N, D, causal = case
    g = torch.Generator(device="cuda").manual_seed(M * N)
    # q as a projection leaves it ([B, M, H, D] transposed), k and v contiguous
    q = torch.randn(B, M, H, D, generator=g, device="cuda").to(dtype).transpose(1, 2).requires_grad_()
    k, v = [torch.randn(B, Hk, N, D, generator=g, device="cuda").to(dtype).requires_grad_() for _ in range(2)]
    do = torch.randn(B, H, M, D, generator=g, device="cuda").to(dtype)
    o = fb.attention(q, k, v, causal)
    o.backward(do)
    fb.check_status()
    qe, ke, ve = [t.detach().double().requires_grad_() for t in (q, k, v)]
    oe, _ = _exact(qe, ke, ve, causal)
    oe.backward(do.double())
    for what, got, want in (("o", o, oe), ("dq", q.grad, qe.grad), ("dk", k.grad, ke.grad), ("dv", v.grad, ve.grad)):
        _close(got.detach(), want.detach(), what)


@pytest.mark.parametrize("H,Hk,M", [(4, 2, 300), (8, 2, 1), (4, 1, 3), (6, 2, 50)])
@pytest.mark.parametrize("splits", [1, 2, 5, 16])
def test_any_number_of_runs(fb, splits, H, Hk, M):
    """Also numbers the rule would not take, among them runs that the causal bound leaves without keys; the lse too, of
    packed tiles as well."""
    from flash_b200 import _lib, ops
    B, N, D = 2, 2048, 64
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(3)
    q, o = torch.randn(B, H, M, D, generator=g, device="cuda").bfloat16(), torch.empty(B, H, M, D, device="cuda", dtype=torch.bfloat16)
    k, v = [torch.randn(B, Hk, N, D, generator=g, device="cuda").bfloat16() for _ in range(2)]
    prob = ops._problem(B, H, Hk, M, N, D, q.dtype, True, 0, 1, D ** -0.5)
    lse = torch.full((B, H, -(-M // 128) * 128), float("nan"), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    n = ctypes.c_size_t(0)
    assert lib.fa_fwd_workspace_bytes(ctypes.byref(prob), splits, ctypes.byref(n)) == 0
    assert (n.value == 0) == (splits == 1)
    work = torch.full((max(4, n.value // 4),), float("nan"), device="cuda")
    tq, tk, tv, to = [ops._tensor(t) for t in (q, k, v, o)]
    args = [ctypes.byref(x) for x in (prob, tq, tk, tv, to)]
    if splits > 1:
        assert lib.fa_fwd_split(*args, lse.data_ptr(), None, splits, work.data_ptr(), n.value - 4, status.data_ptr(), ops._stream()) == 6
    assert lib.fa_fwd_split(*args, lse.data_ptr(), None, 17, work.data_ptr(), 1 << 40, status.data_ptr(), ops._stream()) == 2
    assert lib.fa_fwd_split(*args, lse.data_ptr(), None, splits, work.data_ptr(), n.value, status.data_ptr(), ops._stream()) == 0
    oe, le = _exact(q, k, v, True)
    _close(o, oe, "o")
    assert (lse[..., :M].double() - le).abs().max().item() < 1e-4 and bool(torch.isfinite(lse).all())
    assert int(status.item()) == 0


@pytest.mark.parametrize("what", ["nan in k", "overflowing score", "all of a run is nan", "nan in v", "inf in v", "-inf scores"])
@pytest.mark.parametrize("M,G", [(1, 4), (40, 2), (200, 1)])
def test_values_that_are_not_finite_do_not_get_lost_in_a_run(fb, M, G, what):
    """A call cut into runs gives such rows as the call of one run does: zeros with an lse of -inf where a score is NaN,
    NaN with an lse of -inf where one is +inf, NaN or an infinity where only a value is."""
    from flash_b200 import _lib, ops
    B, Hk, N, D, splits = 2, 2, 1500, 64, 4
    H = G * Hk
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(M)
    q = torch.randn(B, H, M, D, generator=g, device="cuda").bfloat16()
    k, v = [torch.randn(B, Hk, N, D, generator=g, device="cuda").bfloat16() for _ in range(2)]
    if what == "nan in k":
        k[1, 0, 700, 3] = float("nan")
    elif what == "overflowing score":  # +inf for one half of the rows, -inf for the other
        k[1, 0, 700] = 0
        k[1, 0, 700, 0] = 3e38
        odd = (torch.arange(G, device="cuda")[:, None] + torch.arange(M, device="cuda")) % 2
        q[1, :G, :, 0] = (4 - 8 * odd).bfloat16()
    elif what == "all of a run is nan":
        k[1, 0, 256:768] = float("nan")
    elif what == "-inf scores":
        q[1, :G, :, 0] = 1
        k[1, 0, 512:900, 0] = -float("inf")
    else:
        v[1, 0, 700, 3] = float(what.split()[0])
    prob = ops._problem(B, H, Hk, M, N, D, q.dtype, True, 0, 1, D ** -0.5)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    n = ctypes.c_size_t(0)
    assert lib.fa_fwd_workspace_bytes(ctypes.byref(prob), splits, ctypes.byref(n)) == 0
    work = torch.empty(n.value // 4, device="cuda")
    results = []
    for ns in (1, splits):
        o, lse = torch.empty_like(q), torch.empty(B, H, -(-M // 128) * 128, device="cuda")
        assert lib.fa_fwd_split(prob, ops._tensor(q), ops._tensor(k), ops._tensor(v), ops._tensor(o), lse.data_ptr(), None, ns,
                                work.data_ptr(), n.value, status.data_ptr(), ops._stream()) == 0
        results.append((o.double(), lse[..., :M].double()))
    assert int(status.item()) == 0
    (o1, l1), (o2, l2) = results
    dead = l1 == -torch.inf
    if "v" not in what.split()[-1:] and what != "-inf scores":  # the case does what it says: rows of the group are lost
        assert bool(dead[1, :G].any()) and bool(((o1[dead] == 0) | torch.isnan(o1[dead])).all())
    assert torch.equal(dead, l2 == -torch.inf)
    assert bool(((l1 - l2).abs() < 1e-4 + 1e-6 * l1.abs())[~dead].all())
    assert torch.equal(torch.isnan(o1), torch.isnan(o2))
    assert torch.equal(o1.nan_to_num(0, 0, 0).ne(0).any(3), o2.nan_to_num(0, 0, 0).ne(0).any(3))
    finite = (torch.isfinite(o1) & torch.isfinite(o2)).all(3)
    _close(o2[finite].bfloat16(), o1[finite], "o")


@pytest.mark.parametrize("M,N,splits", [(300, 9000, 3), (1, 4000, 11)])
def test_runs_are_dealt_out_alike_with_and_without_a_plan(fb, M, N, splits):
    """A split call for which a plan is optional, with more runs than SMs: the same bits either way, twice with one plan."""
    from flash_b200 import _lib, ops
    B, H, Hk, D = 4, 32, 8, 64
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(N)
    q = torch.randn(B if M == 1 else 1, H, M, D, generator=g, device="cuda").bfloat16()
    B = q.shape[0]
    k, v = [torch.randn(B, Hk, N, D, generator=g, device="cuda").bfloat16() for _ in range(2)]
    prob = ops._problem(B, H, Hk, M, N, D, q.dtype, True, 0, 1, D ** -0.5)
    assert lib.fa_plan_optional(prob, 0) == 1
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    n = ctypes.c_size_t(0)
    assert lib.fa_fwd_workspace_bytes(prob, splits, ctypes.byref(n)) == 0
    work = torch.empty(n.value // 4, device="cuda")
    plan = ops.build_plan(prob, None, None, status)
    results = []
    for p in (None, plan.data_ptr(), plan.data_ptr()):
        o, lse = torch.empty_like(q), torch.empty(B, H, -(-M // 128) * 128, device="cuda")
        assert lib.fa_fwd_split(prob, ops._tensor(q), ops._tensor(k), ops._tensor(v), ops._tensor(o), lse.data_ptr(), p, splits,
                                work.data_ptr(), n.value, status.data_ptr(), ops._stream()) == 0
        results.append((o, lse))
    assert int(status.item()) == 0
    assert all(torch.equal(o, results[0][0]) and torch.equal(lse, results[0][1]) for o, lse in results[1:])


@pytest.mark.parametrize("runs", [1, 3, "whole call"])
def test_pinned_runs_give_a_sequence_the_same_bits_in_any_batch(fb, runs):
    """A sequence (or a share of the heads) by itself chooses another number of runs than the whole call; with
    `attention_in_runs` it gives the bits that it has in the whole call, gradients included."""
    B, H, Hk, M, N, D = 3, 16, 4, 2, 6000, 64
    g = torch.Generator(device="cuda").manual_seed(0)
    q, k, v, do = [torch.randn(B, h, n, D, generator=g, device="cuda").bfloat16() for h, n in ((H, M), (Hk, N), (Hk, N), (H, M))]
    whole = fb.forward_splits(B, H, Hk, M, N, D, q.dtype, True, 0)
    assert whole > 1 and fb.forward_splits(1, H, Hk, M, N, D, q.dtype, True, 0) != whole
    runs = whole if runs == "whole call" else runs

    def step(*at):
        x = [t[at].clone().requires_grad_() for t in (q, k, v)]
        o = fb.attention_in_runs(*x, runs, True)
        return (o.detach(), *torch.autograd.grad(o, x, do[at]))

    full = step(slice(None))
    for b in range(B):
        assert all(torch.equal(a[b:b + 1], p) for a, p in zip(full, step(slice(b, b + 1))))
    heads = [torch.cat([t[:, 4:8] if i in (0, 1) else t[:, 1:2]], 1) for i, t in enumerate(full)]
    x = [t.clone().requires_grad_() for t in (q[:, 4:8], k[:, 1:2], v[:, 1:2])]
    o = fb.attention_in_runs(*x, runs, True)
    part = (o.detach(), *torch.autograd.grad(o, x, do[:, 4:8]))
    assert all(torch.equal(a, p) for a, p in zip(heads, part))
    if runs == whole:
        assert torch.equal(full[0], fb.attention(q, k, v, True))
    # eight arguments, as before: as many gradients
    o = fb.FlashAttention.apply(q.requires_grad_(), k, v, True, None, None, None, 0)
    o.backward(do)
    with pytest.raises(RuntimeError):  # what cannot be cut is refused
        fb.attention_in_runs(q.detach().float(), k.float(), v.float(), 2, True)
