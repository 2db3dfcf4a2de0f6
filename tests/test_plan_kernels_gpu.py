"""Every word of the mask plan against a numpy restatement, on both sides of the size at which one kernel builds it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ANY, LOWEST = 0x7FFFFFFF, -(1 << 31)


def expected(eq, ek, causal):
    """Sections of the plan of one id row (int64 arrays), in their order in the plan."""
    M, N = len(eq), len(ek)
    nq, nk = -(-M // 128), -(-N // 128)
    qc = np.full(nq * 128, ANY, np.int64)
    qc[:M] = np.where(eq >= 0, ANY, np.maximum(eq, LOWEST))
    kc = np.zeros(nk * 128, np.int64)
    kc[:N] = np.where((ek < 0) & (ek >= LOWEST), ek, 0)

    def stats(codes, n, length):
        blocks = [codes[128 * i:min(128 * i + 128, length)] for i in range(n)]
        flags = []
        for i in range(n):
            c = codes[128 * i:128 * i + 128]
            d = np.diff(c)
            many = any(len(np.unique(c[j:j + 32])) > 5 for j in range(0, 128, 32))
            flags.append((0 if (d > 0).any() and (d < 0).any() else 1) | (2 if many else 0))
        return np.array([b.min() for b in blocks]), np.array([b.max() for b in blocks]), np.array(flags)

    qmin, qmax, qf = stats(qc, nq, M)
    kmin, kmax, kf = stats(kc, nk, N)
    visit = ~((qmax[:, None] < 0) & ((kmax[None] < qmin[:, None]) | (kmin[None] > qmax[:, None])))
    if causal:
        last = np.minimum(np.arange(nq) * 128 + 128, M) - 1 + max(0, N - M)
        visit &= np.arange(nk)[None] * 128 <= last[:, None]

    def ranges(v):
        lo = np.where(v.any(1), v.argmax(1), 0)
        hi = np.where(v.any(1), v.shape[1] - v[:, ::-1].argmax(1), 0)
        return lo, hi

    kvlo, kvhi = ranges(visit)
    qlo, qhi = ranges(visit.T)
    natural = np.arange(nq)[::-1]
    ordq = natural[np.argsort(-(kvhi - kvlo)[natural], kind="stable")]
    ordk = np.argsort(-(qhi - qlo), kind="stable")
    return [qc, kc, qmin, qmax, kmin, kmax, kvlo, kvhi, qlo, qhi, qf, kf, ordq, ordk]


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("M,N,causal", [(1, 1, False), (1, 129, True), (128, 128, True), (300, 500, True), (1000, 1000, True),
                                        (4096, 4096, True), (1024, 7168, False), (1025, 7168, True), (4096, 4097, True), (8192, 8193, True)])
def test_every_word(M, N, causal, dtype):
    from flash_b200 import ops
    B, H = 2, 3
    rng = np.random.default_rng(M + N)
    for per_head in (False, True):
        he = H if per_head else 1
        ek = np.zeros((B, he, N), np.int64)
        for b in range(B):
            for h in range(he):
                kind = (b * he + h) % 3
                if kind == 0:  # documents, in an order of their own, and a few ids that see everything
                    cuts = np.sort(rng.integers(0, N + 1, 9))
                    ek[b, h] = -1 - rng.permutation(10)[np.searchsorted(cuts, np.arange(N), side="right")]
                    ek[b, h, rng.random(N) < 0.01] = 7
                elif kind == 1:  # scattered
                    ek[b, h] = -rng.integers(1, 9, N)
                else:  # falling and one at the edge of int32
                    ek[b, h] = -1 - np.arange(N) // 200
                    ek[b, h, -1] = LOWEST
        eq = ek[:, :, N - M:].copy() if N >= M else ek[:, :, :M]
        eq[0, 0, M // 2] = 3
        t = [torch.from_numpy(x).to("cuda", dtype).expand(B, H, x.shape[2]) for x in (eq, ek)]
        prob = ops._problem(B, H, H, M, N, 64, torch.bfloat16, causal, 1, he, 1.0)
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        plan = ops.build_plan(prob, *t, status).cpu().numpy().astype(np.int64)
        rows = [expected(eq[b, h], ek[b, h], causal) for b in range(B) for h in range(he)]
        at = 0
        for i in range(len(rows[0])):
            want = np.concatenate([r[i] for r in rows])
            assert np.array_equal(plan[at:at + len(want)], want), i
            at += len(want) if i < 2 else -(-len(want) // 128) * 128
        assert not plan[at:at + 128].any() and len(plan) == at + 128 and int(status) == 0


def test_ids_below_int32():
    from flash_b200 import ops
    for N in (200, 16500):
        ids = torch.full((1, 1, N), -3, dtype=torch.int64, device="cuda")
        ids[0, 0, N - 1] = LOWEST - 1
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        prob = ops._problem(1, 1, 1, N, N, 64, torch.bfloat16, False, 1, 1, 1.0)
        plan = ops.build_plan(prob, ids, ids, status)
        assert int(status) == 200 and int(plan[N - 1]) == LOWEST
