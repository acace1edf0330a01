"""Split TSMTTSM: columns whose exponents rise long after a CTA's first rows.  The elements jump by more bits than a raise
grants as headroom, in staggered columns, at points placed by the CTAs' own shares of the rows, some in every stage (round)
one after the other, some after long quiet stretches; every CTA has many stages and full periods.

Widths above 16 (jumps of 6 bits; a raise grants 4): more than 32 stages a CTA in each compiled variant.
Widths up to 16 (jumps of 5 bits; a raise grants 2): 20 periods a CTA, so that the sums of digit pairs leave for
the accumulators for either reason: exponents that changed, and the 15 periods that 32 bits hold.

The entries are integers of at most 8 bits times the jumps: every digit product that the scheme drops is zero, every sum is
below 2^53, so the results are exact.  That the raises occur is checked on the data."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def operand(g, pos, cols, jump, at, bits):
    """Integers of `bits` bits; column c jumps by `jump` bits at each position of at(c) (positions within a CTA's share)."""
    lim = 1 << bits
    x = torch.randint(-lim + 1, lim, (pos.numel(), cols), generator=g, device="cuda", dtype=torch.int64)
    for c in range(cols):
        for p in at(c):
            x[:, c] <<= jump * (pos >= p).to(torch.int64)
    return x


def raises(x, unit, pos, head):
    """Stages (rounds) of x's CTAs, other than their first, in which a column exceeds its exponent: [stage] bool."""
    n = x.shape[0] // unit
    e = torch.frexp(x[: n * unit].abs().to(torch.float64).view(n, unit, -1).amax(dim=1))[1].cpu().numpy()
    first = pos[: n * unit : unit].cpu().numpy() == 0
    out, cur = np.zeros(n, dtype=bool), np.zeros(x.shape[1], dtype=int)
    for s in range(n):
        if first[s]:
            cur[:] = 0
        over = e[s] > cur
        out[s] = over.any() and not first[s]
        cur = np.where(over, e[s] + head, cur)
    return out


def shares(units, ctas, K, unit):
    """Position (in units) within its CTA's share of every row, and the shares."""
    b = units * np.arange(ctas + 1) // ctas
    pos = np.concatenate([np.arange(b[i + 1] - b[i]) for i in range(ctas)])
    return torch.from_numpy(np.repeat(pos, unit)[:K]).cuda(), np.diff(b)


def product(handle, A, B, gram, dt, sa, sb):
    exp = (B.to(torch.float64).T @ A.to(torch.float64))
    assert float(exp.abs().max()) < 2.0**53
    Ad = torch.ldexp(A.to(torch.float64), torch.tensor(sa, device="cuda")) if sa > -1000 else \
        torch.from_numpy(np.ldexp(A.cpu().numpy().astype(np.float64), sa)).cuda()
    Bd = torch.ldexp(B.to(torch.float64), torch.tensor(sb, device="cuda"))
    Ad = Ad.to(dt)
    Bd = Ad if gram else Bd.to(dt)
    C = torch.full((B.shape[1], A.shape[1]), float("nan"), dtype=dt, device="cuda")
    handle.tsmttsm(A.shape[1], B.shape[1], A.shape[0], Ad, A.shape[1], 1.0, Bd, B.shape[1], 0.0, C, A.shape[1], acc="split")
    handle.check_device()
    want = np.ldexp(exp.cpu().numpy(), sa + sb)
    assert np.array_equal(C.cpu().numpy(), want.astype(np.float32 if dt == torch.float32 else np.float64))


@pytest.mark.parametrize("dt,sa,sb", [("float64", 0, 0), ("float64", -1070, 900), ("float32", 0, 0)])
@pytest.mark.parametrize("M,N,gram", [(32, 32, False), (17, 9, False), (32, 32, True), (64, 64, False), (40, 64, True),
                                      (64, 64, True), (100, 70, False), (100, 100, True)])
def test_wide(handle, dt, sa, sb, M, N, gram):
    N = M if gram else N
    if gram and sa:
        pytest.skip("squares leave the range")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    unit = 32 if max(M, N) <= 32 else 16
    bm, bn = (M + 63) // 64, (N + 63) // 64
    ctas = sms // (bm * (bm + 1) // 2 if gram else bm * bn)
    units = ctas * 41 + 7
    K = units * unit - 5
    pos, share = shares(units, ctas, K, unit)
    assert share.min() > 32
    g = torch.Generator(device="cuda").manual_seed(M + N)
    # by column: at once in consecutive stages, spread, late, or never
    at = [lambda c: (1, 2, 3), lambda c: (3 + c % 7, 12 + c % 9, 29 + c % 5), lambda c: (35 + c % 6,), lambda c: ()]
    A = operand(g, pos, M, 5 if gram else 6, lambda c: at[c % 4](c)[: 2 if gram else 3], 4 if gram else 8)
    B = A if gram else operand(g, pos, N, 6, lambda c: at[(c + 2) % 4](c)[:1], 6)
    late = raises(torch.cat([A, B], dim=1), unit, pos, 4)
    assert late.sum() >= 8 * ctas and late.sum() <= 32 * ctas  # many, with whole periods between them
    product(handle, A, B, gram, getattr(torch, dt), sa, sb)


@pytest.mark.parametrize("dt", ["float64", "float32"])
@pytest.mark.parametrize("M,N,gram,rr", [(8, 8, False, 256), (16, 16, False, 128), (16, 16, True, 256), (5, 13, False, 128)])
def test_narrow(handle, dt, M, N, gram, rr):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per = 1024 // rr  # rounds of a full period
    rounds = sms * (20 * per + 3) + 11
    K = rounds * rr - 9
    pos, share = shares(rounds, sms, K, rr)
    g = torch.Generator(device="cuda").manual_seed(M + N)
    # in consecutive rounds; in the second and third period; after a quiet stretch of more than 16 periods; never
    at = [lambda c: (1, 2), lambda c: (per + c % per, 2 * per + 1), lambda c: (19 * per + c % 2,), lambda c: ()]
    A = operand(g, pos, M, 5, lambda c: at[c % 4](c), 4 if gram else 8)
    B = A if gram else operand(g, pos, N, 5, lambda c: at[(c + 1) % 4](c)[:1], 6)
    late = raises(torch.cat([A, B], dim=1), rr, pos, 2)
    start = np.flatnonzero(pos[::rr].cpu().numpy()[: late.size] == 0)
    for b, e in zip(start, np.append(start[1:], late.size)):
        r = np.flatnonzero(late[b:e])
        if e - b >= share.min():
            assert r.size >= 4 and r.max() >= 19 * per  # changes, the last one late,
            assert np.diff(r).max() > 16 * per  # and more periods between two than are summed at a time
    product(handle, A, B, gram, getattr(torch, dt), 0, 0)
