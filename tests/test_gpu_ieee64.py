"""The FP64 passes' square root, reciprocals and quotients (csrc/ieee64.cuh) against the operators, bit for bit: on
random operands over the passes' ranges, on mantissas near 1 and near 2, and on the operands whose results lie
nearest to a midpoint of two doubles."""

from __future__ import annotations

import math
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOP, UNIT = 1 << 53, 1 << 52  # an integer mantissa lies in [UNIT, TOP)


def square_root_mod(c, bits):
    """r with r^2 = c mod 2^bits, for c = 1 mod 8 (bit by bit)."""
    r = 1
    for k in range(3, bits):
        if (r * r - c) >> k & 1:
            r += 1 << (k - 1)
    assert (r * r - c) % (1 << bits) == 0
    return r


def hard_square_roots(reach=513):
    """Integer mantissas X and shifts s whose root sqrt(X 2^s) is next to a midpoint M (odd, 54 bits):
    X 2^s = M^2 + k, |k| <= reach."""
    out = []
    for k in range(-reach, reach + 1):
        if k % 8 != 7:
            continue
        for s in (54, 55):
            r = square_root_mod(-k % (1 << s), s)
            roots = {sign * r + half for sign in (1, -1) for half in (0, 1 << (s - 1))}
            for M in {m % (1 << s) + turn * (1 << s) for m in roots for turn in (0, 1)}:
                X = (M * M + k) >> s
                if TOP <= M < 2 * TOP and UNIT <= X < TOP:
                    assert X << s == M * M + k
                    out.append((X, s))
    return out


def hard_quotients(count, rng):
    """Mantissas (A, B) with A 2^54 = Q B + k, Q odd of 54 bits and k small: A / B is next to the midpoint Q 2^-54."""
    out = []
    for B in rng.integers(UNIT // 2, TOP // 2, count):
        B = 2 * int(B) + 1
        inv = pow(B, -1, 1 << 54)
        for k in (-3, -2, -1, 1, 2, 3):
            Q = -k * inv % (1 << 54)
            A = (Q * B + k) >> 54
            for a in (A, 2 * A):  # the quotient's mantissa below and above the numerator's
                if Q >= TOP and UNIT <= a < TOP:
                    out.append((a, B))
    return out


@pytest.fixture(scope="module")
def check():
    import torch

    from dem import _native as N

    ctx = N.Context(1)

    def run(a, b):
        """Number of operands; asserts the four results."""
        a, b = a.contiguous(), b.contiguous()
        ones = 0xFFFFFFFF
        root = a.sqrt()
        ok_root = (root.view(torch.int64) & ones) != ones  # a low word of ones goes to the operators
        ok_b = (b.view(torch.int64) & ones) != ones
        out = torch.empty((4, a.numel()), dtype=torch.float64, device=a.device)
        ctx.ieee64_probe(a, b, out)
        assert torch.equal(out[0], root)
        assert torch.equal(out[1][ok_root], 1 / root[ok_root])
        assert torch.equal(out[2][ok_b], 1 / b[ok_b])
        assert torch.equal(out[3][ok_b], a[ok_b] / b[ok_b])
        return a.numel()

    return run


def _doubles(torch, mantissa, exponent):
    """Doubles of 52-bit fractions and exponents (int64 tensors)."""
    return (mantissa | (exponent + 1023) << 52).view(torch.float64)


def test_operators_round_to_nearest():
    # the operators the others are compared with, against exact integers
    import torch

    rng = np.random.default_rng(5)
    a, b = rng.uniform(1, 4, 2000), rng.uniform(1, 2, 2000)
    root = torch.as_tensor(a, device="cuda").sqrt().cpu().numpy()
    quot = (torch.as_tensor(a, device="cuda") / torch.as_tensor(b, device="cuda")).cpu().numpy()
    for x, g, y, q in zip(a.tolist(), root.tolist(), b.tolist(), quot.tolist()):
        half = Fraction(math.ulp(g)) / 2
        assert (Fraction(g) - half) ** 2 <= Fraction(x) <= (Fraction(g) + half) ** 2
        assert abs(Fraction(x) / Fraction(y) - Fraction(q)) <= Fraction(math.ulp(q)) / 2


# root: 2^-200 <= r^2 < 2^200; divisors: r^3 and r^7 of such; numerators: zero or products of two differences
@pytest.mark.parametrize("ea, eb", [((-200, 200), (-300, 300)), ((-200, 200), (-120, 120)), ((0, 2), (0, 1))])
def test_random(check, ea, eb):
    import torch

    g = torch.Generator("cuda").manual_seed(ea[1] + eb[1])
    kw = dict(device="cuda", generator=g)
    n, total = 1 << 24, 0
    for _ in range(16):
        m = [torch.randint(0, 1 << 52, (n,), **kw) for _ in range(2)]
        total += check(_doubles(torch, m[0], torch.randint(*ea, (n,), **kw)),
                       _doubles(torch, m[1], torch.randint(*eb, (n,), **kw)))
    assert total == 16 << 24


@pytest.mark.parametrize("near_a", ["1", "2"])
@pytest.mark.parametrize("near_b", ["1", "2"])
def test_near_the_ends_of_a_binade(check, near_a, near_b):
    import torch

    k = torch.arange(2048, device="cuda")
    one = {"1": k, "2": (1 << 52) - 1 - k}
    a, b = torch.meshgrid(one[near_a], one[near_b], indexing="ij")
    for e in (0, 1):  # either parity under the root
        check(_doubles(torch, a.reshape(-1), torch.full((), e, device="cuda")),
              _doubles(torch, b.reshape(-1), torch.zeros((), dtype=torch.int64, device="cuda")))


def test_hard_square_roots(check):
    import torch

    hard = hard_square_roots()
    assert len(hard) > 150
    for scale in range(-200, 198, 2):
        x = [math.ldexp(X, s - 106 + scale) for X, s in hard]
        x = torch.tensor([v for v in x if 2.0**-200 <= v < 2.0**200], dtype=torch.float64, device="cuda")
        check(x, torch.ones_like(x))


def test_hard_quotients(check):
    import torch

    hard = np.array(hard_quotients(100000, np.random.default_rng(3)), dtype=np.int64)
    assert len(hard) > 100000
    a, b = (torch.as_tensor(hard[:, c].astype(np.float64), device="cuda") for c in range(2))
    check(a, b)
    check(a * 2.0**-300, b * 2.0**-250)


def test_divisors_next_to_a_midpoint(check):
    """Quotients whose first approximation is 1.5 ulp off and whose divisor's reciprocal is next to a midpoint."""
    import torch

    k = torch.arange(1, 4097, device="cuda")
    a = 2 - k.to(torch.float64) * 2.0**-52
    near = [((1 << 53) - (1 << 27) + 1) * 2.0**-52, 1 - 3 * 2.0**-53, 1 - 5 * 2.0**-53]
    assert (2**106 + 1) % int(near[0] * 2**52) == 0
    for b in near:
        check(a, torch.full_like(a, b))
