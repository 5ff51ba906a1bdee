"""The packed division of the step kernels (div2, csrc/tws_pair.cuh) against the
correctly rounded quotient, over the range that the kernels use it in: d from 2^-100,
t up to 2^20, d < t.  (A quotient of two floats rounded to 53 bits and then to 24
is correctly rounded: 53 >= 2 * 24 + 2.)"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

N = 1 << 24
LO, HI = -100, 20  # exponents of the least d and the largest t


@pytest.fixture(scope="module")
def env():
    import torch
    import terrainwatersim_gb300 as t
    t.lib()
    return torch, t


def check(env, d, t):
    torch, tws = env
    ok = (d >= 2.0 ** LO) & (t <= 2.0 ** HI) & (d < t)
    d, t = d[ok], t[ok]
    n = d.numel() // 2 * 2
    assert n > N // 4
    d, t = d[:n].contiguous(), t[:n].contiguous()
    q = torch.empty_like(d)
    s = torch.cuda.current_stream().cuda_stream
    assert tws.lib().tws_test_divide(d.data_ptr(), t.data_ptr(), q.data_ptr(), n, s) == 0
    want = (d.double() / t.double()).float()
    bad = q.view(torch.int32) != want.view(torch.int32)
    assert not bool(bad.any()), (int(bad.sum()), d[bad][:4].tolist(), t[bad][:4].tolist())


def mantissas(torch, gen, n=N):
    """1 <= m < 2, a fifth of them near the ends and of few bits."""
    m = torch.randint(0, 1 << 23, (n,), generator=gen, device="cuda", dtype=torch.int32)
    k = n // 10
    m[:k] = (1 << 23) - 1 - m[:k] % 64
    m[k:2 * k] = m[k:2 * k] % 64
    p = torch.randperm(n, generator=gen, device="cuda")
    return ((m | (127 << 23)).view(torch.float32))[p]


def scaled(torch, m, e):
    return torch.ldexp(m.double(), e).float()  # (exact: all in the normal range)


def exponents(torch, gen, lo, hi, n=N):
    return torch.randint(lo, hi + 1, (n,), generator=gen, device="cuda")


@pytest.mark.parametrize("seed", range(8))
def test_random_pairs(env, seed):
    """Exponents anywhere in the range, and, as depths and outflows are, close ones."""
    torch, _ = env
    gen = torch.Generator("cuda").manual_seed(seed)
    t = scaled(torch, mantissas(torch, gen), exponents(torch, gen, LO, HI))
    if seed % 2:
        d = scaled(torch, mantissas(torch, gen), exponents(torch, gen, LO, HI))
        d, t = torch.minimum(d, t), torch.maximum(d, t)
    else:
        d = t * (mantissas(torch, gen) - 1.0)
    check(env, d, t)


def test_limits_of_the_range(env):
    torch, _ = env
    gen = torch.Generator("cuda").manual_seed(100)
    t = scaled(torch, mantissas(torch, gen), exponents(torch, gen, LO, HI))
    check(env, torch.full_like(t, 2.0 ** LO), t)
    d = scaled(torch, mantissas(torch, gen), exponents(torch, gen, LO, HI))
    check(env, d, torch.full_like(d, 2.0 ** HI))
    for ulps in (1, 2, 3):  # quotients just below 1
        check(env, (t.view(torch.int32) - ulps).view(torch.float32), t)


@pytest.mark.parametrize("seed", range(4))
def test_closest_to_a_rounding_boundary(env, seed):
    """Pairs whose quotient lies as near the middle of two floats as d's own last
    place allows: d = t * (q + half an ulp), rounded down and up."""
    torch, _ = env
    gen = torch.Generator("cuda").manual_seed(200 + seed)
    t = scaled(torch, mantissas(torch, gen), exponents(torch, gen, -70, HI))
    e = exponents(torch, gen, -30, -1)
    q = scaled(torch, mantissas(torch, gen), e).double()
    half = torch.ldexp(torch.ones_like(q), e - 24)
    for mid in (q + half, q - half):
        d = (mid * t.double()).float()  # (the product is exact in 53 bits)
        i = d.view(torch.int32)
        for step in (-1, 0, 1):
            check(env, (i + step).view(torch.float32), t)
