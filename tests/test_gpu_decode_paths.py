"""Edges of the decode kernel's work split and of its choice of table layout: unit counts
around one and two chains, ragged last units, block counts that are and are not multiples of
the fraction ring, runs of many units per warp, and tables that do and do not take the
narrow entries (frequencies up to 512, usual resolution, no NaN to rewrite).  Everything is
compared with the oracle bit for bit."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests import nzabi as A

pytestmark = pytest.mark.gpu


def values(n, kind, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(n, generator=g, dtype=torch.float32) * 0.02
    if kind == "peaked":          # one exponent for 4 elements of 5: its frequency is above 512
        x = torch.where(torch.rand(n, generator=g) < 0.8, x.sign() * 0.75, x)
    x = x.to(torch.bfloat16)
    if kind == "nan" and n:
        x[torch.randint(0, n, (1 + n // 100,), generator=g)] = float("nan")
    return x


def check(n, s, S, kind, seed):
    x = values(n, kind, seed)
    bits = A.to_bits(x)
    cont, frac = O.compress_bf16(bits, s, S)
    want = O.decompress_bf16(cont, frac, n, s, canonical_nan=True)
    out, status = A.decompress(A.dev_u8(cont), A.dev_u8(frac), n, s, S, canon=True)
    assert status == 0 and np.array_equal(A.to_bits(out), want), (n, s, S, kind)


@pytest.mark.parametrize("s", (7, 3, 1, 0))
@pytest.mark.parametrize("S", (8, 24, 40, 128, 200, 344, 512))
def test_unit_counts_and_ragged_tails(s, S):
    U = 32 * S
    for k in (0, 1, 2, 3):
        for tail in (0, 1, 255, 256, 300, U - 1):
            if 0 < k * U + tail and tail < U:
                check(k * U + tail, s, S, "normal", 100 * S + 10 * k + tail % 7)


@pytest.mark.parametrize("s", (7, 3, 1, 0))
@pytest.mark.parametrize("kind", ("normal", "peaked", "nan"))
def test_table_layouts(s, kind):
    for S in (64, 256):
        check(32 * S * 301 + 777, s, S, kind, 5 + S)


@pytest.mark.parametrize("s", (7, 0))
def test_runs_of_many_units_per_warp(s):
    # more than 32 units per warp at 148 CTAs of 20 warps
    check(256 * 148 * 20 * 34 + 100, s, 8, "normal", 9)


@pytest.mark.parametrize("s,group", ((7, 2), (3, 512), (1, 8), (0, 512), (0, 4)))
def test_normalised_tensors_equal_decode_and_stand_alone_scaling(s, group):
    from neuzip_b200 import _lib
    from neuzip_b200.backend import _cuda
    for n in (300, 32 * 512 * 3, 32 * 512 * 4 + 5001):
        x = values(n, "normal", 31 + n).cuda()
        be = getattr(_cuda, f"Manager_f{s}_n{group}")()
        be.write("w", x)
        e = be.entry("w")
        out, status = A.decompress(e.container, e.fractions, n, s, e.lane_symbols, canon=True)
        assert status == 0
        plain = torch.empty(n + 8, dtype=torch.bfloat16, device="cuda")[:n]
        plain.copy_(out)
        _lib.check(A.lib().nz_denormalize_bf16(plain.data_ptr(), n, group, e.normalizers.data_ptr(),
                                               A.stream()))
        got = be.read("w")
        be.check()
        assert torch.equal(got.view(torch.int16), plain.view(torch.int16)), (s, group, n)
