"""Edges of the decode kernel's work split and of its choice of table layout: unit counts
around one and two chains, ragged last units, block counts that are and are not multiples of
the fraction ring, runs of many units per warp, and tables that do and do not take the
narrow entries (frequencies up to 512, usual resolution, no NaN to rewrite), tables with one or
two copies, raw units.  Everything is compared with the oracle bit for bit."""
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
    if kind in ("raw", "raw nan") and n:       # runs of 4096 whose exponents do not compress
        noise = torch.randint(1, 255, (n,), generator=g).to(torch.int32) << 23
        x = torch.where(torch.arange(n) // 4096 % 3 == 1, noise.view(torch.float32) * x.sign(), x)
    if kind == "inf" and n:
        x[torch.randint(0, n, (1 + n // 100,), generator=g)] = float("inf")
    if kind == "wide11" and n:                 # 33 to 64 exponents: 11 bits
        x = torch.exp2(torch.randint(-30, 20, (n,), generator=g).float()) * x.sign()
    if kind == "wide12" and n:                 # more, none of them with half of the slots: 12 bits
        e = torch.where(torch.rand(n, generator=g) < 0.02, torch.randint(-60, 60, (n,), generator=g),
                        torch.randint(-8, 0, (n,), generator=g))
        x = torch.exp2(e.float()) * x.sign()
    x = x.to(torch.bfloat16)
    if kind in ("nan", "raw nan") and n:
        x[torch.randint(0, n, (1 + n // 100,), generator=g)] = float("nan")
    return x


def check(n, s, S, kind, seed):
    x = values(n, kind, seed)
    bits = A.to_bits(x)
    cont, frac = O.compress_bf16(bits, s, S)
    want = O.decompress_bf16(cont, frac, n, s, canonical_nan=True)
    out, status = A.decompress(A.dev_u8(cont), A.dev_u8(frac), n, s, S, canon=True)
    assert status == 0 and np.array_equal(A.to_bits(out), want), (n, s, S, kind)
    return cont


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


@pytest.mark.parametrize("s", (7, 3, 1, 0))
@pytest.mark.parametrize("kind", ("raw", "raw nan"))
def test_raw_units(s, kind):
    for S in (8, 64, 128):
        for n in (4096 * 9, 4096 * 4 + 1, 4096 * 5 + 255, 4096 * 4 + 300, 4096 * 151 + 777):
            cont = check(n, s, S, kind, S + n)
            offs = np.frombuffer(cont.tobytes(), dtype=np.uint32, count=-(-n // (32 * S)), offset=576)
            assert (offs >> 31).any() and not (offs >> 31).all()


@pytest.mark.parametrize("s", (7, 1))
def test_raw_units_in_operand_order(s):
    rows, cols, S = 64, 512, 64
    bits = A.to_bits(values(rows * cols, "raw", 5))
    cont, frac = O.compress_bf16(O.to_operand_order(bits, rows, cols), s, S)
    assert (np.frombuffer(cont.tobytes(), dtype=np.uint32, count=16, offset=576) >> 31).any()
    want = O.from_operand_order(O.decompress_bf16(cont, frac, bits.size, s, canonical_nan=True), rows, cols)
    out, status = A.decompress_operand(A.dev_u8(cont), A.dev_u8(frac), rows, cols, s, S, canon=True)
    assert status == 0 and np.array_equal(A.to_bits(out), want)


def test_raw_units_of_an_exponent_stream():
    rng = np.random.default_rng(6)
    for n in (2048 * 9, 2048 * 4 + 301):
        e = np.where(np.arange(n) // 2048 % 3 == 1, rng.integers(0, 256, n), rng.integers(118, 122, n)).astype(np.uint8)
        cont, words = A.encode(A.dev_u8(e), 64)
        got, status = A.decode_exponents(cont, n, 64, words)
        assert status == 0 and np.array_equal(got.cpu().numpy(), e)


@pytest.mark.parametrize("kind,bits", (("wide11", 11), ("wide12", 12)))
def test_tables_with_one_and_two_copies(kind, bits):
    # 22 units of 256 symbols per CTA of unknown length: the smallest table leaves room for
    # eleven warps and one round, every larger one takes two
    n = 148 * 21 * 8192 + 8192 * 3 + 5
    cont = check(n, 7, 256, kind, bits)
    assert int(np.frombuffer(cont.tobytes(), dtype=np.uint32, count=1, offset=28)[0]) == bits


@pytest.mark.parametrize("kind", ("normal", "nan", "inf", "raw"))
@pytest.mark.parametrize("s,group", ((7, 2), (3, 512), (1, 8), (0, 512), (0, 4)))
def test_normalised_tensors_equal_decode_and_stand_alone_scaling(s, group, kind):
    from neuzip_b200 import _lib
    from neuzip_b200.backend import _cuda
    for n in (300, 32 * 512 * 3, 32 * 512 * 4 + 5001):
        x = values(n, kind, 31 + n).cuda()
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
