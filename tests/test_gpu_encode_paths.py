"""Branches of the fused encoder, each against the oracle byte for byte: a symbol with more
than half of the slots (the remainder is checked), units above 3 bits per symbol (squeezed in
place), lanes that outgrow their slice (the unit is coded a second time), units stored raw, length
quanta of two words, ragged last units (whole blocks, the block that ends the tensor, blocks of
nothing but padding), and tensors whose units do not fill the GPU evenly."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests import nzabi as A

pytestmark = pytest.mark.gpu


def bits_of(kind, n, seed):
    rng = np.random.default_rng(seed)
    sign_mantissa = rng.integers(0, 256, n).astype(np.uint16)
    if kind == "peaked":
        exp = np.where(rng.random(n) < 0.9, 120, rng.integers(110, 125, n))
    elif kind == "single":
        exp = np.full(n, 121)
    elif kind == "uniform10":                      # 3.3 bits per symbol
        exp = rng.integers(115, 125, n)
    elif kind == "raw":                            # runs of 2048 that do not compress, among others
        exp = np.where(np.arange(n) // 2048 % 3 == 1, rng.integers(1, 255, n), rng.integers(118, 122, n))
    elif kind == "uniform60":                      # 5.9 bits: every lane outgrows its slice
        exp = rng.integers(80, 140, n)
    else:                                          # one lane of 32 has the rare exponents
        lane = (np.arange(n) // 8) % 32
        exp = np.where(lane == 5, rng.integers(60, 180, n), np.where(rng.random(n) < 0.9, 120, 119))
    exp = exp.astype(np.uint16)
    return ((sign_mantissa & 0x80) << 8) | (exp << 7) | (sign_mantissa & 0x7F)


@pytest.mark.parametrize("s", (7, 3, 1, 0))
@pytest.mark.parametrize("kind", ("peaked", "single", "uniform10", "uniform60", "lane"))
def test_encoder_branches(s, kind):
    for S in (8, 64, 256, 776, 1024):
        for n in (1, 32 * S, 32 * S * 5 + 3, 32 * S * 9 + 261):
            bits = bits_of(kind, n, 7 * S + n % 11)
            cont, frac, _ = A.compress(A.from_bits(bits), s, S)
            c_ref, f_ref = O.compress_bf16(bits, s, S)
            assert np.array_equal(cont.cpu().numpy(), c_ref), (s, kind, S, n)
            assert np.array_equal(frac.cpu().numpy(), f_ref), (s, kind, S, n)


def check(bits, s, S):
    cont, frac, _ = A.compress(A.from_bits(bits), s, S)
    c_ref, f_ref = O.compress_bf16(bits, s, S)
    assert np.array_equal(cont.cpu().numpy(), c_ref), (s, S, bits.size)
    assert np.array_equal(frac.cpu().numpy(), f_ref), (s, S, bits.size)
    return c_ref


@pytest.mark.parametrize("s", (7, 3, 1, 0))
@pytest.mark.parametrize("kind", ("peaked", "uniform10", "uniform60", "raw"))
def test_ragged_last_units(s, kind):
    # the last unit's count around every edge of its three parts, alone and behind whole units
    for S in (8, 64, 384):
        U = 32 * S
        for count in {1, 7, 8, 255, 256, 257, 511, 512, U // 2 + 3, U - 257, U - 256, U - 255, U - 1}:
            for units in (0, 3):
                if 0 < count < U:
                    check(bits_of(kind, units * U + count, S + count), s, S)


@pytest.mark.parametrize("s", (7, 3, 1, 0))
def test_raw_units(s):
    for S in (8, 64):
        for n in (2048 * 9, 2048 * 4 + 1, 2048 * 4 + 7, 2048 * 4 + 2043):
            cont = check(bits_of("raw", n, S + n), s, S)
            units = -(-n // (32 * S))
            offs = np.frombuffer(cont.tobytes(), dtype=np.uint32, count=units, offset=576)
            assert (offs >> 31).any() and not (offs >> 31).all()


@pytest.mark.parametrize("s", (7, 1))
def test_raw_units_in_operand_order(s):
    rows, cols, S = 64, 512, 64
    bits = bits_of("raw", rows * cols, 5)
    cont, frac, _ = A.compress_operand(A.from_bits(bits), rows, cols, s, S)
    c_ref, f_ref = O.compress_bf16(O.to_operand_order(bits, rows, cols), s, S)
    assert np.array_equal(cont.cpu().numpy(), c_ref) and np.array_equal(frac.cpu().numpy(), f_ref)
    assert (np.frombuffer(c_ref.tobytes(), dtype=np.uint32, count=16, offset=576) >> 31).any()


@pytest.mark.parametrize("units", (147, 148, 149, 148 * 8, 148 * 8 + 1, 148 * 9, 148 * 16 + 1, 148 * 33))
def test_split_over_the_sms(units):
    # a unit per warp on every SM, several blocks per SM, and more units than warps
    check(bits_of("peaked", 256 * units - 5, 11), 7, 8)


@pytest.mark.parametrize("S", (512, 640, 768, 1024))
def test_long_units_beyond_one_wave(S):
    check(bits_of("uniform10", 32 * S * (148 * 8 + 3) - 77, 12), 1, S)


@pytest.mark.parametrize("units", (255, 256, 257, 148 * 48 * 3 + 4, 131071, 131072, 131072 + 300))
def test_many_units(units):
    # chunks of one and more units, several units per warp; from 131072 units on the offsets, the
    # raw count and the largest unit come from the scan kernel
    n = 256 * units - 23
    bits = bits_of("peaked", n, 3)
    raw = np.random.default_rng(4).integers(0, 256, 256 * 70).astype(np.uint16)
    for first in (0, 100, units // 2, units - 80):          # some units that do not compress
        bits[256 * first:256 * (first + 70)] = (raw << 7)[:max(0, n - 256 * first)]
    cont = check(bits, 7, 8)
    offs = np.frombuffer(cont.tobytes(), dtype=np.uint32, count=units, offset=576)
    assert (offs >> 31).any() and not (offs >> 31).all()
