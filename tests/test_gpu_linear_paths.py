"""Branches of the fused linear: raw units between coded ones (their bytes start on any 16-bit
word), shapes with and without room for the fraction rings beside the operand tiles, and calls
back to back on one workspace (the launches overlap)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests import nzabi as A

pytestmark = pytest.mark.gpu


def reference(w, x):
    return (x.double() @ w.double().t()).cpu()


def check(y, ref):
    # fp32 sums rounded once to bf16: half a unit in the last place (2^-9 of the value) and the
    # fp32 accumulation, bounded by the largest result
    err = (y.double().cpu() - ref).abs()
    assert bool((err <= 2.0 ** -8 * ref.abs() + 2.0 ** -14 * ref.abs().max()).all())


@pytest.mark.parametrize("s", (7, 3, 1, 0))
def test_raw_units_between_coded_ones(s):
    # the identity as input: every weight reaches one result, alone, so each has to be exact
    rows, cols, S = 132, 1024, 64
    g = torch.Generator().manual_seed(s)
    w = (torch.randn(rows, cols, generator=g) * 0.02).to(torch.bfloat16)
    bits = A.to_bits(w).reshape(rows, cols).copy()
    rng = np.random.default_rng(3)
    for row in range(0, rows, 12):                   # row groups whose exponents do not compress
        bits[row:row + 4, :512] = ((rng.integers(1, 250, (4, 512)) << 7) | (bits[row:row + 4, :512] & 0x807F))
    cont, frac, mw = A.compress_operand(A.from_bits(bits.reshape(-1)), rows, cols, s, S)
    offs = np.frombuffer(cont.cpu().numpy().tobytes(), dtype=np.uint32, count=rows // 4 * 2 + 1, offset=576)
    raw = offs[:-1] >> 31 == 1
    assert list(np.flatnonzero(raw)) == list(range(0, rows // 2, 6))
    assert (offs[:-1][raw] & 1).any() and not (offs[:-1][raw] & 1).all()      # at odd and even words
    c_ref, f_ref = O.compress_bf16(O.to_operand_order(bits.reshape(-1), rows, cols), s, S)
    stored = O.from_operand_order(O.decompress_bf16(c_ref, f_ref, bits.size, s), rows, cols)
    y, status = A.linear(cont, frac, rows, cols, s, S, torch.eye(cols, dtype=torch.bfloat16, device="cuda"),
                         max_words=mw)
    assert status == 0
    assert torch.equal(y.cpu().t(), A.from_bits(stored, "cpu").view(rows, cols))


@pytest.mark.parametrize("m", (1, 17, 256))
@pytest.mark.parametrize("cols,S", ((2048, 128), (11008, 344), (4096, 256)))
@pytest.mark.parametrize("nan", (False, True))
def test_with_and_without_room_for_the_rings(cols, S, m, nan):
    rows = 260
    g = torch.Generator().manual_seed(cols + m)
    w = (torch.randn(rows, cols, generator=g) * 0.02).to(torch.bfloat16).cuda()
    if nan:
        w[7, 5] = float("nan")           # its row is NaN, the others take the loop that looks for it
    x = torch.randn(m, cols, generator=g).to(torch.bfloat16).cuda()
    for s in (7, 3, 1, 0):
        cont, frac, mw = A.compress_operand(w, rows, cols, s, S)
        stored = A.decompress_operand(cont, frac, rows, cols, s, S)[0].view(rows, cols)
        if S == 344 and m == 256:
            continue                              # units too long beside this many input rows
        ys = []
        for _ in range(3):
            y, status = A.linear(cont, frac, rows, cols, s, S, x, max_words=mw, canon=nan)
            assert status == 0
            ys.append(y)
        lost = stored.isnan().any(1).cpu()            # (precision 0 rounds the NaN away)
        check(ys[0].cpu()[:, ~lost], reference(stored.cpu(), x.cpu())[:, ~lost])
        assert bool(ys[0].cpu()[:, lost].isnan().all()) and bool(lost.any()) == (nan and s > 0)
        assert all(torch.equal(ys[0].view(torch.int16), y.view(torch.int16)) for y in ys)
