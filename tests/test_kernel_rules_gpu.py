"""Kernels that have several forms chosen by size: at the edges of the rules that choose, and beside them, every form
gives the row the same bits, and the values of the plain float64 reference within a bound from the sums' lengths."""

from __future__ import annotations

import math

import pytest
import torch

from plain import qwen3_plain as plain

pytestmark = pytest.mark.gpu


def K():
    from lockstep_b200 import kernels

    return kernels


def dev():
    return torch.device("cuda:0")


# ---------------------------------------------------------------------------
# sampler: a row over 8, 4, 2 or 1 blocks
# ---------------------------------------------------------------------------

def _draw(k, logits, temperature, top_p, uids, positions, seed=11):
    from lockstep_b200.sampling import philox

    as_i32 = lambda t: t.where(t < 2 ** 31, t - 2 ** 32).to(torch.int32).to(dev())
    keys = torch.tensor([philox.key_words(seed, u) for u in uids], dtype=torch.int64)
    pos = torch.tensor([[p, 0] for p in positions], dtype=torch.int64)
    out = torch.full((len(uids),), -7, dtype=torch.int32, device=dev())
    k.sample(logits.to(dev()), None, temperature.to(dev()), top_p.to(dev()), as_i32(keys), as_i32(pos), out)
    return out.tolist()


@pytest.mark.parametrize("vocab", [3, 777, 49152, 49153, 98305, 163840])
def test_a_sampled_token_does_not_depend_on_how_many_rows_there_are(vocab):
    """1, 18, 19, 37, 74 and 149 rows: every spread that holds the vocabulary; the plain sampler for the first rows."""
    k = K()
    g = torch.Generator().manual_seed(vocab)
    base = torch.randn(6, vocab, generator=g) * 2.5
    base[1] = torch.randint(0, 4, (vocab,), generator=g).float()             # ties everywhere
    base[2, :-1] = -math.inf                                                 # one token has all the mass
    temperature = torch.tensor([0.8, 1.0, 0.7, 0.0, 1.3, 0.9])
    top_p = torch.tensor([0.9, 0.5, 0.9, 1.0, 1.0, 0.05])
    uids, positions = [f"u{i}" for i in range(6)], [3 + 7 * i for i in range(6)]
    first = [_draw(k, base[i:i + 1], temperature[i:i + 1], top_p[i:i + 1], uids[i:i + 1], positions[i:i + 1])[0] for i in range(6)]
    assert first[2] == vocab - 1 and first[3] == int(base[3].argmax())
    for rows in (18, 19, 37, 74, 149):
        pick = [i % 6 for i in range(rows)]
        got = _draw(k, base[pick], temperature[pick], top_p[pick], [uids[i] for i in pick], [positions[i] for i in pick])
        assert got == [first[i] for i in pick], rows
    for i in range(6):
        want = plain.sample_top_p(base[i], 11, uids[i], positions[i], p=float(top_p[i]), temperature=float(temperature[i]))
        # float32 exponentials: a draw within rounding of a boundary may land on the neighbouring rank
        assert want == first[i] or abs(float(base[i, want]) - float(base[i, first[i]])) < 1e-3


def test_rows_that_are_no_distribution_give_token_0_or_the_numbers_in_them():
    k = K()
    vocab = 1000
    logits = torch.zeros(5, vocab)
    logits[0, 500] = math.nan
    logits[1] = math.nan
    logits[2, 30] = math.inf
    logits[3] = -math.inf
    logits[4] = -math.inf
    logits[4, [7, 8]] = -3e38                                                # far below zero, and still the only mass
    one = torch.full((5,), 0.5)
    got = _draw(k, logits, one, torch.tensor([1.0, 0.9, 1.0, 0.9, 1.0]), [f"r{i}" for i in range(5)], [1] * 5)
    assert got[:4] == [0, 0, 0, 0]
    assert got[4] in (0, 7, 8)                                               # -3e38 / 0.5 is -inf in float32


# ---------------------------------------------------------------------------
# rmsnorm: rows kept in 8, 16, 24 or 32 groups a lane
# ---------------------------------------------------------------------------

@pytest.mark.parametrize("parts", [1, 2])
@pytest.mark.parametrize("width", [1020, 1024, 1028, 2048, 2052, 3072, 3076, 4096, 4100, 6146])
def test_a_normed_row_has_the_same_bits_among_few_and_many_rows(width, parts):
    k = K()
    g = torch.Generator().manual_seed(width + parts)
    rows = 1030
    x = (torch.randn(rows, width * parts, generator=g) * 3).to(dev())
    err = k.new_error_word(dev())
    for gain_dtype, out_dtype in ((torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32)):
        gain = (1 + 0.1 * torch.randn(width * parts, generator=g)).to(gain_dtype).to(dev())
        many = torch.empty(rows, width * parts, dtype=out_dtype, device=dev())
        k.rmsnorm(x, gain, many, 1e-6, err, groups=parts)
        few = torch.empty(3, width * parts, dtype=out_dtype, device=dev())
        k.rmsnorm(x, gain, few, 1e-6, err, torch.tensor([1029, 0, 500], dtype=torch.int32, device=dev()), groups=parts)
        assert torch.equal(few, many[[1029, 0, 500]])
        part = x.double().view(rows, parts, width)
        want = (part * torch.rsqrt((part * part).mean(-1, keepdim=True) + 1e-6)).view(rows, -1) * gain.double()
        # a float32 sum of `width` squares in 32 lanes, then three roundings; bfloat16 results round once more
        bound = 1e-6 if out_dtype == torch.float32 else 2.0 ** -8
        assert ((many.double() - want).abs() <= bound * (want.abs() + 1e-3)).all()
    k.raise_on_fault(err)
