"""Kernels that have several forms chosen by size: at the edges of the rules that choose, and beside them, every form
gives the row the same bits, and the values of the plain float64 reference within a bound from the sums' lengths."""

from __future__ import annotations

import math

import numpy as np
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


@pytest.mark.parametrize("rows", [6, 37, 80, 149])
@pytest.mark.parametrize("vocab", [777, 49153, 163840])
def test_a_draw_falls_on_the_token_whose_share_of_the_mass_it_names(vocab, rows):
    """Against the cumulative mass in float64, in the (-p, id) order: the drawn token's share holds the draw to 4e-6 of the
    mass (an exponential's argument below 40 is rounded to 2^-24 of it, so the exponential is right to 2.5e-6, and so is every sum
    of them) and, where there is a nucleus, the share of its last token, which that error may take in or leave out.  Six kinds of
    rows, spread over 8 to 1 blocks."""
    from lockstep_b200.sampling import philox

    k = K()
    g = torch.Generator().manual_seed(vocab)
    base = torch.randn(6, vocab, generator=g) * 2.5
    base[1] = torch.randint(0, 4, (vocab,), generator=g).float()             # four values
    base[2] = torch.randint(0, 2, (vocab,), generator=g).float() * 1e-3      # two that are close
    base[3, ::2] = -math.inf
    base[4, vocab // 2] = 9.0
    temperature = torch.tensor([0.8, 1.0, 0.7, 1.1, 1.3, 0.9])
    top_p = torch.tensor([0.9, 0.5, 0.95, 1.0, 1.0, 0.05])
    pick = [i % 6 for i in range(rows)]
    uids, positions = [f"m{i}" for i in range(rows)], [5 + 3 * i for i in range(rows)]
    got = _draw(k, base[pick], temperature[pick], top_p[pick], uids, positions, seed=23)
    tables = []
    for i in range(6):
        z = (base[i] / temperature[i]).double()
        e = (z - z.max()).exp()
        order = torch.sort(e, descending=True, stable=True).indices
        through = torch.cumsum(e[order], 0) / e.sum()
        place = torch.empty_like(order)
        place[order] = torch.arange(vocab)
        head, slack = 1.0, 4e-6
        if top_p[i] < 1:
            last = min(int(torch.searchsorted(through, top_p[i].double())), vocab - 1)
            head, slack = float(through[last]), 4e-6 + float(e[order[last]] / e.sum())
        tables.append((through, place, head, slack))
    for row, token in enumerate(got):
        through, place, head, slack = tables[pick[row]]
        at, draw = int(place[token]), philox.uniform(23, uids[row], positions[row]) * head
        assert (float(through[at - 1]) if at else 0.0) - slack <= draw <= float(through[at]) + slack, (row, token)


@pytest.mark.parametrize("rows", [1, 37, 80, 149])
@pytest.mark.parametrize("vocab", [5, 777, 49153, 163840])
def test_among_equal_logits_the_draw_names_the_token(vocab, rows):
    """Every token has the same mass, so the sums are exact: the head is the first ceil(top_p V) ids, the token the one on which
    u times its size falls."""
    from fractions import Fraction

    import numpy as np

    from lockstep_b200.sampling import philox

    k = K()
    share = [Fraction(float(np.float32(p))) for p in (1.0, 0.9, 0.3)]
    pick = [i % 3 for i in range(rows)]
    uids, positions = [f"e{i}" for i in range(rows)], [7 * i for i in range(rows)]
    got = _draw(k, torch.full((rows, vocab), 1.5), torch.full((rows,), 0.7), torch.tensor([float(share[i]) for i in pick]), uids,
                positions, seed=3)
    for row, token in enumerate(got):
        u = Fraction(float(np.float32(philox.uniform(3, uids[row], positions[row]))))
        assert token == max(math.ceil(u * math.ceil(share[pick[row]] * vocab)), 1) - 1, row


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

# ---------------------------------------------------------------------------
# float32 products: few tokens on lanes, many tokens in tiles of several sizes
# ---------------------------------------------------------------------------

@pytest.mark.parametrize("epilogue", ["store", "residual", "silu", "gelu", "relu2"])
@pytest.mark.parametrize("n,k_", [(1000, 1060), (2048, 128), (2049, 260), (4736, 64), (4737, 260), (20000, 64)])
def test_a_float32_row_has_the_same_bits_in_every_batch(n, k_, epilogue):
    k = K()
    g = torch.Generator().manual_seed(n)
    code = {"store": k.EPILOGUE_STORE, "residual": k.EPILOGUE_RESIDUAL, "silu": k.EPILOGUE_SILU_MUL, "gelu": k.EPILOGUE_GELU,
            "relu2": k.EPILOGUE_RELU2}[epilogue]
    x = torch.randn(700, k_, generator=g).to(dev())
    w = (torch.randn(2 * n if epilogue == "silu" else n, k_, generator=g) / math.sqrt(k_)).to(dev())
    base = torch.randn(700, n, generator=g).to(dev())
    rows = {}
    for m in (1, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 300, 700):
        c = base[:m].clone()
        k.gemm_nt_simt(x[:m], w, c, code)
        rows[m] = c
    for m, c in rows.items():
        assert torch.equal(c, rows[700][:m]), m
    z = x.double() @ w.double().T
    gelu = lambda a: torch.nn.functional.gelu(a, approximate="tanh")
    want = {"store": lambda: z, "residual": lambda: base.double() + z, "gelu": lambda: gelu(z), "relu2": lambda: z.clamp(min=0) ** 2,
            "silu": lambda: torch.nn.functional.silu(z[:, :n]) * z[:, n:]}[epilogue]()
    # one chain of k_ float32 products of size 1 / sqrt(k_): an error of a few 2^-24 sqrt(k_) against |z| of about 1
    assert (rows[700].double() - want).abs().max() <= 2.0 ** -21 * math.sqrt(k_) * (1 + float(want.abs().max()))


@pytest.mark.parametrize("epilogue", ["store", "residual", "gelu", "relu2"])
@pytest.mark.parametrize("n,k_", [(1024, 260), (1000, 260), (1000, 4092), (1000, 4100)])
def test_a_float32_row_has_the_same_bits_in_tiles_of_128_tokens(n, k_, epilogue):
    """At 148 SMs 1,153 to 2,304 tokens of some 1,024 features take tiles of 128 x 64 (from a depth of 4,096 on with single FMAs),
    one token fewer or more tiles of 64 x 64: the bits of the few-token kernel, and the values in float64."""
    k = K()
    g = torch.Generator().manual_seed(n)
    code = {"store": k.EPILOGUE_STORE, "residual": k.EPILOGUE_RESIDUAL, "gelu": k.EPILOGUE_GELU, "relu2": k.EPILOGUE_RELU2}[epilogue]
    x = torch.randn(2305, k_, generator=g).to(dev())
    w = (torch.randn(n, k_, generator=g) / math.sqrt(k_)).to(dev())
    base = torch.randn(2305, n, generator=g).to(dev())
    few = base.clone()
    for at in range(0, 2305, 32):
        k.gemm_nt_simt(x[at:at + 32], w, few[at:at + 32], code)
    for m in (1152, 1153, 1700, 1800, 2304, 2305):
        c = base[:m].clone()
        k.gemm_nt_simt(x[:m], w, c, code)
        assert torch.equal(c, few[:m]), m
    z = x.double() @ w.double().T
    want = {"store": lambda: z, "residual": lambda: base.double() + z, "relu2": lambda: z.clamp(min=0) ** 2,
            "gelu": lambda: torch.nn.functional.gelu(z, approximate="tanh")}[epilogue]()
    # the bound of the test above
    assert (few.double() - want).abs().max() <= 2.0 ** -21 * math.sqrt(k_) * (1 + float(want.abs().max()))


@pytest.mark.parametrize("epilogue", ["store", "silu"])
def test_a_float32_product_takes_more_rows_than_a_grid_has_tiles(epilogue):
    """More than 65,535 tiles of 64 tokens: the bits of its two halves."""
    k = K()
    g = torch.Generator(device=dev()).manual_seed(7)
    m, n, k_ = 65535 * 64 + 70, 5, 4
    x = torch.randn(m, k_, generator=g, device=dev())
    w = torch.randn(2 * n if epilogue == "silu" else n, k_, generator=g, device=dev())
    code = k.EPILOGUE_SILU_MUL if epilogue == "silu" else k.EPILOGUE_STORE
    whole, halves = torch.full((m, n), math.nan, device=dev()), torch.full((m, n), math.nan, device=dev())
    k.gemm_nt_simt(x, w, whole, code)
    for part in (slice(0, m // 2), slice(m // 2, m)):
        k.gemm_nt_simt(x[part], w, halves[part], code)
    assert bool(torch.isfinite(whole).all()) and torch.equal(whole, halves)


# ---------------------------------------------------------------------------
# float32 attention of prompt portions: tiles of 16, 32 and 64 tokens
# ---------------------------------------------------------------------------

@pytest.mark.parametrize("nq,nkv,d,portions,mask,extra", [
    (4, 2, 128, [(0, 300), (513, 65)], 0, None), (2, 2, 64, [(0, 2), (255, 129), (0, 63)], 0, None),
    (4, 1, 128, [(300, 200)], 100, "sinks"), (2, 1, 64, [(700, 130)], (50, 5), "slopes"),
    (4, 2, 128, [(100, 333)], -64, "log"), (2, 2, 128, [(0, 70), (900, 64)], (64, 300), "cap"), (2, 1, 64, [(640, 64)], -256, None)])
def test_float32_attention_has_the_same_bits_in_tiles_of_every_size(nq, nkv, d, portions, mask, extra):
    from lockstep_b200.engine.batch import mask_parts, plan_attention

    k = K()
    page = 16
    g = torch.Generator().manual_seed(d + len(portions))
    tokens = sum(n for _, n in portions)
    pages_of = [-(-(s + n) // page) for s, n in portions]
    num_pages = sum(pages_of) + 2
    table = torch.zeros(len(portions), max(pages_of) + 1, dtype=torch.int32)
    ids, at, rows, off = torch.randperm(num_pages, generator=g), 0, [], 0
    for i, (s, n) in enumerate(portions):
        table[i, :pages_of[i]] = ids[at:at + pages_of[i]].to(torch.int32)
        at += pages_of[i]
        rows.append((i, off, s, n))
        off += n
    q = torch.randn(tokens, nq * d, generator=g).to(dev())
    pages = torch.randn(num_pages, 2, nkv, page, d, generator=g).to(dev())
    table = table.to(dev())
    slopes = (torch.rand(nq, generator=g) * 0.3).to(dev()) if extra in ("slopes", "log") else None
    rates = torch.rand(nq, generator=g).to(dev()) if extra == "log" else None
    sinks = torch.randn(nq, generator=g).to(dev()) if extra == "sinks" else None
    cap = 5.0 if extra == "cap" else 0.0
    window, keep = mask_parts(mask)
    err = k.new_error_word(dev())
    outs = {}
    for size in (16, 32, 64):
        tile = plan_attention(rows, mask, k.attention_split_size(), size)[0]
        work = torch.from_numpy(tile).to(dev())
        out = torch.full_like(q, float("nan"))
        if size == 16:
            k.attention_tile(q, pages, out, None, None, work, len(tile), table, nq, nkv, d, window, d ** -0.5, err, slopes,
                             rates, sinks, softcap=cap, keep_first=keep)
        else:
            assert k.attention_rows(q, pages, out, work, len(tile), size, table, nq, nkv, d, window, d ** -0.5, err, slopes,
                                    rates, sinks, softcap=cap, keep_first=keep)
        outs[size] = out
    k.raise_on_fault(err)
    assert bool(torch.isfinite(outs[16]).all())
    assert torch.equal(outs[16], outs[32]) and torch.equal(outs[16], outs[64])


@pytest.mark.parametrize("d,start,n,mask", [(128, 0, 130, 0), (64, 0, 130, 0), (128, 290, 75, 100), (64, 640, 64, (40, 300)),
                                            (128, 250, 60, -64)])
def test_a_value_that_is_no_number_reaches_the_rows_it_reaches_in_tiles_of_16_tokens(d, start, n, mask):
    """An infinity or a NaN among the values is NaN in every row of a 16-token tile that reads it, and in no other row."""
    from lockstep_b200.engine.batch import mask_parts, plan_attention

    k = K()
    page, nq, nkv = 16, 2, 1
    g = torch.Generator().manual_seed(d + n)
    q = torch.randn(n, nq * d, generator=g).to(dev())
    count = -(-(start + n) // page)
    pages = torch.randn(count, 2, nkv, page, d, generator=g)
    table = torch.arange(count, dtype=torch.int32).view(1, -1).to(dev())
    for key, value in ((start + 37, math.inf), (start + n - 2, math.nan), (start - 90, -math.inf), (start - 3, math.inf)):
        if key >= 0:
            pages[key // page, 1, 0, key % page, 5:9] = value
    pages = pages.to(dev())
    window, keep = mask_parts(mask)
    err, outs = k.new_error_word(dev()), {}
    for size in (16, 32, 64):
        tile = plan_attention([(0, 0, start, n)], mask, k.attention_split_size(), size)[0]
        work, out = torch.from_numpy(tile).to(dev()), torch.empty_like(q)
        if size == 16:
            k.attention_tile(q, pages, out, None, None, work, len(tile), table, nq, nkv, d, window, d ** -0.5, err, keep_first=keep)
        else:
            assert k.attention_rows(q, pages, out, work, len(tile), size, table, nq, nkv, d, window, d ** -0.5, err, keep_first=keep)
        outs[size] = out
    k.raise_on_fault(err)
    bad = outs[16].isnan()
    assert bool(bad.any())
    for size in (32, 64):
        assert torch.equal(outs[size].isnan(), bad), size
        assert torch.equal(outs[size][~bad], outs[16][~bad]), size


def test_float32_attention_declines_what_it_does_not_cover():
    k = K()
    assert k.attention_rows_tile_tokens(4096, 16, 128, torch.bfloat16) == 16
    assert k.attention_rows_tile_tokens(4096, 16, 96, torch.float32) == 16
    assert k.attention_rows_tile_tokens(3, 16, 128, torch.float32) == 16
    assert k.attention_rows_tile_tokens(4096, 16, 128, torch.float32) == 64
    q = torch.zeros(64, 96, device=dev())
    pages = torch.zeros(4, 2, 1, 16, 96, device=dev())
    work, table = torch.zeros(1, 8, dtype=torch.int32, device=dev()), torch.zeros(1, 4, dtype=torch.int32, device=dev())
    assert not k.attention_rows(q, pages, torch.empty_like(q), work, 1, 64, table, 1, 1, 96, 0, 1.0, k.new_error_word(dev()))


# ---------------------------------------------------------------------------
# the norm in front of a product: inside it or by a kernel of its own
# ---------------------------------------------------------------------------

@pytest.mark.parametrize("width,groups", [(1024, 1), (1024, 2), (2048, 1), (2560, 1)])
def test_rows_normed_inside_the_product_or_before_it_have_the_same_bits(width, groups):
    """Row 3 of 8 tokens (where the norm rides inside) and of 9 and 33 (where it does not)."""
    from lockstep_b200.parts.norm import NormedRows

    k = K()
    g = torch.Generator().manual_seed(width)
    h = (torch.randn(33, width, generator=g) * 2).to(dev())
    gain = (1 + 0.1 * torch.randn(width, generator=g)).to(torch.bfloat16).to(dev())
    w = (torch.randn(4096, width, generator=g) * 0.05).to(torch.bfloat16).to(dev())
    err = k.new_error_word(dev())

    class Norm:
        def __init__(self):
            self.gain, self.eps, self.groups = gain, 1e-6, groups

        def forward(self, rows, row_index):
            out = torch.empty(rows.shape, dtype=torch.bfloat16, device=dev())
            k.rmsnorm(rows, gain, out, 1e-6, err, row_index, groups)
            return out

    outs = []
    for t in (8, 9, 33):
        rows = NormedRows(Norm(), h[:t].contiguous())
        out = torch.empty(t, 4096, dtype=torch.bfloat16, device=dev())
        rows.linear(w, out, k.EPILOGUE_STORE, err)
        assert rows.pending() == (t == 8 and groups == 1 and width <= 2048)
        outs.append(out[3].clone())
    k.raise_on_fault(err)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("width,features,t,inside", [(2304, 1024, 1, True), (2560, 1792, 8, True), (2560, 1024, 9, False),
                                                     (4096, 256, 3, True), (4096, 2048, 8, False), (5120, 640, 8, True),
                                                     (8192, 1024, 16, True), (8192, 1024, 17, False), (8192, 2048, 1, True), (8192, 2048, 9, False),
                                                     (8192, 4096, 2, True), (6144, 2048, 8, True), (6144, 3072, 1, False)])
def test_wide_rows_normed_inside_a_product_of_few_blocks_have_the_bits_of_the_kernel_before_it(width, features, t, inside):
    """Above 2,048 elements the norm rides inside products whose blocks run at one time (14 clusters of eight), or nearly."""
    k = K()
    g = torch.Generator().manual_seed(width + features)
    h = (torch.randn(t, width, generator=g) * 2).to(dev())
    gain = (1 + 0.1 * torch.randn(width, generator=g)).to(torch.bfloat16).to(dev())
    w = (torch.randn(features, width, generator=g) * 0.05).to(torch.bfloat16).to(dev())
    err = k.new_error_word(dev())
    assert k.norm_inside_pays(t, features, w) == inside
    apart, rows = torch.empty(t, features, dtype=torch.bfloat16, device=dev()), torch.empty(t, width, dtype=torch.bfloat16, device=dev())
    k.rmsnorm(h, gain, rows, 1e-6, err)
    k.gemm_nt(rows, w, apart, err=err)
    out = torch.empty_like(apart)
    if inside:
        assert k.gemm_nt_tc_rmsnorm(h, gain, 1e-6, w, out, k.EPILOGUE_STORE, err)
        assert torch.equal(out, apart)
    k.raise_on_fault(err)


# ---------------------------------------------------------------------------
# bfloat16 attention of prompt portions on the tensor cores
# ---------------------------------------------------------------------------

class Prompt:
    """Requests of bfloat16 queries, keys and values in a shuffled cache, and the kernel over portions of them."""

    def __init__(self, nq, nkv, d, page, lengths, mask=0, extra=None, seed=0):
        from lockstep_b200.engine.batch import mask_parts

        g = torch.Generator().manual_seed(seed + nq + d)
        self.nq, self.nkv, self.d, self.mask, self.lengths = nq, nkv, d, mask, lengths
        self.window, self.keep = mask_parts(mask)
        self.scale = d ** -0.5
        self.q = [torch.randn(n, nq, d, generator=g).bfloat16() for n in lengths]
        self.k, self.v = ([torch.randn(n, nkv, d, generator=g).bfloat16() for n in lengths] for _ in range(2))
        count = [-(-n // page) for n in lengths]
        ids, at = torch.randperm(sum(count), generator=g).to(torch.int32), 0
        self.table = torch.zeros(len(lengths), max(count), dtype=torch.int32)
        pages = torch.full((sum(count), 2, nkv, page, d), math.nan).bfloat16()        # behind a request's end: never written
        for r, n in enumerate(lengths):
            self.table[r, :count[r]] = ids[at:at + count[r]]
            at += count[r]
            for which, rows in ((0, self.k[r]), (1, self.v[r])):
                key = torch.arange(n)
                pages[self.table[r, key // page].long(), which, :, key % page] = rows
        self.pages, self.table = pages.to(dev()), self.table.to(dev())
        self.slopes = self.rates = self.sinks = None
        self.cap = 4.0 if extra == "cap" else 0.0
        if extra in ("linear", "log"):
            self.slopes = torch.rand(nq, generator=g) * 0.2
        if extra == "log":
            self.rates = torch.rand(nq, generator=g)
        if extra == "sinks":
            self.sinks = torch.randn(nq, generator=g)

    def run(self, portions):
        """portions (request, start, tokens), two tokens at least; the rows of each, [tokens, nq, d]."""
        from lockstep_b200.engine.batch import plan_attention

        k = K()
        rows, off = [], 0
        for r, start, n in portions:
            rows.append((r, off, start, n))
            off += n
        q = torch.cat([self.q[r][start:start + n] for r, start, n in portions]).view(off, -1).to(dev())
        tile = plan_attention(rows, self.mask, k.attention_split_size(), k.attention_prefill_tc_tile_tokens())[0]
        out, err = torch.full_like(q, math.nan), k.new_error_word(dev())
        on = lambda t: None if t is None else t.to(dev())
        assert k.attention_prefill_tc(q, self.pages, out, torch.from_numpy(tile).to(dev()), len(tile), self.table, self.nq,
                                      self.nkv, self.d, self.window, self.scale, err, on(self.slopes), on(self.rates),
                                      on(self.sinks), softcap=self.cap, keep_first=self.keep)
        k.raise_on_fault(err)
        return [x.view(-1, self.nq, self.d) for x in out.cpu().split([n for _, _, n in portions])]

    def plain(self, r):
        from lockstep_b200.engine.batch import first_key

        n = self.lengths[r]
        pos = np.arange(n)
        seen = (pos[None, :] <= pos[:, None]) & ((pos[None, :] >= first_key(pos, self.window)[:, None]) | (pos[None, :] < self.keep))
        away = torch.from_numpy(np.maximum(pos[:, None] - pos[None, :], 0)).double()
        want = torch.empty(n, self.nq, self.d, dtype=torch.float64)
        for h in range(self.nq):
            kv = h // (self.nq // self.nkv)
            s = self.q[r][:, h].double() @ self.k[r][:, kv].double().T * self.scale
            if self.cap:
                s = self.cap * torch.tanh(s / self.cap)
            if self.rates is not None:
                s = s - self.slopes[h].double() * torch.log1p(self.rates[h].double() * away)
            elif self.slopes is not None:
                s = s - self.slopes[h].double() * away
            s = s.masked_fill(~torch.from_numpy(seen), -math.inf)
            if self.sinks is not None:
                s = torch.cat([s, self.sinks[h].double().expand(n, 1)], 1)
            want[:, h] = torch.softmax(s, 1)[:, :n] @ self.v[r][:, kv].double()
        return want


@pytest.mark.parametrize("extra", [None, "sinks", "log", "linear", "cap"])
@pytest.mark.parametrize("nq,nkv,d,page,mask", [(4, 2, 128, 16, 0), (2, 1, 64, 8, 300), (2, 2, 128, 128, (500, 4)), (4, 1, 64, 32, (300, 200)),
                                                (2, 1, 128, 64, (130, 129)), (2, 1, 128, 16, -200)])
def test_a_bfloat16_row_of_a_prompt_has_the_same_bits_however_it_is_cut(nq, nkv, d, page, mask, extra):
    """A prompt of 1,500 tokens whole, and from 0, 1, 37 and 127 tokens past the edges of two neighbouring tiles on, with
    windows, chunks and kept first keys: the tile that a row's item begins with is another one each time, and a row has the same bits.
    Values against float64: P and the result are rounded to 2^-9 of themselves, of values up to 4.5."""
    prompt = Prompt(nq, nkv, d, page, [1500], mask, extra)
    whole = prompt.run([(0, 0, 1500)])[0]
    assert (whole.double() - prompt.plain(0)).abs().max() <= 2e-2
    for edge in (1024, 1152):
        for past in (0, 1, 37, 127):
            start = edge + past
            assert torch.equal(prompt.run([(0, start, 1500 - start)])[0], whole[start:]), start
    assert torch.equal(prompt.run([(0, 700, 2)])[0], whole[700:702])


@pytest.mark.parametrize("nq,nkv,d,mask,extra", [(16, 8, 128, 0, None), (8, 2, 64, (100, 4), None), (16, 4, 128, 90, "log"), (8, 8, 64, 0, "cap")])
def test_many_short_portions_have_the_rows_of_each_alone(nq, nkv, d, mask, extra):
    """Sixty requests with portions of one, two and three tiles of keys: several items a block, so that a block's items end in
    either team's tile and hand over their places in shared and tensor memory one after the other."""
    lengths = [(37, 128, 129, 200, 257, 300, 384, 2, 90, 250)[i % 10] for i in range(60)]
    starts = [(0, 1, 100, 0)[i % 4] for i in range(60)]
    portions = [(i, s, n - s) for i, (s, n) in enumerate(zip(starts, lengths)) if n - s > 1]
    prompt = Prompt(nq, nkv, d, 16, lengths, mask, extra, seed=3)
    together = prompt.run(portions)
    for (r, start, n), rows in zip(portions, together):
        if r < 10 or r % 7 == 0:
            assert (rows.double() - prompt.plain(r)[start:]).abs().max() <= 2e-2, r
            assert torch.equal(rows, prompt.run([(r, start, n)])[0]), r


@pytest.mark.parametrize("scale", [0.0, -0.125, -3.0])
def test_prompt_attention_takes_a_scale_that_is_not_above_0(scale):
    prompt = Prompt(4, 2, 64, 16, [300], (100, 4))
    prompt.scale = scale
    assert (prompt.run([(0, 0, 300)])[0].double() - prompt.plain(0)).abs().max() <= 2e-2


@pytest.mark.parametrize("d,extra", [(128, None), (64, "log")])
def test_a_row_whose_scores_are_no_numbers_weighs_nothing(d, extra):
    """A query that is NaN gives a row of zeros and leaves the others their bits; a key that is NaN is NaN in every row that sees
    it beside others, and zeros in the row that sees it alone."""
    prompt = Prompt(2, 1, d, 16, [300], 0, extra)
    clean = prompt.run([(0, 0, 300)])[0]
    for row in (0, 130, 299):
        prompt.q[0][row, 1] = math.nan
    got = prompt.run([(0, 0, 300)])[0]
    hit = torch.zeros(300, 2, dtype=torch.bool)
    hit[[0, 130, 299], 1] = True
    assert bool((got[hit] == 0).all()) and torch.equal(got[~hit], clean[~hit])
    prompt = Prompt(2, 1, d, 16, [300], 0, extra)
    prompt.pages[int(prompt.table[0, 0]), 0, 0, 0, 3] = math.nan
    got = prompt.run([(0, 0, 300)])[0]
    assert bool((got[0] == 0).all()) and bool(got[1:].isnan().all())


@pytest.mark.parametrize("nq,nkv,d,page,mask", [(4, 2, 128, 16, 0), (3, 3, 16, 8, 0), (8, 2, 64, 64, 100), (8, 1, 128, 32, (300, 40)),
                                                (2, 1, 112, 16, -96), (4, 4, 128, 128, 0)])
def test_float32_splits_of_single_tokens_have_the_bits_of_the_tile_kernel(nq, nkv, d, page, mask):
    """Partials of every split of single tokens at the edges of tiles and splits, an infinity and a NaN among older values,
    against the tile kernel's, bit for bit."""
    from lockstep_b200.engine.batch import mask_parts, plan_attention

    k = K()
    g = torch.Generator().manual_seed(nq * d + page)
    places = [0, 1, 30, 31, 32, 33, 127, 255, 256, 257, 511, 512, 700, 767]
    count = -(-768 // page)
    pages = torch.randn(count * len(places), 2, nkv, page, d, generator=g)
    table = torch.randperm(count * len(places), generator=g).to(torch.int32).view(len(places), count).contiguous()
    for key, value in ((3, math.inf), (763, math.nan)):          # of the last request alone
        pages[int(table[-1, key // page]), 1, 0, key % page, 5:9] = value
    q = torch.randn(len(places), nq * d, generator=g).to(dev())
    pages, table = pages.to(dev()), table.to(dev())
    _, split, _, n_slots = plan_attention([(i, i, p, 1) for i, p in enumerate(places)], mask, k.attention_split_size())
    work = torch.from_numpy(np.concatenate([split, np.zeros((3, 8), dtype=np.int32)])).to(dev())      # null items at the end
    window, keep = mask_parts(mask)
    err, got = k.new_error_word(dev()), []
    for kernel in (k.attention_split, k.attention_tile):
        acc = torch.full((n_slots, nq, d), 7.0, device=dev())
        ml = torch.full((n_slots, nq, 2), 7.0, device=dev())
        if kernel is k.attention_split:
            assert kernel(q, pages, acc, ml, work, len(work), table, nq, nkv, d, window, d ** -0.5, err, keep_first=keep)
        else:
            kernel(q, pages, None, acc, ml, work, len(work), table, nq, nkv, d, window, d ** -0.5, err, keep_first=keep)
        got.append((acc.view(torch.int32), ml.view(torch.int32), acc.isnan()))
    k.raise_on_fault(err)
    assert bool(got[0][2].any()) and torch.equal(got[0][2], got[1][2])
    assert torch.equal(got[0][0][~got[0][2]], got[1][0][~got[0][2]]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("nq,nkv,d,gain,cache", [(16, 8, 128, torch.bfloat16, True), (3, 1, 128, torch.float32, True), (2, 1, 64, torch.bfloat16, True),
                                                 (7, 7, 64, None, True), (5, 1, 128, torch.bfloat16, False), (200, 8, 128, torch.bfloat16, True)])
def test_whole_heads_have_the_bits_of_the_general_kernel(nq, nkv, d, gain, cache):
    """Odd and even numbers of heads, of 64 and 128 elements, with and without gains and cache, against the kernel that takes any
    alignment (rows that start 8 bytes off)."""
    k = K()
    g = torch.Generator().manual_seed(nq + d)
    tokens, page, num_pages = 37, 16, 5
    raw = torch.randn(tokens * (nq + 2 * nkv) * d + 8, generator=g).bfloat16().to(dev())
    gains = [None, None] if gain is None else [(1 + 0.1 * torch.randn(d, generator=g)).to(gain).to(dev()) for _ in range(2)]
    ang = torch.rand(80, d // 2, generator=g) * 6
    cos, sin = ang.cos().to(dev()), ang.sin().to(dev())
    positions = torch.arange(tokens, dtype=torch.int32, device=dev()) + 11
    table = torch.tensor([[4, 2, 0, 1, 3]], dtype=torch.int32, device=dev())
    req = torch.zeros(tokens, dtype=torch.int32, device=dev())
    err, got, names = k.new_error_word(dev()), [], []
    for off in (0, 4):
        qkv = torch.empty_like(raw)[off:off + raw.numel() - 8].view(tokens, -1)
        qkv.copy_(raw[:-8].view(tokens, -1))
        q = torch.full((tokens, nq * d), 7.0, dtype=torch.bfloat16, device=dev())
        pages = torch.full((num_pages, 2, nkv, page, d), 7.0, dtype=torch.bfloat16, device=dev())
        before = k.kernel_counts()
        k.qk_norm_rope_store(qkv, q, pages, *gains, cos, sin, positions, req, table, nq, nkv, d, d, 1e-6, cache, err)
        after = k.kernel_counts()
        names.append([n for n in after if after[n] > before.get(n, 0)])
        got.append((q, pages))
    k.raise_on_fault(err)
    assert names == [["qk_norm_rope_store_whole"], ["qk_norm_rope_store"]]
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert bool((got[0][1] != 7).any()) == cache
