"""Kernels that only longer steps, one-token steps or certain sizes reach, through one-layer models against the float64 oracles: the
tensor-memory attention kernels (steps of more than 8 tokens) at the edges of their 128-row tiles and 64-key blocks, the scan at each of
its state sizes and at lengths around its blocks of 16 and runs of 8 tokens, the matrix memory at partial rows and columns, steps of one
token per sequence at each count of heads that share a key, more wanted rows than a head chunk, a replayed step against the first one, and
a token's bits alone, in company and under other cuts."""
import numpy as np
import pytest

import fazovik_util as fu
import goponex_util as gu
import zogurax_util as zu
from oracle import fazovik_ref, goponex_ref, zogurax_ref

pytestmark = pytest.mark.gpu

# float32: sums of up to a few hundred terms in another order than the oracle's, amplified by one norm (as in the families' own tests).
# bfloat16: about a dozen independent roundings of 2^-9 / sqrt(3) on the way of a row, 4e-3 together, several times that in a row whose softmax
# is sharp or whose norm is small (most seen: 1.4e-2); a lost or doubled block, row or key moves a row by its own size.
F32, BF16 = 3e-4, 2.5e-2


def engine(path, dtype, tokens, seqs=1, **kw):
    from llama_cpp import models
    return models.open_engine(models.open_model(path), n_ctx=max(tokens + 16, 64), max_seqs=seqs, dtype=dtype, kv_tokens=(tokens + 128) * seqs,
                              max_step_tokens=max(tokens * seqs, 16), **kw)


def whole(eng, prompts):
    """Logits of every token of each prompt, all prompts in one step."""
    from llama_cpp.kv_pages import SequenceSlots
    seqs = SequenceSlots(eng)
    for i in range(len(prompts)):
        seqs.open(i)
    entries = [(seqs.extend(i, len(p)), p) for i, p in enumerate(prompts)]
    lg, _ = eng.step(entries, want=[list(range(len(p))) for p in prompts])
    out = np.split(np.array(lg), np.cumsum([len(p) for p in prompts])[:-1])
    for i in range(len(prompts)):
        seqs.close(i)
    return out


def toks(vocab, n, seed):
    return [int(t) for t in np.random.default_rng(seed).integers(0, vocab, size=n)]


def rows_off(got, want):
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    assert np.isfinite(got).all()
    d, w = got - want, want - want.mean(-1, keepdims=True)
    d -= d.mean(-1, keepdims=True)
    return np.sqrt((d ** 2).mean(-1)) / np.sqrt((w ** 2).mean())


def check(util, ref, cfg, tmp_path, lengths, dtype, bar=None):
    w = util.random_weights(cfg, seed=5)
    prompts = [toks(cfg["vocab"], n, 7 + i) for i, n in enumerate(lengths)]
    eng = engine(util.write_model(str(tmp_path / "m"), cfg, w), dtype, max(lengths), len(lengths))
    got = whole(eng, prompts)
    eng.close()
    for g, p in zip(got, prompts):
        off = rows_off(g, ref.forward(cfg, w, p))
        assert off.max() < (bar or (F32 if dtype == "float32" else BF16)), (int(off.argmax()), float(off.max()))


@pytest.mark.parametrize("dims,lengths", [((16, 16), [256]), ((32, 48), [257]), ((64, 64), [383]), ((80, 128), [385]), ((128, 80), [300, 260]),
                                          ((128, 128), [640]), ((64, 32), [500, 12]), ((32, 32), [9]), ((48, 16), [1, 2, 3, 4, 5, 16, 17, 32, 33, 63, 64, 65])])
@pytest.mark.parametrize("heads,kv", [(4, 2), (6, 1)])
def test_softmax_attention_of_long_steps(native_lib, tmp_path, dims, lengths, heads, kv):
    d, dv = dims
    cfg = zu.config([zu.biased(heads=heads, kv_heads=kv, dim=d, vdim=dv)])
    check(zu, zogurax_ref, cfg, tmp_path, lengths, "bfloat16")


@pytest.mark.parametrize("d,window,keep,lengths", [(16, 1, 0, [256]), (64, 64, 3, [257]), (80, 100, 70, [400]), (128, 129, 1, [511]), (32, 1000, 4, [300, 280]),
                                                  (32, 20, 2, [1, 2, 31, 33, 64, 65])])
def test_window_attention_of_long_steps(native_lib, tmp_path, d, window, keep, lengths):
    cfg = gu.config([gu.parallel(left=gu.attn(heads=4, kv_heads=2, dim=d, rot=8, window=window, keep=keep))])
    check(gu, goponex_ref, cfg, tmp_path, lengths, "bfloat16")


# the same over 32-bit pages: tiles of 32 queries, ranges of 128 keys; tokens that come alone
@pytest.mark.parametrize("d,window,keep,lengths", [(16, 1, 0, [33]), (64, 64, 3, [257]), (80, 100, 70, [200]), (128, 129, 1, [300, 1, 31]), (32, 1000, 4, [100, 64, 2]), (128, 700, 300, [900]), (64, 3000, 1, [1100]),
                                                  (112, 20, 40, [1, 2, 31, 33, 64, 65])])
def test_window_attention_of_long_steps_in_32_bits(native_lib, tmp_path, d, window, keep, lengths):
    cfg = gu.config([gu.parallel(left=gu.attn(heads=4, kv_heads=2, dim=d, rot=8, window=window, keep=keep))])
    check(gu, goponex_ref, cfg, tmp_path, lengths, "float32")


@pytest.mark.parametrize("n,window,keep", [(200, 70, 5), (900, 600, 300)])
def test_cuts_do_not_change_a_token_in_32_bits(native_lib, tmp_path, n, window, keep):
    """Window attention over 32-bit pages: in portions of two tokens and more, each in a step of more than 8, a prompt's logits have the bits of the whole
    (the longer one: with one to eight CTAs a tile, over one to eight ranges of keys)."""
    from llama_cpp.kv_pages import SequenceSlots
    cfg = gu.config([gu.parallel(left=gu.attn(heads=4, kv_heads=2, dim=64, rot=8, window=window, keep=keep))])
    eng = engine(gu.write_model(str(tmp_path / "m"), cfg, gu.random_weights(cfg, seed=9)), "float32", n + 100, 2)
    prompt, side = toks(cfg["vocab"], n, 1), toks(cfg["vocab"], 90, 2)
    rows = []
    for cuts in ([n], [33, n - 33], [2, 60, 7, n - 69], [n - 72, 64, 8]):
        seqs, got, at = SequenceSlots(eng), [], 0
        seqs.open(0), seqs.open(1)
        for k, c in enumerate(cuts):
            entries = [(seqs.extend(0, c), prompt[at:at + c]), (seqs.extend(1, 20), side[20 * k:20 * k + 20])]
            got.append(np.array(eng.step(entries, want=[list(range(c)), list(range(20))])[0])[:c])      # (more than 8 rows for the head: one form of it)
            at += c
        seqs.close(0), seqs.close(1)
        rows.append(np.concatenate(got))
    eng.close()
    for other in rows[1:]:
        assert np.array_equal(rows[0], other)


@pytest.mark.parametrize("d,window,keep,past,pieces", [
    (64, 100, 5, 200, [2] * 10), (128, 600, 300, 900, [2, 3, 4, 5, 2, 2]), (16, 1000, 0, 300, [2, 2, 2, 2, 2, 4]), (48, 40, 1, 63, [4, 3, 2]), (32, 3000, 0, 2200, [2] * 17),
    (80, 70, 3, 150, [1] * 8 + [2]), (128, 3000, 4, 2400, [1, 1, 9]), (64, 300, 4, 310, [1] * 15 + [40]), (64, 300, 0, 290, [1] * 20 + [40]), (112, 20, 40, 64, [1, 1, 1, 65])])
def test_short_portions_in_32_bits(native_lib, tmp_path, d, window, keep, past, pieces):
    """Window attention over 32-bit pages: portions of a few tokens behind others, whose tiles' warps take ranges of keys, more than one round of them, and
    tokens that come alone beside longer ones and join their launch, have the bits that they have in the whole prompts."""
    from llama_cpp.kv_pages import SequenceSlots
    cfg = gu.config([gu.parallel(left=gu.attn(heads=4, kv_heads=2, dim=d, rot=8, window=window, keep=keep))])
    eng = engine(gu.write_model(str(tmp_path / "m"), cfg, gu.random_weights(cfg, seed=9)), "float32", past + 80, len(pieces))
    prompts = [toks(cfg["vocab"], past + k, 20 + i) for i, k in enumerate(pieces)]
    seqs, wholes = SequenceSlots(eng), []
    for p, k in zip(prompts, pieces):
        seqs.open(0)
        wholes.append(np.array(eng.step([(seqs.extend(0, len(p)), p)], want=[list(range(len(p)))])[0])[past:])
        seqs.close(0)
    for i, p in enumerate(prompts):
        seqs.open(i)
        eng.step([(seqs.extend(i, past), p[:past])])
    got = np.array(eng.step([(seqs.extend(i, k), p[past:]) for i, (p, k) in enumerate(zip(prompts, pieces))], want=[list(range(k)) for k in pieces])[0])
    eng.close()
    for i, (g, w) in enumerate(zip(np.split(got, np.cumsum(pieces)[:-1]), wholes)):
        assert np.isfinite(w).all() and np.array_equal(g, w), i


@pytest.mark.parametrize("d,window,keep,past,pieces,at", [(64, 100, 5, 0, [300, 1, 20], 130), (128, 600, 40, 0, [200], 101), (16, 1000, 0, 0, [64, 2, 2, 9], 33),
                                                          (64, 200, 5, 310, [4, 3, 2], 2), (32, 1000, 4, 300, [4, 1, 1, 1, 4], 1), (128, 90, 1, 70, [33, 2], 32)])
def test_window_attention_in_32_bits_beside_a_token_without_numbers(native_lib, tmp_path, d, window, keep, past, pieces, at):
    """Window attention over 32-bit pages: a token whose keys and values are no numbers changes no bit of the tokens ahead of it and of other sequences, nor do
    pages that hold its rows, or others of a longer prompt, when they are used again."""
    from llama_cpp.kv_pages import SequenceSlots
    cfg, bad = gu.config([gu.parallel(left=gu.attn(heads=4, kv_heads=2, dim=d, rot=8, window=window, keep=keep))]), 130
    w = gu.random_weights(cfg, seed=9)
    w["embed"][bad] = np.nan
    eng = engine(gu.write_model(str(tmp_path / "m"), cfg, w), "float32", past + max(pieces), len(pieces))
    prompts, seqs, got = [toks(bad, past + k, 20 + i) for i, k in enumerate(pieces)], SequenceSlots(eng), []

    def run(there, lens):
        for i, p in enumerate(prompts):
            seqs.open(i)
            if past:
                eng.step([(seqs.extend(i, past), p[:past])])
        entries = [(seqs.extend(i, k), [there if i == 0 and j == at else t for j, t in enumerate(p[past:past + k])]) for i, (p, k) in enumerate(zip(prompts, lens))]
        rows = np.split(np.array(eng.step(entries, want=[list(range(k)) for k in lens])[0])[:, :bad], np.cumsum(lens)[:-1])
        for i in range(len(pieces)):
            seqs.close(i)
        return rows

    clean, beside = run(prompts[0][past + at], pieces), run(bad, pieces)
    again = run(prompts[0][past + at], pieces)
    assert all(np.isfinite(g).all() for g in clean) and np.isnan(beside[0][at:]).all()
    assert np.array_equal(beside[0][:at], clean[0][:at])
    for a, b, c in zip(clean[1:], beside[1:], again[1:]):
        assert np.array_equal(a, b) and np.array_equal(a, c)
    assert np.array_equal(clean[0], again[0])
    eng.close()


# (head sizes that are multiples of 8: the products around the attention take rounded rows, without which the general kernel runs)
LATENT = {"plain": lambda heads, rank, **kw: fu.plain(heads=heads, rank=rank, dim=24, vdim=16, **kw),
          "rotated": lambda heads, rank, **kw: fu.rotated(heads=heads, rank=rank, dim=24, vdim=16, rot_dim=16, **kw)}


@pytest.mark.parametrize("rank,heads,lengths", [(64, 3, [256]), (128, 4, [257]), (192, 2, [385]), (256, 2, [511]), (512, 2, [300, 290]), (64, 2, [9]), (512, 3, [65, 1, 2]),
                                                (128, 5, [129, 64, 1])])
@pytest.mark.parametrize("kind", ["plain", "rotated"])
def test_latent_attention_of_long_steps(native_lib, tmp_path, kind, rank, heads, lengths):
    layers = [LATENT[kind](heads, rank)] + ([LATENT[kind](heads, rank, kv_from=0)] if kind == "plain" else [])
    check(fu, fazovik_ref, fu.config(layers), tmp_path, lengths, "bfloat16")


# pairs of CTAs with rotated parts of their own (half of 64 columns each, and fewer), and sizes that leave two stages of values, one of the rotated parts
@pytest.mark.parametrize("rank,rot,lengths", [(512, 64, [300, 129, 2]), (512, 48, [64, 257]), (512, 16, [1, 65]), (256, 256, [257]), (192, 384, [385]), (64, 512, [129, 200])])
def test_rotated_parts_of_latent_attention(native_lib, tmp_path, rank, rot, lengths):
    check(fu, fazovik_ref, fu.config([fu.rotated(heads=3, rank=rank, dim=24, vdim=16, rot_dim=rot)]), tmp_path, lengths, "bfloat16")


@pytest.mark.parametrize("kind,rank", [("rotated", 512), ("plain", 512), ("rotated", 256), ("plain", 64)])
def test_latent_attention_whose_later_keys_outweigh_the_first(native_lib, tmp_path, monkeypatch, kind, rank):
    """Scores spread so far that blocks of 64 keys after the first raise many rows' maxima by more than 2^8, where the sum in tensor memory is rescaled.
    Bar: bf16 queries and cached rows put a score of spread 9 (natural units) off by 9 * 2^-9 * sqrt(2/3) = 1.4e-2, and its row by as much beside what the
    others' are off by; twice their sum."""
    from test_gpu_model import lagging_growth
    layer = LATENT[kind](3, rank, scale=0.45 if kind == "rotated" else 0.9)
    cfg, grown, spread, softmax = fu.config([layer]), [], [], fazovik_ref.causal_softmax

    def seen(scores):
        visible = np.tri(len(scores), dtype=bool)
        grown.append(lagging_growth(np.where(visible, scores * np.log2(np.e), -np.inf), 64)[:, 1:].sum())
        spread.append(scores[visible].std())
        return softmax(scores)

    monkeypatch.setattr(fazovik_ref, "causal_softmax", seen)
    check(fu, fazovik_ref, cfg, tmp_path, [300], "bfloat16", bar=8e-2)
    assert len(grown) == 3 and min(grown) >= 20 and 7 < min(spread) and max(spread) < 11


@pytest.mark.parametrize("rank,heads", [(64, 3), (128, 1), (512, 16)])
@pytest.mark.parametrize("kind", ["plain", "rotated"])
def test_latent_attention_of_one_token_of_every_sequence(native_lib, tmp_path, kind, rank, heads):
    decode_all(fu, fazovik_ref, fu.config([LATENT[kind](heads, rank)]), tmp_path)


# One layer in 32 bits: a handful of roundings of 6e-8 in a row. The scan is off by 1.9e-7 to 2.7e-7, the matrix memory by 1.6e-7 to 3.3e-7; bars: four times that.
@pytest.mark.parametrize("state,inner,conv,lengths", [(1, 24, 2, [67]), (4, 64, 3, [16, 63]), (5, 65, 4, [64]), (8, 40, 4, [9, 70, 3]), (13, 130, 2, [129]),
                                                      (16, 300, 4, [1, 2, 200]), (17, 40, 4, [71]), (32, 72, 1, [66]), (33, 40, 5, [65])])
def test_scan_sizes(native_lib, tmp_path, state, inner, conv, lengths):
    cfg = gu.config([gu.parallel(right=gu.scan(inner=inner, state=state, dt_rank=4, conv=conv))])
    check(gu, goponex_ref, cfg, tmp_path, lengths, "float32", bar=1e-6)


@pytest.mark.parametrize("heads,d,dv,lengths", [(1, 1, 1, [17]), (2, 16, 32, [16]), (1, 17, 33, [31, 1]), (3, 48, 70, [65]), (1, 128, 256, [47]), (2, 100, 31, [33]),
                                                (1, 256, 64, [18])])
def test_matrix_memory_sizes(native_lib, tmp_path, heads, d, dv, lengths):
    cfg = gu.config([gu.mlstm(heads=heads, dim=d, vdim=dv)])
    check(gu, goponex_ref, cfg, tmp_path, lengths, "float32", bar=1.3e-6)


# 32-bit products whose inputs are cut into three bf16 parts: K around 64-entry slices, tokens around 32-column tiles, rows around 128. Without
# the last part a row is off by 2^-17 (8e-6) per product; a few dozen 32-bit roundings in a row stay below half of that. (No matrix memory here:
# its division by a sum that can cancel makes 1.5e-5 of a change of 2e-7 in the embedding, in the oracle itself.)
SPLIT = {"biases": lambda W, ff: (gu, goponex_ref, gu.config([gu.parallel(mlp=ff, right=gu.scan(inner=W, dt_rank=8)), gu.parallel(mlp=2 * ff, left=gu.attn(dim=16))], width=W)),
         "latent": lambda W, ff: (fu, fazovik_ref, fu.config([LATENT["rotated"](3, 64, mlp=fu.dense(ff)), LATENT["plain"](2, 128, mlp=fu.dense(ff), kv_from=None)], width=W)),
         "experts": lambda W, ff: (zu, zogurax_ref, zu.config([zu.biased(heads=4, kv_heads=2, dim=16, vdim=24, mlp=zu.moe(experts=5, ff=ff, shared=40))], width=W))}


@pytest.mark.parametrize("W,ff,lengths", [(72, 200, [9]), (136, 72, [31, 33]), (64, 128, [128]), (200, 328, [129, 1, 65]), (256, 1000, [350])])
@pytest.mark.parametrize("kind", list(SPLIT))
def test_products_in_32_bits(native_lib, tmp_path, kind, W, ff, lengths):
    util, ref, cfg = SPLIT[kind](W, ff)
    check(util, ref, cfg, tmp_path, lengths, "float32", bar=4e-6)


def test_infinite_weight_of_a_32_bit_model(native_lib, tmp_path):
    """A write gate's map with an infinity: the gate is its cap or minus it (the embedding's entries, which the map reads, are not 0), and every
    token's logits are finite, in steps of more than 8 tokens as in short ones."""
    cfg = gu.config([gu.mlstm(heads=2, dim=24, vdim=20, mlp=40)])
    w = gu.random_weights(cfg, seed=5)
    w["l0.mix.i"][1, 7] = np.inf
    prompt = toks(cfg["vocab"], 20, 7)
    assert (w["embed"][prompt, 7] != 0).all()
    eng = engine(gu.write_model(str(tmp_path / "m"), cfg, w), "float32", 20, 1)
    long, short = whole(eng, [prompt])[0], whole(eng, [prompt[:8]])[0]
    eng.close()
    want = goponex_ref.forward(cfg, w, prompt)
    assert rows_off(long, want).max() < F32 and rows_off(short, want[:8]).max() < F32


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("W,dim,inner", [(66, 10, 34), (72, 130, 36), (1020, 20, 24), (1024, 64, 40), (1028, 12, 40), (2052, 16, 40), (4100, 16, 24)])
def test_rows_between_products(native_lib, tmp_path, W, dim, inner, dtype):
    """The row kernels on both sides of their rules: widths that are not multiples of 4, of one, two and four reads a thread and beyond 4096 entries;
    heads of 4-entry groups, of other sizes and beyond 128. (32 bits: rows of whole groups of 8 go through products that sum 64 entries at a time, off by 4e-7
    to 8.4e-7; others sum entry by entry, up to 6.3e-6 at 4100. Bars: four times that.)"""
    cfg = gu.config([gu.parallel(mlp=48, left=gu.attn(heads=2, kv_heads=1, dim=dim, window=9), right=gu.scan(inner=inner)), gu.mlstm(mlp=40, heads=2, dim=24, vdim=20)], width=W)
    check(gu, goponex_ref, cfg, tmp_path, [21, 9], dtype, bar=None if dtype == "bfloat16" else 3.4e-6 if W % 8 == 0 else 2.5e-5)


@pytest.mark.parametrize("W,n", [(70, 17), (1020, 17), (1024, 16), (1028, 40), (1030, 17), (2052, 33), (4096, 17)])
def test_joins_at_the_edges_of_rows(native_lib, tmp_path, W, n):
    """Joins with and without experts, rows of one, two and four reads a thread, rows that are no whole reads, few tokens and more. (Off by 3e-7 to 5e-7, by up
    to 1.9e-6 where products sum entry by entry; bars: four times that.)"""
    cfg = zu.config([zu.biased(mlp=zu.moe(experts=5, ff=24, shared=40)), zu.conved()], width=W)
    check(zu, zogurax_ref, cfg, tmp_path, [n], "float32", bar=2e-6 if W % 8 == 0 else 8e-6)


def test_slots_start_from_empty_states(native_lib, tmp_path):
    """Every recurrent state, tail and stabiliser of a slot is cleared when its next sequence starts, and no other slot's."""
    from llama_cpp.kv_pages import SequenceSlots
    cfg = gu.config([gu.parallel(mlp=40), gu.mlstm(heads=2, dim=17, vdim=33), gu.parallel(right=gu.scan(inner=41, conv=4))])
    w = gu.random_weights(cfg, seed=5)
    eng = engine(gu.write_model(str(tmp_path / "m"), cfg, w), "float32", 40, 3)
    prompts = [toks(cfg["vocab"], n, 7 + n) for n in (20, 33, 12)]
    seqs = SequenceSlots(eng)
    for i in range(3):
        seqs.open(i)
    eng.step([(seqs.extend(i, len(p)), p) for i, p in enumerate(prompts)])
    seqs.close(1)
    seqs.open("again")
    p = toks(cfg["vocab"], 15, 3)
    lg, _ = eng.step([(seqs.extend("again", 15), p), (seqs.extend(0, 1), [5]), (seqs.extend(2, 1), [6])], want=[list(range(15)), [0], [0]])
    eng.close()
    want = [goponex_ref.forward(cfg, w, t) for t in (p, prompts[0] + [5], prompts[2] + [6])]
    assert rows_off(lg[:15], want[0]).max() < F32
    assert rows_off(lg[15:], np.stack([want[1][-1], want[2][-1]])).max() < F32


def decode_all(util, ref, cfg, tmp_path, **kw):
    """Steps that decode all sequences, keys across one to three blocks of 64."""
    from llama_cpp.kv_pages import SequenceSlots
    w = util.random_weights(cfg, seed=6)
    lengths = [1, 2, 63, 64, 65, 127, 128, 130, 20, 40]
    prompts = [toks(cfg["vocab"], n + 2, 30 + i) for i, n in enumerate(lengths)]
    eng = engine(util.write_model(str(tmp_path / "m"), cfg, w), "bfloat16", 136, len(lengths), **kw)
    seqs = SequenceSlots(eng)
    for i in range(len(lengths)):
        seqs.open(i)
    eng.step([(seqs.extend(i, n), p[:n]) for i, (n, p) in enumerate(zip(lengths, prompts))])
    got = [np.array(eng.step([(seqs.extend(i, 1), [p[n + k]]) for i, (n, p) in enumerate(zip(lengths, prompts))], want=[[0]] * len(lengths))[0]) for k in range(2)]
    eng.close()
    for i, (n, p) in enumerate(zip(lengths, prompts)):
        assert rows_off(np.stack([got[0][i], got[1][i]]), ref.forward(cfg, w, p)[n:]).max() < BF16, i


# (17 heads over a key are more than a packed tile holds: a tensor-memory tile, or with pages of 48 a tile for each head)
@pytest.mark.parametrize("heads,kv,d,dv", [(4, 4, 16, 16), (6, 2, 32, 48), (16, 4, 128, 128), (16, 1, 64, 80), (17, 1, 64, 64), (9, 1, 112, 32)])
@pytest.mark.parametrize("block", [64, 48])
def test_one_token_of_every_sequence(native_lib, tmp_path, heads, kv, d, dv, block):
    """Each key/value head's query rows in one tile."""
    decode_all(zu, zogurax_ref, zu.config([zu.biased(heads=heads, kv_heads=kv, dim=d, vdim=dv)]), tmp_path, kv_block_tokens=block)


def test_windows_of_one_token_of_every_sequence(native_lib, tmp_path):
    layers = [gu.parallel(left=gu.attn(heads=8, kv_heads=2, dim=32, rot=8, window=w, keep=k)) for w, k in ((1, 0), (50, 3), (100, 70))]
    decode_all(gu, goponex_ref, gu.config(layers), tmp_path)


WHOLE = {
    "softmax": (zu, lambda: zu.config([zu.biased(heads=8, kv_heads=2, dim=32, vdim=48, mlp=zu.moe()), zu.conved(heads=4, kv_heads=4, dim=64, vdim=32, mlp=zu.moe())])),
    "latent": (fu, lambda: fu.config([LATENT["rotated"](4, 128), LATENT["plain"](3, 64)])),
    "window": (gu, lambda: gu.config([gu.parallel(left=gu.attn(heads=8, kv_heads=2, dim=32, rot=8, window=70, keep=5)),
                                      gu.mlstm(), gu.parallel(left=gu.attn(heads=4, kv_heads=4, dim=64, rot=8, window=200, keep=0))])),
}


@pytest.mark.parametrize("block", [64, 48])
@pytest.mark.parametrize("kind", sorted(WHOLE))
def test_company_and_cuts_do_not_change_a_token(native_lib, tmp_path, kind, block):
    """In steps of more than 8 tokens a prompt's logits have the same bits whole, in portions of two tokens and more, beside other prompts
    and beside sequences that decode; and so have those of the sequences beside it."""
    from llama_cpp.kv_pages import SequenceSlots
    util, make = WHOLE[kind]
    cfg = make()
    V, N, others = cfg["vocab"], 300, 12
    eng = engine(util.write_model(str(tmp_path / "m"), cfg, util.random_weights(cfg, seed=9)), "bfloat16", N + 130, others + 2, kv_block_tokens=block)
    prompt, side, rest = toks(V, N, 1), toks(V, 90, 2), [toks(V, 80, 10 + i) for i in range(others)]

    def run(cuts, company):
        """Rows of the prompt and, in company, of the sequences that decode beside each portion (the head's form depends on the number of
        wanted rows: more than 8 in every step)."""
        seqs, rows, beside = SequenceSlots(eng), [], []
        for i in range(others + 2):
            seqs.open(i)
        eng.step([(seqs.extend(i + 2, 20 + 5 * i), rest[i][:20 + 5 * i]) for i in range(others)])
        at = 0
        for k, n in enumerate(cuts):
            entries, want = [], []
            if company:
                entries += [(seqs.extend(i + 2, 1), [rest[i][20 + 5 * i + k]]) for i in range(others)]
                want += [[0]] * others
            entries.append((seqs.extend(0, n), prompt[at:at + n]))
            want.append(list(range(n)))
            if company and k == 0:
                entries.append((seqs.extend(1, len(side)), side))
                want.append([])
            lg, _ = eng.step(entries, want=want)
            at += n
            beside.append(np.array(lg[:len(lg) - n]))
            rows.append(np.array(lg[len(lg) - n:]))
        for i in range(others + 2):
            seqs.close(i)
        return np.concatenate(rows), beside

    whole_rows, _ = run([N], False)
    alone = []                                            # the sequences beside it, decoding by themselves
    seqs = SequenceSlots(eng)
    for i in range(others):
        seqs.open(i)
    eng.step([(seqs.extend(i, 20 + 5 * i), rest[i][:20 + 5 * i]) for i in range(others)])
    for k in range(4):
        alone.append(np.array(eng.step([(seqs.extend(i, 1), [rest[i][20 + 5 * i + k]]) for i in range(others)], want=[[0]] * others)[0]))
    for i in range(others):
        seqs.close(i)
    for cuts, company in [([N], True), ([129, 171], False), ([17, 283], True), ([256, 44], False), ([100, 9, 191], True), ([298, 2], True), ([2, 128, 165, 5], True), ([33, 60, 40, 167], True)]:
        rows, beside = run(cuts, company)
        assert np.array_equal(rows, whole_rows), (cuts, company, np.abs(rows - whole_rows).max(-1).argmax())
        for got, want in zip(beside, alone):
            assert not company or np.array_equal(got, want), (cuts, np.abs(got - want).max())
    eng.close()


def test_replayed_steps_are_the_first_ones_bits(native_lib, tmp_path):
    """The same step from the same state gives the same bits however often its launches have been replayed, wanted rows or not."""
    from llama_cpp.kv_pages import SequenceSlots
    cfg = zu.config([zu.biased(mlp=zu.moe()), zu.conved(mlp=zu.moe())], vocab=1003)
    eng = engine(zu.write_model(str(tmp_path / "m"), cfg, zu.random_weights(cfg, seed=8)), "bfloat16", 60, 12)
    runs = []
    for _ in range(4):
        seqs, rows = SequenceSlots(eng), []
        for i in range(12):
            seqs.open(i)
        eng.step([(seqs.extend(i, 3 + i), toks(1003, 3 + i, i)) for i in range(12)])
        for k in range(4):
            lg, _ = eng.step([(seqs.extend(i, 1), [17 * i + k]) for i in range(12)], want=[[0] if i % 2 else [] for i in range(12)])
            rows.append(np.array(lg))
        for i in range(12):
            seqs.close(i)
        runs.append(np.concatenate(rows))
    eng.close()
    assert runs[0].shape == (24, 1003)
    for other in runs[1:]:
        assert np.array_equal(runs[0], other)


@pytest.mark.parametrize("vocab", [203, 512])
def test_sampling_in_ragged_steps(native_lib, tmp_path, vocab):
    """Each slot with settings, uniforms and history of its own: sampled rows on both sides of a head chunk's end, some entries sampled and
    others not, steps that run directly, that are captured and that are replayed. The oracle draws from the logits the step returns."""
    from dataclasses import asdict
    from llama_cpp.engine import SamplingSettings
    from oracle import sampler_ref
    cfg = zu.config([zu.biased()], vocab=vocab)
    n = 10
    kinds = [SamplingSettings(temperature=0.0, repeat_penalty=1.0), SamplingSettings(temperature=0.9, top_k=20, top_p=0.8, min_p=0.02, repeat_penalty=1.3),
             SamplingSettings(temperature=1.2, top_p=0.9, frequency_penalty=0.7, presence_penalty=0.8),
             SamplingSettings(temperature=1.5, top_k=vocab, top_p=1.0, min_p=0.0, repeat_penalty=1.8, penalty_last_n=4), SamplingSettings(temperature=0.0, frequency_penalty=2.0)]
    settings, uniforms = [kinds[i % 5] for i in range(n)], [sampler_ref.MT19937Uniforms(40 + i).take(64) for i in range(n)]
    eng = engine(zu.write_model(str(tmp_path / "m"), cfg, zu.random_weights(cfg, seed=5)), "bfloat16", 60, n)
    hist, drawn, seen, off = [toks(vocab, 25, 60 + i) for i in range(n)], [0] * n, 0, 0
    for i in range(n):
        eng.ensure_pages(i, 60)
        eng.seq_begin(i, 0, hist[i], settings[i], uniforms=uniforms[i])

    def draw(entries, sample, rows):
        """Tokens of one step; the wanted rows end with every entry's last one."""
        nonlocal seen, off
        lg, got = eng.step(entries, want=rows, sample=sample)
        ends = np.cumsum([len(r) for r in rows]) - 1
        for i, t in enumerate(got):
            assert (t is not None) == sample[i]
            if sample[i]:
                kw = asdict(settings[i])
                want = sampler_ref.sample(lg[ends[i]], hist[i], float(uniforms[i][drawn[i]]), **kw)
                drawn[i] += 1
                seen, off = seen + 1, off + (want != t)
                assert want == t or settings[i].temperature > 0.0
                hist[i].append(t)
        return got

    last = draw([(i, list(hist[i])) for i in range(n)], [True] * n, [list(range(25))] * n)       # sampled rows 250 .. 259
    for _ in range(4):
        last = draw([(i, [last[i]]) for i in range(n)], [True] * n, [[0]] * n)
    odd = [i % 2 == 1 for i in range(n)]
    for _ in range(3):
        got = draw([(i, [last[i] if last[i] is not None else 7]) for i in range(n)], odd, [[0]] * n)
        last = [t if t is not None else 7 for t in got]
    last = draw([(i, [last[i]] * (1 + 5 * (i == 3))) for i in range(n)], [True] * n, [[0, 5] if i == 3 else [0] for i in range(n)])
    eng.close()
    assert seen == 75 and off <= 1, (seen, off)          # at most one draw at the edge of a 32-bit sum


def test_many_wanted_rows_and_long_rows(native_lib, tmp_path):
    """More wanted rows than a head chunk of 256 holds, rows of a width and vocabulary that are not multiples of the usual sizes."""
    cfg = zu.config([zu.biased()], vocab=1001)
    check(zu, zogurax_ref, cfg, tmp_path, [300, 7, 41], "bfloat16")
    cfg = zu.config([zu.biased()], width=4104, vocab=203)
    check(zu, zogurax_ref, cfg, tmp_path, [20], "bfloat16")


def test_rows_wanted_again_and_again(native_lib, tmp_path):
    """Repeated rows come as often as asked for; more of them than a step's description holds are refused, and nothing has moved."""
    from llama_cpp._cabi import B2Error
    from llama_cpp.kv_pages import SequenceSlots
    cfg = zu.config([zu.biased()], vocab=203)
    eng = engine(zu.write_model(str(tmp_path / "m"), cfg, zu.random_weights(cfg, seed=5)), "bfloat16", 16)
    seqs = SequenceSlots(eng)
    seqs.open(0)
    slot, prompt = seqs.extend(0, 4), toks(203, 4, 1)
    for rows in ([3] * 600, list(range(4)) * 5000):
        with pytest.raises(B2Error):
            eng.step([(slot, prompt)], want=[rows])
    lg, _ = eng.step([(slot, prompt)], want=[[0, 1, 2, 3] * 100 + [2]])
    eng.close()
    assert lg.shape == (401, 203) and all(np.array_equal(lg[i], lg[i % 4]) for i in range(400)) and np.array_equal(lg[400], lg[2])
    assert rows_off(lg[:4], zogurax_ref.forward(cfg, zu.random_weights(cfg, seed=5), prompt)).max() < BF16


@pytest.mark.parametrize("tname", ["Q4_K", "Q6_K", "Q8_0", "Q4_0", "Q5_K", "Q4_1"])
@pytest.mark.parametrize("K,N,T", [(256, 128, 257), (768, 130, 272), (2048, 256, 288), (1024, 257, 385), (512, 384, 512), (4096, 640, 511)])
def test_two_token_tiles_of_quantised_products(native_lib, tname, K, N, T):
    """More than 256 tokens: 256 weight rows and half of the tokens a CTA, at partial row tiles, halves of unequal size, K splits. The weights
    are rounded to f16 once (2^-11 each), as in the test of the other sizes."""
    from test_gpu_ops import _gemm_case
    assert _gemm_case(native_lib, tname, K, N, T) < 2e-3
    assert _gemm_case(native_lib, tname, K, N, T, n_splits=min(3, K // 256)) < 2e-3


@pytest.mark.parametrize("tname", ["Q4_K", "Q6_K", "Q8_0", "Q4_1"])
@pytest.mark.parametrize("K,N,T", [(256, 74 * 256 + 1, 512), (512, 75 * 256 + 130, 257), (256, 123 * 256, 400)])
def test_last_wave_of_quantised_products(native_lib, tname, K, N, T):
    """Row tiles past whole waves of two token tiles: one and two, and as many as fit three token tiles each on the SMs of one wave. Their sums have the
    same bits as in a product of few rows (two token tiles, test above), and so have those of the rows before them."""
    from test_gpu_ops import TYPE_IDS, lib_check, ptr
    from llama_cpp.synth import random_blocks
    from oracle import ggml_blocks as gb
    t = TYPE_IDS[tname]
    w = random_blocks(tname, N * K // gb.BLOCK[t][0], 0.02, seed=N + T).reshape(N, -1)
    x = np.random.default_rng(T).standard_normal((T, K)).astype(np.float32)

    def product(rows, n_splits):
        y = np.zeros((T, len(rows)), np.float32)
        lib_check(native_lib, native_lib.b2_op_gemm(0, t, ptr(rows), len(rows), K, ptr(x), T, None, ptr(y), n_splits))
        return y

    for n_splits in (1, K // 256):
        y = product(w, n_splits)
        for n0 in (0, 73 * 256, 74 * 256):
            part = np.ascontiguousarray(w[n0:n0 + 600])
            assert np.array_equal(y[:, n0:n0 + 600], product(part, n_splits)), (n0, n_splits)
        assert np.array_equal(y[:, -300:], product(np.ascontiguousarray(w[-300:]), n_splits))
