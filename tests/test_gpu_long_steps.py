"""Kernels that only long steps, one-token steps or certain sizes reach, through one-layer models against the float64 oracles: the
tensor-memory attention kernels (256 tokens a sequence and more) at the edges of their 128-row tiles and 64-key blocks, the scan at each of
its state sizes and at lengths around its blocks of 16 and runs of 8 tokens, the matrix memory at partial rows and columns, steps of one
token per sequence at each count of heads that share a key, sampling more rows than a block, and a replayed step against the first one."""
import numpy as np
import pytest

import fazovik_util as fu
import goponex_util as gu
import zogurax_util as zu
from oracle import fazovik_ref, goponex_ref, zogurax_ref

pytestmark = pytest.mark.gpu

# float32: sums of up to a few hundred terms in another order than the oracle's, amplified by one norm (as in the families' own tests).
# bfloat16: activations rounded (2^-9) ahead of each of about six products; a lost or doubled block, row or key moves a row by its own size.
F32, BF16 = 3e-4, 6e-2


def engine(path, dtype, tokens, seqs=1):
    from llama_cpp import models
    return models.open_engine(models.open_model(path), n_ctx=max(tokens + 16, 64), max_seqs=seqs, dtype=dtype, kv_tokens=(tokens + 128) * seqs,
                              max_step_tokens=max(tokens * seqs, 16))


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


def check(util, ref, cfg, tmp_path, lengths, dtype):
    w = util.random_weights(cfg, seed=5)
    prompts = [toks(cfg["vocab"], n, 7 + i) for i, n in enumerate(lengths)]
    eng = engine(util.write_model(str(tmp_path / "m"), cfg, w), dtype, max(lengths), len(lengths))
    got = whole(eng, prompts)
    eng.close()
    for g, p in zip(got, prompts):
        off = rows_off(g, ref.forward(cfg, w, p))
        assert off.max() < (F32 if dtype == "float32" else BF16), (int(off.argmax()), float(off.max()))


@pytest.mark.parametrize("dims,lengths", [((16, 16), [256]), ((32, 48), [257]), ((64, 64), [383]), ((80, 128), [385]), ((128, 80), [300, 260]),
                                          ((128, 128), [640]), ((64, 32), [500, 12])])
def test_softmax_attention_of_long_steps(native_lib, tmp_path, dims, lengths):
    d, dv = dims
    cfg = zu.config([zu.biased(heads=4, kv_heads=2, dim=d, vdim=dv)])
    check(zu, zogurax_ref, cfg, tmp_path, lengths, "bfloat16")


@pytest.mark.parametrize("d,window,keep,lengths", [(16, 1, 0, [256]), (64, 64, 3, [257]), (80, 100, 70, [400]), (128, 129, 1, [511]), (32, 1000, 4, [300, 280])])
def test_window_attention_of_long_steps(native_lib, tmp_path, d, window, keep, lengths):
    cfg = gu.config([gu.parallel(left=gu.attn(heads=4, kv_heads=2, dim=d, rot=8, window=window, keep=keep))])
    check(gu, goponex_ref, cfg, tmp_path, lengths, "bfloat16")


@pytest.mark.parametrize("rank,heads,lengths", [(64, 3, [256]), (128, 4, [257]), (192, 2, [385]), (256, 2, [511]), (512, 2, [300, 290])])
@pytest.mark.parametrize("kind", ["plain", "rotated"])
def test_latent_attention_of_long_steps(native_lib, tmp_path, kind, rank, heads, lengths):
    layer = fu.plain(heads=heads, rank=rank) if kind == "plain" else fu.rotated(heads=heads, rank=rank, rot_dim=16)
    layers = [layer] + ([fu.plain(heads=heads, rank=rank, kv_from=0)] if kind == "plain" else [])
    check(fu, fazovik_ref, fu.config(layers), tmp_path, lengths, "bfloat16")


@pytest.mark.parametrize("state,inner,conv,lengths", [(1, 24, 2, [67]), (4, 64, 3, [16, 63]), (5, 65, 4, [64]), (8, 40, 4, [9, 70, 3]), (13, 130, 2, [129]),
                                                      (16, 300, 4, [1, 2, 200]), (17, 40, 4, [71]), (32, 72, 1, [66]), (33, 40, 5, [65])])
def test_scan_sizes(native_lib, tmp_path, state, inner, conv, lengths):
    cfg = gu.config([gu.parallel(right=gu.scan(inner=inner, state=state, dt_rank=4, conv=conv))])
    check(gu, goponex_ref, cfg, tmp_path, lengths, "float32")


@pytest.mark.parametrize("heads,d,dv,lengths", [(1, 1, 1, [17]), (2, 16, 32, [16]), (1, 17, 33, [31, 1]), (3, 48, 70, [65]), (1, 128, 256, [47]), (2, 100, 31, [33]),
                                                (1, 256, 64, [18])])
def test_matrix_memory_sizes(native_lib, tmp_path, heads, d, dv, lengths):
    cfg = gu.config([gu.mlstm(heads=heads, dim=d, vdim=dv)])
    check(gu, goponex_ref, cfg, tmp_path, lengths, "float32")


@pytest.mark.parametrize("heads,kv,d,dv", [(4, 4, 16, 16), (6, 2, 32, 48), (16, 4, 128, 128), (16, 1, 64, 80), (17, 1, 64, 64), (9, 1, 112, 32)])
def test_one_token_of_every_sequence(native_lib, tmp_path, heads, kv, d, dv):
    """Steps that decode all sequences: each key/value head's query rows in one tile, keys across one to three blocks of 64."""
    from llama_cpp.kv_pages import SequenceSlots
    cfg = zu.config([zu.biased(heads=heads, kv_heads=kv, dim=d, vdim=dv)])
    w = zu.random_weights(cfg, seed=6)
    lengths = [1, 2, 63, 64, 65, 127, 128, 130, 20, 40]
    prompts = [toks(cfg["vocab"], n + 2, 30 + i) for i, n in enumerate(lengths)]
    eng = engine(zu.write_model(str(tmp_path / "m"), cfg, w), "bfloat16", 136, len(lengths))
    seqs = SequenceSlots(eng)
    for i in range(len(lengths)):
        seqs.open(i)
    eng.step([(seqs.extend(i, n), p[:n]) for i, (n, p) in enumerate(zip(lengths, prompts))])
    got = [np.array(eng.step([(seqs.extend(i, 1), [p[n + k]]) for i, (n, p) in enumerate(zip(lengths, prompts))], want=[[0]] * len(lengths))[0]) for k in range(2)]
    eng.close()
    for i, (n, p) in enumerate(zip(lengths, prompts)):
        assert rows_off(np.stack([got[0][i], got[1][i]]), zogurax_ref.forward(cfg, w, p)[n:]).max() < BF16, i


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


def test_many_wanted_rows_and_long_rows(native_lib, tmp_path):
    """More wanted rows than a head chunk of 256 holds, a vocabulary that is not a multiple of four, sampling from the last row."""
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
