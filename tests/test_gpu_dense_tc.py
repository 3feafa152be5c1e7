"""Products of more than 8 tokens on the tensor cores, through one-layer models, against the float64 oracles: token counts at the edges of
its two orientations and their tiles, widths whose last K slice or weight-row tile is partial, expert tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows_close(got, want, tol):
    d = got - want
    err = np.sqrt((d ** 2).mean(-1)) / np.sqrt((want ** 2).mean(-1))
    assert np.isfinite(got).all() and err.max() < tol, (int(err.argmax()), float(err.max()))


def _weights(tensors):
    return {k: np.asarray(t.data) if t.dtype == "I32" else t.to_float32() for k, t in tensors.items()}


# every activation is rounded to bf16 (2^-9 relative) ahead of each of the six products in a row; a lost or doubled tile, row or K
# slice is an error of the order of the row itself
TOL = 2e-2


@pytest.mark.parametrize("width,ff,T", [(256, 512, 9), (256, 512, 16), (264, 520, 17), (328, 200, 63), (256, 512, 65), (264, 520, 127), (256, 264, 128),
                                        (328, 512, 129), (256, 1000, 256), (264, 520, 257), (256, 512, 300), (512, 2048, 513), (328, 1224, 640)])
def test_steps_of_any_length_match_the_oracle(native_lib, width, ff, T):
    from llama_cpp import goponex
    from oracle import goponex_ref
    cfg, tensors = goponex.synthetic(width, 2, 1, ff, 301, pattern="p", seed=T)
    toks = [int(t) for t in np.random.default_rng(T).integers(0, 301, size=T)]
    e = goponex.open_synthetic(cfg, tensors, n_ctx=T + 8, max_seqs=1, dtype="bfloat16", max_step_tokens=T)
    e.ensure_pages(0, T)
    from llama_cpp.engine import SamplingSettings
    e.seq_begin(0, 0, [], SamplingSettings(temperature=0.0))
    logits, _ = e.step([(0, toks)], want=[list(range(T))])
    e.close()
    _rows_close(logits, goponex_ref.forward(cfg, _weights(tensors), toks), TOL)


@pytest.mark.parametrize("T,experts,top,ff", [(9, 4, 2, 64), (33, 8, 2, 136), (200, 4, 4, 128), (600, 4, 2, 200)])
def test_expert_tiles_match_the_oracle(native_lib, T, experts, top, ff):
    from llama_cpp import zogurax
    from llama_cpp.engine import SamplingSettings
    from oracle import zogurax_ref
    cfg, tensors = zogurax.synthetic(256, 4, ff, 300, pattern="b", experts=experts, top=top, seed=T)
    toks = [int(t) for t in np.random.default_rng(T).integers(0, 300, size=T)]
    e = zogurax.open_synthetic(cfg, tensors, n_ctx=T + 8, max_seqs=1, dtype="bfloat16", max_step_tokens=T)
    e.ensure_pages(0, T)
    e.seq_begin(0, 0, [], SamplingSettings(temperature=0.0))
    logits, _ = e.step([(0, toks)], want=[list(range(T))])
    e.close()
    _rows_close(logits, zogurax_ref.forward(cfg, _weights(tensors), toks), TOL)


@pytest.mark.parametrize("family", ["goponex", "zogurax"])
def test_a_row_has_the_same_bits_in_steps_of_any_length(native_lib, family):
    """A prompt whole (token tiles of up to 256, 128-row expert tiles) and in portions that take the other forms (tokens as the 128-row operand,
    one and two tiles of them, several K slices a copy, 64-row expert tiles, the line at 256 tokens from both sides): no sum changes its order."""
    from llama_cpp import goponex, zogurax
    from llama_cpp.engine import SamplingSettings
    N, V = 1100, 301
    if family == "goponex":
        cfg, tensors = goponex.synthetic(264, 2, 1, 520, V, pattern="p", seed=3)
    else:
        cfg, tensors = zogurax.synthetic(256, 4, 136, V, pattern="b", experts=8, top=2, seed=3)
    toks = [int(t) for t in np.random.default_rng(3).integers(0, V, size=N)]
    e = (goponex if family == "goponex" else zogurax).open_synthetic(cfg, tensors, n_ctx=N + 8, max_seqs=1, dtype="bfloat16", max_step_tokens=N)
    e.ensure_pages(0, N)
    got = []
    for cuts in ([N], [9, 256, 257, 578], [128, 129, 300, 16, 17, 510]):
        e.seq_begin(0, 0, [], SamplingSettings(temperature=0.0))
        rows, at = np.full((N, V), np.nan, np.float32), 0
        for n in cuts:
            want = [i for i in range(n) if n - n % 256 > i or n % 256 > 8]      # (the head takes rows by 256, and up to 8 of them its own way)
            rows[[at + i for i in want]] = e.step([(0, toks[at:at + n])], want=[want])[0]
            at += n
        got.append(rows)
    e.close()
    for other in got[1:]:
        seen = ~np.isnan(got[0][:, 0]) & ~np.isnan(other[:, 0])
        assert seen.sum() > 1000 and np.array_equal(other[seen], got[0][seen]), int(np.abs(other - got[0])[seen].max(-1).argmax())
