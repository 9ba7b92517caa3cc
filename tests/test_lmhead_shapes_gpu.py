"""The LM head at the edges of its shapes: token counts around the three padded
sizes, rows that are no whole tile, tiles shared by two and by many thread blocks,
calls of more tokens than the handle has rows (no tile is shared then), hidden
sizes of several launches, and hidden values that do not all fit binary16 (those
calls are multiplied in bf16). Against the product in binary64."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from test_lmhead_affine_gpu import _affine_inputs, _gpu_affine, _widen
from test_lmhead_gpu import _gpu_logits, _head_inputs

pytestmark = pytest.mark.gpu

SHAPES = [  # tokens, hidden, rows, the handle's max_rows
    (1, 512, 1, 1), (16, 512, 255, 64), (17, 8192, 300, 64), (32, 512, 40_003, 32),
    (33, 1536, 38_145, 64), (64, 4096, 12_289, 64), (64, 1024, 50_001, 16), (16, 1024, 151_900, 64)]


@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("bits", [0, 8, 4])  # 0: symmetric bytes
@pytest.mark.parametrize("tokens,hidden,rows,max_rows", SHAPES + [(20, 8192 + 1536, 700, 64)])
def test_head_at_the_edges_of_its_shapes(cuda, lily, tokens, hidden, rows, max_rows, bits, spread):
    if bits and hidden > 8192:
        pytest.skip("an affine head takes a hidden size of at most 8192")
    rng = np.random.default_rng([91, tokens, hidden, rows, bits])
    scratch = lily.SamplerScratch(rows, max_rows=max_rows)
    if bits:
        h, codes, s, b = _affine_inputs(rng, tokens, hidden, rows, bits=bits)
        w = oracle.dequant_affine(codes, _widen(s), _widen(b), rows, hidden, 64, bits)
    else:
        h, codes, s = _head_inputs(cuda, rng, tokens, hidden, rows)
        w = codes.astype(np.float32) * np.repeat(_widen(s), 64, axis=1)
    if spread:  # one column 2^-36 of its size: binary16 cannot hold it beside the others
        h[tokens // 2, 3] -= min(int(h[tokens // 2, 3]) & 0x7F80, 36 << 7)
        h[tokens // 2, 3] |= 1
    got = _gpu_affine(cuda, scratch, h, codes, s, b, bits) if bits else \
        _gpu_logits(cuda, lily, scratch, h, codes, s).cpu().numpy()
    exact = _widen(h).astype(np.float64) @ w.astype(np.float64).T
    # Bound: hidden terms of at most |h| |w|, each with a rounding (2^-24) in its group's sum
    # (depth 64), its scale's product and the sum over the groups; twice for an affine
    # head (codes and offset apart, each up to twice as large as w).
    size = np.abs(_widen(h)).astype(np.float64) @ np.abs(w).astype(np.float64).T
    if bits:
        top = np.abs(_widen(s)) * float(1 << bits) + np.abs(_widen(b))
        size = np.abs(_widen(h)).astype(np.float64) @ np.repeat(top, 64, axis=1).astype(np.float64).T * 2.0
    bound = size * (64 + hidden // 64 + 2) * 2.0 ** -24
    assert np.isfinite(got).all()
    assert np.all(np.abs(got - exact) <= bound), float((np.abs(got - exact) / bound).max())
    scratch.close()


def test_a_handle_of_few_rows_is_small(cuda, lily):
    # (The head's workspaces follow max_rows; those of calls of more tokens are made by such calls.)
    handles = [lily.SamplerScratch(151_936, max_rows=1, max_history=0)]
    before = cuda.cuda.mem_get_info()[0]
    handles += [lily.SamplerScratch(151_936, max_rows=1, max_history=0) for _ in range(32)]
    assert before - cuda.cuda.mem_get_info()[0] <= 32 << 20
    for h in handles:
        h.close()
