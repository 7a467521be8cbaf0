"""The bf16 training step, whose passes are folded into its products, against the fp32 precision's
separate passes (which the float64 oracle checks): batches whose position rows end inside, at and past a
128-row tile, and every sequence length.  bf16 products differ from fp32 ones by about 2^-9 relative per
factor; the bounds are those of the bf16 gradients against the oracle (5 % relative norm, cosine
0.998 per parameter block)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.encoder import SHAPES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [1, 2, 3, 33, 64, 65])
def test_folded_step_matches_the_separate_passes(cuda_ready, pairs):
    from seqtree_b200 import learned
    rng = np.random.default_rng(pairs)
    lens = ((np.arange(2 * pairs) * 7 + 31) % 32 + 1).astype(np.int32)  # 32, 7, 14, ...: all lengths
    codes = rng.integers(0, 24, size=(2 * pairs, 32)).astype(np.uint8)
    codes[np.arange(32)[None, :] >= lens[:, None]] = 0
    scores = rng.integers(0, 120, size=pairs).astype(np.int32)
    params = learned.init_params(3)
    params += rng.normal(0, 0.05, params.size).astype(np.float32)  # biases away from 0
    got = learned.Encoder(params, precision="bf16").loss_grad(codes, lens, scores)
    want = learned.Encoder(params, precision="fp32").loss_grad(codes, lens, scores)
    assert abs(got[0] - want[0]) <= 1e-2 * max(abs(want[0]), 1e-2)
    o = 0
    for name, shape in SHAPES:
        n = int(np.prod(shape))
        a, b = got[1][o:o + n].astype(np.float64), want[1][o:o + n].astype(np.float64)
        o += n
        norm = np.linalg.norm(b)
        if norm < 1e-12:
            assert np.linalg.norm(a) < 1e-9
            continue
        assert np.linalg.norm(a - b) <= 0.05 * norm, name
        assert a @ b >= 0.998 * norm * np.linalg.norm(a), name
