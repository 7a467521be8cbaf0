"""The bf16 embedding where a convolution product that no output uses overflows."""
from __future__ import annotations

import numpy as np
import pytest

import oracle.encoder as oenc

pytestmark = pytest.mark.gpu


def test_products_outside_a_sequence_are_not_seen(cuda_ready):
    """A sequence of one residue has no left neighbour, so conv2's first weights do not reach it: not
    even when h1 times them is infinite."""
    import torch

    from seqtree_b200 import device
    from seqtree_b200.learned import Encoder
    seqs = device.SeqSet(list("ARNDCQEGHILKMFPSTWYV") * 2, "aa")
    flat = oenc.init_params(4).astype(np.float32)
    at = 3 * 24 * 128 + 128  # W1, b1, then W2 [3][128][128]
    rows = []
    for first in (0.0, 3.0e38):
        flat[at:at + 128 * 128] = first
        out = torch.zeros((40, 64), dtype=torch.bfloat16, device="cuda")
        Encoder(flat).embed_into(seqs, out.data_ptr(), 1, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        rows.append(out.float().cpu().numpy())
    assert np.isfinite(rows[0]).all()
    assert np.array_equal(rows[0], rows[1])
