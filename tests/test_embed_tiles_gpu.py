"""The bf16 embedding at the edges of its tiles: 4 sequences a tensor-core tile, 8 a pass of the first
convolution, 16 an output block, one tile and then more for every multiprocessor (148; up to eight,
so that buffers and barrier phases come round), and every sequence length 1..32.  Bounds: bf16 activations (2^-9 relative each) through four products
with fp32 accumulation against the float64 forward, those of the general bf16 test (0.03 a
component, cosine 0.998)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle.encoder as oenc

pytestmark = pytest.mark.gpu

AA = "ARNDCQEGHILKMFPSTWYV"


@pytest.mark.parametrize("n", [1, 3, 4, 5, 15, 16, 17, 592, 593, 1187, 4145])
def test_every_row_of_partial_tiles(cuda_ready, n):
    import torch

    from seqtree_b200 import device
    from seqtree_b200.learned import Encoder, pad_codes
    rng = np.random.default_rng(n)
    lens = (np.arange(n) * 7 + 31) % 32 + 1  # 32, 7, 14, ...: all lengths
    seqs = ["".join(AA[i] for i in rng.integers(0, 20, size=int(L))) for L in lens]
    flat = (oenc.init_params(3) + rng.normal(0, 0.02, oenc.param_count())).astype(np.float32)
    out = torch.full((n + 1, 64), 7.0, dtype=torch.bfloat16, device="cuda")  # one row more
    Encoder(flat).embed_into(device.SeqSet(seqs, "aa"), out.data_ptr(), 1,
                             torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    raw = out.float().cpu().numpy()
    assert (raw[n] == 7.0).all()
    rows = np.arange(n)[:, None]
    got = raw[:n].reshape(n, 8, 8)[rows, np.arange(8)[None, :] ^ (rows & 7)].reshape(n, 64)
    codes, codelens = pad_codes(seqs)
    want = oenc.forward(flat.astype(np.float64), codes, codelens)
    assert np.abs(got - want).max() <= 0.03
    assert ((got * want).sum(1) / np.linalg.norm(got, axis=1)).min() >= 0.998
