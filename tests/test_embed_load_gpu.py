"""The bf16 embedding while copies on another stream load the memory system, so that the kernels' bulk
stores are held up for longer than their tiles take: the rows of an undisturbed call, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5000, 40001])  # 9 tiles a multiprocessor; two chunks, 55 and 13
def test_rows_beside_copies(cuda_ready, n):
    import torch

    from seqtree_b200 import device, workloads
    from seqtree_b200._lib import Packed
    from seqtree_b200.learned import Encoder
    enc = Encoder(seed=5)
    codes, lens = workloads.cdr3_codes(7, n)
    qs = device.SeqSet(Packed.from_arrays(*workloads.codes_to_letters(codes, lens)))

    def embed(stream):
        out = torch.zeros((n, 64), dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        enc.embed_into(qs, out.data_ptr(), 1, stream.cuda_stream)
        return out

    want = embed(torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert np.isfinite(want.float().cpu().numpy()).all() and bool((want != 0).any(dim=1).all())
    src = torch.zeros(1 << 28, dtype=torch.int32, device="cuda")  # 1 GiB
    dst = torch.empty_like(src)
    load, work = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(6):
        out = torch.zeros_like(want)
        torch.cuda.synchronize()
        with torch.cuda.stream(load):
            for _ in range(8):
                dst.copy_(src)
        enc.embed_into(qs, out.data_ptr(), 1, work.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))
