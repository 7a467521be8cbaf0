"""Device memory of an encoder's embedding path."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_an_encoder_gives_its_memory_back(cuda_ready):
    """Encoders that embed and go: free memory does not fall by their 0.84 GB of workspace each."""
    import torch
    from seqtree_b200 import device, workloads
    from seqtree_b200._lib import Packed
    from seqtree_b200.learned import Encoder
    codes, lens = workloads.cdr3_codes(3, 500)
    qs = device.SeqSet(Packed.from_arrays(*workloads.codes_to_letters(codes, lens)))
    out = torch.zeros((500, 64), dtype=torch.bfloat16, device="cuda")
    free = []
    for _ in range(4):
        enc = Encoder(seed=1)
        enc.embed_into(qs, out.data_ptr(), 1, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        del enc
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] < 200 << 20
