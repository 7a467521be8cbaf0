"""The workspace of an encoder's embedding path: its memory, and calls on two streams."""
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


@pytest.mark.parametrize("layout", [0, 1])
def test_one_encoder_on_two_streams(cuda_ready, layout):
    """Calls of one encoder on two streams at once, over sets of other lengths: the rows of lone calls."""
    import torch
    from seqtree_b200 import device, workloads
    from seqtree_b200.learned import Encoder
    enc = Encoder(seed=2)
    n = 20000
    dtype, bits = (torch.bfloat16, torch.int16) if layout else (torch.float32, torch.int32)
    sets = [device.SeqSet(workloads.uniform_strings(s, n, lo, hi, workloads.AA20))
            for s, lo, hi in ((1, 4, 9), (2, 20, 32))]
    outs = [torch.zeros((n, 64), dtype=dtype, device="cuda") for _ in sets]
    want = []
    for s, out in zip(sets, outs):
        enc.embed_into(s, out.data_ptr(), layout, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        want.append(out.view(bits).clone())
    streams = [torch.cuda.Stream() for _ in sets]
    for _ in range(5):
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        for s, out, st in zip(sets, outs, streams):
            enc.embed_into(s, out.data_ptr(), layout, st.cuda_stream)
        torch.cuda.synchronize()
        assert all(torch.equal(out.view(bits), w) for out, w in zip(outs, want))
