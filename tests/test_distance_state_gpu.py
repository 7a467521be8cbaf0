"""What sets keep for the distances, after calls that fail and under graph capture, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from conftest import rand_seqs

pytestmark = pytest.mark.gpu


def into(name, a, b, out):
    import torch
    from seqtree_b200 import device
    getattr(device, name + "_into")(a, b, out.data_ptr(), torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("warm", [None, "levenshtein"])
def test_a_refused_capture_leaves_nothing_behind(cuda_ready, warm):
    """A first Hamming call inside a graph capture is refused, whether or not a Levenshtein call
    has met the sets; eager calls after it are right."""
    import torch
    from seqtree_b200 import device
    rng = np.random.default_rng(9)
    sa, sb = rand_seqs(rng, 40, 19, 19, "ACGT"), rand_seqs(rng, 55, 19, 19, "ACGT")
    a, b = device.SeqSet(sa, None), device.SeqSet(sb, None)
    out = torch.full((40, 55), -1, dtype=torch.int32, device="cuda")
    if warm:
        into(warm, a, b, out)
    torch.cuda.synchronize()
    with pytest.raises(ValueError, match="before capturing"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            into("hamming", a, b, out)
    for name in ("hamming", "levenshtein"):
        out.fill_(-1)
        into(name, a, b, out)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), getattr(oracle, name + "_matrix")(sa, sb))
