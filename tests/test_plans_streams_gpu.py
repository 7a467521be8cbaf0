"""Plans of resident sets made on one stream and read on another, at once, and plans that come and go."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rand_seqs

pytestmark = pytest.mark.gpu


def calls(a, b, raw_a, raw_b, m):
    """name -> (function of (out pointer, stream), shape): the first call on sets makes their plans."""
    from seqtree_b200 import device
    return {
        "gapblock": lambda out, st: device.gapblock_into(a, b, out, st, matrix=m, gap_open=8),
        "strip": lambda out, st: device.align_into(a, b, out, st, matrix=m, dist=True),
        "wave": lambda out, st: device.align_into(a, b, out, st, matrix=m, gap_open=1, gap_extend=3),
        "hamming": lambda out, st: device.hamming_into(raw_a, raw_b, out, st),
        "levenshtein": lambda out, st: device.levenshtein_into(raw_a, raw_b, out, st),
    }


@pytest.mark.parametrize("name", ["gapblock", "strip", "wave", "hamming", "levenshtein"])
def test_a_second_stream_waits_for_the_plans(cuda_ready, name):
    """The plan's stream is busy when the plan is enqueued; a call on another stream follows at once."""
    import torch
    from seqtree_b200 import SubstitutionMatrix, device
    m = SubstitutionMatrix.blosum62()
    rng = np.random.default_rng(4)
    qa, ra = rand_seqs(rng, 300, 12, 12), rand_seqs(rng, 700, 12, 12)
    lens = (40, 90) if name == "wave" else (8, 25)
    q, r = rand_seqs(rng, 300, *lens), rand_seqs(rng, 700, *lens)

    def fresh():
        return calls(device.SeqSet(q), device.SeqSet(r), device.SeqSet(qa, None), device.SeqSet(ra, None), m)[name]

    outs = [torch.zeros((300, 700), dtype=torch.int32, device="cuda") for _ in range(2)]
    warm = fresh()
    for _ in range(3):
        warm(outs[0].data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = outs[0].clone()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(3):
        call = fresh()
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(one):
            torch.cuda._sleep(20_000_000)
        call(outs[0].data_ptr(), one.cuda_stream)
        call(outs[1].data_ptr(), two.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(outs[0], want) and torch.equal(outs[1], want)


def test_plans_that_come_and_go(cuda_ready):
    """Sets used once and dropped: their plans' memory goes back (the library keeps 256 MiB at most) and
    the next sets' results are right."""
    import torch
    from seqtree_b200 import SubstitutionMatrix, device
    m = SubstitutionMatrix.blosum62()
    rng = np.random.default_rng(5)
    q, r = rand_seqs(rng, 4000, 8, 25), rand_seqs(rng, 90000, 8, 25)
    out = torch.zeros((4000, 90000), dtype=torch.int32, device="cuda")
    want, free = None, []
    for _ in range(12):
        out.zero_()
        device.gapblock_into(device.SeqSet(q), device.SeqSet(r), out.data_ptr(),
                             torch.cuda.current_stream().cuda_stream, matrix=m, gap_open=8)
        torch.cuda.synchronize()
        want = out.clone() if want is None else want
        assert torch.equal(out, want)
        free.append(torch.cuda.mem_get_info()[0])
    assert free[1] - free[-1] <= 300 << 20
