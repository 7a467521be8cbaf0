"""Calls that use the library's shared scratch and tables, on two streams at once with different
arguments: each gives what it gives alone."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rand_seqs

pytestmark = pytest.mark.gpu


def calls(name):
    """Two calls (function of (out pointer, stream)) over shapes (nq, nr), and the kernel that runs."""
    from seqtree_b200 import SubstitutionMatrix, device
    rng = np.random.default_rng(7)
    ms = (SubstitutionMatrix.blosum62(), SubstitutionMatrix.pam250())
    if name == "exact":  # alignments past 512 residues: DP rows and self scores
        q, r = (device.SeqSet(rand_seqs(rng, n, 513, 640)) for n in (40, 50))
        return 40, 50, "gotoh_exact_kernel", [
            lambda o, s, m=m: device.align_into(q, r, o, s, matrix=m, dist=True) for m in ms]
    if name == "general":  # gap blocks past 64 residues: penalties
        q, r = (device.SeqSet(rand_seqs(rng, n, 65, 300)) for n in (300, 700))
        return 300, 700, "gapblock_general_kernel", [
            lambda o, s, m=m: device.gapblock_into(q, r, o, s, matrix=m, gap_open=8) for m in ms]
    pairs = [tuple(device.SeqSet(rand_seqs(rng, n, 513, 600, "ACGT"), None) for n in (60, 70)) for _ in ms]
    return 60, 70, "levenshtein_dp_kernel", [lambda o, s, p=p: device.levenshtein_into(*p, o, s) for p in pairs]


@pytest.mark.parametrize("name", ["exact", "general", "levenshtein"])
def test_two_streams(cuda_ready, name):
    import torch
    from seqtree_b200 import _lib
    nq, nr, kernel, two = calls(name)
    outs = [torch.zeros((nq, nr), dtype=torch.int32, device="cuda") for _ in two]
    want = []
    for call, out in zip(two, outs):
        call(out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        want.append(out.clone())
    streams = [torch.cuda.Stream() for _ in two]
    for _ in range(6):
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        for call, out, s in zip(two, outs, streams):
            call(out.data_ptr(), s.cuda_stream)
            assert _lib.last_kernel_name() == kernel
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outs, want))


def test_a_captured_levenshtein_past_512(cuda_ready):
    """The scratch's turn inside a captured call, replayed after other calls of its kind."""
    import torch
    nq, nr, _, two = calls("levenshtein")
    out, other = (torch.zeros((nq, nr), dtype=torch.int32, device="cuda") for _ in range(2))
    two[0](out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        two[0](out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    stream = torch.cuda.Stream()
    for _ in range(3):
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        two[1](other.data_ptr(), stream.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
