"""The kernel of a set's first alignment call, of later ones and of captured ones."""
from __future__ import annotations

import os

import numpy as np
import pytest

import oracle
from conftest import rand_seqs

pytestmark = pytest.mark.gpu


def matrices():
    from seqtree_b200 import SubstitutionMatrix
    return SubstitutionMatrix.blosum62(), SubstitutionMatrix.pam250()


def check(out, q, r, m, **kw):
    import torch
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), oracle.align_matrix(q, r, m.similarity_grid, mode="global", gap_open=11,
                                                                 gap_extend=1, threads=os.cpu_count() or 1, **kw))


def test_first_calls_are_measured_with_their_plans(cuda_ready):
    """The first call on new sets and later calls are tuned under keys of their own; all are right."""
    import torch
    from seqtree_b200 import _lib, device
    m, _ = matrices()
    rng = np.random.default_rng(3)
    q, r = rand_seqs(rng, 61, 9, 23), rand_seqs(rng, 505, 9, 23)
    out = torch.zeros((61, 505), dtype=torch.int32, device="cuda")
    for _ in range(2):  # the second pair of sets meets tuned shapes
        a, b = device.SeqSet(q), device.SeqSet(r)
        for _ in range(3):
            out.zero_()
            device.align_into(a, b, out.data_ptr(), torch.cuda.current_stream().cuda_stream, matrix=m, dist=True)
            check(out, q, r, m, dist=True)
    if os.environ.get("SEQTREE_B200_TUNE") != "0":
        lines = [t for t in _lib.tuning_table().splitlines() if "|0|1|24|23|23|5|8|" in t]
        assert any("|newqr" in t for t in lines) and any("|new" not in t for t in lines), lines


@pytest.mark.parametrize("lo,hi,nq,nr", [(9, 23, 61, 505), (60, 160, 40, 300), (9, 23, 900, 1100)])
def test_one_call_is_enough_before_a_capture(cuda_ready, lo, hi, nq, nr):
    """A call captured after a single eager one, on sets and with a matrix that no call met before."""
    import torch
    from seqtree_b200 import device
    rng = np.random.default_rng(nq)
    for m in matrices():
        for dist in (False, True):
            q, r = rand_seqs(rng, nq, lo, hi), rand_seqs(rng, nr, lo, hi)
            a, b = device.SeqSet(q), device.SeqSet(r)
            out = torch.zeros((nq, nr), dtype=torch.int32, device="cuda")

            def call():
                device.align_into(a, b, out.data_ptr(), torch.cuda.current_stream().cuda_stream, matrix=m,
                                  dist=dist)
            call()
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                call()
            out.zero_()
            graph.replay()
            check(out, q, r, m, dist=dist)


def test_large_shapes_are_measured_once(cuda_ready):
    """Beside a kernel of a millisecond the plans do not count: the first call's choice serves all later ones."""
    import torch
    from seqtree_b200 import _lib, device
    m, _ = matrices()
    rng = np.random.default_rng(5)
    a, b = device.SeqSet(rand_seqs(rng, 130, 150, 210)), device.SeqSet(rand_seqs(rng, 1500, 150, 211))
    out = torch.zeros((130, 1500), dtype=torch.int32, device="cuda")
    tables = []
    for _ in range(3):
        device.align_into(a, b, out.data_ptr(), torch.cuda.current_stream().cuda_stream, matrix=m)
        torch.cuda.synchronize()
        tables.append([t for t in _lib.tuning_table().splitlines() if "|0|0|24|" in t and "|7|10|" in t and "ms" in t])
    assert tables[0] == tables[1] == tables[2]
    if os.environ.get("SEQTREE_B200_TUNE") != "0":
        assert len(tables[0]) == 1
