"""Alignment calls on two streams at once over the same sets, with different matrices, gap costs and
modes: each gives what it gives alone, whichever kernel takes it."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rand_seqs

pytestmark = pytest.mark.gpu

# (lengths, sizes, the two calls' gap costs, kernel): strips take gap_extend <= gap_open at sizes that
# fill the GPU, the wavefront the other order past 32 residues
SETTINGS = {
    "strip": (60, 160, 900, 1100, ((11, 1), (7, 2)), "gotoh_strip_kernel"),
    "strip_short": (8, 25, 3000, 6000, ((11, 1), (7, 2)), "gotoh_strip_kernel"),
    "wave": (60, 160, 400, 500, ((1, 3), (2, 5)), "gotoh_qpair_kernel"),
}


@pytest.mark.parametrize("dist", [True, False])
@pytest.mark.parametrize("setting", list(SETTINGS))
def test_two_calls_at_once(cuda_ready, setting, dist):
    import torch
    from seqtree_b200 import SubstitutionMatrix, _lib, device
    lo, hi, nq, nr, gaps, kernel = SETTINGS[setting]
    rng = np.random.default_rng(nq)
    q, r = device.SeqSet(rand_seqs(rng, nq, lo, hi)), device.SeqSet(rand_seqs(rng, nr, lo, hi))
    matrices = (SubstitutionMatrix.blosum62(), SubstitutionMatrix.pam250())
    outs = [torch.zeros((nq, nr), dtype=torch.int32, device="cuda") for _ in gaps]

    def call(i, stream):
        device.align_into(q, r, outs[i].data_ptr(), stream.cuda_stream, matrix=matrices[i], mode="global",
                          gap_open=gaps[i][0], gap_extend=gaps[i][1], dist=dist)
        assert _lib.last_kernel_name() == kernel

    want = []
    for i in range(2):
        for _ in range(2):
            device.align_into(q, r, outs[i].data_ptr(), torch.cuda.current_stream().cuda_stream,
                              matrix=matrices[i], mode="global", gap_open=gaps[i][0], gap_extend=gaps[i][1],
                              dist=dist)
        torch.cuda.synchronize()
        want.append(outs[i].clone())
    streams = [torch.cuda.Stream() for _ in gaps]
    for _ in range(6):
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        for i, s in enumerate(streams):
            call(i, s)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outs, want))


def test_more_matrices_than_are_kept(cuda_ready):
    """More matrices in turn than a device keeps: each call's own, the first again at the end."""
    import oracle
    from seqtree_b200 import SubstitutionMatrix, pairwise
    rng = np.random.default_rng(2)
    q, r = rand_seqs(rng, 5, 8, 40, "ACGT"), rand_seqs(rng, 40, 8, 40, "ACGT")
    grids = []
    for _ in range(1030):
        g = rng.integers(-4, 6, size=(4, 4))
        grids.append((g + g.T) // 2)
    for g in grids + grids[:2] + grids[-8:]:
        m = SubstitutionMatrix.from_similarity(g)
        got = np.asarray(pairwise.dist_matrix(q, r, m, gap_open=5, gap_extend=2, alphabet="nt"))
        want = oracle.align_matrix(q, r, m.similarity_grid, mode="global", gap_open=5, gap_extend=2, dist=True,
                                   alphabet="nt")
        assert np.array_equal(got, want)
