"""Sparse gap-block rows whose per-(m, n) term (prior minimum + gap cost) is far from 0, against the
thresholded dense matrix: the sums the sparse tile keeps are then larger than the threshold."""
from __future__ import annotations

import os

import numpy as np
import pytest

import oracle
from conftest import rand_seqs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def stb(cuda_ready):
    import seqtree_b200
    return seqtree_b200


def dense_and_rows(q, r, m, thresholds, go, ge, cube, width):
    """The dense device matrix, and (threshold, indptr, ref ids, scores) of each sparse call."""
    import torch
    from seqtree_b200 import _lib, device
    qs, rs = device.SeqSet(q), device.SeqSet(r)
    out = torch.empty((len(q), len(r)), dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    kw = dict(matrix=m, gap_open=go, gap_extend=ge, prior=cube, prior_width=width)
    device.gapblock_into(qs, rs, out.data_ptr(), stream, **kw)
    dense = out.cpu().numpy()
    hits, rows = device.Hits(), []
    for t in thresholds:
        device.gapblock_sparse_into(qs, rs, hits, stream, max_penalty=t, **kw)
        assert _lib.last_kernel_name() == "gapblock_fast_kernel<sparse>"
        rows.append((t, *hits.to_host()))
    return dense, rows


def check_rows(dense, rows):
    for t, indptr, ids, scores in rows:
        keep = dense <= t
        assert np.array_equal(indptr, np.r_[0, np.cumsum(keep.sum(1))]), t
        assert np.array_equal(ids, np.nonzero(keep)[1]), t
        assert np.array_equal(scores, dense[keep]), t


@pytest.mark.parametrize("low", [-9, -240, -7000])
@pytest.mark.parametrize("hi", [25, 64])
def test_priors_below_zero(stb, low, hi):
    """Raw prior cubes with negative cells: a hit's sum exceeds its threshold by up to |low|, more
    than a byte holds from -240 on."""
    rng = np.random.default_rng(-low + hi)
    q, r = rand_seqs(rng, 41, 6, hi), rand_seqs(rng, 700, 6, hi)
    m = stb.SubstitutionMatrix.blosum62()
    cube = rng.integers(low, 20, size=(hi + 1) ** 3).astype(np.int32)
    dense, rows = dense_and_rows(q, r, m, (0, 24, 250, 255, 256), 8, 1, cube, hi)
    want = oracle.gapblock_matrix(q, r, m.penalty_grid, gap_open=8, gap_extend=1, prior=cube,
                                  prior_width=hi, threads=os.cpu_count() or 1)
    assert np.array_equal(dense, want)
    check_rows(dense, rows)


@pytest.mark.parametrize("below", [0, 5, 60, 3000])
@pytest.mark.parametrize("t", [0, 24, 300, 2 ** 31 - 1])
def test_terms_at_the_end_of_int32(stb, below, t):
    """A gap cost so near 2^31 that a score wraps below 0 for some sums and not for others: the rows
    are still those of the dense matrix, which wraps as the reference's int32 arithmetic does."""
    rng = np.random.default_rng(below)
    q, r = rand_seqs(rng, 33, 8, 25), rand_seqs(rng, 600, 8, 25)
    dense, rows = dense_and_rows(q, r, stb.SubstitutionMatrix.blosum62(), (t,), 2 ** 31 - 1 - below, 1, (), 0)
    assert below == 3000 or (dense < 0).any()
    check_rows(dense, rows)
