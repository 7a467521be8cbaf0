"""The fast gap-block kernel at the edges of its tiles against the oracle: partly filled quads,
slices, warp tasks and chunks, lengths mixed inside a warp, 8- and 16-bit penalty words, 8- and
16-bit sparse scores, and thresholds that let the sparse sweep end early or keep every cell."""
from __future__ import annotations

import os

import numpy as np
import pytest

import oracle
from conftest import as_np, prior_by_name, rand_seqs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def stb(cuda_ready):
    import seqtree_b200
    return seqtree_b200


def peak_matrix(stb, peak):
    """Amino-acid penalties spread up to ``peak`` (of the residues Z and X, beside the others)."""
    i, j = np.meshgrid(np.arange(24), np.arange(24), indexing="ij")
    sim = -((i + j + 1) * (peak // 2) // 44) * (i != j)
    sim[21:23, 21:23] = [[peak % 2, -(peak // 2)], [-(peak // 2), 0]]
    sim[23] = sim[:, 23] = 0  # '*' beside anything: no penalty but the own score's
    return stb.SubstitutionMatrix.from_similarity(np.clip(sim, -(peak // 2), None))


def check(stb, q, r, m, prior_name, thresholds, kernel="gapblock_fast_kernel", go=8, ge=1):
    from seqtree_b200 import _lib, gapblock
    prior = prior_by_name(prior_name)
    w = max(map(len, q + r))
    cube = gapblock.prior_cube(prior, w) if prior else []
    pen = 1 - np.eye(24, dtype=np.int32) if m is None else m.penalty_grid
    want = oracle.gapblock_matrix(q, r, pen, gap_open=go, gap_extend=ge, prior=cube,
                                  prior_width=w if prior else 0, threads=os.cpu_count() or 1)
    got = as_np(stb.score_matrix(q, r, m, gap_open=go, gap_extend=ge, gap_prior=prior))
    assert _lib.last_kernel_name() == kernel
    assert np.array_equal(got, want)
    for t in thresholds:
        sp = gapblock.score_sparse(q, r, t, m, gap_open=go, gap_extend=ge, gap_prior=prior)
        keep = want <= t
        assert np.array_equal(sp.indptr, np.r_[0, np.cumsum(keep.sum(1))])
        assert np.array_equal(sp.ref_ids, np.nonzero(keep)[1])
        assert np.array_equal(sp.scores, want[keep])


@pytest.mark.parametrize("prior", ["none", "central21"])
@pytest.mark.parametrize("nq,nr", [(1, 1), (3, 31), (4, 32), (5, 33), (16, 256), (17, 1023),
                                   (31, 1024), (33, 1025), (49, 2049)])
def test_partly_filled_tiles(stb, nq, nr, prior):
    rng = np.random.default_rng(nq * 10007 + nr)
    q, r = rand_seqs(rng, nq, 12, 12 + nq % 3), rand_seqs(rng, nr, 8, 25)
    r[: nr // 3] = [q[i % nq] for i in range(nr // 3)]  # hits, exact ones among them
    check(stb, q, r, stb.SubstitutionMatrix.blosum62(), prior, (0, 24, 60, 10 ** 6))


@pytest.mark.parametrize("prior", ["none", "frame21_5", "positions"])
@pytest.mark.parametrize("lo,hi", [(0, 0), (0, 3), (1, 64), (7, 64), (30, 33), (64, 64)])
def test_lengths_mixed_in_a_warp(stb, lo, hi, prior):
    """Few refs over a wide range of lengths: every warp task mixes lengths, tasks are cut where
    lengths differ by more than a task may hold, empty sequences included."""
    rng = np.random.default_rng(lo * 100 + hi)
    q, r = rand_seqs(rng, 37, lo, hi), rand_seqs(rng, 75, lo, hi)
    check(stb, q, r, stb.SubstitutionMatrix.blosum62(), prior, (8, 40))


@pytest.mark.parametrize("prior", ["none", "central21"])
@pytest.mark.parametrize("peak,hi", [(1, 30), (254, 32), (255, 32), (256, 31), (1000, 8), (8191, 1)])
def test_penalty_words(stb, peak, hi, prior):
    """Penalties at the 8-bit word's edge and beyond, and sums at the int16 bound (8,191)."""
    rng = np.random.default_rng(peak)
    symbols = "ACDEFGHIKLMNPQRSTVWYZX"
    q, r = rand_seqs(rng, 21, 1, hi, symbols), rand_seqs(rng, 300, 1, hi, symbols)
    m = peak_matrix(stb, peak) if peak > 1 else None
    if m is not None:
        assert m.penalty_grid.max() == peak and m.penalty_grid.min() == 0
    check(stb, q, r, m, prior, (4, 254, 255, 256, 2000, 30000))


def test_sparse_scores_do_not_depend_on_the_threshold(stb):
    """The early end of the sweep and the score width change with the threshold; the cells that
    pass two thresholds have the same scores under both."""
    from seqtree_b200 import gapblock
    rng = np.random.default_rng(8)
    q, r = rand_seqs(rng, 70, 8, 25, "ACDEF"), rand_seqs(rng, 3000, 8, 25, "ACDEF")
    m = stb.SubstitutionMatrix.structural()
    dense = as_np(stb.score_matrix(q, r, m, gap_open=8))
    for t in (0, 7, 16, 24, 100, 255, 256):
        got = gapblock.score_sparse(q, r, t, m, gap_open=8).to_dense(-1)
        assert np.array_equal(got, np.where(dense <= t, dense, -1))
