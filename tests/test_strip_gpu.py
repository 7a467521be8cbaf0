"""The strip kernel of the alignment matrices (gotoh_strip.cu) against the oracle, at the edges of
its strips, code words and groups.  The first call of a shape runs every kernel that can take it, the
strip kernel last, so its result is the strip kernel's."""
from __future__ import annotations

import os

import numpy as np
import pytest

import oracle
from conftest import as_np, rand_seqs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def B62(cuda_ready):
    from seqtree_b200 import SubstitutionMatrix
    return SubstitutionMatrix.blosum62()


def check(q, r, matrix, mode, go, ge, dist, alphabet="aa"):
    from seqtree_b200 import _lib, pairwise
    fn = pairwise.dist_matrix if dist else pairwise.score_matrix
    got = as_np(fn(q, r, matrix, mode=mode, gap_open=go, gap_extend=ge, alphabet=alphabet))
    if os.environ.get("SEQTREE_B200_TUNE") != "0":
        assert _lib.last_kernel_name() == "gotoh_strip_kernel"
    want = oracle.align_matrix(q, r, matrix.similarity_grid, mode=mode, gap_open=go, gap_extend=ge,
                               dist=dist, alphabet=alphabet, threads=os.cpu_count() or 1)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("mode", ["global", "local"])
@pytest.mark.parametrize("m", [1, 4, 5, 31, 32, 33, 47, 48, 49, 96, 97, 144, 145, 509, 512])
def test_strip_heights(B62, mode, m):
    """Queries at the strip edges (one more and one less residue beside them, an odd count) against
    refs of 1 to m + 3 residues, 33 of them (two groups, the second with one lane)."""
    rng = np.random.default_rng(m)
    q = [rand_seqs(rng, 1, L, L)[0] for L in (m, max(1, m - 1), max(1, m // 2))]
    r = rand_seqs(rng, 30, 1, min(512, m + 3)) + rand_seqs(rng, 3, min(512, m + 3), min(512, m + 3))
    check(q, r, B62, mode, 11, 1, m % 2 == 0)


@pytest.mark.parametrize("mode", ["global", "local"])
@pytest.mark.parametrize("go,ge,hi", [(7, 7, 21), (0, 0, 22), (3, 0, 23), (900, 30, 24), (4000, 8, 57),
                                      (60, 10, 121)])
def test_gap_costs(B62, mode, go, ge, hi):
    """Linear, free and dear gaps, up to costs near the int16 bound."""
    rng = np.random.default_rng(hi)
    q, r = rand_seqs(rng, 7, 1, hi), rand_seqs(rng, 70, 1, hi)
    q[0], r[0] = rand_seqs(rng, 2, hi, hi)
    check(q, r, B62, mode, go, ge, True)


@pytest.mark.parametrize("mode", ["global", "local"])
@pytest.mark.parametrize("alphabet,symbols,size", [("nt", "ACGT", 4), ("iupac", "ACGTRYSWKMBDHVN", 15)])
def test_small_alphabets_and_matrices_with_negative_diagonals(cuda_ready, mode, alphabet, symbols, size):
    """A random matrix (own scores below others', negative ones among them), so the self scores of
    the distance take the recurrence and not the sum over the diagonal."""
    from seqtree_b200 import SubstitutionMatrix
    rng = np.random.default_rng(size)
    grid = rng.integers(-6, 8, size=(size, size))
    grid = (grid + grid.T) // 2
    m = SubstitutionMatrix.from_similarity(grid)
    hi = 37 + size
    q, r = rand_seqs(rng, 9, 1, hi, symbols), rand_seqs(rng, 40, 1, hi, symbols)
    q[0], r[0] = rand_seqs(rng, 2, hi, hi, symbols)
    check(q, r, m, mode, 5, 2, True, alphabet)


def test_self_scores_of_unplain_residues(B62):
    """X scores below 0 against itself: sequences with it take the self scores' recurrence, up to
    512 residues, beside plain ones."""
    rng = np.random.default_rng(3)
    q = rand_seqs(rng, 6, 300, 510, "ACDEFX") + rand_seqs(rng, 3, 1, 40) + ["X", "XX"]
    r = rand_seqs(rng, 5, 1, 60, "WX") + rand_seqs(rng, 5, 400, 512)
    for mode in ("global", "local"):
        for go, ge in ((11, 1), (1, 3)):
            from seqtree_b200 import pairwise
            got = as_np(pairwise.dist_matrix(q, r, B62, mode=mode, gap_open=go, gap_extend=ge))
            want = oracle.align_matrix(q, r, B62.similarity_grid, mode=mode, gap_open=go,
                                       gap_extend=ge, dist=True, threads=os.cpu_count() or 1)
            assert np.array_equal(got, want)


def test_streams_and_capture(B62):
    """Multi-strip calls enqueued on two streams at once (each with its own scratch), and a captured
    call replayed: the results of separate calls."""
    import torch
    from seqtree_b200 import device
    rng = np.random.default_rng(11)
    sets = [(device.SeqSet(rand_seqs(rng, 300, 60, 160)), device.SeqSet(rand_seqs(rng, 500, 60, 160)))
            for _ in range(2)]
    want, outs = [], [torch.zeros((300, 500), dtype=torch.int32, device="cuda") for _ in sets]

    def call(i, out, stream):
        device.align_into(*sets[i], out.data_ptr(), stream, matrix=B62, mode="global", gap_open=11,
                          gap_extend=1)

    for i in range(2):
        out = torch.zeros_like(outs[i])
        for _ in range(2):
            call(i, out, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        want.append(out)
    streams = [torch.cuda.Stream() for _ in sets]
    for _ in range(4):
        for i, s in enumerate(streams):
            call(i, outs[i], s.cuda_stream)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(outs, want))
    graph = torch.cuda.CUDAGraph()
    outs[0].zero_()
    with torch.cuda.graph(graph):
        call(0, outs[0], torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        outs[0].zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(outs[0], want[0])
