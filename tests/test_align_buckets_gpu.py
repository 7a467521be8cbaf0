"""The query-pair wavefront's two row-bucket widths."""
from __future__ import annotations

import os

import numpy as np
import pytest

import oracle
from conftest import as_np, rand_seqs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["global", "local"])
def test_both_widths_are_measured(cuda_ready, mode):
    """Few queries spread over every bucket (lengths at and beside the 32- and 64-row edges): the first
    call of the shape runs and times both widths, the last one's result is the oracle's."""
    from seqtree_b200 import SubstitutionMatrix, _lib, pairwise
    m = SubstitutionMatrix.blosum62()
    rng = np.random.default_rng(12)
    lens = [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200, 256, 257, 384, 448, 449, 511]
    q = [rand_seqs(rng, 1, L, L)[0] for L in lens]
    r = rand_seqs(rng, 31, 1, 507)
    got = as_np(pairwise.score_matrix(q, r, m, mode=mode, gap_open=1, gap_extend=3))
    assert _lib.last_kernel_name() == "gotoh_qpair_kernel"
    want = oracle.align_matrix(q, r, m.similarity_grid, mode=mode, gap_open=1, gap_extend=3,
                               threads=os.cpu_count() or 1)
    assert np.array_equal(got, want)
    if os.environ.get("SEQTREE_B200_TUNE") != "0":
        line = [t for t in _lib.tuning_table().splitlines() if f"wave|{int(mode == 'local')}|0|24|511|" in t]
        assert any("wW" in t and " 1:" in t for t in line), line
