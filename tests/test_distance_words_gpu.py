"""The bit-vector Levenshtein kernel at the edges of its word counts, and the distance codes that sets
keep, against the oracle."""
from __future__ import annotations

import os

import numpy as np
import pytest

import oracle
from conftest import AA20, as_np, rand_seqs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest", [1, 31, 32, 33, 64, 65, 96, 97, 128, 129, 192, 193, 256, 257, 384,
                                     385, 512])
def test_pattern_words(cuda_ready, longest):
    """Refs up to each word count's last bit and one past it, text longer and shorter than them; the
    count of rows is odd and the last warp of columns partly filled."""
    from seqtree_b200 import _lib, distance
    rng = np.random.default_rng(longest)
    a = rand_seqs(rng, 33, 0, longest + 9, "ACGT")
    b = rand_seqs(rng, 40, 0, longest, "ACGT") + ["A" * longest, "ACGT" * (longest // 4 + 1)][:1]
    got = as_np(distance.levenshtein_matrix(a, b))
    assert _lib.last_kernel_name() == "levenshtein_kernel"
    assert np.array_equal(got, oracle.levenshtein_matrix(a, b, threads=os.cpu_count() or 1))


def test_many_rows_per_block(cuda_ready):
    """Enough rows that a block takes more than sixteen of them."""
    from seqtree_b200 import distance
    rng = np.random.default_rng(5)
    a, b = rand_seqs(rng, 9001, 8, 25), rand_seqs(rng, 6000, 8, 25)
    got = as_np(distance.levenshtein_matrix(a, b))
    rows = np.r_[0:40, 4480:4500, 8990:9001]
    want = oracle.levenshtein_matrix([a[i] for i in rows], b, threads=os.cpu_count() or 1)
    assert np.array_equal(got[rows], want)


def test_sets_shared_between_partners_and_calls(cuda_ready):
    """Sets keep their codes: the same set with partners over the same and over other symbols, as
    both sides, under both distances and on two streams, always gives the oracle's matrix."""
    import torch
    from seqtree_b200 import device
    rng = np.random.default_rng(6)
    strings = {n: rand_seqs(rng, c, 12, 12, s) for n, c, s in
               (("x", 50, "ACGT"), ("y", 60, "ACGT"), ("n", 33, "ACGTN"), ("p", 41, AA20), ("u", 20, "A"))}
    sets = {n: device.SeqSet(s, None) for n, s in strings.items()}
    streams = [torch.cuda.current_stream(), torch.cuda.Stream()]
    turn = 0
    for _ in range(2):
        for a, b in ("xy", "xn", "xy", "yx", "xx", "xp", "pu", "ux", "nn", "xy"):
            for name in ("hamming", "levenshtein"):
                out = torch.full((len(strings[a]), len(strings[b])), -1, dtype=torch.int32, device="cuda")
                torch.cuda.synchronize()
                turn += 1
                getattr(device, name + "_into")(sets[a], sets[b], out.data_ptr(),
                                                streams[turn % 2].cuda_stream)
                torch.cuda.synchronize()
                want = getattr(oracle, name + "_matrix")(strings[a], strings[b])
                assert np.array_equal(out.cpu().numpy(), want), (a, b, name)
