"""Gap-block calls over one pair of resident sets with different arguments: at once on two streams, and
beside a captured one that is replayed in between."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from conftest import rand_seqs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def data(cuda_ready):
    from seqtree_b200 import SubstitutionMatrix, device, gapblock
    rng = np.random.default_rng(21)
    q, r = rand_seqs(rng, 500, 8, 25), rand_seqs(rng, 20000, 8, 25)
    args = []  # (matrix, gap_open, cube): narrow and wide penalties, with and without a prior
    wide = SubstitutionMatrix.from_similarity(np.where(np.eye(24, dtype=int) == 1, 100, -100))
    for m in (SubstitutionMatrix.blosum62(), SubstitutionMatrix.structural(), SubstitutionMatrix.pam250(),
              SubstitutionMatrix.blosum45(), SubstitutionMatrix.blosum80(), wide, None):
        for lam in (None, 21):
            args.append((m, 8 + len(args), () if lam is None else
                         gapblock.prior_cube(gapblock.central_prior(lam), 25)))
    return q, r, device.SeqSet(q), device.SeqSet(r), args


def call(data, i, out, stream):
    from seqtree_b200 import device
    _, _, a, b, args = data
    m, go, cube = args[i]
    device.gapblock_into(a, b, out.data_ptr(), stream.cuda_stream, matrix=m, gap_open=go, prior=cube,
                         prior_width=25 if len(cube) else 0)


def want(data, i, rows):
    q, r, _, _, args = data
    m, go, cube = args[i]
    pen = 1 - np.eye(24, dtype=np.int32) if m is None else m.penalty_grid
    return oracle.gapblock_matrix([q[k] for k in rows], r, pen, gap_open=go, gap_extend=1, prior=cube,
                                  prior_width=25 if len(cube) else 0, threads=8)


def test_two_streams(data):
    """More argument sets than a query set keeps profiles for, in pairs at once."""
    import torch
    streams = [torch.cuda.Stream() for _ in range(2)]
    n = len(data[4])
    outs = [torch.zeros((500, 20000), dtype=torch.int32, device="cuda") for _ in range(n)]
    rows = list(range(0, 500, 50))
    for turn in range(3):  # the first turn tunes
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        for i in range(n):
            call(data, (i * 5) % n, outs[(i * 5) % n], streams[i % 2])
        torch.cuda.synchronize()
        for i in range(n):
            assert np.array_equal(outs[i][rows].cpu().numpy(), want(data, i, rows)), (turn, i)


def test_replays_between_other_calls(data):
    """A captured call keeps its tables, profile and plan while calls with other arguments come by; one
    whose profile would change hands is refused and works eagerly."""
    import torch
    from seqtree_b200 import device
    q, r, _, _, args = data
    mine = (q, r, device.SeqSet(q), device.SeqSet(r), args)
    cur = torch.cuda.current_stream()
    out, other = (torch.zeros((500, 20000), dtype=torch.int32, device="cuda") for _ in range(2))
    rows = list(range(7, 500, 60))
    call(mine, 1, out, cur)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(mine, 1, out, torch.cuda.current_stream())
    expect = want(mine, 1, rows)
    for i in list(range(len(args))) * 2:
        call(mine, i, other, cur)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(other[rows].cpu().numpy(), want(mine, i, rows)), i
        assert np.array_equal(out[rows].cpu().numpy(), expect), i
    call(mine, len(args) - 1, other, cur)
    with pytest.raises(ValueError, match="before capturing"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            call(mine, len(args) - 1, other, torch.cuda.current_stream())
    other.zero_()
    call(mine, len(args) - 1, other, cur)
    torch.cuda.synchronize()
    assert np.array_equal(other[rows].cpu().numpy(), want(mine, len(args) - 1, rows))
