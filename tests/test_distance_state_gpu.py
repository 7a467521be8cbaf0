"""What sets keep for the distances, after calls that fail and under graph capture, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from conftest import rand_seqs

pytestmark = pytest.mark.gpu


def into(name, a, b, out):
    import torch
    from seqtree_b200 import device
    getattr(device, name + "_into")(a, b, out.data_ptr(), torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("warm", [None, "levenshtein"])
def test_a_refused_capture_leaves_nothing_behind(cuda_ready, warm):
    """A first Hamming call inside a graph capture is refused, whether or not a Levenshtein call
    has met the sets; eager calls after it are right."""
    import torch
    from seqtree_b200 import device
    rng = np.random.default_rng(9)
    sa, sb = rand_seqs(rng, 40, 19, 19, "ACGT"), rand_seqs(rng, 55, 19, 19, "ACGT")
    a, b = device.SeqSet(sa, None), device.SeqSet(sb, None)
    out = torch.full((40, 55), -1, dtype=torch.int32, device="cuda")
    if warm:
        into(warm, a, b, out)
    torch.cuda.synchronize()
    with pytest.raises(ValueError, match="before capturing"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            into("hamming", a, b, out)
    for name in ("hamming", "levenshtein"):
        out.fill_(-1)
        into(name, a, b, out)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), getattr(oracle, name + "_matrix")(sa, sb))


SYMBOLS = {"acgt": "ACGT", "acgtn": "ACGTN", "aa": "ACDEFGHIKLMNPQRSTVWY", "two": "AC", "lower": "acgt",
           "digits": "0123456789", "all": "".join(map(chr, range(33, 90))), "gap": "ACGT-", "rna": "ACGU",
           "soft": "ACGTacgt", "iupac": "ACGTRYSWKMBDHVN", "binary": "01"}


def sets_of(rng, count, length=21):
    from seqtree_b200 import device
    strings = {n: rand_seqs(rng, count + 7 * i, length, length, s) for i, (n, s) in enumerate(SYMBOLS.items())}
    return strings, {n: device.SeqSet(s, None) for n, s in strings.items()}


@pytest.mark.parametrize("name", ["hamming", "levenshtein"])
def test_a_captured_call_keeps_its_alphabet(cuda_ready, name):
    """A captured A x B call replayed after A and B have met sets over other symbols, more of them than a
    set keeps packed words for; each of those calls is right too, on either side."""
    import torch
    strings, sets = sets_of(np.random.default_rng(10), 37)
    want = getattr(oracle, name + "_matrix")(strings["acgt"], strings["two"])
    out = torch.full(want.shape, -1, dtype=torch.int32, device="cuda")
    into(name, sets["acgt"], sets["two"], out)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        into(name, sets["acgt"], sets["two"], out)
    for _ in range(2):
        for other in SYMBOLS:
            for a, b in ((other, "acgt"), ("acgt", other), ("two", other)):
                got = torch.full((len(strings[a]), len(strings[b])), -1, dtype=torch.int32, device="cuda")
                into(name, sets[a], sets[b], got)
                torch.cuda.synchronize()
                assert np.array_equal(got.cpu().numpy(),
                                      getattr(oracle, name + "_matrix")(strings[a], strings[b])), (a, b)
            out.fill_(-1)
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), want), other


@pytest.mark.parametrize("name", ["hamming", "levenshtein"])
def test_changing_partners_waits_for_no_other_stream(cuda_ready, name):
    """A set that meets partners over different symbols in turn, while another stream is busy."""
    import torch
    strings, sets = sets_of(np.random.default_rng(11), 33)
    outs = {b: torch.zeros((33, len(strings[b])), dtype=torch.int32, device="cuda") for b in strings}
    for b in strings:
        into(name, sets["acgt"], sets[b], outs[b])
    torch.cuda.synchronize()
    busy = torch.cuda.Stream()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(1_500_000_000)
    for b in ("aa", "acgt", "lower", "aa"):
        into(name, sets["acgt"], sets[b], outs[b])
    assert not busy.query()
    torch.cuda.synchronize()


def test_a_raw_set_takes_its_own_bytes(cuda_ready):
    """Device memory of a set of 256 MiB: its bytes and the allocator's 2 MiB granules, no room for forms
    that only some calls make."""
    import torch
    from seqtree_b200 import device
    device.SeqSet(["ACGT"], None)
    strings = ["ACGT" * (1 << 20)] * 64
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    kept = device.SeqSet(strings, None)
    assert before - torch.cuda.mem_get_info()[0] <= (256 + 16) << 20
    del kept
