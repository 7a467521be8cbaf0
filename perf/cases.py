"""Performance cases of the all-vs-all scoring framework.

Each case is one call that a user's program makes through the public entry points, at the sizes of
the named workloads (``seqtree_b200.workloads``) or of the ranges around them:

* ``gap_host``: ``gapblock.score_matrix`` on two Python lists, result in host memory;
* ``gap_device``: ``device.gapblock_into``, dense gap-block matrix of device-resident sets;
* ``sparse``: ``device.gapblock_sparse_into``, the thresholded CSR rows of device-resident sets;
* ``hamming`` / ``levenshtein``: the distance matrices of device-resident sets;
* ``align``: ``device.align_into``, Needleman-Wunsch / Smith-Waterman scores or distances;
* ``embed``: the encoder's bf16 embeddings of a device-resident set;
* ``train``: one forward and backward pass of the encoder on a batch of labelled pairs.

``listed`` gives the named cases, ``draw`` further ones of the same ranges, ``prepare`` what a
program holds before the call, ``run`` one call, ``work`` the bytes and operations the call cannot
do without, and ``exact`` the same outputs from plain torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from seqtree_b200 import SubstitutionMatrix, device, gapblock, learned, workloads
from seqtree_b200._lib import Packed

# Mean lengths of the generators' length laws (workloads.py), for operation counts.
_MEAN = {"skewed": 14.6, "protein": 203.0}
# Share of the sparse workload's pairs that score at most 24.
_HIT_SHARE = {"blosum62": 1.6e-4, "structural": 0.0275}


# ------------------------------------------------------------------------------- the cases ----
def listed():
    return [
        # An interactive query: a handful of junctions against a small panel.  Latency only.
        {"name": "gap_host_8x200", "kind": "gap_host", "nq": 8, "nr": 200, "lo": 10, "hi": 20,
         "matrix": "blosum62", "lam": 21},
        # The benchmark's headline configuration, as a Python user calls it.
        {"name": "gap_host_1000x10000", "kind": "gap_host", "nq": 1000, "nr": 10000, "lo": 10,
         "hi": 20, "matrix": "blosum62", "lam": 21},
        # A repertoire against a control panel on resident sets, dense, odd counts (rows of the
        # result are not 16-byte aligned), no prior: score_matrix's default.
        {"name": "gap_device_9973x50021", "kind": "gap_device", "nq": 9973, "nr": 50021, "lo": 8,
         "hi": 25, "matrix": "blosum62", "lam": -1},
        # The sparse configuration: a repertoire against a million-junction control, few hits.
        {"name": "sparse_100kx1m", "kind": "sparse", "nq": 100000, "nr": 1000000,
         "matrix": "blosum62", "max_penalty": 24},
        # The Hamming configuration: fixed-length nucleotide tags (barcodes).
        {"name": "hamming_acgt12_20k", "kind": "hamming", "nq": 20000, "nr": 20000,
         "alphabet": "ACGT", "lo": 12, "hi": 12},
        # The Levenshtein configuration: nucleotide reads of 30-60.
        {"name": "lev_acgt30_60_20k", "kind": "levenshtein", "nq": 20000, "nr": 20000,
         "alphabet": "ACGT", "lo": 30, "hi": 60},
        # Edit distances between junctions (amino acids, 8-25), ragged counts.
        {"name": "lev_aa8_25_5003x10007", "kind": "levenshtein", "nq": 5003, "nr": 10007,
         "alphabet": workloads.AA20, "lo": 8, "hi": 25},
        # The protein configuration: global alignment distances.
        {"name": "nw_dist_protein_4096", "kind": "align", "nq": 4096, "nr": 4096,
         "law": "protein", "lo": 0, "hi": 0, "mode": "global", "dist": True},
        # Local alignment scores of a smaller, odd-sized protein panel.
        {"name": "sw_score_protein_1501x4003", "kind": "align", "nq": 1501, "nr": 4003,
         "law": "protein", "lo": 0, "hi": 0, "mode": "local", "dist": False},
        # Alignment distances between junctions, the clustering input of a repertoire.
        {"name": "nw_dist_cdr3_4096", "kind": "align", "nq": 4096, "nr": 4096, "law": "cdr3",
         "lo": 10, "hi": 20, "mode": "global", "dist": True},
        # Embedding a repertoire for the learned search (bf16 inference).
        {"name": "embed_100k", "kind": "embed", "n": 100000},
        # One training batch of the encoder: loss and gradients (forward and backward).
        {"name": "train_2048_pairs", "kind": "train", "pairs": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gap_host", "gap_device", "sparse", "hamming", "levenshtein", "align",
                       "embed", "train"])
    if kind == "gap_host":
        lo = rng.randint(8, 12)
        return {"kind": kind, "nq": _log(rng, 1, 2000), "nr": _log(rng, 50, 20000), "lo": lo,
                "hi": lo + rng.randint(4, 14), "matrix": rng.choice(["blosum62", "structural", "pam250"]),
                "lam": rng.choice([-1, 21])}
    if kind == "gap_device":
        lo = rng.randint(6, 12)
        return {"kind": kind, "nq": _log(rng, 300, 10000), "nr": _log(rng, 3000, 50000), "lo": lo,
                "hi": lo + rng.randint(4, 20), "matrix": rng.choice(["blosum62", "structural", "unit"]),
                "lam": rng.choice([-1, 21])}
    if kind == "sparse":
        matrix = rng.choice(["blosum62", "structural"])
        nr = _log(rng, 20000, 1000000 if matrix == "blosum62" else 200000)
        return {"kind": kind, "nq": _log(rng, 1000, 50000 if matrix == "blosum62" else 10000),
                "nr": nr, "matrix": matrix, "max_penalty": rng.choice([16, 20, 24])}
    if kind == "hamming":
        n = rng.randint(6, 40)
        return {"kind": kind, "nq": _log(rng, 500, 20000), "nr": _log(rng, 500, 20000),
                "alphabet": rng.choice(["ACGT", workloads.AA20]), "lo": n, "hi": n}
    if kind == "levenshtein":
        if rng.random() < 0.5:
            lo = rng.randint(6, 14)
            hi, alphabet = lo + rng.randint(2, 16), workloads.AA20
        else:
            lo = rng.randint(20, 80)
            hi, alphabet = lo + rng.randint(10, 60), "ACGT"
        return {"kind": kind, "nq": _log(rng, 300, 10000), "nr": _log(rng, 1000, 20000),
                "alphabet": alphabet, "lo": lo, "hi": hi}
    if kind == "align":
        c = {"kind": kind, "nq": _log(rng, 64, 2000), "nr": _log(rng, 500, 4096),
             "law": rng.choice(["protein", "cdr3"]), "lo": 0, "hi": 0,
             "mode": rng.choice(["global", "local"]), "dist": rng.random() < 0.5}
        if c["law"] == "cdr3":
            c["lo"] = rng.randint(8, 12)
            c["hi"] = c["lo"] + rng.randint(4, 14)
        return c
    if kind == "embed":
        return {"kind": kind, "n": _log(rng, 1000, 200000)}
    return {"kind": "train", "pairs": _log(rng, 256, 4096)}


# ----------------------------------------------------------------------------- preparation ----
def _matrix(name):
    return None if name == "unit" else getattr(SubstitutionMatrix, name)()


def _gap_open(name):
    return 1 if name == "unit" else 8


def _junctions(seed, n):
    """The sparse workload's junctions, packed (no per-string Python work)."""
    codes, lens = workloads.cdr3_codes(seed, n)
    return Packed.from_arrays(*workloads.codes_to_letters(codes, lens))


def _strings(case, seed):
    """(queries, refs) as lists of str."""
    out = []
    for s, n in ((2 * seed + 1, case["nq"]), (2 * seed, case["nr"])):
        if case["kind"] in ("hamming", "levenshtein"):
            out.append(workloads.uniform_strings(s, n, case["lo"], case["hi"], case["alphabet"]))
        elif case.get("law") == "protein":
            out.append(workloads.proteins(s, n))
        else:
            out.append(workloads.cdr3(s, n, case["lo"], case["hi"]))
    return out


def _train_batch(case, seed):
    codes, lens = learned.training_pairs_codes(seed, case["pairs"])
    # labels from the same range as the exact scores of such pairs (near neighbours, then random)
    rng = np.random.default_rng(seed + 17)
    near = case["pairs"] // 2
    scores = rng.integers(40, 160, size=case["pairs"]).astype(np.int32)
    scores[:near] = rng.integers(4, 60, size=near)
    return codes, lens, scores


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "gap_host":
        st["q"], st["r"] = _strings(case, seed)
        st["prior"] = gapblock.central_prior(case["lam"]) if case["lam"] >= 0 else None
        st["matrix"] = _matrix(case["matrix"])
    elif kind == "gap_device":
        q, r = _strings(case, seed)
        st["q"], st["r"] = device.SeqSet(q), device.SeqSet(r)
        st["matrix"] = _matrix(case["matrix"])
        width = max(map(len, q + r))
        st["prior"] = gapblock.prior_cube(gapblock.central_prior(case["lam"]), width) \
            if case["lam"] >= 0 else ()
        st["width"] = width if case["lam"] >= 0 else 0
        st["out"] = torch.empty((case["nq"], case["nr"]), dtype=torch.int32, device="cuda")
    elif kind == "sparse":
        st["q"] = device.SeqSet(_junctions(2 * seed + 1, case["nq"]))
        st["r"] = device.SeqSet(_junctions(2 * seed, case["nr"]))
        st["matrix"] = _matrix(case["matrix"])
        st["hits"] = device.Hits()
        # the program's own buffers for the rows, larger than any set of this law fills (the rest
        # stays zero)
        room = 65536 + int(2 * _HIT_SHARE[case["matrix"]] * case["nq"] * case["nr"])
        st["ids"] = torch.zeros(room, dtype=torch.int32, device="cuda")
        st["scores"] = torch.zeros(room, dtype=torch.int32, device="cuda")
    elif kind in ("hamming", "levenshtein"):
        q, r = _strings(case, seed)
        st["q"], st["r"] = device.SeqSet(q, None), device.SeqSet(r, None)
        st["out"] = torch.empty((case["nq"], case["nr"]), dtype=torch.int32, device="cuda")
    elif kind == "align":
        q, r = _strings(case, seed)
        st["q"], st["r"] = device.SeqSet(q), device.SeqSet(r)
        st["matrix"] = SubstitutionMatrix.blosum62()
        st["out"] = torch.empty((case["nq"], case["nr"]), dtype=torch.int32, device="cuda")
    elif kind == "embed":
        st["enc"] = learned.Encoder(seed=seed)
        st["set"] = device.SeqSet(_junctions(seed, case["n"]))
        st["out"] = torch.empty((case["n"], 64), dtype=torch.bfloat16, device="cuda")
    elif kind == "train":
        st["enc"] = learned.Encoder(seed=seed)
        st["batch"] = _train_batch(case, seed)
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return st


# --------------------------------------------------------------------------------- one call ----
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gap_host":
        return np.asarray(gapblock.score_matrix(state["q"], state["r"], state["matrix"],
                                                gap_open=_gap_open(case["matrix"]),
                                                gap_prior=state["prior"]))
    if kind == "train":
        loss, grad = state["enc"].loss_grad(*state["batch"])
        return loss, grad
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "gap_device":
        device.gapblock_into(state["q"], state["r"], state["out"].data_ptr(), stream,
                             matrix=state["matrix"], gap_open=_gap_open(case["matrix"]),
                             prior=state["prior"], prior_width=state["width"])
    elif kind == "sparse":
        device.gapblock_sparse_into(state["q"], state["r"], state["hits"], stream,
                                    max_penalty=case["max_penalty"], matrix=state["matrix"],
                                    gap_open=8)
        indptr, ids, scores = device.hits_tensors(state["hits"])
        state["ids"][:ids.numel()].copy_(ids)
        state["scores"][:scores.numel()].copy_(scores)
        return indptr, state["ids"], state["scores"]
    elif kind == "hamming":
        device.hamming_into(state["q"], state["r"], state["out"].data_ptr(), stream)
    elif kind == "levenshtein":
        device.levenshtein_into(state["q"], state["r"], state["out"].data_ptr(), stream)
    elif kind == "align":
        device.align_into(state["q"], state["r"], state["out"].data_ptr(), stream,
                          matrix=state["matrix"], mode=case["mode"], dist=case["dist"])
    elif kind == "embed":
        state["enc"].embed_into(state["set"], state["out"].data_ptr(), 1, stream)
    return state["out"]


# ------------------------------------------------------------------------------------- work ----
def _mean_len(case):
    if case["kind"] == "sparse":
        return _MEAN["skewed"]
    if case.get("law") == "protein":
        return _MEAN["protein"]
    return 0.5 * (case["lo"] + case["hi"])


def _encoder_flops(sequences):
    """Multiply-adds x 2 of one forward pass on padded sequences of 32 positions."""
    per_row = 2 * (3 * 128 + 384 * 128 + 2 * (128 * 384 + 2 * 32 * 128 + 128 * 128))
    return sequences * (32 * per_row + 2 * 128 * 64)


def work(case):
    kind = case["kind"]
    if kind == "embed":
        return {"bytes": case["n"] * (_MEAN["skewed"] + 128), "flops": _encoder_flops(case["n"])}
    if kind == "train":
        params = 4 * 273_000
        return {"bytes": case["pairs"] * (2 * 32 + 12) + 2 * params,
                "flops": 3 * _encoder_flops(2 * case["pairs"])}
    nq, nr, length = case["nq"], case["nr"], _mean_len(case)
    pairs = nq * nr
    inputs = (nq + nr) * length
    if kind == "sparse":
        return {"bytes": inputs + 8 * nq + 8 * _HIT_SHARE[case["matrix"]] * pairs,
                "flops": pairs * 4 * 0.9 * length}
    if kind in ("gap_host", "gap_device"):
        # two table terms added and one minimum taken per block position of the shorter sequence
        return {"bytes": inputs + 4 * pairs, "flops": pairs * 4 * 0.9 * length}
    if kind == "hamming":
        per = 16 if case["alphabet"] == "ACGT" else 6
        return {"bytes": inputs + 4 * pairs, "flops": pairs * 4 * math.ceil(length / per)}
    if kind == "levenshtein":
        # the bit-vector recurrence: ten word operations per text symbol and 32 pattern rows
        return {"bytes": inputs + 4 * pairs, "flops": pairs * 10 * length * math.ceil(length / 32)}
    # three maxima with their additions per cell of the affine recurrence
    return {"bytes": inputs + 4 * pairs, "flops": pairs * 6 * length * length}


# ------------------------------------------------------------------------------------ exact ----
_SHAPES = [("W1", (3, 24, 128)), ("b1", (128,)), ("W2", (384, 128)), ("b2", (128,)),
           ("Wqkv0", (128, 384)), ("bqkv0", (384,)), ("Wo0", (128, 128)), ("bo0", (128,)),
           ("Wqkv1", (128, 384)), ("bqkv1", (384,)), ("Wo1", (128, 128)), ("bo1", (128,)),
           ("Wout", (128, 64)), ("bout", (64,))]


def _parameters(seed):
    """The encoder's initial parameters: uniform +-1/sqrt(fan in) weights, zero biases, drawn in
    the flat order of ``_SHAPES`` and rounded to float32, as doubles."""
    rng = np.random.default_rng(seed)
    fan = {"W1": 3, "W2": 384}
    parts = []
    for name, shape in _SHAPES:
        n = int(np.prod(shape))
        if name[0] == "W":
            parts.append(rng.uniform(-1, 1, n) / np.sqrt(fan.get(name, 128)))
        else:
            parts.append(np.zeros(n))
    return torch.from_numpy(np.concatenate(parts).astype(np.float32)).double().cuda()


def _forward(flat, codes, lens):
    """Unit-length embeddings [S, 64] of codes [S, 32] (CUDA tensors) in the dtype of ``flat``."""
    p, o = {}, 0
    for name, shape in _SHAPES:
        n = int(np.prod(shape))
        p[name] = flat[o:o + n].view(shape)
        o += n
    pos = torch.arange(32, device=codes.device)
    ok = pos[None, :] < lens[:, None]
    mask = ok[..., None].to(flat.dtype)
    x = torch.nn.functional.one_hot(codes.long(), 24).to(flat.dtype) * mask

    def conv(h, w):
        z = torch.zeros_like(h[:, :1])
        return torch.cat([z, h[:, :-1]], 1) @ w[0] + h @ w[1] + torch.cat([h[:, 1:], z], 1) @ w[2]

    h1 = torch.relu(conv(x, p["W1"]) + p["b1"]) * mask
    h = (h1 + torch.relu(conv(h1, p["W2"].view(3, 128, 128)) + p["b2"])) * mask
    for layer in "01":
        q, k, v = (h @ p["Wqkv" + layer] + p["bqkv" + layer]).split(128, dim=2)
        s = (q @ k.transpose(1, 2) / math.sqrt(128.0)).masked_fill(~ok[:, None, :], -math.inf)
        h = (h + torch.softmax(s, dim=2) @ v @ p["Wo" + layer] + p["bo" + layer]) * mask
    e = h.sum(1) / lens[:, None].to(flat.dtype) @ p["Wout"] + p["bout"]
    return e / e.norm(dim=1, keepdim=True)


def exact(case, seed):
    """The floating outputs in 64 bits (whole-number outputs have one right value each and are
    compared as they are)."""
    if case["kind"] == "embed":
        codes, lens = workloads.cdr3_codes(seed, case["n"])
        flat = _parameters(seed)
        z = torch.cat([_forward(flat, torch.from_numpy(codes[i:i + 8192]).cuda(),
                                torch.from_numpy(lens[i:i + 8192]).cuda())
                       for i in range(0, case["n"], 8192)])
        # the proposal kernel's operand layout: 16-byte chunk c of row r stored at c ^ (r & 7)
        row = torch.arange(z.shape[0], device=z.device)
        src = torch.arange(8, device=z.device)[None, :] ^ (row & 7)[:, None]
        return z.view(-1, 8, 8).gather(1, src[:, :, None].expand(-1, 8, 8)).reshape(-1, 64)
    if case["kind"] == "train":
        codes, lens, scores = _train_batch(case, seed)
        flat = _parameters(seed).requires_grad_(True)
        z = _forward(flat, torch.from_numpy(codes).cuda(), torch.from_numpy(lens).cuda())
        d = (z[0::2] - z[1::2]).square().sum(1)
        goal = torch.from_numpy(scores).cuda().double().clamp(max=64.0) / 32.0
        loss = (d - goal).square().mean()
        loss.backward()
        return loss.item(), flat.grad.detach()
    return None
