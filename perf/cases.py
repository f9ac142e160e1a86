"""Workloads of the BPE training engine, over the range its users run it on.

``listed()`` names twelve of them, ``draw(rng)`` gives further ones of the same ranges,
``prepare`` makes what a program has in hand before the call, ``run`` is one pass through the
public entry points.  Every pass trains or counts from the start of its corpus, so it can be repeated.

Kinds of work
  fit       ``GPUBPETrainer.fit`` on padded ``(tokens, valid, lengths)`` CPU batches, as the batchers of a
            data loader yield them
  bytes     ``GPUBPETrainer.fit_bytes`` on one host byte buffer with document offsets (what ``train-bpe``
            does with files: pageable memory; loaders that prepare for the GPU: pinned memory)
  ties      the same with seeded random tie-breaks, which drives the loop from the host merge by merge
  warm      the same with seed merges from an earlier tokenizer applied before the learned ones
  resident  the ``Engine`` handle on bytes that are already on the GPU: reload, count, K merges
  ids       first pair histogram of an id stream over a vocabulary of up to 65 536 (retraining on
            top of an existing tokenizer), down to the sorted histogram
  seam      the operator seam ``count_pairs`` / ``select_best_pair`` / ``apply_merge_once`` on one padded
            CUDA batch, as a host-driven merge loop calls it
"""
from __future__ import annotations

import numpy as np
import torch

from supertoken_b200 import GPUBPETrainer, ops, synth
from supertoken_b200.engine import Engine

DEVICE = "cuda:0"
BASE_VOCAB = 256


def listed():
    return [
        # a few rows and merges: what a test, a notebook or a per-user tokenizer runs; fixed costs only
        {"name": "fit tiny batch", "kind": "fit", "corpus": "text", "batches": 1, "rows": 8, "width": 256,
         "merges": 32},
        # an ordinary loader: eight ragged batches of documents
        {"name": "fit ragged batches", "kind": "fit", "corpus": "mixed", "batches": 8, "rows": 64, "width": 2000,
         "merges": 400},
        # one small file set through train-bpe (pageable memory)
        {"name": "text 1 MiB", "kind": "bytes", "corpus": "text", "bytes": 1 << 20, "merges": 512, "pinned": False},
        # configuration 1 of the benchmark: 16 files of 1 MiB, 1 000 merges
        {"name": "text 16 MiB", "kind": "bytes", "corpus": "text", "bytes": 16 << 20, "merges": 1000,
         "pinned": False},
        # a production vocabulary: configuration 2's mixed-script text, thousands of merges, most of them rare pairs
        {"name": "mixed 256 MiB", "kind": "bytes", "corpus": "mixed", "bytes": 256 << 20, "merges": 8000,
         "pinned": True},
        # configuration 5: long runs of one byte or pattern, text and random bytes (odd size)
        {"name": "adversarial 64 MB", "kind": "bytes", "corpus": "adversarial", "bytes": 64_000_003, "merges": 1000,
         "pinned": False},
        # privacy mode: ties broken by a seeded generator on the host
        {"name": "random ties 512 KiB", "kind": "ties", "corpus": "mixed", "bytes": 512 << 10, "merges": 200},
        # continuing from an earlier tokenizer's merges
        {"name": "warm start 4 MiB", "kind": "warm", "corpus": "mixed", "bytes": 4 << 20, "warm": 200, "merges": 500},
        # the benchmark's default window: first 20 merges of 1 GiB that is already in HBM
        {"name": "resident 1 GiB", "kind": "resident", "corpus": "mixed", "bytes": 1 << 30, "merges": 20},
        # configuration 3's stream at an odd length
        {"name": "ids 200M", "kind": "ids", "tokens": 200_000_003, "vocab": 65536},
        # operator seam, one small batch and one that fills the GPU
        {"name": "seam 16x512", "kind": "seam", "corpus": "text", "rows": 16, "width": 512, "merges": 4},
        {"name": "seam 2048x4096", "kind": "seam", "corpus": "mixed", "rows": 2048, "width": 4096, "merges": 4},
    ]


def draw(rng):
    def log_int(lo, hi):
        return min(hi, int(round(lo * (hi / lo) ** rng.random())))

    kind = rng.choice(["fit", "bytes", "bytes", "bytes", "ties", "warm", "resident", "ids", "seam"])
    corpus = rng.choice(["text", "mixed", "adversarial"])
    if kind == "fit":
        return {"kind": kind, "corpus": corpus, "batches": rng.randint(1, 8), "rows": log_int(4, 128),
                "width": log_int(64, 2000), "merges": log_int(16, 400)}
    if kind == "bytes":
        most, merges = {"text": (64 << 20, 2000), "mixed": (256 << 20, 8000), "adversarial": (64_000_003, 1000)}[corpus]
        n = log_int(32 << 10, most)
        return {"kind": kind, "corpus": corpus, "bytes": n, "merges": log_int(64, min(merges, n // 256 + 64)),
                "pinned": rng.random() < 0.5}
    if kind == "ties":
        return {"kind": kind, "corpus": corpus, "bytes": log_int(32 << 10, 4 << 20), "merges": log_int(32, 300)}
    if kind == "warm":
        merges = log_int(64, 1000)
        return {"kind": kind, "corpus": corpus, "bytes": log_int(256 << 10, 16 << 20),
                "warm": merges // rng.randint(2, 4), "merges": merges}
    if kind == "resident":
        return {"kind": kind, "corpus": "mixed" if corpus == "adversarial" else corpus,
                "bytes": log_int(1 << 20, 1 << 30), "merges": rng.randint(5, 40)}
    if kind == "ids":
        return {"kind": kind, "tokens": log_int(1 << 16, 200_000_003), "vocab": log_int(512, 65536)}
    return {"kind": kind, "corpus": corpus, "rows": log_int(8, 2048), "width": log_int(64, 4096),
            "merges": rng.randint(2, 6)}


# ------------------------------------------------------------------------------------ inputs
def _corpus(case, n_bytes, seed):
    """uint8 bytes on the GPU and row offsets on the host."""
    if case["corpus"] == "text":      # rows are files: sixteen of them
        c = synth.config1_text(n_bytes, seed=seed, file_bytes=max(n_bytes // 16, 1), device=DEVICE)
    elif case["corpus"] == "mixed":
        c = synth.config2_mixed(n_bytes, seed=seed, device=DEVICE)
    else:
        c = synth.config5_adversarial(n_bytes, seed=seed, device=DEVICE)
    return c.data, c.row_offsets.cpu().numpy().astype(np.int64)


def _padded(case, n_batches, seed):
    """Padded batches cut out of a corpus: ragged rows, one of them full, about one in thirty empty."""
    rows, width = case["rows"], case["width"]
    data, _ = _corpus(case, max(rows * width * n_batches, 4096), seed)
    g = np.random.RandomState(seed % (1 << 32))
    out = []
    for b in range(n_batches):
        t = data[b * rows * width:(b + 1) * rows * width].reshape(rows, width).to(torch.int32)
        lens = g.randint(max(width // 4, 1), width + 1, rows)
        lens[g.rand(rows) < 1 / 30] = 0
        lens[g.randint(rows)] = width
        lengths = torch.from_numpy(lens.astype(np.int32)).to(DEVICE)
        valid = (torch.arange(width, device=DEVICE)[None, :] < lengths[:, None])
        out.append(((t * valid).to(torch.int32).contiguous(), valid.to(torch.uint8).contiguous(), lengths))
    return out


def _host(data, pinned):
    if not pinned:
        return data.cpu().numpy()
    h = torch.empty(data.numel(), dtype=torch.uint8, pin_memory=True)
    h.copy_(data)
    return h


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case}
    if kind == "fit":
        state["batches"] = [tuple(x.cpu() for x in b) for b in _padded(case, case["batches"], seed)]
    elif kind in ("bytes", "ties", "warm"):
        data, off = _corpus(case, case["bytes"], seed)
        state["data"], state["offsets"] = _host(data, case.get("pinned", False)), off
        state["tie_seed"] = seed
        if kind == "warm":  # the earlier tokenizer: learned on another, smaller sample of such text
            sample, sample_off = _corpus(case, max(case["bytes"] // 4, 65536), seed + 1)
            earlier = GPUBPETrainer(base_vocab=BASE_VOCAB, merges=case["warm"], device=DEVICE)
            res = earlier.fit_bytes(sample, sample_off)
            state["warm"] = [tuple(p) for p in res["merges"][:len(earlier.merge_counts)]]
    elif kind == "resident":
        state["data"], state["offsets"] = _corpus(case, case["bytes"], seed)
        state["engine"] = Engine(case["bytes"], base_vocab=BASE_VOCAB, max_merges=case["merges"], device=DEVICE)
    elif kind == "ids":
        ids, off = synth.config3_ids(case["tokens"], seed=seed, vocab=case["vocab"], device=DEVICE)
        state["ids"], state["offsets"] = ids, off.cpu().numpy().astype(np.int64)
        state["engine"] = Engine(case["tokens"], base_vocab=case["vocab"], max_merges=1, device=DEVICE)
        # the caller's histogram arrays, long enough for a stream of distinct pairs
        state["keys"] = torch.zeros(case["tokens"], dtype=torch.int64, device=DEVICE)
        state["counts"] = torch.zeros(case["tokens"], dtype=torch.int64, device=DEVICE)
    else:
        tokens, valid, lengths = _padded(case, 1, seed)[0]
        rows, width = tokens.shape
        cap = rows * (width - 1)
        state.update(
            tokens=tokens, valid=valid, work_tokens=torch.empty_like(tokens), work_valid=torch.empty_like(valid),
            lengths=torch.empty_like(lengths), spans=torch.empty((rows, width - 1), dtype=torch.bool, device=DEVICE),
            keys=torch.empty((cap, 2), dtype=torch.int32, device=DEVICE),
            counts=torch.empty((cap,), dtype=torch.int64, device=DEVICE),
            n_pairs=torch.zeros((1,), dtype=torch.int64, device=DEVICE))
    return state


# ------------------------------------------------------------------------------------ one pass
def _rows(values, shape, dtype):
    """The values as an array of the full shape: a run that stops early leaves its last rows at -1."""
    out = np.full(shape, -1, dtype=dtype)
    if len(values):
        out[:len(values)] = values
    return out


def _learned(trainer, result, n_merges):
    """What a training run leaves: the merges it applied or learned, their counts, the live tokens."""
    n = result["warm_start"]["applied"] + len(trainer.merge_counts)
    return {"merges": _rows(result["merges"][:n], (n_merges, 2), np.int32),
            "counts": _rows(trainer.merge_counts, (n_merges,), np.int64),
            "live_tokens": result["telemetry"]["engine"]["live_tokens"]}


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "fit":
        t = GPUBPETrainer(base_vocab=BASE_VOCAB, merges=case["merges"], device=DEVICE)
        return _learned(t, t.fit(state["batches"], log_every=0), case["merges"])
    if kind == "bytes":
        t = GPUBPETrainer(base_vocab=BASE_VOCAB, merges=case["merges"], device=DEVICE)
        return _learned(t, t.fit_bytes(state["data"], state["offsets"]), case["merges"])
    if kind == "ties":
        t = GPUBPETrainer(base_vocab=BASE_VOCAB, merges=case["merges"], device=DEVICE, randomize_ties=True,
                          tie_seed=state["tie_seed"])
        return _learned(t, t.fit_bytes(state["data"], state["offsets"]), case["merges"])
    if kind == "warm":
        t = GPUBPETrainer(base_vocab=BASE_VOCAB, merges=case["merges"], device=DEVICE)
        return _learned(t, t.fit_bytes(state["data"], state["offsets"], warm_start_merges=state["warm"]), case["merges"])
    if kind == "resident":
        e = state["engine"]
        e.reset()
        e.append_bytes(state["data"], state["offsets"])
        e.count_initial()
        e.train(case["merges"])
        merges, counts, live = e.merges()
        n = case["merges"]
        return {"merges": _rows(merges, (n, 2), np.int32), "counts": _rows(counts, (n,), np.int64),
                "live_before": _rows(live, (n,), np.int64), "live_tokens": int(e.state().live_tokens)}
    if kind == "ids":
        e = state["engine"]
        e.reset()
        e.append_ids(state["ids"], state["offsets"])
        e.count_initial()
        keys, counts = e.export_histogram()
        n = keys.numel()
        state["keys"][:n].copy_(keys)
        state["counts"][:n].copy_(counts)
        return {"keys": state["keys"], "counts": state["counts"], "n_pairs": n}
    # seam: the caller's batch is copied to the working buffers, which the operators rewrite in place
    tokens, valid = state["work_tokens"], state["work_valid"]
    tokens.copy_(state["tokens"])
    valid.copy_(state["valid"])
    keys, counts, n_pairs, lengths = state["keys"], state["counts"], state["n_pairs"], state["lengths"]
    chosen, spans = [], None
    for step in range(case["merges"]):
        ops.count_pairs(tokens, valid, keys, counts, n_pairs)
        n = int(n_pairs.item())
        packed = (keys[:n, 0].to(torch.int64) << 32) | keys[:n, 1].to(torch.int64)
        key, count, _ = ops.select_best_pair(ops.PairHistogramResult(packed, counts[:n]))
        if key is None:
            break
        chosen.append((key >> 32, key & 0xFFFFFFFF, count))
        tokens, valid, lengths, spans = ops.apply_merge_once(
            tokens, valid, lengths, key >> 32, key & 0xFFFFFFFF, BASE_VOCAB + step, pair_workspace=state["spans"])
    return {"tokens": tokens, "valid": valid, "lengths": lengths, "spans": spans, "keys": keys, "counts": counts,
            "n_pairs": n_pairs, "chosen": _rows(chosen, (case["merges"], 3), np.int64)}


# ------------------------------------------------------------------------------------ what it costs at least
def work(case):
    """Inputs read once, outputs written once (integer work: no floating-point operations)."""
    kind = case["kind"]
    if kind == "fit":  # int32 token + uint8 valid per cell
        n = 5 * case["batches"] * case["rows"] * case["width"] + 24 * case["merges"]
    elif kind in ("bytes", "ties", "warm", "resident"):
        n = case["bytes"] + 24 * case["merges"]
    elif kind == "ids":  # ids in; a sixth of the positions of such a stream are distinct pairs, 16 bytes each out
        n = 4 * case["tokens"] + 16 * (case["tokens"] // 6)
    else:  # per merge: read by the count and by the merge, written by the merge, the span mask, the histogram buffers
        cells = case["rows"] * case["width"]
        n = case["merges"] * (cells * (5 + 5 + 5 + 1) + 16 * cells)
    return {"bytes": n, "flops": 0}


def tolerance(case):
    return "exact"
