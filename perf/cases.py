"""Performance cases: what a program using this library has it do.

A case is one call (or one short run of calls) through the package's public
front end (rabbitqcplus_gb300.capi, the ctypes mirror of include/care_gpu.h):
correcting anchors against resident tables, a whole session on a new data set,
a file-to-file run, and the learned classifier's training and scoring.

Read sets follow the shapes of rabbitqcplus_gb300/sim.py's workloads (genome
with diverged repeat copies, uniform coverage, both strands, substitutions
rising from 5' to 3', optional indels and pairs, Phred scores from a clipped
normal with low scores at errors), drawn on the GPU from the seed so that they
are quick to make.
"""
from __future__ import annotations

import math
import os
import struct
import tempfile

import numpy as np
import torch

from rabbitqcplus_gb300 import capi, learned

MAPS = 48  # minhash maps, the default of every front end


def _case(name, kind="correct", **kw):
    c = {"name": name, "kind": kind}
    if kind in ("correct", "session", "files"):
        c.update({"reads": 200_000, "anchors": 0, "len_min": 150, "len_max": 150, "coverage": 30, "repeats": 0.0,
                  "paired": False, "quality": False, "err5": 0.01, "err3": 0.01, "indels": 0.0, "driver": "plain",
                  "decision": "classic", "candidates": False})
    c.update(kw)
    return c


def listed():
    return [
        # a program that corrects single reads on demand against a resident index: latency of a small, odd call
        _case("few_anchors", reads=200_000, anchors=37),
        # a small bacterial data set (1 Mbp at 30x), default options
        _case("bacterium_200k", reads=200_000),
        # a 10 Mbp genome with repeats, errors rising along the read, stage-by-stage driver
        _case("repeats_2m", reads=2_000_000, repeats=0.06, err5=0.002, err3=0.02),
        # a large single-end set with the batched driver and the learned decision (the benchmark's main form)
        _case("learned_4m", reads=4_000_000, repeats=0.05, driver="batched", decision="learned"),
        # paired-end reads with indels, a range that is no multiple of any batch size
        _case("paired_1m", reads=1_000_006, repeats=0.01, paired=True, indels=0.0001, driver="batched"),
        # reads trimmed to 50-250 bp, with quality scores
        _case("trimmed_quality_300k", reads=300_001, len_min=50, len_max=250, repeats=0.06, quality=True, err5=0.002,
              err3=0.02),
        # --candidateCorrection: every high-quality anchor also corrects its candidates, then the combine step
        _case("candidates_400k", reads=400_000, repeats=0.05, candidates=True, driver="batched"),
        # 300 bp reads (2 x 300 chemistry, processed as single reads)
        _case("long_300bp_60k", reads=60_000, len_min=300, len_max=300, err5=0.002, err3=0.02),
        # a new data set from host memory: context, append, index build, correction of every read, release
        _case("session_1m", "session", reads=1_000_000, repeats=0.05, driver="batched"),
        # care::performCorrection's job: FASTQ files in, corrected FASTQ files out (a read pair per record)
        _case("files_paired_200k", "files", reads=200_000, paired=True, quality=True, repeats=0.01),
        # training the learned decision's classifier on labelled columns
        _case("train_256k", "train", rows=262_144, batch=4096, epochs=2),
        # scoring a validation set of columns
        _case("score_1m", "score", rows=1_000_003),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["correct"] * 8 + ["session", "session", "files", "train", "score"])
    if kind == "train":
        batch = rng.choice([1024, 2048, 4096, 8192])
        return {"kind": kind, "rows": max(batch, _log_int(rng, 20_000, 300_000)), "batch": batch,
                "epochs": rng.randint(1, 2)}
    if kind == "score":
        return {"kind": kind, "rows": _log_int(rng, 100, 1_000_000)}
    c = _case("", kind)
    del c["name"]
    shape = rng.choice(["fixed", "fixed", "trimmed", "long"] if kind == "correct" else ["fixed", "trimmed"])
    most = {"correct": 3_000_000, "session": 1_000_000, "files": 200_000}[kind]
    if shape == "fixed":
        c["len_min"] = c["len_max"] = rng.choice([75, 100, 101, 125, 150, 151, 250])
    elif shape == "trimmed":
        c["len_min"], c["len_max"] = rng.randint(36, 80), rng.randint(100, 256)
        most = most // 4
    else:
        c["len_max"] = rng.randint(260, 640)
        c["len_min"] = rng.choice([c["len_max"], 200])
        most = 60_000 * 300 // c["len_max"]
    c["reads"] = _log_int(rng, most // 30, most)
    c["coverage"] = rng.choice([20, 30, 30, 40])
    c["repeats"] = rng.choice([0.0, 0.01, 0.05])
    c["err5"], c["err3"] = rng.choice([(0.01, 0.01), (0.002, 0.02)])
    c["quality"] = kind == "files" or rng.random() < 0.3
    c["paired"] = shape != "long" and rng.random() < 0.3
    if c["paired"]:
        c["reads"] += c["reads"] & 1
        c["indels"] = 0.0001
    if kind != "files":
        c["driver"] = rng.choice(["plain", "batched"])
        c["decision"] = rng.choice(["classic", "classic", "learned"]) if shape != "long" else "classic"
        c["candidates"] = c["decision"] == "classic" and not c["paired"] and rng.random() < 0.25
    if kind == "correct" and not c["candidates"] and rng.random() < 0.4:
        c["anchors"] = 2 * _log_int(rng, 1, max(2, c["reads"] // 4)) if c["paired"] else _log_int(rng, 1, c["reads"])
    return c


# ---------------------------------------------------------------- read sets


def _reads(case, seed):
    """(sequences, qualities) as [n][len_max] uint8 host arrays and the read lengths."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    n, lmin, lmax = case["reads"], case["len_min"], case["len_max"]
    size = max(4 * lmax + 1000, int(n * (lmin + lmax) / 2 / case["coverage"]))

    def ints(hi, shape, lo=0, dtype=torch.int64):
        return torch.randint(lo, hi, shape, generator=g, device=dev, dtype=dtype)

    genome = ints(4, (size,), dtype=torch.uint8)
    copies = int(size * case["repeats"] / 3000)
    if copies:  # segments of 1-5 kbp copied elsewhere with 2% divergence
        at = torch.stack([ints(max(1, size - 5000), (copies,)), ints(max(1, size - 5000), (copies,)),
                          ints(5001, (copies,), lo=1000)]).cpu().tolist()
        for src, dst, length in zip(*at):
            seg = genome[src:src + length].clone()
            other = torch.rand(len(seg), generator=g, device=dev) < 0.02
            seg = torch.where(other, (seg + ints(4, (len(seg),), lo=1, dtype=torch.uint8)) & 3, seg)
            genome[dst:dst + len(seg)] = seg[:size - dst]
    lens = torch.full((n,), lmax, device=dev) if lmin == lmax else ints(lmax + 1, (n,), lo=lmin)
    span = lmax + 16  # room for deletions
    if case["paired"]:  # fragments of about 300 bp or one read, read 1 forward and read 2 reverse, either strand
        frag = (torch.randn(n // 2, generator=g, device=dev) * 30 + max(300, lmax + 60)).long().clamp_min(span)
        f0 = (torch.rand(n // 2, generator=g, device=dev, dtype=torch.float64) * (size - frag - span)).long()
        flip = ints(2, (n // 2,)).bool()
        left, right = f0, f0 + frag - span
        start = torch.stack([torch.where(flip, right, left), torch.where(flip, left, right)], 1).reshape(-1)
        rc = torch.stack([flip, ~flip], 1).reshape(-1)
    else:
        start = ints(size - span, (n,))
        rc = ints(2, (n,)).bool()
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=dev)
    col = torch.arange(lmax, device=dev)
    rate = case["err5"] + (case["err3"] - case["err5"]) * col / max(1, lmax - 1)
    seqs = np.empty((n, lmax), np.uint8)
    quals = np.empty((n, lmax), np.uint8) if case["quality"] else None
    chunk = max(1, 60_000_000 // lmax)
    for a in range(0, n, chunk):
        b = min(n, a + chunk)
        m = b - a
        off = col.expand(m, lmax)
        inserted = None
        if case["indels"]:
            u = torch.rand((m, lmax), generator=g, device=dev)
            inserted = u < case["indels"] / 2
            step = 1 + (u > 1 - case["indels"] / 2).long() - inserted.long()
            off = (torch.cumsum(step, 1) - 1).clamp_(0, span - 1)
        r = rc[a:b, None]
        pos = torch.where(r, start[a:b, None] + span - 1 - off, start[a:b, None] + off)
        base = genome[pos]
        base = torch.where(r, 3 - base, base)
        del pos, off
        err = torch.rand((m, lmax), generator=g, device=dev) < rate
        if inserted is not None:
            err = err | inserted
        base = torch.where(err, (base + ints(4, (m, lmax), lo=1, dtype=torch.uint8)) & 3, base)
        torch.from_numpy(seqs[a:b]).copy_(letters[base.long()])
        if quals is not None:
            q = (torch.randn((m, lmax), generator=g, device=dev) * 4 + 34).round_().clamp_(2, 41).to(torch.uint8)
            q = torch.where(err, ints(21, (m, lmax), lo=2, dtype=torch.uint8), q)
            torch.from_numpy(quals[a:b]).copy_(q + 33)
    return seqs, quals, lens.cpu().numpy().astype(np.int64)


def _concatenated(rows, lens):
    """Reads back to back, as cg_append_reads takes them."""
    if int(lens.min()) == rows.shape[1]:
        return rows.reshape(-1)
    keep = torch.arange(rows.shape[1])[None, :] < torch.from_numpy(lens)[:, None]
    return torch.from_numpy(rows).masked_select(keep).numpy()


def _options(case):
    o = capi.CareOptions.defaults(float(case["coverage"]), kmerlength=20, num_hash_functions=MAPS)
    o.pair_mode = capi.CG_PAIR_PE if case["paired"] else capi.CG_PAIR_SE
    o.use_quality_scores = int(case["quality"])
    o.driver = capi.CG_DRIVER_BATCHED if case["driver"] == "batched" else capi.CG_DRIVER_PLAIN
    o.correction_type = capi.CG_CORR_LEARNED if case["decision"] == "learned" else capi.CG_CORR_CLASSIC
    o.correct_candidates = int(case["candidates"])
    return o


def _context(st):
    g = capi.CareGpu(_options(st["case"]))
    g.append_reads(st["sequences"], st["offsets"], st["qualities"])
    g.build_tables()
    if st["case"]["decision"] == "learned":
        g.load_classifier(st["model"])
    return g


def _pinned(shape):
    return torch.empty(shape, dtype=torch.uint8, pin_memory=True).numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "score"):
        return _prepare_classifier(case, seed)
    seqs, quals, lens = _reads(case, seed)
    st = {"case": case, "rows": seqs, "model": open(learned.DEFAULT_MODEL, "rb").read()}
    st["offsets"] = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    st["sequences"] = _concatenated(seqs, lens)
    st["qualities"] = None if quals is None else _concatenated(quals, lens)
    if kind == "files":
        return _prepare_files(st)
    first, count = 0, case["reads"]
    if case.get("anchors"):
        count = min(case["anchors"], case["reads"])
        first = (case["reads"] - count) // 2 & ~1
    st["first"], st["count"] = first, count
    # page-locked results, as a program that corrects window after window keeps them
    st["flags"], st["out"] = _pinned((count,)), _pinned((count, case["len_max"]))
    # bytes past a read's end are not part of its result
    st["past"] = None
    if case["len_min"] != case["len_max"]:
        st["past"] = torch.arange(case["len_max"])[None, :] >= torch.from_numpy(lens[first:first + count])[:, None]
    if kind == "correct":
        st["gpu"] = _context(st)
    else:  # a session reads its input from page-locked memory
        for k in ("sequences", "qualities"):
            if st[k] is not None:
                st[k] = torch.from_numpy(st[k]).pin_memory().numpy()
    return st


def _prepare_files(st):
    case = st["case"]
    where = "/dev/shm" if os.access("/dev/shm", os.W_OK) else None
    st["dir"] = tempfile.TemporaryDirectory(prefix="care_", dir=where)
    d = st["dir"].name
    n = case["reads"]
    files = 2 if case["paired"] else 1
    st["inputs"] = [os.path.join(d, "in_%d.fastq" % f) for f in range(files)]
    st["outputs"] = ["out_%d.fastq" % f for f in range(files)]
    s, q, o = st["sequences"].tobytes(), st["qualities"].tobytes(), st["offsets"].tolist()
    for f, path in enumerate(st["inputs"]):
        rec = [b"@r%d\n%b\n+\n%b\n" % (i, s[o[i]:o[i + 1]], q[o[i]:o[i + 1]]) for i in range(f, n, files)]
        with open(path, "wb") as out:
            out.write(b"".join(rec))
    return st


def _prepare_classifier(case, seed):
    rng = np.random.default_rng(seed)
    n = case["rows"]
    # shares and ratios: mostly near 0 or 1, as the column features are
    x = rng.random((n, capi.CLASSIFIER_FEATURES), np.float32)
    x *= x
    if case["kind"] == "score":
        return {"case": case, "x": x, "model": open(learned.DEFAULT_MODEL, "rb").read()}
    w = rng.normal(0, 1, capi.CLASSIFIER_FEATURES).astype(np.float32)
    z = x @ w
    y = (z > np.quantile(z, 0.05)).astype(np.uint8)
    o = capi.TrainOptions.defaults(epochs=case["epochs"], batch_rows=case["batch"], seed=seed & 0x7FFFFFFF)
    return {"case": case, "x": x, "y": y, "options": o}


# ---------------------------------------------------------------- one pass


def _result(st, flags):
    """The corrected read set: rows without a correction keep the input read."""
    out = st["out"]
    kept = np.flatnonzero((flags & capi.CG_RESULT_CORRECTED) == 0)
    out[kept] = st["rows"][st["first"] + kept]
    if st["past"] is not None:
        torch.from_numpy(out).masked_fill_(st["past"], 0)
    return {"flags": flags, "reads": out}


def run(st):
    kind = st["case"]["kind"]
    if kind == "correct":
        flags, _ = st["gpu"].correct(st["first"], st["count"], st["flags"], st["out"])
        return _result(st, flags)
    if kind == "session":
        g = _context(st)
        flags, _ = g.correct(0, st["count"], st["flags"], st["out"])
        g.close()
        return _result(st, flags)
    if kind == "files":
        records = capi.correct_files(_options(st["case"]), st["inputs"], st["dir"].name, st["outputs"])
        return {"records": records,
                "files": [np.fromfile(os.path.join(st["dir"].name, f), np.uint8) for f in st["outputs"]]}
    if kind == "train":
        model, losses = capi.train_classifier(st["x"], st["y"], st["options"])
        return {"losses": losses, **_parameters(model)}
    return capi.classifier_logits(st["model"], st["x"])


def _parameters(model):
    """The serialized classifier's parameters as FP32 arrays (include/care_gpu.h gives the layout)."""
    f, h1, h2 = struct.unpack_from("<3I", model, 8)

    def bf16(at, n):
        return (np.frombuffer(model, np.uint16, n, at).astype(np.uint32) << 16).view(np.float32)

    at = 32
    w1 = bf16(at, h1 * f)
    w2 = bf16(at + 2 * h1 * f, h2 * h1)
    w3 = bf16(at + 2 * (h1 * f + h2 * h1), h2)
    b = np.frombuffer(model, np.float32, h1 + h2 + 1, at + 2 * (h1 * f + h2 * h1 + h2))
    return {"w1": w1.reshape(h1, f), "w2": w2.reshape(h2, h1), "w3": w3, "b1": b[:h1].copy(),
            "b2": b[h1:h1 + h2].copy(), "b3": b[h1 + h2:].copy()}


def work(case):
    kind = case["kind"]
    macs = 32 * 64 + 64 * 64 + 64
    if kind == "score":
        return {"bytes": case["rows"] * (128 + 4), "flops": 2 * macs * case["rows"]}
    if kind == "train":
        rows = case["rows"] // case["batch"] * case["batch"] * case["epochs"]
        return {"bytes": rows * (128 + 1), "flops": 6 * macs * rows}
    n = case["reads"]
    anchors = min(case["anchors"], n) if case.get("anchors") else n
    length = (case["len_min"] + case["len_max"]) / 2
    # per anchor: its keys and lookup slots (8 + 16 bytes a map), its bucket ids (about 22 per unit of coverage, 4
    # bytes each), the 2-bit rows of the reads it meets (each once over a whole set), and the result
    met = min(n, anchors * 2 * case["coverage"])
    per_read = length / 4 + 2 + (length if case["quality"] else 0)
    b = anchors * (MAPS * 24 + 22 * case["coverage"] * 4 + length + 1) + met * per_read
    if kind in ("session", "files"):
        b += n * (length * (2 if case["quality"] else 1) + 8)  # the input text
        b += n * MAPS * (8 + 16 + 8 + 4 + 16)  # keys written, sorted (read and written once), buckets and slots
    if kind == "files":
        b += n * length
    return {"bytes": int(b), "flops": 0}


def exact(case, seed):
    if case["kind"] != "score":
        return None  # bases, flags and bytes; a trained model follows its own rounding
    st = _prepare_classifier(case, seed)
    p = {k: v.astype(np.float64) for k, v in _parameters(st["model"]).items()}
    x = st["x"].astype(np.float64)
    h = np.maximum(x @ p["w1"].T + p["b1"], 0)
    h = np.maximum(h @ p["w2"].T + p["b2"], 0)
    return h @ p["w3"] + p["b3"]
