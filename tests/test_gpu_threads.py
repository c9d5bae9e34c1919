"""Calls of several threads at once: training (which captures a graph), scoring
and correction with the batched driver (which captures one per pipeline) give
what they give alone."""
import threading

import numpy as np
import pytest

from rabbitqcplus_gb300 import capi, learned, sim

pytestmark = pytest.mark.gpu


def jobs():
    rng = np.random.default_rng(4)
    x = rng.random((4096, capi.CLASSIFIER_FEATURES), np.float32)
    y = (x.sum(1) > 16).astype(np.uint8)
    model = open(learned.DEFAULT_MODEL, "rb").read()
    r = sim.SimReads(sim.SimConfig(seed=81, genome_length=20_000, num_reads=4_000, sub_rate_5p=0.002,
                                   sub_rate_3p=0.02))
    shape = dict(driver=capi.CG_DRIVER_BATCHED, batch_anchors=512, align_blocks=152, msa_warps=4, streams=2)

    def train():
        m, losses = capi.train_classifier(x, y, capi.TrainOptions.defaults(epochs=1, batch_rows=1024, seed=3))
        return np.frombuffer(m, np.uint8), losses

    def score():
        return (capi.classifier_logits(model, x),)

    def correct():
        g = capi.CareGpu(capi.CareOptions.defaults(30.0, **shape))
        g.append_reads(r.sequences, r.offsets)
        g.build_tables()
        flags, out = g.correct()
        g.close()
        return flags, np.where((flags & capi.CG_RESULT_CORRECTED)[:, None] != 0, out, 0)

    return {"train": (train, 100), "score": (score, 200), "correct": (correct, 40)}


@pytest.mark.parametrize("names", [("train", "score"), ("correct", "score"), ("train", "correct"), ("train", "train"),
                                   ("correct", "correct")])
def test_calls_of_two_threads(names):
    todo = [jobs()[n] for n in names]
    want = [f() for f, _ in todo]
    failures = []

    def work(k):
        f, times = todo[k]
        for _ in range(times):
            try:
                got = f()
                if not all(np.array_equal(a, b) for a, b in zip(got, want[k])):
                    failures.append(f"{names[k]}: another result")
            except capi.CareError as e:
                failures.append(f"{names[k]}: {e}")

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, (len(failures), sorted(set(failures)))
