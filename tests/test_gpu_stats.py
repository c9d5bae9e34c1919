"""The stage times of cg_stats in the plain driver, whose batches overlap: each
batch's share is counted once."""
import numpy as np
import pytest

from rabbitqcplus_gb300 import capi, sim

pytestmark = pytest.mark.gpu

STAGES = ("seconds_candidates", "seconds_align", "seconds_msa")


def test_stage_times_of_many_batches():
    torch = pytest.importorskip("torch")
    batch, batches = 65_536, 8  # kernels of a batch far longer than the gaps between launches
    n = batch * batches
    r = sim.SimReads(sim.SimConfig(seed=82, genome_length=n * 150 // 30, num_reads=n))
    g = capi.CareGpu(capi.CareOptions.defaults(30.0, batch_anchors=batch))
    g.append_reads(r.sequences, r.offsets)
    g.build_tables()
    _, lmax = g.read_info()
    flags = torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy()
    out = torch.empty((n, lmax), dtype=torch.uint8, pin_memory=True).numpy()

    def times(first, count):
        a = g.stats()
        g.correct(first, count, flags[first:], out[first:])
        b = g.stats()
        return np.array([b[k] - a[k] for k in STAGES]), b["seconds_correct"]

    times(0, n)
    whole = [times(0, n) for _ in range(3)]
    alone = np.min([sum(times(j * batch, batch)[0] for j in range(batches)) for _ in range(3)], axis=0)
    for stages, total in whole:
        # one after the other on the context's stream: no more than the call's time
        assert stages.sum() <= 1.01 * total
    best = np.min([s for s, _ in whole], axis=0)
    # the same work as in calls of one batch each; a quarter for what the lookups gain or lose beside other kernels
    assert np.all(best >= 0.75 * alone) and np.all(best <= 1.25 * alone), dict(zip(STAGES, zip(best, alone)))
    g.close()
