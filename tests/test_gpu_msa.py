"""The MSA kernel's instances against the oracle: read lengths at the edges of
the instances with quality scores, rows with more mismatches than the list of a
staged group holds, and anchors with several groups of rows."""
import numpy as np
import pytest

import oracle
from rabbitqcplus_gb300 import capi, sim

pytestmark = pytest.mark.gpu


def check(lo, hi, coverage=30, errors=(0.002, 0.02), quality=False, **kw):
    genome = max(4_000, 4 * hi)
    n = int(genome * coverage / ((lo + hi) / 2)) & ~1
    r = sim.SimReads(sim.SimConfig(seed=90 + hi, genome_length=genome, repeat_families=1, repeat_copies=2,
                                   repeat_min_len=300, repeat_max_len=600, num_reads=n, read_len_min=lo,
                                   read_len_max=hi, sub_rate_5p=errors[0], sub_rate_3p=errors[1]))
    q = r.qualities if quality else None
    o = capi.CareOptions.defaults(float(coverage), use_quality_scores=int(quality), **kw)
    g = capi.CareGpu(o)
    g.append_reads(r.sequences, r.offsets, q)
    g.build_tables()
    flags, seqs = g.correct()
    builds = g.stats()["msa_builds"]
    g.close()
    orc = oracle.Oracle(o, r.sequences, r.offsets, q)
    oflags, oseqs, _ = orc.correct(0, n)
    orc.close()
    assert builds > 0
    assert np.array_equal(flags, oflags)
    for i in np.flatnonzero(flags & capi.CG_RESULT_CORRECTED):
        length = int(r.lengths[i])
        assert np.array_equal(seqs[i, :length], oseqs[i, :length]), i


@pytest.mark.parametrize("lo,hi", [(33, 33), (50, 128), (129, 129), (160, 160), (161, 161), (50, 256), (257, 257),
                                   (100, 320), (321, 321), (200, 512), (513, 513), (640, 640), (300, 641), (1024, 1024)])
def test_quality(lo, hi):
    check(lo, hi, quality=True)


@pytest.mark.parametrize("quality", [False, True])
@pytest.mark.parametrize("length", [100, 150, 250, 300, 600, 1000])
def test_many_mismatches(length, quality):
    check(length, length, coverage=60, errors=(0.08, 0.08), quality=quality, max_error_rate=0.45, kmerlength=14)
