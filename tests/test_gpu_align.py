"""The alignment kernel's instances against the oracle: read lengths at the
edges of every instance, one length or several, units of one and of several
parts, and options that loosen the mismatch limit or the smallest overlap."""
import numpy as np
import pytest

import oracle
from rabbitqcplus_gb300 import capi, sim

pytestmark = pytest.mark.gpu


def check(lo, hi, coverage=30, driver=capi.CG_DRIVER_PLAIN, count=None, **kw):
    genome = max(4_000, 4 * hi)
    n = int(genome * coverage / ((lo + hi) / 2)) & ~1
    r = sim.SimReads(sim.SimConfig(seed=70 + hi, genome_length=genome, repeat_families=1, repeat_copies=2,
                                   repeat_min_len=300, repeat_max_len=600, num_reads=n, read_len_min=lo,
                                   read_len_max=hi, sub_rate_5p=0.002, sub_rate_3p=0.02))
    o = capi.CareOptions.defaults(float(coverage), driver=driver, **kw)
    if driver == capi.CG_DRIVER_BATCHED:
        o.batch_anchors, o.msa_warps, o.streams = 64, 2, 2
    g = capi.CareGpu(o)
    g.append_reads(r.sequences, r.offsets)
    g.build_tables()
    first = 0 if count is None else n // 3
    flags, seqs = g.correct(first, count)
    g.close()
    orc = oracle.Oracle(o, r.sequences, r.offsets, None)
    oflags, oseqs, _ = orc.correct(first, len(flags))
    orc.close()
    assert np.array_equal(flags, oflags)
    for i in np.flatnonzero(flags & capi.CG_RESULT_CORRECTED):
        length = int(r.lengths[first + i])
        assert np.array_equal(seqs[i, :length], oseqs[i, :length]), first + i


@pytest.mark.parametrize("length", [33, 64, 95, 96, 97, 128, 129, 159, 160, 161, 255, 256, 257, 319, 320, 321])
def test_one_length(length):
    check(length, length)


@pytest.mark.parametrize("lo,hi", [(22, 40), (25, 96), (36, 101), (50, 160), (20, 161), (50, 256), (60, 257), (30, 320),
                                   (40, 321), (500, 512), (100, 513), (1000, 1024)])
def test_several_lengths(lo, hi):
    check(lo, hi)


@pytest.mark.parametrize("driver", [capi.CG_DRIVER_PLAIN, capi.CG_DRIVER_BATCHED])
@pytest.mark.parametrize("lo,hi", [(100, 100), (60, 150), (700, 700)])
def test_units_of_several_parts(lo, hi, driver):
    check(lo, hi, coverage=180, driver=driver)


@pytest.mark.parametrize("count", [1, 33, 300])
def test_few_anchors(count):
    check(150, 150, coverage=60, count=count)


@pytest.mark.parametrize("kw", [{"max_error_rate": 0.45}, {"max_error_rate": 0.02}, {"min_overlap": 2, "min_overlap_ratio": 0.0},
                                {"min_overlap": 90}, {"min_overlap_ratio": 0.9}])
@pytest.mark.parametrize("lo", [60, 150])
def test_limits(lo, kw):
    check(lo, 150, **kw)


# above one half a shift under its limit can have more hi plane mismatches than matches
@pytest.mark.parametrize("rate", [0.5, 0.55, 0.7, 0.9, 1.5])
@pytest.mark.parametrize("lo,hi", [(150, 150), (60, 150), (300, 300)])
def test_max_error_rate_above_half(lo, hi, rate):
    check(lo, hi, max_error_rate=rate)


def test_max_error_rate_above_half_in_units_of_several_parts():
    check(60, 150, coverage=180, driver=capi.CG_DRIVER_BATCHED, max_error_rate=0.8)


# a shift without overlap is no shift, however far the options let it go
@pytest.mark.parametrize("min_overlap", [0, -1, -70_000])
def test_no_smallest_overlap(min_overlap):
    check(60, 150, min_overlap=min_overlap, min_overlap_ratio=-1000.0)
