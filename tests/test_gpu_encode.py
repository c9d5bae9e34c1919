"""Reads with characters outside ACGT, in either case, at every alignment of the
text: the store must hold what the replacement rule gives (A, C, G, T in turn
over the call's reads), which a second context gets spelled out."""
import numpy as np
import pytest

from rabbitqcplus_gb300 import capi

pytestmark = pytest.mark.gpu


def spelled_out(text):
    out = text.copy()
    upper = text & 0xDF
    good = np.isin(upper, np.frombuffer(b"ACGT", np.uint8))
    out[good] = upper[good]
    bad = np.flatnonzero(~good)
    out[bad] = np.frombuffer(b"ACGT", np.uint8)[np.arange(len(bad)) & 3]
    return out


def state(text, offs):
    g = capi.CareGpu(capi.CareOptions.defaults(30.0, kmerlength=14))
    g.append_reads(text, offs)
    g.build_tables()
    n = len(offs) - 1
    sig = np.array(g.signatures(0, n, 48))
    flags, seqs = g.correct()
    g.close()
    return sig, flags, seqs


@pytest.mark.parametrize("rate", [0.0, 0.01, 0.9])
@pytest.mark.parametrize("lo,hi", [(1, 40), (14, 18), (15, 33), (250, 260), (500, 520), (1020, 1024)])
def test_characters(lo, hi, rate):
    rng = np.random.default_rng(hi)
    genome = rng.choice(np.frombuffer(b"ACGTacgt", np.uint8), 4 * hi)
    lens = rng.integers(lo, hi + 1, 301)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    text = np.concatenate([genome[s:s + n] for s, n in ((int(rng.integers(0, 3 * hi)), int(n)) for n in lens)])
    odd = rng.random(len(text)) < rate
    text[odd] = rng.integers(1, 256, int(odd.sum()), dtype=np.uint8)
    clean = spelled_out(text)
    a, b = state(text, offs), state(clean, offs)
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    for i in np.flatnonzero(a[1] & capi.CG_RESULT_CORRECTED):
        assert np.array_equal(a[2][i, :lens[i]], b[2][i, :lens[i]]), i
