"""The seeded pass on repetitive and on long CDSs.  Above 12288 nucleotides it samples the
words first and leaves a repetitive CDS to the band scan at once, so such a design takes
no longer than with the band scan alone; the hand-over count shows which pass decided."""
import time

import numpy as np
import pytest

from test_gpu_seeded import assert_same, run

pytestmark = pytest.mark.gpu


def repeats(pe, L, motif, seed):
    """A tandem repeat of `motif` residues, one residue in 20 replaced."""
    rng = np.random.default_rng(seed)
    aa = np.where(rng.random(L) < 0.05, rng.integers(0, 20, L), np.resize(rng.integers(0, 20, motif), L))
    return np.append(aa, 20).astype(np.int8)


@pytest.mark.parametrize("motif", [3, 5, 8, 20])
def test_long_repeats_take_no_longer_than_the_band_scan(pe, gpu, motif):
    """Each side's fastest of three; 1.25 leaves room for the sample (under 1 % of the band
    scan) and for noise.  With the thread's bound alone the ratio was 1.9 to 4.4."""
    L, N, gens = 4200, 128, 5
    aa, tab = repeats(pe, L, motif, 7 + L), pe.dirichlet_table(L)
    best = []
    for method in (0, 1):
        with pe.Engine(aa, tab, 2, N, 0.05, objectives=1, seed=3, sl_kind=pe.SL_LRCS, sl_threads=256) as eng:
            eng.set_scan_method(method)
            t = []
            for _ in range(3):
                eng.init()
                eng.synchronize()
                t0 = time.perf_counter()
                eng.step(gens)
                eng.synchronize()
                t.append(time.perf_counter() - t0)
            best.append(min(t))
    assert best[0] <= 1.25 * best[1]


# 3 (L + 1) nucleotides: the first sampled length, either side of the lengths where the number
# of heads may change (24576), and positions above 32767
LENGTHS = [4095, 4096, 4097, 8191, 8192, 8193, 11000]


@pytest.mark.parametrize("kind", ["hairpin", "lrcs"])
@pytest.mark.parametrize("L", LENGTHS)
def test_long_random_is_decided_by_the_seeded_pass(pe, gpu, kind, L):
    k = pe.SL_HAIRPIN if kind == "hairpin" else pe.SL_LRCS
    aa, tab = pe.synthetic_protein(L, 11 + L), pe.dirichlet_table(L)
    pop0, scans0, handed0 = run(pe, aa, tab, 2, 6, 1, k, 0, 5)
    pop1, scans1, handed1 = run(pe, aa, tab, 2, 6, 1, k, 1, 5)
    assert_same(pop0, pop1)
    assert scans0 == scans1 > 0
    assert handed0 == handed1 == 0


@pytest.mark.parametrize("kind", ["hairpin", "lrcs"])
@pytest.mark.parametrize("L", LENGTHS)
def test_long_repetitive_is_handed_over(pe, gpu, kind, L):
    """A hand-over is counted only where the seeded pass was entered.  LRCS: one codon all
    along, so every scan hands over.  Hairpin: AAA or AAG in the first half, UUU or UUC
    in the second; a CDS whose draw pairs few of them (AAG with UUU) has no long chains, so
    some are handed over."""
    k = pe.SL_HAIRPIN if kind == "hairpin" else pe.SL_LRCS
    if kind == "lrcs":
        aa = np.full(L + 1, pe.AMINO.index("M"), np.int8)
    else:
        aa = np.array([pe.AMINO.index("K")] * (L // 2) + [pe.AMINO.index("F")] * (L - L // 2) + [0], np.int8)
    aa[-1] = 20
    tab = pe.dirichlet_table(L)
    pop0, scans0, handed0 = run(pe, aa, tab, 2, 4, 1, k, 0, 5)
    pop1, scans1, handed1 = run(pe, aa, tab, 2, 4, 1, k, 1, 5)
    assert_same(pop0, pop1)
    assert scans0 == scans1 >= handed0 > 0 and handed1 == 0
    if kind == "lrcs":
        assert handed0 == scans0
