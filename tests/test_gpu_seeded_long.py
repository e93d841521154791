"""The seeded pass on CDSs of more than 12288 nucleotides (chains of several words per
table entry): the band scan's runs, for random-like and for repetitive proteins, and
the oracle's stems."""
import numpy as np
import pytest

from test_gpu_hairpin import check
from test_gpu_parity import rand_ids
from test_gpu_seeded import assert_same, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["hairpin", "lrcs"])
@pytest.mark.parametrize("L,repeat", [(4095, False), (4096, False), (5000, True), (8200, False)])
def test_long_seeded_equals_band(pe, gpu, kind, L, repeat):
    k = pe.SL_HAIRPIN if kind == "hairpin" else pe.SL_LRCS
    aa = pe.synthetic_protein(L, 7 + L)
    if repeat:
        aa[:-1] = np.resize(aa[:5], L)
    tab = pe.dirichlet_table(L)
    pop0, scans0, _ = run(pe, aa, tab, 2, 8, 2, k, 0, 5)
    pop1, scans1, _ = run(pe, aa, tab, 2, 8, 2, k, 1, 5)
    assert_same(pop0, pop1)
    assert scans0 == scans1 > 0


def test_long_stems_match_oracle(pe, orc, gpu):
    L = 4501
    tabc = pe.dirichlet_table(L)
    aa = pe.synthetic_protein(L - 1, L)
    ids = rand_ids(np.random.default_rng(L), aa, tabc.arrays(), 2, 1)
    _, handed = check(pe, orc, aa, tabc, ids)
    assert handed == 0


@pytest.mark.parametrize("L", [2730, 2731, 4096, 8191, 8192])
def test_lrcs_head_counts(pe, gpu, L):
    """CDSs of 3 L nucleotides either side of the lengths where the number of table
    heads changes (8192, 12288, 24576)."""
    aa = pe.synthetic_protein(L - 1, L)
    tab = pe.dirichlet_table(L)
    pop0, scans0, _ = run(pe, aa, tab, 2, 8, 2, pe.SL_LRCS, 0, 5)
    pop1, scans1, _ = run(pe, aa, tab, 2, 8, 2, pe.SL_LRCS, 1, 5)
    assert_same(pop0, pop1)
    assert scans0 == scans1 > 0
