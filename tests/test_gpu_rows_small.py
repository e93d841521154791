"""Codon ids of small calls, whose rows the host pads and strips (up to 64 KB of padded rows),
against the oracle: row lengths around multiples of 16, and sizes either side of the
bounds where the device takes over the padding (64 KB of rows of Lp) and the check
(64 KB of ids)."""
import numpy as np
import pytest

from test_gpu_parity import rand_ids, same

pytestmark = pytest.mark.gpu


# positions, CDSs, solutions; bytes of ids and of padded rows beside the bounds
@pytest.mark.parametrize("L,m,n", [
    (15, 2, 1), (16, 2, 1), (17, 2, 1), (33, 3, 2),
    (3, 2, 2048), (3, 2, 2049),      # 12 KB of ids, 64 KB of rows exactly and one more
    (100, 2, 292), (100, 2, 293),    # 57 KB of ids, rows of 65408 and 65632 bytes
    (112, 2, 292), (112, 2, 293),    # whole rows: 65408 and 65632 bytes of ids
    (63, 2, 520), (63, 2, 521),      # padded by the device: 65520 ids, checked by the host, and 65646, by the device
])
def test_small_calls(pe, orc, gpu, L, m, n):
    tabc = pe.dirichlet_table(L)
    tab = tabc.arrays()
    aa = pe.synthetic_protein(L - 1, L)
    ids = rand_ids(np.random.default_rng(L), aa, tab, m, n)
    idx = np.arange(n, dtype=np.int32)
    prob = orc.Problem(aa, tab, m, 8, 0.2, objset=1, p=2)
    with pe.Engine(aa, tabc, m, 8, 0.2, objectives=1, ref_p=2) as eng:
        scores = eng.evaluate(ids)
        for a, b in zip(scores, prob.evaluate(ids)):
            assert same(a, b)
        children, ops = eng.mutate(3, idx, ids, *scores)
        want, want_ops, *_ = prob.mutate(3, idx, ids, *scores)
        assert np.array_equal(children, want) and np.array_equal(ops, want_ops)
        for first in (0, ids.size // 2 + 1, ids.size - 1):
            bad = ids.copy()
            bad.reshape(-1)[first] = 64
            bad.reshape(-1)[-1] |= 128
            for call in (lambda: eng.evaluate(bad), lambda: eng.mutate(3, idx, bad, *scores)):
                with pytest.raises(pe.PeError) as e:
                    call()
                assert e.value.code == 1 and str(e.value).endswith(f"at {first}")


def test_large_calls_stage_in_parts(pe, gpu):
    """96 MB of ids pass through 16 MB of staging at a time: the scores of the parts taken
    one by one, the first bad id of a later part, and no device memory for a second copy."""
    import torch
    L, m, n = 1000, 8, 12000
    tabc = pe.dirichlet_table(L)
    tab = tabc.arrays()
    aa = pe.synthetic_protein(L - 1, L)
    ids = rand_ids(np.random.default_rng(L), aa, tab, m, n)
    with pe.Engine(aa, tabc, m, 8, 0.2, objectives=1, ref_p=2) as eng:
        eng.evaluate(ids[:1])
        before = torch.cuda.mem_get_info()[0]
        whole = eng.evaluate(ids)
        took = before - torch.cuda.mem_get_info()[0]     # the pool keeps what a call had at most
        # the solutions themselves: ids in rows of 1008, bit planes (96 words of 8 bytes a CDS), results
        own = n * m * (1008 + 96 * 8) + n * (16 + 8 + 12 + 8 * m + 4)
        assert took < own + (48 << 20)
        for k in range(0, n, 4000):
            for a, b in zip(whole, eng.evaluate(ids[k:k + 4000])):
                assert same(a[k:k + 4000], b)
        first = (50 << 20) + 7
        ids.reshape(-1)[[first, first + 1, ids.size - 1]] = 64
        with pytest.raises(pe.PeError) as e:
            eng.evaluate(ids)
        assert str(e.value).endswith(f"at {first}")
