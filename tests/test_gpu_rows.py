"""Codon ids on their way between the caller's rows of L bytes and the engine's padded
rows: row lengths below, at and above multiples of 16, and the refusal of an id out of
range with the index of the first one, found by the host up to 64 KB of ids (256 x 256
exactly) and by the device above."""
import numpy as np
import pytest

from test_gpu_parity import rand_ids, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,m,n", [(3, 2, 5), (15, 3, 7), (16, 2, 9), (17, 3, 11), (31, 2, 3), (32, 5, 4), (47, 3, 1),
                                   (257, 2, 21), (256, 2, 128), (257, 2, 128)])
def test_rows_in_and_out(pe, orc, gpu, L, m, n):
    tabc = pe.dirichlet_table(L)
    tab = tabc.arrays()
    aa = pe.synthetic_protein(L - 1, L)
    ids = rand_ids(np.random.default_rng(L), aa, tab, m, n)
    prob = orc.Problem(aa, tab, m, 8, 0.2, objset=1, p=2)
    with pe.Engine(aa, tabc, m, 8, 0.2, objectives=1, ref_p=2) as eng:
        scores = eng.evaluate(ids)
        for a, b in zip(scores, prob.evaluate(ids)):
            assert same(a, b)
        children, ops = eng.mutate(3, np.arange(n, dtype=np.int32), ids, *scores)
        want, want_ops, *_ = prob.mutate(3, np.arange(n, dtype=np.int32), ids, *scores)
        assert np.array_equal(children, want) and np.array_equal(ops, want_ops)
        bad = ids.copy()
        flat = bad.reshape(-1)
        first = flat.size // 2 + 1
        flat[first], flat[-1] = 64, 255
        for call in (lambda: eng.evaluate(bad),
                     lambda: eng.mutate(3, np.arange(n, dtype=np.int32), bad, *scores)):
            with pytest.raises(pe.PeError) as e:
                call()
            assert e.value.code == 1 and f"at {first}" in str(e.value)
        for a, b in zip(scores, eng.evaluate(ids)):
            assert same(a, b)
