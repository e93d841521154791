"""pe_hairpin_noalloc reads 16-byte pieces where the caller's array covers them: arrays
that start at every byte offset, rows of one to a few words, and single rows, against
the allocating evaluator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,m,n", [(3, 1, 1), (10, 1, 3), (11, 2, 5), (16, 3, 7), (43, 1, 2), (86, 2, 9), (333, 3, 4)])
def test_array_at_every_alignment(pe, gpu, L, m, n):
    import torch
    tabc = pe.dirichlet_table(L)
    tab = tabc.arrays()
    aa = pe.synthetic_protein(L - 1, L)
    rng = np.random.default_rng(L)
    ids = (tab["start"][aa] + (rng.random((n, max(m, 2), L)) * tab["count"][aa]).astype(np.int64)).astype(np.uint8)
    if m == 1:
        ids[:, 1] = ids[:, 0]                     # the engine takes two CDSs or more
    with pe.Engine(aa, tabc, ids.shape[1], 8, 0.05, objectives=pe.OBJ_BASE4, ref_p=2) as eng:
        obj, _, pql = eng.evaluate(ids)
    nt = np.asarray(tab["nt"])[ids[:, :m]].astype(np.uint8).ravel()
    dev = torch.device("cuda", 0)
    stream = torch.cuda.current_stream(dev)
    for off in range(17):
        raw = torch.full((off + nt.size,), 3, dtype=torch.uint8, device=dev)
        raw[off:] = torch.from_numpy(nt).to(dev)
        val = torch.zeros(n, dtype=torch.float32, device=dev)
        got = torch.zeros((n, 3), dtype=torch.int32, device=dev)
        cds = torch.zeros(n, dtype=torch.int8, device=dev)
        pe.hairpin_noalloc(raw.data_ptr() + off, n, m, L, val.data_ptr(), got.data_ptr(), cds.data_ptr(),
                           stream.cuda_stream)
        stream.synchronize()
        assert np.array_equal(val.cpu().numpy().view(np.uint32), obj[:, 3].view(np.uint32)), off
        assert np.array_equal(got.cpu().numpy(), pql), off
