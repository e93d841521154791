"""Nearest-reference-point search (k_assoc) at the sizes where its route changes: one
and four solutions per warp (512 points and 4736 solutions), one and several chunks of staged points
(6144 points of four objectives, 3072 of six), solution counts that do not fill a CTA,
and objectives whose normalised values have no usable magnitude.  Whole selections
against the oracle, exactly."""
import numpy as np
import pytest

from test_gpu_parity import same, select_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["uniform", "rounded", "flat", "huge", "tiny"])
@pytest.mark.parametrize("N,M,p", [
    (33, 4, 1), (101, 4, 12), (101, 4, 13),       # 4, 455 and 560 points
    (259, 4, 32),                                 # 6545 points: two chunks
    (77, 6, 6), (77, 6, 7), (131, 6, 11),         # 462, 792 and 4368 points (two chunks)
    (2367, 4, 13), (2371, 4, 13), (2370, 6, 7),   # either side of four solutions a warp
    (2368, 4, 12), (2368, 4, 32),                 # few points; four solutions a warp, two chunks
])
def test_selection_at_the_edges_of_the_association(pe, orc, gpu, N, M, p, kind):
    tabc = pe.dirichlet_table(3)
    aa = pe.synthetic_protein(20, 1)
    rng = np.random.default_rng(N * M + p)
    obj = select_inputs(rng, N, M) if N >= 64 else rng.random((2 * N, M)).astype(np.float32)
    if kind == "rounded":
        obj = np.round(obj * 6) / np.float32(6)
    elif kind == "flat":
        obj[:, 1] = np.float32(0.25)              # a span of the fallback nadir, or zero
    elif kind == "huge":
        obj[: N // 2] *= np.float32(1e25)         # squared norms beyond the pruned range
    elif kind == "tiny":
        obj *= np.float32(1e-3)
    obj = obj.astype(np.float32)
    ext = obj[:M].copy()
    objset = 0 if M == 6 else 1
    with pe.Engine(aa, tabc, 2, N, 0.05, objectives=objset, ref_p=p) as eng:
        gs, gf, ge, gi = eng.select(4, obj, ext)
    os_, of, oe, oi = orc.Problem(aa, tabc.arrays(), 2, N, 0.05, objset=objset, p=p).select(4, obj, ext)
    assert np.array_equal(gf, of)
    assert same(ge, oe)
    assert (gi.rank_count, gi.last_front_size, gi.n_fronts, gi.cut, gi.hyp_exception) == \
        (oi.rank_count, oi.last_front_size, oi.n_fronts, oi.cut, oi.hyp_exception)
    assert np.array_equal(gs, os_)
