"""Selections whose values leave the ordinary range: normalised objectives whose squared
norm lies outside 1e-30 .. 1e30, for which the association evaluates every reference
point, and infinities and NaN in the objectives given to the dominance test, which passes
NaN differences over."""
import numpy as np
import pytest

from test_gpu_parity import same


def wide_values(N, M, kind, seed):
    """huge: the later fronts 1e17 behind the first.  tiny: a first front of a few solutions
    within 1e-17 of the ideal point, so that the nadir is the worst point."""
    rng = np.random.default_rng(seed)
    obj = rng.random((2 * N, M))
    obj /= np.linalg.norm(obj, axis=1, keepdims=True)
    if kind == "huge":
        obj[N // 2:] *= 1e17
    else:
        obj[M:] += 1e-3
        obj[:M] *= 1e-17
    return obj[rng.permutation(2 * N)].astype(np.float32)


def squared_norms(obj, front, info, M):
    """Of the normalised objectives of the solutions that the association takes."""
    ideal, nadir = (np.array(v[:M], np.float64) for v in (info.ideal, info.nadir))
    with np.errstate(all="ignore"):
        f = (obj[front >= 0] - ideal) / (nadir - ideal)
        return (f * f).sum(1)


# one and four solutions a warp (512 points, 4736 solutions), one and two chunks of points
CASES = [(64, 4, 4), (101, 4, 12), (259, 4, 32), (77, 6, 7), (131, 6, 11), (2371, 4, 13), (2370, 6, 7), (2368, 4, 32)]


def reference(pe, orc, N, M, p, obj, ext):
    tabc, aa = pe.dirichlet_table(3), pe.synthetic_protein(20, 1)
    return orc.Problem(aa, tabc.arrays(), 2, N, 0.05, objset=0 if M == 6 else 1, p=p).select(4, obj, ext)


@pytest.mark.parametrize("kind", ["huge", "tiny"])
@pytest.mark.parametrize("N,M,p", CASES)
def test_inputs_leave_the_pruned_range(pe, orc, N, M, p, kind):
    obj = wide_values(N, M, kind, N)
    _, front, _, info = reference(pe, orc, N, M, p, obj, obj[:M].copy())
    F = squared_norms(obj, front, info, M)
    assert (F > 1e30).any() if kind == "huge" else ((F > 0) & (F < 1e-30)).any()
    assert not info.cut                              # or nothing is associated


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["huge", "tiny"])
@pytest.mark.parametrize("N,M,p", CASES)
def test_association_outside_the_pruned_range(pe, orc, gpu, N, M, p, kind):
    obj = wide_values(N, M, kind, N)
    ext = obj[:M].copy()
    with pe.Engine(pe.synthetic_protein(20, 1), pe.dirichlet_table(3), 2, N, 0.05,
                   objectives=0 if M == 6 else 1, ref_p=p) as eng:
        gs, gf, ge, gi = eng.select(4, obj, ext)
    os_, of, oe, oi = reference(pe, orc, N, M, p, obj, ext)
    assert np.array_equal(gf, of) and same(ge, oe)
    assert (gi.rank_count, gi.last_front_size, gi.n_fronts, gi.cut, gi.hyp_exception) == \
        (oi.rank_count, oi.last_front_size, oi.n_fronts, oi.cut, oi.hyp_exception)
    assert np.array_equal(gs, os_)


def unusual_values(N, M):
    """One value in 200 infinite, NaN, subnormal or near the largest, and three rows of them."""
    rng = np.random.default_rng(N + M)
    obj = rng.random((2 * N, M)).astype(np.float32)
    for value in (np.inf, -np.inf, np.nan, 3e38, -3e38, 1e-40):
        obj[rng.random(obj.shape) < 0.005 / 6] = value
    obj[0] = np.nan                                  # every difference NaN
    obj[1] = np.inf
    obj[2, 1:] = np.nan                              # one difference left
    obj[3, 0] = -np.inf
    obj[4, M - 1] = -np.inf
    return obj, rng.random((M, M)).astype(np.float32)


@pytest.mark.parametrize("M", [4, 6])
@pytest.mark.parametrize("N", [7, 100, 200])
def test_unusual_values_still_fill_the_fronts(pe, orc, N, M):
    obj, ext = unusual_values(N, M)
    assert not np.isfinite(obj).all()
    assert reference(pe, orc, N, M, 2, obj, ext)[3].rank_count >= N


@pytest.mark.gpu
@pytest.mark.parametrize("M", [4, 6])
@pytest.mark.parametrize("N", [7, 100, 200])
def test_fronts_of_infinities_and_nan(pe, orc, gpu, N, M):
    """The fronts, which the dominance test alone decides."""
    obj, ext = unusual_values(N, M)
    with pe.Engine(pe.synthetic_protein(20, 1), pe.dirichlet_table(3), 2, N, 0.05,
                   objectives=0 if M == 6 else 1, ref_p=2) as eng:
        _, gf, _, gi = eng.select(4, obj, ext)
    _, of, _, oi = reference(pe, orc, N, M, 2, obj, ext)
    assert np.array_equal(gf, of)
    assert (gi.rank_count, gi.last_front_size, gi.n_fronts, gi.cut) == \
        (oi.rank_count, oi.last_front_size, oi.n_fronts, oi.cut)
