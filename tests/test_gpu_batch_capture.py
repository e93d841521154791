"""A batch's queued scan when its graphs are captured again: with members whose scan
method changed since the first capture (other tables, other shared memory), and while
the generations of the graph that it replaces are still running."""
import pytest

from test_gpu_batch import population_equal

pytestmark = pytest.mark.gpu


def engines_of(pe, jobs):
    out = []
    for L, m, N, nt, kind in jobs:
        e = pe.Engine(pe.synthetic_protein(L, L), pe.dirichlet_table(L), m, N, 0.03, objectives=1, seed=L,
                      sl_threads=nt, sl_kind=kind)
        out.append(e)
    return out


def alone(pe, jobs, gens):
    want = []
    for e in engines_of(pe, jobs):
        with e:
            e.init()
            e.step(gens)
            want.append(e.population())
    return want


@pytest.mark.parametrize("first", [1, 0])
def test_scan_method_changed_between_captures(pe, gpu, first):
    """Two generations with one first pass, then one (a new graph) and two (the buffers'
    parity changed: captured again) with the other."""
    jobs = [(40, 2, 16, 64, pe.SL_LRCS), (300, 2, 32, 64, pe.SL_LRCS), (1400, 2, 16, 128, pe.SL_LRCS),
            (60, 3, 16, 128, pe.SL_HAIRPIN), (4200, 2, 8, 256, pe.SL_LRCS)]
    want = alone(pe, jobs, 5)
    engines = engines_of(pe, jobs)
    for e in engines:
        e.init()
        e.set_scan_method(first)
    with pe.Batch(engines) as b:
        b.set_scan_queue(True)
        b.step(2)
        b.synchronize()
        for e in engines:
            e.set_scan_method(1 - first)
        b.step(1)
        b.step(2)
        b.synchronize()
    for e, w in zip(engines, want):
        assert population_equal(e.population(), w)
        e.close()


def test_captured_again_while_running(pe, gpu):
    """Steps of 2 + 1 and 2 generations, queued without waiting: the second capture of the
    two-generation graph (the buffers' parity changed) writes job tables that the first
    one's generations, some milliseconds each, may not have read yet."""
    jobs = [(6000, 4, 512, 64, pe.SL_LRCS), (300, 2, 64, 64, pe.SL_LRCS)]
    want = alone(pe, jobs, 8)
    engines = engines_of(pe, jobs)
    for e in engines:
        e.init()
    with pe.Batch(engines) as b:
        b.set_scan_queue(True)
        b.step(3)
        b.step(2)
        b.step(3)
        b.synchronize()
    for e, w in zip(engines, want):
        assert population_equal(e.population(), w)
        e.close()
