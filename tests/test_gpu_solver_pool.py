"""A system's first solve launches its kernels, later ones replay a graph: the
same kernels on the same data, so the same bits. Solver objects share a bounded
pool of streams and pinned blocks: more objects alive than the pool keeps, and
objects made and dropped by several threads, give what one alone gives."""

import threading

import pytest

from pymatting_b200.synthetic import make_matting_problem

pytestmark = pytest.mark.gpu


def _problems(n):
    return [make_matting_problem(60 + 7 * k, 90 - 3 * k, k + 1, sigma=1.0, band=1,
                                 unknown_fraction=0.3)[:2] for k in range(n)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_first_solve_and_replay_are_equal(gpu, precision):
    import torch
    from pymatting_b200.batch import AlphaBatch
    probs = _problems(3)
    batch = AlphaBatch([p[0] for p in probs], [p[1] for p in probs], precision=precision)
    first = batch.solve().clone()
    assert torch.equal(first, batch.solve().clone())
    assert torch.equal(first, batch.solve())


def test_more_objects_than_the_pool_keeps_and_threads(gpu):
    import torch
    import pymatting_b200 as pm
    from pymatting_b200.batch import AlphaBatch
    probs = _problems(4)
    one = [pm.solve_alpha([i], [t])[0] for i, t in probs]
    alive = [AlphaBatch([probs[k % 4][0]], [probs[k % 4][1]], precision="mixed")
             for k in range(12)]
    for k, b in enumerate(alive):
        assert torch.equal(b.alphas(b.solve())[0].cpu(), torch.as_tensor(one[k % 4]))
    del alive, b
    bad = []

    def work(k):
        for _ in range(3):
            a = pm.solve_alpha([probs[k][0]], [probs[k][1]])[0]
            if not torch.equal(torch.as_tensor(a), torch.as_tensor(one[k])):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
