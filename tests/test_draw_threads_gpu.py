"""Ancestral draws by several threads, each on a tree of its own over the same
data: every call returns its own draws, as one after the other does."""
import threading

import numpy
import pytest

from p4gpu import pf, sim
from p4gpu.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("given", [False, True])
def test_threads_do_not_share_draws(given, lib):
    sites, calls = 30000, 60
    rng = numpy.random.default_rng(4)
    t = sim.yule_tree(6, rng)
    prob = sim.Problem(t, [sim.make_part(t, rng, "dna", sites)], "threads")
    first = Engine(prob)
    es = [first] + [Engine(prob, shared=(first.cData, first.cParts)) for _ in range(2)]
    u = [numpy.random.default_rng(k).random(sites) for k in range(len(es))]

    def draw(k):
        return pf.drawAncStates(es[k].cTree, 0, sites, u[k] if given else None, 10 + k)
    want = [[draw(k) for _ in range(4)][-1] for k in range(len(es))]   # graphs captured, buffers made
    assert not numpy.array_equal(want[0], want[1])
    wrong, start = [0] * len(es), threading.Barrier(len(es))

    def work(k):
        start.wait()
        for _ in range(calls):
            if not numpy.array_equal(draw(k), want[k]):
                wrong[k] += 1
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(es))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert wrong == [0] * len(es)
    for e in reversed(es):
        e.free()
