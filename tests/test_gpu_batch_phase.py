"""Steps that a batch captured hold every member's MacCormack signs, which
depend on the member's own step counter: a member that advances alone between
two runs of the batch makes them stale."""
import numpy as np
import pytest

from test_gpu_batch import NT, SHAPES, _results, _same, _sim, _synthetic

pytestmark = pytest.mark.gpu
cgfdm = pytest.importorskip("cgfdm")


def _scenarios():
    """Members stretched in z only and skewed ones, side by side."""
    scs = [_synthetic(*d, seed=50 + q) for q, d in enumerate(SHAPES[:4])]
    for sc in scs[::2]:
        c = sc["cjm"].reshape(13, -1)
        for f in (1, 2, 3, 5):
            c[f] = 0.0
    return scs


@pytest.mark.parametrize("graph", [False, True])
def test_member_advanced_alone_between_batch_runs(gpu_available, graph):
    assert NT == 24
    scs = _scenarios()
    alone = []
    for sc in scs:
        s = _sim(sc)
        s.run(NT)
        alone.append(_results(s))
        s.close()
    sims = [_sim(sc) for sc in scs]
    with cgfdm.Batch(sims, graph=graph) as b:
        b.run(17)  # every phase captured, one step replayed
        extra = (1, 3, 0, 2)
        for s, n in zip(sims, extra):
            if n:
                s.run(n)
        b.run(4)
        b.synchronize()
        for s, n in zip(sims, extra):
            s.run(NT - 21 - n)
        for s, r in zip(sims, alone):
            got = _results(s)
            assert np.abs(got[2]).max() > 0
            _same(got, r)
            s.close()
