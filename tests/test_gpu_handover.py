"""Hand-overs of the unweighted shared counts: a threshold above the smallest that
is honoured (2^19), passed by every block of the launch several times: 4.3e9
pairs of one s bin make 7e6 per block of at most 608, and every hand-over comes
at 2^20 or fewer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bintype", [0, 1])
def test_several_handovers(bintype):
    import fcfc_gb300 as fg
    n = 1 << 16
    kw = dict(nmu=2, with_mu_one=True) if bintype else {}
    pc = fg.PairCounter("box", bintype, box=200.0, smin=0, smax=20, ds=20, **kw)
    pc.set_hist_handover(1 << 20)
    rng = np.random.default_rng(1)
    a, b = 70.0 + rng.random((n, 3)), 70.0 + rng.random((n, 3))
    pc.load(0, a)
    pc.load(1, b)
    assert pc.count_pairs(0, 1).sum() == n * n
    assert pc.count_pairs(0).sum() == n * (n - 1) // 2
    cnt, status, _ = pc.count_batch([a, b], [200.0, 200.0])
    assert status == [0, 0]
    assert [c.sum() for c in cnt] == [n * (n - 1) // 2] * 2
