"""Reading trajectory records: one at a time, many at once and across the end of the ring give the
same records, also when the lattices of a batch count differently; none yet reads as zeros."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ensemble():
    import gauge_higgs_b200 as gh
    e = gh.Ensemble([[2, 2], [3, 2], [2, 2]], gh.FundamentalRep(2), seeds=[1, 2, 3], beta=2.0, kappa=0.2, nmd=2)
    e.hot(0.8)
    e.phi_gaussian(12345, 0.3)
    return e


def test_one_at_a_time_equals_many():
    a, b, c = ensemble(), ensemble(), ensemble()
    n = 1030                                   # past the ring's 1024
    one = np.concatenate([a.run(1) for _ in range(n)])
    many = b.run(n)
    c.enqueue(n)
    c.sync()
    assert np.array_equal(one, many)
    assert np.array_equal(c.records(1024), many[-1024:]) and np.array_equal(c.records(3), many[-3:])
    assert np.array_equal(one["traj"][:, 0], np.arange(1, n + 1))
    for e in (a, b, c):
        e.close()


def test_counters_apart_and_zeros():
    e = ensemble()
    assert not e.records(2).view(np.uint8).any()
    e.run(2)
    r = e.records(3)
    assert not r[0].view(np.uint8).any() and np.array_equal(r["traj"][1:], [[1, 1, 1], [2, 2, 2]])
    e.set_traj_count(1, 1022)
    r = e.run(4)
    assert np.array_equal(r["traj"], [[3, 1023, 3], [4, 1024, 4], [5, 1025, 5], [6, 1026, 6]])
    dH, acc = e.trajectory()
    last = e.records(1)[0]
    assert np.array_equal(last["dH"], dH) and np.array_equal(last["accepted"].astype(bool), acc)
    e.close()
