"""Given windows of the travel-time stage on the host (no GPU)."""
import numpy as np

from sparc_flows_gb300 import ttadjoint as TT


def test_given_windows_are_any_iterable():
    """The windows of a source are taken in order from whatever can be iterated, as many as it has receivers."""
    tt = object.__new__(TT.TTAdjoint)
    tt.nx, tt.nt, tt.nb, tt.xlength_cm, tt.plan = 64, 100, 2, 64 * 0.78125e8, None
    modes, x00s = {1: (2.0, 9.0, 4.0)}, [-4.0, 9.0]
    picked = tt._rows(1, x00s, modes, 0.5, None)
    n = [int((picked[:, 0] == b).sum()) for b in range(2)]
    want = {b: [(5 + i, 20 + i) for i in range(n[b] + 3)] for b in range(2)}
    rows = tt._rows(1, x00s, modes, 0.5, want)
    assert min(n) > 0 and [tuple(r) for r in rows[:, 4:6].tolist()] == want[0][:n[0]] + want[1][:n[1]]
    for form in (iter, tuple, np.asarray, lambda v: (w for w in v)):
        assert np.array_equal(tt._rows(1, x00s, modes, 0.5, {b: form(v) for b, v in want.items()}), rows)
