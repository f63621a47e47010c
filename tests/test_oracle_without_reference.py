"""Where the reference's compiled code was not built, the oracle's descent stands in for it."""
import bk_b200 as bk
from oracle import oracle as O


def test_descent_without_the_reference_library(monkeypatch):
    monkeypatch.setattr(O, "ref_lib", lambda: None)
    for n in (3, 20, 32):
        for start in bk.random_states(n, 100 + n, 20):
            for budget in (0, 3 * n + 1):
                assert O.steepest_descent(n, int(start), budget, use_ref=True) == O.steepest_descent(n, int(start), budget)
