"""The autotuner's choice (talus_b200/autotune.py): the fastest candidate whose
solves reach the tolerance they were given."""
from types import SimpleNamespace

from talus_b200 import autotune


def test_a_solve_that_stops_short_is_told_from_one_that_hit_the_cap():
    report = lambda capped, residual: SimpleNamespace(cg_capped_solves=capped, cg_worst_relative_residual=residual)  # noqa: E731
    assert not autotune.stops_short(report(0, 1e-6), 1e-6)
    assert autotune.stops_short(report(0, 1.5e-3), 1e-6)
    assert not autotune.stops_short(report(3, 1.5e-3), 1e-6)


def test_the_fastest_that_converges_is_taken():
    c = lambda ms, short: {"ms_per_step": ms, "stopped_short": short}  # noqa: E731
    assert autotune.fastest([c(3.0, 0), c(2.0, 0), c(1.0, 5)]) == c(2.0, 0)
    assert autotune.fastest([c(3.0, 4), c(2.0, 4), c(1.0, 5)]) == c(2.0, 4)
