"""The ensemble's default plan on the host: which kernel evaluates a system of N
bodies, and that its units of work and scratch fit the arenas."""
import pytest

import nbody_gb300 as nb


@pytest.mark.parametrize("newton3,limit,largest", [(False, 512 << 20, 283008),
                                                   (True, 1 << 30, 401152)])
def test_kinds_change_once_with_the_size(newton3, limit, largest):
    """Tasks, then pairs, then neither: no size between two that are
    evaluated as pairs is not (245,952 to 262,143 bodies were not)."""
    beyond = "blockpairs" if newton3 else "onesided"
    sizes = sorted({1, 2, 1023, 1024, 1025, *range(1100, 70000, 331), *range(70000, 450000, 1013),
                    245000, 245951, 245952, 250000, 262143, 262144, 269000, 269375, 269376,
                    largest - 1, largest, largest + 1, 381504, 381505, 1 << 20, 1 << 30})
    for n in sizes:
        kind, sets, scratch = nb.ensemble_kind(n, newton3)
        assert kind == ("tasks" if n < 1024 else "pairs" if n <= largest else beyond), n
        if kind != "pairs":
            assert scratch == 0
            continue
        assert 0 < scratch <= limit, n
        # units of work: the ensemble holds one for every 12 bodies, and four a system
        nsets, row = -(-n // 128), 4 if n < 8192 else 8
        items = sum(-(-(nsets - a) // sets) for a in range(0, nsets, row))
        assert items <= n // 12 + 4, n


def test_kind_refuses_no_bodies():
    with pytest.raises(nb.NbgbError):
        nb.ensemble_kind(0)
