"""The byte model of the ensemble passes' present loads and stores (no GPU):
the mesh once per pass, state per member, and less than the first program's."""
import pytest

from conftest import ROOT  # noqa: F401  (puts the repository root on sys.path)

L6 = (40962, 122880, 81920)


def test_moved_bytes():
    import bench

    p1, p2, p512 = (bench.inner_ensemble_moved_bytes(*L6, k) for k in (1, 2, 512))
    first = bench.inner_ensemble_pass_bytes(*L6, 512)
    assert set(p1) == set(first)
    for k in p1:
        assert p512[k] == pytest.approx(p1[k] + 511 * (p2[k] - p1[k]))
        assert p512[k] <= first[k] * 1.01  # (vertex and pv moved no less from the start)
    total = bench.inner_ensemble_step_bytes(*L6, 512, bench.inner_ensemble_moved_bytes)
    assert total / 1e9 == pytest.approx(19.74, abs=0.02)
