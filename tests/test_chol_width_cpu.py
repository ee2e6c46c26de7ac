"""The staging schedule of the blocked Cholesky update (test_chol_staging_cpu)
for a chain among longer ones: its column-block width follows from its own 3N,
the staging area from the largest chain of the launch."""
import pytest

from tests import test_chol_staging_cpu as S


def width(n):
    return min((S.SLOTS - S.FIRST_SLOT) * ((n + 7) // 8 * 8) // (2 * S.STRIDE), S.MAX_BLOCK) & ~7


@pytest.mark.parametrize("n_max", [300, 384, 729, 768, 1002, 1452, 1536])
def test_schedule_of_shorter_chains(monkeypatch, n_max):
    for n in sorted({300, 303, 330, 384, 450, 729, 768, 999, n_max}):
        if n <= n_max:
            nb = width(n)
            assert 16 <= nb <= width(n_max)  # the launch's staging area holds the chain's tiles
            monkeypatch.setattr(S, "MAX_BLOCK", nb)
            S.replay(n, n_max)
            monkeypatch.undo()
