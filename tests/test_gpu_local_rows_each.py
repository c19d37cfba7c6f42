"""Rows of the local grids at the numbers of samples a thread (2, 4, 5) that test_gpu_local_rows.py leaves
out."""
import pytest

from test_gpu_local_rows import test_scores_follow_fp64 as follow

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,m", [(64, 17, 2), (96, 24, 1), (96, 27, 3)])
def test_scores_follow_fp64(built, n, R, m):
    follow(built, n, R, m)
