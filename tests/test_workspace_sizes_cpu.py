"""Workspace sizes of joins at the row counts where a path ends: the sorted right
side holds what the sort takes (below 2^30 rows), and no size is computed by a
loop that cannot end. Run in a child process, so that a hang is a failure."""
import subprocess
import sys

import pytest

from yallasql_b200 import _abi as A

CHILD = """
import sys
from yallasql_b200 import _abi as A
print(int(A.load().yq_join_workspace_size(1000, int(sys.argv[1]))))
"""


def size(right_rows):
    r = subprocess.run([sys.executable, "-c", CHILD, str(right_rows)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    return int(r.stdout)


def test_join_sizes_at_the_ends(yq):
    sort_max = (1 << 30) - 1
    inside, past = size(sort_max), size(sort_max + 1)
    assert inside > 16 * sort_max  # the slots alone
    assert past < 40 * (sort_max + 1) < inside  # no sorted table: nothing of it in the size
    for rows in (1_431_655_766, (1 << 31) + 1, (1 << 32) - 1):
        assert past <= size(rows) < 40 * rows


@pytest.mark.parametrize("rows", [0, 1, 1024, 1025, 4096, 4097, 8193])
def test_join_sizes_grow(yq, rows):
    assert 0 < int(A.load().yq_join_workspace_size(1, rows)) <= int(A.load().yq_join_workspace_size(1000, rows + 1))
