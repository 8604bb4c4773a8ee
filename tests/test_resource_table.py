"""Every kernel that profiles/ptxas_resources.md lists is in the sources, and the other way round."""
import os
import re

from test_overlapped_launch_contract import CSRC, KERNELS


def test_the_table_lists_the_kernels_of_the_tree():
    with open(os.path.join(os.path.dirname(CSRC), "profiles", "ptxas_resources.md")) as f:
        table = set(re.findall(r"^\| \w+\.cu \| `(\w+)`", f.read(), re.M))
    assert len(table) > 30 and table == set(KERNELS)
