"""What bench.py's batched line says about the launches it timed, without a GPU."""
import argparse
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench


@pytest.mark.parametrize("split_pass,block_lines,tiles", [(0, 0, True), (0, 128, True), (0, 64, False), (1, 0, False),
                                                          (-1, 0, False)])
def test_batched_line_reports_the_form_that_ran(split_pass, block_lines, tiles):
    # the tile form has no block waves and times no candidates
    r = bench.batch_schedule(argparse.Namespace(split_pass=split_pass, block_lines=block_lines), 8, 456)
    assert r["form"] == ("tiles" if tiles else "marches") and r["blocks"] == 456
    assert ("waves" not in r and "autotuned" not in r["how"]) if tiles else r["waves"] == 8
