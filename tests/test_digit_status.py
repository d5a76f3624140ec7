"""CPU: every call that hands results of a grid to the host, or waits for them, reports a bounded wait of
the ring and column products that gave up (no run makes one give up, so the sources are read)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "springsteel.jl_gb300", "csrc")


def _body(source, name):
    text = open(os.path.join(CSRC, source)).read()
    start = re.search(r"^(?:extern \"C\" )?(?:static )?int32_t (?:\w+::)?%s\([^;{]*\{" % name, text, flags=re.M).end()
    depth, i = 1, start
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[start:i]


@pytest.mark.parametrize("source,name", [
    ("ss_api.cu", "copy_out"), ("ss_api.cu", "ss_grid_transform_to_host"), ("ss_api.cu", "ss_grid_synchronize"),
    ("ss_batch.cu", "ss_batch_synchronize"), ("ss_io.cpp", "ss_grid_save"), ("ss_regular.cu", "regular"),
    ("ss_regular.cu", "unstructured"), ("ss_regular.cu", "ss_relocate_grid"), ("ss_solver.cu", "ss_solve"),
    ("ss_solver.cu", "ss_problem_export"), ("ss_solver.cu", "ss_problem_collect_training")])
def test_timed_out_waits_are_reported(source, name):
    assert "digit_status(" in _body(source, name)
