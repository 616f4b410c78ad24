"""CPU test of the bench's count of its own kernels in a step, against the launches
that a step's host code enqueues (drift, box, keys, the sort, pack, force)."""
import importlib.util
import os

import pytest

from conftest import REPO


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(REPO, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_counts(bench):
    chain = 8 * (1 + 3 + 1)  # histogram, scan in three kernels, scatter
    assert bench.step_kernels(1 << 20) == 1 + 2 + chain + 1 + 1
    assert bench.step_kernels(131073) == bench.step_kernels(1 << 20)
    assert bench.step_kernels(131072) == 1 + 2 + 1 + 1 + 1
    # clock advance, fix-up, kick and clock end of their own
    assert bench.step_kernels(1 << 20, worklist=True) == 1 + 2 + chain + 1 + 1 + 4
