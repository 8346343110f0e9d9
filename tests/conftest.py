"""Test configuration: the `gpu` marker and import paths.

Tests marked `gpu` need a B200 and call the CUDA library through its C ABI;
everything else runs on a CPU-only host."""
import os
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (REPO, os.path.join(REPO, "black-hole-simulator_b200"), os.path.join(REPO, "tests")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200)")


@pytest.fixture(autouse=True)
def launch_knobs_restored(request):
    """The corrected scheme's launch knobs are per process: a GPU test that
    sets them leaves them as they were (else the tests after it no longer run
    by the library's rules)."""
    if request.node.get_closest_marker("gpu") is None:
        yield
        return
    from bhgpu import fixed as fx
    before = {(p, k): fx.tune_get(p, k) for p in fx.PRECISIONS for k in fx.TUNE_KNOBS}
    yield
    for (p, k), v in before.items():
        fx.tune_set(p, k, v)
