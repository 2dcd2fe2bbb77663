"""pytest configuration: registers the `gpu` marker and puts the repository root on sys.path."""
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a B200; run with -m gpu on the GPU box")


@pytest.fixture(scope="session")
def golden():
    import numpy as np

    return np.load(ROOT / "tests" / "golden" / "quant_golden.npz")


@pytest.fixture(autouse=True)
def _launch_mode(request):
    """a GPU test that set the dependent-launch mode leaves the mode the package starts with to the next one."""
    yield
    if request.node.get_closest_marker("gpu"):
        from lightly_trian_quant_b200 import ops

        ops.set_pdl(None)
