import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
# accusim, the framework the plug-ins plug into, from the repository's offline install (baseline/_ref) when it is
# not installed in the environment
from devinproj_b200 import _accusim  # noqa: E402
GOLDEN = os.path.join(ROOT, "tests", "golden")


if _accusim.accusim is None:
    # tests of the C ABI, the engine and the oracle run without accusim; one that asks for it is skipped, not passed
    collect_ignore = ["test_convert.py"]   # asks for it when it is collected

    @pytest.hookimpl(hookwrapper=True)
    def pytest_runtest_call(item):
        outcome = yield
        exc = outcome.excinfo[1] if outcome.excinfo else None
        if isinstance(exc, ImportError) and ("No module named 'accusim" in str(exc) or str(exc) == _accusim.MISSING):
            outcome.force_exception(pytest.skip.Exception("needs accusim, which is not importable"))

    def pytest_report_header():
        return "accusim is not importable: the tests that need it are skipped"


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: longer CPU or GPU case")


def load_golden(name):
    with np.load(os.path.join(GOLDEN, name + ".npz"), allow_pickle=False) as z:
        return {k: z[k] for k in z.files}


@pytest.fixture
def golden():
    return load_golden
