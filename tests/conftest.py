import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200) and the built native libraries")
    config.addinivalue_line("markers", "slow: long-running CPU case")


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    """A comparison with an oracle executable that was not built (it needs the reference tree) is
    skipped, on the GPU as on the CPU."""
    from tests import helpers as H
    outcome = yield
    e = outcome.excinfo[1] if outcome.excinfo else None
    if isinstance(e, FileNotFoundError) and e.filename in (H.ORACLE_EXEC, H.DROPIN_EXEC) and not os.path.exists(e.filename):
        outcome.force_exception(pytest.skip.Exception("oracle/_ref not built (needs the reference tree)"))
