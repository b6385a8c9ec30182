import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); run with -m gpu")


@pytest.fixture(scope="session")
def oracle():
    from oracle import oracle as O

    O.lib()
    return O


@pytest.fixture(scope="session")
def cp():
    import circlepacking_b200 as cp

    cp.lib()
    return cp


@pytest.fixture(scope="session")
def ref():
    from oracle import refcheck

    if not refcheck.available():
        # built from the reference's sources: without them there is nothing to build it from (the
        # golden vectors it left stand in, tests/test_golden.py); with them it is missing by mistake
        from __graft_entry__ import reference_dir

        if not os.path.isdir(reference_dir()):
            pytest.skip(f"no reference sources to build the reference checker {refcheck.SO} from")
        pytest.fail(f"reference checker {refcheck.SO} is missing (build: make -C oracle ref)")
    refcheck.lib()
    return refcheck
