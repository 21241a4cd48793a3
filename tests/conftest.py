"""Shared test set-up: builds the library and the oracle once per session."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "oracle"))
sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (runs the sm_103a kernels)")
    # an empty reference tree is an absent one (oracle.build_reference has the same
    # rule): the test that compiles against its sources then skips
    import oracle
    if os.path.isdir(oracle.REF_DIR) and not os.listdir(oracle.REF_DIR):
        os.environ["CPC_REFERENCE_DIR"] = os.path.join(ROOT, "oracle", "no_reference")


@pytest.fixture(scope="session", autouse=True)
def _built():
    from corr_pc_gb300 import build
    build.build()
    import oracle
    oracle.build_port()
    yield
