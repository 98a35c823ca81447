import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import __graft_entry__ as entry  # noqa: E402

pkg = entry.load_package()


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200) and the built library")


@pytest.fixture(scope="session")
def oracle():
    return entry.load_oracle()


@pytest.fixture(scope="session")
def pt():
    return pkg


@pytest.fixture(scope="session")
def ctx():
    """A context on the wavefront. One whose schedule nobody chose runs small
    refines on the megakernel: tests of that make their own."""
    from oxideav_render_b200 import abi, api
    c = api.Context(0)
    c.set_schedule(abi.PT_SCHEDULE_WAVEFRONT)
    yield c
    c.close()
