import os
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))
sys.path.insert(0, str(Path(__file__).resolve().parent))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (a B200) and the built libqpb.so")


# A test against the reference's compiled code, which can only be built where its
# sources are, has nothing to compare with where the library is absent: skipped
# with that reason, so that a run that stops at its first failure goes on.
@pytest.hookimpl(wrapper=True)
def pytest_runtest_setup(item):
    return (yield from _skip_without_library())


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    return (yield from _skip_without_library())


def _skip_without_library():
    from oracle import ref

    try:
        return (yield)
    except ref.LibraryMissing as missing:
        pytest.skip(str(missing))


def gpu_present() -> bool:
    try:
        from qoraphasecu_b200 import _lib

        return bool(_lib.load().qpb_cuda_available())
    except Exception:
        return False


@pytest.fixture(scope="session")
def gpu():
    """Fails (does not skip) a GPU test that runs without a device or the library."""
    from qoraphasecu_b200 import _lib

    lib = _lib.load()
    assert lib.qpb_cuda_available(), "gpu test run without a CUDA device"
    return lib


@pytest.fixture(scope="session")
def readme():
    from synthetic import readme_triangle

    return readme_triangle()


os.environ.setdefault("OMP_NUM_THREADS", str(len(os.sched_getaffinity(0))))
