import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


@pytest.fixture(scope="session")
def oracle():
    from oracle import oracle as O
    O.port()
    return O


@pytest.fixture(scope="session")
def reflib(oracle):
    """The reference's own library, if it was compiled (oracle/_ref); else the test is skipped."""
    if not oracle.ref_available():
        pytest.skip("oracle/_ref/libojasx_lut.so not built")
    return oracle.RefLib()


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.set_device(0)
    return torch.device("cuda", 0)
