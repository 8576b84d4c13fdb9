import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, "tests", "golden", "ref_golden.npz")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


@pytest.fixture(scope="session")
def oracle():
    from oracle import oracle as O

    O.lib()
    return O


@pytest.fixture(scope="session")
def host_index(tmp_path_factory):
    """tests/native/host_index.cu: host functions of the kernels' headers."""
    from cugridder_b200 import build as B

    so = str(tmp_path_factory.mktemp("native") / "host_index.so")
    src = os.path.join(ROOT, "tests", "native", "host_index.cu")
    subprocess.check_call([B._nvcc(), "-shared", "-o", so, src, "-I", B.CSRC] + B.flags())
    return ctypes.CDLL(so)


@pytest.fixture(scope="session")
def golden():
    if not os.path.exists(GOLDEN):
        pytest.skip("golden outputs of the reference build not recorded")
    return dict(np.load(GOLDEN))


@pytest.fixture(scope="session")
def torch_cuda():
    import torch

    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return torch
