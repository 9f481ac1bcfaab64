import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); everything else runs on CPU")


@pytest.fixture(scope="session")
def oracle():
    from oracle import pyoracle
    pyoracle.build()
    return pyoracle


@pytest.fixture(scope="session")
def golden():
    return np.load(os.path.join(ROOT, "tests", "golden", "sampler_golden.npz"))


@pytest.fixture(scope="session")
def lib():
    """The CUDA library, built in-tree if it is missing (nvcc cross-compiles without a GPU)."""
    from molla_b200 import build, capi
    build.build_library()
    build.build_library(testing=True)
    return capi.lib()


@pytest.fixture(scope="session")
def dev():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


@pytest.fixture(params=["chosen", "tiles", "clusters"])
def route(request, lib, dev):
    """Which row kernels a test's calls go through: those that the library chooses for their size, or one and
    the same kind for all of them. The latter takes the testing build, which counts its launches: a test that did
    not run what its name says fails."""
    if request.param == "chosen":
        yield request.param
        return
    import ctypes as C
    from helpers import ROUTES
    from molla_b200 import capi
    counts = (C.c_int64 * 2)()
    with capi.testing_library() as T:
        T.molla_sample_debug_launches(counts)
        T.molla_sample_debug_knobs(ROUTES[request.param])
        try:
            yield request.param
        finally:
            T.molla_sample_debug_knobs(0)
            T.molla_sample_debug_launches(counts)
    cluster, tiles = counts
    assert (cluster > 0, tiles > 0) == (request.param == "clusters", request.param == "tiles"), (cluster, tiles)
