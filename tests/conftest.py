"""pytest configuration: the `gpu` marker, import paths, and shared helpers.

Layout of what the tests use:
  - `w4a8`   : the package's ctypes binding of libw4a8_b200.so (dgx-serving_b200/__init__.py)
  - `oracle` : the CPU restatement of the reference path (oracle/oracle.py; test infrastructure)
"""
import importlib.util
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))
sys.path.insert(0, ROOT)


def load_package():
    """The package directory is named dgx-serving_b200 (not an identifier); import it as dgx_serving_b200."""
    name = "dgx_serving_b200"
    if name in sys.modules:
        return sys.modules[name]
    path = os.path.join(ROOT, "dgx-serving_b200", "__init__.py")
    spec = importlib.util.spec_from_file_location(name, path, submodule_search_locations=[os.path.dirname(path)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules[name] = mod
    spec.loader.exec_module(mod)
    return mod


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box with -m gpu)")


@pytest.fixture(scope="session")
def w4a8():
    return load_package()


@pytest.fixture(scope="session")
def oracle():
    import oracle as O
    O.lib()
    return O


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a test marked gpu ran without a CUDA device")
    return torch.device("cuda:0")


def to_dev(a, dev):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def launched_kernels(call):
    """Mangled names of the kernels that call(stream) launches, in launch order: the call is captured, not run."""
    import torch
    from cuda.bindings import driver as D

    def ok(r):
        assert r[0] == D.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    stream = torch.cuda.Stream()
    ok(D.cuStreamBeginCapture(stream.cuda_stream, D.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL))
    try:
        call(stream.cuda_stream)
    finally:
        graph = ok(D.cuStreamEndCapture(stream.cuda_stream))
    names = []
    count = ok(D.cuGraphGetNodes(graph, 0))[1]
    for node in ok(D.cuGraphGetNodes(graph, count))[0]:
        if ok(D.cuGraphNodeGetType(node)) == D.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            p = ok(D.cuGraphKernelNodeGetParams(node))
            names.append(ok(D.cuFuncGetName(p.func) if int(p.func) else D.cuKernelGetName(p.kern)).decode())
    ok(D.cuGraphDestroy(graph))
    return names
