"""Shared helpers for the parity tests."""
import os

import numpy as np
import torch

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def load_golden(name):
    return dict(np.load(os.path.join(GOLDEN, name + ".npz")))


def from_bits(arr, dtype):
    """uint16 bit patterns (or fp32 values) stored in a fixture -> torch tensor of `dtype`."""
    if dtype in (torch.bfloat16, torch.float16):
        return torch.from_numpy(arr.view(np.int16).copy()).view(dtype)
    return torch.from_numpy(arr.copy())


def rel_l2(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def max_abs(a, b):
    return float((a.double() - b.double()).abs().max())


def kernels_of_capture(fn):
    """Mangled names of the kernels that ``fn`` launches, from the nodes of a graph captured around a second call."""
    import re
    return re.findall(r"_Z\w+", _dot_of_capture(fn))


def grids_of_capture(fn):
    """(mangled name, CTAs along x) of the kernels that ``fn`` launches."""
    import re
    return [(n, int(x)) for n, x in re.findall(r"(_Z\w+)[\\<]+(\d+)", _dot_of_capture(fn))]


def _dot_of_capture(fn):
    import tempfile
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "graph.dot")
        graph.debug_dump(path)
        with open(path) as f:
            return f.read()
