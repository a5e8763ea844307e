"""The range of the FP64 form's breadth-first draws, from the workspace a
session asks for (no GPU work): they hold a tree node in 32 bits, so a mode whose
tree has more than 2^31 nodes keeps the depth-first kernel, whose state per
sample is smaller."""
import ctypes

import pytest


def size(dims, R, J):
    from rdist_tensor_gb300 import _lib

    lib = _lib.load()
    cfg = _lib.AlsConfig()
    cfg.N, cfg.R, cfg.nnz, cfg.J_max = len(dims), R, 1000, J
    for k, d in enumerate(dims):
        cfg.dims[k] = d
    cfg.sampler, cfg.precision, cfg.preprocessing = 1, 0, 0
    pers, setup = ctypes.c_size_t(), ctypes.c_size_t()
    assert lib.exafac_als_workspace_size(ctypes.byref(cfg), ctypes.byref(pers), ctypes.byref(setup)) == 0
    return pers.value


@pytest.mark.parametrize("rows,R,breadth", [(1 << 28, 1, True), (1 << 30, 1, True), ((1 << 30) + 1, 1, False),
                                            (3 << 30, 2, False), (3 << 30, 3, True)])
def test_node_range(rows, R, breadth):
    J = 1 << 23
    assert J * R * (R + 1) // 2 >= 1 << 22
    # bytes per sample (other arrays sized by the longest mode are the same in both)
    per_sample = (size((rows, 50, 40), R, 2 * J) - size((rows, 50, 40), R, J)) / J
    small = (size((1 << 29, 50, 40), R, 2 * J) - size((1 << 29, 50, 40), R, J)) / J
    if breadth:
        assert abs(per_sample - small) < 1
    else:
        assert per_sample < small - 100
