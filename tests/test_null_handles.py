"""Null handles and bad arguments of entry points, rejected without a GPU."""
from rbffd_gpu_b200 import _lib


def test_wait_failure():
    assert _lib.load().rbffd_pde_inject_wait_failure(None, 1) == -1


def test_path():
    assert _lib.load().rbffd_pde_get_path(None, None, None) == -1


def test_solved_systems():
    assert _lib.load().rbffd_weights_get_solved(None, None) == -1
