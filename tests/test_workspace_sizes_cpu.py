"""Workspace of the FP64 calls: the arrays that the FP64 algorithm itself needs (its matrices, 16 bytes an
entry), plus at most 2 GiB where that lets the eigensolver take all matrices of a call together."""
import ctypes

import pytest

GIB = 1 << 30


@pytest.fixture(scope="module")
def lib():
    from khepri_gb300 import _capi, build
    build.build()
    return _capi.load()


def _bound(arrays, n, batch):
    own = 16 * n * n * batch * arrays
    return own * 1.01 + 64 * n * batch * 16 + (1 << 20), own


@pytest.mark.parametrize("nh", [9, 25, 49, 121, 169, 289])
@pytest.mark.parametrize("batch", [1, 2, 64, 256, 912, 4096])
def test_layer_modes(lib, nh, batch):
    n = 2 * nh
    most, own = _bound(3, n, batch)  # M, the eigensolver's Z, C W
    got = lib.khp_layer_modes_workspace(batch, nh)
    assert got <= (most if own >= 3 * GIB else most + 2 * GIB)


@pytest.mark.parametrize("nh", [9, 25, 49, 121])
@pytest.mark.parametrize("batch", [1, 16, 96, 256, 912])
@pytest.mark.parametrize("kinds,maps", [([1], [0]), ([1, 0], [0, 0]), ([1, 0, 1, 0, 1], [0, 0, 0, 0, 0]),
                                        ([1, 0, 1], [0, 0, 1])])
def test_solve_batched(lib, nh, batch, kinds, maps):
    n, L = 2 * nh, len(kinds)
    used = len({m for k, m in zip(kinds, maps) if k})
    arrays = 5 * used + 4 + sum(2 if k else 1 for k in kinds) + 4
    k, m = (ctypes.c_int32 * L)(*kinds), (ctypes.c_int32 * L)(*maps)
    most, _ = _bound(arrays, n, batch)
    got = lib.khp_solve_batched_workspace(batch, nh, L, k, m)
    free = 16 * n * n * batch * (arrays - 5 * used - 1)  # not in use during the eigensolver
    assert got <= (most if free >= 2 * GIB else most + 2 * GIB - free)
