"""Threads per CTA of the eigensolver: a size set by the caller holds for every batch; the autotuned one is
set only around calls of more than a matrix per SM."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    out = tmp_path_factory.mktemp("teams") / "libteams.so"
    subprocess.run([gxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "khepri_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "host", "teams_host.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    lib.host_chase_team.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_int]
    return lib


@pytest.mark.parametrize("tuned", [32, 64, 128, 256])
@pytest.mark.parametrize("batch", [1, 152, 153, 304, 305, 100000])
@pytest.mark.parametrize("n", [2, 18, 64, 242, 700])
def test_callers_choice_holds(lib, n, batch, tuned):
    assert lib.host_chase_team(n, batch, tuned) == max(64, tuned)
    assert lib.host_eig_team(0, n, tuned) == lib.host_eig_team(1, n, tuned) == tuned


@pytest.mark.parametrize("batch", [1, 152, 153, 304, 305])
@pytest.mark.parametrize("n", [2, 32, 33, 64, 65, 150, 151, 700])
def test_library_choice_is_a_team(lib, n, batch):
    t = lib.host_chase_team(n, batch, 0)
    assert t % 32 == 0 and 64 <= t <= (544 if batch <= 152 else 288)
    assert lib.host_eig_team(0, n, 0) == 256 and lib.host_eig_team(1, n, 0) in (64, 128, 256)


def test_autotuned_size_is_set_for_large_calls_only(monkeypatch):
    from khepri_gb300 import _capi, autotune
    calls = []

    class Fake:
        @staticmethod
        def khp_tune(*a):
            calls.append(a)
            return 0

    monkeypatch.setattr(_capi, "load", lambda: Fake)
    monkeypatch.setattr(autotune, "table", lambda: {18: {"eig_threads": 128}})
    with autotune.tuned_team(18, 153):
        assert calls == [(1, 18, 128)]
    assert calls.pop() == (1, 18, 0)
    calls.clear()
    with autotune.tuned_team(18, 152), autotune.tuned_team(50, 1000):
        assert calls == []
    with autotune.tuned_team(18):
        assert calls == [(1, 18, 128)]
