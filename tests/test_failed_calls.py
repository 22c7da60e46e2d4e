"""Calls that fail halfway, and what the next calls then do.  The library's host
side runs here on a CUDA runtime without a GPU (fake_cudart.cpp: kernels do
nothing but leave their names in a log), in which any one call can be made to
fail; no device is touched."""
import ctypes
import glob
import os
import platform
import subprocess

import pytest

from conftest import PKG

HERE = os.path.dirname(os.path.abspath(__file__))
OOM = 3


class Fake:
    def __init__(self, api):
        self.api = api
        lib = api.lib()
        lib.fake_log.restype = ctypes.c_char_p
        lib.fake_fail.argtypes = [ctypes.c_char_p, ctypes.c_long]
        self.fail = lambda what, nth=1: lib.fake_fail(what.encode(), nth)

    def log(self):
        """The calls since the last look."""
        lines = self.api.lib().fake_log().decode().split("\n")[:-1]
        self.api.lib().fake_log_clear()
        return lines


@pytest.fixture(scope="module")
def fake_lib():
    import build as pkg_build
    pkg_build.build()
    objs = sorted(glob.glob(os.path.join(PKG, "_build", platform.machine(), "*.o")))
    out = os.path.join(PKG, "_build", platform.machine(), f"libimsrg_fake_{os.getpid()}.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I/usr/local/cuda/include",
                    os.path.join(HERE, "fake_cudart.cpp"), *objs, "-Wl,-Bsymbolic", "-o", out], check=True)
    yield out
    os.remove(out)


@pytest.fixture
def fake(fake_lib, monkeypatch):
    from imsrg_gpu import api
    monkeypatch.setattr(api, "LIB_PATH", fake_lib)
    monkeypatch.setattr(api, "_lib", None)
    f = Fake(api)
    yield f
    f.fail("", 0)


def _basis(api, emax=2):
    from imsrg_gpu.layout import ho_basis
    return api.Basis.from_dict(ho_basis(emax))


@pytest.mark.parametrize("what,status", [("malloc", OOM), ("stream", 2), ("event", 2)])
def test_adjoint_after_a_failed_preparation(fake, what, status):
    """Whichever allocation, stream or event of the first reverse-mode call
    fails, the call says so, a second failure too, nothing is launched on the
    half-built tables, and the call works once the cause is gone."""
    api = fake.api
    B = _basis(api)
    X, C, Y = api.Operator(B, -1), api.Operator(B, 1), api.Operator(B, 1)
    fake.log()
    api.commutator_adjoint(X, C, 1, Y)
    first = fake.log()
    launches = [x for x in first if x.startswith("launch")]
    n = 0
    while True:
        B2 = _basis(api)
        X2, C2, Y2 = api.Operator(B2, -1), api.Operator(B2, 1), api.Operator(B2, 1)
        fake.log()
        fake.fail(what, n + 1)
        try:
            api.commutator_adjoint(X2, C2, 1, Y2)
            break  # every one has had its turn
        except api.ImsrgError as e:
            assert e.status == status
        fake.fail(what, n + 1)
        with pytest.raises(api.ImsrgError):
            api.commutator_adjoint(X2, C2, 1, Y2)
        assert not [x for x in fake.log() if x.startswith("launch")]
        api.commutator_adjoint(X2, C2, 1, Y2)
        assert [x for x in fake.log() if x.startswith("launch")] == launches
        for o in (X2, C2, Y2, B2):
            o.close()
        n += 1
    assert n == len([x for x in first if x.startswith(what)]) > 0
    for o in (X, C, Y, B, X2, C2, Y2, B2):
        o.close()


def test_a_dot_product_needs_no_adjoint_tables(fake):
    """op_dot and white_adjoint allocate their own few words, not the adjoint's
    lists."""
    api = fake.api
    B = _basis(api)
    X, Y, Z = api.Operator(B, 1), api.Operator(B, -1), api.Operator(B, 1)
    fake.log()
    api.op_dot(X, Y)
    assert len([x for x in fake.log() if x.startswith("malloc")]) == 1
    api.white_adjoint(X, Y, Z)
    assert len([x for x in fake.log() if x.startswith("malloc")]) == 1
    api.op_dot(X, Y)
    assert not [x for x in fake.log() if x.startswith("malloc")]
    for o in (X, Y, Z, B):
        o.close()


@pytest.mark.parametrize("what", ["k_gemm_fp64", "k_assemble_2body", "k_e0", "malloc"])
def test_an_error_is_reported_once(fake, what):
    """The runtime keeps the last error until it is asked for; a call that has
    returned it leaves none for the next one, which may launch in another way."""
    api = fake.api
    B = _basis(api)
    ops = [api.Operator(B, h) for h in (-1, 1, 1)]
    B.profile(True)  # launches one by one
    fake.fail(what)
    with pytest.raises(api.ImsrgError):
        if what == "malloc":
            api.Operator(B, 1)
        else:
            api.commutator(*ops)
    api.commutator(*ops)
    api.mbpt2(ops[1])
    for o in (*ops, B):
        o.close()
