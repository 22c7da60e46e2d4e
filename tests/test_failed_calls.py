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
    api.lib().fake_fail_none()


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


# calls of a live split commutator between its exponents and their clearing
HALFWAY = ["k_oz_slice", "k_oz_mma", "k_ph_list", "k_assemble_2body"]


def _split_basis(api, emax=2):
    """A basis whose split engine is tuned, and operators of it."""
    B = _basis(api, emax)
    ops = [api.Operator(B, h) for h in (-1, 1, 1)]
    api.commutator(*ops, precision="ozaki")
    return B, ops


def _cleared_before_the_next_front(lines):
    """The block exponents are set to zero ahead of the first kernel that takes
    their maxima (k_front)."""
    front = next(k for k, x in enumerate(lines) if "k_front" in x and x.startswith("launch"))
    return any(x.startswith("memset") and k + 1 < len(lines) and lines[k + 1] != "failed"
               for k, x in enumerate(lines[:front]))


def _fail_a_live_commutator(fake, B, ops, what, clear_fails=False):
    api = fake.api
    B.profile(True)  # launches one by one, no graph
    fake.log()
    fake.fail(what)
    if clear_fails:
        fake.fail("memset")
    with pytest.raises(api.ImsrgError):
        api.commutator(*ops, precision="ozaki")
    B.profile(False)
    return fake.log()


@pytest.mark.parametrize("what", HALFWAY)
@pytest.mark.parametrize("clear_fails", [False, True])
@pytest.mark.parametrize("emax", [2, 5])
def test_cached_commutator_after_a_failed_one(fake, what, clear_fails, emax):
    """Block exponents are maxima taken from zero, and a commutator's last kernel
    leaves them zero.  One that fails before it leaves them large, and a cached
    graph, which holds no memset, would take them over and lose digits."""
    api = fake.api
    if emax == 5 and what == "k_ph_list":
        what = "k_ph_patches"
    B, ops = _split_basis(api, emax)
    for _ in range(2):
        api.commutator(*ops, precision="ozaki")  # captured, then replayed
    lines = _fail_a_live_commutator(fake, B, ops, what, clear_fails)
    api.commutator(*ops, precision="ozaki")
    after = fake.log()
    assert "replay" in after and "end of capture" not in after
    start = next(k for k, x in enumerate(lines) if x == "failed")
    assert _cleared_before_the_next_front(lines[start:] + after)
    # once, not with every call from then on
    api.commutator(*ops, precision="ozaki")
    assert not [x for x in fake.log() if "memset" in x]
    for o in (*ops, B):
        o.close()


def test_a_capture_holds_no_memset_and_clears_nothing(fake):
    """Capturing runs nothing: it neither takes a memset in nor, if it fails,
    leaves the exponents' state changed."""
    api = fake.api
    B, ops = _split_basis(api)
    lines = _fail_a_live_commutator(fake, B, ops, "k_oz_mma", clear_fails=True)
    fake.fail("instantiate")
    with pytest.raises(api.ImsrgError):
        api.commutator(*ops, precision="ozaki")
    lines += fake.log()
    api.commutator(*ops, precision="ozaki")
    lines += fake.log()
    assert not [x for x in lines if x.startswith("capture memset")]
    assert _cleared_before_the_next_front(lines[lines.index("failed"):])
    for o in (*ops, B):
        o.close()


def test_step_graphs_after_a_failed_commutator(fake):
    """The single flow's step graph and the lockstep flow of a batch."""
    api = fake.api
    B, ops = _split_basis(api)
    HS, G = api.Operator(B, 1), api.Operator(B, -1)
    launch = api.lib()["_ZN5imsrg17flow_graph_launchEP11imsrg_basis"]
    # no kernel runs here, so the flow stops before its first step; its graph is built
    api.magnus_decouple_graph(HS, G, max_steps=1, precision="ozaki")
    lines = _fail_a_live_commutator(fake, B, ops, "k_ph_list", clear_fails=True)
    assert launch(B.handle) == 0
    after = fake.log()
    assert "replay" in after
    assert _cleared_before_the_next_front(lines[lines.index("failed"):] + after)
    bt = api.Batch([B])
    bt.magnus_decouple([HS], [G], max_steps=1, precision="ozaki")
    sizes = {x for x in fake.log() if x.startswith("memset")}
    _fail_a_live_commutator(fake, B, ops, "k_ph_list", clear_fails=True)
    bt.magnus_decouple([HS], [G], max_steps=1, precision="ozaki")
    assert {x for x in fake.log() if x.startswith("memset")} - sizes
    bt.close()
    for o in (HS, G, *ops, B):
        o.close()


@pytest.mark.parametrize("what", ["k_oz_mma", "k_oz_slice", "k_assemble_2body"])
def test_batch_after_a_failed_batch(fake, what):
    api = fake.api
    made = [_split_basis(api, e) for e in (2, 3)]
    bt = api.Batch([b for b, _ in made])
    args = [[ops[k] for _, ops in made] for k in range(3)]
    for _ in range(2):
        bt.commutator(*args)
    for b, _ in made:
        b.profile(True)
    fake.log()
    fake.fail(what)
    with pytest.raises(api.ImsrgError):
        bt.commutator(*args)
    for b, _ in made:
        b.profile(False)
    lines = fake.log()
    bt.commutator(*args)
    after = fake.log()
    assert "replay" in after and "end of capture" not in after
    # every basis whose part before the products was enqueued
    fronts = len([x for x in lines if "k_front" in x]) if what != "k_oz_slice" else 1
    both = lines[lines.index("failed"):] + after[:after.index("replay")]
    assert len([x for x in both if x.startswith("memset")]) >= min(fronts, 2)
    bt.close()
    for b, ops in made:
        for o in (*ops, b):
            o.close()
