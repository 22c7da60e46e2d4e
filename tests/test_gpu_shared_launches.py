"""One commutator by its different launch sequences: the graph of a device call
(on small bases and in split precision a chain of launches that several parts
share, else branches), the launches one by one on one stream (kernel timing
on), and the call on packed host operands.  They run the same arithmetic, so
they agree bit for bit; emax 1 to 4 lie on one side of the line between the
sequences, emax 5 on the other, and the sizes give odd term counts, few blocks
and ragged last CTAs.

Tolerances against the oracle: the FP64 bar max |gpu - oracle| <= 1e-10 max
|oracle|; six digits drop at most 2^-42 (6 + 2) K max|A| max|B| per product, K <=
200 and operands up to a few times the result's scale: 1e-9.  The adjoint adds
with atomics in any order: 1e-12 of the largest element."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _pair(lay, hL, hR, seed):
    from imsrg_gpu.synth import random_operator
    return random_operator(lay, hL, seed, 1), random_operator(lay, hR, seed + 1, 2)


@pytest.mark.parametrize("emax,nucleus", [(1, "4He"), (2, "4He"), (3, "16O"), (4, "4He"), (5, "4He")])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("ozaki", 1e-9)])
@pytest.mark.parametrize("hL,hR,with_e0", [(-1, 1, True), (-1, -1, False), (1, 1, True)])
def test_launch_sequences_agree(gpu_lib, oracle_mod, emax, nucleus, precision, tol, hL, hR, with_e0):
    import torch
    from imsrg_gpu.layout import Layout, ho_basis
    bas = ho_basis(emax, nucleus)
    lay = Layout(**bas)
    B = gpu_lib.Basis.from_dict(bas)
    Lh, Rh = _pair(lay, hL, hR, 41)
    ref = oracle_mod.Oracle(**bas).commutator(Lh, hL, Rh, hR)
    L, R, RES = gpu_lib.Operator(B, hL, Lh), gpu_lib.Operator(B, hR, Rh), gpu_lib.Operator(B, 1)
    results = []
    for call in range(3):  # the first one, the graph's capture, its replay
        gpu_lib.commutator(L, R, RES, precision=precision, with_e0=with_e0)
        results.append(RES.download())
    B.profile(True)
    gpu_lib.commutator(L, R, RES, precision=precision, with_e0=with_e0)
    B.synchronize()
    results.append(RES.download())
    packed = RES.download_packed()
    B.profile(False)
    got, want = results[0].copy(), ref.copy()
    if not with_e0:
        got[0] = want[0] = 0.0
    assert rel_err(got, want) <= tol
    for r in results[1:]:
        assert np.array_equal(r[1:], results[0][1:]) and (not with_e0 or r[0] == results[0][0])
    hosts = []
    for x in (L.download_packed(), R.download_packed(), np.full(packed.size, np.nan)):
        t = torch.empty(x.size, dtype=torch.float64, pin_memory=True)
        t.numpy()[:] = x
        hosts.append(t)
    gpu_lib.commutator_host_packed(B, hosts[0].numpy(), hL, hosts[1].numpy(), hR, hosts[2].numpy(),
                                   precision=precision, with_e0=with_e0)
    assert np.array_equal(hosts[2].numpy()[1:], packed[1:])


@pytest.mark.parametrize("emax", [2, 5])
@pytest.mark.parametrize("digits", [5, 8])
def test_block_exponents_do_not_outlive_a_commutator(gpu_lib, emax, digits):
    """Large operands, then small ones: the second result has the bits of a fresh
    basis (exponents left over from the first would cost it 20 bits)."""
    from imsrg_gpu.layout import Layout, ho_basis
    bas = ho_basis(emax, "4He")
    lay = Layout(**bas)
    Lh, Rh = _pair(lay, -1, 1, 51)

    def run(scales):
        B = gpu_lib.Basis.from_dict(bas)
        B.set_split_digits(digits)
        RES = gpu_lib.Operator(B, 1)
        for s in scales:
            L, R = gpu_lib.Operator(B, -1, s * Lh), gpu_lib.Operator(B, 1, Rh / s)
            for _ in range(2):
                gpu_lib.commutator(L, R, RES, precision="ozaki")
        return RES.download()

    assert np.array_equal(run([1024.0 ** 2, 1.0]), run([1.0]))


@pytest.mark.parametrize("emax", [2, 5])
def test_adjoint_on_one_stream_and_on_two(gpu_lib, emax):
    from imsrg_gpu.layout import Layout, ho_basis
    bas = ho_basis(emax, "16O")
    lay = Layout(**bas)
    B = gpu_lib.Basis.from_dict(bas)
    X = gpu_lib.Operator(B, -1, _pair(lay, -1, 1, 61)[0])
    C = gpu_lib.Operator(B, 1, np.random.default_rng(62).standard_normal(lay.nfull))
    Y = gpu_lib.Operator(B, 1)
    gpu_lib.commutator_adjoint(X, C, 1, Y)
    two = Y.download()
    B.profile(True)
    gpu_lib.commutator_adjoint(X, C, 1, Y)
    B.synchronize()
    B.profile(False)
    assert rel_err(Y.download(), two) <= 1e-12
