"""The FP64 product tiles at ragged block sizes (odd emax, both hole spaces:
row and column groups of every remainder, contractions of one to a few
hundred, tiles that split K and tiles that do not), forward against the oracle
and the adjoint as the forward's transpose.

Tolerances: max |gpu - oracle| <= 1e-10 max |oracle|, the FP64 bar; the
adjoint's inner products to 1e-12 of their terms' magnitude (sums of the same
products in different orders)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("emax,nucleus", [(1, "4He"), (2, "16O"), (3, "4He"), (3, "16O"), (4, "4He"), (5, "16O")])
def test_fp64_products(gpu_lib, oracle_mod, emax, nucleus):
    from imsrg_gpu.layout import Layout, ho_basis
    from imsrg_gpu.synth import random_operator
    bas = ho_basis(emax, nucleus)
    lay = Layout(**bas)
    B = gpu_lib.Basis.from_dict(bas)
    Lh, Rh = random_operator(lay, -1, 15, 1), random_operator(lay, 1, 16, 2)
    ref = oracle_mod.Oracle(**bas).commutator(Lh, -1, Rh, 1)
    L, R, RES = gpu_lib.Operator(B, -1, Lh), gpu_lib.Operator(B, 1, Rh), gpu_lib.Operator(B, 1)
    gpu_lib.commutator(L, R, RES)
    assert rel_err(RES.download(), ref) <= 1e-10
    Cb = np.random.default_rng(17).standard_normal(lay.nfull)
    Yb = gpu_lib.Operator(B, 1)
    gpu_lib.commutator_adjoint(L, gpu_lib.Operator(B, 1, Cb), 1, Yb)
    scale = float(np.dot(np.abs(Cb), np.abs(ref))) + 1.0
    assert abs(float(np.dot(Cb, ref)) - float(np.dot(Yb.download(), Rh))) <= 1e-12 * scale


@pytest.mark.parametrize("emax,nucleus", [(1, "4He"), (3, "16O"), (5, "4He")])
@pytest.mark.parametrize("digits", [4, 5, 6, 7, 8])
def test_split_products(gpu_lib, oracle_mod, emax, nucleus, digits):
    """The split engine's tiles and digit images at the same ragged sizes.  The
    dropped levels and the digit rounding are below 2^-(7 S) (S + 2) K max|A|
    max|B| per product; with |elements| <= 5, K <= 200 and results of some
    hundreds that is 2^-(7 S) 200 of the result's scale, plus the FP64 bar."""
    from imsrg_gpu.layout import Layout, ho_basis
    from imsrg_gpu.synth import random_operator
    bas = ho_basis(emax, nucleus)
    lay = Layout(**bas)
    B = gpu_lib.Basis.from_dict(bas)
    B.set_split_digits(digits)
    Lh, Rh = random_operator(lay, -1, 25, 1), random_operator(lay, 1, 26, 2)
    ref = oracle_mod.Oracle(**bas).commutator(Lh, -1, Rh, 1)
    L, R, RES = gpu_lib.Operator(B, -1, Lh), gpu_lib.Operator(B, 1, Rh), gpu_lib.Operator(B, 1)
    for _ in range(2):  # the autotuning call, then the graph
        gpu_lib.commutator(L, R, RES, precision="ozaki")
        assert rel_err(RES.download(), ref) <= 200.0 * 2.0 ** (-7 * digits) + 1e-10
