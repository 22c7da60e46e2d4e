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
