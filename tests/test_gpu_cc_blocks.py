"""The |Tz| = 1 cross-coupled blocks as two independent ones (proton-neutron
and neutron-proton pairs), with different hole shells for the two isospins so
that the halves have different column counts, one of them none at all; emax = 5
forms its recoupling inputs patch by patch, the others one by one.

Tolerances: the FP64 bar max |gpu - oracle| <= 1e-10 max |oracle|; six digits
truncate each product at 2^-42 K max|A| max|B| (K <= 200 here, operands up to
a few times the result's scale): 1e-9.  The adjoint's two inner products are
sums of the same products in different orders: 1e-12 of their magnitude."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("emax,protons,neutrons", [(2, 1, 0), (2, 0, 1), (3, 1, 2), (3, 2, 1), (4, 2, 0), (5, 1, 2)])
def test_unequal_hole_shells(gpu_lib, oracle_mod, emax, protons, neutrons):
    from imsrg_gpu.layout import Layout, ho_basis
    from imsrg_gpu.synth import random_operator
    bas = ho_basis(emax)
    shell = 2 * bas["nn"] + bas["ll"]
    bas["con"] = (shell < np.where(bas["itzp"] < 0, protons, neutrons)).astype(np.int32)
    lay = Layout(**bas)
    B, orc = gpu_lib.Basis.from_dict(bas), oracle_mod.Oracle(**bas)
    for hL, hR in ((-1, 1), (1, 1), (-1, -1)):
        Lh, Rh = random_operator(lay, hL, 5, 1), random_operator(lay, hR, 6, 2)
        ref = orc.commutator(Lh, hL, Rh, hR)
        L, R, RES = gpu_lib.Operator(B, hL, Lh), gpu_lib.Operator(B, hR, Rh), gpu_lib.Operator(B, 1)
        for precision, tol in (("fp64", 1e-10), ("ozaki", 1e-9)):
            gpu_lib.commutator(L, R, RES, precision=precision)
            assert rel_err(RES.download(), ref) <= tol, (precision, hL, hR)
        Cb = np.random.default_rng(9).standard_normal(lay.nfull)
        Yb = gpu_lib.Operator(B, 1)
        gpu_lib.commutator_adjoint(L, gpu_lib.Operator(B, 1, Cb), hR, Yb)
        lhs = float(np.dot(Cb, ref))
        scale = float(np.dot(np.abs(Cb), np.abs(ref))) + 1.0
        assert abs(lhs - float(np.dot(Yb.download(), Rh))) <= 1e-12 * scale
