"""Block exponents that a commutator left behind: its part before the products
runs alone on operands 2^20 times larger, as in a call that fails there, and then
a cached graph is replayed on the ordinary ones.  Its result has the bits of the
replay before (with the exponents left over it would lose 20 bits of 35)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAUNCHES = "_ZN5imsrg19commutator_launchesEP11imsrg_basisPKdiS3_iPdiiiPKNS_6HostIOEi"
FRONT = 1


@pytest.mark.parametrize("emax", [2, 5])
def test_cached_commutator_after_a_lone_front(gpu_lib, emax):
    import torch
    from imsrg_gpu.layout import Layout, ho_basis
    from imsrg_gpu.synth import random_operator
    bas = ho_basis(emax, "4He")
    lay = Layout(**bas)
    B = gpu_lib.Basis.from_dict(bas)
    B.set_split_digits(5)
    Lh, Rh = random_operator(lay, -1, 71, 1), random_operator(lay, 1, 72, 2)
    L, R, RES = gpu_lib.Operator(B, -1, Lh), gpu_lib.Operator(B, 1, Rh), gpu_lib.Operator(B, 1)
    bigL, bigR, out = (gpu_lib.Operator(B, -1, Lh * 2.0 ** 20), gpu_lib.Operator(B, 1, Rh * 2.0 ** 20),
                       gpu_lib.Operator(B, 1))
    for _ in range(3):  # tuned, captured, replayed
        gpu_lib.commutator(L, R, RES, precision="ozaki")
    want = RES.download()
    launches = gpu_lib.lib()[LAUNCHES]
    p, i = ctypes.c_void_p, ctypes.c_int
    launches.argtypes = [p, p, i, p, i, p, i, i, i, p, i]
    assert launches(B.handle, bigL.device_ptr(), -1, bigR.device_ptr(), 1, out.device_ptr(), 1, 1, 1, None, FRONT) == 0
    torch.cuda.synchronize()
    gpu_lib.commutator(L, R, RES, precision="ozaki")
    assert np.array_equal(RES.download(), want)
