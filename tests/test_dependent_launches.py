"""Kernels that start before their predecessor ends (device.cuh: launch_after)
may not read what it writes through the non-coherent path, whose data has to be
unchanged from the kernel's start on.  Read from the sources: such a kernel takes
no `const T *__restrict__` but tables of the plan and operands that were whole
before its predecessor began, the functions it shares with others take none at
all, and __ldg is applied to tables only."""
import glob
import os
import re

import pytest

from conftest import PKG

CSRC = os.path.join(PKG, "csrc")
TABLE_TYPES = {"AdjProb", "GemmTile", "GemmProb", "OzMatrix", "uint16_t", "OzTile", "CUtensorMap", "Asm2Head"}
# sched_off: the schedule's table; act: read by ordinary launches of a batch alone
OPERANDS = {"X", "Cb", "L", "R", "sched_off", "act"}
TABLES = ("slots", "ph", "T.ph_slots", "reinterpret_cast<const uint4 *>(tiles")


def _sources():
    out = {}
    for p in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        out[os.path.basename(p)] = re.sub(r"//[^\n]*", "", open(p).read())
    return out


def _kernels():
    """name -> (file, parameters, body) of every kernel that calls pdl_wait."""
    out = {}
    for name, src in _sources().items():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(\w+)\(", src):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(src[i], 0)
                i += 1
            params = src[m.end():i - 1]
            j = src.index("{", i)
            depth, k = 1, j + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[k], 0)
                k += 1
            if "pdl_wait()" in src[j:k]:
                out[m.group(1)] = (name, params, src[j:k])
    return out


def _restricted(params):
    return [(t, n) for t, n in re.findall(r"const\s+([\w:]+)\s*\*\s*__restrict__\s*(\w+)", params)]


def test_every_dependent_kernel_waits():
    """Whatever launch_after may start calls pdl_wait."""
    waiting = _kernels()
    launched = set()
    for src in _sources().values():
        for args in re.findall(r"launch_after\(([^;]*);", src):
            launched |= set(re.findall(r"\bk_\w+", args))
    launched |= {"k_ph_list", "k_ph_patches", "k_oz_slice"}  # chosen through a pointer
    assert len(launched) >= 9 and launched <= set(waiting)


@pytest.mark.parametrize("kernel", sorted(_kernels()))
def test_no_noncoherent_reads_of_a_predecessors_output(kernel):
    file, params, body = _kernels()[kernel]
    bad = [(t, n) for t, n in _restricted(params) if t not in TABLE_TYPES and n not in OPERANDS]
    assert not bad, (file, kernel, bad)
    assert "double *__restrict__" not in re.sub(r"const\s+double \*__restrict__", "", params)
    for arg in re.findall(r"__ldg\((.*?)\)", body):
        assert arg.startswith(TABLES), (file, kernel, arg)


@pytest.mark.parametrize("file,functions", [("front.cuh", None), ("gemm_fp64.cuh", None),
                                            ("device.cuh", ("series_chunk", "sum_partials")),
                                            ("adjoint.cu", ("adj_ph",))])
def test_shared_functions_take_no_restricted_data(file, functions):
    src = _sources()[file]
    for m in re.finditer(r"__device__ __forceinline__ \w+ (\w+)\(([^{]*)\)\s*\{", src):
        if functions is None or m.group(1) in functions:
            assert not _restricted(m.group(2)), m.group(1)
    if functions is None:
        assert "__ldg" not in src
