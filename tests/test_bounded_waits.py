"""The product kernel's waits give up after a time limit, and then every warp has
to leave together: a lane that gave up while its neighbour saw the phase complete
would wait at the CTA's last barrier, the neighbour at the warp's next
instruction for all lanes, and the kernel would hang after its limit.  Read from
the source (a time limit is not provoked on a GPU): outside the producer, which is
one lane, every wait is the warp's, and no loop or branch around a warp-wide
instruction depends on a lane's own look at the abort flag."""
import os
import re

from conftest import PKG


def _roles():
    src = re.sub(r"//[^\n]*", "", open(os.path.join(PKG, "csrc", "ozaki.cu")).read())
    body = src[src.index("k_oz_mma(const OzTile"):]
    body = body[:body.index("tcgen05.dealloc")]
    producer, issuer = body.index("if (warp == 0) {"), body.index("} else if (warp == 1) {")
    epilogue = body.rindex("} else {", 0, body.index("const int quad = warp & 3"))
    end = body.index("__syncthreads();", epilogue)
    return src, body[producer:issuer], body[issuer:epilogue], body[epilogue:end]


def test_waits_of_whole_warps_have_one_outcome():
    src, producer, issuer, epilogue = _roles()
    assert "if (lane == 0)" in producer and "mbar_wait(" in producer
    for role, waits in ((issuer, 2), (epilogue, 1)):
        assert "mbar_wait(" not in role
        assert len(re.findall(r"ok = mbar_wait_warp\(", role)) == waits
        # the flag itself is one lane's affair
        rest = re.sub(r"mbar_wait_warp\([^;]*;", "", role)
        rest = re.sub(r"if \(lane == 0\) \{[^{}]*\}", "", rest)
        rest = re.sub(r"if \([^()]*\bleader\) [^;]*;", "", rest)
        assert "abort_flag" not in rest
    wait = re.search(r"bool mbar_wait_warp\([^)]*\) \{(.*?)\n\}", src, re.S).group(1)
    assert "__all_sync(0xffffffffu, mbar_wait(" in wait
