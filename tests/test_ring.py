"""The stage ring of the tcgen05 K3 kernel (fdga_ring.h, fdga_k3_oz.cu): the parities that its waits name, on the
CPU against the mbarrier's rule (a wait on parity p returns once the barrier's current phase has the other parity).
"""
import ctypes
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fddgasolver.jl_gb300", "csrc")


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    src, lib = d / "ring.cpp", d / "ring.so"
    src.write_text('#include "fdga_ring.h"\n'
                   'extern "C" int stage(int c, int ns) { return fdga::ring_stage(c, ns); }\n'
                   'extern "C" unsigned parity(int c, int ns) { return fdga::ring_parity(c, ns); }\n')
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)])
    return ctypes.CDLL(str(lib))


@pytest.mark.parametrize("ns", [2, 3])
def test_waits_end_with_their_use_and_not_before(ring, ns):
    """For every number of committed chunks (the release after an abort waits for the last) and every number of
    those done: chunk c is issued only once use c - ns of its stage is done, so at least committed - ns are."""
    for committed in range(1, 17):
        last = committed - 1
        for done in range(max(0, committed - ns), committed + 1):
            phases = sum(1 for c in range(done) if ring.stage(c, ns) == ring.stage(last, ns))
            returns = (phases & 1) != ring.parity(last, ns)
            assert returns == (done == committed)


def test_every_wait_of_the_kernel_names_its_use():
    src = open(os.path.join(CSRC, "fdga_k3_oz.cu"), encoding="utf-8").read()
    calls = re.findall(r"mbar_wait\((\w+\((?:[^()]|\([^()]*\))*\)), ((?:[^(),]|\([^()]*\))*),", src)
    assert len(calls) == 7
    assert all(p == "par" or p.startswith("ring_parity(") for _, p in calls), calls
    assert "const uint32_t par = ring_parity(c, NS);" in src
