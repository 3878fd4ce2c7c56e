"""Words that blocks pass one another are read and written whole.  The PTX
memory model treats a vector access as scalar accesses in no stated order, so
an ordered or strong access (relaxed, acquire, release, volatile) whose
elements belong together must be a scalar one."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gridinfcuda_gb300", "csrc")
STRONG_VECTOR = re.compile(r"\b(?:ld|st)\.(?:[\w:]+\.)*(?:relaxed|acquire|release|volatile)\.(?:[\w:]+\.)*v[248]\.")


def test_pattern_finds_vector_forms():
    assert STRONG_VECTOR.search("ld.relaxed.cluster.shared::cluster.v2.u32 {%0, %1}, [%2];")
    assert STRONG_VECTOR.search("st.volatile.shared.v4.f32")
    assert not STRONG_VECTOR.search("ld.relaxed.gpu.global.u32 %0, [%1];")
    assert not STRONG_VECTOR.search("ld.global.nc.v4.f32")


def test_no_strong_vector_accesses():
    sources = glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))
    assert sources
    found = [(os.path.basename(f), n + 1) for f in sorted(sources)
             for n, line in enumerate(open(f).read().splitlines()) if STRONG_VECTOR.search(line)]
    assert not found, found
