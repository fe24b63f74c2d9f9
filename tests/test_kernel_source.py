"""Rules of the kernels' sources whose breach could hang or fault the device, and so has no test
that runs it: read from the text."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "mojoblas_b200" / "csrc"
SOURCES = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*"))}


def functions(text):
    """(head, body) of every function whose closing brace is in the first column."""
    for m in re.finditer(r"^(?:template|__global__|__device__|inline|int|void|static)[^;{}]*\{\n(.*?)^\}", text, re.M | re.S):
        yield text[m.start():m.start(1)], m.group(1)


def test_cluster_barrier_has_converged_warps():
    """barrier.cluster's aligned forms need a converged warp: the one place that issues them sees to it."""
    users = [name for name, text in SOURCES.items() if "barrier.cluster" in text]
    assert users == ["cluster.cuh"]
    bodies = [b for _, b in functions(SOURCES["cluster.cuh"]) if "barrier.cluster" in b]
    assert len(bodies) == 1
    assert "__syncwarp();" in bodies[0].split("barrier.cluster")[0]


def test_kernels_with_tmem_let_no_kernel_in():
    """A dependent kernel's blocks may start once every block has called pdl_next().  They could take the TMEM
    that this kernel is yet to allocate, and then wait for this kernel, which waits for them."""
    seen = 0
    for name, text in SOURCES.items():
        for head, body in functions(text):
            if "tmem_alloc" in body and "pdl_wait" in body:
                assert "pdl_next" not in body, (name, head)
                seen += 1
    assert seen == 4


def test_kernels_of_a_chain_wait_on_every_path():
    """A kernel that lets the next one in, or waits for the one before, takes part in a chain of dependent
    launches, whose order holds because each waits: pdl_wait() follows pdl_next(), and a block
    that leaves before the kernel's wait has waited too."""
    for name, text in SOURCES.items():
        for head, body in functions(text):
            if "pdl_next();" in body:
                assert re.search(r"pdl_next\(\);\s*pdl_wait\(\);", body), (name, head)
            if "pdl_wait();" in body:
                before = body[:body.rindex("pdl_wait();")]
                assert all(re.search(r"pdl_wait\(\);\s*$", part) for part in before.split("return;")[:-1]), (name, head)
