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


def test_next_kernel_is_let_in_after_the_tmem_allocation():
    """A dependent kernel's blocks may start once every block has called pdl_next().  Before this
    kernel has its TMEM they could take it, and then wait for this kernel, which waits for them."""
    seen = 0
    for name, text in SOURCES.items():
        for head, body in functions(text):
            if "tmem_alloc" in body and "pdl_next" in body:
                alloc = body.rindex("tmem_alloc")
                ready = re.search(r"__syncthreads\(\)|clu::sync_all\(\)", body[alloc:])
                assert ready and body.index("pdl_next") > alloc + ready.start(), (name, head)
                seen += 1
    assert seen == 4


def test_kernels_of_a_chain_wait_on_every_path():
    """A kernel that lets the next one in takes part in a chain of dependent launches, whose order holds
    because each waits for the one before: pdl_wait() follows pdl_next(), and a block that
    leaves before that has waited too."""
    for name, text in SOURCES.items():
        for head, body in functions(text):
            if "pdl_next();" not in body or "pdl_wait() {" in head:
                continue
            assert re.search(r"pdl_next\(\);\s*pdl_wait\(\);", body), (name, head)
            before = body[:body.index("pdl_next();")]
            assert all(re.search(r"pdl_wait\(\);\s*$", part) for part in before.split("return;")[:-1]), (name, head)
