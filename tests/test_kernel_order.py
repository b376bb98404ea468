"""Orders that the kernels' results rest on but that a run cannot show to be
missing (a block that starts late, a compiler that moves a load), checked in
the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sca2012_b200", "csrc")


def _code(name):
    """A source file without its comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _block(code, start):
    """The braced block that follows the first match of `start`."""
    i = code.index("{", re.search(start, code).end())
    depth = 0
    for j in range(i, len(code)):
        depth += {"{": 1, "}": -1}.get(code[j], 0)
        if depth == 0:
            return code[i:j + 1]
    raise AssertionError(f"no end of block after {start}")


def test_remote_shared_memory_is_written_only_to_started_blocks():
    """A block may touch another block's shared memory only once that block is
    known to have started: a cluster barrier stands before the first remote store,
    outside any branch that part of the block would skip."""
    body = _block(_code("sph_scan.cuh"), r"uint32_t\s+cluster_scan_body\(")
    remote = body.index("st.shared::cluster")
    before = body[:remote]
    arrive, wait = before.find("barrier.cluster.arrive"), before.find("barrier.cluster.wait")
    assert 0 <= arrive < wait
    for at in (arrive, wait):
        assert body[:at].count("{") - body[:at].count("}") == 1   # the function's own level
    # and none is left unread when a block ends: the barrier behind the stores
    after = body[remote:]
    assert 0 <= after.find("barrier.cluster.arrive.release") < after.find("barrier.cluster.wait.acquire")


def test_remote_shared_memory_has_one_user():
    """The check above covers the only function that maps remote shared memory."""
    uses = {f: len(re.findall(r"\bmapa\b|st\.shared::cluster|ld\.shared::cluster", _code(f)))
            for f in os.listdir(CSRC) if f.endswith((".cuh", ".cu"))}
    assert {f for f, n in uses.items() if n} == {"sph_scan.cuh"}
    body = _block(_code("sph_scan.cuh"), r"uint32_t\s+cluster_scan_body\(")
    assert len(re.findall(r"\bmapa\b|shared::cluster", body)) == len(
        re.findall(r"\bmapa\b|shared::cluster", _code("sph_scan.cuh")))


def test_density_buffer_drain_is_fenced_from_the_appends():
    """The density walk appends to its buffer by inline assembly that names no
    memory; the drain's plain loads and stores of the same buffer stay between
    two compiler barriers."""
    body = _block(_code("sph_kernels.cuh"), r"void\s+density_walk\(")
    drain = re.sub(r"\s+", "", _block(body, r"auto\s+drain\s*=\s*\[&\]\(bool\s+last\)")[1:-1])
    fence = 'asmvolatile("":::"memory");'
    assert drain.startswith(fence) and drain.endswith(fence)
    # every other plain use of the buffer is inside the drain
    assert len(re.findall(r"\bcol\[", body)) == drain.count("col[")
