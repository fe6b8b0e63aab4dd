"""Memory order of the grid-wide barriers, from their source: a missing fence shows in no run of the kernels that
use them (most of their loads go past L1), so the order of the operations is checked where it is written."""
import os
import re

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parameter_server_b200", "csrc", "cuda")


def _body(path, name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CUDA, path)).read())
    at = re.search(r"\b%s\([^)]*\)\s*\{" % name, src).end()
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(src[end], 0)
        end += 1
    return src[at:end]


def test_last_cta_of_the_grid_barrier_acquires_before_it_releases():
    b = _body("psb_common.cuh", "grid_barrier")
    arrive = b.index("atomicAdd(bar")
    assert "__threadfence()" in b[:arrive], "every CTA releases its stores before it arrives"
    last = b[b.index("if (arrived"):b.index("else")]
    assert last.index("__threadfence()") < last.index("st_relaxed_gpu(bar,") < last.index("st_release_gpu(bar + 1,")
    assert "while (ld_acquire_gpu(bar + 1)" in b[b.index("else"):]


def test_every_cta_of_the_pass_barrier_acquires():
    b = _body("darlin.cu", "pass_barrier")
    assert "red.release.gpu" in b and "ld_acquire_gpu(word) < target" in b
