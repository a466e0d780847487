"""Order of barrier, fence and release in the elimination kernels, checked on
the source: a wrong order shows on no device reliably, and must not be run."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "parallel-randomized-cholesky_b200", "csrc")


def code(name):
    """The file without its comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def test_counters_drop_after_barrier_then_fence():
    """release_row's relaxed decrement publishes what every thread of the warp
    or CTA wrote.  That holds only if the releasing thread passes a fence of its
    own after the barrier that joins the other threads' writes."""
    text = code("factor.cu")
    calls = [m.start() for m in re.finditer(r"\brelease_row\(a,", text)]
    assert len(calls) == 3  # one warp, register lists, slabs in global memory
    for at in calls:
        before = text[:at]
        barrier = max(before.rfind("__syncthreads"), before.rfind("__syncwarp"))
        fence = before.rfind("__threadfence()")
        assert 0 <= barrier < fence, text[barrier:at]


def test_block_tickets_are_taken_between_fences():
    """The last block of a reduction reads what every thread of the other blocks
    wrote: barrier, fence, ticket, fence, barrier, the fences in the thread that
    takes the ticket."""
    text = code("solve.cu")
    at = text.index("bool last_block(")
    body = text[at:text.index("\n}", at)]
    steps = re.findall(r"__syncthreads|__threadfence|atomicAdd", body)
    assert steps == ["__syncthreads", "__threadfence", "atomicAdd", "__threadfence", "__syncthreads"]
    lead = body[body.index("if (threadIdx.x == 0) {"):body.rindex("__syncthreads")]
    assert lead.count("__threadfence") == 2 and "atomicAdd" in lead
