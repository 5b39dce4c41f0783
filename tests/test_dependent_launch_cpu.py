"""Kernels launched as programmatic dependents (prior_grids_done()) start while
the kernel before them still writes: what that one writes must not be read
through loads that are only defined for data no kernel writes (__ldg, const
__restrict__ pointers), nor through __ldcg, which the compiler may move ahead
of the wait.  Read from the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tsuner_b200", "csrc")
# what only the host writes, or this grid itself behind a fence
READ_ONLY = ("A.mask + g", "A.tCC + (A.timeCC - 2)",
             "reinterpret_cast<const unsigned long long *>(&E.members[m].g) + threadIdx.x")
OWN_GRID = ("A.partials + i", "A.partials + nb + i", "A.partials + 2 * nb + i")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def arguments(text, call):
    """The argument texts of every call(...)."""
    for m in re.finditer(re.escape(call) + r"\(", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        yield " ".join(text[m.end():k - 1].split())


def dependents(text):
    """(signature, body) of every kernel that waits for the grid before it."""
    for m in re.finditer(r"__global__", text):
        at = text.index("{", m.end())
        depth, k = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        if "prior_grids_done()" in text[at:k]:
            yield text[m.end():at], text[at:k]


def test_stage_kernels_read_state_through_coherent_loads():
    text = source("stage32.cu")
    stage = text[:text.index("to32_kernel")]  # what the dependent kernels run
    assert set(arguments(stage, "__ldg")) <= set(READ_ONLY)
    assert set(arguments(stage, "__ldcg")) <= set(OWN_GRID)
    text = source("stage64.cu")
    stage = text[:text.index("dt_partials_kernel")]
    assert not list(arguments(stage, "__ldg"))
    assert set(arguments(stage, "__ldcg")) <= set(OWN_GRID)


def test_dependent_kernels_take_no_read_only_pointers():
    found = 0
    for name in ("stage32.cu", "stage64.cu", "corrector.cu"):
        for signature, body in dependents(source(name)):
            found += 1
            assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", signature), signature
            if name == "corrector.cu":
                assert "__ldg(" not in body and "__ldcg(" not in body, signature
    assert found == 5  # FP64 and FP32 stages, ensemble stage, weight gradient and its reduction
