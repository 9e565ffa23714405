"""What kernels may and may not do around a programmatic dependent launch, read from their source (with
several GPUs a breach shows as a hang, and as stale data only now and then)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "csrc" / "kernels"


def _source(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def _functions(text):
    """(head, body) of every function of the file: the text between two ends of a top-level block."""
    out, depth, start, head = [], 0, 0, ""
    for i, c in enumerate(text):
        if c == "{":
            if depth == 0:
                head, at = text[start:i], i
                if re.search(r"\bnamespace\s+\w*\s*$", head):
                    start = i + 1
                    continue
            depth += 1
        elif c == "}" and depth:
            depth -= 1
            if depth == 0:
                out.append((head, text[at:i]))
                start = i + 1
    return out


def test_kernels_that_wait_for_peers_let_nobody_in_early():
    waits, checked = ("block_barrier", "plan_body", "scatter_body", "combine_body"), 0
    for head, body in _functions(_source("moe.cu")):
        if "__global__" in head and any(re.search(r"\b%s\b" % w, body) for w in waits):
            checked += 1
            free = re.sub(r"if \(a\.coll\.nranks == 1\) \{[^}]*\}", "", body)
            assert "pdl_launch_dependents" not in free, head
    assert checked >= 6      # plan, scatter, combine, and their emulated forms
    for name in ("collectives.cu", "coll_bodies.inl", "coll_device.cuh", "gemm_sm100.cu", "gemm_ag_cta_movers.cu"):
        assert "pdl_launch_dependents" not in _source(name), name


def test_overlapped_kernels_promise_nothing_about_their_inputs():
    """Neither read-only loads nor restricted pointers in what may start under its predecessor."""
    overlapped = 0
    for path in sorted(CSRC.glob("*.cu")):
        text = _source(path.name)
        if "pdl.cuh" not in text:
            continue
        assert not re.search(r"\b(__ldg|ld\.global\.nc)\b", text), path.name
        for head, body in _functions(text):
            if "__global__" in head and "pdl_wait" in body:
                overlapped += 1
                assert "__restrict__" not in head, (path.name, head)
    assert overlapped >= 8
