"""What every kernel launched as a programmatic dependent has to keep to, checked on the sources (no GPU): such a kernel starts while
its predecessor on the stream is still running, so before its wait it may neither touch memory nor hold what the predecessor needs."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "all_quant_b200", "csrc")


def kernels(name):
    """{kernel: body} of a source file, comments taken out."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    out = {}
    for m in re.finditer(r"__global__[^;{]*?\b(uq_\w+_kernel)\s*\(", text):
        at = text.index("{", m.end())
        depth, end = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            if depth == 0:
                break
            end += 1
        out[m.group(1)] = text[at:end + 1]
    return out


def test_tensor_memory_is_allocated_after_the_wait():
    """A block that held all 512 columns while it waits for the kernel before it would starve a block of that kernel on the same SM
    that lets its successor go first and allocates tensor memory afterwards: each would wait for the other."""
    body = kernels("uq_verify_tc.cu")["uq_verify_tc_kernel"]
    wait = [m.end() for m in re.finditer(r"uq_pdl_wait\w*\(", body)]
    alloc = body.index("tcgen05.alloc")
    assert len(wait) == 2 and body.count("tcgen05.alloc") == 1   # (the first one is that of the early exit on a misplaced buffer)
    assert "return;" in body[wait[0]:wait[1]] and alloc > wait[1]


def test_indexes_of_read_only_loads_come_out_of_the_wait():
    """What is read through a const __restrict__ pointer or __ldg counts as unchanged during the whole kernel, so the compiler may
    move such a load above the wait - where the kernel before it may still be writing.  In the kernels that read their inputs this
    way every address is made of a thread index that the wait itself returns."""
    bodies = kernels("uq_append.cu")
    assert len(bodies) == 5
    for name, body in bodies.items():
        assert body.count("uq_pdl_wait_index()") == 1 and "threadIdx" not in body, name
        wait = body.index("uq_pdl_wait_index()")
        assert not re.search(r"\b(key|value|slots|src|x)\s*\[|__ldg|\.load\(", body[:wait]), name


def test_appends_release_their_successors_after_their_own_wait():
    """Before it, a waiting kernel would let the next one in, and that one the next: a pile of waiting grids in the working one's way.
    Only a grid of several waves, whose last blocks start late, may release first."""
    for name, body in kernels("uq_append.cu").items():
        wait = body.index("uq_pdl_wait_index()")
        first = "if (pdl && bulk_blocks() >= kReleaseFrom) uq_pdl_release();" in body[:wait]
        assert first == ("bulk" in name) and body[:wait].count("uq_pdl_release()") == first and body[wait:].count("uq_pdl_release()") == 1, name


def test_no_multiprocessor_count_is_written_down():
    """The grid and the rules that compare with it ask the device for its count."""
    for name in ("uq_verify_tc.cu", "uq_combine.cu", "uq_append.cu"):
        assert not re.search(r"\b148\b", re.sub(r"//[^\n]*|asm volatile\([^;]*;", "", open(os.path.join(CSRC, name)).read())), name
