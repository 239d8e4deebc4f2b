"""No kernel leaves a thread block while copies into its shared memory are in
flight, whichever wait gave up.

The waits of a pipeline (mbar_wait, wait_count) return at once when another
thread has recorded an error, long before a copy has landed, so the waits
before a block's end are mbar_drain, which only a time limit ends.  Read from
the sources: making the copies outlive a block on a GPU could hang it.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "sycl-bench_gb300" / "csrc"


def source(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def body(text, head):
    """The braces that follow `head`."""
    i = text.index("{", text.index(head))
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError(head)


def test_the_drain_ends_only_by_completion_or_time():
    drain = body(source("gbpoly_internal.cuh"), "bool mbar_drain(")
    assert "mbar_try_wait" in drain and "kWaitTimeoutNs" in drain
    assert "volatile" not in drain  # (the other waits read the error word through one)


@pytest.mark.parametrize("name", ["split_gemm.cu", "sgemm_simt.cu"])
def test_producers_drain_their_stages(name):
    text = source(name)
    assert "kDevErrDrainWait" not in text  # no drain through a wait that an error ends
    assert re.search(r"mbar_drain\(&full\[", text)


def test_every_load_of_c_is_counted_and_drained():
    kernel = body(source("split_gemm.cu"), "void __launch_bounds__(F::THREADS, 1) split_gemm_kernel(")
    epilogue = kernel[kernel.index("float acc[F::HALF]"):]
    loads = [m.start() for m in re.finditer(r"tma_load_2d\([^;]*sched\.cmap", epilogue)]
    assert len(loads) == 4  # the C-tile form, box by box, the whole tile, its transpose
    for at in loads:
        # counted before the next wait or load
        rest = epilogue[at + 1:]
        nxt = min(rest.index(w) for w in ("mbar_wait(", "c_landed()", "tma_load_2d(") if w in rest)
        assert "++c_loads" in rest[:nxt] or "++c_loads" in rest[:rest.index("};")], rest[:200]
    # the one way out: after the loop over the units, if any wait failed
    end = epilogue[epilogue.rindex("if(!ok && c_loads > 0)"):]
    assert re.match(r"if\(!ok && c_loads > 0\) mbar_drain\(&cbar\[warp - 4\], \(c_loads - 1\) & 1, err\);", end)
