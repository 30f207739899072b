"""How the kernels use block barriers, read from their source (a missed or early
barrier shows on a GPU only by chance): warps arrive with their lanes apart, so
every barrier is the unaligned block_sync."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fringe-sgc_gb300", "csrc")


def kernel_sources():
    """(file name, text without comments) of every device source."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            text = f.read()
        text = re.sub(r"/\*.*?\*/", lambda m: "\n" * m.group().count("\n"), text, flags=re.S)
        yield os.path.basename(path), re.sub(r"//[^\n]*", "", text)


def test_barriers_take_warps_with_their_lanes_apart():
    aligned = r"__syncthreads|__barrier_sync|\bbar\.(sync|red|arrive)|barrier\.[a-z.]*aligned"
    for name, text in kernel_sources():
        for i, line in enumerate(text.split("\n"), 1):
            assert not re.search(aligned, line), f"{name}:{i}: {line.strip()}"


def test_shared_queue_items_are_replaced_behind_a_barrier():
    """A block's thread 0 fetches the next queue item into shared memory that all
    warps read, also in the condition by which they leave the last item's loop:
    a barrier stands directly before it."""
    found = 0
    for name, text in kernel_sources():
        lines = [line.strip() for line in text.split("\n") if line.strip()]
        for i, line in enumerate(lines):
            if not re.match(r"(S\.|s_)\w+ = atomicAdd\(queue\b", line):
                continue
            at = i - 1
            while not re.match(r"if \((tid|threadIdx\.x) == 0\)", lines[at]):
                at -= 1
            assert at >= i - 2 and lines[at - 1] == "block_sync();", f"{name}: {lines[at - 1:i + 1]}"
            found += 1
    assert found >= 2
