"""Sorts, scans and selections whose results the next pass indexes with: the
status of each is looked at before that pass is launched (a failed one leaves
uninitialised indices).  Read from the source, because such a failure cannot be
brought about safely on a GPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fringe-sgc_gb300", "csrc")


def test_status_of_every_device_wide_call_is_used():
    calls = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"cub::Device\w+::\w+\(", text):
            before = text[:m.start()].rstrip()
            assert re.search(r"(=|\(|\|\||&&|return)$", before), (os.path.basename(path), before[-60:])
            calls += 1
    assert calls >= 8
