"""The autotuner's command times settings that a kernel reads and no others: a setting
that steers nothing would be picked by timing noise."""
import os
import re
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "fringe-sgc_gb300"))
import autotune  # noqa: E402
import fsgc  # noqa: E402


def test_unread_fields_are_those_that_only_the_range_check_names():
    read = set()
    csrc = os.path.join(ROOT, "fringe-sgc_gb300", "csrc")
    for name in os.listdir(csrc):
        if name.endswith(".cu"):
            with open(os.path.join(csrc, name)) as f:
                text = f.read()
            read |= set(re.findall(r"tune\.(\w+)", text))  # the range check takes its settings as `t`
    assert set(autotune.CANDIDATES) - read == autotune.UNREAD


def test_the_command_leaves_them_at_their_defaults(monkeypatch, tmp_path):
    import bench
    timed = []

    class Ctx:
        def __init__(self, device):
            pass

        def __enter__(self):
            return self

        def __exit__(self, *a):
            pass

        upload = prepare = release = lambda self, g: 1

    def tune(ctx, gid, mos, repeats, fields=None, log=None):
        timed.extend(fields if fields is not None else list(autotune.CANDIDATES))
        return fsgc.Tuning.default().as_dict(), {}

    monkeypatch.setattr(fsgc, "Context", Ctx)
    monkeypatch.setattr(autotune, "tune", tune)
    monkeypatch.setattr(bench, "matching_orders", lambda: [])
    monkeypatch.setattr(sys, "argv", ["autotune.py", "--scale", "6", "--out", str(tmp_path / "t.json")])
    autotune.main()
    assert timed and not autotune.UNREAD & set(timed)
    assert set(timed) | autotune.UNREAD == set(autotune.CANDIDATES)
