"""bench.py's report of a batch group: the name and the tuned time are those of
the kernel that runs, the line and warp kernels included, or there is no time."""
import bench


def group(p, variant, **ms):
    g = {"p": p, "variant": variant, "ms_pipe": 0.0, "ms_block": 0.0, "ms_block8": 0.0,
         "ms_split": 0.0, "ms_line": 0.0}
    return {**g, **ms}


def test_line_group():
    name, ms = bench.group_kernels(group(9, 6, ms_pipe=2.0, ms_line=1.5, ms_split=1.8))
    assert name == "line" and ms[name] == 1.5


def test_warp_group():
    name, ms = bench.group_kernels(group(7, 2, ms_pipe=1.0))
    assert name == "warp" and ms[name] == 1.0 and "pipe" not in ms


def test_other_groups():
    for variant, name, key in [(1, "block", "ms_block"), (2, "pipe", "ms_pipe"),
                               (3, "block8", "ms_block8"), (4, "split", "ms_split")]:
        got, ms = bench.group_kernels(group(5, variant, **{key: 0.7}))
        assert got == name and ms[got] == 0.7


def test_a_kernel_without_a_name_has_no_time():
    name, ms = bench.group_kernels(group(5, 9, ms_pipe=1.0))
    assert ms.get(name, 0.0) == 0.0
