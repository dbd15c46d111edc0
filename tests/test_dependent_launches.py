"""What the kernels that are launched as programmatic dependents rely on, as
far as their sources show it (no GPU needed).  Such a kernel may start before
the launch before it has ended, and only its own griddepcontrol.wait makes
that launch's output visible."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dim2d_finite_volume_b200", "csrc")
# template parameters of the kernels: fixed when a kernel is compiled
TEMPLATE = {"MODE", "UN", "EDGES", "MIX", "KEEP", "WALLS"}


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as fh:
            yield os.path.basename(path), re.sub(r"//[^\n]*", "", fh.read())


def test_no_wait_depends_on_the_launch():
    """A wait that a launch's arguments can switch off leaves a kernel that
    reads its input unordered."""
    found = 0
    for name, text in _sources():
        for m in re.finditer(r"(if \((?P<cond>[^;{]*)\) )?wait_for_launch_before\(\);", text):
            found += 1
            names = set(re.findall(r"[A-Za-z_][\w.]*", m["cond"] or ""))
            assert names <= TEMPLATE, (name, m[0])
    assert found >= 4


def test_no_dependent_reads_through_the_read_only_path():
    """ld.global.nc is specified for data that nothing writes from a kernel's
    start to its end; a dependent starts before its input is complete.  The
    sources that may use it hold plain launches only."""
    plain = {"dim2d_open.cuh", "dim2d_interior.cu"}
    for name, text in _sources():
        if name in plain:
            assert "wait_for_launch_before();" not in text, name
        else:
            assert "__ldg(" not in text and "ld.global.nc" not in text, name
