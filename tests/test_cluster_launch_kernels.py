"""Source check of the time step's dependent launches of a whole cluster (no GPU).

`launch_dep_cluster` (delta_b200/csrc/pdl.cuh) starts a kernel while the one before it may
still run, as `launch_dep` does, so the kernel has to wait first (`dep_sync();`). Its CTAs may
wait on one another, which only a cluster's may: the hardware starts it as a whole. So no
kernel of another launch uses a cluster's barrier, and pdl.cuh has no launcher that neither
this test nor that of `launch_dep` covers.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "delta_b200" / "csrc"
SOURCES = {p.name: p.read_text() for p in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))}


def _code(text):
    return re.sub(r"//[^\n]*", "", text)


def _launched(launcher):
    """Kernels given to `launcher`, directly or through a variable set to one of several."""
    out = set()
    for name, text in SOURCES.items():
        if name == "pdl.cuh":
            continue
        for m in re.finditer(r"\b" + launcher + r"\(\s*(?:\w+\s*,\s*)?([A-Za-z_]\w*)", _code(text)):
            kernel = m.group(1)
            if kernel.startswith("k_"):
                out.add(kernel)
                continue
            d = re.search(r"\bauto\s+" + kernel + r"\s*=([^;]*);", text)
            assert d, f"{name}: {launcher} of {kernel}, whose kernels are not found"
            out |= set(re.findall(r"\bk_\w+", d.group(1)))
    return out


def _kernels():
    """Name and body of every __global__ function."""
    for text in SOURCES.values():
        text = _code(text)
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            depth, j = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[j], 0)
                j += 1
            i = text.index("{", j)
            depth, j = 1, i + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                j += 1
            yield m.group(1), text[i + 1:j - 1]


def test_every_cluster_launch_waits_for_its_predecessor_first():
    launched = _launched("launch_dep_cluster")
    assert launched == {"k_skin_step"}
    bodies = [b for k, b in _kernels() if k in launched]
    assert bodies
    for b in bodies:
        assert b.lstrip().startswith("dep_sync();")


def test_only_clusters_wait_on_their_ctas():
    clusters = _launched("launch_dep_cluster")
    for kernel, body in _kernels():
        if kernel not in clusters:
            assert not re.search(r"barrier\.cluster|this_cluster|this_grid|skin_sync|cluster_exclusive_scan", body), kernel


def test_the_launchers_are_the_two_that_are_tested():
    assert set(re.findall(r"\b(launch_\w+)\(", _code(SOURCES["pdl.cuh"]))) == {"launch_dep", "launch_dep_cluster"}
