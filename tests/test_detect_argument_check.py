"""delta_detect's check of the meshes and pairs comes before everything that follows a
body's triangle range or a pair's bodies.

A triangle range out of order, or a body index out of range, may name memory outside the
caller's arrays, so the box and culling kernels must not read through it. They are enqueued
before the host has read the check's result, hence two rules that the sources are tested for
(a GPU run with such a mesh would show nothing, or read out of range): the check is launched
first, and those kernels return on its result before they read anything. The GPU test then
checks the refusals on meshes whose arrays hold every vertex that the ranges name.
"""
import ctypes
import re
from pathlib import Path

import numpy as np
import pytest

SRC = (Path(__file__).resolve().parents[1] / "delta_b200" / "csrc" / "detect.cu").read_text()


def _body(marker):
    """The braces' content of the first function whose head contains `marker`."""
    m = re.search(marker, SRC)
    assert m, marker
    depth, j = 1, m.end()
    while depth:  # the parameter list
        depth += {"(": 1, ")": -1}.get(SRC[j], 0)
        j += 1
    i = SRC.index("{", j)
    depth, j = 1, i + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(SRC[j], 0)
        j += 1
    return SRC[i + 1:j - 1]


def test_the_check_is_launched_before_the_kernels_it_protects():
    body = _body(r"static delta_status detect_culled\(")
    check = body.index("k_check_detect<<<")
    for later in ("k_body_boxes<<<", "launch_cull(", "launch_survivors("):
        assert body.count(later) == 1 and body.index(later) > check, later


@pytest.mark.parametrize("kernel,guard", [("k_body_boxes", r"if \(\*bad\) return;"),
                                          ("k_cull_pairs", r"(dep_sync\(\);\s*)if \(rc\.bad && \*rc\.bad\) return;")])
def test_the_protected_kernels_return_on_a_failed_check(kernel, guard):
    assert re.match(r"\s*" + guard, _body(r"\b" + kernel + r"\(delta_meshes m"))


def _call(ctx, driver, tri_offset, pair_a, pair_b, triangles):
    """Status and contact count of delta_detect on well separated copies of one triangle."""
    import torch

    from delta_b200 import detection, lib

    n = len(tri_offset) - 1
    xyz = np.tile([[0.0, 0.0, 0.0], [0.01, 0.0, 0.0], [0.0, 0.01, 0.0]], (triangles, 1))
    xyz[:, 2] += np.repeat(0.1 * np.arange(triangles), 3)
    m = detection.Meshes(np.asarray(tri_offset, np.int64), xyz[:, 0].copy(), xyz[:, 1].copy(), xyz[:, 2].copy(),
                         np.full(n, 1e-4), np.zeros(n, np.uint8))
    contacts, count = detection.Contacts(64), ctypes.c_int64(-1)
    pa, pb = (torch.tensor(p, dtype=torch.int32).cuda() for p in (pair_a, pair_b))
    status = lib().delta_detect(ctx.handle, driver, 0, ctypes.byref(m.struct()), pa.data_ptr(), pb.data_ptr(),
                                len(pair_a), ctypes.byref(contacts.struct()), ctypes.byref(count), None)
    return status, count.value


@pytest.mark.gpu
@pytest.mark.parametrize("driver", range(11))
def test_bad_meshes_and_pairs_are_refused(ctx, driver):
    from delta_b200 import lib

    cases = [([0, 500, 160], [0], [1], b"65536"),            # a range out of order
             ([0, 65536, 65540], [0], [1], b"65536"),        # one triangle too many
             ([0, 4, 8], [0], [2], b"out of range"),         # no such body
             ([0, 4, 8], [-1], [1], b"out of range")]
    for off, pa, pb, text in cases:
        status, count = _call(ctx, driver, off, pa, pb, max(off))
        assert status != 0 and count == 0, (off, status, count)
        assert text in lib().delta_last_error(), off
    # the same context goes on, at the largest body that is accepted
    assert _call(ctx, driver, [0, 65535, 65537], [0], [1], 65537) == (0, 0)
