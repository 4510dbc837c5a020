"""The graph step on a context whose stream does not wait for the default stream.

Its buffers are initialised by memsets, among them the skin list's keys. On the default stream
a memset runs when that stream's own work is done, which the replays do not wait for: a list
cleared after it was built has no pairs. So the sources are checked for none, and a run is
compared with single steps while the default stream is busy.
"""
import re
from pathlib import Path

import numpy as np
import pytest

STEP = (Path(__file__).resolve().parents[1] / "delta_b200" / "csrc" / "step.cu").read_text()


def test_the_graph_buffers_are_initialised_in_the_contexts_order():
    body = STEP[STEP.index("static delta_status graph_alloc_all("):]
    body = re.sub(r"//[^\n]*", "", body[:body.index("\n}\n")])
    assert not re.search(r"\bcudaMemset\(|\bcudaMemcpy\(", body)
    last = max(m.start() for m in re.finditer(r"\bcudaMemsetAsync\(", body))
    assert "cudaStreamSynchronize(s->ctx->stream)" in body[last:]


@pytest.mark.gpu
def test_a_busy_default_stream_changes_nothing(scene_seed=12):
    import torch

    from delta_b200.engine import Simulation, StepParams
    from delta_b200.narrowphase import Context
    from delta_b200.scenarios import lattice_scene

    scene, prm, runs = lattice_scene(seed=scene_seed), StepParams.make(dt=1e-5), []
    side = torch.cuda.Stream()
    for busy in (False, True):
        ctx = Context(0, side.cuda_stream)
        sim = Simulation(ctx, scene, 8)
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(400_000_000)  # about 0.2 s of the default stream
        cps = sim.step(40, prm, graph=True)
        torch.cuda.synchronize()
        runs.append((cps, sim.state(), sim.skin_stats()["rebuilds"]))
        sim.close()
        ctx.close()
    (c0, s0, r0), (c1, s1, r1) = runs
    assert np.array_equal(c0, c1) and c0.sum() > 0 and r0 == r1
    for k in ("pos", "vel", "ang", "rot", "x", "y", "z"):
        assert np.array_equal(s0[k], s1[k]), k
