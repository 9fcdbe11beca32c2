"""Projections of host arrays after the session has moved to another stream: they work in
the session's scratch, which a refresh or a set_object queued on the old stream may still
need, so they run after it. The old stream is kept busy (a spin of about 50 ms) while the
calls are made, and both results are compared with the same calls on one stream.

The forward projections and the error sinogram are FP64 sums in any order, rounded once:
1.2e-7 of the value; back projection and FBP are the same arithmetic on the same data.
"""
import numpy as np
import pytest

import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem

pytestmark = pytest.mark.gpu


def test_projections_wait_for_the_old_stream():
    import torch
    pb, obj = make_problem(ncol=32, nrow=8, nview=40)
    s = pc.Session(to_gpu_problem(pb))
    rng = np.random.default_rng(1)
    x = rng.random(s.shape).astype(np.float32)
    y = rng.random(s.sino_shape).astype(np.float32)
    s.set_object(obj)
    ref = dict(err=s.get_error(), back=s.back_project(y), fwd=s.forward_project(x), fbp=s.fbp())
    calls = [lambda: np.array_equal(s.back_project(y), ref["back"]), lambda: np.array_equal(s.fbp(), ref["fbp"]),
             lambda: np.all(np.abs(s.forward_project(x) - ref["fwd"]) <= 1.2e-7 * np.abs(ref["fwd"]))]
    for call in calls:
        old, new = torch.cuda.Stream(), torch.cuda.Stream()
        s.set_stream(old.cuda_stream)
        s.get_error()  # the session's scratch is idle
        with torch.cuda.stream(old):
            torch.cuda._sleep(100_000_000)
        s.refresh_error()
        done = torch.cuda.Event()
        done.record(old)
        s.set_stream(new.cuda_stream)
        assert call()
        assert done.query()  # the refresh came first
        assert np.all(np.abs(s.get_error() - ref["err"]) <= 1.2e-7 * np.abs(pb.projections).max())
    s.close()
