"""Field calls of one plan in flight on two streams at once.

Recovery and adjoint share the plan's scratch: the element pass of one call must not start
over it before the node pass of the call before has read it, on whichever stream that is.
The calls go through the C ABI, which does not wait on the host, and queue behind a kernel
that keeps both streams busy, so that they meet on the GPU. Bar: the same bits as one call
after the other."""
import numpy as np
import pytest
import torch

from calculixpp_b200 import Plan, _lib
from calculixpp_b200 import meshgen as mg
from tests.helpers import box_model

pytestmark = pytest.mark.gpu


def test_scratch_is_ordered_between_streams(cuda):
    model = box_model(mg.C3D8, 24, 24, 24, jitter=0.05)
    n, e = model.mesh.n_nodes, model.mesh.n_elems
    rng = np.random.default_rng(0)
    us = [torch.as_tensor(rng.uniform(-1e-3, 1e-3, 3 * n), device=cuda) for _ in range(4)]
    with Plan(model) as plan:
        def buffers(k):
            sizes = (6 * n, 6 * n, 3 * n) if k % 3 else (e, 3 * n)
            return [torch.empty(s, dtype=torch.float64, device=cuda) for s in sizes]

        def call(k, out, stream):
            p = [t.data_ptr() for t in (us[k % 4], *out)]
            if k % 3:
                rc = plan.lib.cxg_recover_fields(plan.h, p[0], None, *p[1:], stream)
            else:
                rc = plan.lib.cxg_adjoint_compliance(plan.h, *p, stream)
            _lib.check(rc)

        want, got = ([buffers(k) for k in range(16)] for _ in range(2))
        for k, out in enumerate(want):
            call(k, out, None)
            torch.cuda.synchronize()
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        for s in streams:
            with torch.cuda.stream(s):
                torch.cuda._sleep(4_000_000)
        for k, out in enumerate(got):
            call(k, out, streams[k % 2].cuda_stream)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for w, g in zip(want, got) for a, b in zip(w, g))
