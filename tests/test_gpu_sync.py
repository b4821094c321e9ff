"""What a context's calls wait for."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_sync_waits_for_a_component_call_after_a_run(cuda):
    """n4_sync after an asynchronous run and an evaluation behind it, on a
    non-blocking stream: the evaluation is done as well, and the run's report
    is filled."""
    import n4b200
    from n4b200 import _lib
    ctx = n4b200.Context(0)
    im = cuda.rand((64, 64, 48), device="cuda") + 1
    p = n4b200.N4Param(NumberOfFittingLevels=1, MaximumNumberOfIterations=[2], ConvergenceThreshold=0.0, low_value=0.0)
    n4b200.N4(im, None, p, ctx=ctx)
    lattice = cuda.rand((7, 7, 7), device="cuda")
    s = cuda.cuda.Stream()
    s.wait_stream(cuda.cuda.current_stream())
    with cuda.cuda.stream(s):
        for _ in range(40):
            n4b200.EvaluateBspline3D(lattice, (7, 7, 7), (400, 400, 300), ctx=ctx)
        rep = (_lib.n4_report_t * 1)()
        _lib.check(_lib.load().n4_sync(ctx.handle, rep, 1))
        assert s.query()
    assert rep[0].status == 0 and rep[0].levels == 1
