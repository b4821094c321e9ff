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


@pytest.mark.parametrize("call", ["sharpen", "convergence"])
def test_default_stream_calls_wait_for_a_fit_on_another_stream(cuda, call):
    """A fit on a non-blocking stream keeps its row and plane sums in the scratch
    that sharpening and the convergence value use on the default stream, which
    does not wait for that stream by itself: the fit's lattice has the same bits
    as alone, at every distance between the calls."""
    import n4b200
    from n4b200 import _lib
    lib = _lib.load()
    shape, nc = (256, 256, 200), (7, 7, 7)
    field = cuda.rand(shape, device="cuda")
    x = cuda.rand(4096, device="cuda")
    y = cuda.rand(4096, device="cuda")
    out = cuda.empty_like(x)
    E, cv = np.zeros(200, np.float32), ctypes.c_double()
    want = n4b200.FitBspline3D(field, None, nc)
    cuda.cuda.synchronize()
    ctx = n4b200.Context(0)
    s = cuda.cuda.Stream()
    for _ in range(20):
        with cuda.cuda.stream(s):
            got = n4b200.FitBspline3D(field, None, nc, ctx=ctx)
        if call == "sharpen":
            _lib.check(lib.n4_sharpen_image(ctx.handle, x.data_ptr(), None, 4096, 200, 0.01, 0.15, out.data_ptr(), None,
                                            None, E.ctypes.data))
        else:
            _lib.check(lib.n4_convergence(ctx.handle, x.data_ptr(), y.data_ptr(), None, 4096, 0, ctypes.byref(cv)))
        s.synchronize()
        assert cuda.equal(got, want)
