"""What the server's admission counts for a request against what its solve and its
mesh take on the device: no less (admitted solves stay within the budget), and
not far more (1.25 times and the megabyte of small buffers)."""
import pytest

from axisem_gb300.serve import Request, Server, _solve_bytes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("comp", [False, True])
@pytest.mark.parametrize("period,pole", [(50, 0), (50, 1), (50, 2), (25, 0), (25, 2)])
def test_estimate_covers_a_solve(gpu_lib, period, pole, comp):
    req = Request(0, 0.0, period, pole, 200.0, 300, 3600.0, 0.3)
    srv = Server(lib=gpu_lib, compensated=comp)
    try:
        before = srv._estimate(req)
        srv.preload([(period, pole)])
        own_estimate = srv._estimate(req)
        s = srv._solver(req, share=True)
        own, _ = _solve_bytes(s)
        s.close()
        assert own <= own_estimate <= 1.25 * own + (1 << 20)
        total = own + srv.used
        assert total <= before <= 1.25 * total + (1 << 20)
    finally:
        srv.close()
