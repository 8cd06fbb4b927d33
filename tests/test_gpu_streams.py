"""Other streams beside a batch solve: the CTAs of a size bucket leave their SMs when its queue is empty."""
import numpy as np
import pytest

from conicxx_gb300 import BatchSolver, generators

pytestmark = pytest.mark.gpu


def test_sms_are_free_once_a_bucket_is_done():
    """One FP64 instance of 480 rows (some 100 ms on one SM) and 3000 of 12 rows (some 10 ms on the other SMs,
    whose registers their CTAs fill). Work of another stream, behind a few milliseconds of waiting, ends
    long before the large instance does."""
    torch = pytest.importorskip("torch")
    big = generators.random_conic_qp(0, n=480, m_zero=0, m_nonneg=100, soc=(3,) * 5, density=0.3, family=9)
    small = [generators.random_conic_qp(s, n=12, m_zero=0, m_nonneg=8, soc=(3,), density=0.5, family=9) for s in range(16)]
    B = BatchSolver([big] + [small[i % 16] for i in range(3000)], precision=0, warm_start=0)
    out = [torch.zeros(k, dtype=torch.float64, device="cuda") for k in (B.n_total, B.m_total, B.m_total)]
    a = torch.randn(4096, 4096, dtype=torch.float32, device="cuda")
    c = torch.empty_like(a)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]

    def solve():
        B.solve_device(*[t.data_ptr() for t in out], s1.cuda_stream)

    with torch.cuda.stream(s2):
        torch.mm(a, a, out=c)  # both kernels loaded
        torch.cuda._sleep(1000)
    solve()
    torch.cuda.synchronize()
    ev[0].record(s1)
    solve()
    ev[1].record(s1)
    with torch.cuda.stream(s2):
        torch.cuda._sleep(int(30e6))  # about 15 ms: the small instances are done
        for _ in range(4):
            torch.mm(a, a, out=c)
        ev[2].record(s2)
    torch.cuda.synchronize()
    whole, other = ev[0].elapsed_time(ev[1]), ev[0].elapsed_time(ev[2])
    print("solve %.1f ms, other stream's work done at %.1f ms" % (whole, other))
    assert whole > 40.0
    assert other < 0.8 * whole
