"""Which launches of a step overlap: on fields of at most 10 MB a component most of them, on larger
ones only the sin/cos y passes (two in each of the four stages).  Read from the captured graph of
a step, whose edges say whether a kernel may start before its predecessor has ended."""
import pytest

from capture import captured

pytestmark = pytest.mark.gpu

# (basis, precision, sizes, launches that overlap; None: most of them)
CASES = [(b, "f32", (32, 32, 32), None) for b in ("FFF", "SFF", "SSF", "SSS")]
CASES += [("FFF", "f32", (128, 128, 256), 0), ("FFF", "f64", (128, 128, 128), 0), ("SFF", "f32", (128, 128, 256), 0),
          ("SSF", "f32", (128, 128, 256), 8), ("SSS", "f32", (128, 128, 256), 8), ("SSF", "f64", (128, 128, 128), 8)]


@pytest.mark.parametrize("basis,prec,N,count", CASES)
def test_overlapped_launches_of_a_step(cuda, basis, prec, N, count):
    import tarang_b200 as tb
    plan = tb.Plan(N, basis=basis, precision=prec, dealias="two_thirds", nu=0.01, kappa=0.01, dt=1e-4, Ra=1e4, Pr=1.0)
    u, T = plan.field(3), plan.field(1)
    step = (lambda: plan.rk4_step(u, 1)) if basis == "FFF" else (lambda: plan.rk4_step_rbc(u, T, 1))
    step()
    types = captured(plan, step)[1]
    overlapped = types.count(1)
    assert len(types) > 16 and (overlapped > len(types) // 2 if count is None else overlapped == count)
