"""The cell update's reciprocal, quotient, root and third (csrc/lattice.cuh)
against CUDA's correctly rounded operations: equal bits over the ranges that
their comment states (all floats of the range; 2e9 pairs for the quotient),
and their results at the ends of the range and beyond it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import gpu as ogpu  # noqa: E402

RECIP, ROOT, THIRD, QUOTIENT = range(4)
INF, NAN = float("inf"), float("nan")


@pytest.fixture(scope="module")
def probe():
    return C.CDLL(str(ogpu.build_probe()))


def _bits(v):
    return int(np.float32(v).view(np.uint32))


@pytest.mark.parametrize("op,first,n", [
    (RECIP, _bits(1e-37), _bits(2.0 ** 126) - _bits(1e-37)),
    (ROOT, _bits(1e-30), _bits(3.4e38) - _bits(1e-30)),
    (THIRD, _bits(1e-30), _bits(3.4e38) - _bits(1e-30)),
    (THIRD, _bits(-1e-30), _bits(-3.4e38) - _bits(-1e-30)),
    (QUOTIENT, 12345, 2_000_000_000),
], ids=["recip", "root", "third", "third_negative", "quotient"])
def test_results_are_correctly_rounded(probe, op, first, n):
    bad = torch.zeros(1, dtype=torch.int64, device="cuda:0")
    ex = torch.zeros(2, dtype=torch.int32, device="cuda:0")
    rc = probe.olp_compare(op, C.c_uint32(first), C.c_uint32(n), C.c_void_p(bad.data_ptr()),
                           C.c_void_p(ex.data_ptr()))
    assert rc == 0
    assert int(bad) == 0, ex.view(torch.float32).tolist()


@pytest.mark.parametrize("op,a,b,want", [
    # what `/` gives, where a diverging flow can reach it
    (QUOTIENT, 1.0, INF, 0.0), (QUOTIENT, INF, 2.0, INF), (QUOTIENT, -INF, 2.0, -INF),
    (QUOTIENT, INF, INF, NAN), (QUOTIENT, NAN, 1.0, NAN), (QUOTIENT, 0.0, 2.0, 0.0),
    (QUOTIENT, -1.5, 0.5, -3.0), (QUOTIENT, 1.0, -4.0, -0.25),
    # a reciprocal too small for a normal float is 0
    (RECIP, 2.0 ** 126, 1.0, 2.0 ** -126), (RECIP, 3e38, 1.0, 0.0), (RECIP, NAN, 1.0, NAN),
    (ROOT, 3.4e38, 1.0, float(np.sqrt(np.float32(3.4e38)))), (ROOT, NAN, 1.0, NAN),
    (ROOT, 1e-30, 1.0, float(np.sqrt(np.float32(1e-30)))),
    (THIRD, 0.0, 1.0, 0.0), (THIRD, NAN, 1.0, NAN),
])
def test_results_at_and_beyond_the_range(probe, op, a, b, want):
    t = lambda v: torch.tensor([v], dtype=torch.float32, device="cuda:0")  # noqa: E731
    x, y, got, rounded = t(a), t(b), t(0.0), t(0.0)
    p = lambda v: C.c_void_p(v.data_ptr())  # noqa: E731
    assert probe.olp_values(op, p(x), p(y), 1, p(got), p(rounded)) == 0
    assert np.array_equal(np.float32(float(got)), np.float32(want), equal_nan=True)
