"""Spans of right-hand sides per block of the anterpolation and interpolation:
the autotuner times each launch once (a span is rounded up to a round of 16, so
that several values name one launch), and matvecs repeat bit for bit, with the
same bits, for spans that give other grids."""
import numpy as np
import pytest

from scadyn_b200 import api
from tests.diag_operator import diagonal_solver
from tests.gpu_helpers import solver_from_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs,spans", [(1, 0), (7, 1), (12, 0), (16, 0), (40, 4)])
def test_tuner_times_each_launch_once(nrhs, spans):
    """FP64: the default, the three-pass FFT chain (nine launches a matvec, seven
    fused) and at most `spans` other spans, reps timed matvecs and a warm-up each."""
    s = diagonal_solver(np.full(3000, 1.0 + 0.1j))
    s.profile_matvec(1, nrhs, api.PREC_FP64)
    s.timing(reset=True)
    reps = 2
    s.tune_matvec(nrhs, api.PREC_FP64, reps)
    launches = s.timing()["launches"]
    s.close()
    assert launches <= (7 + 9 + 9 * spans) * (reps + 1)


@pytest.mark.parametrize("precision", [api.PREC_MIXED, api.PREC_FP64])
def test_spans_keep_the_bits(small_op, precision):
    s = solver_from_oracle(small_op)
    rng = np.random.default_rng(4)
    mat = rng.standard_normal((40, s.n)) + 1j * rng.standard_normal((40, s.n))
    kw = dict(tol=1e-6, m=20, cycles=6, block=40, precision=precision, inner_tol=1e-3, want_x=True)
    want = s.solve_columns(mat, **kw)[2]
    for spans in ((16, 32), (32, 16), (48, 48)):
        s.apply_tuning(dict(nrhs=40, precision=precision, scatter_span=spans[0], gather_span=spans[1]))
        assert s.check_matvec_repeat(20, 40, precision) == (0, 0), spans
        assert np.array_equal(s.solve_columns(mat, **kw)[2], want), spans
    s.close()
