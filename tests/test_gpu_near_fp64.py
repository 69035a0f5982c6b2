"""The FP64 near zone at the sizes where its kernels change: right-hand-side
counts around the passes of 8 and 16 (one on the FMA units, more as DMMAs),
group sizes whose 3n unknowns leave every remainder of the blocks of 4 and 8,
complex64 and complex128 storage, one and two partial sums.  A host operator
with a zero grid part isolates it: A x is the near-zone product alone, compared
with numpy in FP64; every column of a batch has the bits of the column alone."""
import numpy as np
import pytest

from scadyn_b200 import api

pytestmark = pytest.mark.gpu


def _operator(per_box, storage, seed=3):
    """per_box tets in each of 3 x 2 boxes; all pairs of neighbouring boxes."""
    rng = np.random.default_rng(seed)
    n = (12, 12, 12)
    boxes = [(x, y, 2) for y in (1, 2) for x in (0, 1, 2)]
    cube = np.array([b for b, c in zip(boxes, per_box) for _ in range(c)])
    T = len(cube)
    first = 2 * cube[:, 0] + n[0] * (2 * cube[:, 1] + n[1] * 2 * cube[:, 2])
    j = np.arange(27)
    indS = (first[:, None] + j % 3 + n[0] * (j // 3 % 3 + n[1] * (j // 9)) + 1).astype(np.int32)
    a, b = np.nonzero((np.abs(cube[:, None] - cube[None]) <= 1).all(2) & (np.arange(T)[:, None] <= np.arange(T)))
    sp = rng.standard_normal((len(a), 3, 3)) + 1j * rng.standard_normal((len(a), 3, 3))
    sp = (0.3 / np.sqrt(T) * sp).astype(storage)
    sp[a == b] += np.eye(3, dtype=storage)
    return n, indS, sp, np.stack([a, b], 1).astype(np.int32) + 1


def _dense(sp, ind, T):
    V = sp.astype(np.complex128).transpose(0, 2, 1)
    A = np.zeros((T, 3, T, 3), np.complex128)
    for v, (i, j) in zip(V, ind - 1):
        A[i, :, j] = v
        if i != j:
            A[j, :, i] = v.T
    return A.reshape(3 * T, 3 * T)


@pytest.mark.parametrize("split", [1, 2])
@pytest.mark.parametrize("storage", [np.complex64, np.complex128])
@pytest.mark.parametrize("per_box", [(1, 2, 3, 1, 2, 1), (5, 8, 7, 11, 13, 4), (24, 23, 16, 24, 25, 30)])
def test_near_zone_fp64(per_box, storage, split):
    n, indS, sp, ind = _operator(per_box, storage)
    T = len(indS)
    s = api.Solver(*n, 1.0, (0.0, 0.0, 0.0), T, near_split=split)
    s.set_wavenumber(0.3)
    zero = np.zeros((T, 27), np.complex128)
    s.set_projectors(zero, zero, zero, zero, indS)
    s.build_G()
    s.set_nearzone(sp, ind)
    A = _dense(sp, ind, T)
    rng = np.random.default_rng(7)
    mat = rng.standard_normal((35, 3 * T)) + 1j * rng.standard_normal((35, 3 * T))
    y = s.compute_Ax2(mat[0])
    want = A @ mat[0]
    # 3T products per sum: a few thousand roundings of 1.1e-16 of the terms at most
    assert np.linalg.norm(y - want) <= 1e-14 * np.linalg.norm(np.abs(A) @ np.abs(mat[0]))
    kw = dict(tol=1e-9, m=12, cycles=3, precision=api.PREC_FP64, want_x=True)
    _, it1, X1, _ = s.solve_columns(mat, block=1, **kw)
    for block in (2, 7, 8, 9, 16, 17, 24, 25, 33, 35):
        _, it, X, _ = s.solve_columns(mat[:block], block=block, **kw)
        assert np.array_equal(X, X1[:block]) and np.array_equal(it, it1[:block]), block
    s.close()
