"""The 9 x 9 trial-step decomposition with the matrix in registers (gr_svd9,
through me_svd_u at order 9) where its paths part: matrices per warp (1 to 32,
from the count), the cancellation of rank-deficient matrices, deflations
before the first sweep, and radii outside the normal range.

w and U come from backward-stable transformations (a few hundred rounding
errors of 1.1e-16 each, growing as their square root in practice): singular
values within 1e-13 of |a| of numpy's, U^T U within 1e-13 of 1 and U diag(w) U^T
within 1e-12 |a| of a symmetric semidefinite a (V = U up to signs, which squares
remove: U diag(w^2) U^T = a a^T)."""
import numpy as np
import pytest

import me_b200

pytestmark = pytest.mark.gpu


def _jacobians(rng, count):
    return rng.normal(size=(count, 60, 9)) * np.logspace(0, 2, 9)


def _inputs(kind, count):
    rng = np.random.default_rng(count)
    j = _jacobians(rng, count)
    if kind == "zero_columns":
        for m in range(count):
            j[m][:, rng.choice(9, size=1 + m % 4, replace=False)] = 0.0
    if kind == "rank4":
        j = j[:, :4]
    h = np.einsum("mki,mkj->mij", j, j)
    if kind == "orthogonal":
        return np.linalg.qr(rng.normal(size=(count, 9, 9)))[0]
    if kind == "diagonal":
        return np.einsum("mi,ij->mij", rng.normal(size=(count, 9)), np.eye(9))
    if kind == "zero_pivot":
        a = np.triu(rng.normal(size=(count, 9, 9)))
        a[:, 4, 4] = 0.0
        return a
    return {"tiny": h * 1e-130, "huge": h * 1e130}.get(kind, h)


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("lanes", [1, 32])
@pytest.mark.parametrize("count", [1, 33, 1184, 1185, 2369, 18945])
def test_counts(count, lanes, fast):
    _check(_inputs("normal", count), lanes, fast)


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("kind", ["zero_columns", "rank4", "orthogonal", "diagonal", "zero_pivot",
                                  "tiny", "huge"])
def test_kinds(kind, lanes, fast):
    _check(_inputs(kind, 257), lanes, fast)


def _check(a, lanes, fast):
    u, w, hits = me_b200.svd_u(a, lanes=lanes, fast=fast)
    assert hits == 0
    scale = np.linalg.norm(a, axis=(1, 2))
    unit = a / scale[:, None, None]
    want = np.linalg.svd(unit, compute_uv=False)
    got = np.sort(w / scale[:, None], axis=1)[:, ::-1]
    assert np.max(np.abs(got - want)) < 1e-13
    eye = np.einsum("mki,mkj->mij", u, u)
    live = np.abs(w / scale[:, None]) > 1e-13  # a zero singular value has no column of its own
    both = live[:, :, None] & live[:, None, :]
    assert np.max(np.abs(np.where(both, eye - np.eye(9), 0.0))) < 1e-13
    ws = w / scale[:, None]
    gram = np.einsum("mik,mk,mjk->mij", u, ws * ws, u)
    assert np.max(np.abs(gram - unit @ unit.transpose(0, 2, 1))) < 1e-12


def test_zero_matrix():
    u, w, hits = me_b200.svd_u(np.zeros((3, 9, 9)))
    assert hits == 0 and np.all(w == 0) and np.all(u == np.eye(9))


@pytest.mark.parametrize("count", [1, 33, 1185, 20011])
@pytest.mark.parametrize("kind", ["normal", "rank4", "orthogonal", "zero_pivot"])
def test_full_decomposition(kind, count):
    """me_svd at order 9 (gr_svd9_v): a = u diag(w) v^T, u and v orthogonal
    where w is not zero, to the bounds above."""
    a = _inputs(kind, count)
    u, w, v = me_b200.svd(a)
    scale = np.linalg.norm(a, axis=(1, 2))[:, None]
    unit, ws = a / scale[:, :, None], w / scale
    assert np.all(w >= 0)
    assert np.max(np.abs(np.einsum("mik,mk,mjk->mij", u, ws, v) - unit)) < 1e-12
    eye = np.einsum("mki,mkj->mij", v, v)
    assert np.max(np.abs(eye - np.eye(9))) < 1e-13
    live = ws > 1e-13
    both = live[:, :, None] & live[:, None, :]
    eye = np.einsum("mki,mkj->mij", u, u)
    assert np.max(np.abs(np.where(both, eye - np.eye(9), 0.0))) < 1e-13
