"""GPU: roundings of the one-launch sweeps: a small-block solve's quotients round once,
and the dominant term of a selected inverse's diagonal or of a solve's row is added
last."""

import numpy as np
import pytest
import torch

import serinv_gb300 as sg

pytestmark = pytest.mark.gpu


def _diagonal(n, b, a, dt, rng):
    d = np.exp2(rng.uniform(-20, 20, (n, b))).astype(dt)
    t = np.exp2(rng.uniform(-20, 20, a)).astype(dt)
    D = np.zeros((n, b, b), dt)
    D[:, np.arange(b), np.arange(b)] = d
    L = [D, np.zeros((n - 1, b, b), dt), np.zeros((n, a, b), dt), np.diag(t).astype(dt)]
    return [torch.from_numpy(x).cuda() for x in L], np.concatenate([d.ravel(), t])


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("case", [(3, 5, 3, np.float64), (6, 8, 32, np.float64), (4, 16, 0, np.float64), (5, 20, 7, np.float32),
                                  (2, 32, 1, np.float32), (9, 1, 1, np.float64)])
def test_quotients_round_once(case, trans):
    n, b, a, dt = case
    rng = np.random.default_rng(b)
    L, d = _diagonal(n, b, a, dt, rng)
    B = rng.standard_normal((n * b + a, 700)).astype(dt)
    X = torch.from_numpy(B).cuda()
    sg.pobtas(*L, X, trans=trans)
    got, ref = X.cpu().numpy(), B / d[:, None]
    # one correction with a reciprocal that is off by at most a little over half an
    # ulp gives the rounded quotient but for ties; a product with it misses a quarter
    assert (np.abs(got - ref) <= np.spacing(np.abs(ref))).all()
    assert np.mean(got != ref) < 1e-3


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_quotients_at_the_ends_of_the_range(dt):
    f = np.finfo(dt)
    B = np.array([np.inf, -np.inf, np.nan, 0.0, -0.0, f.max, f.tiny, -f.tiny * 64, 1.0, 3.0], dt)
    for d in (f.tiny, f.max, 1.0, 3.0, np.inf):
        L = [torch.full((1, 1, 1), float(d), dtype=torch.from_numpy(B).dtype, device="cuda")]
        L += [torch.empty(s, dtype=L[0].dtype, device="cuda") for s in ((0, 1, 1), (1, 0, 1), (0, 0))]
        for trans in ("N", "T"):
            X = torch.from_numpy(B[None].copy()).cuda()
            sg.pobtas(*L, X, trans=trans)
            got = X.cpu().numpy()[0]
            with np.errstate(all="ignore"):
                ref = B / dt(d)
            # a quotient below the normal range may round twice
            assert np.isclose(got, ref, rtol=2 * f.eps, atol=2 * f.smallest_subnormal, equal_nan=True).all(), (d, got, ref)


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("case", [(3, 8, 0), (2, 5, 9), (4, 16, 32), (2, 2, 1), (1, 7, 20)])
def test_smaller_terms_are_summed_before_the_dominant_one(case, dt):
    """L_ii^{-1} = I minus a first column of 2**-k: the first entry of the product with
    its transpose is 1 + (b - 1) 2**-2k, its terms too small to change 1 one by one.
    All products here are exact, so the sum is the rounded one."""
    n, b, a = case
    k = 27 if dt == np.float64 else 13  # 2**-2k: a quarter (an eighth) of the spacing at 1
    D = np.tile(np.eye(b, dtype=dt), (n, 1, 1))
    D[:, 1:, 0] = 2.0 ** -k
    T = np.eye(a, dtype=dt)
    T[1:, :1] = 2.0 ** -k
    L = [torch.from_numpy(x).cuda() for x in (D, np.zeros((n - 1, b, b), dt), np.zeros((n, a, b), dt), T)]
    sg.pobtasi(*L)
    got, tip = L[0].cpu().numpy(), L[3].cpu().numpy()
    assert (got[:, 0, 0] == dt(1 + (b - 1) * np.longdouble(2) ** (-2 * k))).all()
    if a:
        assert tip[0, 0] == dt(1 + (a - 1) * np.longdouble(2) ** (-2 * k))
    for x, m in ((got[0], b), (tip, a)):
        ref = np.eye(m, dtype=dt)
        ref[1:, :1] = -(2.0 ** -k)
        np.testing.assert_array_equal(np.tril(x, -1), np.tril(ref, -1))
        np.testing.assert_array_equal(np.diag(x)[1:], np.ones(max(m - 1, 0), dt))


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("case", [(2, 5, 4, 1, np.float64), (2, 17, 33, 1, np.float64), (3, 40, 0, 3, np.float64),
                                  (2, 64, 20, 16, np.float64), (1, 100, 128, 2, np.float64), (3, 128, 1, 5, np.float64),
                                  (2, 33, 9, 1, np.float32), (2, 90, 0, 4, np.float32), (2, 127, 100, 20, np.float32)])
def test_a_row_of_a_solve_adds_its_diagonals_term_last(case, trans):
    """Unit factors with -2**-k in the last row (the first column for L^T), right-hand
    sides of 2**-k with 1 in that row: it becomes 1 + (rows - 1) 2**-2k.  All terms and
    their sums below 1 are exact."""
    n, b, a, nrhs, dt = case
    k = 27 if dt == np.float64 else 13

    def factor(m):
        L = np.eye(m, dtype=dt)
        if m > 1 and trans == "N":
            L[-1, :-1] = -(2.0 ** -k)
        elif m > 1:
            L[1:, 0] = -(2.0 ** -k)
        return L

    def rows(m, one):
        x = np.full(m, 2.0 ** -k, dtype=dt)
        if m:
            x[-1 if trans == "N" else 0] = one(m)
        return x

    L = [np.tile(factor(b), (n, 1, 1)), np.zeros((n - 1, b, b), dt), np.zeros((n, a, b), dt), factor(a)]
    L = [torch.from_numpy(x).cuda() for x in L]
    B, ref = (np.concatenate([rows(b, one)] * n + [rows(a, one)])[:, None].repeat(nrhs, 1)
              for one in (lambda m: 1.0, lambda m: dt(1 + (m - 1) * np.longdouble(2) ** (-2 * k))))
    X = torch.from_numpy(B.copy()).cuda()
    sg.pobtas(*L, X, trans=trans)
    np.testing.assert_array_equal(X.cpu().numpy(), ref)
