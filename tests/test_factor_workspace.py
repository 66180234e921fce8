"""Host replay of the workspace of the recursive Cholesky-with-inverse (chol_inv64 in
dynemol_gb300/csrc/elhl_api.cu): a split forms L21 in n1 columns of W, which are its own until
the second stream has copied them into place, so the second block's splits take the columns
after them and the first block's, done before, the same ones.  No two open splits overlap,
every column used lies inside W, chol_inv_fits says so, and the factors come out right although
L21 is in place only at the end."""
import os
import re

import numpy as np
import pytest

API = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynemol_gb300", "csrc",
                        "elhl_api.cu")).read()
LEAF = 64


def ru(x, m):
    return (x + m - 1) // m * m


def test_replay_is_the_source():
    body = re.sub(r"\s+", " ", API)
    assert ("return (size_t)ld * n1 <= wcap && chol_inv_fits(n1, ld, wcap) && "
            "chol_inv_fits(n2, ld, wcap - (size_t)ld * n1);") in body
    assert "if (int rc = chol_inv64(A, G, n1, ld, row0, W, info, tc)) return rc;" in body
    assert "if (int rc = chol_inv64(A22, G22, n2, ld, row0 + n1, W + (size_t)n1 * ld, info, tc)) return rc;" in body
    assert "const int n1 = round_up(n / 2, leaf), n2 = n - n1;" in body


def fits(n, wcap):  # in columns
    if n <= LEAF:
        return True
    n1 = ru(n // 2, LEAF)
    return n1 <= wcap and fits(n1, wcap) and fits(n - n1, wcap - n1)


@pytest.mark.parametrize("n", list(range(1, 700, 3)) + list(range(700, 4200, 31)) + [3720, 8192, 12000, 16384])
def test_open_splits_lie_side_by_side_inside_w(n):
    assert fits(n, n)
    owner = [None] * n

    def rec(m, w, depth):
        if m <= LEAF:
            return
        n1 = ru(m // 2, LEAF)
        rec(n1, w, depth + 1)                       # before L21: the same columns
        assert w + n1 <= n
        assert all(o is None for o in owner[w:w + n1])
        owner[w:w + n1] = [depth] * n1              # L21 until the side work is done
        rec(m - n1, w + n1, depth + 1)
        assert owner[w:w + n1] == [depth] * n1
        owner[w:w + n1] = [None] * n1               # the main stream has waited for the side

    rec(n, 0, 0)
    assert owner == [None] * n


@pytest.mark.parametrize("n", [65, 130, 200, 513, 700, 1000])
def test_factors_with_l21_left_in_w(n):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, n))
    S = X @ X.T / n + np.eye(n)
    A, G, W = np.tril(S), np.full((n, n), np.nan), np.full((n, n), np.nan)

    def rec(a, m, w):
        i = slice(a, a + m)
        if m <= LEAF:
            Lb = np.linalg.cholesky(np.tril(A[i, i]) + np.tril(A[i, i], -1).T)
            A[i, i], G[i, i] = Lb, np.tril(np.linalg.inv(Lb))
            return
        n1 = ru(m // 2, LEAF)
        i1, i2, c = slice(a, a + n1), slice(a + n1, a + m), slice(w, w + n1)
        rec(a, n1, w)
        W[:m - n1, c] = A[i2, i1] @ np.tril(G[i1, i1]).T
        A[i2, i1] = np.nan                           # its copy lands at any time before the split ends
        A[i2, i2] -= np.tril(W[:m - n1, c] @ W[:m - n1, c].T)
        rec(a + n1, m - n1, w + n1)
        A[i2, i1] = W[:m - n1, c]
        G[i2, i1] = -np.tril(G[i2, i2]) @ (W[:m - n1, c] @ np.tril(G[i1, i1]))

    rec(0, n, 0)
    L = np.linalg.cholesky(S)
    assert np.abs(np.tril(A) - L).max() < 1e-12
    assert np.abs(np.tril(G) - np.linalg.inv(L)).max() < 1e-12
