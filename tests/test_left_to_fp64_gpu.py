"""Residue products of values whose large elements meet only small ones: whole
tiles are summed in FP64 inside the reconstruction, beside tiles that are not, in
each of its forms (columns of a block, few rows, form of the result)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.fixture(scope="module")
def api():
    from rimp2_gpu_gb300 import api
    return api


def apart(rng, rows, k, low):
    """Rows (C order): the first `low` with values in the first half of the terms
    only, the next with a factor of 1e-12 there, the rest everywhere."""
    x = rng.standard_normal((rows, k))
    x[:low, k // 2:] = 0.0
    x[low:2 * low, : k // 2] *= 1e-12
    return x


def check(got, ref, mag, k):
    # both sides: sums of k terms in FP64, or rounded once
    assert np.isfinite(got).all()
    assert (np.abs(got - ref) <= 2 * (k + 4) * U * mag).all()


@pytest.mark.parametrize("m,n,k", [
    (65, 33, 400), (64, 64, 400),  # one tile and a row past it
    (300, 300, 200), (129, 700, 331),
    (49, 900, 330), (48, 900, 330), (47, 901, 330), (17, 3000, 250), (16, 3000, 250), (900, 40, 333),  # few rows, few columns
    (1950, 1930, 33), (1900, 1900, 33),  # either side of six tiles an SM
])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 1.0), (0.5, -2.0)])
def test_product(api, m, n, k, alpha, beta):
    rng = np.random.default_rng(m + n + k)
    A, B = apart(rng, m, k, 2 * m // 5), apart(rng, n, k, n // 3)
    B[:, :] = B[:, ::-1]  # the columns' halves against the rows'
    C = np.asfortranarray(rng.standard_normal((m, n)))
    ref = alpha * (A @ B.T) + beta * C
    mag = abs(alpha) * (np.abs(A) @ np.abs(B).T) + 2 * abs(beta) * np.abs(C) + np.abs(ref)
    At, Bt = np.asfortranarray(A.T), np.asfortranarray(B.T)
    before = api.kernel_launch_count()
    api.dgemm("T", "N", m, n, k, alpha, At, k, Bt, k, beta, C, m)
    assert api.kernel_launch_count() - before >= (3 if k <= 64 else 4)  # residues
    check(C, ref, mag, k)


@pytest.mark.parametrize("nvirt,nocc,nba", [(60, 5, 200), (93, 7, 130), (351, 8, 70)])
def test_symmetric_product(api, nvirt, nocc, nba):
    """g of one set of vectors with itself: the mirror of every tile."""
    rng = np.random.default_rng(nvirt)
    n = nvirt * nocc
    X = apart(rng, n, nba, n // 3)[rng.permutation(n)]
    X[: n // 2] = X[: n // 2][np.argsort(np.abs(X[: n // 2, -1]))]  # tiles of one kind and mixed ones
    C = np.asfortranarray(X.T).reshape((nba, nvirt, nocc), order="F")
    G = np.zeros((nvirt, nocc, nvirt, nocc), order="F")
    api.calc_gocc(nvirt, nocc, nba, C, G)
    got = G.reshape((n, n), order="F")
    check(got, X @ X.T, np.abs(X) @ np.abs(X).T, nba)
    assert (got == got.T).all()


@pytest.mark.parametrize("nvirt,nocc,nba", [(60, 5, 200), (30, 9, 130)])
def test_quotients(api, nvirt, nocc, nba):
    """g / D with whole tiles in FP64; U = 1 keeps them as they are."""
    rng = np.random.default_rng(nvirt)
    n = nvirt * nocc
    X = apart(rng, n, nba, n // 3)
    C = np.asfortranarray(X.T).reshape((nba, nvirt, nocc), order="F")
    eo, ev = np.sort(rng.random(nocc) - 1.5), np.sort(rng.random(nvirt) + 0.1)
    t = np.zeros((nocc, nocc, nvirt, nvirt), order="F")
    api.calc_toccA(nvirt, nocc, nocc, nba, C, eo, ev, t, np.asfortranarray(np.eye(nocc)))
    X3 = X.reshape((nocc, nvirt, nba))
    d = eo[:, None, None, None] + eo[None, :, None, None] - ev[None, None, None, :] - ev[None, None, :, None]
    ref = np.einsum("iak,jbk->ijab", X3, X3, optimize=True) / d
    mag = np.einsum("iak,jbk->ijab", np.abs(X3), np.abs(X3), optimize=True) / np.abs(d)
    check(t, ref, mag + np.abs(ref), nba + nocc)


def test_magnitudes_of_a_long_sum(api):
    """sum |a||b| is 2^-5.8 of ||a|| ||b||, spread over sixteen sums of 1024 of which
    none has 2^-8: no element is left to FP64, whose sums depend on the order of the
    terms; residues' do not."""
    rng = np.random.default_rng(4)
    m, n, k, big = 64, 80, 16384, 1000.0

    def rows(r, at):
        x = (0.5 + 0.5 * rng.random((r, k))) * np.where(rng.random((r, k)) < 0.5, -1.0, 1.0)
        x[:, at] = big * (0.75 + 1e-3 * rng.random(r))
        return x
    A, B = rows(m, 0), rows(n, 1)
    norms = np.linalg.norm(A, axis=1)[:, None] * np.linalg.norm(B, axis=1)[None, :]
    mag = np.abs(A) @ np.abs(B).T
    assert (mag > norms / 64).all()  # whatever the scales
    assert (np.abs(A[:, :1024]) @ np.abs(B[:, :1024]).T < norms / 256).all()

    def product(p):
        C = np.zeros((m, n), order="F")
        api.dgemm("T", "N", m, n, k, 1.0, np.asfortranarray(A[:, p].T), k, np.asfortranarray(B[:, p].T), k, 0.0, C, m)
        return C
    same = np.arange(k)
    C = product(same)
    check(C, A @ B.T, mag, k)
    for _ in range(3):
        # the large terms stay in the first sum, the others change places
        assert (C == product(np.concatenate([same[:2], 2 + rng.permutation(k - 2)]))).all()
