"""Residue products in parts: large ones are cut into parts of rows and columns
with a workspace of bounded size.  Smaller bounds (RIMP2_RESIDUE_PARTS) reach every kind
of part at small sizes.  Residues do not depend on the parts: the same bits as in one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.fixture(scope="module")
def api():
    from rimp2_gpu_gb300 import api
    return api


def both(monkeypatch, api, parts, run):
    """run() in one part and in parts, and the launches of each."""
    n0 = api.kernel_launch_count()
    one = run()
    n1 = api.kernel_launch_count()
    monkeypatch.setenv("RIMP2_RESIDUE_PARTS", parts)
    cut = run()
    monkeypatch.delenv("RIMP2_RESIDUE_PARTS")
    return one, cut, n1 - n0, api.kernel_launch_count() - n1


FORMS = [
    # m, n, k, parts (rows, columns), how many of each
    (700, 150, 300, "256,4096", 3, 1),    # rows in three parts, the last one short
    (300, 900, 300, "4096,320", 1, 3),    # columns
    (513, 700, 300, "256,256", 3, 3),     # both; a last part of one row
    (640, 641, 50, "256,320", 3, 3),      # sums of one K chunk
    (520, 530, 1500, "256,256", 3, 3),    # sums beyond 1024
    (900, 40, 400, "256,256", 1, 4),      # few columns: transposed
]


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
@pytest.mark.parametrize("m,n,k,parts,rows,cols", FORMS)
def test_product_in_parts(api, monkeypatch, ta, tb, m, n, k, parts, rows, cols):
    rng = np.random.default_rng(m + n + k)
    A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    C0 = rng.standard_normal((m, n))
    At, Bt = np.asfortranarray(A if ta == "N" else A.T), np.asfortranarray(B if tb == "N" else B.T)
    for alpha, beta in ((1.0, 0.0), (-1.0, 1.0), (0.5, -2.0)):
        def run():
            C = np.asfortranarray(C0.copy())
            api.dgemm(ta, tb, m, n, k, alpha, At, At.shape[0], Bt, Bt.shape[0], beta, C, m)
            return C
        one, cut, n1, n2 = both(monkeypatch, api, parts, run)
        per = 3 if k <= 64 else 4
        assert n1 == per and n2 == per * rows * cols
        assert (one == cut).all()
        mag = abs(alpha) * (np.abs(A) @ np.abs(B)) + 2 * np.abs(beta * C0)
        assert (np.abs(cut - (alpha * (A @ B) + beta * C0)) <= 2 * (k + 4) * U * mag).all()


@pytest.mark.parametrize("m,n,k,parts", [f[:4] for f in FORMS])
def test_values_left_to_fp64_in_parts(api, monkeypatch, m, n, k, parts):
    """Single elements and whole tiles in FP64 in later parts; infinities and NaN there."""
    rng = np.random.default_rng(k)
    A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    A[m // 2:, k // 2:] = 0.0
    B[: k // 2, 2 * n // 3:] = 0.0
    A[m // 3] *= 1e200
    A[m - 1, 3], B[5, n - 1] = np.inf, np.nan
    B[3, n // 2] = 0.0
    At, Bt = np.asfortranarray(A.T), np.asfortranarray(B)

    def run():
        C = np.zeros((m, n), order="F")
        api.dgemm("T", "N", m, n, k, 1.0, At, k, Bt, k, 0.0, C, m)
        return C
    one, cut, n1, n2 = both(monkeypatch, api, parts, run)
    assert n2 > n1
    with np.errstate(all="ignore"):
        ref = A @ B
        mag = np.abs(A) @ np.abs(B)
    f = np.isfinite(ref)
    assert (np.isnan(ref) == np.isnan(cut)).all() and (np.isinf(ref) == np.isinf(cut)).all()
    assert (np.abs(cut - ref)[f] <= 2 * (k + 4) * U * mag[f]).all()
    assert (np.abs(one - ref)[f] <= 2 * (k + 4) * U * mag[f]).all()


@pytest.mark.parametrize("parts", ["256,4096", "4096,256", "256,256"])
def test_integrals_and_quotients_in_parts(api, monkeypatch, parts):
    """g and g / D: no symmetric form in parts; denominators of rows and columns that
    begin at a part."""
    rng = np.random.default_rng(7)
    nvirt, nocc, nba = 75, 7, 200
    X = rng.standard_normal((nocc, nvirt, nba)) * 0.05
    C = np.asfortranarray(X.transpose(2, 1, 0))
    eo, ev = np.sort(rng.random(nocc) - 1.5), np.sort(rng.random(nvirt) + 0.1)

    def run():
        G = np.zeros((nvirt, nocc, nvirt, nocc), order="F")
        api.calc_gocc(nvirt, nocc, nba, C, G)
        t = np.zeros((nocc, nocc, nvirt, nvirt), order="F")
        api.calc_toccA(nvirt, nocc, nocc, nba, C, eo, ev, t, np.asfortranarray(np.eye(nocc)))
        return G, t
    one, cut, n1, n2 = both(monkeypatch, api, parts, run)
    assert n2 > n1 + 8
    assert (one[0] == cut[0]).all()
    # the mirror's denominators subtract the virtual energies in the other order: an ulp of D
    d = eo[:, None, None, None] + eo[None, :, None, None] - ev[None, None, None, :] - ev[None, None, :, None]
    mag = np.einsum("iak,jbk->ijab", np.abs(X), np.abs(X), optimize=True) / np.abs(d)
    ref = np.einsum("iak,jbk->ijab", X, X, optimize=True) / d
    for t in (one[1], cut[1]):
        assert (np.abs(t - ref) <= 2 * (nba + nocc + 4) * U * mag).all()


@pytest.mark.parametrize("parts", ["256,4096", "300,300", "512,512"])
@pytest.mark.parametrize("amplitudes", [False, True])
def test_energies_by_blocks(api, monkeypatch, parts, amplitudes):
    """Pair energies from blocks of occupied orbitals with themselves and with others."""
    rng = np.random.default_rng(3)
    nvirt, nocc, nba = 90, 7, 400
    C = np.asfortranarray(rng.standard_normal((nba, nvirt, nocc)) * 0.05)
    eo, ev = np.sort(rng.random(nocc) - 1.5), np.sort(rng.random(nvirt) + 0.1)
    one, cut, n1, n2 = both(monkeypatch, api, parts,
                            lambda: api.energy(nvirt, nocc, nba, C, eo, ev, amplitudes=amplitudes))
    assert n1 > 6 and n2 > n1
    # the integrals are the same bits; tiles of 32 or 64 and their order by the shape alone
    for a, b in zip(one, cut):
        assert np.array_equal(a, b)


def test_sum_beyond_the_longest(api):
    """More than 16384 terms: FP64 in one launch."""
    rng = np.random.default_rng(9)
    m, n, k = 70, 65, 16385
    A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    C = np.zeros((m, n), order="F")
    before = api.kernel_launch_count()
    api.dgemm("T", "N", m, n, k, 1.0, np.asfortranarray(A.T), k, np.asfortranarray(B), k, 0.0, C, m)
    assert api.kernel_launch_count() - before == 1
    assert (np.abs(C - A @ B) <= 2 * k * U * (np.abs(A) @ np.abs(B))).all()


def test_cholesky_in_parts(api, monkeypatch):
    """A triangle that would need parts is left to FP64; the other updates are cut."""
    import torch
    rng = np.random.default_rng(11)
    n = 900
    X = rng.standard_normal((n, n))
    V = X @ X.T / n + np.eye(n)
    monkeypatch.setenv("RIMP2_RESIDUE_PARTS", "256,256")
    d = torch.from_numpy(V).cuda()
    torch.cuda.synchronize()
    api.cholesky_dev(n, d.data_ptr())
    L = d.cpu().numpy().T  # column-major
    assert (np.triu(L, 1) == 0).all()
    # backward error of a Cholesky factorisation, (n + 1) u |L| |L^T| (Higham, Theorem 10.3)
    assert (np.abs(L @ L.T - V) <= 2 * (n + 2) * U * (np.abs(L) @ np.abs(L).T)).all()
