"""FP64 contractions through residues on the FP16 tensor cores (mod_gemm.cu):
the general product over its forms and tile edges, against exactly rounded
sums, and the elements and tiles that it leaves to FP64 arithmetic."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.fixture(scope="module")
def api():
    from rimp2_gpu_gb300 import api
    return api


def exact_dot(a, b):
    """sum a b rounded once: error-free products (Dekker), math.fsum."""
    c = 134217729.0
    p = a * b
    ah = a * c - (a * c - a)
    bh = b * c - (b * c - b)
    e = ((ah * bh - p) + ah * (b - bh) + (a - ah) * bh) + (a - ah) * (b - bh)
    return math.fsum(np.concatenate([p, e]))


def product(api, ta, tb, A, B, alpha, beta, C, pad=0):
    """C := alpha A B + beta C through the library; the number of launches."""
    m, k = A.shape
    n = B.shape[1]

    def store(x, t):
        x = x.T if t == "T" else x
        s = np.zeros((x.shape[0] + pad, x.shape[1]), order="F")
        s[:x.shape[0]] = x
        return s
    As, Bs = store(A, ta), store(B, tb)
    before = api.kernel_launch_count()
    api.dgemm(ta, tb, m, n, k, alpha, As, As.shape[0], Bs, Bs.shape[0], beta, C, m)
    return api.kernel_launch_count() - before


@pytest.mark.parametrize("residues,ta,tb,m,n,k,alpha,beta,pad", [
    (True, "N", "N", 257, 255, 1025, 1.0, 0.0, 0),   # one value past a tile, a sum and a K chunk
    (True, "T", "N", 256, 512, 1024, -1.0, 1.0, 0),  # whole tiles and sums
    (True, "N", "T", 511, 321, 639, 0.5, -2.0, 3),   # ragged, leading dimensions beyond the extents
    (True, "T", "T", 385, 700, 2049, 1.0, 0.0, 1),   # three sums, odd leading dimensions
    (True, "T", "N", 4100, 4097, 31, 1.0, 0.0, 0),   # a short sum
    (False, "T", "N", 4100, 4097, 8, 1.0, 0.0, 0),   # DMMA on 64 x 64 tiles
    (False, "N", "N", 70000, 3, 61, 1.0, 0.0, 0),    # on 128 x 8 tiles
    (False, "N", "T", 50001, 13, 29, 2.0, 1.0, 2),   # on 16 x 16 tiles, odd leading dimensions
    (False, "T", "N", 7, 40003, 30, 1.0, 0.0, 0),    # few rows: transposed
    (False, "N", "N", 100, 77, 45, 1.0, -1.0, 0),    # on 16 x 16 tiles
    (False, "T", "T", 380, 384, 12, 1.0, 0.0, 0),    # on 32 x 32 tiles
    (False, "N", "N", 33, 1, 3, 1.0, 0.0, 0),
])
def test_product_forms(api, residues, ta, tb, m, n, k, alpha, beta, pad):
    r = np.random.Generator(np.random.Philox(key=[k, m]))
    A, B = r.standard_normal((m, k)), r.standard_normal((k, n))
    C0 = np.asfortranarray(r.standard_normal((m, n)))
    C = C0.copy(order="F")
    assert (product(api, ta, tb, A, B, alpha, beta, C, pad) > 1) == residues
    I = np.concatenate([r.integers(0, m, 300), [0, m - 1, m - 1, 0]])
    J = np.concatenate([r.integers(0, n, 300), [0, n - 1, 0, n - 1]])
    for i, j in zip(I, J):
        d = alpha * exact_dot(A[i], B[:, j])
        ref = d + beta * C0[i, j]
        # rounding to 62-bit integers: sqrt(K)/2 u sum|a||b| at most (an element
        # under 2^-8 of the norms' product is summed in FP64); FP64 sums: K u
        # sum|a||b|; then alpha, beta
        tol = abs(alpha) * (math.sqrt(k) / 2 + 2 if residues else k) * U * \
            np.abs(A[i] * B[:, j]).sum() + 3 * U * (abs(d) + abs(beta * C0[i, j]))
        assert abs(C[i, j] - ref) <= tol


@pytest.mark.parametrize("n", range(1, 9))
@pytest.mark.parametrize("ta,m,k,alpha,beta", [
    ("N", 160001, 33, 1.0, 0.0),   # rows along the fast direction, one past a block
    ("N", 156000, 65, -1.0, 1.0),  # two chunks of the columns' operand
    ("T", 160001, 30, 1.0, 0.0),   # sums along it
    ("T", 158000, 64, 0.5, -2.0),
])
def test_thin_products(api, ta, m, n, k, alpha, beta):
    """At most eight columns: FP64's own bound, K u sum|a||b|, then alpha and beta."""
    r = np.random.Generator(np.random.Philox(key=[n, k]))
    A, B = r.standard_normal((m, k)), r.standard_normal((k, n))
    C0 = np.asfortranarray(r.standard_normal((m, n)))
    C = C0.copy(order="F")
    assert product(api, ta, "N", A, B, alpha, beta, C) == 1
    ref, mag = A @ B, np.abs(A) @ np.abs(B)  # numpy's own error: the same bound
    tol = 2 * abs(alpha) * k * U * mag + 3 * U * (np.abs(alpha * ref) + np.abs(beta * C0))
    assert (np.abs(C - (alpha * ref + beta * C0)) <= tol).all()


def test_product_exact_and_special_values(api):
    r = np.random.Generator(np.random.Philox(key=[5, 9]))
    m = n = k = 640
    # integers, sums that cancel, a permutation: results that FP64 holds come out exact
    A = r.integers(-1000, 1000, (m, k)).astype(float)
    B = r.integers(-1000, 1000, (k, n)).astype(float)
    A[5, 0], A[5, 1], B[0, 7], B[1, 7] = 2.0 ** 45, 2.0 ** 45, 1.0, -1.0
    C = np.zeros((m, n), order="F")
    assert product(api, "N", "N", A, B, 1.0, 0.0, C) > 1
    ref = A.astype(np.int64) @ B.astype(np.int64)
    held = ref.astype(float).astype(np.int64) == ref  # row 5 has sums beyond 53 bits
    assert held[6:].all() and not held.all()
    assert np.array_equal(C[held], ref[held].astype(float))
    assert (np.abs(C.astype(np.int64) - ref) <= np.spacing(np.abs(C))).all()
    perm = np.eye(k)[r.permutation(k)]
    X = r.standard_normal((m, k)) * np.exp(4 * r.standard_normal((m, k)))
    product(api, "N", "N", X, perm, 1.0, 0.0, C)
    assert np.array_equal(C, X @ perm)
    # infinities, NaN, zeros, extreme magnitudes: as FP64 sums them
    X = r.standard_normal((m, k))
    X[3, 5], X[70, 2], X[100], X[400, 9] = np.nan, np.inf, 0.0, -np.inf
    X[200] *= 1e-200
    X[201] *= 1e300
    X[:, 7] = 1e-310
    Y = r.standard_normal((k, n))
    Y[11, 13] = np.inf
    product(api, "N", "N", X, Y, 1.0, 0.0, C)
    with np.errstate(all="ignore"):
        ref, mag = X @ Y, np.abs(X) @ np.abs(Y)
    assert np.array_equal(np.isnan(C), np.isnan(ref))
    assert np.array_equal(np.isinf(C), np.isinf(ref))
    f = np.isfinite(ref)
    assert np.array_equal(np.sign(C[~f & ~np.isnan(ref)]), np.sign(ref[~f & ~np.isnan(ref)]))
    assert (np.abs(C - ref)[f] <= 2 * k * U * mag[f]).all()


@pytest.mark.parametrize("spread", [2.0, 6.0])
def test_rows_of_wide_range(api, spread):
    """Log-normal values: a part, or nearly all, of the elements is summed in FP64."""
    r = np.random.Generator(np.random.Philox(key=[17, int(spread)]))
    m, n, k = 500, 520, 700
    A = r.standard_normal((m, k)) * np.exp(spread * r.standard_normal((m, k)))
    B = r.standard_normal((k, n)) * np.exp(spread * r.standard_normal((k, n)))
    C = np.zeros((m, n), order="F")
    assert product(api, "T", "N", A, B, 1.0, 0.0, C) > 1
    for i, j in zip(r.integers(0, m, 400), r.integers(0, n, 400)):
        ref = exact_dot(A[i], B[:, j])
        assert abs(C[i, j] - ref) <= k * U * np.abs(A[i] * B[:, j]).sum()  # FP64's own bound


def test_subroutine_forms(api):
    """Every stride pattern that the drop-in subroutines hand to the product,
    at sizes that take the residue form, against numpy's FP64."""
    r = np.random.Generator(np.random.Philox(key=[3, 8]))
    nv, no, ne, ve, nb = 201, 19, 9, 37, 333
    F = np.asfortranarray
    Ca = F(r.standard_normal((nb, nv, no)) * 0.03)
    eo, ev = np.sort(-r.random(no) - 0.3), np.sort(r.random(nv) + 0.1)
    UoE, UvT = F(r.standard_normal((no, ne))), F(r.standard_normal((nv, nv)))
    UoT, UvE = F(r.standard_normal((no, no))), F(r.standard_normal((nv, ve)))
    tocc, tvirt, gocc, gvirt = api.steps5to8(nv, no, ne, ve, nb, Ca, eo, ev, UoE, UvT, UoT, UvE)
    g = np.tensordot(Ca, Ca, (0, 0))  # a i b j
    t = g / (eo[None, :, None, None] + eo - ev[:, None, None, None] - ev[None, None, :, None])

    def local(x, uo, uv):
        x = np.tensordot(uv, x, (0, 0))
        x = np.moveaxis(np.tensordot(uo, x, (0, 1)), 0, 1)
        x = np.moveaxis(np.tensordot(uv, x, (0, 2)), 0, 2)
        return np.moveaxis(np.tensordot(uo, x, (0, 3)), 0, 3)
    for got, x, uo, uv, chain in ((tocc, t, UoE, UvT, nb + 2 * no + 2 * nv),
                                  (tvirt, t, UoT, UvE, nb + 2 * no + 2 * nv),
                                  (gocc, g, UoE, UvT, nb + 2 * no + 2 * nv),
                                  (gvirt, g, UoT, UvE, nb + 2 * no + 2 * nv)):
        ref, mag = local(x, uo, uv), None
        gm = np.tensordot(np.abs(Ca), np.abs(Ca), (0, 0))
        mag = local(gm / np.abs(g / x), np.abs(uo), np.abs(uv))
        # the classical bound of the chain of sums, for either side
        assert (np.abs(got - ref) <= 2 * chain * U * mag).all()


def fp64_energies(nocc, nvirt, nba, Ca, eo, ev):
    """The DMMA kernels (the allocation-free entry point keeps to them)."""
    import torch
    from rimp2_gpu_gb300._lib import call
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (Ca.ravel(order="F"), eo, ev)]
    E = torch.zeros(nocc * nocc, dtype=torch.float64, device="cuda")
    T = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    call("rimp2_energy_fp64_noalloc_dev", nvirt, nocc, nba, *(x.data_ptr() for x in d), E.data_ptr(),
         T.data_ptr(), None)
    torch.cuda.synchronize()
    return E.cpu().numpy().reshape(nocc, nocc, order="F"), float(T[0])


@pytest.mark.parametrize("nocc,nvirt,nba,spread", [
    (1, 515, 900, 0.0),     # one pair, i = j
    (7, 129, 700, 0.0),     # one virtual past two tiles, odd row padding
    (16, 65, 1025, 0.0),    # two sums
    (5, 256, 2048, 0.0),    # whole tiles
    (64, 256, 70, 0.0),     # two blocks of occupied orbitals
    (6, 190, 640, 2.5),     # some elements summed in FP64
    (4, 250, 640, 7.0),     # most tiles left to FP64
])
def test_fp64_energies(api, nocc, nvirt, nba, spread):
    r = np.random.Generator(np.random.Philox(key=[nocc, nvirt]))
    Ca = r.standard_normal((nba, nvirt, nocc)) * np.exp(spread * r.standard_normal((nba, nvirt, nocc)))
    Ca = np.asfortranarray(Ca * 0.03 / np.abs(Ca).max())
    eo, ev = np.sort(-r.random(nocc) - 0.3), np.sort(r.random(nvirt) + 0.1)
    Er, Tr = fp64_energies(nocc, nvirt, nba, Ca, eo, ev)
    before = api.kernel_launch_count()
    E, T = api.energy(nvirt, nocc, nba, Ca, eo, ev)
    assert api.kernel_launch_count() - before > 7, "expected the residue form"
    # both sides sum FP64 terms of g and 1/D that are a few ulp off; the terms
    # of a pair cancel by no more than their number: sums of magnitudes over
    # |e_ij| stay below ~10 here, the sums' rounding below sqrt(nvirt) u each
    assert (np.abs(E - Er) <= 1e-13 * np.abs(Er)).all()
    assert abs(T - Tr) <= 1e-13 * abs(Tr)


@pytest.mark.parametrize("nocc,nvirt,nba", [(6, 131, 640), (9, 64, 900)])
def test_fp64_amplitudes(api, nocc, nvirt, nba):
    r = np.random.Generator(np.random.Philox(key=[nvirt, nba]))
    Ca = np.asfortranarray(r.standard_normal((nba, nvirt, nocc)) * 0.03)
    eo, ev = np.sort(-r.random(nocc) - 0.3), np.sort(r.random(nvirt) + 0.1)
    before = api.kernel_launch_count()
    E, T, t = api.energy(nvirt, nocc, nba, Ca, eo, ev, amplitudes=True)
    assert api.kernel_launch_count() - before > 7, "expected the residue form"
    g = np.tensordot(Ca, Ca, (0, 0))
    mag = np.tensordot(np.abs(Ca), np.abs(Ca), (0, 0))
    d = eo[None, :, None, None] + eo - ev[:, None, None, None] - ev[None, None, :, None]
    assert (np.abs(t - g / d) <= (nba + 4) * U * np.abs(mag / d)).all()
    e = (t * (2 * g - g.transpose(2, 1, 0, 3))).sum((0, 2))
    assert np.abs(E - e).max() <= 1e-12 * np.abs(e).max()


@pytest.mark.parametrize("n,k", [(300, 700), (321, 1500)])
def test_symmetric_product(api, n, k):
    """A set of vectors with itself: both triangles, and the elements left to FP64."""
    r = np.random.Generator(np.random.Philox(key=[n, k]))
    X = r.standard_normal((k, n, 2))
    X[:, 5, 1] = 0.0
    X[:, 100, 0] *= np.exp(6 * r.standard_normal(k))
    X[3, 200, 1] = np.inf
    X = np.asfortranarray(X)
    G = np.zeros((n, 2, n, 2), order="F")
    before = api.kernel_launch_count()
    api.calc_gocc(n, 2, k, X, G)
    assert api.kernel_launch_count() - before > 1
    F, G = X.reshape(k, 2 * n, order="F"), G.reshape(2 * n, 2 * n, order="F")
    assert np.array_equal(G, G.T, equal_nan=True)
    with np.errstate(all="ignore"):
        ref, mag = F.T @ F, np.abs(F).T @ np.abs(F)
    ok = np.isfinite(ref)
    assert np.array_equal(ok, np.isfinite(G))
    assert (np.abs(G - ref)[ok] <= 2 * k * U * mag[ok]).all()
    for i, j in [(0, 1), (1, 0), (2 * n - 1, 3), (3, 2 * n - 1), (70, 100), (64, 63), (256, 255)]:
        d = exact_dot(F[:, i], F[:, j])
        assert abs(G[i, j] - d) <= (math.sqrt(k) / 2 + 1) * U * np.abs(F[:, i] * F[:, j]).sum()
