"""Calls that run on residue products: what they report, at which limits they
still run, and on which streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_NOMEM, ERR_TIMEOUT = 3, 5


@pytest.fixture(scope="module")
def api():
    from rimp2_gpu_gb300 import api
    return api


def metric(n, seed=3):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, n))
    return np.asfortranarray(X @ X.T / n + np.eye(n))


@pytest.mark.parametrize("call", ["cholesky_dev", "calpha_from_ao", "calpha_from_ao metric", "dgemm"])
def test_product_that_gave_up(api, monkeypatch, call):
    """A product whose kernel gave up on a wait (its error word is set here by the
    host) fails the synchronising call that used it, and no later one."""
    import torch
    from rimp2_gpu_gb300._lib import Rimp2Error
    rng = np.random.default_rng(1)

    def run():
        if call == "cholesky_dev":
            V = torch.from_numpy(metric(600)).cuda()
            torch.cuda.synchronize()
            api.cholesky_dev(600, V.data_ptr())
        elif call == "dgemm":
            A = np.asfortranarray(rng.standard_normal((300, 300)))
            api.dgemm("N", "N", 300, 300, 300, 1.0, A, 300, A, 300, 0.0, np.zeros((300, 300), order="F"), 300)
        else:  # products in the transform and the solve only, or in the metric too
            nba = 600 if "metric" in call else 200
            nbas, nocc, nvirt = 100, 20, 80
            ao = np.asfortranarray(rng.standard_normal((nba, nbas, nbas)))
            api.calpha_from_ao(nba, nbas, nocc, nvirt, ao, metric(nba),
                               np.asfortranarray(rng.standard_normal((nbas, nbas))))

    run()
    monkeypatch.setenv("RIMP2_FAULT_INJECT", "wait")
    with pytest.raises(Rimp2Error) as e:
        run()
    assert e.value.status == ERR_TIMEOUT
    monkeypatch.delenv("RIMP2_FAULT_INJECT")
    api.sync_status()
    run()


def fragment(seed, no=6, nv=90, nb=400):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda")
    C = torch.randn(no, nv, nb, generator=g, **f64) * 0.05
    eo = torch.sort(torch.rand(no, generator=g, **f64) - 1.5)[0]
    ev = torch.sort(torch.rand(nv, generator=g, **f64) + 0.1)[0]
    return (nv, no, nb), (C, eo, ev, torch.zeros(no, no, **f64), torch.zeros(1, **f64))


def enqueue(api, frag, stream):
    sizes, t = frag
    api.energy_dev(*sizes, *(x.data_ptr() for x in t), precision=api.PREC_FP64, stream=stream.cuda_stream)


@pytest.mark.parametrize("threads", [1, 3])
def test_contractions_on_several_streams(api, threads):
    """Energies in turn on three streams, from one thread and from a thread for
    each stream: the bits of every call alone, and no error afterwards."""
    import threading

    import torch
    streams = [torch.cuda.Stream() for _ in range(3)]
    frags = [[fragment(10 * k + r) for r in range(4)] for k in range(3)]
    want = []
    for k in range(3):
        for f in frags[k]:
            torch.cuda.synchronize()
            before = api.kernel_launch_count()
            enqueue(api, f, streams[0])
            assert api.kernel_launch_count() - before > 6  # residue products
            torch.cuda.synchronize()
            want.append(f[1][3].clone())
            f[1][3].zero_()
    torch.cuda.synchronize()
    errors = []

    def work(ks):
        try:
            for _ in range(5):
                for r in range(4):
                    for k in ks:
                        enqueue(api, frags[k][r], streams[k])
        except Exception as e:  # shown by the assertion below
            errors.append(e)

    parts = [[0, 1, 2]] if threads == 1 else [[0], [1], [2]]
    ts = [threading.Thread(target=work, args=(p,)) for p in parts]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    api.sync_status()
    for w, f in zip(want, (f for k in range(3) for f in frags[k])):
        assert torch.equal(w, f[1][3])


def test_end_that_cannot_be_recorded(api, monkeypatch):
    """The call fails (the order of contractions would be lost otherwise), has
    waited for its kernels, and later calls run."""
    import torch
    from rimp2_gpu_gb300._lib import Rimp2Error
    s = torch.cuda.Stream()
    f = fragment(1)
    torch.cuda.synchronize()
    enqueue(api, f, s)
    torch.cuda.synchronize()
    want = f[1][3].clone()
    f[1][3].zero_()
    torch.cuda.synchronize()
    monkeypatch.setenv("RIMP2_FAULT_INJECT", "record")
    with pytest.raises(Rimp2Error):
        enqueue(api, f, s)
    assert s.query()
    monkeypatch.delenv("RIMP2_FAULT_INJECT")
    enqueue(api, f, s)
    torch.cuda.synchronize()
    api.sync_status()
    assert torch.equal(want, f[1][3])


def lost_allocations(api, monkeypatch, run, tol=4 * 600 * 2.0 ** -53, count=60):
    """run() with the first, the second, ... of its device allocations failing (of
    `count`, more than it makes): how many of them it did not get over."""
    from rimp2_gpu_gb300._lib import Rimp2Error
    want = run()
    lost = 0
    for n in range(1, count + 1):
        monkeypatch.setenv("RIMP2_FAULT_INJECT", f"alloc:{n}")
        try:
            got = run()
        except Rimp2Error as e:
            assert e.status == ERR_NOMEM
            lost += 1
            got = want
        monkeypatch.delenv("RIMP2_FAULT_INJECT")
        api.sync_status()
        for w, g in zip(want, got):
            # FP64 kernels instead of residues: four products in a row, sums of at most 600 terms
            assert np.abs(w - g).max() <= tol * np.abs(w).max()
    return lost


def local_orbitals(nv, no, ne, ve, nb):
    rng = np.random.default_rng(2)
    q = lambda n: np.asfortranarray(np.linalg.qr(rng.standard_normal((n, n)))[0])  # noqa: E731
    C = np.asfortranarray(rng.standard_normal((nb, nv, no)) * 0.05)
    eo, ev = np.sort(rng.random(no) - 1.5), np.sort(rng.random(nv) + 0.1)
    Uo, Uv = q(no), q(nv)
    return C, eo, ev, np.asfortranarray(Uo[:, :ne]), Uv, Uo, np.asfortranarray(Uv[:, :ve])


def test_steps5to8_short_of_memory(api, monkeypatch):
    """What the call cannot do without are its seven inputs, g/D and its first
    projection, and the last three arrays of Steps 6, 7 and 8 each.  Neither the
    products' workspaces nor what it keeps for Step 6 beside Step 5 may make it fail."""
    nv, no, ne, ve, nb = 100, 8, 3, 30, 300
    x = local_orbitals(nv, no, ne, ve, nb)
    run = lambda: api.steps5to8(nv, no, ne, ve, nb, *x)  # noqa: E731
    assert lost_allocations(api, monkeypatch, run) == 7 + 2 + 3 * 3


def test_energies_short_of_memory(api, monkeypatch):
    """One fragment in FP64 cannot do without its three inputs and its results."""
    nv, no, nb = 100, 8, 300
    x = local_orbitals(nv, no, 3, 30, nb)
    assert lost_allocations(api, monkeypatch, lambda: api.energy(nv, no, nb, *x[:3])) == 4


def test_local_energies_short_of_memory(api, monkeypatch):
    """Local orbitals in split form, one residual slice: the seven inputs, three
    results and checks, the two projectors of more than half rank, both halves of
    the two low-rank projections; not both partitionings' slices at once."""
    nv, no, ne, ve, nb = 300, 8, 3, 30, 300
    assert api.split_nslices(nv, no, nb) == 1
    x = local_orbitals(nv, no, ne, ve, nb)
    run = lambda: [np.array(api.energy_eos(nv, no, ne, ve, nb, *x, api.PREC_SPLIT))]  # noqa: E731
    assert lost_allocations(api, monkeypatch, run, tol=1e-7) == 7 + 3 + 2 + 4  # accuracy of the split form
