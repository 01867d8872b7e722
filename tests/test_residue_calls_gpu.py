"""Calls that run on residue products: what they report, at which limits they
still run, and on which streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_TIMEOUT = 5


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
