"""Stream-ordered calls captured by the caller: a replay gives the call's own
results, also when the host memory of the captured call has been used again."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["energy fp64", "energy fp64 small", "energy fp64 amplitudes", "energy split",
                                  "ao2mo split", "ao2mo split sliced", "ao2mo fp64", "trsm"])
def test_captured_call(monkeypatch, call):
    import torch
    from rimp2_gpu_gb300 import api
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    rnd = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    zeros = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")  # noqa: E731
    if call.startswith("energy"):
        no, nv, nb = (2, 20, 60) if "small" in call else (8, 200, 600)
        C = rnd(no, nv, nb) * 0.05
        eo = torch.sort(rnd(no).abs() * -0.3 - 0.5)[0]
        ev = torch.sort(rnd(nv).abs() * 0.3 + 0.1)[0]
        E, T = zeros(no, no), zeros(1)
        t = zeros(nv, no, nv, no) if "amplitudes" in call else None
        out = [E, T] + ([t] if t is not None else [])
        prec = api.PREC_SPLIT if "split" in call else api.PREC_FP64

        def run(s):
            api.energy_dev(nv, no, nb, C.data_ptr(), eo.data_ptr(), ev.data_ptr(), E.data_ptr(), T.data_ptr(),
                           t.data_ptr() if t is not None else 0, precision=prec, stream=s)
    elif call.startswith("ao2mo"):
        nba, nbas, no, nv = 129, 64, 6, 58
        ao, cm, o = rnd(nbas, nbas, nba), rnd(nbas, nbas), zeros(no, nv, nba)
        out = [o]
        if "sliced" in call:
            monkeypatch.setenv("RIMP2_AO_FUSED", "0")

        def run(s):
            api.ao2mo_dev(nba, nbas, no, nv, ao.data_ptr(), cm.data_ptr(), o.data_ptr(), split="split" in call,
                          stream=s)
    else:
        n, m = 200, 50
        L = torch.tril(rnd(n, n)).T.contiguous()  # column-major lower
        L += 20 * torch.eye(n, dtype=torch.float64, device="cuda")
        B0, B, X = rnd(m, n), zeros(m, n), zeros(m, n)
        out = [X]

        def run(s):  # B is the call's workspace
            with torch.cuda.stream(st):
                B.copy_(B0)
            api.trsm_lower_dev(n, m, L.data_ptr(), B.data_ptr(), X.data_ptr(), stream=s)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    run(st.cuda_stream)
    torch.cuda.synchronize()
    plain = [x.clone() for x in out]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(st):
        graph.capture_begin(capture_error_mode="relaxed")
        run(st.cuda_stream)
        graph.capture_end()
    # other calls take the host memory that the captured one has given back
    c2, e2, v2, p2, t2 = rnd(120), rnd(1), rnd(3), zeros(1), zeros(1)
    torch.cuda.synchronize()
    for k in range(1, 40):
        api.energy_dev(3, 1, k, c2.data_ptr(), e2.data_ptr(), v2.data_ptr(), p2.data_ptr(), t2.data_ptr(),
                       precision=api.PREC_FP64, stream=st.cuda_stream)
    torch.cuda.synchronize()
    for x in out:
        x.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    first = [x.clone() for x in out]
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    api.sync_status()
    for x, f, p in zip(out, first, plain):
        assert torch.equal(x, f)
        # FP64 sums: a captured call takes the FP64 kernels, sums of up to 600 terms and their
        # energies in another order (2 x 600 x 2^-53 of the largest value, tenfold for the energy's sum)
        tol = 0.0 if "split" in call else 1.4e-12
        assert float((x - p).abs().max()) <= tol * float(p.abs().max())
