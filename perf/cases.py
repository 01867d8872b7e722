"""Performance cases: what a user of this package has it do, through its public entry points.

The sizes span what the tests, the benchmark and the tuning tables of this
repository use: fragments from a few occupied orbitals to nocc = 128, nvirt =
1024, NBA = 4096, uneven batches, AO bases of 128 to 600 functions with three
auxiliary functions each.  Odd and ragged sizes are the rule in real fragments,
so most cases have them.

Kinds of case:
  energy       pair and total energies of one fragment resident on the device
               (precision "split" or "fp64"): a driver that keeps Calpha there
  amplitudes   FP64 energies and the amplitude array t(a,i,b,j) from host
               arrays: small fragments whose amplitudes are used further
  energy_host  split energies from a pinned host Calpha, copied in each call
  batch        a planned batch of uneven fragments resident on the device
  eos          fragment energies with local orbitals, host arrays, both
               partitionings
  steps        the reference driver's Steps 5-8 on host arrays (four arrays of
               amplitudes and integrals come back)
  integrals    the drop-in integral subroutine on host arrays
  calpha       Calpha from AO integrals: transform, metric Cholesky, solve
  ao2mo        the AO to MO transform alone
"""
import math
import random

import numpy as np
import torch

from rimp2_gpu_gb300 import api

DEV = "cuda"


def listed():
    return [
        # the smallest calls: launches and latency count
        dict(name="energy_tiny", kind="energy", precision="split", nocc=8, nvirt=96, nba=256),
        dict(name="amplitudes_small", kind="amplitudes", nocc=6, nvirt=53, nba=187),
        # an ordinary ragged fragment, and the largest the benchmark quotes
        dict(name="energy_mid", kind="energy", precision="split", nocc=24, nvirt=301, nba=1203),
        dict(name="energy_large", kind="energy", precision="split", nocc=128, nvirt=1024, nba=4096),
        # reference-accuracy energies
        dict(name="energy_fp64", kind="energy", precision="fp64", nocc=16, nvirt=512, nba=2048),
        # fragments of a whole molecule in one plan
        dict(name="batch", kind="batch", nfrag=40, shapes=4),
        # the reference generator's production fragment from host memory
        dict(name="energy_host", kind="energy_host", nocc=59, nvirt=741, nba=2173),
        dict(name="eos", kind="eos", nvirt=741, nocc=59, nocc_eos=14, nvirt_eos=45, nba=2173),
        # the drop-in driver at half of that fragment's extents
        dict(name="steps5to8", kind="steps", nvirt=370, nocc=30, nocc_eos=7, nvirt_eos=22, nba=1086),
        dict(name="integrals", kind="integrals", nvirt=301, nocc_eos=9, nba=1203),
        # the front end from AO integrals
        dict(name="calpha_ao", kind="calpha", nbas=384),
        dict(name="ao2mo", kind="ao2mo", nbas=509),
    ]


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["energy", "energy_fp64", "amplitudes", "batch", "energy_host", "eos", "steps",
                       "integrals", "calpha", "ao2mo"])
    if kind == "energy":
        return dict(kind="energy", precision="split", nocc=span(4, 100), nvirt=span(48, 1000),
                    nba=span(128, 4000))
    if kind == "energy_fp64":
        return dict(kind="energy", precision="fp64", nocc=span(4, 18), nvirt=span(48, 500),
                    nba=span(128, 2400))
    if kind == "amplitudes":
        return dict(kind="amplitudes", nocc=span(2, 12), nvirt=span(20, 120), nba=span(60, 600))
    if kind == "batch":
        return dict(kind="batch", nfrag=span(6, 40), shapes=rng.randrange(10, 10000))
    if kind == "energy_host":
        return dict(kind="energy_host", nocc=span(12, 64), nvirt=span(100, 760), nba=span(400, 2200))
    if kind == "eos":
        nocc, nvirt = span(12, 59), span(100, 741)
        return dict(kind="eos", nvirt=nvirt, nocc=nocc, nocc_eos=rng.randint(3, max(3, nocc // 3)),
                    nvirt_eos=rng.randint(5, max(5, nvirt // 8)), nba=span(400, 2173))
    if kind == "steps":
        nocc, nvirt = span(6, 30), span(40, 370)
        return dict(kind="steps", nvirt=nvirt, nocc=nocc, nocc_eos=rng.randint(2, max(2, nocc // 3)),
                    nvirt_eos=rng.randint(5, max(5, nvirt // 10)), nba=span(150, 1086))
    if kind == "integrals":
        return dict(kind="integrals", nvirt=span(40, 400), nocc_eos=rng.randint(2, 10),
                    nba=span(150, 1500))
    if kind == "calpha":
        return dict(kind="calpha", nbas=span(128, 440))
    return dict(kind="ao2mo", nbas=span(128, 600))


def batch_shapes(case):
    """Uneven fragments: nocc U[8,64], nvirt U[64,512], NBA U[256,2048]."""
    r = random.Random(case["shapes"])
    return [(r.randint(8, 64), r.randint(64, 512), r.randint(256, 2048)) for _ in range(case["nfrag"])]


def ao_sizes(case):
    nbas = case["nbas"]
    nocc = max(1, nbas // 10)
    return nbas, 3 * nbas, nocc, nbas - nocc


# ---- inputs ---------------------------------------------------------------------


def generator(seed, k=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + k)


def fragment(seed, nocc, nvirt, nba, k=0):
    """Calpha(NBA, nvirt, nocc), alpha fastest, decaying with alpha; sorted orbital energies."""
    g = generator(seed, k)
    c = torch.randn(nocc, nvirt, nba, dtype=torch.float64, device=DEV, generator=g)
    c *= 0.03 / torch.sqrt(1.0 + torch.arange(nba, dtype=torch.float64, device=DEV) / 64)
    eo = torch.rand(nocc, dtype=torch.float64, device=DEV, generator=g) * 1.2 - 1.5
    ev = torch.rand(nvirt, dtype=torch.float64, device=DEV, generator=g) * 2.9 + 0.1
    return c, eo.sort().values, ev.sort().values


def orthonormal(seed, k, m, n):
    """n orthonormal columns of length m (local orbitals in the canonical basis)."""
    r = np.random.Generator(np.random.Philox(key=[int(seed), k])).standard_normal((m, m))
    q, t = np.linalg.qr(r)
    return np.asfortranarray((q * np.sign(np.diag(t)))[:, :n])


def ao_integrals(seed, nbas, nba):
    """(alpha | mu nu), symmetric in mu and nu, decaying with |mu - nu|; the metric; MO columns."""
    g = generator(seed, 7)
    ao = torch.randn(nbas, nbas, nba, dtype=torch.float64, device=DEV, generator=g)
    i = torch.arange(nbas, device=DEV)
    ao *= torch.exp(-(i[:, None] - i[None, :]).abs().double() / 32)[:, :, None]
    for m in range(1, nbas):
        ao[m, :m] = ao[:m, m]
    a = torch.randn(nba, nba, dtype=torch.float64, device=DEV, generator=g)
    v = a @ a.T / nba
    v = (v + v.T) / 2 + 0.1 * torch.eye(nba, dtype=torch.float64, device=DEV)
    return ao, v, orthonormal(seed, 5, nbas, nbas)


def host(t, pinned):
    """A Fortran-ordered numpy array of the tensor's values: (k, j, i) becomes (i, j, k)."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned)
    h.copy_(t)
    return h.numpy().T


def local_orbitals(case, seed):
    no, nv = case["nocc"], case["nvirt"]
    return (orthonormal(seed, 1, no, case["nocc_eos"]), orthonormal(seed, 2, nv, nv),
            orthonormal(seed, 3, no, no), orthonormal(seed, 4, nv, case["nvirt_eos"]))


class DeviceFragments:
    """Fragments resident on the device, their pair energies and totals back to back."""

    def __init__(self, seed, sizes):
        self.sizes = sizes
        self.inputs = [fragment(seed, *sh, k=k) for k, sh in enumerate(sizes)]
        self.pairs = torch.zeros(sum(sh[0] ** 2 for sh in sizes), dtype=torch.float64, device=DEV)
        self.totals = torch.zeros(len(sizes), dtype=torch.float64, device=DEV)

    def pointers(self):
        at = 0
        for k, (sh, x) in enumerate(zip(self.sizes, self.inputs)):
            yield [*(t.data_ptr() for t in x), self.pairs[at:].data_ptr(), self.totals[k:].data_ptr()]
            at += sh[0] ** 2


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, stream=torch.cuda.Stream())
    if kind == "energy":
        s["f"] = DeviceFragments(seed, [(case["nocc"], case["nvirt"], case["nba"])])
        s["pointers"] = next(s["f"].pointers())
    elif kind == "batch":
        f = s["f"] = DeviceFragments(seed, batch_shapes(case))
        torch.cuda.current_stream().synchronize()
        s["plan"] = api.BatchPlan([(*sh, *p) for sh, p in zip(f.sizes, f.pointers())], graph=True,
                                  stream=s["stream"].cuda_stream)
    elif kind in ("energy_host", "eos", "amplitudes", "steps"):
        c, eo, ev = fragment(seed, case["nocc"], case["nvirt"], case["nba"])
        # large Calphas are kept in pinned memory, the drop-in driver's arrays are plain ones
        s["c"] = host(c, kind in ("energy_host", "eos"))
        s["eo"], s["ev"] = eo.cpu().numpy(), ev.cpu().numpy()
        if kind in ("eos", "steps"):
            s["u"] = local_orbitals(case, seed)
    elif kind == "integrals":
        c, _, _ = fragment(seed, case["nocc_eos"], case["nvirt"], case["nba"])
        s["c"] = host(c, False)
        n = (case["nvirt"], case["nocc_eos"])
        s["out"] = np.zeros(n + n, order="F")
    else:
        nbas, nba, nocc, nvirt = ao_sizes(case)
        s["ao"], s["v"], cmo = ao_integrals(seed, nbas, nba)
        s["cmo"] = torch.from_numpy(cmo.T.copy()).to(DEV)
        s["out"] = torch.zeros(nocc, nvirt, nba, dtype=torch.float64, device=DEV)
    s["stream"].wait_stream(torch.cuda.current_stream())
    return s


# ---- one pass -------------------------------------------------------------------


def run(s):
    c, kind, sp = s["case"], s["case"]["kind"], s["stream"].cuda_stream
    if kind == "energy":
        prec = api.PREC_SPLIT if c["precision"] == "split" else api.PREC_FP64
        api.energy_dev(c["nvirt"], c["nocc"], c["nba"], *s["pointers"], precision=prec, stream=sp)
        return s["f"].pairs, s["f"].totals
    if kind == "batch":
        s["plan"].execute(stream=sp)
        return s["f"].pairs, s["f"].totals
    if kind == "amplitudes":
        return api.energy(c["nvirt"], c["nocc"], c["nba"], s["c"], s["eo"], s["ev"], amplitudes=True)
    if kind == "energy_host":
        return api.energy(c["nvirt"], c["nocc"], c["nba"], s["c"], s["eo"], s["ev"],
                          precision=api.PREC_SPLIT)
    if kind == "eos":
        return api.energy_eos(c["nvirt"], c["nocc"], c["nocc_eos"], c["nvirt_eos"], c["nba"], s["c"],
                              s["eo"], s["ev"], *s["u"], precision=api.PREC_SPLIT)
    if kind == "steps":
        return api.steps5to8(c["nvirt"], c["nocc"], c["nocc_eos"], c["nvirt_eos"], c["nba"], s["c"],
                             s["eo"], s["ev"], *s["u"])
    if kind == "integrals":
        api.calc_gocc(c["nvirt"], c["nocc_eos"], c["nba"], s["c"], s["out"])
        return s["out"]
    nbas, nba, nocc, nvirt = ao_sizes(c)
    if kind == "calpha":
        api.calpha_from_ao_split_dev(nba, nbas, nocc, nvirt, s["ao"].data_ptr(), s["v"].data_ptr(),
                                     s["cmo"].data_ptr(), s["out"].data_ptr(), stream=sp)
    else:
        api.ao2mo_dev(nba, nbas, nocc, nvirt, s["ao"].data_ptr(), s["cmo"].data_ptr(),
                      s["out"].data_ptr(), split=True, stream=sp)
    return s["out"]


# ---- what a pass cannot do without ------------------------------------------------


def energy_work(nocc, nvirt, nba):
    n = nocc * nvirt  # g is symmetric: n (n + 1) / 2 elements
    return 8.0 * (nba * n + nocc + nvirt + nocc * nocc), 1.0 * nba * n * (n + 1)


def work(case):
    kind = case["kind"]
    if kind in ("energy", "energy_host", "amplitudes"):
        b, f = energy_work(case["nocc"], case["nvirt"], case["nba"])
        if kind == "amplitudes":
            b += 8.0 * (case["nocc"] * case["nvirt"]) ** 2
        return dict(bytes=b, flops=f)
    if kind == "batch":
        w = [energy_work(*sh) for sh in batch_shapes(case)]
        return dict(bytes=sum(x[0] for x in w), flops=sum(x[1] for x in w))
    if kind == "integrals":
        n, k = case["nvirt"] * case["nocc_eos"], case["nba"]
        return dict(bytes=8.0 * (n * k + n * n), flops=1.0 * k * n * (n + 1))
    if kind in ("eos", "steps"):
        no, nv, nb = case["nocc"], case["nvirt"], case["nba"]
        ne, ve = case["nocc_eos"], case["nvirt_eos"]
        b, f = energy_work(no, nv, nb)
        b += 8.0 * (no * ne + nv * nv + no * no + nv * ve)
        if kind == "eos":  # g, the two projected integrals, the projections
            return dict(bytes=b, flops=3 * f + 4.0 * nb * nv * no * (ne + ve))
        b += 8.0 * (2 * (nv * ne) ** 2 + 2 * (ve * no) ** 2)
        # amplitudes to local orbitals, the smaller index first
        f += 2.0 * nv * nv * no * ne * (no + ne) + 4.0 * ne * ne * nv ** 3
        f += 2.0 * no * no * nv * ve * (nv + ve) + 4.0 * ve * ve * no ** 3
        # Calpha to local orbitals and the two integral arrays
        f += 2.0 * nb * nv * ne * (no + nv) + 1.0 * nb * (nv * ne) ** 2
        f += 2.0 * nb * no * ve * (nv + no) + 1.0 * nb * (ve * no) ** 2
        return dict(bytes=b, flops=f)
    nbas, nba, nocc, nvirt = ao_sizes(case)
    b = 8.0 * (nba * nbas * nbas + nbas * nbas + nba * nocc * nvirt)
    f = 2.0 * nba * nbas * nocc * (nbas + nvirt)
    if kind == "calpha":
        b += 8.0 * nba * nba
        f += nba ** 3 / 3 + 1.0 * nba * nba * nocc * nvirt
    return dict(bytes=b, flops=f)


# ---- the results in 64 bits, by torch ---------------------------------------------


def mm(a, b):
    """a.T @ b over the leading (alpha) extent, in blocks of it: a short rounding chain."""
    out = None
    for k in range(0, a.shape[0], 256):
        p = a[k:k + 256].T @ b[k:k + 256]
        out = p if out is None else out.add_(p)
    return out


def exact_energy(c, eo, ev, ct=None):
    """Pair energies; ct: the projected Calpha of the integral side (total only)."""
    no, nv, nb = c.shape
    cols = [c[i].T.contiguous() for i in range(no)]
    tcols = cols if ct is None else [ct[i].T.contiguous() for i in range(no)]
    e = torch.zeros(no, no, dtype=torch.float64, device=c.device)
    vv = ev[:, None] + ev[None, :]
    step = max(1, min(no, 16))
    for i in range(no):
        for j0 in range(i, no, step):
            js = range(j0, min(no, j0 + step))
            g = mm(cols[i], torch.cat([cols[j] for j in js], 1)).view(nv, len(js), nv).permute(1, 0, 2)
            h = g if ct is None else (mm(tcols[i], torch.cat([tcols[j] for j in js], 1))
                                      .view(nv, len(js), nv).permute(1, 0, 2))
            d = eo[i] + eo[j0:j0 + len(js)][:, None, None] - vv[None]
            v = (g / d * (2 * h - h.transpose(1, 2))).sum((1, 2))
            e[i, j0:j0 + len(js)] = v
            e[j0:j0 + len(js), i] = v
    return e


def to_local(x, uo, uv):
    """x(i, a, j, b) in local orbitals, as (aL, iL, bL, jL)."""
    y = torch.einsum("iajb,ik->kajb", x, uo)
    y = torch.einsum("kajb,jl->kalb", y, uo)
    y = torch.einsum("kalb,ac->kclb", y, uv)
    return torch.einsum("kclb,bd->ckdl", y, uv)


def exact(case, seed):
    kind = case["kind"]
    if (3 if kind == "eos" else 1) * work(case)["flops"] > 1.2e13:
        return None  # over about 20 s in 64 bits
    if kind in ("energy", "energy_host"):
        e = exact_energy(*fragment(seed, case["nocc"], case["nvirt"], case["nba"]))
        return (e.view(-1), e.sum().view(1)) if kind == "energy" else (e.cpu().numpy(), float(e.sum()))
    if kind == "batch":
        es = [exact_energy(*fragment(seed, *sh, k=k)) for k, sh in enumerate(batch_shapes(case))]
        return torch.cat([e.view(-1) for e in es]), torch.stack([e.sum() for e in es])
    if kind in ("amplitudes", "eos", "steps"):
        c, eo, ev = fragment(seed, case["nocc"], case["nvirt"], case["nba"])
        no, nv, nb = c.shape
        if kind == "eos":
            uoe, uv, uo, uve = (torch.from_numpy(u).to(DEV) for u in local_orbitals(case, seed))
            e = []
            for a, b in ((uoe, uv), (uo, uve)):
                ct = torch.einsum("iax,ik,jk->jax", c, a, a)
                e.append(float(exact_energy(c, eo, ev, torch.einsum("iax,ak,bk->ibx", ct, b, b)).sum()))
            return tuple(e)
        flat = c.reshape(no * nv, nb).T.contiguous()
        g = mm(flat, flat).view(no, nv, no, nv)
        t = (eo[:, None, None, None] - ev[None, :, None, None] + eo[None, None, :, None] -
             ev[None, None, None, :])
        t = torch.div(g, t)
        if kind == "amplitudes":
            e = (t * (2 * g - g.transpose(1, 3))).sum((1, 3))
            return e.cpu().numpy(), float(e.sum()), t.permute(1, 0, 3, 2).contiguous().cpu().numpy()
        del g
        uoe, uv, uo, uve = (torch.from_numpy(u).to(DEV) for u in local_orbitals(case, seed))
        out = [to_local(t, uoe, uv), to_local(t, uo, uve)]
        for a, b in ((uoe, uv), (uo, uve)):
            ct = torch.einsum("iax,ik->kax", c, a)
            ct = torch.einsum("kax,ab->xbk", ct, b).contiguous()
            f = ct.view(nb, -1)
            out.append(mm(f, f).view(ct.shape[1:] + ct.shape[1:]))
        return tuple(x.cpu().numpy() for x in out)
    if kind == "integrals":
        c, _, _ = fragment(seed, case["nocc_eos"], case["nvirt"], case["nba"])
        f = c.permute(2, 1, 0).reshape(case["nba"], -1).contiguous()
        n = (case["nvirt"], case["nocc_eos"])
        return mm(f, f).view(n + n).cpu().numpy()
    nbas, nba, nocc, nvirt = ao_sizes(case)
    ao, v, cmo = ao_integrals(seed, nbas, nba)
    cmo = torch.from_numpy(cmo).to(DEV)
    half = torch.einsum("mnx,ni->imx", ao, cmo[:, :nocc])
    out = torch.einsum("imx,ma->iax", half, cmo[:, nocc:]).contiguous()
    if kind == "calpha":
        low = torch.linalg.cholesky(v)
        out = torch.linalg.solve_triangular(low, out.view(-1, nba).T, upper=False).T
        out = out.reshape(nocc, nvirt, nba).contiguous()
    return out
