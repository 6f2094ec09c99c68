"""Performance cases of the triples engine: what its users have it do, through its public entry points.

Kinds of a case (``kind``):

* ``run``      one ``Context.run`` over a stretch of the tuple list of a system whose tensors are resident
               (the step of a driver that checkpoints, shards or samples the list), and its tuple energies;
* ``dropin``   a whole ``Atrip.run(Input)`` on host arrays: context, uploads, every tuple, E(T);
* ``batch``    one ``Batch.run`` over many small systems;
* ``noalloc``  the entry point for hosts that may not allocate, on the caller's own device arrays.

Inputs have the value distributions of the benchmark workloads (atrip_gb300/synth.py), drawn on the GPU.
"""
import ctypes
import math

import numpy as np
import torch

from atrip_gb300 import atrip, capi

REAL7 = ("epsi", "epsa", "Tai", "Tabij", "Vabij", "Vijka", "Vabci")
J2 = ("Jijka", "Jabci")


def _run(name, form, no, nv, count, first=0, j=False, slices=0, field="real", tuned=False):
    c = dict(kind="run", form=form, slices=slices, no=no, nv=nv, first=first, count=count, j=j, field=field, tuned=tuned)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call a host program makes: a unit-test sized molecule through the drop-in interface
        dict(name="dropin_no4_nv12", kind="dropin", no=4, nv=12, j=False),
        # a small molecule end to end from host memory, with the (cT) intermediates
        dict(name="dropin_no12_nv60_ct", kind="dropin", no=12, nv=60, j=True),
        # the parity workload: a whole list in FP64, the default form
        _run("fp64_no8_nv40", "fp64", 8, 40, 11440),
        # one chunk of a medium system's list in FP64 (what a checkpointing driver runs at a time)
        _run("fp64_no24_nv240", "fp64", 24, 240, 8000, first=1000000),
        # (cT), two W builds a tuple, at sizes that fit no tile
        _run("fp64_no37_nv151_ct", "fp64", 37, 151, 900, first=200000, j=True),
        # the headline workload in the form its tuner chooses, with that tuner's launch parameters
        _run("f16_no40_nv400", "split_f16", 40, 400, 9000, first=5000000, tuned=True),
        # the accurate split form as called without a tuner
        _run("bf16x3_no24_nv240", "split_bf16", 24, 240, 16000, first=1000000, slices=3),
        # many occupied orbitals, odd sizes, split form with default launch parameters
        _run("f16_no53_nv201", "split_f16", 53, 201, 3000, first=400000),
        # a set of small molecules in one call, FP64
        dict(name="batch_fp64", kind="batch", form="fp64",
             systems="4:67 5:52 6:70 7:44 8:61 9:38 10:57 11:49 12:66 13:33 14:58 15:41 16:47 17:36 19:54 20:30"),
        # a set of small molecules in one call, split form
        dict(name="batch_f16", kind="batch", form="split_f16",
             systems="4:117 5:82 6:150 7:64 8:131 9:58 10:97 11:109 12:126 13:73 14:88 15:61 16:77 17:56 19:94 20:70"),
        # complex orbitals
        _run("complex_no13_nv50", "fp64", 13, 50, 9000, first=3000, field="complex"),
        # a host with its own allocator, column-major arrays in place
        dict(name="noalloc_no24_nv120", kind="noalloc", no=24, nv=120, first=100000, count=2500),
    ]


def _stretch(rng, form, no, nv, work, j, slices=0, field="real", tuned=False):
    n = capi.n_tuples(nv)
    per = 12.0 * no ** 3 * (no + nv) * (2 if j else 1) * (4 if field == "complex" else 1)
    count = int(min(n, max(64, work / per)))
    return _run(None, form, no, nv, count, first=rng.randrange(n - count + 1), j=j, slices=slices, field=field, tuned=tuned)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "fp64", "fp64", "fp64", "f16", "f16", "bf16", "bf16", "batch", "complex", "noalloc"])
    if kind == "dropin":
        return dict(kind="dropin", no=_log(rng, 2, 12), nv=_log(rng, 8, 60), j=rng.random() < 0.4)
    if kind == "fp64":
        return _stretch(rng, "fp64", _log(rng, 6, 42), _log(rng, 36, 240), math.exp(rng.uniform(math.log(4e9), math.log(2.8e11))),
                        rng.random() < 0.3)
    if kind == "f16":
        return _stretch(rng, "split_f16", rng.randint(8, 56), _log(rng, 60, 300), math.exp(rng.uniform(math.log(1e11), math.log(2e12))),
                        rng.random() < 0.2, tuned=rng.random() < 0.5)
    if kind == "bf16":
        return _stretch(rng, "split_bf16", rng.randint(8, 40), _log(rng, 60, 260), math.exp(rng.uniform(math.log(5e10), math.log(6e11))),
                        rng.random() < 0.2, slices=rng.choice([2, 3, 3, 4]), tuned=rng.random() < 0.3)
    if kind == "batch":
        fp64 = rng.random() < 0.5
        sizes, left = [], 5e11 if fp64 else 5e12
        for _ in range(rng.randint(4, 16)):
            no, nv = rng.randint(4, 20), rng.randint(30, 60 if fp64 else 120)
            left -= _work(no, nv, capi.n_tuples(nv))[1]
            if left < 0:
                break
            sizes.append("%d:%d" % (no, nv))
        return dict(kind="batch", form="fp64" if fp64 else "split_f16", systems=" ".join(sizes or ["8:40"]))
    if kind == "complex":
        return _stretch(rng, "fp64", _log(rng, 5, 20), _log(rng, 24, 90), math.exp(rng.uniform(math.log(4e9), math.log(1e11))),
                        rng.random() < 0.3, field="complex")
    no, nv = rng.randint(8, 40), _log(rng, 40, 140)
    n = capi.n_tuples(nv)
    count = int(min(n, max(64, math.exp(rng.uniform(math.log(4e9), math.log(4e10))) / (12.0 * no ** 3 * (no + nv)))))
    return dict(kind="noalloc", no=no, nv=nv, first=rng.randrange(n - count + 1), count=count)


# ------------------------------------------------------------------ inputs

def _inputs(no, nv, seed, j=False, field="real"):
    """Column-major tensors on the GPU: each has its indices reversed in torch's (row-major) order."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + no * 1009 + nv)

    def normal(shape, sigma):
        x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64).mul_(sigma)
        if field == "complex":
            x = torch.complex(x, torch.randn(shape, generator=g, device="cuda", dtype=torch.float64).mul_(sigma))
        return x

    def pair(sigma):  # X[a,b,i,j] == X[b,a,j,i]
        x = normal((no, no, nv, nv), sigma)
        return (x + x.permute(1, 0, 3, 2)).mul_(0.5).contiguous()

    def uniform(n, lo, hi):
        x = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo
        return torch.complex(x, torch.zeros_like(x)) if field == "complex" else x

    d = {"epsi": uniform(no, -2.0, -0.3), "epsa": uniform(nv, 0.1, 3.0), "Tai": normal((no, nv), 0.01),
         "Tabij": pair(0.05), "Vabij": pair(0.1), "Vijka": normal((nv, no, no, no), 0.1)}
    d["Vabci"] = normal((no, nv, nv, nv), 0.1)
    if j:
        d["Jijka"] = normal((nv, no, no, no), 0.1)
        d["Jabci"] = normal((no, nv, nv, nv), 0.1)
    torch.cuda.synchronize()
    return d


def _systems(case):
    return [tuple(int(v) for v in s.split(":")) for s in case["systems"].split()]


def _context(no, nv, seed, j=False, field="real"):
    ctx = capi.Context(no, nv, 0, field=field)
    d = _inputs(no, nv, seed, j, field)
    for n in REAL7 + (J2 if j else ()):
        ctx.upload(n, d[n])
    del d
    torch.cuda.empty_cache()  # the column-major originals are done with
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        ctx = _context(case["no"], case["nv"], seed, case["j"], case["field"])
        if case["tuned"]:
            ctx.set_tuning(split_variant=2, split_w_global=1, tuple_block=4)
        return dict(case=case, ctx=ctx)
    if kind == "batch":
        ctxs = [_context(no, nv, seed * 100 + k) for k, (no, nv) in enumerate(_systems(case))]
        return dict(case=case, ctxs=ctxs, batch=capi.Batch(ctxs))
    d = _inputs(case["no"], case["nv"], seed, case.get("j", False))
    if kind == "dropin":
        return dict(case=case, host={k: np.asfortranarray(v.cpu().numpy().T) for k, v in d.items()})
    n = case["count"]
    out = torch.empty(2 * n + 2, device="cuda", dtype=torch.float64)
    ptr = capi.DeviceInputs(*[d[k].data_ptr() for k in REAL7], None, None)
    return dict(case=case, d=d, out=out, ptr=ptr, lib=capi.load())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        t0, n = case["first"], case["count"]
        r = state["ctx"].run(form=case["form"], slices=case["slices"], use_j=case["j"], first_iteration=t0,
                             max_iterations=t0 + n - 1)
        e, ect = state["ctx"].tuple_energies(t0, n)
        return {"energy": r.energy, "ct_energy": r.ct_energy, "tuple_e": e, "tuple_ect": ect}
    if kind == "batch":
        res = state["batch"].run(form=case["form"], use_j=False)
        return {"energy": np.array([r.energy for r in res]),
                "tuple_e": [c.tuple_energies(0, r.tuples_done)[0] for c, r in zip(state["ctxs"], res)]}
    if kind == "dropin":
        h = state["host"]
        inp = atrip.Input().with_epsilon_i(h["epsi"]).with_epsilon_a(h["epsa"]).with_Tai(h["Tai"]).with_Tabij(h["Tabij"])
        inp.with_Vabij(h["Vabij"]).with_Vijka(h["Vijka"]).with_Vabci(h["Vabci"])
        if case["j"]:
            inp.with_Jijka(h["Jijka"]).with_Jabci(h["Jabci"])
        out = atrip.Atrip.run(inp)
        return {"energy": out.energy, "ct_energy": out.ct_energy}
    n, out = case["count"], state["out"]
    capi.check(state["lib"].atrip_gpu_run_fp64_noalloc(
        case["no"], case["nv"], ctypes.byref(state["ptr"]), case["first"], case["first"] + n - 1, 0, 0,
        out.data_ptr() + 16, out.data_ptr() + 16 + 8 * n, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return {"energy": out[:2], "tuple_e": out[2:2 + n]}


# ------------------------------------------------------------------ work

def _work(no, nv, n, j=False, field="real"):
    w, elem = (2 if j else 1), (16 if field == "complex" else 8)
    flops = n * (12.0 * no ** 3 * (no + nv) * w + 45.0 * no ** 3 / 6 * w) * (4 if field == "complex" else 1)
    # each input once: the whole tensors, or what n tuples can touch of them
    t2 = min(float(nv * nv * no * no), n * (3.0 * nv * no * no + 3 * no * no))
    v = min(float(nv ** 3 * no), n * 6.0 * nv * no) + min(float(no ** 3 * nv), n * 3.0 * no ** 3)
    vv = min(float(nv * nv * no * no), n * 3.0 * no * no)
    return elem * (t2 + vv + v * w + nv * no + nv + no) + 16.0 * n, flops


def work(case):
    if case["kind"] == "batch":
        ws = [_work(no, nv, capi.n_tuples(nv)) for no, nv in _systems(case)]
        return {"bytes": sum(w[0] for w in ws), "flops": sum(w[1] for w in ws)}
    n = case["count"] if "count" in case else capi.n_tuples(case["nv"])
    b, f = _work(case["no"], case["nv"], n, case.get("j", False), case.get("field", "real"))
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact

def _tuples(nv, first, count):
    """Positions first .. first + count - 1 of the list a <= b <= c without a == b == c."""
    out, pos = [], 0
    for a in range(nv):
        m = nv - a
        size = m * (m + 1) // 2 - 1
        if pos + size > first and pos < first + count:
            b, c = np.triu_indices(m)
            keep = (b + c) > 0
            b, c = b[keep] + a, c[keep] + a
            lo, hi = max(0, first - pos), min(size, first + count - pos)
            out.append(np.stack([np.full(hi - lo, a), b[lo:hi], c[lo:hi]], 1))
        pos += size
    return torch.from_numpy(np.concatenate(out)).cuda()


def _w(d, vh, vp, a, b, c):
    """Tijk of the tuples, [tuple, i, j, k]: particle terms minus hole terms."""
    T = d["Tabij"]  # [j, i, b, a]
    Vh, Vp = d[vh], d[vp]  # [a, k, j, i], [i, c, b, a]
    conj = T.is_complex()

    def slab(x):  # T[x,E,p,q] -> [n, (p,q), E]
        return T[:, :, :, x].permute(3, 1, 0, 2).reshape(len(x), -1, T.shape[2])

    def hole(w):  # Vh[p,q,L,w] -> [n, (p,q), L]
        h = Vh[w].permute(0, 3, 2, 1).reshape(len(w), -1, Vh.shape[1])
        return h.conj() if conj else h

    def vcol(y, z):  # V[y,z,E,r] -> [n, E, r]
        return Vp[:, :, z, y].permute(2, 1, 0)

    def tuv(u, v, flip):  # T[u,v,L,r] (or T[u,v,r,L]) -> [n, L, r]
        x = T[:, :, v, u]  # [j, i, n]
        return x.permute(2, 0, 1) if flip else x.permute(2, 1, 0)

    no = T.shape[0]

    def term(x, w, y, z, u, v, flip):
        r = torch.bmm(slab(x), vcol(y, z)) - torch.bmm(hole(w), tuv(u, v, flip))
        return r.reshape(len(x), no, no, no)  # [n, p, q, r]

    W = term(a, b, b, c, a, c, False)                                  # (i, j, k)
    W = W + term(a, c, c, b, a, b, False).permute(0, 1, 3, 2)          # (i, k, j)
    W += term(c, a, a, b, b, c, True).permute(0, 2, 3, 1)              # (k, i, j)
    W += term(c, b, b, a, a, c, True).permute(0, 3, 2, 1)              # (k, j, i)
    W += term(b, a, a, c, b, c, False).permute(0, 2, 1, 3)             # (j, i, k)
    W += term(b, c, c, a, a, b, True).permute(0, 3, 1, 2)              # (j, k, i)
    return W


def _energies(d, tup, j, limit=6e8):
    """Per-tuple energies (and (cT) energies) in 64 bits."""
    no, nv = d["Tabij"].shape[0], d["Tabij"].shape[2]
    tri = [(i, jj, k) for k in range(no) for jj in range(k, no) for i in range(jj, no)]
    I, J, K = (torch.tensor([t[m] for t in tri], device="cuda") for m in range(3))
    fac = torch.where(J == K, 0.5, 1.0).double() * torch.where(I == J, 0.5, 1.0).double()
    ei, ea, t1, V = d["epsi"], d["epsa"], d["Tai"], d["Vabij"]
    eijk = (ei[I] + ei[J]) + ei[K]
    e, ect = [], []
    step = max(1, min(len(tup), int(limit / (8.0 * (14 * no ** 3 + no * no * nv * 2)))))
    for lo in range(0, len(tup), step):
        a, b, c = tup[lo:lo + step].T.contiguous()
        W = _w(d, "Vijka", "Vabci", a, b, c)

        def vv(x, y):  # V[x,y,m,n] -> [n, m, n]
            return V[:, :, y, x].permute(2, 1, 0)

        Z = W + t1[:, a].T[:, :, None, None] * vv(b, c)[:, None, :, :]
        Z += t1[:, b].T[:, None, :, None] * vv(a, c)[:, :, None, :]
        Z += t1[:, c].T[:, None, None, :] * vv(a, b)[:, :, :, None]
        eabc = (ea[a] + ea[b] + ea[c]).real
        same = ((a == b) | (b == c))[:, None]

        def energy(T):
            def six(X):
                return [X[:, p, q, r] for p, q, r in ((I, J, K), (I, K, J), (J, I, K), (J, K, I), (K, I, J), (K, J, I))]

            U, Vv, Ww, X, Y, Zz = six(Z)
            A, B, C, D, E, F = six(T.conj() if T.is_complex() else T)
            first = A * U + (B * Vv + (C * Ww + (D * X + (E * Y + F * Zz))))
            uxy, vwz, ade, bcf = U + X + Y, Vv + Ww + Zz, A + D + E, B + C + F
            val = 3.0 * first + (uxy - 2.0 * vwz) * ade + (vwz - 2.0 * uxy) * bcf
            val_s = 3.0 * (A * U + D * X + E * Y) - ade * uxy
            q = 2.0 * torch.where(same, val_s, val) / (eabc[:, None] - eijk[None, :])
            return ((q.real if q.is_complex() else q) * fac).sum(1)

        e.append(energy(W))
        if j:
            ect.append(energy(_w(d, "Jijka", "Jabci", a, b, c)))
    e = torch.cat(e)
    return e, torch.cat(ect) if j else e


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        es = []
        for k, (no, nv) in enumerate(_systems(case)):
            d = _inputs(no, nv, seed * 100 + k)
            es.append(_energies(d, _tuples(nv, 0, capi.n_tuples(nv)), False)[0].cpu().numpy())
        return {"energy": np.array([-math.fsum(e) for e in es]), "tuple_e": es}
    no, nv, j = case["no"], case["nv"], case.get("j", False)
    first, count = case.get("first", 0), case.get("count", capi.n_tuples(nv))
    d = _inputs(no, nv, seed, j, case.get("field", "real"))
    e, ect = (x.cpu().numpy() for x in _energies(d, _tuples(nv, first, count), j))
    E, Ect = -math.fsum(e), -math.fsum(ect)
    if kind == "dropin":
        return {"energy": E, "ct_energy": Ect}
    if kind == "noalloc":
        return {"energy": np.array([E, Ect]), "tuple_e": e}
    return {"energy": E, "ct_energy": Ect, "tuple_e": e, "tuple_ect": ect}
