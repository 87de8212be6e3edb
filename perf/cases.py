"""The workloads whose speed this package is judged by: what each stands for, its
inputs, one pass through the public entry points, the work a pass cannot do without,
and the same pass in plain torch.

Sizes follow the measured configurations (24-site Lanczos, mTPQ and DSF, the 18-site
S = 1 cluster, the 30-site product, the served lattices of 18-26 sites, the Sz sector of
the Heisenberg model) and the sizes of the tests.  Chains are as long as their
coefficients stay a function of the input (Lanczos coefficients are chaotic once a Ritz
value has converged), which is the first few dozen steps.

A case's keys: kind, n (sites), s2 (2S), R (interleaved vectors), J, K, gamma, h (couplings
and the field along [111]), sector (Sz = 0 basis), host (start vector in host memory), steps.
"""
import math

import numpy as np
import torch

import pned_b200 as P
from pned_b200 import couplings as CP
from pned_b200.lattice import cluster_for_sites

KH = {"J": math.cos(0.3 * math.pi), "K": 2.0 * math.sin(0.3 * math.pi)}   # the 24- and 30-site workloads
S1 = {"J": 0.2, "K": -1.0}                                                # the S = 1 workload


def _case(name, kind, n, steps, s2=1, R=1, J=KH["J"], K=KH["K"], gamma=0.0, h=0.0, sector=False, host=False):
    c = {"kind": kind, "n": n, "s2": s2, "R": R, "J": J, "K": K, "gamma": gamma, "h": h, "sector": sector, "host": host,
         "steps": steps}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one H.v of a small cluster, as a host loop calls p_mltply_v3: latency
        _case("hv-n12", "hv", 12, 1),
        # one H.v of the largest cluster that a GPU holds with its Krylov vectors
        _case("hv-n30", "hv", 30, 1),
        # the smallest served lattice: a chain to the first convergence check, from a host vector (Fortran host)
        _case("lanczos-n18-host", "lanczos", 18, 32, host=True),
        # ground state of the 24-site cluster: chain, Ritz value, eigenvector pass
        _case("ground-n24", "ground", 24, 40),
        # the largest lattice of the served mix, with Gamma and a field (complex coefficients)
        _case("lanczos-n26-field", "lanczos", 26, 10, gamma=0.1, h=0.05),
        # Heisenberg model in its Sz = 0 sector
        _case("sector-n28", "lanczos", 28, 8, J=1.0, K=0.0, sector=True),
        # S = 1, 18 sites, one chain
        _case("s1-lanczos-n18", "lanczos", 18, 4, s2=2, **S1),
        # finite temperature: 16 random vectors on 24 sites with Gamma and a field
        _case("tps-n24-r16", "tps", 24, 5, R=16, gamma=0.1, h=0.05),
        # finite temperature for S = 1: 4 random vectors
        _case("s1-tps-n16-r4", "tps", 16, 4, s2=2, R=4, **S1),
        # dynamical structure factor: the 12 momenta of the 24-site cluster in one launch
        _case("dsf-n24-r12", "dsf", 24, 6, R=12),
        # a serving lane: four chains with couplings of their own (Lanczos and mTPQ side by side)
        _case("slots-n20-r4", "slots", 20, 24, R=4),
        # inverse iteration by conjugate gradients
        _case("cg-n20", "cg", 20, 30),
    ]


def draw(rng):
    kind = rng.choice(["hv", "lanczos", "ground", "sector", "s1-lanczos", "s1-tps", "tps", "dsf", "slots", "cg"])
    j, k = round(math.cos(a := rng.uniform(0.0, 2.0 * math.pi)), 4), round(2.0 * math.sin(a), 4)
    field = {"gamma": round(rng.uniform(-0.2, 0.2), 4), "h": round(rng.uniform(0.0, 0.1), 4)} if rng.random() < 0.5 else {}
    even = lambda lo, hi: 2 * rng.randint(lo // 2, hi // 2)  # noqa: E731  (honeycomb clusters have an even number of sites)
    wide = lambda n, most: rng.choice([r for r in (1, 2, 3, 4, 6, 8, 12, 16) if r <= most and r << n <= 1 << 28])  # noqa: E731
    if kind == "hv":
        n = even(8, 28)
        return _case(None, "hv", n, 1, R=wide(n, 16), J=j, K=k, **field)
    if kind == "lanczos":
        n = even(14, 26)
        return _case(None, "lanczos", n, rng.randint(6, 14 if n < 24 else 8), R=wide(n, 4) if n < 25 else 1, J=j, K=k, host=n < 22 and rng.random() < 0.3, **field)
    if kind == "sector":
        return _case(None, "lanczos", even(14, 28), rng.randint(5, 8), J=1.0, K=0.0, sector=True)
    if kind == "s1-lanczos":
        return _case(None, "lanczos", even(8, 16), rng.randint(4, 8), s2=2, J=j, K=k, **field)
    if kind == "s1-tps":
        return _case(None, "tps", even(8, 14), rng.randint(3, 6), s2=2, R=rng.choice([1, 2, 3, 4, 6, 8]), J=j, K=k, **field)
    if kind == "tps":
        n = even(14, 24)
        return _case(None, "tps", n, rng.randint(3, 12 if n < 22 else 5), R=wide(n, 16), J=j, K=k, **field)
    if kind == "dsf":
        n = even(14, 24)
        return _case(None, "dsf", n, rng.randint(4, 6), R=rng.choice([1, 2, 3, 4, 6, 8, 12]), J=j, K=k)
    if kind == "slots":
        n = even(14, 22)
        return _case(None, "slots", n, rng.randint(12, 24), R=wide(n, 8), J=j, K=k)
    n = even(12, 24 if kind == "ground" else 22)
    return _case(None, kind, n, rng.randint(12, 24 if n < 24 else 14), J=j, K=k, **field)


# ----------------------------------------------------------------------------- inputs

def _dim(c):
    return math.comb(c["n"], c["n"] // 2) if c["sector"] else (c["s2"] + 1) ** c["n"]


def _L(c):
    """mTPQ shift: l n with the l of the S = 1/2 and S = 1 workloads."""
    return (2.0 if c["s2"] == 1 else 3.0) * c["n"]


def _cg_E(c):
    """The energy that the inverse iteration is shifted by: a tenth below a short chain's lowest Ritz value."""
    v = _vectors(c, 1, 1, True)[0].view(-1, 1)
    al, be = _chain(lambda x: _apply(c, c, x), v, 16)
    return 1.1 * float(_ritz(al, be)[0])


def _vectors(c, seed, count, normalise):
    """`count` seeded complex Gaussian [dim][R] vectors on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    out = []
    for _ in range(count):
        v = torch.randn(_dim(c) * c["R"], dtype=torch.complex128, device="cuda", generator=g)
        if normalise:
            m = v.view(-1, c["R"])
            for r in range(c["R"]):
                m[:, r] /= torch.linalg.vector_norm(m[:, r])
        out.append(v)
    return out


def _slot_couplings(c, seed):
    """Couplings of each slot (those of a served stream): phi, Gamma and h by the seed."""
    rng = np.random.default_rng(int(seed))
    out = []
    for _ in range(c["R"]):
        phi = rng.uniform(0.0, 2.0 * math.pi)
        out.append({"s2": 1, "J": math.cos(phi), "K": 2.0 * math.sin(phi), "gamma": rng.uniform(-0.2, 0.2), "h": rng.uniform(0.0, 0.1)})
    return out


def _model_args(c, k):
    fld = CP.field_111(k["h"]) if k["h"] else None
    return dict(couplings=CP.kitaev_heisenberg(k["J"], k["K"], gamma=k["gamma"]), q=c["s2"] + 1, tree=0 if c["s2"] == 1 else 1, field=fld)


def _model(c, tps_L=None):
    cl = cluster_for_sites(c["n"])
    a = _model_args(c, c)
    if not c["sector"]:
        return P.Model.from_couplings(cl, a["couplings"], q=a["q"], tree=a["tree"], field=a["field"], tps_L=tps_L)
    X, skip, pt = P.build_xlocal(2, 0, a["couplings"])
    return P.Model(c["n"], 2, 0, cl.ipair, cl.ibond_type, X, skip, pt, total_sz=c["n"] // 2)


def _qr(c):
    cl = cluster_for_sites(c["n"])
    return np.ascontiguousarray([cl.qr(r % len(cl.q_list)) for r in range(c["R"])])


def prepare(c, seed):
    cl = cluster_for_sites(c["n"])
    s = {"c": c}
    kind = c["kind"]
    if kind == "slots":
        s["batch"] = P.SlotBatch(P.ModelInput.structure(cl), c["R"], c["steps"])
        s["couplings"] = []
        for k in _slot_couplings(c, seed):
            a = _model_args(c, k)
            s["couplings"].append(P.ModelInput.from_couplings(cl, a["couplings"], field=a["field"]))
        v = _vectors(dict(c, R=1), seed, c["R"], False)
        s["v"] = v
        return s
    s["model"] = _model(c, tps_L=_L(c) if kind == "tps" else None)
    s["ctx"] = P.Context(s["model"], R=c["R"])
    if kind == "hv":
        s["v1"], s["v0"] = _vectors(c, seed, 2, False)
    elif kind == "dsf":
        s["x"] = _vectors(dict(c, R=1), seed, 1, True)[0]
        s["qr"] = _qr(c)
    else:
        v = _vectors(c, seed, 1, True)[0]
        s["v"] = v.cpu().numpy() if c["host"] else v
    if kind == "cg":
        s["E"] = _cg_E(c)
    return s


# ----------------------------------------------------------------------------- one pass

def run(s):
    c = s["c"]
    kind, m = c["kind"], c["steps"]
    if kind == "hv":
        pr = s["ctx"].p_mltply_v3(s["v1"], s["v0"], 0.0625)
        return {"v0": s["v0"], "prdct": pr}
    if kind == "lanczos":
        r = s["ctx"].lanczos(s["v"], m)
        return {"alpha": r["alpha"], "beta": r["beta"], "ene": r["ene"]}
    if kind == "ground":
        r = s["ctx"].lanczos(s["v"], m)
        a, b = r["alpha"][:, 0], r["beta"][:, 0]
        E = P.bisec(a, b, m, 1)
        x = s["ctx"].lanczos_vector(s["v"], a, b, P.vec12(a, b, E, m, 1)[0])
        return {"alpha": r["alpha"], "beta": r["beta"], "ene": r["ene"], "x": x}
    if kind == "tps":
        return s["ctx"].tps(_L(c), s["v"], m)
    if kind == "dsf":
        return s["ctx"].dsf(s["x"], s["qr"], m)
    if kind == "cg":
        x, n_inv, n_cg = s["ctx"].cg(s["E"], s["v"], inv_max=1, cg_max=m)
        return {"x": x, "n_inv": n_inv, "n_cg": n_cg}
    b = s["batch"]
    for r in range(c["R"]):
        if r % 2 == 0:
            b.load(r, "lanczos", s["couplings"][r], s["v"][r], m)
        else:
            b.load(r, "tps", s["couplings"][r], s["v"][r], m, L=_L(c))
    b.step(m)
    out = []
    for r in range(c["R"]):
        d = b.read(r)
        out.append({k: d[k] for k in ("steps", "status", "alpha", "beta") + (("coef",) if r % 2 else ())})
        b.release(r)
    return out


def work(c):
    """Bytes: each vector that a pass or step reads once and writes once (H.v: v1, v0 in, v0 out;
    a Lanczos or TPS step: two vectors in, one out).  Flops: the nonzero products."""
    elems = float(_dim(c)) * c["R"]
    q = c["s2"] + 1
    per = 0.0   # flops of H.v per element
    cl = cluster_for_sites(c["n"])
    if q == 2:
        nb = cl.nbond if not c["sector"] else cl.nbond / 2
        sites = c["n"] if (c["h"] or c["gamma"]) else 0
        per = (nb + sites) * (8.0 if sites else 4.0)
    else:
        loc = _local(c, c)
        for t in cl.ibond_type:
            x = loc[int(t)] - np.diag(np.diag(loc[int(t)]))
            per += np.count_nonzero(np.abs(x) > 1e-14) / float(q * q) * (8.0 if np.iscomplexobj(x) and np.any(x.imag) else 4.0)
    m = c["steps"]
    # bytes per element of a step (or pass)
    step = {"hv": 48.0, "lanczos": 48.0, "tps": 48.0, "dsf": 48.0, "slots": 48.0, "ground": 48.0 + 80.0, "cg": 112.0}[c["kind"]]
    rounds = 2.0 if c["kind"] == "ground" else 1.0
    return {"bytes": m * step * elems, "flops": m * rounds * (per + 16.0) * elems}


# ----------------------------------------------------------------------------- the same in plain torch

def _spin(q, s2):
    """S^x, S^y, S^z as the package's two conventions have them (S = 1/2: digit 0 up; S >= 1: digit d is m = d - S)."""
    if s2 == 1:
        return (np.array([[0, .5], [.5, 0]], complex), np.array([[0, -.5j], [.5j, 0]]), np.array([[.5, 0], [0, -.5]], complex))
    S = 0.5 * s2
    up = np.zeros((q, q), complex)   # element (i, i + 1)
    for i in range(q - 1):
        mz = i - S
        up[i, i + 1] = math.sqrt((S - mz) * (S + mz + 1.0))
    return 0.5 * (up + up.T), -0.5j * (up - up.T), np.diag(np.arange(q) - S).astype(complex)


def _local(c, k):
    """{bond type: two-site matrix} of J S.S + K S^g S^g + Gamma (S^a S^b + S^b S^a) - h.(S_1 + S_2) / 3,
    the first site on the fast digit."""
    q = c["s2"] + 1
    s = _spin(q, c["s2"])
    hf = k["h"] / math.sqrt(3.0)
    out = {}
    for t, g in ((1, 0), (2, 1), (3, 2)):
        a, b = [i for i in range(3) if i != g]
        m = sum(k["J"] * np.kron(s[i], s[i]) for i in range(3)) + k["K"] * np.kron(s[g], s[g])
        m = m + k["gamma"] * (np.kron(s[a], s[b]) + np.kron(s[b], s[a]))
        one = np.eye(q)
        for i in range(3):
            m = m - hf / 3.0 * (np.kron(one, s[i]) + np.kron(s[i], one))
        out[t] = m
    return out


def _apply(c, k, v, shift=0.0, sign=1.0):
    """sign * H^T v + shift v (the package applies the transpose, as the reference does), v [q^n][R]."""
    n, q, R = c["n"], c["s2"] + 1, v.shape[1]
    cl = cluster_for_sites(n)
    loc = _local(c, k)
    out = v * shift
    for (a, b), t in zip(cl.site_pairs0(), cl.ibond_type):
        lo, hi = int(min(a, b)), int(max(a, b))
        x = loc[int(t)]
        shape = (q ** (n - 1 - hi), q, q ** (hi - lo - 1), q, q ** lo * R)
        vi, oi = v.view(shape), out.view(shape)
        for tgt in range(q * q):
            for cur in range(q * q):
                z = complex(sign * x[tgt, cur])
                if abs(z) > 1e-15:
                    oi[:, cur // q, :, cur % q].add_(vi[:, tgt // q, :, tgt % q], alpha=z if z.imag else z.real)
    return out


def _sector_index(n):
    """States with n / 2 set bits, ascending (the package's sector order)."""
    parts = []
    chunk = 1 << min(n, 24)
    for lo in range(0, 1 << n, chunk):
        s = torch.arange(lo, lo + chunk, device="cuda", dtype=torch.int64)
        cnt = torch.zeros_like(s)
        for b in range(n):
            cnt += (s >> b) & 1
        parts.append(s[cnt == n // 2])
    return torch.cat(parts)


def _dots(a, b):
    return torch.stack([torch.vdot(a[:, r], b[:, r]) for r in range(a.shape[1])])


def _chain(H, v, m):
    """Lanczos coefficients [m][R] of the columns of v."""
    al, be = [], []
    prev, beta = None, None
    for _ in range(m):
        w = H(v)
        a = _dots(v, w).real
        w -= v * a
        if prev is not None:
            w -= prev * beta
        beta = torch.stack([torch.linalg.vector_norm(w[:, r]) for r in range(w.shape[1])])
        al.append(a.cpu().numpy())
        be.append(beta.cpu().numpy())
        prev, v = v, w / beta
    return np.array(al), np.array(be)


def _tps(H, v, m, L):
    """mTPQ norms and coefficients of the columns of v, H = L - H."""
    R = v.shape[1]
    al, be, co = np.zeros((m, R)), np.zeros((m, R)), np.zeros((m, R, 5))
    g = None
    for k in range(m):
        w = H(v)
        a1 = _dots(v, w).real.cpu().numpy()
        b = torch.stack([torch.linalg.vector_norm(w[:, r]) for r in range(R)])
        al[k], be[k] = L - a1, b.cpu().numpy()
        co[k, :, 0], co[k, :, 1], co[k, :, 2], co[k, :, 3] = 2.0 * (k + 1) / a1, L, be[k], al[k]
        if g is not None:
            co[k, :, 4] = (L * _dots(g, v).real - _dots(g, w).real).cpu().numpy()
        g, v = v, w / b
    return {"alpha": al, "beta": be, "coef": co}


def _ritz(al, be):
    m = len(al)
    e = np.zeros(8)
    t = np.diag(al[:, 0]) + np.diag(be[:m - 1, 0], 1) + np.diag(be[:m - 1, 0], -1)
    w = np.linalg.eigvalsh(t)[:min(m, 8)]
    e[:len(w)] = w
    return e


def exact(c, seed):
    kind, m, R = c["kind"], c["steps"], c["R"]
    if kind == "slots":
        out = []
        vs = _vectors(dict(c, R=1), seed, R, False)
        for r, k in enumerate(_slot_couplings(c, seed)):
            v = (vs[r] / torch.linalg.vector_norm(vs[r])).view(-1, 1)
            if r % 2 == 0:
                al, be = _chain(lambda x: _apply(c, k, x), v, m)
                out.append({"steps": m, "status": 0, "alpha": al[:, 0], "beta": be[:, 0]})
            else:
                d = _tps(lambda x: _apply(c, k, x, shift=_L(c), sign=-1.0), v, m, _L(c))
                out.append({"steps": m, "status": 0, "alpha": d["alpha"][:, 0], "beta": d["beta"][:, 0], "coef": d["coef"][:, 0]})
        return out
    if kind == "hv":
        v1, v0 = (v.view(-1, R) for v in _vectors(c, seed, 2, False))
        w = _apply(c, c, v1, shift=-0.0625 * cluster_for_sites(c["n"]).nbond)
        pr = _dots(v1, w).cpu().numpy()
        return {"v0": v0.add_(w).view(-1), "prdct": pr}
    if kind == "dsf":
        x = _vectors(dict(c, R=1), seed, 1, True)[0]
        q, n = c["s2"] + 1, c["n"]
        qr = _qr(c)
        w = torch.zeros(q ** n, R, dtype=torch.complex128, device="cuda")
        for j in range(n):
            f = torch.tensor([d - 0.5 * c["s2"] for d in range(q)], dtype=torch.float64, device="cuda").view(1, q, 1, 1)
            ph = torch.tensor(np.exp(1j * qr[:, j]), device="cuda").view(1, 1, 1, R)
            w.view(q ** (n - 1 - j), q, q ** j, R).add_(f * ph)
        w *= x.view(-1, 1)
        raw = torch.stack([torch.linalg.vector_norm(w[:, r]) ** 2 for r in range(R)])
        w /= raw.sqrt()
        al, be = _chain(lambda y: _apply(c, c, y), w, m)
        cn = (raw / n).cpu().numpy()
        # S^z_q at q = 0 is the total spin: its chain is as well defined as the others on a random vector
        return {"cnorm": cn, "salpha": al, "sbeta": np.concatenate([cn[None], be])}
    v = _vectors(c, seed, 1, True)[0].view(-1, R)
    if kind == "tps":
        return _tps(lambda x: _apply(c, c, x, shift=_L(c), sign=-1.0), v, m, _L(c))
    if kind == "cg":
        E = _cg_E(c)
        b = v[:, 0]
        x, r, p = torch.zeros_like(b), b.clone(), b.clone()
        for _ in range(m):
            y = _apply(c, c, p.view(-1, 1), shift=-E)[:, 0]
            rr = torch.vdot(r, r).real
            a = torch.vdot(p, r) / torch.vdot(p, y)
            x += a * p
            r = r - a * y
            p = r + (torch.vdot(r, r).real / rr) * p
        return {"x": x / torch.linalg.vector_norm(x), "n_inv": 1, "n_cg": m}
    if c["sector"]:
        idx = _sector_index(c["n"])

        def H(y):
            full = torch.zeros(1 << c["n"], 1, dtype=torch.complex128, device="cuda")
            full[idx] = y
            return _apply(dict(c, sector=False), c, full)[idx]
    else:
        def H(y):
            return _apply(c, c, y)
    al, be = _chain(H, v, m)
    out = {"alpha": al, "beta": be, "ene": _ritz(al, be)}
    if kind == "ground":
        out["x"] = None   # a Ritz vector's sign is the inverse iteration's choice
    return out
