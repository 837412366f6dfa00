"""Workloads on which the library's speed is measured, each one call (or one
measurement cycle) a user's program makes through the public entry points.

The physics is the Falicov-Kimball model on the reference's lattices: periodic
hopping -t, U on f-occupied sites, mu_c = mu_f = U/2, f occupations
Bernoulli(0.5) from the seed. `listed()` spans one N = 64 chain to 1024 chains
of uneven size, both precisions, the drop-in calc_ed call, the free-energy
gradients, an eigenvector measure, the Chebyshev method and the rank-one
update; `draw()` varies lattice, size, batch, precision and step count over the
same ranges.
"""
import math

import numpy as np
import torch

NDIM = {"cubic1d": 1, "cubic2d": 2, "cubic3d": 3, "triangular": 2}
# the lattices of the uneven batch: N = 144 .. 1024
UNEVEN = [("cubic2d", 12), ("cubic2d", 16), ("cubic2d", 20), ("cubic2d", 24), ("cubic2d", 32), ("triangular", 12),
          ("triangular", 18), ("triangular", 24)]
NW, ETA = 64, 0.05  # conductivity grid of the stiffness measure
EXACT_N3 = 2.0e11   # sum of n^3 over the dense solves exact() may spend


def listed():
    return [
        # one Markov chain of the reference's smallest benchmark (cubic2d L=8), one sweep of single-site
        # proposals and the measurement's read-back: the smallest call, latency and launches count
        {"name": "sweep_f64_n64_b1", "op": "chains", "precision": "f64", "method": "ed", "kind": "cubic2d", "L": 8,
         "batch": 1, "steps": 64, "U": 1.0, "beta": 1.0, "device": False},
        # the drop-in configuration_t::calc_ed of one configuration of odd order (cubic3d L=7, N=343):
        # spectrum, exp, fermi, logZ, host buffers
        {"name": "calc_ed_f64_n343_b1", "op": "calc_ed", "precision": "f64", "kind": "cubic3d", "L": 7, "batch": 1,
         "U": 2.0, "beta": 5.0},
        # 512 independent chains at N=256 on the plain FP64 path (a scan of U and beta run as one batch)
        {"name": "chains_f64_n256_b512", "op": "chains", "precision": "f64", "method": "ed", "kind": "cubic2d",
         "L": 16, "batch": 512, "steps": 2, "U": 2.0, "beta": 5.0, "device": False},
        # 128 chains on the cubic lattice L=8 (N=512), mixed precision
        {"name": "chains_mixed_n512_b128", "op": "chains", "precision": "mixed", "method": "ed", "kind": "cubic3d",
         "L": 8, "batch": 128, "steps": 2, "U": 2.0, "beta": 5.0, "device": False},
        # the benchmark workload: 256 chains, cubic2d L=24 (N=576), inputs resident on the device; mixed ...
        {"name": "chains_mixed_n576_b256", "op": "chains", "precision": "mixed", "method": "ed", "kind": "cubic2d",
         "L": 24, "batch": 256, "steps": 2, "U": 2.0, "beta": 4.0, "device": True},
        # ... and plain FP64
        {"name": "chains_f64_n576_b256", "op": "chains", "precision": "f64", "method": "ed", "kind": "cubic2d",
         "L": 24, "batch": 256, "steps": 1, "U": 2.0, "beta": 4.0, "device": True},
        # a small temperature scan on the largest lattice (cubic2d L=32, N=1024): 16 chains, mixed
        {"name": "chains_mixed_n1024_b16", "op": "chains", "precision": "mixed", "method": "ed", "kind": "cubic2d",
         "L": 32, "batch": 16, "steps": 2, "U": 3.0, "beta": 8.0, "device": False},
        # 1024 chains of uneven size and lattice, U in [0.5, 4], beta in [1, 10]: the largest call
        {"name": "uneven_mixed_b1024", "op": "chains", "precision": "mixed", "method": "ed", "kind": "uneven", "L": 0,
         "batch": 1024, "steps": 1, "U": 0.0, "beta": 0.0, "device": True},
        # free energy and its derivatives through torch.autograd for 256 configurations at N=576
        {"name": "grad_mixed_n576_b256", "op": "grad", "precision": "mixed", "kind": "cubic2d", "L": 24, "batch": 256,
         "U": 2.0, "beta": 4.0},
        # Drude stiffness and conductivity of 32 configurations, triangular L=15 (N=225, odd), FP64 eigenvectors
        {"name": "stiffness_f64_n225_b32", "op": "stiffness", "precision": "f64", "kind": "triangular", "L": 15,
         "batch": 32, "U": 2.0, "beta": 10.0},
        # the same 256 chains as the benchmark with logZ from the Chebyshev expansion (cheb_moves)
        {"name": "cheb_n576_b256", "op": "chains", "precision": "f64", "method": "chebyshev", "kind": "cubic2d",
         "L": 24, "batch": 256, "steps": 3, "U": 2.0, "beta": 4.0, "device": True},
        # rank-one evaluation of 256 single-site proposals at N=576 from resident eigenpairs
        {"name": "rank1_n576_b256", "op": "rank1", "precision": "f64", "kind": "cubic2d", "L": 24, "batch": 256,
         "U": 2.0, "beta": 4.0},
    ]


def draw(rng):
    log = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))
    op = rng.choice(["chains"] * 5 + ["calc_ed", "calc_ed", "grad", "stiffness", "ipr", "cheb", "rank1"])
    if op in ("chains",) and rng.random() < 0.15:
        return {"op": "chains", "precision": rng.choice(["mixed", "f64"]), "method": "ed", "kind": "uneven", "L": 0,
                "batch": int(log(8, 200)), "steps": 1, "U": 0.0, "beta": 0.0, "device": rng.random() < 0.5}
    kind = rng.choice(["cubic1d", "cubic2d", "cubic2d", "cubic2d", "cubic3d", "triangular"])
    if op in ("stiffness", "ipr") and kind == "cubic1d":  # nearly degenerate localized states: vectors not unique
        kind = "cubic2d"
    d = NDIM[kind]
    lo, hi = (36, 1024) if op not in ("cheb", "stiffness", "ipr") else (64, 729)
    L = max(int(round(log(lo, hi) ** (1.0 / d))), 3)
    while L ** d > hi:
        L -= 1
    n = L ** d
    precision = rng.choice(["f64", "mixed"])
    most = {"cheb": 512, "rank1": 512}.get(op, 768)
    cap = 1.5e11 if precision == "mixed" else 4.5e10  # batch n^3 of the largest listed calls
    if op in ("stiffness", "ipr", "grad"):
        cap = min(cap, 2.0e10 if precision == "f64" else 4.9e10)
    if op == "calc_ed":
        most = 32
    batch = max(1, min(int(log(1, most)), int(cap / n ** 3)))
    c = {"op": op, "precision": precision, "kind": kind, "L": L, "batch": batch,
         "U": rng.choice([0.5, 1.0, 2.0, 4.0]), "beta": rng.choice([1.0, 3.0, 5.0, 10.0])}
    if op == "stiffness":  # a near-cancellation of two sums: measured on the FP64 path
        c["precision"] = "f64"
        c["batch"] = max(1, min(batch, int(2.0e10 / n ** 3)))
    if op == "rank1":
        c["precision"] = "f64"
    if op in ("chains", "cheb"):
        c["method"] = "chebyshev" if op == "cheb" else "ed"
        c["op"] = "chains"
        c["steps"] = rng.choice([1, 2, 4, 8]) if batch * n ** 3 < cap / 16 else 1
        c["device"] = rng.random() < 0.5
    return c


# ---- inputs -----------------------------------------------------------------

def _csr(kind, L):
    """(rows, cols, vals) of the periodic hopping matrix, -1 per bond, entries that coincide added."""
    d = NDIM[kind]
    n = L ** d
    pos = np.stack(np.unravel_index(np.arange(n), (L,) * d), axis=1)
    mult = np.array([L ** (d - 1 - a) for a in range(d)])
    rows, cols = [], []
    steps = [(a, s) for a in range(d) for s in (-1, 1)]
    for a, s in steps:
        p = pos.copy()
        p[:, a] = (p[:, a] + s) % L
        rows.append(np.arange(n))
        cols.append(p @ mult)
    if kind == "triangular":
        for s in (-1, 1):
            rows.append(np.arange(n))
            cols.append(((pos + s) % L) @ mult)
    return n, np.concatenate(rows), np.concatenate(cols)


def _dense(kind, L):
    n, r, c = _csr(kind, L)
    H = np.zeros((n, n))
    np.add.at(H, (r, c), -1.0)
    return H


def _lattices(case):
    return UNEVEN if case["kind"] == "uneven" else [(case["kind"], case["L"])]


def _inputs(case, seed):
    """Everything a pass reads, as numpy arrays, from the seed alone."""
    rng = np.random.default_rng(seed)
    B = case["batch"]
    lat = _lattices(case)
    ids = (np.arange(B) % len(lat)).astype(np.int32)
    ns = np.array([lat[i][1] ** NDIM[lat[i][0]] for i in ids])
    if case["kind"] == "uneven":
        U, beta = rng.uniform(0.5, 4.0, B), rng.uniform(1.0, 10.0, B)
    else:
        U, beta = np.full(B, case["U"]), np.full(B, case["beta"])
    f = [rng.integers(0, 2, n).astype(np.int32) for n in ns]
    steps = case.get("steps", 1)
    site = (rng.random((steps, B)) * ns).astype(np.int32)
    u = rng.random((steps, B))
    return {"lat": lat, "ids": ids, "ns": ns, "U": U, "beta": beta, "f": f, "site": site, "u": u}


def _cheb_size(n):
    m = int(math.log(n) * 2.2)
    m += m % 2
    return m, max(2 * m, 10)


def _rank1_inputs(case, seed):
    """8 configurations with their eigenpairs, batch/8 proposed sites on each (a chain's sites tried in turn)."""
    rng = np.random.default_rng(seed)
    H0 = _dense(case["kind"], case["L"])
    n, B = H0.shape[0], case["batch"]
    nc = min(8, B)
    fs = rng.integers(0, 2, (nc, n))
    own = np.arange(B) % nc
    sites = rng.integers(0, n, B)
    ev, z, rho = np.empty((B, n)), np.empty((B, n)), np.empty(B)
    for c in range(nc):
        w, V = np.linalg.eigh(H0 + np.diag(case["U"] * (fs[c] - 0.5)))
        for b in np.nonzero(own == c)[0]:
            ev[b], z[b] = w, V[sites[b]]
            rho[b] = case["U"] if fs[c, sites[b]] == 0 else -case["U"]
    return {"H0": H0, "fs": fs, "own": own, "sites": sites, "ev": ev, "z": z, "rho": rho,
            "beta": np.full(B, case["beta"])}


def prepare(case, seed):
    import fk_mc_gb300
    B, op = case["batch"], case["op"]
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
    lat = _lattices(case)
    nmax = max(L ** NDIM[k] for k, L in lat)
    s = fk_mc_gb300.Solver(max_n=nmax, max_batch=B, precision=case["precision"])
    ns = [s.set_lattice(i, k, L) for i, (k, L) in enumerate(lat)]
    st = {"case": case, "solver": s, "n": ns[0]}
    if op == "rank1":
        x = _rank1_inputs(case, seed)
        for k in ("ev", "z", "rho", "beta"):
            st[k] = dev(x[k])
        st["logz"] = torch.zeros(B, dtype=torch.float64, device="cuda")
        st["evnew"] = torch.zeros((B, ns[0]), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return st
    x = _inputs(case, seed)
    st.update(ids=x["ids"], beta=x["beta"])
    if op == "chains":
        if case["method"] == "chebyshev":
            s.set_chebyshev(*_cheb_size(ns[0]))
            s.set_method("chebyshev")
        s.chains_init(x["ids"], np.concatenate(x["f"]), x["U"], x["U"] / 2, x["U"] / 2, x["beta"])
        if case["device"]:
            st.update(site=dev(x["site"]), u=dev(x["u"]))
            st["acc"] = torch.zeros(x["site"].shape, dtype=torch.int32, device="cuda")
            st["dlogz"] = torch.zeros(x["site"].shape, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
        else:
            st.update(site=x["site"], u=x["u"])
        return st
    if op == "grad":
        st["f"] = np.concatenate(x["f"])
        for k, v in (("U", x["U"]), ("t", np.ones(B)), ("mu", x["U"] / 2), ("tbeta", x["beta"])):
            st[k] = dev(v).requires_grad_(True)
        return st
    st["diag"] = np.concatenate([U * (f - 0.5) for U, f in zip(x["U"], x["f"])])
    if op == "stiffness":
        s.set_stiffness_ops(0, case["kind"], case["L"])
        st["wgrid"] = np.linspace(-4.0, 4.0, NW)
    return st


def run(st):
    case, s = st["case"], st["solver"]
    op = case["op"]
    if op == "chains":
        if case["device"]:
            s.propose_accept_device(case["steps"], st["site"].data_ptr(), st["u"].data_ptr(), st["acc"].data_ptr(),
                                    st["dlogz"].data_ptr())
            acc, dlogz = st["acc"], st["dlogz"]
        else:
            acc, dlogz = s.propose_accept(st["site"], st["u"])
        f, logz, w = s.chains_get()  # what the energy and occupation measures read
        return {"accepted": acc, "dlogz": dlogz, "f": f, "logz": logz, "spectrum": w}
    if op == "calc_ed":
        r = s.eigh_logz(st["ids"], st["diag"], st["beta"], exp_fermi=True)
        return {k: r[k] for k in ("evals", "exp", "fermi", "logz")}
    if op == "grad":
        from fk_mc_gb300.autograd import FreeEnergy
        p = [st["U"], st["t"], st["mu"], st["tbeta"]]
        F = FreeEnergy.apply(*p, s, st["ids"], st["f"])
        g = torch.autograd.grad(F.sum(), p)
        return {"F": F, "dU": g[0], "dt": g[1], "dmu": g[2], "dbeta": g[3]}
    if op == "stiffness":
        d, cond = s.measure_stiffness(st["ids"], st["diag"], st["beta"], st["wgrid"], ETA)
        return {"stiffness": d, "cond": cond}
    if op == "ipr":
        return {"ipr": np.concatenate(s.measure_ipr(st["ids"], st["diag"], st["beta"]))}
    s.rank1_logz_device(case["batch"], st["n"], st["ev"].data_ptr(), st["z"].data_ptr(), st["rho"].data_ptr(),
                        st["beta"].data_ptr(), st["logz"].data_ptr(), st["evnew"].data_ptr())
    return {"logz": st["logz"], "evals": st["evnew"]}


def work(case):
    """Eigenvalues only: 4/3 n^3 flops (Householder reduction); eigenvectors: 10/3 n^3; inputs read and outputs
    written once."""
    B, op = case["batch"], case["op"]
    lat = _lattices(case)
    ns = [lat[c % len(lat)][1] ** NDIM[lat[c % len(lat)][0]] for c in range(B)]
    n1, n2, n3 = (float(sum(n ** q for n in ns)) for q in (1, 2, 3))
    steps = case.get("steps", 1)
    if op == "chains" and case["method"] == "chebyshev":
        m, _ = _cheb_size(ns[0])
        d, r = NDIM[case["kind"]], m // 2
        ball = min(ns[0], {1: 2 * r + 1, 2: 2 * r * r + 2 * r + 1, 3: (4 * r ** 3 + 6 * r * r + 8 * r + 3) // 3}[d])
        deg = 2 * d + (2 if case["kind"] == "triangular" else 0)
        return {"bytes": steps * 24.0 * B + 12.0 * n1, "flops": steps * n1 * ball * r * 2.0 * (deg + 3)}
    if op == "chains":
        return {"bytes": steps * 24.0 * B + 12.0 * n1, "flops": steps * 4.0 / 3.0 * n3}
    if op == "calc_ed":
        return {"bytes": 32.0 * n1, "flops": 4.0 / 3.0 * n3}
    if op == "grad":
        return {"bytes": 4.0 * n1 + 72.0 * B, "flops": 10.0 / 3.0 * n3}
    if op == "stiffness":
        return {"bytes": 8.0 * n1 + 8.0 * B * (NW + 1), "flops": 13.0 / 3.0 * n3 + 5.0 * NW * n2}
    if op == "ipr":
        return {"bytes": 16.0 * n1, "flops": 10.0 / 3.0 * n3}
    return {"bytes": 24.0 * n1, "flops": 2 * 7.0 * n2}


# ---- the same in 64 bits, without the library --------------------------------

def _logz(w, beta):
    return float(np.sum(np.logaddexp(0.0, -beta * w)))


def _cheb_logz(w, beta):
    """logZ by the Chebyshev expansion on the Lobatto grid (trapezoid rule in theta), moments from the spectrum."""
    n = w.size
    M, G = _cheb_size(n)
    a, b = (w[-1] - w[0]) / 2, (w[-1] + w[0]) / 2
    t = np.arccos(np.clip((w - b) / a, -1.0, 1.0))
    x = -np.cos(np.pi * np.arange(G) / (G - 1))
    fx = n * np.logaddexp(0.0, -beta * (a * x + b))
    wt = np.full(G, 1.0 / (G - 1))
    wt[[0, -1]] *= 0.5
    c = [np.sum(wt * fx * np.cos(m * np.arccos(x))) for m in range(M)]
    return float(sum((1 if m == 0 else 2) * c[m] * np.mean(np.cos(m * t)) for m in range(M)))


def exact(case, seed):
    op, B = case["op"], case["batch"]
    lat = _lattices(case)
    n3 = sum((lat[c % len(lat)][1] ** NDIM[lat[c % len(lat)][0]]) ** 3 for c in range(B))
    vectors = op in ("grad", "stiffness", "ipr")
    if n3 * (1 + case.get("steps", 0)) * (4 if vectors else 1) > EXACT_N3:
        return None
    if op == "rank1":
        x = _rank1_inputs(case, seed)
        w = []
        for b in range(B):
            H = x["H0"] + np.diag(case["U"] * (x["fs"][x["own"][b]] - 0.5))
            H[x["sites"][b], x["sites"][b]] += x["rho"][b]
            w.append(np.linalg.eigvalsh(H))
        return {"logz": np.array([_logz(v, case["beta"]) for v in w]), "evals": np.array(w)}
    x = _inputs(case, seed)
    H0 = [_dense(k, L) for k, L in lat]
    ham = lambda c, f: H0[x["ids"][c]] + np.diag(x["U"][c] * (f - 0.5))
    if op == "chains":
        cheb = case["method"] == "chebyshev"
        lz = _cheb_logz if cheb else _logz
        out = {"accepted": np.zeros(x["site"].shape, np.int32), "dlogz": np.zeros(x["site"].shape)}
        fe, ze, we = [], [], []
        for c in range(B):
            f, beta, mu = x["f"][c].copy(), x["beta"][c], x["U"][c] / 2
            w = np.linalg.eigvalsh(ham(c, f))
            z = lz(w, beta)
            for s in range(case["steps"]):
                g = f.copy()
                i = x["site"][s, c]
                g[i] ^= 1
                wn = np.linalg.eigvalsh(ham(c, g))
                zn = lz(wn, beta)
                out["dlogz"][s, c] = zn - z
                if math.exp(zn - z) * math.exp(beta * mu if g[i] else -beta * mu) > x["u"][s, c]:
                    out["accepted"][s, c] = 1
                    f, w, z = g, wn, zn
            fe.append(f)
            ze.append(z)
            we.append(np.zeros_like(w) if cheb else w)
        out.update(f=np.concatenate(fe), logz=np.array(ze), spectrum=np.concatenate(we))
        return out
    if op == "calc_ed":
        w = np.array([np.linalg.eigvalsh(ham(c, x["f"][c])) for c in range(B)])
        e = np.exp(x["beta"][:, None] * w)
        return {"evals": w.ravel(), "exp": e.ravel(), "fermi": (1 / (1 + e)).ravel(),
                "logz": np.array([_logz(w[c], x["beta"][c]) for c in range(B)])}
    out = {k: np.zeros(B) for k in ("F", "dU", "dt", "dmu", "dbeta")}
    ipr, stiff, cond = [], np.zeros(B), np.zeros((B, NW))
    if op == "stiffness":
        n, L, d = x["ns"][0], case["L"], NDIM[case["kind"]]
        pos = np.stack(np.unravel_index(np.arange(n), (L,) * d), axis=1)
        T, J = np.zeros((n, n)), np.zeros((n, n))
        for s in (-1, 1):
            p = pos.copy()
            p[:, 0] = (p[:, 0] + s) % L
            q = p @ np.array([L ** (d - 1 - a) for a in range(d)])
            np.add.at(T, (np.arange(n), q), -1.0)
            np.add.at(J, (np.arange(n), q), float(s))
    for c in range(B):
        w, V = np.linalg.eigh(ham(c, x["f"][c]))
        beta, U = x["beta"][c], x["U"][c]
        fer = 1 / (1 + np.exp(beta * w))
        if op == "ipr":
            ipr.append(np.sum(V ** 4, axis=0) ** 0.25 / np.sum(V ** 2, axis=0))
        elif op == "grad":
            rho = (V ** 2) @ fer
            F, E = -_logz(w, beta) / beta, float(np.sum(w * fer))
            dU, dmu = float(np.sum(x["f"][c] * rho)), -float(np.sum(rho))
            for k, v in (("F", F), ("dU", dU), ("dmu", dmu), ("dt", E - U * dU - U / 2 * dmu), ("dbeta", (E - F) / beta)):
                out[k][c] = v
        else:
            mJ = V.T @ J @ V
            sig = np.pi * (fer[None, :] - fer[:, None]) * mJ.T * mJ   # [i, j]
            de = w[:, None] - w[None, :]
            ok = np.tril(np.ones((n, n), bool), -1) & (np.abs(de) > 1e-12) & (np.abs(sig) > 1e-13)
            sg, dd = sig[ok], de[ok]
            stiff[c] = (np.sum(2 * sg / dd) - np.pi * np.sum(fer * np.sum(V * (T @ V), axis=0))) / n
            lor = lambda y: ETA / np.pi / (y * y + ETA * ETA)
            for q, wq in enumerate(np.linspace(-4.0, 4.0, NW)):
                cond[c, q] = np.sum(sg * (lor(wq - dd) - lor(wq + dd)))
    if op == "ipr":
        return {"ipr": np.concatenate(ipr)}
    return out if op == "grad" else {"stiffness": stiff, "cond": cond}
