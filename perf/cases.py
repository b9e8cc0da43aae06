"""The work a user of this framework has it do, as timed cases.

Eight kinds of call, each through the public entry points: a pairwise
contraction and a network contraction of labelled tensors, the QR and the
truncated SVD of a site or two-site tensor, the compression of an MPS through
the drop-in class, the MPO application, the native apply + compress sweep, and
a queue of uneven states.  ``listed()`` names the fixed cases, ``draw()`` gives
more of the same ranges.

SVD factors and the sites of a compressed MPS are defined up to a gauge (a
phase per singular vector), so those cases return what is not: the tensor the
factors stand for, the state's amplitudes, or, where 2^N amplitudes are too
many, the bond dimensions, the kept weights, the norm and the fidelity to the
state before truncation, and in double precision the one-site density matrices
(in single precision a cut through a dense spectrum does not determine them).
"""
import math
import random

import numpy as np
import torch

import tncontract_gb300 as tn
from tncontract_gb300 import engine

_DTYPE = {"f32": torch.float32, "f64": torch.float64, "c64": torch.complex64, "c128": torch.complex128}
_WIDE = {"f32": torch.float64, "f64": torch.float64, "c64": torch.complex128, "c128": torch.complex128}
_BYTES = {"f32": 4, "f64": 8, "c64": 8, "c128": 16}


def listed():
    return [
        # two neighbouring sites of a small MPS merged: the call of an interactive user, all latency
        {"name": "contract small c128", "kind": "contract", "dtype": "c128", "l": 16, "m": 16, "r": 16, "d": 2, "mixed": False},
        # the same at the bonds of an applied MPS (256 x 3), single precision, the first site in the
        # [phys, right, left] order that a right canonisation leaves
        {"name": "contract large c64", "kind": "contract", "dtype": "c64", "l": 768, "m": 768, "r": 256, "d": 2, "mixed": True},
        # a real double-precision merge at odd bonds
        {"name": "contract odd f64", "kind": "contract", "dtype": "f64", "l": 171, "m": 203, "r": 97, "d": 3, "mixed": True},
        # one environment update <bra|MPO|ket>, as energies and variational updates make it at every site
        {"name": "con environment c64", "kind": "con", "dtype": "c64", "chi": 256, "D": 3, "d": 2},
        # the QR of the left sweep at the bulk of a chi = 256, D = 3 apply + compress
        {"name": "qr site c64", "kind": "qr", "dtype": "c64", "d": 2, "l": 768, "r": 768},
        # a ragged double-precision canonisation step
        {"name": "qr odd f64", "kind": "qr", "dtype": "f64", "d": 3, "l": 85, "r": 85},
        # splitting a two-site tensor of a small chain
        {"name": "svd small f64", "kind": "svd", "dtype": "f64", "d": 2, "l": 32, "r": 32, "chi": 32},
        # the split after a two-site gate at bond 128, complex double precision
        {"name": "svd gate c128", "kind": "svd", "dtype": "c128", "d": 2, "l": 128, "r": 128, "chi": 128},
        # a whole MatrixProductState.svd_compress, bond 32 to 16
        {"name": "svd_compress f64", "kind": "compress", "dtype": "f64", "N": 16, "d": 2, "chi": 32, "to": 16},
        # MPO application alone at large bonds (XXZ D = 5, float32): moving data
        {"name": "mpo apply f32", "kind": "mpo", "dtype": "f32", "N": 8, "d": 2, "chi": 512, "D": 5},
        # the headline sweep, mixed precision, on a short chain, and the fidelity of what it kept
        {"name": "sweep mixed c64", "kind": "sweep", "precision": "mixed", "N": 20, "chi": 256},
        # independent uneven states on worker streams: left-canonise, compress to chi / 2, norm
        {"name": "uneven queue", "kind": "queue", "count": 8, "N": 24, "chi": 96, "specs": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["contract", "con", "qr", "svd", "compress", "mpo", "sweep", "queue"])
    dtype = rng.choice(["f32", "f64", "c64", "c128"])
    single = dtype in ("f32", "c64")
    if kind == "contract":
        top = 768 if single else 320
        return {"kind": kind, "dtype": dtype, "l": _log(rng, 8, top), "m": _log(rng, 8, top), "r": _log(rng, 8, top),
                "d": rng.choice([2, 3, 4]), "mixed": rng.random() < 0.5}
    if kind == "con":
        return {"kind": kind, "dtype": dtype, "chi": _log(rng, 8, 320 if single else 128), "D": rng.choice([2, 3, 5]),
                "d": rng.choice([2, 3])}
    if kind == "qr":
        top = 640 if single else 256
        return {"kind": kind, "dtype": dtype, "d": rng.choice([2, 3, 4]), "l": _log(rng, 8, top), "r": _log(rng, 8, top)}
    if kind == "svd":
        d, l, r = rng.choice([2, 3]), _log(rng, 6, 96), _log(rng, 6, 96)
        # single-precision splits keep every value (a cut through a dense spectrum is not determined at that precision)
        return {"kind": kind, "dtype": dtype, "d": d, "l": l, "r": r, "chi": 0 if single else max(2, min(l, r) * d // 2)}
    if kind == "compress":
        d = rng.choice([2, 3, 4])
        chi = _log(rng, 6, 48)
        return {"kind": kind, "dtype": rng.choice(["f64", "c128"]), "N": rng.randint(5, {2: 16, 3: 10, 4: 8}[d]), "d": d,
                "chi": chi, "to": max(2, chi // 2)}
    if kind == "mpo":
        return {"kind": kind, "dtype": dtype, "N": rng.randint(3, 8), "d": rng.choice([2, 3]),
                "chi": _log(rng, 16, 400 if dtype == "f32" else 256 if dtype != "c128" else 160), "D": rng.choice([2, 3, 5])}
    if kind == "sweep":
        precision = rng.choice(["mixed", "mixed", "fp32", "fp64"])
        return {"kind": kind, "precision": precision, "N": rng.randint(6, 20), "chi": _log(rng, 12, 64 if precision == "fp64" else 224)}
    return {"kind": kind, "count": rng.randint(3, 8), "N": rng.randint(8, 24), "chi": _log(rng, 16, 96), "specs": rng.randrange(1 << 20)}


# ---------------------------------------------------------------- inputs


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, shape, dtype):
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


def _mps(g, N, d, chi, dtype):
    """Random sites (phys, left, right) with normal entries, scaled so that the state's norm stays near one."""
    out = []
    for i in range(N):
        a = _randn(g, (d, chi if i else 1, chi if i < N - 1 else 1), dtype)
        out.append(a * (math.sqrt(a.shape[2]) / torch.linalg.vector_norm(a)))
    return out


def _mpo(g, N, d, D, dtype):
    return [_randn(g, (d, d, D if i else 1, D if i < N - 1 else 1), dtype) for i in range(N)]


def _tfim(N, dtype, J=1.0, h=0.5):
    """-J sum Z Z - h sum X as lower-triangular sites (physout, physin, left, right)."""
    eye, X, Z = torch.eye(2), torch.tensor([[0.0, 1.0], [1.0, 0.0]]), torch.diag(torch.tensor([1.0, -1.0]))
    W = torch.zeros(3, 3, 2, 2)
    W[0, 0], W[1, 0], W[2, 0], W[2, 1], W[2, 2] = eye, Z, -h * X, -J * Z, eye
    W = W.permute(2, 3, 0, 1).to("cuda", dtype)
    return [W[:, :, 2 * (i == 0):, :1 if i == N - 1 else 3].contiguous() for i in range(N)]


def _two_site(g, case):
    """A two-site tensor (left, p, q, right) whose values fall off exponentially, as those of a state near its
    ground state do: ratio e^-10 from the largest to the smallest."""
    wide = _WIDE[case["dtype"]]
    m, n = case["l"] * case["d"], case["d"] * case["r"]
    k = min(m, n)
    u = torch.linalg.qr(_randn(g, (m, k), wide))[0]
    v = torch.linalg.qr(_randn(g, (n, k), wide))[0]
    s = torch.exp(-10.0 * torch.arange(k, device="cuda", dtype=torch.float64) / k)
    return ((u * s) @ v.conj().T).to(_DTYPE[case["dtype"]]).reshape(case["l"], case["d"], case["d"], case["r"])


def _specs(case):
    """(N, d, chi, dtype) of every state of an uneven queue."""
    r = random.Random(case["specs"])
    return [(r.randint(max(4, case["N"] // 4), case["N"]), r.choice([2, 3, 4]), r.randint(max(8, case["chi"] // 8), case["chi"]),
             "c64" if b % 2 else "f32") for b in range(case["count"])]


def _inputs(case, seed):
    """The plain device arrays of a case."""
    g, kind = _gen(seed), case["kind"]
    dt = _DTYPE.get(case.get("dtype"))
    if kind == "contract":
        l, m, r, d = case["l"], case["m"], case["r"], case["d"]
        return [_randn(g, (d, m, l) if case["mixed"] else (l, d, m), dt), _randn(g, (m, d, r), dt)]
    if kind == "con":
        chi, D, d = case["chi"], case["D"], case["d"]
        return [_randn(g, s, dt) for s in ((chi, D, chi), (chi, d, chi), (D, d, d, D), (chi, d, chi))]
    if kind == "qr":
        return [_randn(g, (case["d"], case["l"], case["r"]), dt)]
    if kind == "svd":
        return [_two_site(g, case)]
    if kind == "compress":
        return _mps(g, case["N"], case["d"], case["chi"], dt)
    if kind == "mpo":
        return [_mps(g, case["N"], case["d"], case["chi"], dt), _mpo(g, case["N"], case["d"], case["D"], dt)]
    if kind == "sweep":
        dt = engine.compute_dtype(case["precision"], True)
        return [_mps(g, case["N"], 2, case["chi"], dt), _tfim(case["N"], dt)]
    return [_mps(g, N, d, chi, _DTYPE[t]) for N, d, chi, t in _specs(case)]


_SITE = ["phys", "left", "right"]


def prepare(case, seed):
    x, kind = _inputs(case, seed), case["kind"]
    state = {"case": case}
    if kind == "contract":
        state["a"] = tn.Tensor(x[0], ["phys", "right", "left"] if case["mixed"] else ["left", "phys", "right"])
        state["b"] = tn.Tensor(x[1], ["left2", "phys2", "right2"])
    elif kind == "con":
        labels = (["ea", "ew", "eb"], ["kl", "kp", "kr"], ["wl", "wo", "wi", "wr"], ["bl", "bp", "br"])
        state["tensors"] = [tn.Tensor(t, list(lb)) for t, lb in zip(x, labels)]
    elif kind == "qr":
        state["a"] = tn.Tensor(x[0], list(_SITE))
    elif kind == "svd":
        state["a"] = tn.Tensor(x[0], ["left", "p", "q", "right"])
    elif kind == "compress":
        state["psi"] = tn.onedim.MatrixProductState([tn.Tensor(t, list(_SITE)) for t in x])
    elif kind == "mpo":
        state["psi"] = tn.onedim.MatrixProductState([tn.Tensor(t, list(_SITE)) for t in x[0]])
        state["mpo"] = tn.onedim.MatrixProductOperator([tn.Tensor(t, ["physout", "physin", "left", "right"]) for t in x[1]])
    elif kind == "sweep":
        state["sites"], state["mpo"] = x
    else:
        state["states"] = x
        state["streams"] = [torch.cuda.Stream() for _ in range(4)]
    return state


# ---------------------------------------------------------------- one pass


def _densities(sites):
    """One-site density matrices, normalised, of a right-canonical state: its left environment taken along the chain."""
    env, out = None, []
    for a in sites:
        ket, bra = tn.Tensor(a, ["p", "l", "r"]), tn.conjugate(tn.Tensor(a, ["q", "m", "s"]))
        if env is None:
            env = tn.Tensor(torch.eye(1, dtype=a.dtype, device=a.device), ["m", "l"])
        half = tn.contract(env, ket, "l", "l")  # m, p, r
        rho = tn.contract(half, bra, ["m", "r"], ["m", "s"])  # p, q
        out.append(rho.data)
        bra.replace_label(["q"], ["p"])
        env = tn.contract(bra, half, ["m", "p"], ["m", "p"])  # s, r
        env.replace_label(["s", "r"], ["m", "l"])
    rho = torch.stack(out)
    return rho / torch.diagonal(rho, dim1=1, dim2=2).sum(1)[0].real


def _compress_one(sites, chi):
    """left-canonise + svd_compress(chi), and the norm of what comes out."""
    stats = engine.SweepStats()
    out, log_norm = engine.compress(sites, chi, stats=stats, fold_norm=False)
    mantissa, scale = engine.inner_product(out, out, log_scale=True)
    return out, stats, log_norm, mantissa.real, scale


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "contract":
        return tn.contract(state["a"], state["b"], "right", "left2").data
    if kind == "con":
        return tn.con(*state["tensors"], ("eb", "kl"), ("ew", "wl"), ("kp", "wi"), ("ea", "bl"), ("wo", "bp")).data
    if kind == "qr":
        q, r = tn.tensor.tensor_qr(state["a"], ["phys", "left"])
        return q.data, r.data
    if kind == "svd":
        if case["chi"]:
            u, v, cut = tn.truncated_svd(state["a"], ["left", "p"], chi=case["chi"])
            return tn.contract(u, v, "svd_in", "svd_out").data, cut
        u, s, v = tn.tensor_svd(state["a"], ["left", "p"])
        return tn.contract(tn.contract(u, s, "svd_in", "svd_out"), v, "svd_in", "svd_out").data, s.data
    if kind == "compress":
        psi = state["psi"].copy()
        psi.svd_compress(chi=case["to"])
        whole = tn.onedim.contract_virtual_indices(psi, 0, case["N"], periodic_boundaries=False)
        return whole.data, np.array(psi.bonddims(), dtype=np.int64)
    if kind == "mpo":
        return [t.data for t in tn.onedim.contract_mps_mpo(state["psi"], state["mpo"])]
    if kind == "sweep":
        real = np.float64 if case["precision"] == "fp64" else np.float32
        stats = engine.SweepStats()
        out = engine.apply_compress_native(state["sites"], state["mpo"], case["chi"], stats=stats,
                                           core=engine.mixed_core(case["precision"]))
        fidelity = engine.fidelity(engine.apply_mpo(state["sites"], state["mpo"]), out)
        return {"bonds": np.array(stats.bonds, dtype=np.int64), "kept": np.array([1.0 - x for x in stats.discarded], dtype=real),
                "log_norm": np.array(stats.log_norm, dtype=real), "fidelity": np.array(fidelity, dtype=real),
                "densities": _densities(out) if real is np.float64 else None}
    jobs = [(lambda s=s, c=max(2, chi // 2): _compress_one(s, c))
            for s, (N, d, chi, t) in zip(state["states"], _specs(case))]
    res = engine.run_queue(jobs, 4, streams=state["streams"])
    return {"bonds": np.array([b for r in res for b in r[1].bonds], dtype=np.int64),
            "discarded": np.array([x for r in res for x in r[1].discarded], dtype=np.float32),
            "log_norm": np.array([r[2] for r in res], dtype=np.float32),
            "norm": np.array([r[3] * math.exp(r[4]) for r in res], dtype=np.float32)}


# ---------------------------------------------------------------- what a pass cannot do without


def _bonds(N, d, chi, top=None):
    """Bond dimensions of a chain of bond chi after truncation to ``top``."""
    b = [1] + [chi] * (N - 1) + [1]
    for i in range(1, N):
        b[i] = min(b[i], b[i - 1] * d)
    c = [1] + [chi] * (N - 1) + [1]
    for i in range(N - 1, 0, -1):
        c[i] = min(b[i], c[i + 1] * d, top or chi)
    return b, c


def _compress_flops(N, d, chi, to):
    """QR left sweep and truncating SVD right sweep (2 m n^2 - 2 n^3 / 3 for R and the same to form Q, 6 m n^2 + 20 n^3 for
    a thin SVD, and the absorptions)."""
    full = [1] + [chi] * (N - 1) + [1]
    b, c = _bonds(N, d, chi, to)
    f = 0.0
    for i in range(N - 1):
        m, n = d * b[i], full[i + 1]
        hi, lo = max(m, n), min(m, n)
        f += 4.0 * hi * lo * lo - 4.0 / 3.0 * lo ** 3 + 2.0 * lo * n * d * full[i + 2]
    for i in range(N - 1, 0, -1):
        m, n = d * c[i + 1], b[i]
        hi, lo = max(m, n), min(m, n)
        f += 6.0 * hi * lo * lo + 20.0 * lo ** 3 + 2.0 * d * b[i - 1] * n * c[i]
    sizes = sum(d * full[i] * full[i + 1] + d * c[i] * c[i + 1] for i in range(N))
    return f, sizes


def work(case):
    kind = case["kind"]
    if kind in ("sweep", "queue"):
        if kind == "sweep":
            parts = [(case["N"], 2, case["chi"], "c128" if case["precision"] == "fp64" else "c64", 3, case["chi"])]
        else:
            parts = [(N, d, chi, t, 1, max(2, chi // 2)) for N, d, chi, t in _specs(case)]
        flops = size = 0.0
        for N, d, chi, t, D, to in parts:
            f, s = _compress_flops(N, d, chi * D, to)
            flops += f * (4 if t[0] == "c" else 1)
            read = sum(d * (chi if i else 1) * (chi if i < N - 1 else 1) for i in range(N))
            _, c = _bonds(N, d, chi * D, to)
            size += (read + sum(d * c[i] * c[i + 1] for i in range(N))) * _BYTES[t]
        return {"bytes": size, "flops": flops}
    t = case["dtype"]
    cx, es, d = (4.0 if t[0] == "c" else 1.0), _BYTES[t], case["d"]
    if kind == "contract":
        l, m, r = case["l"], case["m"], case["r"]
        return {"bytes": es * (d * l * m + d * m * r + d * d * l * r), "flops": cx * 2.0 * d * d * l * m * r}
    if kind == "con":
        chi, D = case["chi"], case["D"]
        n = chi * chi
        return {"bytes": es * (2.0 * n * D + 2 * n * d + D * D * d * d), "flops": cx * 2.0 * (2 * n * chi * D * d + n * D * d * D * d)}
    if kind == "qr":
        m, n = d * case["l"], case["r"]
        hi, lo = max(m, n), min(m, n)
        return {"bytes": es * (m * n + m * lo + lo * n), "flops": cx * (4.0 * hi * lo * lo - 4.0 / 3.0 * lo ** 3)}
    if kind == "svd":
        m, n = d * case["l"], d * case["r"]
        hi, lo = max(m, n), min(m, n)
        return {"bytes": es * 2.0 * m * n, "flops": cx * (6.0 * hi * lo * lo + 20.0 * lo ** 3 + 2.0 * m * n * (case["chi"] or lo))}
    if kind == "compress":
        N = case["N"]
        f, size = _compress_flops(N, d, case["chi"], case["to"])
        _, c = _bonds(N, d, case["chi"], case["to"])
        f += sum(2.0 * d ** (i + 1) * c[i] * c[i + 1] for i in range(1, N))
        return {"bytes": es * (size + float(d) ** N), "flops": cx * f}
    b = [1] + [case["chi"]] * (case["N"] - 1) + [1]
    w = [1] + [case["D"]] * (case["N"] - 1) + [1]
    size = flops = 0.0
    for i in range(case["N"]):
        out = d * b[i] * w[i] * b[i + 1] * w[i + 1]
        size += out + d * b[i] * b[i + 1] + d * d * w[i] * w[i + 1]
        flops += 2.0 * d * out
    return {"bytes": es * size, "flops": cx * flops}


# ---------------------------------------------------------------- the same in 64 bits


def _host(t):
    return t.to(torch.complex128 if t.is_complex() else torch.float64).cpu().numpy()


def _compress64(sites, to, threshold=1e-15):
    """QR left sweep, then the truncating SVD sweep from the right, on (phys, left, right) arrays: (sites with the norm in
    the first one, bonds, kept weights, log norm)."""
    P, log_norm = [np.array(a) for a in sites], 0.0
    N = len(P)
    for i in range(N - 1):
        d, l, r = P[i].shape
        q, x = np.linalg.qr(P[i].reshape(d * l, r))
        P[i] = q.reshape(d, l, -1)
        n = np.linalg.norm(x)
        log_norm += math.log(n)
        P[i + 1] = np.einsum("ab,pbc->pac", x / n, P[i + 1], optimize=True)
    n = np.linalg.norm(P[-1])
    log_norm += math.log(n)
    P[-1] = P[-1] / n
    bonds, kept, scale = [], [], 1.0
    for i in range(N - 1, 0, -1):
        d, l, r = P[i].shape
        u, s, v = np.linalg.svd(P[i].transpose(0, 2, 1).reshape(d * r, l), full_matrices=False)
        k = min(int((s / s[0] > threshold).sum()), to)
        bonds.append(k)
        kept.append((float((s[:k] ** 2).sum()), float((s ** 2).sum()), float(s[0])))
        P[i] = u[:, :k].reshape(d, r, k).transpose(0, 2, 1)
        P[i - 1] = np.einsum("pab,kb->pak", P[i - 1], s[:k, None] * v[:k], optimize=True) / s[0]
        scale *= s[0]
    P[0] = P[0] * scale
    return P, bonds[::-1], kept[::-1], log_norm, scale


def exact(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    if kind == "contract":
        a, b = (t.to(_WIDE[case["dtype"]]) for t in x)
        return torch.tensordot(a.permute(0, 2, 1) if case["mixed"] else a, b, ([2], [0]))
    if kind == "con":
        e, k, w, b = (t.to(_WIDE[case["dtype"]]) for t in x)
        # the free labels in the order that the arguments leave them: ket right, MPO right, bra right
        t = torch.tensordot(e, k, ([2], [0]))  # ea ew kp kr
        t = torch.tensordot(t, w, ([1, 2], [0, 2]))  # ea kr wo wr
        return torch.tensordot(t, b, ([0, 2], [0, 1]))  # kr wr br
    if kind == "qr":
        q, r = np.linalg.qr(_host(x[0]).reshape(case["d"] * case["l"], case["r"]))
        return q.reshape(case["d"], case["l"], -1), r
    if kind == "svd":
        a = _host(x[0])
        u, s, v = np.linalg.svd(a.reshape(case["l"] * case["d"], -1), full_matrices=False)
        k = case["chi"] or len(s)
        whole = ((u[:, :k] * s[:k]) @ v[:k]).reshape(a.shape)
        return (whole, s[k:]) if case["chi"] else (whole, np.diag(s).astype(a.dtype))
    if kind == "compress":
        P, bonds, _, log_norm, _ = _compress64([_host(t) for t in x], case["to"])
        v = np.ones((1, 1))
        for a in P:
            v = np.tensordot(v, a, (-1, 1)).reshape(-1, a.shape[2])
        shape = (1,) + (case["d"],) * case["N"] + (1,)
        return v.reshape(shape) * math.exp(log_norm), None
    if kind == "mpo":
        out = []
        for a, w in zip(*x):
            a, w = a.to(_WIDE[case["dtype"]]), w.to(_WIDE[case["dtype"]])
            t = torch.einsum("plr,opab->laorb", a, w)
            l, a_, o, r, b_ = t.shape
            out.append(t.reshape(l * a_, o, r * b_))
        return out
    if kind == "sweep":
        sites = []
        for a, w in zip(*x):
            t = np.einsum("plr,opab->olarb", _host(a), _host(w), optimize=True)
            o, l, a_, r, b_ = t.shape
            sites.append(t.reshape(o, l * a_, r * b_))
        P, _, kept, log_norm, scale = _compress64(sites, case["chi"])
        double = case["precision"] == "fp64"
        env, rho, over, full = np.ones((1, 1)), [], np.ones((1, 1)), np.ones((1, 1))
        for a, w in zip(P, sites):
            w = w / np.linalg.norm(w)
            over = np.einsum("pms,mpr->sr", w.conj(), np.einsum("ml,plr->mpr", over, a, optimize=True), optimize=True)
            full = np.einsum("pms,mpr->sr", w.conj(), np.einsum("ml,plr->mpr", full, w, optimize=True), optimize=True)
            t = np.einsum("ml,plr->mpr", env, a, optimize=True)
            if double:
                rho.append(np.einsum("mpr,qmr->pq", t, a.conj(), optimize=True))
            env = np.einsum("pms,mpr->sr", a.conj(), t, optimize=True)
        fidelity = abs(over.item()) ** 2 / (full.item().real * env.item().real)
        return {"bonds": None, "kept": np.array([a / b for a, b, _ in kept]), "log_norm": np.array(log_norm + math.log(scale)),
                "fidelity": np.array(fidelity), "densities": np.array(rho) / np.trace(rho[0]).real if double else None}
    cut, logs, norms = [], [], []
    for sites, (N, d, chi, t) in zip(x, _specs(case)):
        P, _, k, log_norm, scale = _compress64([_host(a) for a in sites], max(2, chi // 2))
        cut += [(b - a) / s ** 2 for a, b, s in k[::-1]]  # the engine lists its bonds from the right, over the largest value's square
        logs.append(log_norm + math.log(scale))
        norms.append((np.linalg.norm(P[0]) / scale) ** 2)
    return {"bonds": None, "discarded": np.array(cut), "log_norm": np.array(logs), "norm": np.array(norms)}
