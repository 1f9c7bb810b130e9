"""Timed cases of the library: what its users call, over the sizes they call it with.

Every case goes through the public Python layer (`ttcuda`), which marshals to the C entry points a
Julia program binds.  The one-shot methods take host tensors and return host tensors; the batched
roundings work on TTs resident on the GPU and return TTs to page-locked host memory.

A truncated-SVD rounding defines its cores up to the signs of the singular vectors, so the cases
that round this way go on as a solver does, to the next step, whose result does not depend on these
signs: a single TT is orthogonalised at its other end, a basis is compressed to a fixed rank (below
its TTs' ranks: the compressed TTs then depend on the large singular values).

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call
    run(state)          one pass, and everything it computes
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the result in 64 bits without the library (None for a whole basis, and where
                        the sketch has reduced precision)
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "tensor-train-julia_b200"))


def _lib():
    import ttcuda
    return ttcuda


# ------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call of a solver's inner loop: a sum of three short TTs rounded
        {"name": "round_small", "kind": "round", "d": 12, "n": 2, "terms": 3, "rank": 5, "tol": 1e-10, "rmax": 16384,
         "right": False},
        # a linear combination of 8 rank-8 TTs rounded after the additions
        {"name": "round_sum", "kind": "round", "d": 20, "n": 2, "terms": 8, "rank": 8, "tol": 1e-8, "rmax": 64,
         "right": False},
        # the same from the other side, odd ranks and mode size, rank-limited
        {"name": "round_right", "kind": "round", "d": 17, "n": 3, "terms": 3, "rank": 37, "tol": 1e-10, "rmax": 51,
         "right": True},
        # one large TT, as a solution that is kept at full accuracy
        {"name": "round_large", "kind": "round", "d": 28, "n": 2, "terms": 2, "rank": 124, "tol": 1e-8, "rmax": 16384,
         "right": False},
        # a Krylov basis kept on the GPU, uneven ranks: rounded to a tolerance, compressed to rank 24
        # for the next cycle and read back
        {"name": "batch_det", "kind": "batch", "count": 60, "d": 32, "n": 2, "rlo": 48, "rhi": 256, "tol": 1e-8,
         "rmax": 16384, "sketch": 0, "precision": "fp64", "next": 24},
        # the same basis rounded to rank 64 with a BF16 sketch first
        {"name": "batch_rand_bf16", "kind": "batch", "count": 60, "d": 32, "n": 2, "rlo": 48, "rhi": 256, "tol": 1e-8,
         "rmax": 64, "sketch": 64, "precision": "bf16", "next": 24},
        # operator times TT rounded without forming the product: a nearest-neighbour chain
        {"name": "op_round", "kind": "op_round", "d": 32, "n": 2, "r": 128, "R": 6, "s": 138, "precision": "fp64"},
        # the same with a long-range operator and the sketch in BF16
        {"name": "op_round_bf16", "kind": "op_round", "d": 24, "n": 2, "r": 320, "R": 64, "s": 320,
         "precision": "bf16"},
        # operator times TT, formed
        {"name": "apply", "kind": "apply", "d": 32, "n": 2, "r": 96, "R": 6},
        # energy gradient of a variational step, in both precisions
        {"name": "grad_fp64", "kind": "grad", "d": 32, "n": 2, "r": 192, "R": 18, "ckpt": 4, "precision": "fp64"},
        {"name": "grad_fp32", "kind": "grad", "d": 32, "n": 2, "r": 192, "R": 18, "ckpt": 4, "precision": "fp32"},
        # an inner product and its interface matrices, as the Gram matrix of a basis needs them
        {"name": "interfaces", "kind": "interfaces", "d": 32, "n": 2, "ra": 128, "rb": 77},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["round", "round", "batch", "batch", "op_round", "op_round", "apply", "grad", "grad",
                       "interfaces"])
    n = rng.choice([2, 2, 2, 3, 4])
    if kind == "round":
        terms = rng.randint(2, 8)
        return {"kind": kind, "d": rng.randint(8, 28), "n": n, "terms": terms,
                "rank": max(1, _log_int(rng, 8, 240 if n == 2 else 160) // terms), "tol": rng.choice([1e-10, 1e-8, 1e-6]),
                "rmax": rng.choice([16384, 64, 33]), "right": rng.random() < 0.4}
    if kind == "batch":
        rhi = _log_int(rng, 24, 240)
        rand = rng.random() < 0.5
        rlo = max(6, rhi // rng.choice([1, 2, 8]))
        rank = _log_int(rng, 8, max(9, rhi // 2))
        return {"kind": kind, "count": _log_int(rng, 2, 56), "d": rng.randint(10, 32), "n": 2 if rhi > 160 else n,
                "rlo": rlo, "rhi": rhi, "tol": rng.choice([1e-8, 1e-6]),
                "rmax": rank if rand else rng.choice([16384, rank]), "sketch": rank if rand else 0,
                "precision": rng.choice(["fp64", "bf16", "tf32"]) if rand else "fp64", "next": rng.randint(3, max(3, min(rlo, rank) // 2))}
    if kind == "op_round":
        R = _log_int(rng, 3, 60)
        r = _log_int(rng, 16, 300 if R < 16 else 200)
        return {"kind": kind, "d": rng.randint(10, 32 if R < 24 else 24), "n": n if r * R < 4000 else 2, "r": r, "R": R,
                "s": min(360, r + rng.randint(0, 10)), "precision": rng.choice(["fp64", "fp64", "bf16", "tf32"])}
    if kind == "apply":
        R = _log_int(rng, 3, 12)
        return {"kind": kind, "d": rng.randint(10, 32), "n": n, "r": _log_int(rng, 8, 600 // (R * n) if R * n < 60 else 9),
                "R": R}
    if kind == "grad":
        return {"kind": kind, "d": rng.randint(10, 30), "n": n, "r": _log_int(rng, 12, 180 // (n - 1)),
                "R": _log_int(rng, 4, 18), "ckpt": rng.choice([1, 4, 7]), "precision": rng.choice(["fp64", "fp32"])}
    return {"kind": kind, "d": rng.randint(8, 40), "n": n, "ra": _log_int(rng, 8, 256), "rb": _log_int(rng, 8, 256)}


# ------------------------------------------------------------------------------------- the inputs
def _clamp(ranks, d, n):
    """Bond ranks no larger than the dimension on either side."""
    return [min(r, n ** min(k, d - k, 30)) for k, r in enumerate(ranks)]


def _gauss(g, d, n, ranks, decay=None):
    """Cores (n, r_{k-1}, r_k) with N(0,1) entries scaled to interfaces of norm about one; with
    `decay`, the singular values of a bond fall like 10^(-i/decay)."""
    out, prev = [], np.ones(1)
    for k in range(d):
        c = g.standard_normal((ranks[k + 1], ranks[k], n)).T / math.sqrt(n * ranks[k])
        out.append(c if decay is None else np.asfortranarray(c * prev[None, :, None]))
        if decay is not None:
            prev = 10.0 ** (-np.arange(ranks[k + 1]) / decay)
            prev /= math.sqrt(np.mean(prev ** 2))
    return out


def _sum_cores(g, case):
    """Direct sum of `terms` TTs of rank `rank`, term j scaled by 2^-j (the cores tt_add gives)."""
    d, n, m, r = case["d"], case["n"], case["terms"], case["rank"]
    parts = [_gauss(g, d, n, _clamp([1] + [r] * (d - 1) + [1], d, n)) for _ in range(m)]
    ranks = [1] + [sum(p[k].shape[2] for p in parts) for k in range(d - 1)] + [1]
    out = []
    for k in range(d):
        c = np.zeros((n, ranks[k], ranks[k + 1]), order="F")
        a = b = 0
        for j, p in enumerate(parts):
            q = p[k] * (2.0 ** -j if k == 0 else 1.0)
            c[:, a:a + q.shape[1], b:b + q.shape[2]] = q
            a += q.shape[1] if k > 0 else 0
            b += q.shape[2] if k < d - 1 else 0
        out.append(c)
    return out, ranks


def _operator(g, case, symmetric=False):
    """MPO cores (n, n, R_{k-1}, R_k) of rank up to R, of norm about one."""
    d, n, R = case["d"], case["n"], case["R"]
    rk = [min(R, n ** (2 * min(k, d - k, 15))) for k in range(d + 1)]
    out = []
    for k in range(d):
        c = g.standard_normal((rk[k + 1], rk[k], n, n)).T / math.sqrt(n * rk[k])
        out.append(np.asfortranarray((c + c.transpose(1, 0, 2, 3)) / math.sqrt(2.0)) if symmetric else c)
    return out, rk


def _ranks(case, r):
    d, n = case["d"], case["n"]
    return _clamp([1] + [r] * (d - 1) + [1], d, n)


def _batch_ranks(case):
    """Rank lists of the basis: interior ranks drawn from [rlo, rhi] for every TT and bond."""
    d, n = case["d"], case["n"]
    g = np.random.default_rng([case["rlo"], case["rhi"], d])
    return [_clamp([1] + [int(v) for v in g.integers(case["rlo"], case["rhi"] + 1, d - 1)] + [1], d, n)
            for _ in range(case["count"])]


def _sketch_ranks(case, s):
    """Sketch ranks of a single Gaussian block per bond (block_rks = s): min(s, n^(d-k))."""
    d, n = case["d"], case["n"]
    return [min(s, n ** min(d - k, 30)) for k in range(d + 1)]


def _range_finder_ranks(d, n, rks):
    """Ranks of ttrand_rounding(y, rks) with its default blocks of d columns: whole blocks, as many
    at a bond as at the one before it or more, and at most n times the left neighbour's rank."""
    b, p = [d] * d + [1], [1] * (d + 1)
    for k in range(d - 1, -1, -1):
        b[k] = min(b[k], n * b[k + 1])
    for k in range(d):
        p[k] = max(-(-rks[k] // b[k]), p[k - 1] if k else 1)
    out = [1] * (d + 1)
    for k in range(d - 1):
        out[k + 1] = min(n * out[k], b[k + 1] * p[k + 1])
    return out


def _inputs(case, seed):
    """The host tensors of a one-shot case, from the seed alone."""
    g = np.random.default_rng([seed, 77])
    k = case["kind"]
    if k == "round":
        return {"x": _sum_cores(g, case)}
    if k in ("op_round", "apply", "grad"):
        r = _ranks(case, case["r"])
        return {"x": (_gauss(g, case["d"], case["n"], r), r), "H": _operator(g, case, symmetric=k == "grad")}
    ra, rb = _ranks(case, case["ra"]), _ranks(case, case["rb"])
    return {"x": (_gauss(g, case["d"], case["n"], ra), ra), "y": (_gauss(g, case["d"], case["n"], rb), rb)}


# ------------------------------------------------------------------------------------- one pass
def prepare(case, seed):
    T = _lib()
    d, n = case["d"], case["n"]
    dims = (n,) * d
    st = {"case": case, "T": T}
    if case["kind"] == "batch":
        g = np.random.default_rng([seed, 78])
        ranks = _batch_ranks(case)
        tts = [T.TTvector(d, _gauss(g, d, n, r, decay=32.0), dims, r) for r in ranks]
        st["x"] = T.DeviceBatch.from_tts(tts)
        if case["sketch"]:
            rks = [1] + [case["sketch"]] * (d - 1) + [1]
            st["rks"], caps = rks, [_range_finder_ranks(d, n, rks)] * case["count"]
        else:
            caps = ranks
        st["y"] = T.DeviceBatch(dims, caps)
        st["next"] = [1] + _sketch_ranks(case, case["next"])[1:]
        caps = [1] * (d + 1)
        for k in range(d - 1):
            caps[k + 1] = min(n * caps[k], st["next"][k + 1])
        st["z"] = T.DeviceBatch(dims, [caps] * case["count"])
        # the page-locked result blocks, allocated (and cleared) once by a program that reads back
        # into the same memory on every pass
        for block in _blocks(st["z"].download(reuse=True)):
            block[:] = 0.0
        return st
    for name, (cores, ranks) in _inputs(case, seed).items():
        st[name] = T.TToperator(d, cores, dims, ranks) if name == "H" else T.TTvector(d, cores, dims, ranks)
    return st


def _blocks(tts):
    """The one host block that holds a downloaded TT's cores, for every TT."""
    out = []
    for t in tts:
        v = t.ttv_vec[0]
        while isinstance(v.base, np.ndarray):
            v = v.base
        out.append(v)
    return out


def run(state):
    T, case = state["T"], state["case"]
    k = case["kind"]
    if k == "round":
        right = case["right"]
        y = T.tt_rounding(state["x"], tol=case["tol"], rmax=case["rmax"], direction="right" if right else "left")
        y = T.orthogonalize(y, 1 if right else case["d"])
        return {"ranks": np.array(y.ttv_rks), "cores": y.ttv_vec}
    if k == "batch":
        if case["sketch"]:
            state["x"].round_rand(state["y"], state["rks"], precision=case["precision"], after_tol=case["tol"],
                                  rmax=case["rmax"])
        else:
            state["x"].round_det(state["y"], tol=case["tol"], rmax=case["rmax"])
        state["y"].round_rand(state["z"], state["next"], block_rks=case["next"])
        tts = state["z"].download(reuse=True)
        return {"ranks": np.array([t.ttv_rks for t in tts]), "cores": _blocks(tts)}
    if k == "op_round":
        y = T.ttrand_rounding_op([1.0], state["H"], [state["x"]], [1] + _sketch_ranks(case, case["s"])[1:],
                                 orthogonal=False, seed=5, block_rks=case["s"], precision=case["precision"])
        return {"cores": y.ttv_vec}
    if k == "apply":
        return {"cores": T.mpo_apply(state["H"], state["x"]).ttv_vec}
    if k == "grad":
        value, grads = T.rayleigh_grad(state["H"], state["x"], ckpt_every=case["ckpt"], precision=case["precision"])
        return {"value": value, "grads": grads}
    return {"dot": T.dot(state["x"], state["y"]), "w": T.partial_contraction(state["x"], state["y"])}


# ------------------------------------------------------------------------------------- its work
def _svd_sweep(d, n, rp, out):
    """Operations of the right-to-left truncated-SVD sweep over ranks rp keeping the ranks `out`:
    the SVD of an r x (n r') unfolding by way of its triangular factor, and the product with the
    neighbouring core."""
    f = 0.0
    for j in range(d - 1, 0, -1):
        q, p = rp[j], n * out[j + 1]
        m, k = max(p, q), min(p, q)
        f += 2.0 * m * k * k - 2.0 * k ** 3 / 3 + 12.0 * k ** 3 + 4.0 * m * k * out[j] + 2.0 * rp[j - 1] * n * q * out[j]
    return f


def _qr(m, k):
    return 4.0 * m * k * k - 4.0 * k ** 3 / 3


def work(case):
    d, n, k = case["d"], case["n"], case["kind"]
    if k == "round" or k == "batch":
        if k == "round":
            r = [1] + [0] * (d - 1) + [1]
            for j in range(1, d):
                r[j] = case["terms"] * min(case["rank"], n ** min(j, d - j, 30))
            lists = [r]
        else:
            lists = _batch_ranks(case)
        byt = flo = 0.0
        for r in lists:
            e = [1] * (d + 1)     # ranks after the left-to-right sweep
            for j in range(d - 1):
                e[j + 1] = min(n * e[j], r[j + 1], case.get("sketch") or r[j + 1])
                flo += 2.0 * e[j] * n * r[j] * r[j + 1] + _qr(max(n * e[j], e[j + 1]), e[j + 1])
                if case.get("sketch"):
                    flo += 4.0 * n * r[j] * r[j + 1] * e[j + 1] + 4.0 * e[j] * n * r[j + 1] * e[j + 1]
            o = [1] * (d + 1)     # kept ranks
            for j in range(d - 1, 0, -1):
                o[j] = min(n * o[j + 1], e[j], case["rmax"])
            flo += _svd_sweep(d, n, e, o)
            z = o
            if k == "round":      # orthogonalised at the other end
                flo += sum(2.0 * n * o[j] ** 2 * o[j + 1] + _qr(max(n * o[j], o[j + 1]), o[j + 1]) for j in range(d - 1))
            else:                 # compressed to the next rank
                z = [1] * (d + 1)
                for j in range(d - 1):
                    z[j + 1] = min(n * z[j], o[j + 1], _sketch_ranks(case, case["next"])[j + 1])
                    flo += _qr(max(n * z[j], z[j + 1]), z[j + 1]) + 2.0 * n * z[j] * o[j] * o[j + 1]
                    flo += 4.0 * n * o[j] * o[j + 1] * z[j + 1] + 4.0 * n * z[j] * o[j + 1] * z[j + 1]
            byt += 8.0 * n * sum(r[j] * r[j + 1] + z[j] * z[j + 1] for j in range(d))
        return {"bytes": byt, "flops": flo}
    if k in ("op_round", "apply", "grad"):
        r = _ranks(case, case["r"])
        R = [min(case["R"], n ** (2 * min(j, d - j, 15))) for j in range(d + 1)]
        byt = 8.0 * sum(n * r[j] * r[j + 1] + n * n * R[j] * R[j + 1] for j in range(d))
        if k == "apply":
            out = sum(n * r[j] * r[j + 1] * R[j] * R[j + 1] for j in range(d))
            return {"bytes": byt + 8.0 * out, "flops": 2.0 * n * out}

        def env(a, b, g, a1, b1, g1):   # (a, b, g) from (a1, b1, g1) through a TT, an MPO and a TT core
            return 2.0 * n * (a * a1 * b1 * g1 + n * a * g1 * b * b1 + a * b * g1 * g)
        if k == "grad":
            flo = sum(3 * env(r[j], R[j], r[j], r[j + 1], R[j + 1], r[j + 1]) + 12.0 * n * r[j] * r[j + 1] * r[j]
                      for j in range(d))
            return {"bytes": byt + 8.0 * n * sum(r[j] * r[j + 1] for j in range(d)), "flops": flo}
        s = _sketch_ranks(case, case["s"])
        rho, flo = [1] * (d + 1), 0.0
        for j in range(d - 1):
            rho[j + 1] = min(n * rho[j], s[j + 1])
        for j in range(d):
            flo += env(r[j], R[j], s[j], r[j + 1], R[j + 1], s[j + 1])
            if j + 1 < d:
                q, m = r[j + 1] * R[j + 1], n * rho[j]
                flo += 4.0 * m * q * rho[j + 1] + _qr(max(m, rho[j + 1]), rho[j + 1])
                flo += 2.0 * rho[j + 1] * n * (q * r[j + 2] + n * r[j + 2] * R[j + 1] * R[j + 2])
        return {"bytes": byt + 8.0 * n * sum(rho[j] * rho[j + 1] for j in range(d)), "flops": flo}
    a, b = _ranks(case, case["ra"]), _ranks(case, case["rb"])
    byt = 8.0 * n * sum(a[j] * a[j + 1] + b[j] * b[j + 1] for j in range(d))
    return {"bytes": 2 * byt + 8.0 * sum(a[j] * b[j] for j in range(d + 1)),
            "flops": 2 * sum(2.0 * n * (a[j] * a[j + 1] * b[j + 1] + a[j] * b[j] * b[j + 1]) for j in range(d))}


# ------------------------------------------------------------------------------------- in 64 bits
def _normals(seed, stream, count):
    """Philox4x32-10 (Salmon et al., SC'11) and Box-Muller: the library's sketch entries."""
    q = np.arange((count + 3) // 4, dtype=np.uint64)
    mask = np.uint64(0xFFFFFFFF)
    c = [q & mask, np.full_like(q, stream), np.zeros_like(q), np.zeros_like(q)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = [(v.astype(np.float64) + 0.5) / 2.0 ** 32 for v in c]
    z = []
    for i in (0, 2):
        rad, ang = np.sqrt(-2.0 * np.log(u[i])), 2.0 * np.pi * u[i + 1]
        z += [rad * np.cos(ang), rad * np.sin(ang)]
    return np.stack(z, 1).reshape(-1)[:count]


def _range_finder(case, seed, y0, interface, step):
    """Left-to-right orthogonalise-and-project sweep: Z = Y W_{k+1}, core k = Q of Z's Householder
    QR, Y <- Q^T Y A_{k+1}.  `interface`: the sketch (q_k, s_k) of every bond; `step(k, P)`: Y of
    site k from P (rho, q_k)."""
    d, n = case["d"], case["n"]
    dev = y0.device
    s = _sketch_ranks(case, case["s"])
    S = [torch.from_numpy(_normals(seed, k, s[k + 1] * n * s[k]) / math.sqrt(s[k])).to(dev)
         .reshape(s[k], n, s[k + 1]).permute(2, 1, 0) for k in range(d)]
    W = interface(S)
    out, Y, rho = [], y0, 1
    for k in range(d - 1):                                   # Y: (rho, n, q); rows with rho fastest
        m = Y.permute(1, 0, 2).reshape(n * rho, -1)
        Q = torch.linalg.qr((m @ W[k + 1]).cpu())[0].to(dev)
        out.append(Q.reshape(n, rho, -1))
        rho = Q.shape[1]
        Y = step(k + 1, Q.T @ m)
    out.append(Y.reshape(rho, n, 1).permute(1, 0, 2))
    return [c.cpu().numpy() for c in out]


def _orth_left(v):
    """Left-orthogonal cores 1 .. d-1 by Householder QR, unfolding rows with the rank index fastest."""
    v = list(v)
    for j in range(len(v) - 1):
        n, a, b = v[j].shape
        q, r = np.linalg.qr(v[j].reshape(n * a, b))
        v[j] = q.reshape(n, a, -1)
        v[j + 1] = np.einsum("pa,iab->ipb", r, v[j + 1])
    return v


def _orth_right(v):
    """Right-orthogonal cores 2 .. d by Householder QR of the transposed unfoldings."""
    v = list(v)
    for j in range(len(v) - 1, 0, -1):
        n, a, b = v[j].shape
        q, r = np.linalg.qr(v[j].transpose(2, 0, 1).reshape(b * n, a))
        v[j] = q.reshape(b, n, -1).transpose(1, 2, 0)
        v[j - 1] = np.einsum("iab,pb->iap", v[j - 1], r)
    return v


def _exact_round(case, seed):
    """Orthogonalisation sweep, truncated-SVD sweep back (the tail of each bond below tol times its
    norm, then rmax), orthogonalisation again; from the right, on the mirror image."""
    right = case["right"]
    v = _inputs(case, seed)["x"][0]
    if right:
        v = [c.transpose(0, 2, 1) for c in reversed(v)]
    v = _orth_left(v)
    for j in range(len(v) - 1, 0, -1):
        n, a, b = v[j].shape
        u, s, w = np.linalg.svd(v[j].transpose(1, 0, 2).reshape(a, n * b), full_matrices=False)
        tail = np.cumsum(s[::-1] ** 2)[::-1]
        keep = min(max(1, int(np.sum(tail >= case["tol"] ** 2 * tail[0]))), case["rmax"], int(np.sum(s > 0)))
        v[j] = w[:keep].reshape(keep, n, b).transpose(1, 0, 2)
        v[j - 1] = np.einsum("iab,bp->iap", v[j - 1], u[:, :keep] * s[:keep])
    if right:
        v = _orth_right([c.transpose(0, 2, 1) for c in reversed(v)])
    else:
        v = _orth_left(v)
    return {"ranks": np.array([c.shape[1] for c in v] + [1]), "cores": v}


def exact(case, seed):
    k = case["kind"]
    if k == "batch" or (k == "op_round" and case["precision"] != "fp64"):
        return None
    if k == "round":
        return _exact_round(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    d, n = case["d"], case["n"]
    given = _inputs(case, seed)
    t = {name: [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in v[0]] for name, v in given.items()}
    one = torch.ones(1, 1, dtype=torch.float64, device=dev)
    x = t["x"]
    if k == "apply":
        return {"cores": [torch.einsum("ijab,jcd->iacbd", h, c).permute(0, 2, 1, 4, 3)
                          .reshape(n, h.shape[2] * c.shape[1], -1).cpu().numpy() for h, c in zip(t["H"], x)]}
    if k == "interfaces":
        w = [one]
        for a, b in zip(reversed(x), reversed(t["y"])):
            w.append(torch.einsum("zab,zcb->ac", torch.einsum("zab,bd->zad", a, w[-1]), b))
        w = [v.cpu().numpy() for v in reversed(w)]
        return {"dot": float(w[0][0, 0]), "w": w}
    if k == "grad":
        H = t["H"]
        L, Ln = [one.reshape(1, 1, 1)], [one]
        for c, h in zip(x, H):
            v = torch.einsum("abc,jcf->abjf", L[-1], c)
            v = torch.einsum("abjf,ijbe->aief", v, h)
            L.append(torch.einsum("iad,aief->def", c, v))
            Ln.append(torch.einsum("iad,ac,icf->df", c, Ln[-1], c))
        e, nn = float(L[-1][0, 0, 0]), float(Ln[-1][0, 0])
        R, Rn, grads = one.reshape(1, 1, 1), one, [None] * d
        for j in range(d - 1, -1, -1):
            c, h = x[j], H[j]
            u = torch.einsum("jcf,def->cjde", c, R)
            u = torch.einsum("cjde,ijbe->bcid", u, h)
            grads[j] = (2.0 / nn) * (torch.einsum("abc,bcid->iad", L[j], u) -
                                     (e / nn) * torch.einsum("ac,icf,df->iad", Ln[j], c, Rn))
            R = torch.einsum("iad,bcid->abc", c, u)
            Rn = torch.einsum("iad,icf,df->ac", c, c, Rn)
        return {"value": e / nn, "grads": [v.cpu().numpy() for v in grads]}
    H = t["H"]

    def interface(S):
        W = [None] * d + [one.reshape(1, 1, 1)]
        for j in range(d - 1, -1, -1):
            v = torch.einsum("zae,ebg->zabg", x[j], W[j + 1])
            v = torch.einsum("zabg,yzcb->acyg", v, H[j])
            W[j] = torch.einsum("acyg,gys->acs", v, S[j])
        return [w.reshape(-1, w.shape[2]) for w in W]

    def step(j, P):                                          # P: (rho, a, b)
        v = torch.einsum("pab,zae->pbze", P.reshape(P.shape[0], x[j].shape[1], -1), x[j])
        return torch.einsum("pbze,yzbc->pyec", v, H[j]).reshape(P.shape[0], n, -1)
    return {"cores": _range_finder(case, 5, step(0, one), interface, step)}
