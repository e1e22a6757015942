"""Performance cases of the two-site DMRG engine, through its public entry points.

Kinds of case (the ``kind`` field):

  matvec  one H_eff application on device-resident operands
          (``dmrg2_op_heff_noalloc``): what a program that drives its own
          eigensolver calls, and the inner step of every sweep
  bond    one two-site ground-state solve (``dmrg2.optimize_two_site``), host arrays
  split   one truncated split of theta (``dmrg2.truncated_svd``), host arrays
  env     one left and one right environment update (``dmrg2.update_*_env``), host arrays
  solve   a whole solve from a seeded MPS: set_mps, run with a chi ramp, energy,
          the local magnetisation or charge, and the MPS
  sweep   one further full sweep (left-to-right and back) at the bond cap on an engine
          that a ramp has brought there (``resume``): the steady state of a long run
  batch   several independent solves through ``dmrg2.Server``

The models are those of ``dmrg2.models``: XXZ (d = 2, D = 5), J1-J2 (d = 2, D = 8) and the
complex Josephson array (d = 2 n_max + 1, D = 4). Chains carry weak seeded on-site terms,
so that local expectation values are not zero by symmetry and another seed is another
problem.

A returned MPS is defined up to its bond gauge, so solves of short chains return the state
vector it stands for (with its largest entry real and positive) and the large sweeps return the
energy and the local expectation values. Splits return left and right with the phase of each
singular pair fixed by the largest entry of the left vector.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dmrg-implementations_b200"))
import dmrg2  # noqa: E402
from dmrg2 import models  # noqa: E402


# ----------------------------------------------------------------------------- cases
def listed():
    return [
        # a bond near the end of a chain: small matrices, launches and latency
        {"name": "matvec_edge", "kind": "matvec", "model": "xxz", "cL": 8, "cR": 16, "n_max": 0},
        # a bond of a J1-J2 chain whose kept dimensions the cutoff left ragged
        {"name": "matvec_j1j2", "kind": "matvec", "model": "j1j2", "cL": 171, "cR": 187, "n_max": 0},
        # the bulk bond of the benchmark chain (XXZ, chi = 256)
        {"name": "matvec_xxz256", "kind": "matvec", "model": "xxz", "cL": 256, "cR": 256, "n_max": 0},
        # the bulk bond of the complex benchmark (Josephson, d = 5, chi = 128)
        {"name": "matvec_josephson", "kind": "matvec", "model": "josephson", "cL": 128, "cR": 128, "n_max": 2},
        # a caller that drives its own sweep: one Lanczos solve on host arrays
        {"name": "bond_xxz128", "kind": "bond", "model": "xxz", "cL": 128, "cR": 120, "n_max": 0},
        # the exact split of a bulk bond at chi = 256, left-to-right
        {"name": "split_f64_512", "kind": "split", "complex": False, "m": 512, "n": 512, "keep": 256, "dir": "R"},
        # the exact complex split of a ragged bond, right-to-left
        {"name": "split_c128_ragged", "kind": "split", "complex": True, "m": 275, "n": 320, "keep": 64, "dir": "L"},
        # environment updates in both directions, ragged bond
        {"name": "env_xxz", "kind": "env", "model": "xxz", "cL": 256, "cR": 243, "n_max": 0},
        # a small chain solved from scratch (the short-chain configuration)
        {"name": "solve_xxz_L12", "kind": "solve", "model": "xxz", "L": 12, "chi": 64, "n_max": 0, "sweeps": 6,
         "truncation": 0, "single_site": False},
        # the steady sweep of the benchmark chain
        {"name": "sweep_xxz_L100", "kind": "sweep", "model": "xxz", "L": 100, "chi": 256, "n_max": 0},
        # the steady sweep of the complex benchmark chain, at half its bond cap
        {"name": "sweep_josephson_L24", "kind": "sweep", "model": "josephson", "L": 24, "chi": 64, "n_max": 2},
        # a small batch of served solves
        {"name": "batch_xxz", "kind": "batch", "model": "xxz", "L": 24, "chi": 64, "n_max": 0, "requests": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "bond", "split", "split", "env", "solve", "sweep", "sweep", "batch"])
    model = rng.choice(["xxz", "j1j2", "josephson"])
    n_max = rng.choice([1, 2]) if model == "josephson" else 0
    if kind in ("matvec", "bond", "env"):
        hi = {"xxz": 300, "j1j2": 260, "josephson": 140 if n_max == 1 else 128}[model]
        if kind == "bond":
            hi //= 2
        return {"kind": kind, "model": model, "cL": _log(rng, 8, hi), "cR": _log(rng, 8, hi), "n_max": n_max}
    if kind == "split":
        cplx = rng.random() < 0.4
        m, n = _log(rng, 24, 320 if cplx else 512), _log(rng, 24, 320 if cplx else 512)
        return {"kind": kind, "complex": cplx, "m": m, "n": n, "keep": max(4, min(m, n) // rng.choice([2, 3, 4])),
                "dir": rng.choice("RL")}
    if kind == "solve":
        if model == "josephson":
            L, n_max, chi = rng.randint(5, 7), 1, rng.randint(12, 27)
        else:
            L, chi = rng.randint(6, 12), rng.randint(24, 64)
        return {"kind": kind, "model": model, "L": L, "chi": chi, "n_max": n_max, "sweeps": rng.randint(5, 8),
                "truncation": rng.choice([0, 1]), "single_site": rng.random() < 0.25}
    if kind == "sweep":
        if model == "josephson":
            L, chi = rng.randint(12, 24), _log(rng, 24, 64)
        else:
            L, chi = rng.randint(24, 96 if model == "xxz" else 56), _log(rng, 32, 250 if model == "xxz" else 128)
        return {"kind": kind, "model": model, "L": L, "chi": chi, "n_max": n_max}
    return {"kind": "batch", "model": rng.choice(["xxz", "j1j2"]), "L": rng.randint(16, 24), "chi": rng.randint(32, 64),
            "n_max": 0, "requests": rng.randint(2, 6)}


# ----------------------------------------------------------------------------- inputs
def _dims(case):
    """(d, D, complex) of the case's model."""
    if case["model"] == "josephson":
        return 2 * case["n_max"] + 1, 4, True
    return 2, (5 if case["model"] == "xxz" else 8), False


def _local_op(case):
    d = _dims(case)[0]
    return np.diag(np.arange(d) - (d - 1) / 2.0) if case["model"] == "josephson" else np.diag([0.5, -0.5])


def _chain(case, rng):
    """MPO of the case's chain with seeded weak on-site terms."""
    L, op = case["L"], _local_op(case)
    if case["model"] == "xxz":
        Ws = models.xxz(L, delta=rng.uniform(0.8, 1.2))
    elif case["model"] == "j1j2":
        Ws = models.j1j2(L, J2=rng.uniform(0.15, 0.35))
    else:
        Ws = models.josephson(L, n_max=case["n_max"], E_J=2.0, E_C=1.0, n_g=0.25, phi=2 * np.pi * 0.1 / L, onsite="shifted")
    Ws = [W.copy() for W in Ws]
    for W, h in zip(Ws, 0.1 * rng.uniform(-1, 1, L)):
        W[0, -1] += h * op
    return Ws


def _bulk(case):
    """Two neighbouring bulk MPO tensors of the case's model."""
    L = 8
    if case["model"] == "xxz":
        Ws = models.xxz(L)
    elif case["model"] == "j1j2":
        Ws = models.j1j2(L, J2=0.25)
    else:
        Ws = models.josephson(L, n_max=case["n_max"], E_J=2.0, E_C=1.0, n_g=0.25, phi=0.1, onsite="shifted")
    return Ws[3], Ws[4]


def _rand(rng, shape, cplx):
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if cplx else x


def _block_env(rng, chi, case, side):
    """(bra, mpo, ket) environment of a block of `chi` states: the identity, bounded block
    operators in the coupling channels, and a block Hamiltonian with a gap at the bottom."""
    _, D, cplx = _dims(case)
    E = np.zeros((chi, D, chi), np.complex128 if cplx else np.float64)
    idle, full = (0, D - 1) if side == "L" else (D - 1, 0)
    E[:, idle] = np.eye(chi)
    H = _rand(rng, (chi, chi), cplx) / np.sqrt(chi)
    E[:, full] = 0.05 * (H + H.conj().T) + np.diag(6.0 * np.sqrt(np.arange(chi) / chi))
    ladder = {1: 2, 4: 5} if case["model"] == "j1j2" else {1: 2}  # channels of an operator and its adjoint
    for w in range(1, D - 1):
        if w in ladder.values():
            E[:, w] = E[:, w - 1].conj().T
        else:
            O = 0.2 * _rand(rng, (chi, chi), cplx) / np.sqrt(chi)
            E[:, w] = O if w in ladder else 0.5 * (O + O.conj().T)
    return E


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind in ("matvec", "bond", "env"):
        d, D, cplx = _dims(case)
        cL, cR = case["cL"], case["cR"]
        L, R = _block_env(rng, cL, case, "L"), _block_env(rng, cR, case, "R")
        WL, WR = _bulk(case)
        th = _rand(rng, (cL, d, d, cR), cplx)
        if kind == "bond":  # a start vector that decays towards the blocks' high states, as a previous sweep's does
            th *= np.exp(-np.arange(cL) / 8.0)[:, None, None, None] * np.exp(-np.arange(cR) / 8.0)
        th /= np.linalg.norm(th)
        st["host"] = [L, R, WL, WR, th]
        if kind == "matvec":
            dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in st.pop("host")]
            st["dev"], st["out"] = dev, torch.empty_like(dev[4])
            st["lib"] = dmrg2.load_library()
            p = [ctypes.c_void_p(t.data_ptr()) for t in dev + [st["out"]]]
            st["args"] = [dmrg2.C128 if cplx else dmrg2.F64, cL, cR, d, D, D, D] + p
        elif kind == "env":
            st["A"] = np.linalg.qr(_rand(rng, (cL * d, min(cR, cL * d)), cplx))[0].reshape(cL, d, -1)
            q = np.linalg.qr(_rand(rng, (cR * d, min(cL, cR * d)), cplx))[0]
            st["B"] = np.ascontiguousarray(q.T).reshape(-1, d, cR)
    elif kind == "split":
        m, n, cplx = case["m"], case["n"], case["complex"]
        r = min(m, n)
        U = np.linalg.qr(_rand(rng, (m, r), cplx))[0]
        V = np.linalg.qr(_rand(rng, (n, r), cplx))[0]
        s = np.exp(-8.0 * np.arange(r) / r)  # a Schmidt spectrum that falls by 3000 over the bond
        s *= 1.0 + 0.2 * rng.uniform(-1, 1, r) * (8.0 / r)
        st["M"] = (U * (s / np.linalg.norm(s))) @ V.conj().T
    elif kind in ("solve", "sweep"):
        d, D, cplx = _dims(case)
        dt = np.complex128 if cplx else np.float64
        single = bool(case.get("single_site", False))
        g = dmrg2.DMRG2GPU(case["L"], d, case["chi"], D, dtype=dt, krylov_max=30, cutoff=1e-12, tol=1e-11,
                           truncation=case.get("truncation", 0), single_site=single, seed=int(seed) & 0xFFFF)
        g.set_mpo(_chain(case, rng))
        mps = models.random_mps(case["L"], d, case["chi"] if single else min(16, case["chi"]), seed=seed, dtype=dt)
        st["engine"], st["mps"], st["op"] = g, mps, _local_op(case).astype(dt)
        chi = case["chi"]
        ramp = [c for c in (16, 32, 64, 128) if c < chi]
        if kind == "solve":
            st["schedule"] = [chi] * case["sweeps"] if single else (ramp + [chi] * case["sweeps"])
        else:
            g.set_mps(mps)
            g.run(schedule=ramp + [chi, chi, chi])
    else:
        st["chains"] = [_chain(case, rng) for _ in range(case["requests"])]
        st["server"] = dmrg2.Server(max_active=case["requests"])
        st["seeds"] = [int(x) for x in rng.integers(1, 1 << 30, case["requests"])]
        chi = case["chi"]
        st["schedule"] = [c for c in (16, 32) if c < chi] + [chi] * 6
    return st


# ----------------------------------------------------------------------------- one pass
def _state_vector(As):
    """The state an MPS stands for, largest entry real and positive."""
    v = As[0].reshape(As[0].shape[1], -1)
    for A in As[1:]:
        v = (v @ A.reshape(A.shape[0], -1)).reshape(-1, A.shape[2])
    return _fix_vector(v.ravel())


def _fix_vector(v):
    p = v.ravel()[np.argmax(np.abs(v))]
    return v * (np.conj(p) / np.abs(p))


def _fix_pairs(left, right):
    p = left[np.argmax(np.abs(left), axis=0), np.arange(left.shape[1])]
    p = p / np.abs(p)
    return left * np.conj(p), right * p[:, None]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "matvec":
        if st["lib"].dmrg2_op_heff_noalloc(*st["args"], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)):
            raise RuntimeError(st["lib"].dmrg2_last_error(None).decode())
        return st["out"]
    if kind == "bond":
        e, th = dmrg2.optimize_two_site(*st["host"], max_iter=60, tol=1e-12, max_restarts=2)
        return [e, _fix_vector(th)]
    if kind == "split":
        left, S, right, _ = dmrg2.truncated_svd(st["M"], case["keep"], 0.0, case["dir"])
        return [*_fix_pairs(left, right), S]
    if kind == "env":
        L, R, WL, WR, _ = st["host"]
        return [dmrg2.update_left_env(L, st["A"], WL), dmrg2.update_right_env(R, st["B"], WR)]
    if kind == "solve":
        g = st["engine"]
        g.set_mps(st["mps"])
        g.run(schedule=st["schedule"])
        return [g.get_energy(), g.expect_local(st["op"]), _state_vector(g.get_mps())]
    if kind == "sweep":
        g = st["engine"]
        g.resume([case["chi"]])
        return [g.get_energy(), g.expect_local(st["op"])]
    ids = [st["server"].submit(W, st["schedule"], seed=s, init=dmrg2.INIT_RANDOM, cutoff=1e-12, tol=1e-11)
           for W, s in zip(st["chains"], st["seeds"])]
    out = [st["server"].result(i) for i in ids]
    for r in out:
        if r["state"] != dmrg2.REQ_DONE:
            raise RuntimeError(r["message"])
    return [r["energy"] for r in out]


# ----------------------------------------------------------------------------- necessary work
def _matvec_flops(cL, cR, d, D, cplx):
    f = 2.0 * D * d * d * cL * cR * (cL + cR)  # the two environment contractions
    return 4 * f if cplx else f


def _bond_profile(case):
    """Bond dimensions of the case's chain at its cap (the cutoff may leave fewer)."""
    d, L, chi = _dims(case)[0], case["L"], case["chi"]
    return [min(d ** min(i, L - i), chi) for i in range(L + 1)]


def _sweep_work(case, per_bond_matvecs=3):
    """One full sweep: theta, three Krylov vectors (the fewest the stop rule accepts), a
    rank-k orthonormal basis and the projection on it, one environment update per bond."""
    d, D, cplx = _dims(case)
    b = _bond_profile(case)
    fl = by = 0.0
    for i in range(case["L"] - 1):
        cL, k, cR = b[i], b[i + 1], b[i + 2]
        m, n = cL * d, d * cR
        f = 2.0 * m * k * n + 4.0 * m * n * k + 2.0 * min(m, n) * k * k
        f += 2.0 * D * d * cL * k * (cL + k)
        f = (4 * f if cplx else f) + per_bond_matvecs * _matvec_flops(cL, cR, d, D, cplx)
        fl += 2 * f
        # both environments and both sites read, the sites and one environment written
        by += 2 * (16 if cplx else 8) * (D * (cL * cL + cR * cR + k * k) + 2.0 * (m * k + k * n))
    return {"bytes": by, "flops": fl}


def work(case):
    kind = case["kind"]
    if kind == "split":
        m, n, k, s = case["m"], case["n"], case["keep"], 16 if case["complex"] else 8
        g = m if case["dir"] == "R" else n
        o = m * n // g
        f = g * g * o + 4.0 / 3 * g ** 3 + 2.0 * g * g * k + 2.0 * m * n * k
        return {"bytes": s * (m * n + (m + n) * k) + 8 * min(m, n), "flops": 4 * f if case["complex"] else f}
    d, D, cplx = _dims(case)
    s = 16 if cplx else 8
    if kind in ("matvec", "bond", "env"):
        cL, cR = case["cL"], case["cR"]
        n, envs = cL * d * d * cR, D * (cL * cL + cR * cR)
        if kind == "matvec":
            return {"bytes": s * (envs + 2 * n), "flops": _matvec_flops(cL, cR, d, D, cplx)}
        if kind == "bond":  # at least ten Krylov vectors from a rough start
            f = 10 * _matvec_flops(cL, cR, d, D, cplx)
            return {"bytes": s * (envs + 2 * n), "flops": f + 10 * 4.0 * n * 10}
        a, b = min(cR, cL * d), min(cL, cR * d)
        f = 2.0 * D * d * (cL * a * (cL + a) + cR * b * (cR + b))
        return {"bytes": s * (envs + D * (a * a + b * b) + d * (cL * a + cR * b)), "flops": 4 * f if cplx else f}
    one = _sweep_work(case)
    sweeps = 1 if kind == "sweep" else (case["sweeps"] if kind == "solve" else 4 * case["requests"])
    return {k: v * sweeps for k, v in one.items()}


def tolerance(case):
    """About four times the differences measured from plain 64-bit answers and between two
    builds that sum in different orders (over the listed cases and sixteen drawn ones)."""
    kind = case["kind"]
    if kind in ("matvec", "env"):  # up to 1e-15 from the 64-bit answer
        return {"rel": 4e-15}
    if kind == "bond":  # a Ritz value settled to 1e-12 fixes the vector to 4.6e-7
        return {"rel": 2e-6}
    if kind == "split":  # up to 2.9e-13 (density matrix of a spectrum that falls by 3000)
        return {"rel": 1.2e-12}
    if kind == "solve":  # the state 7e-8 from the exact one, by the same Ritz value rule in every bond
        return {"rel": 3e-7}
    if kind == "sweep":  # local values 1.2e-11 between builds, energies to rounding
        return {"rel": 1e-7}
    return {"rel": 1e-10}  # energies alone


# ----------------------------------------------------------------------------- plain 64-bit answers
def _exact_matvec(L, R, WL, WR, th):
    x = torch.einsum("awc,csre->awsre", L, th)
    x = torch.einsum("wmsp,awsre->ampre", WL, x)
    x = torch.einsum("mnrq,ampre->anpqe", WR, x)
    return torch.einsum("anpqe,fne->apqf", x, R)


def _exact_ground(L, R, WL, WR, th):
    """Lanczos with full reorthogonalisation (twice), restarted from the Ritz vector."""
    v = th / torch.linalg.norm(th)
    e = 0.0
    for _ in range(6):
        V, al, be = [v.reshape(-1)], [], []
        for j in range(60):
            w = _exact_matvec(L, R, WL, WR, V[j].reshape(th.shape)).reshape(-1)
            al.append(float(torch.vdot(V[j], w).real))
            B = torch.stack(V)
            for _ in range(2):
                w = w - B.T @ (B.conj() @ w)
            b = float(torch.linalg.norm(w))
            if b < 1e-13 or j == 59:
                break
            be.append(b)
            V.append(w / b)
        k = len(al)
        ev, y = np.linalg.eigh(np.diag(al) + np.diag(be[:k - 1], 1) + np.diag(be[:k - 1], -1))
        e = float(ev[0])
        v = torch.stack(V[:k]).T @ torch.from_numpy(y[:, 0]).to(v.device, v.dtype)
        v = v / torch.linalg.norm(v)
    return e, v.reshape(th.shape)


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind in ("sweep", "batch"):
        return None
    if kind == "solve":
        d, L = _dims(case)[0], case["L"]
        if d ** L > 4096 or case["single_site"]:
            return None
        if case["chi"] < d ** (L // 2):
            return None  # the kept space does not hold the exact state
        H = _chain(case, np.random.default_rng(seed))
        M = torch.from_numpy(H[0]).to(dev)[0].permute(0, 2, 1)  # (mpo_r, out, in)
        for W in H[1:]:
            W = torch.from_numpy(W).to(dev)
            a, b = M.shape[1], W.shape[2]
            M = torch.einsum("xoi,xyst->yotis", M, W).reshape(W.shape[1], a * b, a * b)
        ev, vec = torch.linalg.eigh(M[0])
        psi = vec[:, 0].cpu().numpy()
        op = np.diag(_local_op(case))
        p = (np.abs(psi) ** 2).reshape([d] * L)
        loc = np.array([float((p.sum(axis=tuple(j for j in range(L) if j != i)) * op).sum()) for i in range(L)])
        return [float(ev[0]), loc.astype(complex) if case["model"] == "josephson" else loc, _fix_vector(psi)]
    st = prepare(case, seed)
    if kind == "split":
        U, S, Vh = np.linalg.svd(st["M"], full_matrices=False)
        k = case["keep"]
        if case["dir"] == "R":
            left, right = U[:, :k], S[:k, None] * Vh[:k]
        else:
            left, right = U[:, :k] * S[:k], Vh[:k]
        return [*_fix_pairs(left, right), S]
    if kind == "matvec":
        return _exact_matvec(*st["dev"])
    t = [torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in st["host"]]
    if kind == "bond":
        e, th = _exact_ground(*t)
        return [e, _fix_vector(th.cpu().numpy())]
    L, R, WL, WR, _ = t
    A, B = torch.from_numpy(st["A"]).to(dev), torch.from_numpy(st["B"]).to(dev)
    x = torch.einsum("awc,csk->awsk", L, A)
    x = torch.einsum("wnst,awsk->antk", WL, x)
    left = torch.einsum("atb,antk->bnk", A.conj(), x)
    y = torch.einsum("awc,ksc->awsk", R, B)
    y = torch.einsum("nwst,awsk->antk", WR, y)
    right = torch.einsum("bta,antk->bnk", B.conj(), y)
    return [left.cpu().numpy(), right.cpu().numpy()]
