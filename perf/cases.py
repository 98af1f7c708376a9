"""The calls whose speed this repository looks after.

``listed()`` names twelve of them: effective-Hamiltonian applications from the smallest bond
dimension to the flagship Hubbard one, a raw complex GEMM, a QRpos, a gauge fixing, an
eigensolve, an environment build, an entanglement spectrum, and two whole calls (a TDVP step
and a VUMPS iteration).  ``draw(rng)`` gives another case of the same kinds and ranges.
``prepare`` makes what a user's program holds before the call, ``run`` is one call through the
public entry points, ``work`` what it cannot do without, and ``exact`` the same result from
plain torch or numpy in 64 bits.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from infinitempsalgorithms_b200 import _lib as L
from infinitempsalgorithms_b200 import api

# model -> (physical dimension, MPO levels)
SHAPE = {"tfim": (2, 3), "xxz": (2, 5), "hubbard": (4, 6)}
# which bond dimensions a drawn case of a kind and model may have (inclusive); the listed
# cases lie inside, and nothing drawn costs more than the largest of them
RANGE = {
    ("heff", "tfim"): (8, 512), ("heff", "xxz"): (16, 768), ("heff", "hubbard"): (32, 1000),
    ("gauge", "tfim"): (16, 256), ("gauge", "xxz"): (16, 256), ("gauge", "hubbard"): (16, 192),
    ("eig", "tfim"): (16, 320), ("eig", "xxz"): (16, 256), ("eig", "hubbard"): (16, 160),
    ("envs", "tfim"): (16, 320), ("envs", "xxz"): (16, 256), ("envs", "hubbard"): (16, 256),
    ("tdvp", "tfim"): (16, 256), ("tdvp", "xxz"): (16, 160),
}


def listed():
    return [
        # the inner loop of a VUMPS run at the smallest bond dimension (TFIM, N = 1, D = 16):
        # one matvec is launches and nothing else
        {"name": "heff_tfim_d16", "kind": "heff", "model": "tfim", "D": 16, "slices": 0},
        # an ordinary chain, an odd bond dimension
        {"name": "heff_xxz_d251", "kind": "heff", "model": "xxz", "D": 251, "slices": 0},
        # the flagship matvec (Hubbard, Jordan-Wigner, D = 1024), in FP64
        {"name": "heff_hubbard_d1024", "kind": "heff", "model": "hubbard", "D": 1024, "slices": 0},
        # and in the split-precision mode, with the context's default slice count
        {"name": "heff_hubbard_d1024_split", "kind": "heff", "model": "hubbard", "D": 1024, "slices": 5},
        # a contraction that a caller makes itself on device arrays: odd sizes, op(A) = A^H,
        # an update of C
        {"name": "gemm_odd", "kind": "gemm", "M": 1537, "N": 771, "K": 2049, "opA": 2, "opB": 0, "beta": 1.0},
        # leftorth of one site tensor (D = 512, d = 4)
        {"name": "qr_2048x512", "kind": "qr", "m": 2048, "n": 512, "left": True},
        # the constructor every run starts with: CanonicalIMPS of random tensors (XXZ cell, D = 256)
        {"name": "gauge_xxz_d256", "kind": "gauge", "model": "xxz", "D": 256},
        # one eigensolve of the effective Hamiltonian from the current centre tensor
        {"name": "eig_xxz_d256", "kind": "eig", "model": "xxz", "D": 256},
        # the environments of a new state, built from nothing
        {"name": "envs_hubbard_d256", "kind": "envs", "model": "hubbard", "D": 256},
        # the entanglement spectrum of one bond, the usual observable after a run
        {"name": "spectrum_d256", "kind": "spectrum", "D": 256},
        # one step of a real-time quench
        {"name": "tdvp_tfim_d256", "kind": "tdvp", "model": "tfim", "D": 256},
        # the first VUMPS iteration of a Hubbard ground-state search in the adaptive split mode
        {"name": "vumps_hubbard_d384_split", "kind": "vumps", "model": "hubbard", "D": 384},
    ]


def _log(rng, lo, hi):
    """An integer in [lo, hi], uniform in its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["heff", "heff", "heff", "gemm", "qr", "gauge", "eig", "envs", "spectrum", "tdvp", "vumps"])
    if kind == "gemm":
        m, n, k = (_log(rng, 24, 2600) for _ in range(3))
        return {"kind": kind, "M": m, "N": n, "K": k, "opA": rng.choice([0, 1, 2]), "opB": rng.choice([0, 1, 2]),
                "beta": rng.choice([0.0, 1.0])}
    if kind == "qr":
        n = _log(rng, 12, 600)
        return {"kind": kind, "m": min(2600, round(n * rng.uniform(1.0, 4.0))), "n": n, "left": rng.random() < 0.5}
    if kind == "spectrum":
        return {"kind": kind, "D": _log(rng, 16, 320)}
    if kind == "vumps":
        return {"kind": kind, "model": "hubbard", "D": _log(rng, 64, 384)}
    model = rng.choice([m for k, m in RANGE if k == kind])
    case = {"kind": kind, "model": model, "D": _log(rng, *RANGE[kind, model])}
    if kind == "heff":
        case["slices"] = rng.choice([0, 0, 4, 5, 6])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_contexts = {}


def _context(slices):
    """The program's context: FP64 (0), a fixed slice count, or the adaptive split mode (-1),
    on torch's stream."""
    if slices not in _contexts:
        ctx = api.Context(0) if slices == 0 else api.Context(0, precision=L.IMPS_PREC_SPLIT_I8, nslices=slices)
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        _contexts[slices] = ctx
    return _contexts[slices]


def _cell(model):
    return 1 if model == "tfim" else 2


def _hamiltonian(model, sites):
    """The model's MPO on a unit cell of this many sites."""
    if model == "tfim":
        H = api.tfim_hamiltonian(1.0, 1.5)
    elif model == "xxz":
        H = api.heisenberg_hamiltonian(1.0, 0.5)
    else:
        H = api.hubbard_hamiltonian(1.0, 4.0, 2.0)
    return api.SparseIMPO(H.Ws * sites)


def _randn(gen, *shape):
    """A column-major complex128 device tensor of this shape, Re, Im ~ N(0, 1/2)."""
    x = torch.randn(*reversed(shape), dtype=torch.complex128, device="cuda", generator=gen)
    return x.permute(*reversed(range(len(shape))))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _host(x):
    """The column-major host array of a device tensor."""
    n = x.dim()
    return x.permute(*reversed(range(n))).contiguous().cpu().numpy().transpose(*reversed(range(n)))


def _heff_inputs(case, seed):
    """Environments as a canonical state has them (an identity level each, the others of
    order one) and a unit centre tensor."""
    d, w = SHAPE[case["model"]]
    D, g = case["D"], _gen(seed)
    GL, GR = _randn(g, D, w, D) / math.sqrt(D), _randn(g, D, w, D) / math.sqrt(D)
    eye = torch.eye(D, dtype=torch.complex128, device="cuda")
    GL[:, 0, :] = eye
    GR[:, w - 1, :] = eye
    x = _randn(g, D, d, D)
    return GL, GR, x / torch.linalg.vector_norm(x)


def _sites(case, seed):
    d, _ = SHAPE[case["model"]]
    g = _gen(seed)
    return [_host(_randn(g, case["D"], d, case["D"])) for _ in range(_cell(case["model"]))]


def _gemm_inputs(case, seed):
    g = _gen(seed)
    a = (case["M"], case["K"]) if case["opA"] == 0 else (case["K"], case["M"])
    b = (case["K"], case["N"]) if case["opB"] == 0 else (case["N"], case["K"])
    return _randn(g, *a), _randn(g, *b), _randn(g, case["M"], case["N"])


def _qr_input(case, seed):
    shape = (case["m"], case["n"]) if case["left"] else (case["n"], case["m"])
    return _host(_randn(_gen(seed), *shape))


def _bond_matrix(case, seed):
    """A bond matrix with decaying Schmidt values in a general basis."""
    D, g = case["D"], _gen(seed)
    s = torch.exp(-16.0 * torch.arange(D, dtype=torch.float64, device="cuda") / D)
    c = (_randn(g, D, D) * s) @ _randn(g, D, D)
    return _host(c / torch.linalg.vector_norm(c))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "heff":
        ctx = _context(case["slices"])
        H = _hamiltonian(case["model"], 1)
        d, _ = SHAPE[case["model"]]
        GL, GR, x = _heff_inputs(case, seed)
        psi = api.CanonicalIMPS(ctx, [d], [case["D"]])
        envs = api.DMRGCache(psi, H, build=False)
        envs.set_leftenv(1, _host(GL))
        envs.set_rightenv(1, _host(GR))
        return {"case": case, "ctx": ctx, "psi": psi, "envs": envs, "H": H, "x": x, "y": torch.empty_like(x)}
    if kind == "gemm":
        A, B, C0 = _gemm_inputs(case, seed)
        return {"case": case, "ctx": _context(0), "A": A, "B": B, "C0": C0, "C": torch.empty_like(C0)}
    if kind == "qr":
        return {"case": case, "ctx": _context(0), "M": _qr_input(case, seed)}
    if kind == "gauge":
        return {"case": case, "ctx": _context(0), "As": _sites(case, seed)}
    if kind == "spectrum":
        ctx = _context(0)
        psi = api.CanonicalIMPS(ctx, [2], [case["D"]])
        psi.set(L.IMPS_C, 0, _bond_matrix(case, seed))
        return {"case": case, "psi": psi}
    ctx = _context(-1 if kind == "vumps" else 0)
    H = _hamiltonian(case["model"], _cell(case["model"]))
    psi = api.CanonicalIMPS.from_sites(_sites(case, seed), ctx=ctx)
    state = {"case": case, "ctx": ctx, "psi": psi, "H": H}
    if kind == "eig":
        state["envs"] = api.DMRGCache(psi, H)
        state["x0"] = psi.get(L.IMPS_AC, 0)
    return state


# ---------------------------------------------------------------------------
# one call
# ---------------------------------------------------------------------------
def _tensors(psi):
    return {"AL": list(psi.AL), "AR": list(psi.AR), "C": list(psi.C), "AC": list(psi.AC)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "heff":
        ctx = state["ctx"]
        L.check(ctx.lib.imps_ac_apply_dev(state["envs"].h, state["H"].handle(ctx), 0, state["x"].data_ptr(),
                                          state["y"].data_ptr()), ctx.h)
        return state["y"]
    if kind == "gemm":
        ctx = state["ctx"]
        A, B, out = state["A"], state["B"], state["C"]
        if case["beta"]:
            out.copy_(state["C0"])
        L.check(ctx.lib.imps_zgemm(ctx.h, case["opA"], case["opB"], case["M"], case["N"], case["K"], 1.0, 0.0,
                                   A.data_ptr(), A.shape[0], B.data_ptr(), B.shape[0], case["beta"], 0.0,
                                   out.data_ptr(), case["M"]), ctx.h)
        return out
    if kind == "qr":
        return (api.qrpos if case["left"] else api.lqpos)(state["M"], ctx=state["ctx"])
    if kind == "gauge":
        return _tensors(api.CanonicalIMPS.from_sites(state["As"], ctx=state["ctx"]))
    if kind == "eig":
        h = api.AC_hamiltonian(1, state["psi"], state["H"], state["psi"], state["envs"])
        return api.fixedpoint(h, state["x0"], "SR", dict(tol=1e-10, krylovdim=30, maxiter=300, eager=True))
    if kind == "envs":
        envs = api.DMRGCache(state["psi"], state["H"])
        return {"left": list(envs.lefts), "right": list(envs.rights)}
    if kind == "spectrum":
        return api.entanglement_spectrum(state["psi"], 1)
    if kind == "tdvp":
        psi, _ = api.timestep(state["psi"], state["H"], -0.01j)
        return _tensors(psi)
    psi, envs, info = api.find_groundstate(state["psi"], state["H"], api.VUMPS(D=case["D"], maxiter=1))
    return {"state": _tensors(psi), "losses": list(info.losses),
            "energy": api.expectationvalue(psi, state["H"], envs).real}


# ---------------------------------------------------------------------------
# what a call cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "gemm":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 16.0 * (M * K + K * N + (2 if case["beta"] else 1) * M * N), "flops": 8.0 * M * N * K}
    if kind == "qr":
        m, n = max(case["m"], case["n"]), min(case["m"], case["n"])
        return {"bytes": 16.0 * (2 * m * n + n * n), "flops": 16.0 * (m * n * n - n ** 3 / 3.0)}
    D = case["D"]
    if kind == "spectrum":
        return {"bytes": 16.0 * D * D + 8.0 * D, "flops": 16.0 * D ** 3}
    d, w = SHAPE[case["model"]]
    N = _cell(case["model"])
    site, env = d * D * D, w * D * D
    apply = 16.0 * w * d * D ** 3 + 8.0 * w * w * d * d * D * D
    qr = 16.0 * (d - 1.0 / 3.0) * D ** 3
    push = 16.0 * d * D ** 3
    if kind == "heff":
        return {"bytes": 16.0 * (2 * env + 2 * site), "flops": apply}
    if kind == "gauge":
        # eleven sweeps each way (the gauge iteration solves for the fixed point from the tenth on)
        return {"bytes": 16.0 * N * 4 * site, "flops": N * 22 * (8.0 * d * D ** 3 + qr)}
    if kind == "eig":
        return {"bytes": 16.0 * (2 * env + 2 * site), "flops": 20 * apply}
    if kind == "envs":
        return {"bytes": 16.0 * N * (2 * site + 2 * env), "flops": N * 2 * (2 * w + 10) * push}
    if kind == "tdvp":
        return {"bytes": 16.0 * N * (5 * site + 2 * env), "flops": N * (10 * apply + 22 * qr + 20 * push)}
    return {"bytes": 16.0 * N * (5 * site + 2 * env),
            "flops": N * (10 * apply + 11 * (8.0 * d * D ** 3 + qr) + 4 * (2 * w + 10) * push)}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch / numpy
# ---------------------------------------------------------------------------
def _apply(GL, W, GR, x):
    t = torch.einsum("bia,asc->bisc", GL, x)
    t = torch.einsum("iujs,bisc->bujc", W, t)
    return torch.einsum("bujc,cjd->bud", t, GR)


def _qr_pos(M):
    Q, R = torch.linalg.qr(M)
    ph = torch.diagonal(R)
    ph = torch.where(ph.abs() > 0, ph / ph.abs(), torch.ones_like(ph))
    return Q * ph, R * ph.conj()[:, None]


def _left_sweeps(As, C):
    """QRpos sweeps of the unit cell until the bond matrix stands still: AL, C with AL C = C A."""
    for _ in range(400):
        old, AL, Cs = C, [], []
        for A in As:
            Dl, d, Dr = A.shape
            Q, C = _qr_pos(torch.einsum("ab,bsc->asc", C, A).permute(1, 0, 2).reshape(d * Dl, Dr))
            # rows run over (a, s) with a first, as in the column-major (Dl d) x Dr matrix
            AL.append(Q.reshape(d, Dl, Dr).permute(1, 0, 2))
            Cs.append(C)
        C = C / torch.linalg.vector_norm(C)
        if torch.linalg.vector_norm(C - old) < 1e-14:
            break
    Cs[-1] = C
    return AL, Cs


def _mirror(A):
    return A.permute(2, 1, 0).conj()


def _canonical(As):
    """AL, AR, C, AC of the uniform state of these site tensors; C[l] right of site l."""
    As = [torch.from_numpy(np.ascontiguousarray(A)).cuda() for A in As]
    D = As[0].shape[0]
    AL, Cs = _left_sweeps(As, torch.eye(D, dtype=torch.complex128, device="cuda") / math.sqrt(D))
    # the right orthogonalisation is the left one of the mirrored tensors; its row order runs
    # over (s, c) with s first
    N = len(As)
    C = Cs[-1]
    for _ in range(400):
        old, AR, Cr = C, [None] * N, [None] * N
        for l in range(N - 1, -1, -1):
            A = AL[l]
            Dl, d, Dr = A.shape
            M = torch.einsum("asb,bc->asc", A, C).permute(0, 2, 1).reshape(Dl, Dr * d)
            Q, R = _qr_pos(M.conj().T)
            Cr[l - 1] = C = R.conj().T
            AR[l] = Q.conj().T.reshape(Dl, Dr, d).permute(0, 2, 1)
        nrm = torch.linalg.vector_norm(C)
        C = C / nrm
        Cr[N - 1] = C
        if torch.linalg.vector_norm(C - old) < 1e-14:
            break
    AC = [torch.einsum("asb,bc->asc", AL[l], Cr[l]) for l in range(N)]
    return AL, AR, Cr, AC


def _environments(AL, AR, Cs, Ws):
    """Regularised left and right Schur environments, levels in order, the closing ones by the
    geometric series of the transfer matrix."""
    N, D, w = len(AL), AL[0].shape[0], Ws[0].shape[0]
    dev = AL[0].device
    eye = torch.eye(D, dtype=torch.complex128, device=dev)

    def push_left(GL, A, W):
        t = torch.einsum("bia,asc->bisc", GL, A)
        t = torch.einsum("iujs,bisc->bujc", W, t)
        return torch.einsum("buk,bujc->kjc", A.conj(), t)

    def push_right(GR, A, W):
        t = torch.einsum("asc,cjk->asjk", A, GR)
        t = torch.einsum("iujs,asjk->auik", W, t)
        return torch.einsum("auik,buk->aib", t, A.conj())

    def fixed(rhs, chain, rho):
        x = rhs - torch.einsum("ab,ba->", rho, rhs) * eye
        base, term = x.clone(), x
        for _ in range(400):
            term = chain(term)
            term = term - torch.einsum("ab,ba->", rho, term) * eye
            base = base + term
            if torch.linalg.vector_norm(term) < 1e-15 * torch.linalg.vector_norm(base):
                break
        return base

    def chain_left(x):
        for A in AL:
            x = torch.einsum("buk,buc->kc", A.conj(), torch.einsum("ba,asc->bsc", x, A))
        return x

    def chain_right(x):
        for A in reversed(AR):
            x = torch.einsum("auk,buk->ab", torch.einsum("asc,ck->ask", A, x), A.conj())
        return x

    lefts, rights = [], []
    GL = torch.zeros(D, w, D, dtype=torch.complex128, device=dev)
    GL[:, 0, :] = eye
    for _ in range(w):  # the middle levels follow from the ones above within w cells
        for l in range(N):
            GL = push_left(GL, AL[l], Ws[l])
        rhs = GL[:, w - 1, :].clone()
        GL[:, w - 1, :] = 0
    rho = Cs[N - 1] @ Cs[N - 1].conj().T
    GL[:, w - 1, :] = fixed(rhs, chain_left, rho)
    for l in range(N):
        rho = Cs[l - 1] @ Cs[l - 1].conj().T
        keep = GL.clone()
        keep[:, w - 1, :] -= torch.einsum("ab,ba->", rho, GL[:, w - 1, :]) * eye
        lefts.append(keep)
        GL = push_left(GL, AL[l], Ws[l])
    GR = torch.zeros(D, w, D, dtype=torch.complex128, device=dev)
    GR[:, w - 1, :] = eye
    for _ in range(w):
        for l in range(N - 1, -1, -1):
            GR = push_right(GR, AR[l], Ws[l])
        rhs = GR[:, 0, :].clone()
        GR[:, 0, :] = 0
    rho = Cs[N - 1].conj().T @ Cs[N - 1]
    GR[:, 0, :] = fixed(rhs, chain_right, rho)
    for l in range(N - 1, -1, -1):
        rho = Cs[l].conj().T @ Cs[l]
        keep = GR.clone()
        keep[:, 0, :] -= torch.einsum("ab,ba->", rho, GR[:, 0, :]) * eye
        rights.insert(0, keep)
        GR = push_right(GR, AR[l], Ws[l])
    return lefts, rights


def _lowest(apply, x0):
    """Lowest eigenpair by restarted Lanczos with full orthogonalisation, in phase with x0."""
    v = x0 / torch.linalg.vector_norm(x0)
    shape, value, kmax = v.shape, 0.0, min(120, v.numel())
    for _ in range(40):
        V, a, b = [v.reshape(-1)], [], []
        for k in range(kmax):
            w = apply(V[k].reshape(shape)).reshape(-1)
            B = torch.stack(V, 1)
            h = B.conj().T @ w
            w = w - B @ h
            w = w - B @ (B.conj().T @ w)
            a.append(h[k].real.item())
            n = torch.linalg.vector_norm(w).item()
            if k + 1 == kmax or n < 1e-13:
                break
            b.append(n)
            V.append(w / n)
        T = np.diag(a) + np.diag(b[:len(a) - 1], 1) + np.diag(b[:len(a) - 1], -1)
        e, U = np.linalg.eigh(T)
        u = torch.from_numpy(U[:, 0]).to(v.device, torch.complex128)
        v = (torch.stack(V[:len(a)], 1) @ u).reshape(shape)
        v = v / torch.linalg.vector_norm(v)
        r = apply(v)
        value = torch.einsum("asb,asb->", v.conj(), r).real.item()
        if torch.linalg.vector_norm(r - value * v).item() < 1e-13 * max(1.0, abs(value)) or n < 1e-13:
            break
    ph = torch.einsum("asb,asb->", x0.conj(), v)
    return value, v * (ph.conj() / ph.abs())


def _op(X, op):
    return X if op == 0 else X.transpose(0, 1) if op == 1 else X.conj().transpose(0, 1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("tdvp", "vumps"):
        return None
    if kind == "gemm":
        A, B, C0 = _gemm_inputs(case, seed)
        return _op(A, case["opA"]) @ _op(B, case["opB"]) + case["beta"] * C0
    if kind == "qr":
        M = torch.from_numpy(np.ascontiguousarray(_qr_input(case, seed)))
        if case["left"]:
            Q, R = _qr_pos(M)
            return Q.numpy(), R.numpy()
        Q, R = _qr_pos(M.conj().T)
        return R.conj().T.numpy(), Q.conj().T.numpy()
    if kind == "spectrum":
        s = np.linalg.svd(_bond_matrix(case, seed), compute_uv=False) ** 2
        return s / s.sum()
    W = [torch.from_numpy(np.ascontiguousarray(X)).cuda() for X in _hamiltonian(case["model"], 1).Ws]
    if kind == "heff":
        GL, GR, x = _heff_inputs(case, seed)
        return _apply(GL, W[0], GR, x)
    AL, AR, Cs, AC = _canonical(_sites(case, seed))
    if kind == "gauge":
        return {n: [X.cpu().numpy() for X in v] for n, v in (("AL", AL), ("AR", AR), ("C", Cs), ("AC", AC))}
    lefts, rights = _environments(AL, AR, Cs, W * len(AL))
    if kind == "envs":
        return {"left": [X.cpu().numpy() for X in lefts], "right": [X.cpu().numpy() for X in rights]}
    value, v = _lowest(lambda x: _apply(lefts[0], W[0], rights[0], x), AC[0])
    return value, v.cpu().numpy()
