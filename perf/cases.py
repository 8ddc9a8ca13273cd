"""Performance cases: the work that users of this framework have it do, through its public entry points.

Three groups.  Whole searches and evolutions by the reference-shaped API (`MPS.FindVariationalGroundState`,
`MPS.Sweep`, `iTEBDState.Step`, `FullState.FindGroundState`, `LearnedCorrection`); the site operators that a host
solver calls through the C ABI on device buffers (`tn_heff_apply`, `tn_env_left` / `tn_env_right`); and the dense
solvers behind the same ABI (`tn_qr`, `tn_lq`, `tn_svd`).  Sizes are those of the repository's benchmark (L = 100,
D up to 256 at S = 1/2; D = 512 at S = 1), of its tests (L = 10, D = 8; iTEBD D = 32) and generic odd ones.

Matrices are column-major, as the C ABI takes them: an m x n matrix is a contiguous torch tensor of shape (n, m).
"""
import ctypes as C
import math

import numpy as np
import torch

from tensornetworks_b200 import api

F64 = torch.float64
PRECISION = {"fp64": api.FP64, "mixed": api.MIXED}
_stream = None


def _context():
    """The program's one context, on a torch stream of its own, so that torch work in between is ordered with it."""
    global _stream
    ctx = api.default_context()
    if _stream is None:
        _stream = torch.cuda.Stream()
        api.check(ctx._lib.tn_ctx_set_stream(ctx.handle, C.c_void_p(_stream.cuda_stream)), "tn_ctx_set_stream")
    return ctx


def listed():
    return [
        # the reference's own example (test_Unittest1.py): a whole search where every launch is small
        {"name": "search_L10_D8", "kind": "search", "twoS": 1, "L": 10, "D0": 8, "D": 8, "sweeps": 3, "precision": "fp64"},
        # the benchmark's search on a shorter chain: D grown 16 -> 256, split precision
        {"name": "search_L32_D256_mixed", "kind": "search", "twoS": 1, "L": 32, "D0": 16, "D": 256, "sweeps": 1, "precision": "mixed"},
        # one FP64 sweep pair from a random state, spin 1, a bond dimension that no tile divides
        {"name": "sweep_S1_L12_D90", "kind": "sweep", "twoS": 2, "L": 12, "D": 90, "precision": "fp64"},
        # the benchmark's bulk matvec by the operator handle
        {"name": "heff_D256_mixed", "kind": "heff", "twoS": 1, "D1": 256, "D2": 256, "precision": "mixed"},
        # the largest site operator: spin 1, D = 512, FP64
        {"name": "heff_S1_D512", "kind": "heff", "twoS": 2, "D1": 512, "D2": 512, "precision": "fp64"},
        # environment updates of both sweep directions, ragged site
        {"name": "env_D250_D203", "kind": "env", "twoS": 1, "D1": 250, "D2": 203, "precision": "fp64"},
        # gauge move left to right at the benchmark's size
        {"name": "qr_512x256", "kind": "qr", "m": 512, "n": 256},
        # gauge move right to left, spin 1, D = 512
        {"name": "lq_512x1536", "kind": "lq", "m": 512, "n": 1536},
        # SVDSolver / compressor input: two-site matrix of a modest bond dimension
        {"name": "svd_150x128", "kind": "svd", "m": 150, "n": 128},
        # the reference's iTEBD test size, a few second-order Trotter steps from a random state
        {"name": "itebd_D32", "kind": "itebd", "twoS": 1, "D": 32, "steps": 3},
        # exact diagonalisation of a chain that no longer fits a dense solver
        {"name": "fullstate_L18", "kind": "fullstate", "twoS": 1, "L": 18},
        # learned correction: one gradient for training and inference on one bulk site vector
        {"name": "learned_131072", "kind": "learned", "n": 131072},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["search", "sweep", "heff", "heff", "env", "qr", "lq", "svd", "itebd", "fullstate", "learned"])
    twoS = rng.choice([1, 1, 2])
    if kind == "search":
        if rng.random() < 0.5:
            D = rng.randint(4, 40)
            return {"kind": kind, "twoS": twoS, "L": rng.randint(4, 16), "D0": D, "D": D, "sweeps": 2, "precision": "fp64"}
        return {"kind": kind, "twoS": 1, "L": rng.randint(12, 32), "D0": 16, "D": 16 * rng.randint(2, 12), "sweeps": 1, "precision": "mixed"}
    if kind == "sweep":
        return {"kind": kind, "twoS": twoS, "L": rng.randint(6, 16), "D": _log(rng, 8, 128 if twoS == 1 else 90), "precision": "fp64"}
    if kind == "heff":
        D1, D2 = _log(rng, 16, 512), _log(rng, 16, 512)
        if rng.random() < 0.5:
            return {"kind": kind, "twoS": twoS, "D1": 16 * max(1, D1 // 16), "D2": 16 * max(1, D2 // 16), "precision": "mixed"}
        return {"kind": kind, "twoS": twoS, "D1": D1, "D2": D2, "precision": "fp64"}
    if kind == "env":
        return {"kind": kind, "twoS": twoS, "D1": _log(rng, 8, 512), "D2": _log(rng, 8, 512), "precision": "fp64"}
    if kind in ("qr", "lq"):
        n = _log(rng, 8, 512)
        m = min(1536, int(round(n * rng.choice([1.0, 1.3, 2.0, 2.0, 3.0]))))
        return {"kind": kind, "m": m, "n": n} if kind == "qr" else {"kind": kind, "m": n, "n": m}
    if kind == "svd":
        return {"kind": kind, "m": _log(rng, 8, 160), "n": _log(rng, 8, 160)}
    if kind == "itebd":
        return {"kind": kind, "twoS": twoS, "D": _log(rng, 4, 32 if twoS == 1 else 16), "steps": rng.randint(1, 3)}
    if kind == "fullstate":
        return {"kind": kind, "twoS": twoS, "L": rng.randint(6, 18) if twoS == 1 else rng.randint(4, 11)}
    return {"kind": kind, "n": _log(rng, 1024, 131072)}


# ---- inputs -----------------------------------------------------------------


def _randn(rng, *shape):
    return torch.from_numpy(rng.standard_normal(shape))


def _graded(rng, m, n, span):
    """m x n with singular values falling evenly on a logarithmic scale from 1 to 10^-span, as a site matrix's do."""
    k = min(m, n)
    U = np.linalg.qr(rng.standard_normal((m, k)))[0]
    V = np.linalg.qr(rng.standard_normal((n, k)))[0]
    s = 10.0 ** (-span * (np.arange(k) + 0.4 * rng.random(k)) / k)
    return torch.from_numpy((U * s) @ V.T)


def _environment(rng, D, done, side):
    """Dw = 5 blocks as a chain's environments are: the identity, three operators of norm ~ 1/2, an accumulated energy."""
    E = torch.empty(5, D, D, dtype=F64)
    for w in range(5):
        X = _randn(rng, D, D) / math.sqrt(D)
        E[w] = 0.125 * (X + X.T)
    E[done] = torch.eye(D, dtype=F64)
    E[side] = E[side] - 10.0 * torch.eye(D, dtype=F64) * (1.0 + 0.02 * _randn(rng, D, 1))
    return E


def _mpo(twoS):
    """The bulk MPO tensor of the Heisenberg chain, (Dw, Dw, d, d)."""
    H = api.Factory.GetFactory(_context()).Make1D_NN_HeisenbergHamiltonian(10, twoS / 2, 1.0, 1.0, 0.0)
    return np.ascontiguousarray(H.GetW(5))


def _site_operands(case, seed):
    """Left and right environments and a site tensor (d, D2, D1), on the host."""
    rng = np.random.default_rng(seed)
    d, D1, D2 = case["twoS"] + 1, case["D1"], case["D2"]
    F = _environment(rng, D1, 4, 0)   # lower MPO form: row 4 is complete on the left of the interaction
    G = _environment(rng, D2, 0, 4)
    x = _randn(rng, d, D2, D1)
    return F, G, x / x.norm()


def _schedule(case):
    """One line at D0, then the bond dimension doubled up to D, one line each."""
    sched, D = api.IterationSchedule(), case["D0"]
    last = D
    while True:
        eps = api.Epsilons(1e-12)
        eps.itsEigenSolverEpsilon = 1e-10
        sched.Insert(api.IterationScheduleLine(case["sweeps"], D, max(1, D - last), eps))
        if D >= case["D"]:
            return sched
        last, D = D, min(2 * D, case["D"])


def _chain(case, seed):
    """Couplings of the chain, spread with the seed as a parameter scan's are."""
    rng = np.random.default_rng(seed)
    return 1.0, float(rng.uniform(0.8, 1.2)), float(rng.uniform(0.0, 0.1))


def prepare(case, seed):
    kind = case["kind"]
    ctx = _context()
    st = {"case": case, "seed": seed, "ctx": ctx, "lib": ctx._lib}
    if kind in ("search", "sweep"):
        st["H"] = api.Factory.GetFactory(ctx).Make1D_NN_HeisenbergHamiltonian(case["L"], case["twoS"] / 2, *_chain(case, seed))
        st["psi"] = None
        st["options"] = api.SolverOptions(precision=PRECISION[case["precision"]])
        st["schedule"] = _schedule(case) if kind == "search" else None
        if kind == "sweep":
            st["psi"] = st["H"].CreateMPS(case["D"])
    elif kind in ("heff", "env"):
        F, G, x = _site_operands(case, seed)
        st["W"], st["F"], st["G"], st["x"] = _mpo(case["twoS"]), F.cuda(), G.cuda(), x.cuda()
        d, D1, D2 = case["twoS"] + 1, case["D1"], case["D2"]
        if kind == "heff":
            st["y"] = torch.empty_like(st["x"])
            torch.cuda.synchronize()
            st["op"] = _Heff(ctx, PRECISION[case["precision"]], d, D1, D2, st)
        else:
            st["Fout"] = torch.empty(5, D2, D2, dtype=F64, device="cuda")
            st["Gout"] = torch.empty(5, D1, D1, dtype=F64, device="cuda")
    elif kind in ("qr", "lq", "svd"):
        m, n = case["m"], case["n"]
        k = min(m, n)
        st["A"] = _graded(np.random.default_rng(seed), m, n, 3 if kind == "svd" else 5).T.contiguous().cuda()
        st["B"] = torch.empty(k, m, dtype=F64, device="cuda")    # m x k: Q, L or U
        st["C"] = torch.empty(n, k, dtype=F64, device="cuda")    # k x n: R, Q or Vt
        st["s"] = torch.empty(k, dtype=F64, device="cuda")
    elif kind == "itebd":
        st["psi"] = api.iTEBDState(case["twoS"] / 2, case["D"], *_chain(case, seed), seed=seed, ctx=ctx)
        st["sites"] = [st["psi"].GetSite(i) for i in range(2)]
        st["bonds"] = [st["psi"].GetBond(i) for i in range(2)]
    elif kind == "fullstate":
        st["H"] = api.Factory.GetFactory(ctx).Make1D_NN_HeisenbergHamiltonian(case["L"], case["twoS"] / 2, *_chain(case, seed))
    else:
        F, T, p = _pairs(case["n"], seed)
        st["F"], st["T"] = torch.from_numpy(F).cuda(), torch.from_numpy(T).cuda()
        st["model"] = api.LearnedCorrection(seed=1, ctx=ctx)
        st["model"].set_params(p)
    return st


class _Heff:
    """The operator handle of a site, freed with the state that holds it."""

    def __init__(self, ctx, precision, d, D1, D2, st):
        self.ctx, self.keep = ctx, (st["F"], st["G"])
        h = C.c_void_p()
        api.check(ctx._lib.tn_heff_create(ctx.handle, precision, d, 5, 5, D1, D2, st["W"].ctypes.data, st["F"].data_ptr(),
                                          st["G"].data_ptr(), C.byref(h)), "tn_heff_create")
        self.handle = h

    def apply(self, x, y):
        api.check(self.ctx._lib.tn_heff_apply(self.handle, x.data_ptr(), y.data_ptr()), "tn_heff_apply")

    def __del__(self):
        self.ctx._lib.tn_heff_destroy(self.handle)


def _pairs(n, seed):
    """Training pairs (features with the recorded ones' scales, targets) and a network's parameters."""
    rng = np.random.default_rng(seed)
    F = rng.standard_normal((n, 4)).astype(np.float32)
    F[:, 0] = np.abs(F[:, 0]) * 2.0
    F[:, 3] = rng.random(n, dtype=np.float32)
    T = np.clip(0.3 * F[:, 1] / (0.2 + F[:, 0]) + 0.1 * rng.standard_normal(n), -50, 50).astype(np.float32)
    p = np.zeros(4 * 64 + 64 + 64 * 64 + 64 + 64 + 1, dtype=np.float32)
    p[:256] = 0.3 * rng.standard_normal(256)
    p[256:320] = 0.1 * rng.standard_normal(64)
    p[320:4416] = 0.125 * rng.standard_normal(4096)
    p[4416:4480] = 0.1 * rng.standard_normal(64)
    p[4480:4544] = 0.125 * rng.standard_normal(64)
    return F, T, p


# ---- one pass ---------------------------------------------------------------


def run(st):
    case, ctx, lib = st["case"], st["ctx"], st["lib"]
    kind = case["kind"]
    if kind == "search":
        psi = st["H"].CreateMPS(case["D0"])
        psi.InitializeWith(api.Random, st["seed"])
        psi.FindVariationalGroundState(st["H"], st["schedule"], st["options"])
        return _measured(psi, case)
    if kind == "sweep":
        psi = st["psi"]
        psi.InitializeWith(api.Random, st["seed"])
        psi.PrepareSweeps(st["H"])
        psi.Sweep(st["H"], 1, 1e-10, st["options"])
        return _measured(psi, case)
    if kind == "heff":
        st["op"].apply(st["x"], st["y"])
        if case["precision"] == "fp64":
            return st["y"]
        with torch.cuda.stream(_stream):  # a split-precision product is carried on in single precision
            return st["y"].float()
    if kind == "env":
        d, D1, D2, W = case["twoS"] + 1, case["D1"], case["D2"], st["W"].ctypes.data
        api.check(lib.tn_env_left(ctx.handle, api.FP64, d, 5, 5, D1, D2, W, st["x"].data_ptr(), st["F"].data_ptr(),
                                  st["Fout"].data_ptr()), "tn_env_left")
        api.check(lib.tn_env_right(ctx.handle, api.FP64, d, 5, 5, D1, D2, W, st["x"].data_ptr(), st["G"].data_ptr(),
                                   st["Gout"].data_ptr()), "tn_env_right")
        return st["Fout"], st["Gout"]
    if kind in ("qr", "lq"):
        m, n = case["m"], case["n"]
        f = lib.tn_qr if kind == "qr" else lib.tn_lq
        api.check(f(ctx.handle, m, n, st["A"].data_ptr(), m, st["B"].data_ptr(), m, st["C"].data_ptr(), min(m, n)), kind)
        return st["B"], st["C"]
    if kind == "svd":
        m, n = case["m"], case["n"]
        api.check(lib.tn_svd(ctx.handle, m, n, st["A"].data_ptr(), m, st["B"].data_ptr(), m, st["s"].data_ptr(),
                             st["C"].data_ptr(), min(m, n)), "tn_svd")
        return _signed(st["B"], st["s"], st["C"])
    if kind == "itebd":
        psi = st["psi"]
        for i in range(2):
            psi.SetSite(i, st["sites"][i])
            psi.SetBond(i, st["bonds"][i])
        psi.Step(0.1, case["D"], case["steps"])
        # the Gammas are fixed up to the signs of the Schmidt vectors
        return [psi.GetBond(i) for i in range(2)], [np.abs(psi.GetSite(i)) for i in range(2)]
    if kind == "fullstate":
        fs = st["H"].CreateFullState(st["seed"])
        E = fs.FindGroundState(st["H"], 1e-10)
        return E, fs.GetAmplitudes()
    g, loss = st["model"].gradient(st["F"], st["T"])
    return g, loss, st["model"].forward(st["F"])


def _measured(psi, case):
    """What a search is run for: its energies and the bond spectra.  The spectra of a split-precision search are
    those of vectors solved to single precision."""
    s = np.concatenate([psi.GetBondSVs(b) for b in range(1, case["L"])])
    return psi.GetSiteEnergies(), s if case["precision"] == "fp64" else s.astype(np.float32)


def _signed(U, s, Vt):
    """Singular vectors with the sign that makes each left vector's largest entry positive (tensors are transposed)."""
    at = U.abs().argmax(dim=1, keepdim=True)
    sign = torch.sign(U.gather(1, at))
    return U * sign, s, Vt * sign.T


# ---- what a pass cannot do without -------------------------------------------


def _heff_flops(d, D1, D2):
    return 2.0 * d * 5 * D1 * D2 * (D1 + D2)


def work(case):
    kind = case["kind"]
    if kind in ("search", "sweep"):
        d, L = case["twoS"] + 1, case["L"]
        Ds = [case["D"]]
        if kind == "search":
            Ds = [case["D0"]]
            while Ds[-1] < case["D"]:
                Ds += [Ds[-1], min(2 * Ds[-1], case["D"])]  # each line first repeats the dimension before it
        flops = nbytes = 0.0
        for D in Ds:
            dims = [min(D, d ** min(i, L - i, 40)) for i in range(L + 1)]
            for a, b in zip(dims, dims[1:]):
                big, small = max(d * a, b), min(d * a, b)
                # twice each site: one application, one environment, one thin QR
                flops += 2.0 * case.get("sweeps", 1) * (2 * _heff_flops(d, a, b) + 4.0 * big * small * small)
                nbytes += 2.0 * case.get("sweeps", 1) * 8.0 * (2.0 * d * a * b + 5.0 * (a * a + b * b) + small * small)
        return {"bytes": nbytes, "flops": flops}
    if kind in ("heff", "env"):
        d, D1, D2 = case["twoS"] + 1, case["D1"], case["D2"]
        if kind == "heff":
            out = 4.0 if case["precision"] == "mixed" else 8.0
            return {"bytes": 8.0 * (5 * (D1 * D1 + D2 * D2) + d * D1 * D2) + out * d * D1 * D2, "flops": _heff_flops(d, D1, D2)}
        return {"bytes": 8.0 * (10 * (D1 * D1 + D2 * D2) + 2 * d * D1 * D2), "flops": 2 * _heff_flops(d, D1, D2)}
    if kind in ("qr", "lq", "svd"):
        m, n = max(case["m"], case["n"]), min(case["m"], case["n"])
        flops = 4.0 * m * n * n - 4.0 * n ** 3 / 3.0
        if kind == "svd":
            flops = 6.0 * m * n * n + 11.0 * n ** 3  # thin U, s, V by a Golub-Reinsch count
        return {"bytes": 8.0 * (2.0 * m * n + n * n), "flops": flops}
    if kind == "itebd":
        d, D = case["twoS"] + 1, case["D"]
        m = d * D
        return {"bytes": case["steps"] * 3 * 8.0 * 4 * d * D * D, "flops": case["steps"] * 3 * (2.0 * d * d * D ** 3 + 17.0 * m ** 3)}
    if kind == "fullstate":
        d, L = case["twoS"] + 1, case["L"]
        N = float(d ** L)
        return {"bytes": 20 * 2 * 8.0 * N, "flops": 20 * 2.0 * (L - 1) * N * (d if d == 2 else 3)}  # a Krylov space of 20
    n = case["n"]
    per = 2.0 * (4 * 64 + 64 * 64 + 64)
    return {"bytes": n * (16.0 + 4 + 16 + 4), "flops": n * (3 * per + per)}


# ---- the same values in 64 bits ---------------------------------------------


def exact(case, seed):
    kind = case["kind"]
    if kind in ("heff", "env"):
        F, G, x = (t.cuda() for t in _site_operands(case, seed))
        W = torch.from_numpy(_mpo(case["twoS"])).cuda()
        # torch blocks are transposed: F[w, j, i] with i the bra index, x[n, i2, i1]
        if kind == "heff":
            P = torch.einsum("wji,nbj->wnib", F, x)
            Q = torch.einsum("vwmn,vnib->wmib", W, P)
            return torch.einsum("wmib,wbc->mci", Q, G)
        P = torch.einsum("wji,nbj->wnib", F, x)
        Q = torch.einsum("vwmn,vnib->wmib", W, P)
        left = torch.einsum("mai,wmib->wba", x, Q)
        P = torch.einsum("wba,nbj->wnaj", G, x)
        Q = torch.einsum("vwmn,wnaj->vmaj", W, P)
        right = torch.einsum("mai,vmaj->vji", x, Q)
        return left, right
    if kind in ("qr", "lq", "svd"):
        A = _graded(np.random.default_rng(seed), case["m"], case["n"], 3 if kind == "svd" else 5)
        if kind == "qr":
            Q, R = torch.linalg.qr(A)
            return Q.T.contiguous(), R.T.contiguous()
        if kind == "lq":
            Q, R = torch.linalg.qr(A.T)
            return R.contiguous(), Q.contiguous()
        U, s, Vt = torch.linalg.svd(A, full_matrices=False)
        return _signed(U.T, s, Vt.T)
    if kind == "learned":
        return _learned_exact(case["n"], seed)
    return None


def _learned_exact(n, seed):
    F, T, p = (torch.from_numpy(a).double() for a in _pairs(n, seed))

    def net(q, F):
        h1 = torch.tanh(F @ q[:256].view(4, 64) + q[256:320])
        h2 = torch.tanh(h1 @ q[320:4416].view(64, 64) + q[4416:4480])
        return h2 @ q[4480:4544] + q[4544]

    q = p.clone().requires_grad_(True)
    loss = ((net(q, F) - T) ** 2).mean()
    loss.backward()
    with torch.no_grad():
        y = net(p.bfloat16().double(), F)  # inference reads the weights rounded to BF16
    return q.grad, loss.detach().item(), y
