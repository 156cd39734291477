"""Performance cases: the work a user of the framework has it do, by public entry point.

Five paths, each over the range of sizes its entry point is used at:

* ``newton``: one predictor-corrector Newton step of a dense SDP on a handle that
  stays on the GPU (`CudaBackend`, the backend seam a host interior-point loop
  drives): residuals and block factors, Schur assembly, its factorization, the
  predictor, the affine step bounds, the corrector with refinement, the step
  lengths.  FP64 or mixed precision, with or without equality rows.
* ``solve``: a bounded number of interior-point iterations of a whole solve,
  through `solve` (upload and teardown included) or on a kept handle.
* ``normal``: the reduced normal system of an LP with Lorentz cones
  (`NormalSystem`): NT scaling, assembly, factorization, one solve.
* ``batch``: many small SDPs at once (`BatchSolver`).
* ``adjoint``: the backward direction, gradients of a loss of the solution with
  respect to the data, with the refactorization it needs.

Solves run a fixed number of iterations (three; two for the tiny problems of a batch,
which are feasible to the last digit by then): from there on the controller compares
residuals at the rounding floor, so which branch a complete solve takes, and with it
the last digits of its answer, is decided by rounding.  They run in FP64: the mixed
mode's predictor is only solved to 1e-8, which stays in the iterates, so that mode is
covered by its Newton steps, refined in both stages.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "sdpx.jl_b200"))

import sdpx_b200  # noqa: E402
from sdpx_b200.batch import BatchSolver, batch_options  # noqa: E402
from sdpx_b200.controller import SolverOptions  # noqa: E402
from sdpx_b200.cuda_backend import CudaBackend  # noqa: E402
from sdpx_b200.generators import sdpa_dense  # noqa: E402
from sdpx_b200.normal import NormalSystem  # noqa: E402
from sdpx_b200.problem import SDPProblem  # noqa: E402

DEV = "cuda"
F64 = torch.float64


def _newton(name, m, blocks, lp=0, n_eq=0, precision="fp64"):
    case = dict(kind="newton", m=m, blocks=blocks, lp=lp, n_eq=n_eq, precision=precision)
    return dict(case, name=name) if name else case


def _solve(name, m, blocks, lp=0, iterations=3, handle=False):
    case = dict(kind="solve", m=m, blocks=blocks, lp=lp, n_eq=0, iterations=iterations,
                handle=handle)
    return dict(case, name=name) if name else case


def _normal(name, m, n_lp, cones, order):
    case = dict(kind="normal", m=m, n_lp=n_lp, cones=cones, order=order)
    return dict(case, name=name) if name else case


def _batch(name, count, n_min, n_max, m_cap, iterations=2):
    case = dict(kind="batch", count=count, n_min=n_min, n_max=n_max, m_cap=m_cap,
                iterations=iterations)
    return dict(case, name=name) if name else case


def _adjoint(name, m, blocks):
    case = dict(kind="adjoint", m=m, blocks=blocks, lp=0, n_eq=0, wrt=10)
    return dict(case, name=name) if name else case


def listed():
    return [
        # The smallest step, as in a control loop or a test model: launches and
        # read-backs are all there is.
        _newton("newton_m24_n12", 24, "12"),
        # Odd orders, two unequal blocks, nonnegatives and a few equality rows:
        # what a modelling front end hands over.
        _newton("newton_m333_61_17_eq5", 333, "61+17", lp=29, n_eq=5),
        # The differentiable-SDP size of the benchmark.
        _newton("newton_m500_n200", 500, "200"),
        # Half the headline size (two blocks and nonnegatives), all FP64.
        _newton("newton_m1000_200_100_lp250", 1000, "200+100", lp=250),
        # The headline size in the mixed mode, which the headline solve runs in.
        _newton("newton_mixed_m2000_400_200", 2000, "400+200", lp=500, precision="mixed"),
        # A user's whole call on a small model: upload, cold start, iterations.
        _solve("solve_m100_n50", 100, "50"),
        # The headline instance's solve on a kept handle.
        _solve("solve_m2000_400_200_lp500", 2000, "400+200", lp=500, handle=True),
        # A small ragged LP + Lorentz-cone system.
        _normal("normal_m317_ragged", 317, 2111, 9, 33),
        # The benchmark's LP + Lorentz-cone system.
        _normal("normal_m3000", 3000, 20000, 100, 64),
        # A few dozen tiny SDPs (one per node of a search tree).
        _batch("batch_48_tiny", 48, 4, 24, 60),
        # A slice of the small-SDP workload of uneven sizes.
        _batch("batch_512_uneven", 512, 4, 64, 200),
        # Gradients at the differentiable-SDP size.
        _adjoint("adjoint_m500_n200", 500, "200"),
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["newton", "newton", "newton", "solve", "normal", "batch", "adjoint"])
    if kind == "normal":
        m = _log_int(rng, 150, 2600)
        return _normal(None, m, _log_int(rng, 3 * m, 7 * m), rng.randint(3, 90),
                       rng.randint(5, 64))
    if kind == "batch":
        return _batch(None, _log_int(rng, 24, 400), 4, rng.randint(12, 64), rng.randint(40, 200))
    k = _log_int(rng, 12, 300)
    # fewer variables than the block has entries, so that S is nonsingular
    m = min(1600, max(16, _log_int(rng, k, 6 * k)), k * (k + 1) // 3)
    if kind == "adjoint":
        return _adjoint(None, m, str(k))
    blocks = str(k) + ("+%d" % rng.randint(3, max(4, k // 2)) if rng.random() < 0.5 else "")
    lp = rng.choice([0, rng.randint(1, 500)])
    if kind == "solve":
        if k <= 80:
            return _solve(None, m, blocks, lp=lp % 40)
        return _solve(None, m, blocks, lp=lp, handle=True)
    n_eq = rng.choice([0, 0, rng.randint(1, max(1, min(40, m // 8)))])
    mixed = k >= 60 and rng.random() < 0.4
    return _newton(None, m, blocks, lp=lp, n_eq=n_eq, precision="mixed" if mixed else "fp64")


# ---------------------------------------------------------------------------
#   Inputs
# ---------------------------------------------------------------------------

def _orders(case):
    return [int(b) for b in case["blocks"].split("+")]


def _spd(g, k, lo, hi):
    """Q·diag(d)·Qᵀ, d log-uniform in [lo, hi]."""
    q, _ = torch.linalg.qr(torch.randn(k, k, generator=g, dtype=F64, device=DEV))
    e = torch.rand(k, generator=g, dtype=F64, device=DEV)
    d = lo * (hi / lo) ** e
    x = (q * d) @ q.T
    return 0.5 * (x + x.T)


def _near_identity(g, k):
    w = torch.randn(k, k, generator=g, dtype=F64, device=DEV)
    return torch.eye(k, dtype=F64, device=DEV) + 0.1 * (w @ w.T) / k


def _sdp(case, seed):
    """A strictly feasible SDP in SDPX's form and an interior iterate in mid-solve.

    Per block A_i = (G + Gᵀ)/2, c = 𝒜ᵀX0 (+ B·y1), C = 𝒜y0 − Z0 and b = Bᵀy0 with
    X0, Z0 ≻ 0; the nonnegatives are one 'lp' vector here and 1×1 blocks in
    the library.  The iterate has eigenvalues over two decades."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    m, ks, lp, ne = case["m"], _orders(case), case["lp"], case["n_eq"]
    A, C, X, Y = [], [], [], []
    y0 = torch.randn(m, generator=g, dtype=F64, device=DEV)
    c = torch.zeros(m, dtype=F64, device=DEV)
    for k in ks:
        a = torch.randn(m, k, k, generator=g, dtype=F64, device=DEV)
        a += a.transpose(1, 2).clone()
        a *= 0.5
        a = a.reshape(m, k * k)
        c += a @ _near_identity(g, k).reshape(-1)
        r = (y0 @ a).reshape(k, k) - _near_identity(g, k)
        A.append(a)
        C.append(0.5 * (r + r.T))
        x = _spd(g, k, 0.1, 10.0)
        lam, v = torch.linalg.eigh(x)
        xis = (v * lam.rsqrt()) @ v.T  # X^{-1/2}
        y = xis @ _near_identity(g, k) @ xis
        X.append(x)
        Y.append(0.5 * (y + y.T))
    alp = torch.randn(m, lp, generator=g, dtype=F64, device=DEV)
    c += alp @ (0.5 + torch.rand(lp, generator=g, dtype=F64, device=DEV))
    clp = y0 @ alp - (0.5 + torch.rand(lp, generator=g, dtype=F64, device=DEV))
    xlp = 0.1 * 100.0 ** torch.rand(lp, generator=g, dtype=F64, device=DEV)
    ylp = (0.9 + 0.2 * torch.rand(lp, generator=g, dtype=F64, device=DEV)) / xlp
    B = torch.randn(m, ne, generator=g, dtype=F64, device=DEV)
    b = B.T @ y0
    y1 = torch.randn(ne, generator=g, dtype=F64, device=DEV)
    c += B @ y1
    x = y0 + 0.1 * torch.randn(m, generator=g, dtype=F64, device=DEV)
    wx = torch.randn(m, generator=g, dtype=F64, device=DEV)
    WY = [torch.randn(k, k, generator=g, dtype=F64, device=DEV) for k in ks]
    return dict(m=m, ks=ks, lp=lp, ne=ne, A=A, C=C, c=c, alp=alp, clp=clp, B=B, b=b, x=x, X=X, Y=Y,
                xlp=xlp, ylp=ylp, wx=wx, WY=[w + w.T for w in WY])


def _problem(d):
    """The `SDPProblem` (host arrays) of `_sdp`."""
    lp = d["lp"]
    alp = d["alp"].T.contiguous().cpu().numpy().reshape(lp, d["m"], 1)
    clp = d["clp"].cpu().numpy()
    return SDPProblem(d["c"].cpu().numpy(), d["ks"] + [1] * lp,
                      [a.cpu().numpy() for a in d["A"]] + [alp[j] for j in range(lp)],
                      [a.cpu().numpy() for a in d["C"]] + [clp[j:j + 1].reshape(1, 1)
                                                           for j in range(lp)],
                      d["B"].cpu().numpy(), d["b"].cpu().numpy())


def _iterate(d):
    def blocks(dense, lp):
        lp = lp.cpu().numpy()
        return [a.cpu().numpy() for a in dense] + [v.reshape(1, 1) for v in lp]
    return d["x"].cpu().numpy(), blocks(d["X"], d["xlp"]), blocks(d["Y"], d["ylp"])


def _normal_data(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    m, nl, nc, q = case["m"], case["n_lp"], case["cones"], case["order"]
    n = nl + nc * q
    B = torch.randn(n, m, generator=g, dtype=F64, device=DEV)
    B *= torch.rand(n, m, generator=g, dtype=torch.float32, device=DEV) < 0.1
    w = (0.5 + torch.rand(nl, generator=g, dtype=F64, device=DEV))
    w /= 0.5 + torch.rand(nl, generator=g, dtype=F64, device=DEV)

    def points():
        u = torch.randn(nc, q, generator=g, dtype=F64, device=DEV)
        u[:, 0] = 1.5 * u[:, 1:].norm(dim=1) + 1.0
        return u
    s, z = points(), points()
    rhs = torch.randn(n + m, generator=g, dtype=F64, device=DEV)
    return dict(B=B, w=w, s=s, z=z, rhs=rhs, n=n, m=m)


NORMAL_REG = 1e-10


def _batch_sizes(case):
    """(n, m) of every instance, the distribution of `batch_instances`: a
    program that solves batch after batch keeps the sizes and changes the data."""
    rng = np.random.default_rng(0)
    out = []
    for _ in range(case["count"]):
        n = int(rng.integers(case["n_min"], case["n_max"] + 1))
        out.append((n, int(rng.integers(3, min(case["m_cap"], n * (n + 1) // 2) + 1))))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        probs = [sdpa_dense(m=m, blocks=[n], seed=int(seed) * 1_000_003 + i)
                 for i, (n, m) in enumerate(_batch_sizes(case))]
        return dict(kind=kind, solver=BatchSolver(probs), opts=batch_options(
            1e-8, iter_max=case["iterations"]))
    if kind == "normal":
        d = _normal_data(case, seed)
        ns = NormalSystem(np.asfortranarray(d["B"].cpu().numpy()), case["n_lp"],
                          [case["order"]] * case["cones"])
        host = {k: d[k].reshape(-1).cpu().numpy() for k in ("w", "s", "z", "rhs")}
        torch.cuda.empty_cache()
        return dict(kind=kind, system=ns, **host)
    d = _sdp(case, seed)
    prob = _problem(d)
    x, X, Y = _iterate(d)
    wx, WY = d["wx"].cpu().numpy(), [w.cpu().numpy() for w in d["WY"]]
    del d
    torch.cuda.empty_cache()
    if kind == "solve":
        opts = SolverOptions(iter_max=case["iterations"]).with_tolerance(1e-8)
        return dict(kind=kind, prob=prob, be=CudaBackend(prob) if case["handle"] else None,
                    opts=opts, iterations=case["iterations"])
    be = CudaBackend(prob, precision=case.get("precision", "fp64"))
    be.set_iterate(x, X, Y, y=np.zeros(case["n_eq"]))
    L = prob.L
    mu = [0.1 * float(np.vdot(a, b)) / a.shape[0] for a, b in zip(X, Y)]
    if kind == "newton":
        be.begin_iteration(None)  # leaves the cold start: the requested precision from here on
        return dict(kind=kind, be=be, mu=mu, mixed=case["precision"] == "mixed")
    return dict(kind=kind, be=be, x=x, X=X, Y=Y, wx=wx, WY=WY, zero=[0.0] * L,
                wrt=list(range(min(case["wrt"], prob.m))))


# ---------------------------------------------------------------------------
#   One pass
# ---------------------------------------------------------------------------

def _stack(blocks):
    return np.concatenate([np.asarray(b).reshape(-1) for b in blocks])


def _run_newton(s):
    be = s["be"]
    be.compute_residuals(s["mu"], True, True)
    be.schur_build()
    be.factorize()
    be.predictor_rhs()
    be.solve_direction()
    if s["mixed"]:
        be.refine("auto", 0.0, 8, 1)
    be.direction_blocks()
    p = be.affine_diagnostics(True)
    sigma = min(1.0, max(p["mu_aff"] / p["mu"], 0.0)) ** 3
    be.mehrotra_corrector_rhs(sigma, p["mu"], not p["uniform"])
    be.solve_direction()
    be.refine("auto", 0.0, 8, 1)
    be.direction_residual()
    be.direction_blocks()
    tX, tY = be.line_search("backtrack", 0.9, 0.9, 0.9, 1e-10, 1.4901161193847656e-08)
    dx, dX, dY = be.get_direction()
    return dict(dx=dx, dX=_stack(dX), dY=_stack(dY), dy=be.get_equality_direction(),
                steps=np.array([p["tX"], p["tY"], tX, tY]))


def _run_adjoint(s):
    be = s["be"]
    be.set_iterate(s["x"], s["X"], s["Y"])
    be.compute_residuals(s["zero"], True, True)
    be.schur_build()
    be.factorize()
    g = be.adjoint(wx=s["wx"], WY=s["WY"], A_index=s["wrt"])
    return dict(grad_c=g["grad_c"], grad_C=_stack(g["grad_C"]),
                grad_A=_stack([_stack(a) for a in g["grad_A"]]))


def run(state):
    kind = state["kind"]
    if kind == "newton":
        return _run_newton(state)
    if kind == "adjoint":
        return _run_adjoint(state)
    if kind == "normal":
        ns = state["system"]
        _, _, nt = ns.soc_nt_scaling(state["s"], state["z"])
        ns.factor_reduced(state["w"], NORMAL_REG)
        return dict(sol=ns.solve_factor(state["rhs"]), w=nt["w"], lam=nt["lambda"])
    if kind == "batch":
        res = state["solver"].optimize(state["opts"])
        return dict(x=np.concatenate([r.x for r in res]),
                    X=_stack([r.X[0] for r in res]), Y=_stack([r.Y[0] for r in res]),
                    iterations=np.array([r.iterations for r in res]))
    if state["be"] is not None:
        state["be"].reset()
        r = state["be"].optimize(state["opts"])
    else:
        r = sdpx_b200.solve(state["prob"], maximum_iterations=state["iterations"])
    return dict(x=r.x, X=_stack(r.X), Y=_stack(r.Y), iterations=r.iterations)


# ---------------------------------------------------------------------------
#   What a pass cannot do without
# ---------------------------------------------------------------------------

def _step_work(m, ks, lp):
    """(bytes, flops) of one Newton step: the lower triangles of 𝒜 read once, S
    written and read once, the iterate and the direction; the products
    L_X⁻¹·A_i·L_Y, the Gram, its Cholesky and the step-length factors."""
    kt = sum(k * (k + 1) // 2 for k in ks) + lp
    kf = sum(k * k for k in ks) + lp
    b = 8.0 * (kt * m + m * m + 6 * kf + 4 * m)
    f = 2.0 * m * sum(k ** 3 for k in ks) + float(m) * m * kf + m ** 3 / 3.0
    f += sum(20.0 * k ** 3 for k in ks) + 8.0 * kt * m
    return b, f


def work(case):
    kind = case["kind"]
    if kind == "normal":
        n, m = case["n_lp"] + case["cones"] * case["order"], case["m"]
        return dict(bytes=8.0 * (n * m + m * m + 4 * n), flops=float(m) * m * n + m ** 3 / 3.0)
    if kind == "batch":
        b = f = 0.0
        for k, m in _batch_sizes(case):
            bi, fi = _step_work(m, [k], 0)
            b, f = b + bi, f + case["iterations"] * fi
        return dict(bytes=b, flops=f)
    b, f = _step_work(case["m"], _orders(case), case["lp"])
    if kind == "solve":
        it = case["iterations"]
        # 𝒜 does not stay on the chip between iterations where it exceeds the L2
        return dict(bytes=b * (it if b > 1.2e8 else 1), flops=f * it)
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------
#   The same in plain 64-bit torch
# ---------------------------------------------------------------------------

class _Exact:
    """The HKM Newton system at the iterate of `_sdp`."""

    def __init__(self, d):
        self.d, m = d, d["m"]
        self.Xi = [torch.linalg.inv(x) for x in d["X"]]
        S = torch.zeros(m, m, dtype=F64, device=DEV)
        for k, A, Xi, Y in zip(d["ks"], d["A"], self.Xi, d["Y"]):
            a = A.reshape(m, k, k)
            for i in range(0, m, 250):  # rows ⟨X⁻¹·A_i·Y, A_j⟩
                S[i:i + 250] += (Xi @ a[i:i + 250] @ Y).reshape(-1, k * k) @ A.T
        S += (d["alp"] * (d["ylp"] / d["xlp"])) @ d["alp"].T
        self.S = 0.5 * (S + S.T)
        self.P = [((d["x"] @ A).reshape(k, k) - X - C)
                  for k, A, X, C in zip(d["ks"], d["A"], d["X"], d["C"])]
        self.Plp = d["x"] @ d["alp"] - d["xlp"] - d["clp"]
        self.dres = d["c"] - self.at(d["Y"], d["ylp"])
        self.p = d["b"] - d["B"].T @ d["x"]
        ne = d["ne"]
        K = torch.zeros(m + ne, m + ne, dtype=F64, device=DEV)
        K[:m, :m] = self.S
        K[:m, m:] = -d["B"]
        K[m:, :m] = d["B"].T
        self.K, self.lu = K, torch.linalg.lu_factor(K)

    def at(self, Z, zlp):
        d = self.d
        v = d["alp"] @ zlp
        for A, z in zip(d["A"], Z):
            v = v + A @ z.reshape(-1)
        return v

    def kkt(self, r, p):
        b = torch.cat([r, p])[:, None]
        s = torch.linalg.lu_solve(*self.lu, b)
        s = s + torch.linalg.lu_solve(*self.lu, b - self.K @ s)
        return s[:self.d["m"], 0], s[self.d["m"]:, 0]

    def direction(self, R, Rlp):
        d = self.d
        Z = [Xi @ (P @ Y - r) for Xi, P, Y, r in zip(self.Xi, self.P, d["Y"], R)]
        zlp = (self.Plp * d["ylp"] - Rlp) / d["xlp"]
        dx, dy = self.kkt(-(self.dres + self.at(Z, zlp)), self.p)
        dX = [(dx @ A).reshape(k, k) + P for k, A, P in zip(d["ks"], d["A"], self.P)]
        dX = [0.5 * (v + v.T) for v in dX]
        dY = [Xi @ (r - u @ Y) for Xi, r, u, Y in zip(self.Xi, R, dX, d["Y"])]
        dxl = dx @ d["alp"] + self.Plp
        return dx, dy, dX, [0.5 * (v + v.T) for v in dY], dxl, (Rlp - dxl * d["ylp"]) / d["xlp"]


def _bound(M, dM, v, dv):
    """Largest t ≤ 1 with M + t·dM ⪰ 0 in every block."""
    t = 1.0
    for a, da in zip(M, dM):
        L = torch.linalg.cholesky(a)
        G = torch.linalg.solve_triangular(L, da, upper=False)
        G = torch.linalg.solve_triangular(L, G.T.contiguous(), upper=False)
        low = float(torch.linalg.eigvalsh(0.5 * (G + G.T))[0])
        t = min(t, -1.0 / low) if low < -1.0 else t
    neg = dv < -v
    return min(t, float((-v[neg] / dv[neg]).min())) if bool(neg.any()) else t


def _exact_newton(d):
    e = _Exact(d)
    X, Y, xl, yl = d["X"], d["Y"], d["xlp"], d["ylp"]
    R = [-(x @ y) for x, y in zip(X, Y)]
    dx, dy, dX, dY, dxl, dyl = e.direction(R, -xl * yl)
    aX, aY = _bound(X, dX, xl, dxl), _bound(Y, dY, yl, dyl)
    n = sum(d["ks"]) + d["lp"]
    dots = [float((x * y).sum()) for x, y in zip(X, Y)]
    mu = (sum(dots) + float(xl @ yl)) / n
    aff = sum(float(((x + aX * u) * (y + aY * v)).sum()) for x, u, y, v in zip(X, dX, Y, dY))
    aff = (aff + float((xl + aX * dxl) @ (yl + aY * dyl))) / n
    sigma = min(1.0, max(max(0.0, aff) / mu, 0.0)) ** 3
    one = len(d["ks"]) + d["lp"] == 1  # a single block: its own mean is the common one
    eye = [torch.eye(k, dtype=F64, device=DEV) for k in d["ks"]]
    R = [sigma * (mu if one else t / k) * i - x @ y - u @ v
         for t, k, i, x, y, u, v in zip(dots, d["ks"], eye, X, Y, dX, dY)]
    Rlp = sigma * xl * yl - xl * yl - dxl * dyl
    dx, dy, dX, dY, dxl, dyl = e.direction(R, Rlp)
    steps = [aX, aY]
    for M, dM, v, dv in ((X, dX, xl, dxl), (Y, dY, yl, dyl)):
        t, top = 1.0, _bound(M, dM, v, dv)
        while t > top or (t == 1.0 and top == 1.0 and not _interior(M, dM, v, dv)):
            t *= 0.9
        steps.append(t)

    def stack(dense, lp):
        return torch.cat([a.reshape(-1) for a in dense] + [lp]).cpu().numpy()
    return dict(dx=dx.cpu().numpy(), dX=stack(dX, dxl), dY=stack(dY, dyl), dy=dy.cpu().numpy(),
                steps=np.array(steps))


def _interior(M, dM, v, dv):
    return bool((v + dv > 0).all()) and all(
        int(torch.linalg.cholesky_ex(a + da)[1]) == 0 for a, da in zip(M, dM))


def _exact_adjoint(d, wrt):
    e = _Exact(d)
    G = [Xi @ W @ Y for Xi, W, Y in zip(e.Xi, d["WY"], d["Y"])]
    lx, _ = e.kkt(d["wx"] - e.at(G, torch.zeros(0, dtype=F64, device=DEV)), e.p * 0)
    gC = []
    for k, A, Xi, Y, g in zip(d["ks"], d["A"], e.Xi, d["Y"], G):
        z = Xi @ (lx @ A).reshape(k, k) @ Y
        gC.append(0.5 * (z + z.T) + 0.5 * (g + g.T))
    gA = [torch.cat([(lx[i] * Y - d["x"][i] * c).reshape(-1) for Y, c in zip(d["Y"], gC)])
          for i in range(wrt)]
    return dict(grad_c=(-lx).cpu().numpy(),
                grad_C=torch.cat([c.reshape(-1) for c in gC]).cpu().numpy(),
                grad_A=torch.cat(gA).cpu().numpy())


def _exact_normal(case, d):
    nl, q = case["n_lp"], case["order"]
    B, s, z = d["B"], d["s"], d["z"]
    det = lambda v: (v[:, 0] - v[:, 1:].norm(dim=1)) * (v[:, 0] + v[:, 1:].norm(dim=1))  # noqa: E731
    ss, zs = det(s).sqrt()[:, None], det(z).sqrt()[:, None]
    J = torch.ones(q, dtype=F64, device=DEV)
    J[1:] = -1.0
    a, b = s / ss, z / zs
    gamma = ((1.0 + (a * b).sum(1, keepdim=True)) / 2.0).sqrt()
    w = (a + J * b) / (2.0 * gamma)
    eta2 = ss / zs
    wd = eta2.sqrt()
    zt = (w[:, 1:] * z[:, 1:]).sum(1, keepdim=True)
    lam = torch.cat([wd * (w[:, :1] * z[:, :1] + zt),
                     wd * (z[:, 1:] + (z[:, :1] + zt / (1.0 + w[:, :1])) * w[:, 1:])], 1)

    def hinv(v):  # (2·Jw·(Jw)ᵀ − J)/eta² on each cone's coordinates, v: n × columns
        top = v[:nl] / (d["w"] + NORMAL_REG)[:, None]
        u = v[nl:].reshape(case["cones"], q, -1)
        jw = (J * w)[:, :, None]
        low = (2.0 * jw * (jw * u).sum(1, keepdim=True) - J[None, :, None] * u) / eta2[:, :, None]
        return torch.cat([top, low.reshape(-1, v.shape[1])])
    Q = B.T @ hinv(B)
    Q = 0.5 * (Q + Q.T)
    Q.diagonal().add_(NORMAL_REG)
    rx, ry = d["rhs"][:d["n"], None], d["rhs"][d["n"]:, None]
    t = hinv(rx)
    lu = torch.linalg.lu_factor(Q)
    r = ry - B.T @ t
    dy = torch.linalg.lu_solve(*lu, r)
    dy = dy + torch.linalg.lu_solve(*lu, r - Q @ dy)
    dx = t + hinv(B @ dy)
    return dict(sol=torch.cat([dx, dy])[:, 0].cpu().numpy(), w=w.reshape(-1).cpu().numpy(),
                lam=lam.reshape(-1).cpu().numpy())


def exact(case, seed):
    kind = case["kind"]
    if kind == "normal":
        return _exact_normal(case, _normal_data(case, seed))
    if kind in ("batch", "solve"):
        return None  # iterates of a loop: no closed form
    d = _sdp(case, seed)
    return _exact_newton(d) if kind == "newton" else _exact_adjoint(d, min(case["wrt"], d["m"]))
