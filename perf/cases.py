"""What a program does with this package, as cases that can be timed and compared.

The unit of almost every use is one alpha of the sweep: a warm-started leading-eigenvector solve of
D^{-a/2} (J/c) D^{-a/2}. Around it stand the fused operator by itself, the batched local search of the
rounded candidates, whole solves (single and batched) and the differentiation form. The graphs are the
package's own seeded generators with the sizes of its benchmark configurations: Erdos-Renyi
n = 1024 (expected degree 20), Barabasi-Albert n = 2^16 (precision study), n = 2^18 (differentiation) and
n = 2^20 (headline), and the ragged batch of n = 2^10 .. 2^14.

An eigenvector is unique up to its sign. The alpha cases are warm-started, so the previous vector fixes
it; the whole FP64 solve reports the side of the cut on which each vertex lies relative to vertex 0.
In FP32 the signs of eigenvector entries at rounding level decide single spins, so FP32 solves are
compared by the eigenvalues of all their alphas, and the local search by its exact integers from given
candidates.
"""
import numpy as np
import scipy.sparse as sp
import torch

from specann_b200 import _lib, graphs
from specann_b200.batch import BatchedSpectralAnnealing
from specann_b200.differentiation import EigenProblem, smoothed_energy
from specann_b200.engine import Engine
from specann_b200.spectral_annealing import SpectralAnnealing, default_ncv, gershgorin_bound

STARTS = {"diagonal": _lib.SA_START_DIAGONAL, "prev": _lib.SA_START_PREV}
STEPS = 60           # Lanczos steps that one alpha takes (20 .. 150 over a sweep)
LS_PASSES = 60       # local-search passes until no candidate improves (40 .. 110)


def listed():
    return [
        # the smallest instance in use (Gset-sized MaxCut): every phase is latency
        {"name": "alpha_er1024", "do": "alpha", "graph": "er", "n": 1024, "deg": 20, "couplings": "unit",
         "precision": 32, "alpha": 0.6, "before": 0.59, "start": "diagonal"},
        # a mid-sized signed Ising instance with an odd number of spins, continued from the vector before
        {"name": "alpha_ba23456_pm1", "do": "alpha", "graph": "ba", "n": 23456, "deg": 10, "couplings": "pm1",
         "precision": 32, "alpha": 0.35, "before": 0.34, "start": "prev"},
        # the all-FP64 arm of the precision study
        {"name": "alpha_ba65536_f64", "do": "alpha", "graph": "ba", "n": 1 << 16, "deg": 20, "couplings": "unit",
         "precision": 64, "alpha": 0.75, "before": 0.745, "start": "diagonal"},
        # one alpha of the headline solve: where most of a large run's time goes
        {"name": "alpha_ba1048576", "do": "alpha", "graph": "ba", "n": 1 << 20, "deg": 20, "couplings": "unit",
         "precision": 32, "alpha": 0.7, "before": 0.695, "start": "diagonal"},
        # the fused operator alone (power iterations, residual checks) at the headline size, and with
        # couplings of many magnitudes at a ragged one
        {"name": "operator_ba1048576", "do": "operator", "graph": "ba", "n": 1 << 20, "deg": 20, "couplings": "unit",
         "precision": 32, "alpha": 0.5},
        {"name": "operator_ba150001_int", "do": "operator", "graph": "ba", "n": 150001, "deg": 20,
         "couplings": "int100", "precision": 32, "alpha": 0.8},
        # the local search of a full sweep's candidates, and of a part of them on a larger weighted graph
        {"name": "search_ba65536_k128", "do": "search", "graph": "ba", "n": 1 << 16, "deg": 20, "couplings": "unit",
         "precision": 32, "k": 128},
        {"name": "search_ba200003_k40_int", "do": "search", "graph": "ba", "n": 200003, "deg": 15,
         "couplings": "int100", "precision": 32, "k": 40},
        # whole solves from a host CSR: the small configuration in FP64, the headline graph on a short schedule
        {"name": "solve_er1024_f64", "do": "solve", "graph": "er", "n": 1024, "deg": 20, "couplings": "unit",
         "precision": 64, "alphas": 128},
        {"name": "solve_ba1048576", "do": "solve", "graph": "ba", "n": 1 << 20, "deg": 20, "couplings": "unit",
         "precision": 32, "alphas": 24},
        # the ragged batch in one launch
        {"name": "batch_12x2", "do": "batch", "count": 12, "seeds": 2, "log2_max": 14, "alphas": 16},
        # one training step of the differentiation form: smoothed energy and its gradients, in the precision
        # that its finite-difference checks use
        {"name": "gradient_ba262144_pm1", "do": "gradient", "graph": "ba", "n": 1 << 18, "deg": 20,
         "couplings": "pm1", "precision": 64, "alpha": 0.5},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    do = rng.choice(["alpha", "alpha", "alpha", "operator", "operator", "search", "solve", "batch", "gradient"])
    graph = rng.choice(["ba", "ba", "er"])
    deg = rng.choice([20, 30]) if graph == "er" else rng.choice([10, 12, 15, 20])
    couplings = rng.choice(["unit", "pm1", "int100"])
    case = {"do": do, "graph": graph, "deg": deg, "couplings": couplings, "precision": 32}
    if do == "alpha":
        # unit couplings: their leading eigenvalue stays separated over these alphas
        case["couplings"] = "unit"
        case["n"] = size(1000, 1 << 20)
        case["precision"] = rng.choice([32, 32, 64]) if case["n"] < 300000 else 32
        case["alpha"] = round(rng.uniform(0.2, 0.85), 4)
        case["before"] = round(case["alpha"] - rng.uniform(0.003, 0.02), 4)
        case["start"] = rng.choice(["diagonal", "prev"])
    elif do == "operator":
        case["n"] = size(1000, 1 << 20)
        case["precision"] = rng.choice([32, 32, 64]) if case["n"] < 300000 else 32
        case["alpha"] = round(rng.uniform(0.0, 1.0), 4)
    elif do == "search":
        case["n"] = size(1000, 200000)
        case["k"] = rng.choice([1, 7, 16, 33, 64, 128]) if case["n"] < 70000 else rng.choice([1, 8, 24, 40])
    elif do == "solve":
        case["n"] = size(1000, 1 << 18)
        case["precision"] = 64 if case["n"] < 4000 else 32
        case["alphas"] = rng.choice([16, 32]) if case["n"] > 20000 else rng.choice([32, 64, 128])
    elif do == "batch":
        case = {"do": "batch", "count": rng.randrange(4, 13), "seeds": rng.choice([1, 2]),
                "log2_max": rng.choice([11, 12, 13, 14]), "alphas": rng.choice([8, 12, 16])}
    else:
        case["couplings"] = "pm1"
        case["precision"] = 64
        case["n"] = size(2000, 1 << 18)
        case["alpha"] = round(rng.uniform(0.3, 0.7), 4)
    return case


def _graph(case, seed):
    couplings = case["couplings"]
    dtype = np.float32 if case["precision"] == 32 else np.float64
    if case["graph"] == "er":
        J = graphs.erdos_renyi(case["n"], case["deg"] / (case["n"] - 1), seed=seed, couplings=couplings, dtype=dtype)
        return graphs.drop_isolated(J)
    return graphs.barabasi_albert(case["n"], case["deg"], seed=seed, couplings=couplings, dtype=dtype)


def _engine(J, precision, candidates):
    eng = Engine(J.shape[0], J.nnz, precision=precision, ncv_max=max(2, default_ncv(J.shape[0], None)),
                 max_candidates=candidates)
    info = eng.upload_csr(J.indptr, J.indices, J.data)
    if eng.panels_pay():
        eng.build_panels()
    return eng, info


class _Plain:
    """The normalised operator and its leading eigenvector in plain 64-bit torch on the GPU."""

    def __init__(self, J):
        self.n = J.shape[0]
        self.J = torch.sparse_csr_tensor(torch.from_numpy(J.indptr.astype(np.int64)),
                                         torch.from_numpy(J.indices.astype(np.int64)),
                                         torch.from_numpy(J.data.astype(np.float64)), size=J.shape,
                                         check_invariants=False).cuda()
        deg = torch.from_numpy(np.asarray(abs(J).sum(axis=1), dtype=np.float64).ravel()).cuda()
        self.c = float(deg.max())
        self.d = deg / self.c

    def scale(self, alpha):
        return self.d.pow(alpha).clamp_min(1e-12).rsqrt() / self.c ** 0.5

    def apply(self, x, alpha):
        s = self.scale(alpha)
        return s * (self.J @ (s * x))

    def leading(self, alpha, start, tol, restarts=60):
        """Unit leading eigenvector: Lanczos with full reorthogonalisation, restarted from its Ritz vector."""
        m = min(50, self.n - 1)
        y = start / start.norm()
        for _ in range(restarts):
            V = torch.zeros(m, self.n, dtype=torch.float64, device="cuda")
            T = torch.zeros(m, m, dtype=torch.float64)
            V[0] = y
            k = m
            for j in range(m):
                w = self.apply(V[j], alpha)
                h = V[: j + 1] @ w
                w = w - h @ V[: j + 1]
                w = w - (V[: j + 1] @ w) @ V[: j + 1]
                b = float(w.norm())
                T[j, j] = float(h[j])
                if j + 1 < m:
                    if b < 1e-14:
                        k = j + 1
                        break
                    T[j, j + 1] = T[j + 1, j] = b
                    V[j + 1] = w / b
            e, S = torch.linalg.eigh(T[:k, :k])
            z = S[:, -1].cuda() @ V[:k]
            z = z / z.norm()
            y = z if float(z @ y) >= 0 else -z
            if float((self.apply(y, alpha) - e[-1].cuda() * y).norm()) <= tol:
                break
        return float(e[-1]), y


def _start_vector(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, generator=g, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    do = case["do"]
    if do == "batch":
        inst = [J for _, J in graphs.ragged_batch(case["count"], seed=seed, log2_max=case["log2_max"])]
        b = BatchedSpectralAnnealing(seeds=range(1, case["seeds"] + 1), num_alphas=case["alphas"])
        return {"do": do, "batch": b.load(inst)}
    J = _graph(case, seed)
    n, precision = J.shape[0], case["precision"]
    vtype = torch.float32 if precision == 32 else torch.float64
    if do == "alpha":
        # the sweep's own situation: the graph is bound, the eigenvector of the alpha before is known
        plain = _Plain(J)
        lam, y = plain.leading(case["before"], _start_vector(n, seed), 1e-6)
        eng, info = _engine(J, precision, 4)
        last = y.to(vtype)
        eng.set_last_vector(last)
        g = gershgorin_bound(info.d_min, info.d_max, case["alpha"])
        return {"do": do, "engine": eng, "last": last, "args": dict(
            alpha=case["alpha"], alpha_prev=case["before"], rho=1.001 * max(g, lam), gershgorin=g, tol=1e-6,
            pred_tol=1e-3, maxiter=1000, ncv=default_ncv(n, None), start_mode=STARTS[case["start"]], seed=42,
            stream_id=4)}
    if do == "operator":
        eng, _ = _engine(J, precision, 4)
        x = _start_vector(n, seed).to(vtype)
        return {"do": do, "engine": eng, "x": x, "y": torch.empty_like(x), "alpha": case["alpha"]}
    if do == "search":
        # rounded vectors along the path between two ends, as a sweep leaves them
        plain = _Plain(J)
        a, z = (plain.leading(t, _start_vector(n, seed), 1e-2, restarts=1)[1] for t in (0.1, 0.95))
        eng, _ = _engine(J, precision, case["k"])
        z = z if float(a @ z) >= 0 else -z
        for c in range(case["k"]):
            t = (c + 0.5) / case["k"]
            eng.set_candidate(c, np.where(((1 - t) * a + t * z).cpu().numpy() >= 0, 1, -1).astype(np.int8))
        return {"do": do, "engine": eng, "k": case["k"]}
    if do == "solve":
        s = SpectralAnnealing("case", "cases", random_seed=42, precision=precision, num_alphas=case["alphas"],
                              write_results=False)
        return {"do": do, "solver": s, "J": J, "precision": precision}
    p = EigenProblem(J, precision=precision)
    return {"do": do, "problem": p, "alpha": case["alpha"], "offsets": torch.zeros(n, device="cuda")}


def run(state):
    do = state["do"]
    if do == "alpha":
        rec = state["engine"].alpha_solve(**state["args"])
        return {"mu": rec.mu, "y": state["engine"].result_vector()}
    if do == "operator":
        return state["engine"].spmv(state["alpha"], 1.001, state["x"], state["y"])
    if do == "search":
        before, after, _ = state["engine"].local_search(state["k"], seed=42)
        best = int(np.argmin(after))
        return {"before": before, "after": after, "spins": state["engine"].candidate_spins(best, refined=True)}
    if do == "solve":
        energy, spins, _ = state["solver"].solve(state["J"])
        lam = np.array([r["lambda1"] for r in state["solver"].alpha_results], dtype=spins.dtype)
        if state["precision"] == 32:
            return {"lambda1": lam}
        return {"lambda1": lam, "energy": energy, "side": spins == spins[0]}
    if do == "batch":
        b = state["batch"]
        b.sweep()
        rows = [r["rows"] for r in b.results()]
        return {"lambda1": np.array([[r["lambda1"] for r in p] for p in rows], dtype=np.float32)}
    alpha = torch.tensor(state["alpha"], requires_grad=True)
    offsets = state["offsets"].detach().requires_grad_()
    loss = smoothed_energy(state["problem"], alpha, offsets)
    loss.backward()
    return {"loss": loss.item(), "alpha": alpha.grad, "offsets": offsets.grad}


def exact(case, seed):
    do = case["do"]
    if do == "batch":
        return None
    J = _graph(case, seed)
    if do == "alpha":
        plain = _Plain(J)
        lam, before = plain.leading(case["before"], _start_vector(J.shape[0], seed), 1e-6)
        deg = np.asarray(abs(J).sum(axis=1), dtype=np.float64).ravel() / plain.c
        g = gershgorin_bound(float(deg.min()), float(deg.max()), case["alpha"])
        top, y = plain.leading(case["alpha"], before, 1e-12)
        return {"mu": 1.001 * max(g, lam) - top, "y": y if float(y @ before) >= 0 else -y}
    if do == "operator":
        dtype = torch.float32 if case["precision"] == 32 else torch.float64
        x = _start_vector(J.shape[0], seed).to(dtype).double()
        return 1.001 * x - _Plain(J).apply(x, case["alpha"])
    if do == "gradient" and J.shape[0] <= 4096:
        deg = torch.from_numpy(np.asarray(abs(J).sum(axis=1), dtype=np.float64).ravel()).cuda()
        d = deg / deg.max()
        A = torch.from_numpy(J.toarray().astype(np.float64)).cuda()
        s = d.pow(-0.5 * case["alpha"])
        M = s[:, None] * A * s[None, :] / deg.max()
        lam, Y = torch.linalg.eigh(M)
        y, beta = Y[:, -1], 8.0
        t = torch.tanh(beta * s * y)
        At = A @ t
        gx = -At * beta * (1 - t * t)
        r = s * gx
        w = Y[:, :-1] @ ((Y[:, :-1].T @ r) / (lam[-1] - lam[:-1]))
        l = -0.5 * torch.log(d)
        off = l * (y * (M @ w) + w * (M @ y)) + l * gx * s * y
        return {"loss": -0.5 * t @ At, "alpha": off.sum(), "offsets": off}
    return None


def work(case):
    """Bytes and operations without which a pass cannot do: the couplings are streamed once per operator
    application (4-byte columns and values) with the vectors that it reads and writes."""
    do = case["do"]
    if do == "batch":
        # sizes are log-uniform from 2^10 to 2^log2_max, of mean degree 25
        lo, hi = 2.0 ** 10, 2.0 ** case["log2_max"]
        mean = (hi - lo) / np.log(hi / lo)
        entries = 25 * mean * case["count"] * case["seeds"] * case["alphas"] * STEPS
        return {"bytes": 8 * entries, "flops": 2 * entries}
    n = case["n"]
    t = 4 if case["precision"] == 32 else 8
    nnz = n * case["deg"] * (1 if case["graph"] == "er" else 2)
    apply_bytes = nnz * (4 + t) + 4 * n + 3 * n * t
    if do == "operator":
        return {"bytes": apply_bytes, "flops": 2 * nnz}
    if do == "search":
        k = case["k"]
        row = nnz * (4 + t) + 4 * n + 2 * n * ((k + 7) // 8)
        return {"bytes": row + 4 * n * k + 2 * n * k * LS_PASSES // 64, "flops": 2.0 * nnz * k}
    # Lanczos: one application, and the basis (16 vectors on average) read for the dots and the update
    step = apply_bytes + 2 * 16 * n * t
    flops = 2 * nnz + 8 * 16 * n
    if do == "solve":
        return {"bytes": step * STEPS * case["alphas"], "flops": flops * STEPS * case["alphas"]}
    return {"bytes": step * STEPS, "flops": flops * STEPS}
