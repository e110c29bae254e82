"""The alpha solve at the edges of its paths: one cluster of 8 or 16 CTAs and the whole grid (by the
tiles of the work list), vector phases in registers and streamed (by n), sizes that are no multiple of
a 16-byte position, the column panels at small n, and basis and restart sizes other than the default.
Each against SciPy's FP64 eigensolver on the exact operator, with a rounding that is bit-exact given
the vector."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import specann_oracle as O  # noqa: E402
from specann_b200 import _lib, graphs  # noqa: E402
from specann_b200.engine import Engine  # noqa: E402


def check(J, precision, alpha, ncv=33, keep=0, layout="worklist", tol=1e-6):
    J = sp.csr_matrix(J)
    n = J.shape[0]
    eng = Engine(n, J.nnz, precision=precision, ncv_max=ncv, max_candidates=2)
    eng.upload_csr(J.indptr, J.indices, J.data.astype(np.float32 if precision == 32 else np.float64))
    if layout == "panel":
        eng.build_panels()
    rec = eng.alpha_solve(alpha=alpha, alpha_prev=alpha, rho=1.001, gershgorin=1.0, tol=tol, pred_tol=1e-3,
                          maxiter=4000, ncv=ncv, start_mode=_lib.SA_START_RANDOM, seed=7, stream_id=0, align=False,
                          restart_keep=keep)
    assert rec.status == _lib.SA_OK, rec.status
    deg = np.asarray(abs(J).sum(axis=1)).ravel()
    M, _ = O.scaled_operator_f64(J, deg, deg.max(), alpha)
    y = eng.result_vector().double().cpu().numpy()
    lam = 1.001 - rec.mu
    # the solver stops at a residual estimate of tol; the FP32 operator adds its rounding
    assert np.linalg.norm(M @ y - lam * y) <= (1e-5 if precision == 32 else 2 * tol)
    ref = spla.eigsh(spla.aslinearoperator(M), k=1, which="LA", v0=y, tol=1e-10, return_eigenvectors=False)[0]
    assert abs(lam - ref) <= (1e-6 if precision == 32 else 1e-8)
    eng.keep_candidate(0)
    assert np.array_equal(eng.candidate_spins(0).cpu().numpy(), np.where(y >= 0, 1, -1).astype(np.int8))
    again = eng.alpha_solve(alpha=alpha, alpha_prev=alpha, rho=1.001, gershgorin=1.0, tol=tol, pred_tol=1e-3,
                            maxiter=4000, ncv=ncv, start_mode=_lib.SA_START_RANDOM, seed=7, stream_id=0, align=False,
                            restart_keep=keep)
    assert again.mu == rec.mu and again.iterations == rec.iterations   # no dependence on timing
    assert torch.equal(eng.result_vector().double().cpu(), torch.from_numpy(y))
    eng.close()


@pytest.mark.parametrize("precision", [32, 64])
# 37: under a warp of positions; 1283 / 1290: about 128 tiles (8 or 16 CTAs); 2559 / 2566: about 256 (16 or the grid)
@pytest.mark.parametrize("n", [37, 130, 1283, 1290, 2559, 2566])
def test_cluster_and_grid_edges(n, precision):
    check(graphs.barabasi_albert(n, 10, seed=n), precision, 0.5)


@pytest.mark.parametrize("precision,n", [(32, 151549), (32, 151557), (64, 75775), (64, 75779)])
def test_register_and_streamed_vector_phases(precision, n):
    check(graphs.barabasi_albert(n, 4, seed=5), precision, 0.4)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [591, 4099])
def test_streamed_phases_on_few_rows_per_cta(n, precision):
    check(graphs.barabasi_albert(n, 20, seed=3), precision, 0.5, layout="panel")


@pytest.mark.parametrize("ncv,keep", [(4, 0), (9, 3), (33, 16), (64, 8)])
def test_basis_and_restart_sizes(ncv, keep):
    # a leading gap small enough to restart several times
    check(graphs.erdos_renyi(3000, 20 / 2999, seed=11), 64, 0.9, ncv=ncv, keep=keep, tol=1e-7)


@pytest.mark.parametrize("n,m,precision,pays", [(65535, 20, 64, False), (65536, 20, 64, True), (65536, 10, 64, False),
                                                (65536, 10, 32, True)])
def test_panel_rule(n, m, precision, pays, monkeypatch):
    J = graphs.barabasi_albert(n, m, seed=2)
    eng = Engine(n, J.nnz, precision=precision, ncv_max=4, max_candidates=1)
    eng.upload_csr(J.indptr, J.indices, J.data.astype(np.float32 if precision == 32 else np.float64))
    assert eng.panels_pay() == pays
    # FP64: a layout of more than half of the free memory is left out
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (2 * eng.panel_plan()[0] - 1, 1 << 37))
    assert eng.panels_pay() == (pays and precision == 32)
    eng.close()


@pytest.mark.parametrize("layout", ["worklist", "panel"])
@pytest.mark.parametrize("precision", [32, 64])
def test_operator_calls_in_a_row_and_captured(layout, precision):
    # each call's scaling writes the buffers that the call before still reads: nothing may overlap there
    J = graphs.barabasi_albert(70003, 20, seed=6, couplings="pm1")
    n, dt = J.shape[0], torch.float32 if precision == 32 else torch.float64
    eng = Engine(n, J.nnz, precision=precision, ncv_max=4, max_candidates=1, stream=torch.cuda.Stream())
    eng.upload_csr(J.indptr, J.indices, J.data.astype(np.float32 if precision == 32 else np.float64))
    if layout == "panel":
        eng.build_panels()
    g = torch.Generator(device="cuda").manual_seed(3)
    X = torch.randn(12, n, device="cuda", generator=g, dtype=dt)
    alphas = np.linspace(0.0, 1.0, 12)
    torch.cuda.synchronize()
    alone = torch.empty_like(X)
    for q in range(12):
        eng.spmv(alphas[q], 1.001, X[q], alone[q])
        torch.cuda.synchronize()
    row = torch.zeros_like(X)
    torch.cuda.synchronize()
    for q in range(12):
        eng.spmv(alphas[q], 1.001, X[q], row[q])
    torch.cuda.synchronize()
    assert torch.equal(row, alone)
    captured = torch.zeros_like(X)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=eng.stream):
        for q in range(12):
            eng.spmv(alphas[q], 1.001, X[q], captured[q])
    for _ in range(2):
        captured.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, alone)
    assert eng.operator_status() == 0
    eng.close()


def test_work_list_spmv_keeps_its_l1():
    # the vector phases' shared memory comes out of the L1 that the gathers need: a step's SpMV against the
    # standalone operator on the same work list (1.3 times as long; 1.9 times with only 28 KB of L1)
    J = graphs.barabasi_albert(1 << 20, 4, seed=42, dtype=np.float32)
    eng = Engine(J.shape[0], J.nnz, precision=32, ncv_max=33, max_candidates=1)
    eng.upload_csr(J.indptr, J.indices, J.data)

    def step():
        rec = eng.alpha_solve(alpha=0.6, alpha_prev=0.6, rho=1.001, gershgorin=1.0, tol=1e-30, pred_tol=1e-3, maxiter=30,
                              ncv=33, start_mode=_lib.SA_START_RANDOM, seed=7, stream_id=0, align=False)
        return rec.phase_ms[1] / rec.iterations

    x = torch.randn(J.shape[0], device="cuda")
    y = torch.empty_like(x)

    def operator(reps=10):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            eng.spmv(0.6, 1.001, x, y)
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / reps

    step(), operator()
    assert min(step() for _ in range(5)) < 1.6 * min(operator() for _ in range(5))
    eng.close()
