"""The alpha solve where its kernels differ: vector phases streamed over few rows a CTA (column splits at
small n), over several tiles a CTA with a ragged last one, and behind the column panels; and every start
vector, accepted and rejected, on one cluster and on the whole grid. Against SciPy's FP64 eigensolver on the
exact operator, and bit-equal when repeated."""
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


def engine(J, precision, layout):
    eng = Engine(J.shape[0], J.nnz, precision=precision, ncv_max=33, max_candidates=2)
    eng.upload_csr(J.indptr, J.indices, J.data.astype(np.float32 if precision == 32 else np.float64))
    if layout == "panel":
        eng.build_panels()
    elif layout == "split":
        eng.build_splits(3)
    return eng


def solve(eng, alpha, **kw):
    args = dict(alpha=alpha, alpha_prev=alpha, rho=1.001, gershgorin=1.0, tol=1e-6, pred_tol=1e-3, maxiter=4000, ncv=33,
                start_mode=_lib.SA_START_RANDOM, seed=7, stream_id=0, align=False)
    args.update(kw)
    rec = eng.alpha_solve(**args)
    assert rec.status == _lib.SA_OK, rec.status
    return rec, eng.result_vector().double().cpu().numpy()


def check(J, precision, alpha, rec, y):
    J = sp.csr_matrix(J)
    deg = np.asarray(abs(J).sum(axis=1)).ravel()
    M, _ = O.scaled_operator_f64(J, deg, deg.max(), alpha)
    lam = 1.001 - rec.mu
    # the solver stops at a residual estimate of 1e-6; the FP32 operator adds its rounding
    assert np.linalg.norm(M @ y - lam * y) <= (1e-5 if precision == 32 else 2e-6)
    ref = spla.eigsh(spla.aslinearoperator(M), k=1, which="LA", v0=y, tol=1e-9, return_eigenvectors=False)[0]
    assert abs(lam - ref) <= (1e-6 if precision == 32 else 1e-8)


# few rows a CTA; one tile and several of 4096 (FP32) or 2048 (FP64) rows, none a multiple of a position
@pytest.mark.parametrize("precision,n,m,layout", [
    (32, 591, 20, "split"), (64, 591, 20, "split"), (32, 4099, 20, "split"), (64, 4099, 20, "split"),
    (32, 151557, 8, "panel"), (64, 75779, 8, "panel"), (32, 620003, 4, "panel"), (64, 310001, 4, "panel"),
    (32, 620003, 4, "worklist"), (64, 310001, 4, "worklist"), (32, 1250007, 3, "split")])
def test_streamed_vector_phases(precision, n, m, layout):
    J = graphs.barabasi_albert(n, m, seed=5)
    eng = engine(J, precision, layout)
    rec, y = solve(eng, 0.4)
    check(J, precision, 0.4, rec, y)
    again, y2 = solve(eng, 0.4)
    assert (again.mu, again.iterations) == (rec.mu, rec.iterations) and np.array_equal(y, y2)
    eng.close()


@pytest.mark.parametrize("precision", [32, 64])
# clusters of 8 and 16 CTAs, the whole grid, the panels
@pytest.mark.parametrize("n,m,layout", [(1283, 10, "worklist"), (2500, 10, "worklist"), (5001, 10, "worklist"),
                                        (5001, 20, "panel")])
@pytest.mark.parametrize("start", ["prev", "diagonal", "secant", "tangent", "given"])
@pytest.mark.parametrize("rejected", [False, True])
def test_start_vectors(n, m, layout, precision, start, rejected):
    J = graphs.barabasi_albert(n, m, seed=9)
    eng = engine(J, precision, layout)
    ys = []
    for a in (0.48, 0.5):
        rec, y = solve(eng, a, align=bool(ys))
        eng.commit()
        ys.append(y)
    v0 = None
    if start == "tangent":
        v0 = torch.from_numpy((ys[1] - ys[0]) / 0.02).to("cuda", eng.vdtype)
    elif start == "given":
        v0 = torch.from_numpy(ys[1] + 1e-3 * np.random.default_rng(0).standard_normal(n)).to("cuda", eng.vdtype)
    mode = {"prev": _lib.SA_START_PREV, "diagonal": _lib.SA_START_DIAGONAL, "secant": _lib.SA_START_SECANT,
            "tangent": _lib.SA_START_TANGENT, "given": _lib.SA_START_GIVEN}[start]
    kw = dict(alpha_prev=0.5, start_mode=mode, v0=v0, align=True, pred_tol=1e-12 if rejected else 1.0)
    rec, y = solve(eng, 0.52, **kw)
    predicted = start in ("diagonal", "secant", "tangent")
    assert rec.pred_accepted == ((0 if rejected else 1) if predicted else -1)
    check(J, precision, 0.52, rec, y)
    assert y @ ys[1] > 0.0
    again, y2 = solve(eng, 0.52, **kw)
    assert (again.mu, again.iterations, again.pred_residual) == (rec.mu, rec.iterations, rec.pred_residual) or (
        not predicted and (again.mu, again.iterations) == (rec.mu, rec.iterations))
    assert np.array_equal(y, y2)
    eng.close()
