"""Teams of one CTA: the update of a Lanczos step with one thread a position and with positions shared by
lanes, around the size where the rule changes (64 16-byte positions for 128 threads), against the dense FP64
eigenvalues."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import specann_oracle as O  # noqa: E402
from specann_b200 import graphs  # noqa: E402
from specann_b200.batch import BatchedSpectralAnnealing  # noqa: E402


# 256 and 257 entries (FP32), 128 and 129 (FP64): the largest that lanes share and the smallest that they do not;
# 515 and 1030: more positions than threads, no multiple of a position
@pytest.mark.parametrize("precision,sizes", [(32, (255, 256, 257, 515, 1030)), (64, (127, 128, 129, 515, 1030))])
def test_update_on_either_side_of_the_rule(precision, sizes):
    Js = [graphs.barabasi_albert(n, 6, seed=n, couplings="pm1") for n in sizes]
    b = BatchedSpectralAnnealing(seeds=range(1, 151), num_alphas=3, schedule="linear", precision=precision)
    b.load(Js)
    b.sweep()
    res = b.results()
    assert len(res) == 150 * len(sizes)
    exact = []
    for J in Js:
        deg = np.asarray(abs(J).sum(axis=1)).ravel()
        exact.append([np.linalg.eigvalsh(O.scaled_operator_f64(J, deg, deg.max(), r["alpha"])[0].toarray())[-1]
                      for r in res[0]["rows"]])
    for p, r in enumerate(res):
        assert r["team"][1] == 1
        lam = np.array([row["lambda1"] for row in r["rows"]])
        # residuals of 1e-6 leave eigenvalues far closer; FP32 adds the operator's rounding
        assert np.max(np.abs(lam - exact[p // 150])) <= (2e-6 if precision == 32 else 1e-9)
    b.close()
