"""The automatic choice of the operator layout: a function of the problem and the device, whatever else is in
memory; in FP64 the work list where the panels' values would have to be streamed for short rows, or where
there is no memory for them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from specann_b200 import graphs  # noqa: E402
from specann_b200.differentiation import EigenProblem  # noqa: E402
from specann_b200.engine import Engine  # noqa: E402
from specann_b200.spectral_annealing import SpectralAnnealing  # noqa: E402


def layouts(J, precision):
    p = EigenProblem(J, precision=precision)
    s = SpectralAnnealing("t", "t", random_seed=1, num_alphas=2, precision=precision, write_results=False)
    s.solve(J)
    out = p.operator_layout, s.operator_layout
    p.close()
    return out


# rows of about 2 m entries; 36 and 32 are the shortest of one magnitude on either side of n = 80000, 80 of several
@pytest.mark.parametrize("n,m,couplings,layout", [(65535, 20, "pm1", "worklist"), (65536, 20, "pm1", "panel"),
                                                  (65536, 19, "pm1", "panel"), (65536, 17, "pm1", "worklist"),
                                                  (80000, 17, "pm1", "panel"), (80000, 15, "pm1", "worklist"),
                                                  (65536, 20, "int100", "worklist"), (65536, 39, "int100", "worklist"),
                                                  (65536, 41, "int100", "panel")])
def test_fp64_rule(n, m, couplings, layout):
    J = graphs.barabasi_albert(n, m, seed=2, couplings=couplings)
    assert layouts(J, 64) == (layout, layout)


def test_layout_does_not_depend_on_free_memory(monkeypatch):
    J = graphs.barabasi_albert(65536, 20, seed=2, couplings="pm1")
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (1 << 20, 1 << 37))
    assert layouts(J, 64) == ("panel", "panel")


def test_work_list_where_the_panels_find_no_memory(monkeypatch):
    J = graphs.barabasi_albert(65536, 20, seed=2, couplings="pm1")

    def refuse(self):
        raise torch.cuda.OutOfMemoryError("no memory for the panels")

    monkeypatch.setattr(Engine, "build_panels", refuse)
    assert layouts(J, 64) == ("worklist", "worklist")
    with pytest.raises(torch.cuda.OutOfMemoryError):    # FP32 has always needed them
        layouts(J, 32)
