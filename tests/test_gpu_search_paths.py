"""The batched local search at the edges of its passes: candidate counts around the word and tile widths,
rows around the length from which a whole CTA checks them, both pass semantics; spins, energies and
pass counts exact against the oracle."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import specann_oracle as O  # noqa: E402
from specann_b200 import _lib, graphs  # noqa: E402
from specann_b200.engine import Engine  # noqa: E402


def with_hubs(n, degrees, seed):
    """A +-1 Barabasi-Albert graph whose first nodes are joined to more nodes, up to the given degrees."""
    J = graphs.barabasi_albert(n, 6, seed=seed, couplings="pm1").tolil()
    rng = np.random.default_rng(seed)
    for hub, deg in enumerate(degrees):
        have = set(J.rows[hub]) | {hub}
        free = np.array([v for v in range(n) if v not in have])
        for v in rng.permutation(free)[: max(0, deg - len(J.rows[hub]))]:
            J[hub, v] = J[v, hub] = float(rng.choice([-1, 1]))
    return sp.csr_matrix(J)


@pytest.fixture(scope="module")
def hubs():
    # 512 / 513: the longest row of a warp and the shortest of a CTA; 1400: several chunks
    return with_hubs(1501, (512, 513, 1400), seed=4)


@pytest.mark.parametrize("semantics", ["priority", "snapshot"])
@pytest.mark.parametrize("k", [1, 8, 9, 16, 17, 33, 70, 128])
def test_search_matches_oracle(hubs, k, semantics):
    n = hubs.shape[0]
    S = np.where(np.random.default_rng(k).random((k, n)) < 0.5, 1, -1).astype(np.int8)
    eng = Engine(n, hubs.nnz, precision=32, ncv_max=4, max_candidates=k)
    eng.upload_csr(hubs.indptr, hubs.indices, hubs.data.astype(np.float32))
    for c in range(k):
        eng.set_candidate(c, S[c])
    iters, rounds = (1000, 25) if semantics == "priority" else (12, 3)   # snapshot passes may oscillate
    eb, ea, res = eng.local_search(k, max_iterations=iters, num_rounds=rounds, seed=5, semantics=semantics)
    ref = O.local_search(hubs, S, seed=5, max_iterations=iters, num_rounds=rounds, semantics=semantics)
    got = np.stack([eng.candidate_spins(c, refined=True).cpu().numpy() for c in range(k)])
    assert np.array_equal(got, ref.spins)
    assert np.array_equal(ea, np.asarray(ref.energies_after, dtype=np.float64))
    assert res.iterations == ref.iterations
    eng.close()


# nodes that a pass leaves out keep their changes for a later one: small subsets, and a final sweep over
# a part of the nodes
@pytest.mark.parametrize("k, sub, final", [(3, 0.3, 1.0), (40, 0.3, 0.6), (70, 0.05, 0.5), (128, 0.6, 0.9)])
def test_search_with_small_subsets(hubs, k, sub, final):
    n = hubs.shape[0]
    S = np.where(np.random.default_rng(k).random((k, n)) < 0.5, 1, -1).astype(np.int8)
    eng = Engine(n, hubs.nnz, precision=32, ncv_max=4, max_candidates=k)
    eng.upload_csr(hubs.indptr, hubs.indices, hubs.data.astype(np.float32))
    for c in range(k):
        eng.set_candidate(c, S[c])
    kw = dict(seed=9, max_iterations=60, subset_fraction=sub, final_sweep_fraction=final, num_rounds=4)
    eb, ea, res = eng.local_search(k, **kw)
    ref = O.local_search(hubs, S, **kw)
    got = np.stack([eng.candidate_spins(c, refined=True).cpu().numpy() for c in range(k)])
    assert np.array_equal(got, ref.spins)
    assert np.array_equal(ea, np.asarray(ref.energies_after, dtype=np.float64))
    assert res.iterations == ref.iterations
    eng.close()


# one CTA per SM and two (from 2^21 fields on)
@pytest.mark.parametrize("n", [16383, 16384])
def test_search_on_either_side_of_the_second_cta(n):
    J, k = graphs.barabasi_albert(n, 3, seed=8, couplings="pm1"), 128
    S = np.where(np.random.default_rng(n).random((k, n)) < 0.5, 1, -1).astype(np.int8)
    eng = Engine(n, J.nnz, precision=32, ncv_max=4, max_candidates=k)
    eng.upload_csr(J.indptr, J.indices, J.data.astype(np.float32))
    for c in range(k):
        eng.set_candidate(c, S[c])
    kw = dict(seed=2, max_iterations=4, num_rounds=1, final_sweep_iters=2)
    eb, ea, res = eng.local_search(k, **kw)
    ref = O.local_search(J, S, **kw)
    got = np.stack([eng.candidate_spins(c, refined=True).cpu().numpy() for c in range(k)])
    assert np.array_equal(got, ref.spins)
    assert np.array_equal(ea, np.asarray(ref.energies_after, dtype=np.float64))
    assert res.iterations == ref.iterations
    eng.close()


def test_flip_total_beyond_32_bits():
    # 2^25 antiferromagnetic pairs, all spins up in 32 candidates: a snapshot pass flips every spin of every
    # candidate, 2^31 in all
    n, k = 1 << 26, 32
    eng = Engine(n, n, precision=32, ncv_max=2, max_candidates=k)
    rowptr = torch.arange(n + 1, dtype=torch.int32, device="cuda")
    col = torch.arange(n, dtype=torch.int32, device="cuda") ^ 1
    eng.bind(rowptr, col, torch.full((n,), -1.0, device="cuda"))
    up = torch.full((n // 32,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for c in range(k):
        _lib.check("sa_candidate_set", eng.lib.sa_candidate_set(eng.h, c, up.data_ptr()))
    eb, ea, res = eng.local_search(k, max_iterations=1, subset_fraction=1.0, final_sweep_iters=0, semantics="snapshot")
    assert res.total_flips == n * k
    assert np.all(eb == n // 2) and np.all(ea == n // 2)
    eng.close()
