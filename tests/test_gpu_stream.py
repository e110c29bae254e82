"""The streamed vector phases by themselves: both against NumPy in FP64, with one to three groups of tiles in
flight, at sizes around a 16-byte position, a thread's share of a tile and whole tiles; and a wait for a
copy that is made to run out."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from specann_b200 import _lib  # noqa: E402


def run(precision, buffers, blocks, n, j, withhold=False, spin_limit=1 << 22):
    dt, wide = (torch.float32, 4) if precision == 32 else (torch.float64, 2)
    ldv = (n + wide - 1) // wide * wide
    rng = np.random.default_rng(1000 * n + j)
    host = rng.standard_normal((j + 4, ldv)).astype(np.float32 if precision == 32 else np.float64)
    host[:, n:] = 0.0
    X = torch.from_numpy(host).cuda()
    h = torch.from_numpy(rng.standard_normal(j + 1)).cuda()
    dots = torch.zeros(blocks, j + 2, dtype=torch.float64, device="cuda")
    words = torch.zeros(1 + blocks, dtype=torch.int32, device="cuda")
    w, u, sigma, a3, b3 = X[j + 1].clone(), torch.full((ldv,), 9.0, dtype=dt, device="cuda"), X[j + 3].clone(), 0.75, -0.5
    p = _lib.StreamTest(precision=precision, buffers=buffers, blocks=blocks, j=j, n=n, ldv=ldv,
                        V=X.data_ptr(), w=w.data_ptr(), u=u.data_ptr(), sigma=sigma.data_ptr(), h=h.data_ptr(),
                        dots=dots.data_ptr(), a3=a3, b3=b3, spin_limit=spin_limit, withhold=int(withhold))
    st, passed = C.c_int32(-1), C.c_int32(-1)
    torch.cuda.synchronize()
    rc = _lib.load().sa_stream_selftest(C.byref(p), C.c_void_p(words.data_ptr()), C.byref(st), C.byref(passed),
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == _lib.SA_OK
    V, w0, sg, hh = (t.double().cpu().numpy() for t in (X[: j + 1], X[j + 1], X[j + 3], h))
    eps = 2.0 ** (-24 if precision == 32 else -53)
    u0 = w0 - a3 * V[j] - (b3 * V[j - 1] if j > 0 else 0.0)
    return st.value, passed.value, dots.sum(0).cpu().numpy(), w.double().cpu().numpy(), u.double().cpu().numpy(), V, u0, sg, hh, eps


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("buffers", [1, 2, 3])
# one CTA: a position, a thread's share of a tile, tiles of 4096 (FP32) or 2048 (FP64) rows, several of them
# with a ragged last one; the vectors of one group, of several, and a last group of one vector
@pytest.mark.parametrize("blocks,n,j", [(1, 1, 0), (1, 5, 3), (1, 2049, 1), (1, 4097, 2), (1, 12301, 4), (1, 30001, 33),
                                        (3, 2, 7), (3, 40003, 9), (7, 100003, 62)])
def test_phases_match_numpy(precision, buffers, blocks, n, j):
    st, passed, dots, w, u, V, u0, sg, h, eps = run(precision, buffers, blocks, n, j)
    assert st == _lib.SA_OK and passed == blocks
    # rounded to the working precision: u0, w and u; the sums are in FP64
    ref, absolute = np.append(V @ u0, u0 @ u0), np.append(np.abs(V) @ np.abs(u0), u0 @ u0)
    assert np.all(np.abs(dots - ref) <= (4 * eps + 1e-12) * absolute)
    w_ref = u0 - h @ V
    err = 2 * eps * (np.abs(u0) + np.abs(w_ref)) + 1e-13 * (np.abs(u0) + np.abs(h) @ np.abs(V))
    assert np.all(np.abs(w - w_ref) <= err)
    assert np.all(np.abs(u - sg * w_ref) <= np.abs(sg) * (err + 2 * eps * np.abs(w_ref)))


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("buffers", [1, 3])
def test_wait_for_a_copy_runs_out(precision, buffers):
    st, passed, *_ = run(precision, buffers, 4, 50001, 6, withhold=True, spin_limit=64)
    assert st == _lib.SA_ERR_BARRIER_TIMEOUT and passed == 0
    # the context is still usable
    st, passed, *_ = run(precision, buffers, 4, 50001, 6)
    assert st == _lib.SA_OK and passed == 4
