"""The barrier between the phases of the persistent kernels, by itself: no CTA leaves it early over many
barriers and solves, and a wait that nothing ends runs out in every CTA and leaves the context usable."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from specann_b200 import _lib  # noqa: E402


def meet(blocks, expected, solves=1, meets=1, first_epoch=0, spin_limit=1 << 20):
    scratch = torch.zeros(32 + 4 * 1024, dtype=torch.uint8, device="cuda")
    st, passed, early = C.c_int32(-1), C.c_int32(-1), C.c_int32(-1)
    rc = _lib.load().sa_meet_selftest(blocks, expected, solves, meets, first_epoch, spin_limit,
                                      C.c_void_p(scratch.data_ptr()), scratch.numel(), C.byref(st), C.byref(passed),
                                      C.byref(early), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return rc, st.value, passed.value, early.value


@pytest.mark.parametrize("blocks", [1, 2, 3, 7, 148])
def test_no_cta_leaves_early(blocks):
    blocks = min(blocks, torch.cuda.get_device_properties(0).multi_processor_count)
    assert meet(blocks, blocks, solves=20, meets=37) == (_lib.SA_OK, _lib.SA_OK, blocks, 0)


@pytest.mark.parametrize("blocks", [2, 3, 7, 100])
def test_counter_past_its_end(blocks):
    # a counter wraps after 2^32 arrivals, between two barriers of a solve or in the midst of one's, and the
    # solves after it are counted anew
    for before in (0, 1, 18):
        first = ((1 << 32) // blocks - before) & 0xffffffff
        assert meet(blocks, blocks, solves=6, meets=5, first_epoch=first) == (_lib.SA_OK, _lib.SA_OK, blocks, 0)


@pytest.mark.parametrize("blocks", [2, 8, 148])
@pytest.mark.parametrize("spin_limit", [1, 64, 4096, 20000])
def test_wait_runs_out_in_every_cta(blocks, spin_limit):
    blocks = min(blocks, torch.cuda.get_device_properties(0).multi_processor_count)
    assert meet(blocks, blocks + 1, spin_limit=spin_limit) == (_lib.SA_OK, _lib.SA_ERR_BARRIER_TIMEOUT, 0, 0)
    assert meet(blocks, blocks, solves=3, meets=5) == (_lib.SA_OK, _lib.SA_OK, blocks, 0)


def test_unbounded_or_oversized_requests_are_refused():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for bad in (dict(blocks=sms + 1, expected=sms + 1), dict(blocks=0, expected=1), dict(blocks=4, expected=3),
                dict(blocks=4, expected=4, spin_limit=0), dict(blocks=4, expected=4, spin_limit=(1 << 25) + 1),
                dict(blocks=4, expected=4, meets=0), dict(blocks=4, expected=4, solves=1001)):
        assert meet(**bad)[0] == _lib.SA_ERR_INVALID_ARG
