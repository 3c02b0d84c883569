"""A kernel that gives up a bounded wait leaves a result that is not valid: the next call on its stream says so.  The wait is
one that nothing satisfies, on its own and with a limit of a millisecond; nothing faults."""
import numpy as np
import pytest
import torch

from oracle import fp8_oracle as O
from helpers import kernels, run_linear, upload_case

pytestmark = pytest.mark.gpu


def give_up(pkg, ws):
    L = pkg._lib
    L.raise_for(L.load().fp8lin_debug_wait_timeout(ws.data_ptr(), 1000, torch.cuda.current_stream().cuda_stream), "probe")
    torch.cuda.synchronize()


@pytest.mark.parametrize("inference", [False, True])
def test_the_next_call_raises_and_the_one_after_is_clean(pkg, inference):
    Kn, dev = kernels(), torch.device("cuda", 0)
    d = upload_case(O.make_case(3, 130, 448, 576))
    with torch.inference_mode(inference):
        want = run_linear("fp8_w8a8_static", d)
        give_up(pkg, Kn.workspace(dev, pkg._lib.WS_HEADER_BYTES))
        other = torch.cuda.Stream()
        with torch.cuda.stream(other):                              # another stream's scratch has nothing to report
            np.testing.assert_array_equal(run_linear("fp8_w8a8_static", d), want)
    with pytest.raises(RuntimeError, match="gave up a bounded wait .device status 0x101."):
        run_linear("fp8_w8a8_static", d)
    np.testing.assert_array_equal(run_linear("fp8_w8a8_static", d), want)
    assert Kn.read_status(dev) == 0


def test_scratch_that_grows_keeps_reporting(pkg):
    Kn, dev = kernels(), torch.device("cuda", 0)
    with torch.cuda.stream(torch.cuda.Stream()):
        small = Kn.workspace(dev, pkg._lib.WS_HEADER_BYTES)
        large = Kn.workspace(dev, 4 * small.numel())
        assert large.data_ptr() != small.data_ptr()
        for ws in (small, large):                                   # (a CUDA graph may still use the outgrown buffer)
            give_up(pkg, ws)
            with pytest.raises(RuntimeError, match="gave up"):
                Kn.workspace(dev, pkg._lib.WS_HEADER_BYTES)
        assert Kn.read_status(dev) == 0
        give_up(pkg, large)
        with pytest.raises(RuntimeError, match="bounded wait"):      # a blocking read reports it once, and for all
            Kn.read_status(dev)
        Kn.workspace(dev, pkg._lib.WS_HEADER_BYTES)
