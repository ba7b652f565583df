"""Matrix memories in chunks of 128 tokens (33 to 128 rows a head): what chunks of 64 are asked for, at the edges of the longer ones.  The bounds
are those of the tests they are called from."""
import pytest

from tests import test_linear_chunks_gpu as chunks

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def wide(monkeypatch):
    from tensorline_b200 import ops
    monkeypatch.setattr(ops, "WIDE_CHUNKS_BLOCKS", {False: 0, True: 0})
    monkeypatch.setattr(ops, "WIDE_CHUNKS_SHARE", 1.0)
    yield
    ops.check_device_status()


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("H,d,dv,lens,rot,interleaved", [
    (3, 128, 256, [128, 129, 1], 64, False), (2, 64, 64, [300], 64, True), (1, 36, 128, [127, 63, 256], 0, False), (1, 96, 20, [400, 32], 96, False),
    (2, 68, 388, [160, 257], 8, True), (2, 52, 132, [33, 96], 0, False), (40, 128, 512, [513], 0, False)])
def test_wide_chunks_against_the_recurrence_in_float64_and_the_scan_kernel(gated, H, d, dv, lens, rot, interleaved):
    chunks.test_chunks_against_the_recurrence_in_float64_and_the_scan_kernel(gated, H, d, dv, lens, rot, interleaved)


@pytest.mark.parametrize("seed", [0, 1])
@pytest.mark.parametrize("gated,H,d,dv,T", [(True, 8, 128, 256, 300), (True, 16, 64, 128, 200), (False, 4, 128, 128, 130), (False, 8, 96, 64, 300),
                                            (True, 8, 128, 256, 1000)])
def test_errors_are_no_larger_than_token_by_token(gated, H, d, dv, T, seed):
    chunks.test_errors_are_no_larger_than_token_by_token(gated, H, d, dv, T, seed)


@pytest.mark.parametrize("what,value", [("v", float("nan")), ("k", -float("inf")), ("k", 1e30), ("q", float("nan"))])
@pytest.mark.parametrize("gated,d,dv", [(True, 64, 64), (False, 128, 132), (True, 128, 256)])
def test_a_value_that_is_no_number_reaches_what_it_reaches_token_by_token(what, value, gated, d, dv):
    chunks.test_a_value_that_is_no_number_reaches_what_it_reaches_token_by_token(what, value, gated, d, dv)
