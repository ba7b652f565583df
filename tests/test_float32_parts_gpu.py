"""The 32-bit engine's product on the tensor cores (bfloat16 weights, large matrices) at the edges of its tiles, segments and groups: a
row's floats do not depend on the rows beside it, and the formula in float64.  Bound of an output's error: its sums round at most once
a chunk of 64 k, a segment and a group, and a chunk is cut off at most at each of its twelve instructions, each time by less than
2^-22 of the sum of absolute products."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from tensorline_b200 import ops
    return ops


def product(ops, a, w, bias=None):
    out = torch.full((a.shape[0], w.shape[0]), 7.0, device="cuda")
    ops.gemm_f32(a, w, out, bias)
    return out


@pytest.mark.parametrize("N,K", [(2048, 1024), (257, 4104), (1029, 1088), (300, 8200), (4608, 3584), (200, 18944)])
def test_rows_of_every_tile_width_have_the_same_floats(ops, N, K):
    g = torch.Generator().manual_seed(N + K)
    top = 2100
    a = torch.randn(top, K, generator=g).cuda()
    w = torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
    bias = torch.randn(N, generator=g).to(torch.bfloat16).cuda()
    assert ops.core().tl_gemm_f32_parts_scratch(a.data_ptr(), K, w.data_ptr(), 1, N, K) > 0
    whole = product(ops, a, w, bias)                     # more rows than are taken at a time
    want, size = a.double() @ w.double().T + bias.double(), a.double().abs() @ w.double().abs().T + 1.0
    chunks = -(-K // 64)
    assert float(((whole.double() - want).abs() / size).max()) <= (chunks + chunks // 16 + 60) * 2.0 ** -24
    for n in (1, 2, 31, 33, 64, 65, 97, 128, 129, 177, 336, 353, 700):
        lo = (n * 37) % (top - n)
        assert torch.equal(product(ops, a[lo:lo + n], w, bias), whole[lo:lo + n]), n
    ops.check_device_status()


def test_rows_apart_and_odd_values(ops):
    g = torch.Generator().manual_seed(3)
    N, K = 700, 1600
    wide = torch.randn(40, K + 12, generator=g).cuda()
    a = wide[:, 4:4 + K]                                 # 16 bytes into its rows
    w = torch.randn(N, K, generator=g).clamp_(-0.9, 0.9).to(torch.bfloat16).cuda()
    assert torch.equal(product(ops, a, w), product(ops, a.contiguous(), w))
    odd = a.contiguous().clone()
    odd[1, 3] = 3.4028e38                                # would round up to an infinity in bfloat16
    odd[2] *= 2.0 ** -140                                # below the smallest normal number
    odd[3, 5] = float("inf")
    odd[4, 7] = float("nan")
    odd[5, 9] = torch.tensor(0x7f800001, dtype=torch.int32).view(torch.float32)      # a not-a-number whose high half is an infinity's
    got = product(ops, odd, w)
    keep = [0] + list(range(6, 40))
    assert torch.equal(got[keep], product(ops, a, w)[keep])
    want = odd.double() @ w.double().T
    assert torch.equal(torch.isinf(got[3]), torch.isinf(want[3])) and torch.equal(got[3].sign(), want[3].sign().float())
    assert bool(torch.isnan(got[4]).all()) and bool(torch.isnan(got[5]).all())
    assert float((got[2].double() - want[2]).abs().max()) <= K * 2.0 ** -132
    assert float(((got[1].double() - want[1]).abs() / want[1].abs().clamp_min(1.0)).max()) <= 2.0 ** -20
    ops.check_device_status()


def test_infinite_weights(ops):
    """An infinite weight meets parts of a float that are zero: still what a chain of multiply-adds gives, an infinity, or none where
    the value is zero or infinities of both signs meet.  With sums along K in one piece, in several, and in several kernels."""
    for M, N, K in ((5, 1029, 1088), (200, 1029, 8200), (1, 300, 18944)):
        g = torch.Generator().manual_seed(K)
        a = torch.randn(M, K, generator=g).cuda()
        a[:, 3], a[:, 7], a[0, 3] = 2.0, -0.37, 0.0      # in bfloat16 exactly, not so, zero
        w = torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
        w[1, 3], w[130, 7], w[257, 3], w[257, 7] = float("inf"), float("inf"), -float("inf"), -float("inf")
        assert ops.core().tl_gemm_f32_parts_scratch(a.data_ptr(), K, w.data_ptr(), M, N, K) > 0
        bias = torch.randn(N, generator=g).to(torch.bfloat16).cuda()
        got, want, clean = product(ops, a, w, bias), product(ops, a, w.float(), bias.float()), product(ops, a, w.nan_to_num(0.0, 0.0, 0.0), bias)
        rows = [1, 130, 257]
        assert int(want[1:, rows].isnan().sum()) == M - 1 and bool(want[1:, 1].isinf().all())
        assert torch.equal(got[:, rows].isnan(), want[:, rows].isnan())
        assert torch.equal(got[:, rows].nan_to_num(0.0), want[:, rows].nan_to_num(0.0))
        rest = [n for n in range(N) if n not in rows]
        assert torch.equal(got[:, rest], clean[:, rest])
    ops.check_device_status()


@pytest.mark.parametrize("M,N,K", [(2048, 152064, 5120), (2048, 37888, 18944), (700, 152064, 8192), (1, 152064, 18944), (2048, 3584, 18944)])
def test_the_scratch_has_a_bound(ops, M, N, K):
    """The parts of 2,048 rows, and sums along K in pieces only as far as they are small."""
    a = torch.zeros(256, device="cuda")
    blocks = ops.core().tl_gemm_f32_parts_scratch(a.data_ptr(), K, a.data_ptr(), M, N, K)
    assert 0 < blocks * 256 <= 6 * 2048 * K + 256 + (256 << 20)


@pytest.mark.parametrize("N,K", [(16640, 4104), (152064, 4104)])
def test_rows_in_slabs_have_the_same_floats(ops, N, K):
    """So many outputs that the sums along K of all rows would be more than the scratch may hold: 1,936 and 176 rows at a time."""
    g = torch.Generator().manual_seed(K)
    a, w = torch.randn(2048 if N < 20000 else 400, K, generator=g).cuda(), torch.randn(N, K, generator=g, dtype=torch.bfloat16).cuda()
    whole = product(ops, a, w)
    for lo, n in ((0, 33), (100, 128), (a.shape[0] - 148, 148)):
        assert torch.equal(product(ops, a[lo:lo + n], w), whole[lo:lo + n]), n
    ops.check_device_status()


@pytest.mark.parametrize("N,K", [(2048, 1024), (1029, 2040)])
def test_short_rows_of_weights_are_chains(ops, N, K):
    """One launch there, two or three here: a few rows were slower.  The floats of the widened weights' chains."""
    g = torch.Generator().manual_seed(K)
    a, w = torch.randn(40, K, generator=g).cuda(), torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
    for n in (1, 4, 40):
        assert torch.equal(product(ops, a[:n], w), product(ops, a[:n], w.float()))


@pytest.mark.parametrize("N,K", [(2048, 2048), (257, 4104), (300, 8200), (4608, 3584), (200, 18944)])
def test_errors_are_those_of_three_parts(ops, N, K):
    """In the norm: a chunk's cuts and the additions behind it come to less than 4e-7 of a sum of random signs (two parts only: 1e-5), and to
    no more than what chains of multiply-adds on the same values are off by.  For every width of the tiles."""
    g = torch.Generator().manual_seed(K)
    a, w = torch.randn(353, K, generator=g).cuda(), torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
    for n in (1, 32, 64, 96, 128, 176, 353):
        want = a[:n].double() @ w.double().T
        err, chains = (float((x.double() - want).norm() / want.norm()) for x in (product(ops, a[:n], w), product(ops, a[:n], w.float())))
        assert err <= 4e-7 and err <= chains, (n, err, chains)
    ops.check_device_status()
