"""An index that a kernel reported and skipped does not stop the kernels behind it."""
import pytest
import torch

from pisceslx_b200.ops import KernelStatusError, check_status, functional as F_, moe as moe_ops, status_word

pytestmark = pytest.mark.gpu
DEV = "cuda"
INDEX_OUT_OF_RANGE = 8


@pytest.fixture
def reported():
    check_status(torch.device(DEV, torch.cuda.current_device()))
    word = status_word(torch.device(DEV, torch.cuda.current_device()))
    word[0] = INDEX_OUT_OF_RANGE
    yield word
    word.zero_()


def _rand(*shape):
    return torch.randn(*shape, device=DEV).bfloat16()


@pytest.mark.parametrize("rows,N,K", [(1, 256, 2048), (64, 4096, 1024), (128, 100, 64), (300, 512, 1024)])
def test_products_are_written(reported, rows, N, K):
    w = _rand(N, K)
    for _ in range(3):                           # each in memory that held another product
        x = _rand(rows, K)
        got, want = F_.linear(x, w), x.double() @ w.double().t()
        # one rounding to bf16
        assert (got.double() - want).norm() < 2.0 ** -8 * want.norm()
        del got
    assert int(reported[0]) == INDEX_OUT_OF_RANGE


def test_attention_and_experts_are_written(reported):
    q, k, v = (_rand(300, 4 * 64) for _ in range(3))
    cu = torch.tensor([0, 300], dtype=torch.int32, device=DEV)
    x, w13, w2 = _rand(40, 128), _rand(4, 256, 128) * 0.1, _rand(4, 128, 128) * 0.1
    idx = torch.rand(40, 4, device=DEV).topk(2, -1).indices.int()
    weights = torch.rand(40, 2, device=DEV)
    seen = []
    for bits in (INDEX_OUT_OF_RANGE, 0):
        reported[0] = bits
        with torch.no_grad():
            seen.append((F_.attention(q, k, v, cu, cu, 300, 300, 4, 4, 64, True), moe_ops.moe_experts(x, w13, w2, weights, idx)))
    assert all(torch.equal(a, b) for a, b in zip(*seen))


def test_the_report_still_reaches_the_host(reported):
    with pytest.raises(KernelStatusError):
        check_status(torch.device(DEV, torch.cuda.current_device()))
    check_status(torch.device(DEV, torch.cuda.current_device()))
