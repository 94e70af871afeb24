"""The p = inf forward of a handful of input rows against the tiled and generic kernels: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2, 3, 5, 8, 9, 16])
@pytest.mark.parametrize("CI,CO,G", [(784, 1024, 1), (1027, 333, 1), (64, 32, 1), (258, 130, 2), (4096, 4100, 1)])
def test_same_bits(cuda, lib, B, CI, CO, G):
    torch.manual_seed(B)
    x = (torch.randn(B, CI, 1, device="cuda") * 8).round() / 8          # ties
    w = (torch.randn(CO, CI // G, device="cuda") * 8).round() / 8
    x[0, 1] = float("nan")
    w[3] = x[B - 1, : CI // G, 0]                                       # a row of zero distance
    sub, add = torch.randn(CO, device="cuda"), torch.randn(CO, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    got = []
    try:
        for never in (0, 1):
            lib.linf_tune_set(8, never)
            y, z = (torch.empty(B, CO, 1, device="cuda") for _ in range(2))
            pos = torch.empty(B, CO, 1, dtype=torch.int32, device="cuda")
            assert lib.linf_inf_dist_forward(x.data_ptr(), w.data_ptr(), B, CO, CI, G, 1, y.data_ptr(), pos.data_ptr(), s) == 0
            assert lib.linf_inf_dist_forward_post(x.data_ptr(), w.data_ptr(), B, CO, CI, G, 1, sub.data_ptr(), add.data_ptr(), 1, z.data_ptr(), None, 0, s) == 0
            got.append((y, pos, z))
    finally:
        lib.linf_tune_set(8, 0)
    for a, b in zip(*got):
        assert torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))


@pytest.mark.parametrize("B,CI,CO", [(8, 20000, 800), (8, 20004, 1024), (2, 125004, 264), (3, 53400, 304), (16, 165000, 33)])
def test_same_bits_at_long_rows(cuda, lib, B, CI, CO):
    """Either side of the line above which the tiled kernel takes long rows."""
    test_same_bits(cuda, lib, B, CI, CO, 1)
