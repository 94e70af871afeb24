"""Convolution-shaped distance layers: the unfold and fold kernels against torch's (the same values), and the weight gradient of few
rows with many sources against the oracle's order of additions (the same bits)."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C,H,W,k,dil,pad,stride", [(3, 8, 16, 16, 3, 1, 1, 1), (2, 5, 7, 9, 3, 2, 0, 1), (4, 4, 11, 6, 2, 1, 3, 2),
                                                      (1, 300, 5, 5, 5, 1, 2, 3), (2, 4, 6, 6, 1, 1, 0, 2)])
def test_unfold_and_fold(cuda, lib, B, C, H, W, k, dil, pad, stride):
    from linfdist_b200.norm_dist import PatchRowsF
    torch.manual_seed(0)
    x = torch.randn(B, C, H, W, device="cuda", requires_grad=True)
    cols = F.unfold(x, k, dil, pad, stride)
    rows = PatchRowsF.apply(x, k, dil, pad, stride, cols.size(2))
    assert torch.equal(rows.view(B, cols.size(2), -1).permute(0, 2, 1), cols)
    g = torch.randn_like(cols)
    want, = torch.autograd.grad(cols, x, g)
    got, = torch.autograd.grad(rows, x, g.permute(0, 2, 1).reshape(rows.shape))
    # at most k * k numbers are added: k * k roundings of 2^-24 of their sum of magnitudes
    assert (got - want).abs().max() <= k * k * 2.0 ** -23 * max(1.0, float(g.abs().max())) * k * k


@pytest.mark.parametrize("R,CI,CO,G", [(1024, 64, 40, 1), (5000, 36, 7, 1), (4097, 576, 130, 2), (8192, 9, 33, 1)])
def test_weight_gradient_of_few_rows(cuda, lib, R, CI, CO, G):
    import oracle
    gen = torch.Generator().manual_seed(R)
    g = torch.randn(R, CO, 1, generator=gen)
    g[torch.rand(R, CO, 1, generator=gen) < 0.3] = 0.0
    idx = (torch.rand(R, CO, 1, generator=gen) ** 3 * (CI // G)).int().clamp(max=CI // G - 1)      # some bins far fuller than others
    pos = torch.where(torch.rand(R, CO, 1, generator=gen) < 0.5, idx, idx | -2147483648).int()
    _, want = oracle.inf_dist_backward(g.numpy(), pos.numpy(), CI, G)
    gd, pd, gw = g.cuda(), pos.cuda(), torch.empty(CO, CI // G, device="cuda")
    assert lib.linf_inf_dist_backward_weight(gd.data_ptr(), pd.data_ptr(), R, CO, CI, G, 1, gw.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert np.array_equal(gw.cpu().numpy(), want)


@pytest.mark.parametrize("above", [0, 1])
def test_weight_gradient_at_the_most_rows_of_the_bins_kernel(cuda, lib, above):
    test_weight_gradient_of_few_rows(cuda, lib, 1100, 52, torch.cuda.get_device_properties(0).multi_processor_count + above, 1)


@pytest.mark.parametrize("p", [float("inf"), 8.0, 23.7])
@pytest.mark.parametrize("form", ["contiguous", "channels_last", "sliced"])
@pytest.mark.parametrize("group,stride,padding,dilation", [(1, 1, 1, 1), (2, 2, 0, 2)])
def test_module_on_patch_rows(cuda, lib, p, form, group, stride, padding, dilation):
    """Value and gradients of a NormDistConv against torch's unfold and one dense call per image, whatever the image's strides."""
    import linfdist_b200 as L
    torch.manual_seed(5)
    layer = L.NormDistConv(16, 64, 3, stride=stride, padding=padding, dilation=dilation, group=group, p=p, bias=True).cuda()
    x = torch.randn(6, 16, 13, 14, device="cuda")
    if form == "channels_last":
        x = x.contiguous(memory_format=torch.channels_last)
    if form == "sliced":
        x = torch.randn(6, 20, 13, 20, device="cuda")[:, 2:18, :, 3:17]
    x.requires_grad_()
    y = layer(x)[0]
    g = torch.randn_like(y)
    got = torch.autograd.grad(y, [x, layer.weight, layer.bias], g)
    cols = F.unfold(x, 3, dilation, padding, stride)                     # [B, C * 9, L]
    per_image = [L.norm_dist(c.t().unsqueeze(-1).contiguous(), layer.weight.view(64, -1), group, p) for c in cols]
    want_y = torch.stack([v[:, :, 0].t() for v in per_image]).view_as(y) + layer.bias.view(1, -1, 1, 1)
    want = torch.autograd.grad(want_y, [x, layer.weight, layer.bias], g)
    limit = 1e-6 if p == float("inf") else 2.0 ** -20 + p * 2.0 ** -22       # rounding of the terms, twice that of a call against 64 bits
    assert torch.linalg.norm(y - want_y) <= limit * torch.linalg.norm(want_y)
    for a, b in zip(got, want):
        assert torch.linalg.norm(a - b) <= max(limit, 1e-5) * torch.linalg.norm(b)
