"""Limits that decide on the host how a call is run: no GPU needed."""
from types import SimpleNamespace

import pytest
import torch


def own_bytes(B, CO, CI, G, inputs):
    return 4 * (inputs * B * CI + CO * CI // G + 2 * B * CO)


@pytest.mark.parametrize("B,CO,CI,G", [(512, 5120, 5120, 1), (131000, 72, 512, 1), (100000, 64, 256, 1), (16384, 128, 576, 1), (20000, 132, 579, 1), (512, 5120, 3072, 4), (203, 1333, 1027, 1)])
def test_scratch_of_the_lists(lib, B, CO, CI, G):
    """The lists take 64 MB or half of the call's own tensors; counters, the list of failed outputs (4 bytes for 128 of them) and, in the forward, the dense
    kernel's scratch come on top."""
    rest = 4 * (B * G + CO) + B * CO // 32 + (1 << 17)
    bound = lib.linf_inf_dist_bound_pruned_workspace_bytes(B, CO, CI, G, 1)
    assert 0 <= bound <= max(64 << 20, own_bytes(B, CO, CI, G, 2) // 2) + rest
    forward = lib.linf_inf_dist_forward_pruned_workspace_bytes(B, CO, CI, G, 1)
    dense = lib.linf_inf_dist_forward_workspace_bytes(B, CO, CI, G, 1)
    assert 0 <= forward <= max(64 << 20, own_bytes(B, CO, CI, G, 1) // 2) + rest + dense
    assert forward > 0 or bound > 0


def test_images_that_the_unfold_kernel_does_not_take():
    """More than 2^31 pixels, of which a stride leaves fewer patches: torch's unfold takes them, the kernel with its 32-bit counts does not."""
    import linfdist_b200 as L
    layer = L.NormDistConv(4, 32, 2, stride=4)

    def image(b, c, h, w):
        sizes = (b, c, h, w)
        return SimpleNamespace(is_cuda=True, dtype=torch.float32, dim=lambda: 4, numel=lambda: b * c * h * w, size=lambda k: sizes[k])

    assert layer._rows_from_patches(image(64, 4, 64, 64), 16, 16)
    assert not layer._rows_from_patches(image(200, 4, 2048, 2048), 512, 512)
