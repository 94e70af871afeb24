"""Limits that decide on the host how a call is run: no GPU needed."""
from types import SimpleNamespace

import torch


def test_images_that_the_unfold_kernel_does_not_take():
    """More than 2^31 pixels, of which a stride leaves fewer patches: torch's unfold takes them, the kernel with its 32-bit counts does not."""
    import linfdist_b200 as L
    layer = L.NormDistConv(4, 32, 2, stride=4)

    def image(b, c, h, w):
        sizes = (b, c, h, w)
        return SimpleNamespace(is_cuda=True, dtype=torch.float32, dim=lambda: 4, numel=lambda: b * c * h * w, size=lambda k: sizes[k])

    assert layer._rows_from_patches(image(64, 4, 64, 64), 16, 16)
    assert not layer._rows_from_patches(image(200, 4, 2048, 2048), 512, 512)
