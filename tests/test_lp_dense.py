"""Finite-p kernels of dense layers at the sizes where they can go wrong (edges of tiles and of the packed rows, sizes that are
multiples of nothing, groups, the smallest and the largest p), against the same sums in double precision."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(x, w, g, G, p):
    B, CI = x.shape
    CO, cig = w.shape
    cog = CO // G
    x, w, g = x.double(), w.double(), g.double()
    y = torch.empty(B, CO, dtype=torch.float64, device=x.device)
    gx = torch.zeros(B, CI, dtype=torch.float64, device=x.device)
    gw = torch.zeros(CO, cig, dtype=torch.float64, device=x.device)
    for k in range(G):
        rows, cols = slice(k * cog, (k + 1) * cog), slice(k * cig, (k + 1) * cig)
        t = x[:, cols][:, None, :] - w[None, rows]
        M = t.abs().amax(-1, keepdim=True).clamp_min(1e-300)
        yk = M[..., 0] * ((t.abs() / M) ** p).sum(-1) ** (1 / p)
        f = g[:, rows, None] * (t.abs() / yk[..., None].clamp_min(1e-300)) ** (p - 1) * t.sign()
        y[:, rows], gx[:, cols], gw[rows] = yk, f.sum(1), -f.sum(0)
    return y, gx, gw


def norm_error(a, b):
    return float((a.double() - b).norm() / b.norm())


def check(L, x, w, g, G, p):
    """A term's rounding (a few units of 2^-24) is raised to the power p: 2^-22 + p * 2^-23 in the 2-norm."""
    x, w = x.clone().requires_grad_(), w.clone().requires_grad_()
    y = L.norm_dist(x, w, G, p)
    gx, gw = torch.autograd.grad(y, [x, w], g)
    ref = reference(x.detach()[:, :, 0], w.detach(), g[:, :, 0], G, p)
    limit = 2.0 ** -22 * 4 + p * 2.0 ** -23
    for name, a, b in zip(("y", "grad_input", "grad_weight"), (y.detach()[:, :, 0], gx[:, :, 0], gw), ref):
        assert norm_error(a, b) <= limit, (name, norm_error(a, b), limit)
    return y.detach(), gx, gw


@pytest.mark.parametrize("p", [2.0, 2.5, 8.0, 16.0, 23.7, 40.0, 64.0, 97.3, 1000.0])
@pytest.mark.parametrize("B,CI,CO,G", [(33, 33, 33, 1), (8, 64, 32, 1), (70, 96, 130, 2), (130, 68, 36, 1), (203, 207, 101, 1), (2100, 64, 64, 1)])
def test_dense_gradients(cuda, lib, B, CI, CO, G, p):
    import linfdist_b200 as L
    torch.manual_seed(B)
    x, w, g = (torch.randn(*s, device="cuda") for s in ((B, CI, 1), (CO, CI // G), (B, CO, 1)))
    y, gx, gw = check(L, x, w, g, G, p)
    # one gradient alone: the same numbers to the rounding of another summation order
    for need in (0, 1):
        t = [x.clone(), w.clone()]
        t[need].requires_grad_()
        one, = torch.autograd.grad(L.norm_dist(t[0], t[1], G, p), t[need], g)
        both = (gx, gw)[need]
        assert torch.linalg.norm(one - both) <= 1e-5 * torch.linalg.norm(both)


@pytest.mark.parametrize("p", [8.0, 16.0, 23.7, 64.0])
@pytest.mark.parametrize("scale", [1e-6, 1e6])
def test_dense_far_from_one(cuda, lib, p, scale):
    """Differences whose p-th power leaves the range of a float."""
    import linfdist_b200 as L
    torch.manual_seed(1)
    x, w, g = (torch.randn(*s, device="cuda") for s in ((130, 100, 1), (65, 100), (130, 65, 1)))
    check(L, x * scale, w * scale, g, 1, p)


@pytest.mark.parametrize("p", [8.0, 16.0])
def test_dense_large_common_offset(cuda, lib, p):
    """Inputs and weights far from zero with small differences: neither the rows past the batch nor the outputs past the
    group, which exist only to fill a tile, may bring in the power of a lone large number."""
    import linfdist_b200 as L
    torch.manual_seed(2)
    x, w, g = (torch.randint(-4, 5, s, device="cuda").float() for s in ((33, 36, 1), (33, 36), (33, 33, 1)))
    x, w = x + 2.0 ** 20, w + 2.0 ** 20
    x[:, 0] += 1
    check(L, x, w, g, 1, p)


def off_by_one_float(t):
    """The same values in memory that starts 4 bytes past a 16-byte boundary (a view of a flat buffer)."""
    flat = torch.empty(t.numel() + 4, device=t.device)
    v = flat[1: 1 + t.numel()].view(t.shape)
    assert v.data_ptr() % 16 == 4
    return v.copy_(t)


@pytest.mark.parametrize("p", [2.0, 3.0, 7.5, 100.5, 300.0])
def test_unaligned_tensors_keep_the_generic_kernel(cuda, lib, p):
    """Channel counts that are multiples of four do not make a dense layer an aligned one.  The generic kernel, which serves spatial layouts
    as well, adds the same powers in the same order there: the same bits."""
    import linfdist_b200 as L
    torch.manual_seed(3)
    B, CI, CO = 70, 96, 64
    x, w = torch.randn(B, CI, 1, device="cuda"), torch.randn(CO, CI, device="cuda")
    y = L.norm_dist(off_by_one_float(x), off_by_one_float(w), 1, p)
    s = torch.cuda.current_stream().cuda_stream
    spatial, want = x[:, :, 0].t().contiguous().view(1, CI, B), torch.empty(1, CO, B, device="cuda")
    assert lib.linf_norm_dist_forward(spatial.data_ptr(), w.data_ptr(), 1, CO, CI, 1, B, want.data_ptr(), p, s) == 0
    assert torch.equal(y[:, :, 0], want[0].t())


@pytest.mark.parametrize("p", [2.5, 8.0, 16.0, 23.7, 64.0, 300.0])
@pytest.mark.parametrize("B,CI,CO,G", [(33, 64, 36, 1), (70, 97, 65, 1), (130, 2052, 64, 1), (2100, 64, 64, 2)])
def test_unaligned_tensors(cuda, lib, B, CI, CO, G, p):
    import linfdist_b200 as L
    torch.manual_seed(B)
    CI, CO = CI * G, CO * G
    x, w, g = (off_by_one_float(torch.randn(*s, device="cuda")) for s in ((B, CI, 1), (CO, CI // G), (B, CO, 1)))
    x.requires_grad_(); w.requires_grad_()
    y = L.norm_dist(x, w, G, p)
    gx, gw = torch.autograd.grad(y, [x, w], g)
    ref = reference(x.detach()[:, :, 0], w.detach(), g[:, :, 0], G, p)
    limit = 2.0 ** -22 * 4 + p * 2.0 ** -23          # as in `check`
    for name, a, b in zip(("y", "grad_input", "grad_weight"), (y.detach()[:, :, 0], gx[:, :, 0], gw), ref):
        assert norm_error(a, b) <= limit, (name, norm_error(a, b), limit)


def clamped(x, w, p, y=None, g=None):
    """What a call that the generic kernel served gives for any data, in double precision: a term is min(|t| / M, 1)^p with min(NaN, 1) = 1, M the
    largest |t| that is a number; in the gradients min(|t| / y, 1)^(p-1) with 1 / y = 0 where y is not positive, and the sign of x - w or w - x (minus for 0 and NaN)."""
    t = x.double()[:, None, :] - w.double()[None]
    unit = lambda u: torch.where(u < 1.0, u, torch.ones_like(u))
    if g is None:
        M = torch.where(t.isnan(), torch.zeros_like(t), t.abs()).amax(-1, keepdim=True)
        S = (unit(t.abs() * torch.where(M > 0, 1 / M, torch.zeros_like(M))) ** p).sum(-1)
        return torch.where(M[..., 0] > 0, S ** (1 / p) * M[..., 0], torch.zeros_like(S))
    y = y.double()[..., None]
    T = unit(t.abs() * torch.where(y > 0, 1 / y, torch.zeros_like(y))) ** (p - 1)
    T = g.double()[..., None] * T
    return torch.where(t > 0, T, -T).sum(1), torch.where(t < 0, T, -T).sum(0)


def spoil(x, w):
    x, w = x.clone(), w.clone()
    x[1, 3, 0], x[2, 5, 0], x[4, 0, 0] = float("inf"), float("nan"), -float("inf")
    x[7] = float("nan")
    w[2, 6], w[5, 1], w[9] = float("inf"), float("nan"), float("nan")
    w[8, 4], x[8, 4, 0] = float("inf"), float("inf")
    return x, w


def assert_same_kind(a, b, limit, what):
    """Infinities and NaN in the same places, and the numbers close in the 2-norm."""
    a, b = a.double(), b.double()
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isposinf(), b.isposinf()) and torch.equal(a.isneginf(), b.isneginf()), what
    ok = b.isfinite()
    assert norm_error(a[ok], b[ok]) <= limit, (what, norm_error(a[ok], b[ok]), limit)


@pytest.mark.parametrize("p", [8.0, 16.0, 23.7, 64.0, 100.0])
@pytest.mark.parametrize("B,CI,CO,aligned", [(70, 99, 65, True), (70, 96, 65, True), (203, 1027, 301, True), (130, 64, 36, False)])
def test_infinities_and_nan_forward(cuda, lib, B, CI, CO, aligned, p):
    """Calls that are no aligned dense layer: ragged channel counts, tensors off a 16-byte boundary."""
    import linfdist_b200 as L
    torch.manual_seed(B)
    x, w = spoil(torch.randn(B, CI, 1, device="cuda"), torch.randn(CO, CI, device="cuda"))
    place = (lambda t: t) if aligned else off_by_one_float
    x, w = place(x), place(w)
    y = L.norm_dist(x, w, 1, p)[:, :, 0]
    assert_same_kind(y, clamped(x[:, :, 0], w, p), 2.0 ** -22 * 4 + p * 2.0 ** -23, "y")
    tiny = 2.0 ** -140          # 1 / M is infinite: every term counts 1
    y = L.norm_dist(place(torch.full_like(x, tiny)), place(torch.zeros_like(w)), 1, p)
    assert torch.allclose(y, torch.full_like(y, CI ** (1 / p)) * tiny, rtol=1e-5, atol=2.0 ** -149)


@pytest.mark.parametrize("p", [8.0, 16.0, 23.7, 64.0, 100.0])
@pytest.mark.parametrize("B,CI,CO,aligned", [(70, 99, 65, True), (20, 96, 65, True), (203, 1027, 301, True), (2100, 64, 36, False), (2100, 64, 36, True)])
def test_infinities_and_nan_backward(cuda, lib, B, CI, CO, aligned, p):
    import linfdist_b200 as L
    torch.manual_seed(B)
    x, w = torch.randn(B, CI, 1, device="cuda"), torch.randn(CO, CI, device="cuda")
    generic = not aligned or CI % 4 != 0 or CO % 4 != 0
    if generic:
        x, w = spoil(x, w)      # (aligned layers have no rule for such data: NaN)
    g = torch.randn(B, CO, 1, device="cuda")
    place = (lambda t: t) if aligned else off_by_one_float
    x, w = place(x).requires_grad_(), place(w).requires_grad_()
    y = L.norm_dist(x, w, 1, p)
    with torch.no_grad():
        xs, ws, ys = x[:, :, 0].detach(), w.detach(), y[:, :, 0].detach()
    limit = 2.0 ** -22 * 4 + p * 2.0 ** -23
    for bad in (None, float("inf")):
        if bad is not None and p > 8.0:
            break               # (factors that underflow in 32 bits: inf * 0)
        if bad is not None:
            g[3, 7, 0] = bad
        grads = torch.autograd.grad(y, [x, w], g, retain_graph=True)
        for name, a, b in zip(("grad_input", "grad_weight"), (grads[0][:, :, 0], grads[1]), clamped(xs, ws, p, ys, g[:, :, 0])):
            assert_same_kind(a, b, limit, (name, bad))


def separate_gradients(lib, x, w, y, g, G, p):
    """Both gradients by the entry points that work out one each."""
    B, CI, _ = x.shape
    CO, s = w.shape[0], torch.cuda.current_stream().cuda_stream
    gx, gw = torch.empty_like(x), torch.empty_like(w)
    a = (g.data_ptr(), x.data_ptr(), w.data_ptr(), y.data_ptr(), B, CO, CI, G, 1)
    assert lib.linf_norm_dist_backward_input(*a, gx.data_ptr(), p, s) == 0
    assert lib.linf_norm_dist_backward_weight(*a, gw.data_ptr(), p, s) == 0
    return gx, gw


@pytest.mark.parametrize("B,CI,CO,p,aligned", [(2100, 64, 64, 150.0, False), (2048, 36, 40, 1000.0, False), (70, 35, 65, 64.0, True), (2100, 60, 64, 64.0, False)])
def test_large_powers_keep_the_clamped_kernels(cuda, lib, B, CI, CO, p, aligned):
    import linfdist_b200 as L
    torch.manual_seed(B)
    place = (lambda t: t) if aligned else off_by_one_float
    x, w, g = (place(torch.randn(*s, device="cuda")) for s in ((B, CI, 1), (CO, CI), (B, CO, 1)))
    x.requires_grad_(); w.requires_grad_()
    y = L.norm_dist(x, w, 1, p)
    got = torch.autograd.grad(y, [x, w], g)
    want = separate_gradients(lib, x.detach(), w.detach(), y.detach(), g, 1, p)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("p,size,g_size", [(16.0, 2.0, 2.0 ** -75), (16.0, 2.0, 2.0 ** -100), (8.0, 16.0, 2.0 ** -95), (8.0, 1.0, 2.0 ** -60)])
def test_gradients_of_small_grad_output(cuda, lib, p, size, g_size):
    """g / y^(p-1) below the normal numbers although the gradients are not."""
    import linfdist_b200 as L
    torch.manual_seed(4)
    x, w, g = (torch.randn(*s, device="cuda") for s in ((70, 99, 1), (65, 99), (70, 65, 1)))
    check(L, x * size, w * size, g * g_size, 1, p)


@pytest.mark.parametrize("B,CI,CO,p,alone", [(2048, 64, 64, 8.0, "input"), (8200, 64, 36, 23.7, "input"), (16, 130, 65, 23.7, "weight"), (70, 99, 37, 8.0, "input")])
def test_one_gradient_that_its_own_kernel_does(cuda, lib, B, CI, CO, p, alone):
    import linfdist_b200 as L
    torch.manual_seed(B)
    x, w, g = (torch.randn(*s, device="cuda") for s in ((B, CI, 1), (CO, CI), (B, CO, 1)))
    (x if alone == "input" else w).requires_grad_()
    y = L.norm_dist(x, w, 1, p)
    got, = torch.autograd.grad(y, [x if alone == "input" else w], g)
    want = separate_gradients(lib, x.detach(), w.detach(), y.detach(), g, 1, p)
    assert torch.equal(got, want[0 if alone == "input" else 1])
