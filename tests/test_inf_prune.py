"""The p = inf forward and bounds through lists of large entries against the full scan: the same bits for every kind of data, whether
the lists serve, some outputs have to be scanned again, or the dense kernel does the layer."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def make_x(kind, *shape):
    x = torch.randn(*shape, device="cuda")
    if kind == "uniform":
        return torch.rand(*shape, device="cuda")
    if kind == "narrow":
        return 0.25 * x
    if kind == "ties":
        return (x * 4).round() / 4
    if kind == "equal":
        return torch.ones_like(x)
    if kind == "rows":                       # rows of very different size: the smallest output says little about the others
        return x * torch.exp(torch.randn(shape[0], 1, 1, device="cuda"))
    if kind == "spikes":                     # more outputs fail the test than the list of them holds
        x = 0.01 * x
        x[:: 2, 0] = 50.0
        return x
    if kind == "special":
        x[3, 5] = x[9] = float("nan")
        x[11, 7] = float("inf")
        x[12] = 0.0
    return x


@pytest.mark.parametrize("kind", ["normal", "uniform", "narrow", "ties", "equal", "rows", "spikes", "special"])
@pytest.mark.parametrize("B,CI,CO,G", [(203, 1027, 1333, 1), (512, 784, 3780, 1), (130, 3001, 700, 1), (517, 4096, 1432, 2), (20000, 580, 132, 1), (64, 9999, 300, 1)])
def test_same_bits_as_the_full_scan(cuda, lib, B, CI, CO, G, kind):
    torch.manual_seed(B)
    x, w = make_x(kind, B, CI, 1), torch.randn(CO, CI // G, device="cuda")
    if kind == "ties":
        w = (w * 4).round() / 4
    if kind == "special":
        w[5, 3], w[6, 2] = float("inf"), float("nan")
    s = torch.cuda.current_stream().cuda_stream
    clean = lambda t: torch.nan_to_num(t, nan=7.0, posinf=8.0, neginf=9.0)
    new = lambda dtype=torch.float32: torch.full((B, CO, 1), -7, dtype=dtype, device="cuda")

    y, pos, y2, pos2, y3 = new(), new(torch.int32), new(), new(torch.int32), new()
    sub, add = torch.randn(CO, device="cuda"), torch.randn(CO, device="cuda")
    n = lib.linf_inf_dist_forward_pruned_workspace_bytes(B, CO, CI, G, 1)
    assert n > 0
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    sizes = (B, CO, CI, G, 1)
    assert lib.linf_inf_dist_forward_pruned(x.data_ptr(), w.data_ptr(), *sizes, None, None, 0, y.data_ptr(), pos.data_ptr(), ws.data_ptr(), n, s) == 0
    assert lib.linf_inf_dist_forward(x.data_ptr(), w.data_ptr(), *sizes, y2.data_ptr(), pos2.data_ptr(), s) == 0
    assert torch.equal(clean(y), clean(y2)) and torch.equal(pos, pos2)
    assert lib.linf_inf_dist_forward_pruned(x.data_ptr(), w.data_ptr(), *sizes, sub.data_ptr(), add.data_ptr(), 1, y3.data_ptr(), None, ws.data_ptr(), n, s) == 0
    assert torch.equal(clean(y3), clean(-((y2 - sub.view(1, -1, 1)) + add.view(1, -1, 1))))

    lo, up = x - 0.03, x + 0.03
    if kind == "special":
        lo[2, 4] = up[2, 4] + 1.0            # an empty interval
    n = lib.linf_inf_dist_bound_pruned_workspace_bytes(B, CO, CI, G, 1)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    a = [new() for _ in range(4)]
    for post in ((None, None, 0), (sub.data_ptr(), add.data_ptr(), 1)):
        assert lib.linf_inf_dist_bound_pruned(lo.data_ptr(), up.data_ptr(), w.data_ptr(), *sizes, *post, a[0].data_ptr(), a[1].data_ptr(), ws.data_ptr(), n, s) == 0
        assert lib.linf_inf_dist_bound_forward_post(lo.data_ptr(), up.data_ptr(), w.data_ptr(), *sizes, *post, a[2].data_ptr(), a[3].data_ptr(), s) == 0
        assert torch.equal(clean(a[0]), clean(a[2])) and torch.equal(clean(a[1]), clean(a[3]))


@pytest.mark.parametrize("kind", ["tight", "spikes", "special"])
@pytest.mark.parametrize("B,CI,CO,G", [(256, 2048, 1024, 1), (520, 2060, 1300, 2)])
def test_bounds_by_two_halves_behind_the_lists(cuda, lib, B, CI, CO, G, kind):
    """Data that the lists do not serve, at sizes where the dense kernel behind them splits the reduction: the halves meet in outputs that
    the list pass has written before."""
    torch.manual_seed(B)
    CI, CO = CI * G, CO * G
    x, w = make_x(kind, B, CI, 1), torch.randn(CO, CI // G, device="cuda")
    if kind == "tight":
        x, w = torch.rand_like(x), torch.rand_like(w)
    lo, up = x - 0.03, x + 0.03
    if kind == "special":
        lo[2, 4] = up[2, 4] + 1.0
    s, sizes = torch.cuda.current_stream().cuda_stream, (B, CO, CI, G, 1)
    sub, add = torch.randn(CO, device="cuda"), torch.randn(CO, device="cuda")
    n = lib.linf_inf_dist_bound_pruned_workspace_bytes(*sizes)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    for post in ((None, None, 0), (sub.data_ptr(), add.data_ptr(), 1)):
        a = [torch.full((B, CO, 1), 1e30, device="cuda") for _ in range(4)]
        assert lib.linf_inf_dist_bound_pruned(lo.data_ptr(), up.data_ptr(), w.data_ptr(), *sizes, *post, a[0].data_ptr(), a[1].data_ptr(), ws.data_ptr(), n, s) == 0
        assert lib.linf_inf_dist_bound_forward_post(lo.data_ptr(), up.data_ptr(), w.data_ptr(), *sizes, *post, a[2].data_ptr(), a[3].data_ptr(), s) == 0
        assert torch.equal(a[0].nan_to_num(7.0), a[2].nan_to_num(7.0)) and torch.equal(a[1].nan_to_num(7.0), a[3].nan_to_num(7.0))


def off_by_one_float(t):
    """The same values in memory that starts 4 bytes past a 16-byte boundary."""
    return torch.empty(t.numel() + 4, dtype=t.dtype, device=t.device)[1: 1 + t.numel()].view(t.shape).copy_(t)


def pruned_forward(lib, x, w, y, pos, ws):
    B, CO, CI, s = x.size(0), w.size(0), x.size(1), torch.cuda.current_stream().cuda_stream
    assert lib.linf_inf_dist_forward_pruned(x.data_ptr(), w.data_ptr(), B, CO, CI, 1, 1, None, None, 0, y.data_ptr(), pos.data_ptr(), ws.data_ptr(), ws.numel(), s) == 0


def new_outputs(lib, x, w):
    n = lib.linf_inf_dist_forward_pruned_workspace_bytes(x.size(0), w.size(0), x.size(1), 1, 1)
    assert n > 0
    shape = (x.size(0), w.size(0), 1)
    return (torch.full(shape, -7.0, device="cuda"), torch.full(shape, -7, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.uint8, device="cuda"))


def full_scan(lib, x, w):
    y, pos, _ = new_outputs(lib, x, w)
    assert lib.linf_inf_dist_forward(x.data_ptr(), w.data_ptr(), x.size(0), w.size(0), x.size(1), 1, 1, y.data_ptr(), pos.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    return y, pos


@pytest.mark.parametrize("kind", ["normal", "narrow", "spikes"])
@pytest.mark.parametrize("which", ["x", "w", "outputs", "all"])
def test_unaligned_tensors(cuda, lib, which, kind):
    torch.manual_seed(1)
    x, w = make_x(kind, 640, 1024, 1), torch.randn(2304, 1024, device="cuda")
    want, want_pos = full_scan(lib, x, w)
    lo, up = x - 0.03, x + 0.03
    s, sizes = torch.cuda.current_stream().cuda_stream, (640, 2304, 1024, 1, 1)
    want_lo, want_up = torch.empty_like(want), torch.empty_like(want)
    assert lib.linf_inf_dist_bound_forward(lo.data_ptr(), up.data_ptr(), w.data_ptr(), *sizes, want_lo.data_ptr(), want_up.data_ptr(), s) == 0
    y, pos, ws = new_outputs(lib, x, w)
    out_lo, out_up = torch.empty_like(y), torch.empty_like(y)
    if which in ("x", "all"):
        x, lo, up = off_by_one_float(x), off_by_one_float(lo), off_by_one_float(up)
    if which in ("w", "all"):
        w = off_by_one_float(w)
    if which in ("outputs", "all"):
        y, pos, out_lo, out_up = (off_by_one_float(t) for t in (y, pos, out_lo, out_up))
    pruned_forward(lib, x, w, y, pos, ws)
    assert torch.equal(y, want) and torch.equal(pos, want_pos)
    n = lib.linf_inf_dist_bound_pruned_workspace_bytes(*sizes)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    assert lib.linf_inf_dist_bound_pruned(lo.data_ptr(), up.data_ptr(), w.data_ptr(), *sizes, None, None, 0, out_lo.data_ptr(), out_up.data_ptr(), ws.data_ptr(), n, s) == 0
    assert torch.equal(out_lo, want_lo) and torch.equal(out_up, want_up)


def test_under_graph_capture(cuda, lib):
    """The decision between the lists and the dense kernel is taken on the device, at each replay on the data that are there then."""
    torch.manual_seed(2)
    w = torch.randn(2304, 1024, device="cuda")
    x = make_x("narrow", 640, 1024, 1)
    y, pos, ws = new_outputs(lib, x, w)
    pruned_forward(lib, x, w, y, pos, ws)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pruned_forward(lib, x, w, y, pos, ws)
    for kind in ("narrow", "equal", "uniform", "spikes", "narrow"):
        x.copy_(make_x(kind, 640, 1024, 1))
        y.fill_(-7.0); pos.fill_(-7)
        graph.replay()
        want, want_pos = full_scan(lib, x, w)
        assert torch.equal(y, want) and torch.equal(pos, want_pos), kind


@pytest.mark.parametrize("streams", [1, 2])
def test_two_host_threads(cuda, lib, streams):
    """Two threads that call at the same time, on one stream or on one each, do not disturb each other's scratch."""
    import threading
    import linfdist_b200 as L
    torch.manual_seed(3)
    w = torch.randn(2304, 1024, device="cuda")
    xs = [make_x("narrow", 640, 1024, 1), make_x("uniform", 640, 1024, 1)]
    wants = [full_scan(lib, x, w)[0] for x in xs]
    torch.cuda.synchronize()
    side = [torch.cuda.Stream() for _ in range(streams)]
    got, errors = [[], []], []

    def work(k):
        try:
            with torch.cuda.stream(side[k % streams]):
                for _ in range(20):
                    got[k].append(L.norm_dist(xs[k], w, 1, float("inf")))
        except Exception as e:                  # (a thread's exception would be lost)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    assert all(torch.equal(y, wants[k]) for k in (0, 1) for y in got[k])
