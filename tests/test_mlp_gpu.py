"""The learned warm start's network: the library's tensor-core forward and
backward kernels against the numpy oracle (which mirrors the device's BF16
roundings; the tolerance covers FP32 summation order), and training."""
import numpy as np
import pytest

from hl2sdk_tools_sharp_b200 import learned as LN, tracer as T

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net():
    import torch
    tr = T.CudaRayTracer(T.make_triangles(np.zeros((1, 9), np.float32), np.zeros(1, np.int32)))
    n = LN.Network(tr, seed=3)
    yield n, torch
    n.close()
    tr.close()


def _data(torch, n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, LN.INPUTS)).astype(np.float32)
    xt = torch.from_numpy(x).to("cuda").to(torch.bfloat16).contiguous()
    bits = xt.cpu().view(torch.int16).numpy().view(np.uint16)
    t = rng.normal(size=(n, LN.OUTPUTS)).astype(np.float32)
    return xt, bits, torch.from_numpy(t).cuda(), t


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def test_forward_matches_oracle(net):
    from oracle import mlp_oracle as MO
    n, torch = net
    xt, bits, _, _ = _data(torch, 1000, 1)       # not a multiple of the 128-row tile
    y = n.forward(xt).cpu().numpy()
    want, _, _ = MO.forward(n.params(), bits)
    assert _rel(y, want) < 2e-3


def test_gradient_matches_oracle(net):
    from oracle import mlp_oracle as MO
    n, torch = net
    xt, bits, tt, t = _data(torch, 777, 2)
    g, loss = n.gradient(xt, tt)
    want, want_loss = MO.gradient(n.params(), bits, t)
    assert abs(loss - want_loss) < 1e-3 * want_loss
    gs, ws = LN.split(g), LN.split(want.astype(np.float32))
    for name in ("w1", "b1", "w2", "b2", "w3", "b3"):
        assert _rel(gs[name], ws[name]) < 1e-2, name
    # Two calls give the same gradient but for the atomics' order.
    g2, _ = n.gradient(xt, tt)
    assert _rel(g2, g) < 1e-5


@pytest.mark.parametrize("rows", [1, 15, 17, 127, 128, 129, 148 * 128 + 1, 2 * 148 * 128 + 130])
def test_gradient_at_tile_edges(net, rows):
    """Row counts about a warp's 16 rows, a tile's 128 and the tiles the
    chip's CTAs take in one and two turns; the tolerances are
    test_gradient_matches_oracle's (BF16 activations and gradients)."""
    from oracle import mlp_oracle as MO
    n, torch = net
    xt, bits, tt, t = _data(torch, rows, 3 + rows)
    g, loss = n.gradient(xt, tt)
    want, want_loss = MO.gradient(n.params(), bits, t)
    assert abs(loss - want_loss) < 1e-3 * want_loss
    gs, ws = LN.split(g), LN.split(want.astype(np.float32))
    for name in ("w1", "b1", "w2", "b2", "w3", "b3"):
        assert _rel(gs[name], ws[name]) < 1e-2, name


def test_training_fits_a_function(net):
    import torch
    n, _ = net
    rng = np.random.default_rng(5)
    x = rng.uniform(-1, 1, size=(20000, LN.INPUTS)).astype(np.float32)
    t = np.stack([np.sin(2 * x[:, 0]) + x[:, 1] * x[:, 2], np.abs(x[:, 3]) - 0.5, x[:, 4] ** 2], 1).astype(np.float32)
    xt = torch.from_numpy(x).cuda().to(torch.bfloat16).contiguous()
    tt = torch.from_numpy(t).cuda()
    _, first = n.gradient(xt, tt)
    for step in range(400):
        n.train_step(xt, tt, 3e-3)
    torch.cuda.synchronize()
    last = n.loss()
    assert last < first / 10, (first, last)


def test_tcgen05_forward_at_scale_and_alignment(net):
    """The tcgen05 forward over a million rows (7,813 tiles on 2 CTAs per SM,
    the last tile partial) against the oracle on a spread of rows, and the
    same rows from a 4-byte-aligned (not 16-byte-aligned) input."""
    from oracle import mlp_oracle as MO
    n, torch = net
    rows = 1_000_003
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    xt = torch.randn((rows, LN.INPUTS), device="cuda", generator=g).to(torch.bfloat16).contiguous()
    y = n.forward(xt)
    torch.cuda.synchronize()
    n.status()
    pick = np.unique(np.concatenate([np.arange(0, 300), np.linspace(0, rows - 1, 3000).astype(np.int64),
                                     np.arange(rows - 300, rows)]))
    idx = torch.from_numpy(pick).cuda()
    bits = xt[idx].cpu().view(torch.int16).numpy().view(np.uint16)
    want, _, _ = MO.forward(n.params(), bits)
    got = y[idx].cpu().numpy()
    assert np.isfinite(got).all()
    assert _rel(got, want) < 2e-3
    # A view two elements in: rows start 4 bytes past a 16-byte boundary.
    buf = torch.zeros((4096 * LN.INPUTS + 2,), dtype=torch.bfloat16, device="cuda")
    view = buf[2:].view(4096, LN.INPUTS)
    view.copy_(xt[:4096])
    assert view.data_ptr() % 16 == 4
    y2 = n.forward(view)
    torch.cuda.synchronize()
    assert torch.equal(y2, y[:4096])


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 148 * 128 + 1, 2 * 148 * 128, 5 * 148 * 128 - 1])
def test_forward_at_tile_edges(net, rows):
    """One tile, a part of one, as many as the SMs, as many as are in flight,
    several rounds with a partial last one; a row of infinities and one of
    NaNs stay in their rows."""
    from oracle import mlp_oracle as MO
    n, torch = net
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    x = torch.randn((rows, LN.INPUTS), device="cuda", generator=g).to(torch.bfloat16).contiguous()
    y = n.forward(x)
    torch.cuda.synchronize()
    n.status()
    assert y.shape == (rows, 3)
    want, _, _ = MO.forward(n.params(), x.cpu().view(torch.int16).numpy().view(np.uint16))
    assert _rel(y.cpu().numpy(), want) < 2e-3
    bad = x.clone()
    bad[rows // 2] = float("nan")
    bad[rows - 1, 0] = float("inf")
    y2 = n.forward(bad)
    torch.cuda.synchronize()
    keep = torch.ones(rows, dtype=torch.bool, device="cuda")
    keep[rows // 2] = keep[rows - 1] = False
    assert torch.equal(y2[keep], y[keep])


def test_gradient_of_a_million_rows_is_summed_in_fp32(net):
    """Against 64-bit products of the same BF16 activations and gradients.
    A tile's 128 rows may lose an ulp (2^-23) a product step, eight steps;
    the tiles' sums are FP32 adds, 55 a CTA and an atomic add per CTA, whose
    roundings are as often up as down (2^-24 sqrt(203)); and an activation
    that FP32 and 64 bits round to different BF16 values moves a sum by some
    1e-6 at most.  1e-6 + 1e-6 + 2e-6 together."""
    n, torch = net
    rows = 1 << 20
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    x = torch.rand((rows, LN.INPUTS), device="cuda", generator=g).to(torch.bfloat16).contiguous()
    target = (6.0 * x[:, :LN.OUTPUTS].float() + torch.rand((rows, LN.OUTPUTS), device="cuda", generator=g)).contiguous()

    def bf(v):
        return v.float().to(torch.bfloat16).double()

    p = {k: torch.from_numpy(np.asarray(v, np.float32)).cuda() for k, v in LN.split(n.params()).items()}
    p = {k: bf(v) if k[0] == "w" else v.double() for k, v in p.items()}
    xd = x.double()
    h1 = bf(torch.relu(xd @ p["w1"] + p["b1"]))
    h2 = bf(torch.relu(h1 @ p["w2"] + p["b2"]))
    e = h2 @ p["w3"] + p["b3"] - target.double()
    dy = bf(2.0 * e / e.numel())
    dz2 = bf((dy @ p["w3"].T) * (h2 > 0))
    dz1 = bf((dz2 @ p["w2"].T) * (h1 > 0))
    want = {"w1": xd.T @ dz1, "b1": dz1.sum(0), "w2": h1.T @ dz2, "b2": dz2.sum(0), "w3": h2.T @ dy, "b3": dy.sum(0)}
    got, _ = n.gradient(x, target)
    off = {k: _rel(np.asarray(v, np.float64).ravel(), want[k].cpu().numpy().ravel()) for k, v in LN.split(got).items()}
    assert all(v < 4e-6 for v in off.values()), off


def test_gradients_from_several_threads(net):
    """More networks than pinned blocks are kept, their gradients taken at
    once from a thread each, on a stream each: every caller gets its own."""
    import threading
    n, torch = net
    tr = T.CudaRayTracer(T.make_triangles(np.zeros((1, 9), np.float32), np.zeros(1, np.int32)))
    nets = [LN.Network(tr, seed=s) for s in range(12)]
    data = [_data(torch, 300 + 7 * k, k) for k in range(len(nets))]
    torch.cuda.synchronize()
    want = [m.gradient(d[0], d[2]) for m, d in zip(nets, data)]
    got = [None] * len(nets)

    def work(k):
        stream = torch.cuda.Stream()
        for _ in range(20):
            got[k] = nets[k].gradient(data[k][0], data[k][2], stream=stream.cuda_stream)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(nets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (g, loss), (w, wl) in zip(got, want):
        assert _rel(g, w) < 1e-5 and abs(loss - wl) < 1e-5 * wl
    for m in nets:
        m.close()
    tr.close()
