"""The sums over triangles and bands of the device-resident triangulation.

Accuracy: nd of many bands against the exact sum of the float64 contributions.
The additions at the size of the total dominate: a tree over the blocks' parts
rounds at total / 2^k, 2^k times, in all 0.41 units in the last place rms, and the
sums within blocks and the contributions themselves at most as much again, so
0.6 units = 1 to 1.3e-16 of the total; 1.5e-16 rms over the energies.  (One addition
after the other over 76 blocks: 2.3e-16.)  Beside it: calls on several streams at
once, which share the arrays for the parts, and a captured call."""
import math

import numpy as np
import pytest

from parphom_gb300 import dos, geometry, synth

pytestmark = pytest.mark.gpu


def _bands(grid, nb, seed):
    rng = np.random.default_rng(seed)
    q = synth.uniform_grid(grid)
    base = np.sort(rng.uniform(5.0, 1600.0, nb))
    amp, phase, hop = rng.uniform(2.0, 60.0, nb), rng.uniform(0, 2 * np.pi, nb), rng.integers(-2, 3, (nb, 2))
    freq = base + amp * np.cos(2 * np.pi * (q[:, :2] @ hop.T) + phase) + rng.uniform(0, 0.3, (len(q), nb))
    tri = dos.triangulate(q, geometry.reciprocal_lattice(synth.tblg_cell(3).lat))
    return np.sort(freq, axis=1), rng.uniform(0.1, 3.0, freq.shape), tri


def _exact_nd(freq, f, tri, E):
    e = freq[tri]
    o = np.argsort(e, axis=1)
    e, f = np.take_along_axis(e, o, 1), np.take_along_axis(f[tri], o, 1)
    (e0, e1, e2), (f0, f1, f2) = e.transpose(1, 0, 2), f.transpose(1, 0, 2)
    out = []
    for x in E:
        a, b = (x - e0) / (e1 - e0), (x - e0) / (e2 - e0)
        c, d = (e2 - x) / (e2 - e0), (e2 - x) / (e2 - e1)
        low = ((3 - a - b) * f0 + a * f1 + b * f2) * a * b
        up = (1 - d * c * c) * f0 + (1 - c * d * d) * f1 + (1 - 3 * c * d + d * c * c + c * d * d) * f2
        v = np.where(x <= e0, 0.0, np.where(x < e1, low, np.where(x < e2, up, f0 + f1 + f2)))
        out.append(math.fsum(v.ravel()))
    return np.array(out)


@pytest.mark.parametrize("weighted", [False, True])
def test_sums_round_like_a_tree(weighted):
    import torch
    freq, w, tri = _bands(16, 300, 1)
    E = np.linspace(30.0, 1650.0, 700)
    dev = torch.device("cuda")
    F, T, X = (torch.tensor(a, device=dev) for a in (freq, tri, E))
    W = torch.tensor(w, device=dev) if weighted else None
    _, nd = dos.linear_triangulation_device(F, T, X, func_dev=W)
    exact = _exact_nd(freq, w if weighted else np.ones_like(freq), tri, E)
    err = (nd.cpu().numpy() - exact) / exact
    assert np.sqrt((err ** 2).mean()) <= 1.5e-16


def test_streams_share_the_parts():
    import torch
    dev = torch.device("cuda")
    sets = []
    for k in range(5):
        freq, w, tri = _bands(8 + k, 60 + 31 * k, k)
        E = np.linspace(0.0, 1650.0, 300 + 177 * k)
        sets.append([torch.tensor(a, device=dev) for a in (freq, tri, E, w)])
    alone = [[t.clone() for t in dos.linear_triangulation_device(F, T, X, func_dev=W)] for F, T, X, W in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    for _ in range(20):
        got = []
        for s, (F, T, X, W) in zip(streams, sets):
            with torch.cuda.stream(s):
                got.append(dos.linear_triangulation_device(F, T, X, func_dev=W, stream=s.cuda_stream))
        torch.cuda.synchronize()
        for g, a in zip(got, alone):
            assert torch.equal(g[0], a[0]) and torch.equal(g[1], a[1])


def test_captured_call():
    import torch
    dev = torch.device("cuda")
    freq, w, tri = _bands(10, 80, 3)
    E = np.linspace(0.0, 1650.0, 600)
    F, T, X, W = (torch.tensor(a, device=dev) for a in (freq, tri, E, w))
    d, n = dos.linear_triangulation_device(F, T, X, func_dev=W)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        dc, nc = dos.linear_triangulation_device(F, T, X, func_dev=W, stream=torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        for a, b in ((dc, d), (nc, n)):
            assert float((a - b).abs().max()) <= 1e-13 * float(b.abs().max())


@pytest.mark.parametrize("vals", [(0.0, 1e-310, 1.0), (-1.0, 0.0, 3e-309), (0.0, 4e-310, 9e-310)])
def test_values_a_subnormal_apart(vals):
    """nd of a triangle whose frequencies lie so close that 1 / difference overflows: finite, as the quotients give it."""
    freq = np.array(vals)[:, None]
    gap = [k for k in range(2) if vals[k + 1] - vals[k] < 1e-308]
    E = np.array([vals[k] + f * (vals[k + 1] - vals[k]) for k in gap for f in (0.25, 0.5, 0.75)])
    _, nd = dos.linear_triangulation(freq, np.array([[0, 1, 2]]), E)
    for x, n in zip(E, nd):
        e0, e1, e2 = vals
        if x < e1:
            a, b = (x - e0) / (e1 - e0), (x - e0) / (e2 - e0)
            want = (3 - a - b + a + b) * a * b
        else:
            c, d = (e2 - x) / (e2 - e0), (e2 - x) / (e2 - e1)
            want = (1 - d * c * c) + (1 - c * d * d) + (1 - 3 * c * d + d * c * c + c * d * d)
        assert abs(n - want) <= 1e-12 * want


def test_call_while_another_thread_captures():
    """A call on an ordinary stream while another thread captures its own in the global mode: neither disturbs the other."""
    import threading
    import torch
    dev = torch.device("cuda")
    freq, w, tri = _bands(8, 50, 4)
    E = np.linspace(0.0, 1650.0, 300)
    F, T, X = (torch.tensor(a, device=dev) for a in (freq, tri, E))
    d, n = dos.linear_triangulation_device(F, T, X)
    outs = [(torch.zeros_like(d), torch.zeros_like(n)) for _ in range(4)]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    begun, called, err = threading.Event(), threading.Event(), []
    y = torch.zeros(16, device=dev)
    g = torch.cuda.CUDAGraph()

    def capture():
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                g.capture_begin(capture_error_mode="global")
                y.add_(1.0)
                begun.set()
                called.wait(20)
                y.add_(1.0)
                g.capture_end()
        except Exception as ex:   # noqa: BLE001
            err.append(ex)
            begun.set()

    t = threading.Thread(target=capture)
    t.start()
    begun.wait(20)
    L, p = dos._lib(), dos._ptr
    import ctypes
    rcs = [L.pp_dos_triangulation_device(p(F), F.shape[1], F.shape[0], F.shape[1], None, F.shape[1], p(T), len(T),
                                         p(X), len(X), p(a), p(b), ctypes.c_void_p(side.cuda_stream)) for a, b in outs]
    called.set()
    t.join()
    torch.cuda.synchronize()
    assert not err and rcs == [0] * 4, (err, rcs)
    for a, b in outs:
        assert torch.equal(a, d) and torch.equal(b, n)
    g.replay()
    torch.cuda.synchronize()
    assert float(y[0]) == 2.0
