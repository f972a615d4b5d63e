"""Observables at the edges of their blocks: networks smaller than a warp, without links or
heads, FREE rods, more terms than one window of a chain, long chains and one giant component;
against numpy's order-free results (the ordered sums: tests/test_gpu_observables.py)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _components(n, edges):
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components
    e = np.array(edges, np.int64).reshape(-1, 2)
    _, comp = connected_components(coo_matrix((np.ones(len(e)), (e[:, 0], e[:, 1])), shape=(n, n)), directed=False)
    return comp


@pytest.mark.parametrize("sizes,links", [((1, 5, 31), 0), ((256, 257, 1000), 40), ((20000, 3), 30000), ((40000,), 0)])
def test_extent_and_clusters(sizes, links):
    from softbox_b200.runtime import default_context
    rng = np.random.default_rng(sum(sizes))
    n = sum(sizes)
    base = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    c = rng.normal(size=3 * n)
    state = np.where(rng.random(n) < 0.1, -1, 0).astype(np.int32)
    e2 = np.full(n, -1, np.int32)
    for a, b in zip(base[:-1], base[1:]):               # one chain through the whole network
        e2[a:b - 1] = np.arange(a + 1, b)
    e2[rng.random(n) < 0.02] = -1
    la, lb = (rng.integers(base[0], base[1], links).astype(np.int32) for _ in range(2))
    ls = np.where(rng.random(links) < 0.3, -1, 0).astype(np.int32)
    dev = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    ctx = default_context()
    nn = len(sizes)
    d = [dev(x) for x in (base, c, state, e2, la, lb, ls)]
    ext = torch.zeros(2 * nn, dtype=torch.float64, device="cuda")
    ctx("sbx_obs_extent", nn, d[0], n, None, d[1], d[2], ext)
    label, size = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    flags = torch.zeros(3, dtype=torch.int32, device="cuda")
    out = torch.full((2 * nn,), 9, dtype=torch.int32, device="cuda")
    ctx("sbx_obs_clusters", nn, d[0], n, d[2], d[3], links, d[4], d[5], d[6], 0, None, None, 0, 2, label, size, flags, out)
    torch.cuda.synchronize()
    live = state >= 0
    edges = [(i, e2[i]) for i in range(n) if e2[i] >= 0 and live[i] and live[e2[i]]]
    edges += [(a, b) for a, b, s in zip(la, lb, ls) if s >= 0 and live[a] and live[b]]
    comp = _components(n, edges)
    first = np.full(comp.max() + 1, n)
    np.minimum.at(first, comp, np.arange(n))
    assert np.array_equal(label.cpu().numpy(), np.where(live, first[comp], -1))
    assert flags.cpu().numpy()[1] == 0
    counts = np.bincount(comp[live], minlength=comp.max() + 1)
    got, ex = out.cpu().numpy().reshape(-1, 2), ext.cpu().numpy().reshape(-1, 2)
    xyz = c.reshape(3, n)
    for k in range(nn):
        s = slice(base[k], base[k + 1])
        m = live[s]
        assert got[k, 1] == m.sum() and got[k, 0] == (counts[comp[s][m]].max() if m.any() else 0)
        p = xyz[:, s][:, m]
        want = np.sqrt(((p - p.mean(axis=1, keepdims=True)) ** 2).sum(axis=0).mean()) if m.any() else 0.0
        assert ex[k, 1] == m.sum() and abs(ex[k, 0] - want) <= 1e-12 * max(want, 1.0)


@pytest.mark.parametrize("n,links", [(300_000, 0), (300_000, 1), (1 << 21, 0)])
def test_one_long_chain(n, links):
    # a walk along the chain takes fewer steps than a walk's limit (2^20), and every label is right
    from softbox_b200.runtime import default_context
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    ctx = default_context()
    e2 = torch.arange(1, n + 1, dtype=torch.int32, device="cuda")
    e2[-1] = -1
    label, size = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    flags, out, ends = dev([0, 0, 0]), dev([0, 0]), dev([0, n - 1, 0])
    for _ in range(3):                                 # (the third call is timed)
        torch.cuda.synchronize()
        s, e = torch.cuda.Event(True), torch.cuda.Event(True)
        s.record()
        ctx("sbx_obs_clusters", 1, dev([0, n]), n, None, e2, links, ends[:1], ends[1:2], ends[2:], 0, None, None, 0, 2,
            label, size, flags, out)
        e.record()
        torch.cuda.synchronize()
    assert out.tolist() == [n, n] and flags[1].item() == 0 and label.max().item() == 0
    assert s.elapsed_time(e) < 20                      # ms: hooking and compressing in rounds takes 3 at 2^21
