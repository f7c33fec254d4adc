"""Builds of one work list replayed as a captured graph (a small molecule's builds after some twenty):
each repeat has other densities and other buffers, and the density screen, the spin, the FP64 forms
and a caller's own capture change in between.  Every build against the first (direct) build of a
fresh context on the same inputs: 1e-11 of the largest element (the order of the atomics), the
same quartet count."""
import numpy as np
import pytest

from conftest import golden, golden_basis, load_sqb200


def _fresh(sqb, g, P, **kw):
    eng = sqb.JKEngine(golden_basis(g), schwarz=g["schwarz"])
    out = eng.build(P[0], P[1], **kw)
    q = eng.stats()["quartets"]
    eng.close()
    return out, q


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["water_321g", "h2co_631gs"])
def test_replayed_builds_match_direct(case):
    import torch
    sqb = load_sqb200()
    g = golden(case)
    n = golden_basis(g).nbf
    rng = np.random.default_rng(6)
    eng = sqb.JKEngine(golden_basis(g), schwarz=g["schwarz"])
    f64 = dict(dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()
    steps = [(True, np.inf, None)] * 3 + [(True, 0.0, None)] * 2 + [(False, np.inf, None)] * 3 + [(True, np.inf, 1)] * 3 \
        + [(True, 1e-6, None)]
    for k, (restricted, rmax, form) in enumerate(steps):
        A = 10.0 ** -(k % 3) * rng.standard_normal((2, n, n))
        P = [A[0] + A[0].T, A[1] + A[1].T]
        if restricted:
            P[1] = P[0]
        kw = dict(restricted=restricted, scf_cutoff=1e-10, dscreen_rmax=rmax)
        if form is not None:
            eng.set_tiles(np.full(256, form, np.int32))
        d = [torch.tensor(p, **f64) for p in P]
        out = [torch.full((n, n), np.nan, **f64) for _ in range(3)]
        torch.cuda.synchronize()
        for _ in range(40 if k % 3 else 1):     # one in three is direct, the others are replays
            eng.build_tensors(d[0], d[1], *out, stream=st, **kw)
        st.synchronize()
        q = eng.stats()["quartets"]
        ref, q0 = _fresh(sqb, g, P, **kw)
        assert q == q0, k
        for x, y in zip(out, ref):
            assert np.abs(x.cpu().numpy() - y).max() <= 1e-11 * max(1.0, np.abs(y).max()), k
    # inside a caller's own capture the launches are the caller's nodes
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=st):
        eng.build_tensors(d[0], d[1], *out, stream=st, **kw)
    d[0].mul_(0.5)
    d[1].copy_(d[0])
    graph.replay()
    torch.cuda.synchronize()
    ref, _ = _fresh(sqb, g, [d[0].cpu().numpy()] * 2, **kw)
    assert np.abs(out[0].cpu().numpy() - ref[0]).max() <= 1e-11 * max(1.0, np.abs(ref[0]).max())
    eng.close()


class _Calls:
    """Builds of one context on one stream, each against a fresh context's first build."""

    def __init__(self, sqb, g, seed):
        import torch
        self.torch, self.sqb, self.g = torch, sqb, g
        self.n = golden_basis(g).nbf
        self.eng = sqb.JKEngine(golden_basis(g), schwarz=g["schwarz"])
        self.st = torch.cuda.Stream()
        rng = np.random.default_rng(seed)
        self.P = [A + A.T for A in rng.standard_normal((2, self.n, self.n))]
        self.d = [torch.tensor(p, dtype=torch.float64, device="cuda") for p in self.P]
        self.out = [torch.empty((self.n, self.n), dtype=torch.float64, device="cuda") for _ in range(3)]
        torch.cuda.synchronize()

    def build(self, **kw):
        self.eng.build_tensors(*self.d, *self.out, stream=self.st, scf_cutoff=1e-10, **kw)

    def check(self, **kw):
        self.st.synchronize()
        ref, _ = _fresh(self.sqb, self.g, self.P, scf_cutoff=1e-10, **kw)
        for x, y in zip(self.out, ref):
            assert np.abs(x.cpu().numpy() - y).max() <= 1e-11 * max(1.0, np.abs(y).max())

    def until_replayed(self, **kw):
        """Builds until one is a replay; how many were direct."""
        n0 = self.eng.replays()
        for k in range(100):
            self.build(**kw)
            if self.eng.replays() > n0:
                return k
        raise AssertionError("no build of this work list was replayed")


@pytest.mark.gpu
def test_which_builds_are_replays():
    import torch
    sqb = load_sqb200()
    c = _Calls(sqb, golden("h2co_631gs"), 9)
    kw = dict(restricted=False)
    # making the graph costs some twenty replays' gain: the builds of an ordinary SCF are direct
    assert c.until_replayed(**kw) >= 20
    c.check(**kw)
    for _ in range(3):                          # from then on every build is a replay
        n = c.eng.replays()
        c.build(**kw)
        assert c.eng.replays() == n + 1
    c.build(dscreen_rmax=0.0, **kw)             # the density screen is no part of the graph
    assert c.eng.replays() == n + 2
    c.check(dscreen_rmax=0.0, **kw)

    def direct(**k):
        n = c.eng.replays()
        c.build(**k)
        assert c.eng.replays() == n
        c.check(**k)

    direct(restricted=False, fixed_cutoff=1e-9)   # another work list
    c.eng.set_tiles(np.full(256, 2, np.int32))    # other forms
    direct(**kw)
    c.until_replayed(**kw)
    c.check(**kw)
    c.eng.profile(True)
    direct(**kw)
    c.eng.profile(False)
    c.eng.set_persistent(True)
    direct(**kw)
    c.eng.set_persistent(False)
    n = c.eng.replays()
    graph = torch.cuda.CUDAGraph()
    c.st.synchronize()
    with torch.cuda.graph(graph, stream=c.st):
        c.build(**kw)
    assert c.eng.replays() == n
    for x in c.out:
        x.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    c.check(**kw)
    c.build(**kw)
    assert c.eng.replays() == n + 1
    c.check(**kw)
    del graph
    c.eng.close()
