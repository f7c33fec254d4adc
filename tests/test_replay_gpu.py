"""Builds of one work list replayed as a captured graph (a small molecule's builds from the second on):
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
