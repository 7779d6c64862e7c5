"""The rounds scheduler (launches of fewer than 64 instances) where it can go wrong:
grids that do not divide into tiles, fewer tiles than CTAs and many tiles per
CTA, launches of one, a few and 63 instances of different ends, and the reverse
solve on a graph with a cycle."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import make_dictin
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(model, shape, seed, nseeds=2):
    rng = np.random.default_rng(seed)
    nd = len(shape)
    h = 1.0 / max(shape)
    case = dict(model=model, dims=np.array(shape, np.float32), gridScales=np.full(nd, h, np.float32),
                origin=np.zeros(nd, np.float32))
    idx = np.stack([rng.integers(0, n, nseeds) for n in shape], -1)
    case["seeds"] = ((idx + 0.5) * h).astype(np.float32)
    cost = rng.uniform(0.8, 1.2, shape).astype(np.float32)
    if model.startswith("Isotropic"):
        case["cost"] = cost
    else:
        a = rng.standard_normal((nd, nd))
        m = 0.3 * np.eye(nd) + a @ a.T
        case["metric"] = (cost[..., None] * m[np.tril_indices(nd)]).astype(np.float32)
    return case


def _interfaces(cases):
    from adaptivegriddiscretizations_b200.Eikonal.HFM_CUDA import Interface
    itfs = []
    for c in cases:
        it = Interface(make_dictin(c, extra={"exportValues": True}))
        it.SetKernelTraits()
        it.SetGeometry()
        it.SetArgs()
        itfs.append(it)
    return itfs


def _close(v, case):
    ref = O.run(dict(case, atol=1e-12, rtol=1e-12), np.float64)["values"]
    fin = np.isfinite(ref)
    assert np.array_equal(fin, np.isfinite(v))
    # four stopping tolerances (5e-6 relative to the value, 5e-6 of the cost absolute)
    assert (np.abs(v - ref)[fin] <= 2e-5 * ref[fin] + 2.5e-5).all()


@pytest.mark.parametrize("ctas", [0, 1, 5, 148])
@pytest.mark.parametrize("model,shape", [("Isotropic2", (1, 1)), ("Isotropic2", (17, 33)), ("Riemann2", (9, 70)),
                                         ("Riemann3", (5, 4, 13)), ("Isotropic3", (21, 6, 9)), ("Riemann2", (163, 129))])
def test_rounds_tiles_and_ctas(model, shape, ctas):
    from adaptivegriddiscretizations_b200 import _lib
    from adaptivegriddiscretizations_b200.Eikonal.HFM_CUDA import BatchPlan
    case = _case(model, shape, 3, nseeds=1 if shape == (1, 1) else 2)
    it, = _interfaces([case])
    plan = BatchPlan([it], launch=_lib.AgdLaunch(ctas=ctas, warps_per_cta=0, timeout_ns=0))
    plan.run()
    torch.cuda.synchronize()
    niter, status, visits = plan.read_stats()
    assert status[0] == 0 and niter[0] >= 1 and visits[0] >= niter[0]
    _close(it.squeeze(it.values_t).cpu().numpy(), case)


@pytest.mark.parametrize("count", [2, 63])
def test_rounds_instances(count):
    """Instances of different sizes, models and ends share the epochs; one has an iteration limit."""
    from adaptivegriddiscretizations_b200 import _lib
    from adaptivegriddiscretizations_b200.Eikonal.HFM_CUDA import BatchPlan
    cases = [_case(("Riemann2", "Isotropic2")[k % 2], (20 + 7 * k % 90, 9 + 11 * k % 70), k) for k in range(count)]
    itfs = _interfaces(cases)
    itfs[0].nitermax_o = 2
    plan = BatchPlan(itfs)
    plan.run()
    torch.cuda.synchronize()
    niter, status, visits = plan.read_stats()
    assert status[0] == _lib.AGD_STATUS_NOT_CONVERGED and niter[0] == 2
    assert not status[1:].any()
    for k in list(range(1, count))[:: max(1, count // 8)]:
        _close(itfs[k].squeeze(itfs[k].values_t).cpu().numpy(), cases[k])


def test_reverse_with_a_cycle():
    """A hand-made graph: a chain of points across tiles that feeds a cycle of two, and a row
    outside the grid that must be ignored, against a dense solve in float64."""
    from adaptivegriddiscretizations_b200 import _lib
    it, = _interfaces([_case("Isotropic2", (40, 40), 1)])
    N, n = it.size_tot, 40
    rng = np.random.default_rng(0)
    fw = np.zeros((2, N), np.float32)
    fi = np.full((2, N), 2 ** 31 - 1, np.int64)
    chain = rng.permutation(N)[:200]
    for a, b in zip(chain[:-1], chain[1:]):
        fw[0, a], fi[0, a] = rng.uniform(0.2, 0.9), b
    x, y = chain[-1], chain[-2]
    fw[1, x], fi[1, x] = 0.3, y  # the cycle
    fw[1, chain[0]], fi[1, chain[0]] = 0.5, N + 3  # outside: no edge
    wsum = np.ones(N, np.float32)
    sens = np.zeros(N, np.float32)
    sens[chain[:100]] = rng.uniform(-1, 1, 100)
    W = np.zeros((N, N))
    for k in range(2):
        for z in np.nonzero(fw[k])[0]:
            if fi[k, z] < N:
                W[z, fi[k, z]] += fw[k, z]
    ref = np.linalg.solve(np.diag(wsum.astype(np.float64)) - W.T, sens)
    dev = lambda a, t: torch.as_tensor(a.astype(t)).cuda()  # noqa: E731
    fw_t, fi_t, ws_t, s_t = dev(fw, np.float32), dev(fi, np.int32), dev(wsum, np.float32), dev(sens, np.float32)
    lam, stats = torch.empty(N, device="cuda"), torch.zeros(2, dtype=torch.int64, device="cuda")
    inst = it.instance()
    L = _lib.lib()
    nbytes = L.agd_reverse_workspace_bytes(ctypes.byref(inst))
    ws = torch.empty(int(nbytes), dtype=torch.uint8, device="cuda")
    _lib.check(L.agd_reverse(ctypes.byref(inst), _lib.ptr(fw_t), _lib.ptr(fi_t), _lib.ptr(ws_t), _lib.ptr(s_t),
                             _lib.ptr(lam), ctypes.c_float(0.0), ctypes.c_float(5e-6), _lib.ptr(ws), int(nbytes),
                             _lib.ptr(stats), None, _lib.stream_ptr()))
    torch.cuda.synchronize()
    assert int(stats[0].item()) >> 32 == 0
    # 200 steps, each passing changes above 5e-6 of the value on
    assert np.abs(lam.cpu().numpy() - ref).max() <= 2e-5 * np.abs(ref).max()


def test_rounds_captured_and_two_streams():
    """The rounds' cooperative launch in a captured graph, replayed, and two solves in flight
    on two streams: the values are the plain run's (the schedule may differ: within tolerance)."""
    from adaptivegriddiscretizations_b200.Eikonal.HFM_CUDA import BatchPlan
    cases = [_case("Riemann2", (163, 129), 5), _case("Isotropic2", (130, 257), 6)]
    itfs = _interfaces(cases)
    plans = [BatchPlan([it]) for it in itfs]

    def step(k):
        itfs[k].values_t.fill_(float("inf"))
        plans[k].run()

    streams = [torch.cuda.Stream() for _ in plans]
    for _ in range(3):
        for k, s in enumerate(streams):
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                step(k)
    torch.cuda.synchronize()
    for it, c in zip(itfs, cases):
        _close(it.squeeze(it.values_t).cpu().numpy(), c)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for k in range(2):
            step(k)
    for it in itfs:
        it.values_t.zero_()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for p, it, c in zip(plans, itfs, cases):
        assert not p.read_stats()[1].any()
        _close(it.squeeze(it.values_t).cpu().numpy(), c)
