"""The kernels that the default shape chooses among (a block per flight, 32 lanes with a hand-over, four
flights per warp) against the explicit 32-lane shape: one summation order, so every distance, step count
and score is equal bit for bit, at the edges of each kernel's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _flights(torch, pe, G, seeds, shape=None, vary=0, max_steps=7200, smooth=0):
    e = pe.Engine(0)
    if shape:
        e.set_config(**shape)
    e.set_smooth_landing(smooth)
    pop, n = G.shape[0], G.shape[0] * len(seeds)
    g = torch.from_numpy(G).cuda()
    dist = torch.full((n,), 7.0, device="cuda")
    steps = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    scores = torch.empty(pop, device="cuda")
    out = []
    for _ in range(2):  # the second call finds the first one's lists and states
        e.eval_batch(g, pop, seeds, vary, max_steps, dist, steps, scores)
        torch.cuda.synchronize()
        out.append([x.cpu().numpy().view(np.int32).copy() for x in (dist, steps, scores)])
    e.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    return out[0]


def _same(torch, pe, G, seeds, **kw):
    want = _flights(torch, pe, G, seeds, shape=dict(lanes=32, warps=4, reg_cap=0, chunk=7200), **kw)
    got = _flights(torch, pe, G, seeds, **kw)
    for name, a, b in zip(("dist", "steps", "scores"), got, want):
        assert np.array_equal(a, b), (name, int((a != b).sum()))


@pytest.mark.parametrize("per_sm, extra", [(0, 1), (0, 3), (1, 0), (8, -1), (8, 0), (8, 1), (10, 0), (10, 1), (14, 5),
                                            (24, 0), (24, 1), (32, 0), (32, 1), (50, 7)])
def test_default_kernels_at_their_edges(cuda, pe, oracle, per_sm, extra):
    n = per_sm * cuda.cuda.get_device_properties(0).multi_processor_count + extra
    G = oracle.grand(400 + n, n)
    if n > 20:
        G[3, 11] = np.nan  # nose ballast: flies one step and reports a NaN flight
    _same(cuda, pe, G, [5])


@pytest.mark.parametrize("max_steps", [1, 2, 8, 9, 16, 17, 599, 600, 601, 1300])
@pytest.mark.parametrize("pop", [40, 300, 900])  # a block per flight, 32 lanes, four per warp
def test_default_kernels_horizon(cuda, pe, oracle, pop, max_steps):
    """Horizons about the polls for the hand-over and the clock's restart."""
    _same(cuda, pe, oracle.grand(11, pop), [1, 2, 3, 4, 5, 6, 7], max_steps=max_steps)


@pytest.mark.parametrize("pop", [40, 300, 900])
@pytest.mark.parametrize("vary, smooth", [(1, 0), (0, 1)])
def test_default_kernels_options(cuda, pe, oracle, pop, vary, smooth):
    _same(cuda, pe, oracle.grand(12, pop), [3, 7922, 15841, 23760, 31679, -4, 9], vary=vary, smooth=smooth)


@pytest.mark.parametrize("every", [1, 59, 60, 600])
def test_gradient_forward_kernels(cuda, pe, oracle, every):
    """The same genomes in a batch of a block per flight and in one that is handed over: distances and
    objectives bit for bit, gradients to the reverse kernels' own 1e-5 of the norm."""
    torch = cuda
    G, seeds, out = oracle.grand(21, 240), list(range(1, 9)), []
    for n in (20, 240):
        e = pe.Engine(0)
        g = torch.from_numpy(G[:n]).cuda()
        grad, obj = torch.empty(n, 35, device="cuda"), torch.empty(n, device="cuda")
        dist = torch.empty(n * 8, device="cuda")
        e.grad(g, n, seeds, grad, max_steps=2400, checkpoint_every=every, d_obj=obj, d_dist=dist)
        torch.cuda.synchronize()
        out.append((dist[:160].cpu().numpy(), obj[:20].cpu().numpy(), grad[:20].cpu().numpy().astype(np.float64)))
        e.close()
    a, b = out
    assert np.array_equal(a[0].view(np.int32), b[0].view(np.int32))
    assert np.array_equal(a[1].view(np.int32), b[1].view(np.int32))
    assert np.linalg.norm(a[2] - b[2]) <= 1e-5 * np.linalg.norm(b[2])


@pytest.mark.parametrize("knob, value", [("PE_GRAD_GROUP", "2"), ("PE_GRAD_GROUP", "0"), ("PE_GRAD_STEPS", "300"),
                                         ("PE_GRAD_STEPS", "1"), ("PE_GRAD_STEPS", "511"), ("PE_GRAD_STEPS", "513")])
@pytest.mark.parametrize("pop, nseeds, max_steps, every", [(1, 1, 1, 1), (5, 3, 31, 7), (33, 5, 33, 60), (40, 8, 513, 60),
                                                           (60, 4, 2400, 600)])
def test_gradient_parallel_in_time(cuda, pe, oracle, monkeypatch, pop, nseeds, max_steps, every, knob, value):
    """The reverse pass parallel in time against the serial kernels, and with its longer flights left to
    them: objectives and distances bit for bit, each genome's gradient to 1e-5 of its norm (two float
    adjoints of one trajectory; the serial kernels differ among themselves by 1e-6).  Horizons about its
    chunks of 32 steps and its parts of 512."""
    torch = cuda
    G = oracle.grand(31, pop)
    if pop > 4:
        G[2, 11] = np.nan
    e = pe.Engine(0)
    g, out = torch.from_numpy(G).cuda(), []
    for i in range(2):
        if i:
            monkeypatch.setenv(knob, value)
        grad, obj = torch.full((pop, 35), 3.0, device="cuda"), torch.empty(pop, device="cuda")
        dist = torch.empty(pop * nseeds, device="cuda")
        e.grad(g, pop, list(range(1, nseeds + 1)), grad, max_steps=max_steps, checkpoint_every=every, d_obj=obj, d_dist=dist)
        torch.cuda.synchronize()
        out.append((dist.cpu().numpy(), obj.cpu().numpy(), grad.cpu().numpy().astype(np.float64)))
    e.close()
    a, b = out
    assert np.array_equal(a[0].view(np.int32), b[0].view(np.int32)) and np.array_equal(a[1].view(np.int32), b[1].view(np.int32))
    bad = np.isnan(b[2]).any(axis=1)  # the NaN genome's row: its zero adjoints times a NaN mesh, on either side
    assert np.array_equal(np.isnan(a[2]), np.isnan(b[2])) and bad.sum() <= 1
    norm = np.linalg.norm(b[2][~bad], axis=1)
    assert (np.linalg.norm((a[2] - b[2])[~bad], axis=1) <= 1e-5 * norm).all()


@pytest.mark.parametrize("max_steps", [1, 2, 600, 601, 900])
def test_objective_flights_per_block(cuda, pe, oracle, max_steps):
    """pe_objective with a flight per block (few flights, FP32) and with four (more than 14 per SM): the same
    distances bit for bit, and FP64 (four per block) within FP32's rounding of them for flights this short
    of chaos (1e-3 of a metre for 99 % of flights; the rest pass through the FP32 gust sine's worst arguments)."""
    torch = cuda
    sm = torch.cuda.get_device_properties(0).multi_processor_count
    pop = 14 * sm // 7 + 1  # 7 scenarios: just over 14 flights per SM
    G, seeds = oracle.grand(51, pop), list(range(2, 9))
    e = pe.Engine(0)

    def dist(g, precision):
        n = g.shape[0]
        obj, d = (torch.empty(k, dtype=torch.float64, device="cuda") for k in (n, 7 * n))
        e.objective(torch.from_numpy(g).cuda(), n, seeds, precision=precision, max_steps=max_steps, d_obj=obj, d_dist=d)
        torch.cuda.synchronize()
        return obj.cpu().numpy(), d.cpu().numpy()

    many, few = dist(G, 32), dist(np.ascontiguousarray(G[5:45]), 32)
    assert np.array_equal(many[1][35:315], few[1]) and np.array_equal(many[0][5:45], few[0])
    wide = dist(G, 64)
    assert np.mean(np.abs(wide[1] - many[1]) <= 1e-3) >= 0.99
    e.close()


@pytest.mark.parametrize("pop,S,max_steps,chunk", [(1, 1, 7200, 7200), (7, 3, 1, 1), (40, 19, 601, 600), (40, 20, 1200, 599),
                                                   (200, 16, 7200, 600), (800, 16, 7200, 7200)])
def test_reference_order_blocks(cuda, pe, oracle, pop, S, max_steps, chunk):
    """The reference arithmetic with one to four flights per block (by the number of flights), in one launch
    and in chunks: the first planes' flights bit for bit as they fly alone, oversize planes left at -100."""
    torch = cuda
    G, seeds = oracle.grand(17, pop), list(range(4, 4 + S))

    def fly(g, steps_per_launch):
        e = pe.Engine(0)
        e.set_config(formulation=0, lanes=32, reg_cap=0, chunk=steps_per_launch)
        n = g.shape[0] * S
        d, st = torch.empty(n, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
        e.eval_batch(torch.from_numpy(g).cuda(), g.shape[0], seeds, 0, max_steps, d, st)
        torch.cuda.synchronize()
        nt = torch.empty(g.shape[0], dtype=torch.int32, device="cuda")
        e.plane_table(g.shape[0], d_nt=nt)
        torch.cuda.synchronize()
        e.close()
        return d.cpu().numpy(), st.cpu().numpy(), nt.cpu().numpy()

    d, st, nt = fly(G, chunk)
    over = np.repeat(nt <= 0, S)
    assert np.all(d[over] == -100.0) and np.all(st[over] == 0) and np.all(st[~over] > 0) and st.max() <= max_steps
    for p in range(min(pop, 5)):
        a = fly(G[p:p + 1], 7200)
        assert np.array_equal(a[0], d[p * S:(p + 1) * S]) and np.array_equal(a[1], st[p * S:(p + 1) * S])


@pytest.mark.parametrize("pop,S", [(1, 1), (3, 5), (32, 511), (32, 512)])  # results in one copy, and just beyond
@pytest.mark.parametrize("want", ["dist", "steps", "scores", "all"])
def test_host_results(cuda, pe, oracle, pop, S, want):
    torch = cuda
    G, seeds = oracle.grand(23, pop), list(range(5, 5 + S))
    e = pe.Engine(0)
    d, st, sc = torch.empty(pop * S, device="cuda"), torch.empty(pop * S, dtype=torch.int32, device="cuda"), torch.empty(pop, device="cuda")
    e.eval_batch(torch.from_numpy(G).cuda(), pop, seeds, 0, 40, d, st, sc)
    torch.cuda.synchronize()
    ref = {"dist": d, "steps": st, "scores": sc}
    for _ in range(2):
        out = e.evaluate_population(G, seeds, max_steps=40, **{"want_" + k: want in (k, "all") for k in ref})
        assert set(out) == {k for k in ref if want in (k, "all")}
        for k, v in out.items():
            assert np.array_equal(v, ref[k].cpu().numpy())
    e.close()


@pytest.mark.parametrize("pop", [1, 2, 31, 33, 127, 128, 129, 300])
def test_panel_offsets(cuda, pe, oracle, pop):
    """Panel offsets counted by the mesh's own blocks (at most 128 planes) and by the scan: the exclusive
    prefix of the topology's triangle counts, and the planes' panels as those of a plane alone."""
    torch = cuda
    G = oracle.grand(61, pop)

    def table(g):
        e, n = pe.Engine(0), g.shape[0]
        e.eval_batch(torch.from_numpy(g).cuda(), n, [1], 0, 1, torch.empty(n, device="cuda"))
        off, nt = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
        ext, pc = torch.empty(n, 4, device="cuda"), torch.zeros(n * 344, 4, device="cuda")
        total = e.plane_table(n, d_off=off, d_nt=nt, d_ext=ext, d_pc=pc)
        torch.cuda.synchronize()
        e.close()
        return off.cpu().numpy(), nt.cpu().numpy(), ext[:, 3].cpu().numpy().astype(int), pc.cpu().numpy(), total

    off, nt, topo, pc, total = table(G)
    assert np.array_equal(off, np.cumsum(topo) - topo) and total == topo.sum()
    for p in {0, pop // 2, pop - 1}:
        one = table(G[p:p + 1])
        assert one[1][0] == nt[p] and np.array_equal(one[3][:nt[p]], pc[off[p]:off[p] + nt[p]])


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("pop, nseeds", [(1, 1), (1, 8), (40, 8), (80, 8), (310, 8)])  # one to four flights per block
def test_objective_few_flights(cuda, pe, oracle, precision, pop, nseeds):
    """pe_objective's flights do not depend on how many share a block: the first planes as they fly alone."""
    torch = cuda
    G, seeds = oracle.grand(53, pop), list(range(2, 2 + nseeds))
    e = pe.Engine(0)

    def dist(g):
        n = g.shape[0]
        obj, d = (torch.empty(k, dtype=torch.float64, device="cuda") for k in (n, nseeds * n))
        e.objective(torch.from_numpy(np.ascontiguousarray(g)).cuda(), n, seeds, precision=precision, max_steps=700, d_obj=obj, d_dist=d)
        torch.cuda.synchronize()
        return obj.cpu().numpy(), d.cpu().numpy()

    obj, d = dist(G)
    for p in range(min(pop, 4)):
        alone = dist(G[p:p + 1])
        assert np.array_equal(alone[0], obj[p:p + 1]) and np.array_equal(alone[1], d[p * nseeds:(p + 1) * nseeds])
    e.close()


@pytest.mark.parametrize("blocks, warps", [(1, 8), (1, 1), (5, 7), (300, 2), (1000, 8)])
def test_reference_order_given_grid(cuda, pe, oracle, blocks, warps):
    """The reference arithmetic in a grid that is given: as in its own, bit for bit."""
    G, shape = oracle.grand(17, 50), dict(formulation=0, lanes=32, reg_cap=0)
    want = _flights(cuda, pe, G, [3, 4, 5, 6], shape=shape, max_steps=700)
    got = _flights(cuda, pe, G, [3, 4, 5, 6], shape=dict(blocks=blocks, warps=warps, **shape), max_steps=700)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
