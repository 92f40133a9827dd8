"""pe_grad's serial reverse kernels, which take the calls that the pass parallel in time does not: flights that
share blocks, the pipelined pass of the longest ones, and the line between the two kinds of pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEEDS = list(range(25, 33))


def _run(torch, e, G, seeds, max_steps=3600, K=60, vary=0):
    """Objectives, gradients and distances of a call, and how many kernels it launched."""
    n, S = G.shape[0], len(seeds)
    grad, obj, dist = (torch.full(s, 3.0, device="cuda") for s in ((n, 35), (n,), (n * S,)))
    e.grad(torch.from_numpy(np.ascontiguousarray(G)).cuda(), n, seeds, grad, vary=vary, max_steps=max_steps,
           checkpoint_every=K, d_obj=obj, d_dist=dist)
    torch.cuda.synchronize()
    return obj.cpu().numpy(), grad.cpu().numpy(), dist.cpu().numpy(), e.last_timing()["launches"]


def _norms(a, b, tol=1e-5):
    return np.linalg.norm(a.astype(np.float64) - b, axis=1) <= tol * np.linalg.norm(b.astype(np.float64), axis=1)


@pytest.mark.parametrize("pop, nseeds, max_steps, K, vary", [(256, 8, 3600, 60, 0), (101, 3, 2400, 7, 0), (101, 3, 2400, 61, 0),
                                                             (101, 3, 2400, 96, 0), (64, 3, 2400, 60, 1), (64, 3, 2400, 97, 0)])
def test_shared_blocks_change_nothing(cuda, engine, oracle, monkeypatch, pop, nseeds, max_steps, K, vary):
    """The serial kernels with the flights two to a block (PE_GRAD_GROUP=2; rebuilt a segment ahead up to
    checkpoints every 60 steps, not so up to 96, not shared beyond) and with a block each (3) give the same
    objectives, distances and gradients bit for bit; the one-flight kernel (0), whose sums run over four warps
    instead of three, the same objectives and distances and gradients to 1e-5 of their norm."""
    G = oracle.grand(4, pop)
    usual, out = _run(cuda, engine, G, SEEDS[:nseeds], max_steps, K, vary), {}
    for group in ("2", "3", "0"):
        monkeypatch.setenv("PE_GRAD_GROUP", group)
        out[group] = _run(cuda, engine, G, SEEDS[:nseeds], max_steps, K, vary)
    for k in range(4):
        np.testing.assert_array_equal(out["2"][k], out["3"][k])
    for k in (0, 2):
        np.testing.assert_array_equal(out["0"][k], out["2"][k])
    assert _norms(out["0"][1], out["2"][1]).all()
    assert usual[3] > out["2"][3]  # not the pass parallel in time, which has four kernels more


def test_longest_flights_pass(cuda, engine, oracle, monkeypatch):
    """A small batch gives its longest flights a block of three roles each, a large one fewer of them: 24 genomes
    alone (192 flights) and among 256, objectives and distances bit for bit, gradients to 1e-5 of their norm."""
    monkeypatch.setenv("PE_GRAD_GROUP", "2")
    G = oracle.grand(4, 256)
    some, all_ = _run(cuda, engine, G[100:124], SEEDS), _run(cuda, engine, G, SEEDS)
    np.testing.assert_array_equal(some[0], all_[0][100:124])
    np.testing.assert_array_equal(some[2], all_[2][800:992])
    assert _norms(some[1], all_[1][100:124]).all()


@pytest.mark.parametrize("steps", [31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 257])
@pytest.mark.parametrize("knob", [None, "PE_GRAD_STEPS"])
def test_parts_and_stages(cuda, engine, oracle, monkeypatch, steps, knob):
    """Horizons about the chunks of 32 steps, the Jacobians' items of 64, the panels' stages of 96 and parts of
    128, and the same lengths as the limit beyond which a flight takes the serial kernel."""
    G = oracle.grand(31, 60)
    monkeypatch.setenv("PE_GRAD_GROUP", "2")
    want = _run(cuda, engine, G, SEEDS[:4], 700 if knob else steps)
    monkeypatch.delenv("PE_GRAD_GROUP")
    monkeypatch.setenv("PE_GRAD_STEPS", str(steps if knob else 3072))  # set, it takes the pass at any horizon
    got = _run(cuda, engine, G, SEEDS[:4], 700 if knob else steps)
    for k in (0, 2):
        np.testing.assert_array_equal(got[k], want[k])
    assert _norms(got[1], want[1]).all() and got[3] > want[3]


def test_records_that_do_not_fit(cuda, pe, oracle, monkeypatch):
    """The pass parallel in time within a bound on its memory and the serial kernels beyond it, on one engine, back and
    forth: objectives and distances bit for bit, gradients to 1e-5 of their norm.  40 x 8 flights of 513 steps take 320 x
    (544 entries of 96 B, 17 chunks of 17,168 B, four more parts of 9,664 B, 64 B and 14 items) = 122,513,920 bytes."""
    G, e = oracle.grand(31, 40), pe.Engine(0)
    need = 320 * (544 * 96 + 17 * 17168 + 4 * 9664 + 64 + 14 * 4)
    out = []
    for bytes_ in (need, need - 1, None, 0):
        if bytes_ is None:
            monkeypatch.delenv("PE_GRAD_BYTES")
        else:
            monkeypatch.setenv("PE_GRAD_BYTES", str(bytes_))
        out.append(_run(cuda, e, G, SEEDS, 513))
    e.close()
    for a, b in ((0, 2), (1, 3)):
        for k in range(4):
            np.testing.assert_array_equal(out[a][k], out[b][k])
    for k in (0, 2):
        np.testing.assert_array_equal(out[0][k], out[1][k])
    assert out[0][3] > out[1][3] and _norms(out[0][1], out[1][1]).all()


def test_records_at_their_largest(cuda, pe, oracle):
    """About the bound itself: 557 planes x 8 flights of 3,072 steps take the pass parallel in time (8.99 GiB), 558
    the serial kernels; objectives and distances bit for bit, gradients to 1e-5 of their norm for 98 % of the planes
    (two float adjoints of one trajectory, amplified by the worst-conditioned flights) and 1e-3 for all."""
    G, e = oracle.grand(31, 558), pe.Engine(0)
    within, beyond = _run(cuda, e, G[:557], SEEDS, 3072), _run(cuda, e, G, SEEDS, 3072)
    e.close()
    assert within[3] > beyond[3]
    np.testing.assert_array_equal(within[0], beyond[0][:557])
    np.testing.assert_array_equal(within[2], beyond[2][:557 * 8])
    assert _norms(within[1], beyond[1][:557]).mean() >= 0.98 and _norms(within[1], beyond[1][:557], 1e-3).all()


@pytest.mark.parametrize("pop, nseeds, short, longer", [(8, 8, (1, 48, 64, 65, 95), (96,)), (64, 8, (1, 48), (49, 64, 65, 95, 96)),
                                                        (400, 8, (1, 48, 65, 95), (49, 64, 96))])
def test_short_horizons_take_the_serial_kernels(cuda, engine, oracle, monkeypatch, pop, nseeds, short, longer):
    """Where the pass parallel in time does not pay for its launches and its items of 64 steps: below 96 steps for few
    flights, below 49 for all, from 65 to 95 for more than 16 per SM."""
    G = oracle.grand(31, pop)
    for steps in short + longer:
        monkeypatch.delenv("PE_GRAD_GROUP", raising=False)
        got = _run(cuda, engine, G, SEEDS[:nseeds], steps)
        monkeypatch.setenv("PE_GRAD_GROUP", "2")
        want = _run(cuda, engine, G, SEEDS[:nseeds], steps)
        for k in (0, 2):
            np.testing.assert_array_equal(got[k], want[k])
        assert _norms(got[1], want[1]).all()
        assert (got[3] > want[3]) == (steps in longer), steps
