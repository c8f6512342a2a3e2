"""Full global placement on the GPU (CPU-runnable design, 10k cells, 128x128 bins).

* the graph-captured engine and the reference-shaped autograd path follow the
  same trajectory (same kernels, same operation order) for the first iterations;
* GP reaches the 0.07 overflow stop, and the split-BF16 Poisson solve ends
  within 0.1% HPWL of the plain fp32 form."""
import pytest
import torch

from dreamplace_b200 import synthetic
from dreamplace_b200.nonlinear_place import place
from dreamplace_b200.params import Params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def design():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return synthetic.cells_10k()


def run(design, engine, precision, iters=None, deterministic=0):
    traj = []
    p = Params(target_density=design.target_density, stop_overflow=0.07, dct_precision=precision, gp_engine=engine,
               deterministic_flag=deterministic)
    placer, res = place(design, p, max_iterations=iters, callback=lambda it, m: traj.append((m.hpwl, m.overflow)))
    return placer, res, traj


def test_engine_matches_autograd_path(design):
    _, _, a = run(design, "autograd", "fp32", 8, deterministic=1)
    _, _, b = run(design, "graph", "fp32", 8, deterministic=1)
    _, _, c = run(design, "eager", "fp32", 8, deterministic=1)
    for (ha, oa), (hb, ob), (hc, oc) in zip(a, b, c):
        assert abs(ha - hb) <= 1e-4 * ha and abs(oa - ob) <= 1e-4
        assert hb == hc and ob == oc  # graph replay == the same kernels launched eagerly


def test_gp_converges_and_split_bf16_matches_plain(design):
    """Deterministic mode (int64 density maps), so the two runs differ only in
    the Poisson-solve arithmetic."""
    _, plain, _ = run(design, "graph", "fp32", deterministic=1)
    _, split, _ = run(design, "graph", "split_bf16", deterministic=1)
    for r in (plain, split):
        assert r["overflow"] <= 0.07 + 1e-9 and r["iterations"] < 1000
    print("plain", plain, "split", split, "rel", abs(split["hpwl"] - plain["hpwl"]) / plain["hpwl"])
    assert abs(split["hpwl"] - plain["hpwl"]) <= 1e-3 * plain["hpwl"], (split, plain)


def test_recapture_with_one_timed_piece_keeps_the_trajectory(design):
    """GPEngine.time_only (the bench's timed window): the trial graphs,
    captured again mid-GP with one piece's events, follow the run that kept
    its first graphs bit for bit (deterministic mode), and the piece is timed."""
    p = lambda **kw: Params(target_density=design.target_density, stop_overflow=0.07,  # noqa: E731
                            dct_precision="split_bf16", deterministic_flag=1, **kw)
    t1, t2 = [], []
    place(design, p(time_pieces=True), max_iterations=40, callback=lambda it, m: t1.append((m.hpwl, m.overflow)))
    holder = {}

    def cb(it, m):
        t2.append((m.hpwl, m.overflow))
        if it == 12:
            eng = holder["placer"].stepper.eng
            eng.time_only(["wa_forward"])
            holder["eng"] = eng

    from dreamplace_b200.nonlinear_place import NonLinearPlace
    params = p(time_pieces=True)
    placer = NonLinearPlace(params, design, "cuda")
    holder["placer"] = placer
    placer(params, design, max_iterations=40, callback=cb)
    assert t1 == t2
    means = holder["eng"].piece_means()
    assert set(means) == {"wa_forward"} and means["wa_forward"] > 0


def test_gp_deterministic_mode_is_reproducible(design):
    p = lambda: Params(target_density=design.target_density, stop_overflow=0.07, dct_precision="fp32",  # noqa: E731
                       deterministic_flag=1)
    t1, t2 = [], []
    place(design, p(), max_iterations=30, callback=lambda it, m: t1.append((m.hpwl, m.overflow)))
    place(design, p(), max_iterations=30, callback=lambda it, m: t2.append((m.hpwl, m.overflow)))
    assert t1 == t2


def test_trial_metrics_match_direct_evaluation(design):
    """The HPWL summed inside the trial's WA forward and the overflow from the
    trial's movable-only map equal a direct evaluation of the same position
    (bit for bit in deterministic mode), and the HPWL matches the oracle."""
    import numpy as np
    import oracle
    placer, _, _ = run(design, "graph", "fp32", 6, deterministic=1)
    eng = placer.stepper.eng
    q = eng.parity  # v_k, produced by the last accepted trial
    h_trial, o_trial = eng.H[q][0].item(), eng.O[q][0:2].clone()
    eng.evaluate(q)
    assert eng.H[q][0].item() == h_trial
    assert torch.equal(eng.O[q][0:2], o_trial)
    d = design
    pos = eng.V[q].cpu().numpy()
    n, P = d.num_nodes, d.num_pins
    px = pos[d.pin2node_map] + d.pin_offset_x
    py = pos[n + d.pin2node_map] + d.pin_offset_y
    ref = oracle.hpwl(np.concatenate([px, py]).astype(np.float32), d.flat_net2pin_map, d.flat_net2pin_start_map,
                      np.ones(d.num_nets, np.uint8), d.net_weights)
    ref = ref[0] if isinstance(ref, tuple) else ref
    assert abs(h_trial - ref) <= 1e-6 * ref


def test_iteration_head_matches_host_loop():
    """dp_iteration_head against the host loop's formulas (NonLinearPlace
    density-weight update in RePlAce HPWL mode, gamma update, Nesterov advance):
    HPWL up and down, both clamps of mu, the first iteration (no update)."""
    import math
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dreamplace_b200._native import C
    base_gamma, area, ref, lower, upper = 4.0 * 46.875, 2.5e6, 350000.0, 0.95, 1.05
    cases = [(0, 1.0e6, 9.0e5, 0.9), (1, 1.0e6, 9.0e5, 0.5), (7, 1.0e6, 1.1e6, 0.3), (12, 1.0e6, 1.0e6 + 1e9, 0.12),
             (30, 2.0e6, 2.0e6 + 1.0, 0.07), (400, 5.0e5, 4.0e5, 0.2)]
    for k, hp_prev, hp, ovf in cases:
        st_prev = torch.zeros(8 + 2 * 1280, dtype=torch.float64, device="cuda")
        st_prev[0:4] = torch.tensor([0.3, 2.5, 3.1, 0.4], dtype=torch.float64)
        st_new = torch.zeros_like(st_prev)
        sched_prev = torch.tensor([float(k), hp_prev], dtype=torch.float64, device="cuda")
        sched_new = torch.zeros(2, dtype=torch.float64, device="cuda")
        w_prev = torch.tensor([1.7e-4, 20.0, 0.05], dtype=torch.float32, device="cuda")
        w_new = torch.zeros(3, dtype=torch.float32, device="cuda")
        hpk = torch.tensor([hp], dtype=torch.float64, device="cuda")
        ovk = torch.tensor([ovf * area], dtype=torch.float64, device="cuda")
        C.iteration_head(st_prev, st_new, sched_prev, sched_new, hpk, ovk, w_prev, w_new, base_gamma, area, ref,
                         lower, upper)
        # the host loop (nonlinear_place.py run_gen)
        f = k + 1
        lam = torch.tensor([1.7e-4], dtype=torch.float32)
        if f > 1:
            delta = hp - hp_prev
            if delta < 0:
                mu = upper * max(math.pow(0.9999, float(f)), 0.98)
            else:
                mu = upper * min(max(math.pow(upper, -delta / ref), lower), upper)
            lam.mul_(mu)
        gamma = torch.zeros((), dtype=torch.float32).fill_(base_gamma * math.pow(10, ((ovf * area) / area - 0.1) * 20 / 9 - 1))
        w = w_new.cpu()
        assert w[0].item() == lam.item(), (k, w[0].item(), lam.item())
        assert w[1].item() == gamma.item()
        assert w[2].item() == (1.0 / gamma.reshape(1)).item()
        a = 3.1
        an = (1.0 + math.sqrt(4.0 * a * a + 1.0)) / 2.0
        got = st_new[0:4].cpu().tolist()
        assert got == [0.3, a, an, (a - 1.0) / an]
        assert sched_new.cpu().tolist() == [float(f), hp]


def test_speculative_iterations_match_serial(design):
    """Iteration k+1 enqueued ahead of the host (speculate) gives the serial
    loop's trajectory bit for bit in deterministic mode, retries included."""
    traj = {}
    for spec in (False, True):
        t = []
        p = Params(target_density=design.target_density, stop_overflow=0.07, dct_precision="fp32",
                   deterministic_flag=1, speculate=spec)
        placer, res = place(design, p, max_iterations=120, callback=lambda it, m: t.append((m.hpwl, m.overflow)))
        traj[spec] = (t, placer.stepper.eng.trials, placer.pos[0].detach().cpu())
    (t0, n0, p0), (t1, n1, p1) = traj[False], traj[True]
    assert n0 == n1 and n0 > 120  # some iterations needed a retry
    assert t0 == t1
    assert torch.equal(p0, p1)


def test_trial_gate_skips_gated_kernels():
    """Launches made while a trial gate is installed return at once when the
    word is set, and run when it is clear; dp_trial_gate sets it from an
    accept flag; launches after removal ignore the word."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dreamplace_b200._native import C
    n = 1000
    xy = torch.arange(2 * n, dtype=torch.float32, device="cuda")
    order = torch.arange(n - 1, -1, -1, dtype=torch.int32, device="cuda")
    gate = torch.zeros(1, dtype=torch.int32, device="cuda")
    rejected = torch.zeros(1, dtype=torch.float64, device="cuda")
    accepted = torch.ones(1, dtype=torch.float64, device="cuda")
    out = torch.full((2 * n,), -1.0, device="cuda")
    C.set_trial_gate(gate)
    try:
        C.trial_gate(gate, rejected)
        C.gather_order_xy(xy, order, n, out)
        assert gate.item() == 1 and bool((out == -1.0).all())
        C.trial_gate(gate, accepted)
        C.gather_order_xy(xy, order, n, out)
        assert gate.item() == 0
        assert torch.equal(out.view(-1, 2), xy.view(-1, 2)[order.long()])
        C.trial_gate(gate, rejected)
    finally:
        C.set_trial_gate(None)
    out.fill_(-1.0)
    C.gather_order_xy(xy, order, n, out)  # gate removed: runs although the word is set
    assert gate.item() == 1 and torch.equal(out.view(-1, 2), xy.view(-1, 2)[order.long()])


@pytest.mark.parametrize("xyo_mode,wa_grad_order", [("order", "lane"), ("trial", "lane"), ("gather", "csr")])
def test_engine_layout_options_give_the_same_trajectory(design, xyo_mode, wa_grad_order):
    """The engine's layout options (how the scatter reads the trial point, where
    the WA gradient is written) change no arithmetic: deterministic runs give
    the default layout's trajectory bit for bit."""
    def traj(**kw):
        t = []
        p = Params(target_density=design.target_density, stop_overflow=0.07, dct_precision="fp32",
                   deterministic_flag=1, **kw)
        place(design, p, max_iterations=40, callback=lambda it, m: t.append((m.hpwl, m.overflow, m.objective)))
        return t
    assert traj(xyo_mode=xyo_mode, wa_grad_order=wa_grad_order) == traj()


def test_best_position_copied_before_its_slot_is_reused(design):
    """The GP loop's best position is copied lazily: a newer best supersedes a
    pending copy, a pending copy is made on the stream before a trial
    overwrites the slot holding it, and the divergence rollback
    (set_position) completes it first."""
    p = Params(target_density=design.target_density, stop_overflow=0.07, dct_precision="fp32", deterministic_flag=1)
    placer, _ = place(design, p, max_iterations=10)
    eng = placer.stepper.eng

    def step():
        g = eng.step_gen()
        next(g)
        try:
            next(g)
        except StopIteration:
            pass

    step()
    first = eng.current_position().clone()
    buf = eng.mark_best(None)
    step()
    second = eng.current_position().clone()
    assert eng.mark_best(buf) is buf  # supersedes the first best before any copy
    for _ in range(4):
        step()  # the trials write every slot, the second best's included
    torch.cuda.synchronize()
    assert eng.best_slot is None
    assert torch.equal(buf, second) and not torch.equal(buf, first)
    step()
    third = eng.current_position().clone()
    eng.mark_best(buf)
    eng.set_position(buf)  # completes the pending copy, then restores from it
    torch.cuda.synchronize()
    assert torch.equal(buf, third) and torch.equal(eng.current_position(), third)


def test_profile_piece_runs_every_piece():
    """The profiling entry point runs each piece of the trial on a GP state."""
    from dreamplace_b200 import profile_piece
    for piece in profile_piece.PIECES:
        profile_piece.main(["--piece", piece, "--design", "cells_10k", "--iterations", "3", "--repeat", "1"])


@pytest.mark.parametrize("precision,deterministic", [("split_bf16", 1), ("split_bf16", 0), ("fp32", 1), ("tf32", 1)])
def test_fused_trial_equals_its_pieces(design, precision, deterministic):
    """A trial through dp_trial_* (head, zeroing, finishers and scalar kernels
    folded into the heavy kernels) against the stand-alone entry points launched
    one by one: every sum keeps its order, so deterministic maps give the same
    bits; fp32 atomics may add in another order (1e-4 of the largest entry)."""
    from dreamplace_b200._native import C
    from dreamplace_b200.electric_potential import poisson_solve
    placer, _, _ = run(design, "graph", precision, 6, deterministic=deterministic)
    eng = placer.stepper.eng
    ep, d = eng.ep, eng.design
    torch.cuda.synchronize()
    s = eng.slot
    r, t = (s - 1) % 3, (s + 1) % 3
    # an iteration ahead may have run from slot s: start from its inputs
    eng._trial(s, head=True)
    torch.cuda.synchronize()
    names = ("V", "U", "G", "XY", "XYO")
    got = {k: getattr(eng, k)[t].clone() for k in names}
    got.update(row=eng.metrics[s].clone(), host=eng.metrics_host[s].clone().cuda(), state=eng.S[s][:8].clone(),
               weights=eng.weights[s].clone(), sched=eng.sched[s].clone(), hpwl=eng.H[t][0].clone(),
               ovf=eng.O[t][:2].clone())
    for k in names:
        getattr(eng, k)[t].fill_(-1.0)
    C.iteration_head(eng.S[r], eng.S[s], eng.sched[r], eng.sched[s], eng.H[r][0:1], eng.O[r][0:1], eng.weights[r],
                     eng.weights[s], *eng.head_scalars, gate=eng.gate)
    assert eng.gate.item() == 0
    eng.nesterov_trial_only(s)
    w = eng.weights[s]
    eng.wirelength(eng.V[t], eng.H[t], w[2:3])
    eng.scatter_maps(eng.V[t], eng.O[t])
    ex, ey, energy = poisson_solve(eng.dmap, ep.bin_size_x, ep.bin_size_y, eng.prec, bool(ep.fast_mode),
                                   1.0 / (ep.bin_size_x * ep.bin_size_y), eng.poisson_ws)
    C.objective_finish(eng.wl64, energy, w[0:1], eng.factor_quad, eng.obj64, eng.grad_scale)
    eng.field_force(eng.V[t], ex, ey)
    eng.assemble(eng.V[s], eng.G[s], eng.V[t], eng.G[t], s)
    C.trial_metrics(eng.H[s], eng.O[s], eng.S[s], eng.obj64, eng.wl64, energy, eng.metrics[s])
    want = {k: getattr(eng, k)[t] for k in names}
    want.update(row=eng.metrics[s], host=eng.metrics[s], state=eng.S[s][:8], weights=eng.weights[s],
                sched=eng.sched[s], hpwl=eng.H[t][0], ovf=eng.O[t][:2])
    for k, v in want.items():
        # the energy is an atomic fp64 sum of the solve's tiles: its last bits vary
        rel = 1e-12 if deterministic and k in ("row", "host") else 0.0 if deterministic else 1e-4
        assert (got[k].double() - v.double()).abs().max() <= rel * v.double().abs().max(), k


def test_pinned_rows_outlive_the_warm_up_of_the_graphs(design):
    """A trial's last kernel writes the host's metrics row, which the pinned
    allocator does not see.  The warm-up of the graphs enqueues such a trial
    before any step has: an engine dropped then keeps its rows until that trial
    is done, and the next engine's set-up gives them back."""
    import gc
    from dreamplace_b200 import engine
    placer, _, _ = run(design, "graph", "fp32", 2, deterministic=1)
    first = placer.stepper.eng
    eng = engine.GPEngine(placer.params, design, placer.data_collections, placer.op_collections, placer.model, True)
    eng.load_state_dict(first.state_dict())
    eng._check_graph_key()
    eng._graph(eng.slot, False)
    rows = eng.metrics_host
    del eng
    gc.collect()
    assert any(kept is rows for kept, _ in engine._RETIRED)
    torch.cuda.synchronize()
    engine._release_retired()
    assert not any(kept is rows for kept, _ in engine._RETIRED)


@pytest.mark.parametrize("bins,precision,launches,bound", [(128, "split_bf16", 3, "hbm"), (256, "split_bf16", 4, "tensor"),
                                                          (256, "fp32", 3, "hbm"), (136, "fp32", 4, "fp32")])
def test_timed_pieces_are_the_trials_own(bins, precision, launches, bound):
    """GPEngine.trial_pieces (what the bench and the profiler time) run in order is
    a trial, bit for bit, and its solve is the one that the trial runs: three
    passes of the fast transforms, rated by their maps, or four products."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import bench
    from dreamplace_b200._native import C
    d = synthetic.scaled(3000, num_bins=bins, seed=9)
    placer, _, _ = run(d, "graph", precision, 5, deterministic=1)
    eng = placer.stepper.eng
    torch.cuda.synchronize()
    s = eng.slot
    t = (s + 1) % 3
    state = lambda: [eng.V[t].clone(), eng.U[t].clone(), eng.G[t].clone(), eng.S[s][:8].clone(),  # noqa: E731
                     eng.metrics[s][:7].clone()]
    eng._trial(s, head=True)
    want = state()
    for buf in (eng.V[t], eng.U[t], eng.G[t]):
        buf.fill_(-1.0)
    count = {}
    for name, piece in eng.trial_pieces(s).items():
        before = C.launch_count()
        piece()
        count[name] = C.launch_count() - before
    got = state()
    assert all(torch.equal(a, b) for a, b in zip(got[:4], want[:4]))
    # the objective adds the energy, an atomic fp64 sum: its last bits vary
    assert torch.allclose(got[4], want[4], rtol=1e-12, atol=0.0)
    assert count["poisson_gemms"] == launches
    assert bench.piece_work(d, eng)["poisson_gemms"][1] == bound
    work = bench.kernel_roofline(placer, d, {}, reps=1)
    assert set(work) == set(count) and all(ms > 0 for ms, _, _ in work.values())
    eng.step()  # the engine goes on from slot s
    assert all(torch.equal(a, b) for a, b in zip(state()[:3], want[:3]))
