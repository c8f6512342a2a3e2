"""Kernels of the module path at the sizes where their tiling can go wrong: the
warp-staged folds over a CSR, pin positions through the interleaved copy, the
WA value with gamma, the preconditioner and the force in node order.  Sums keep
their order, so results equal the plain expression bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dreamplace_b200._native import C
    return C


def _csr(degrees, rng):
    start = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
    flat = rng.permutation(int(start[-1])).astype(np.int32)
    return flat, start


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# tiles of 32 segments, chunks of 128 entries: one short, exact, one over; empty segments; one long segment
DEGREES = [[0], [1], [5] * 31, [4] * 32, [4] * 33, [0, 3, 0] * 21 + [129], [128], [1000] + [2] * 63, [0] * 40,
           [7] * 4096 + [1]]


@pytest.mark.parametrize("degrees", DEGREES, ids=[str(i) for i in range(len(DEGREES))])
def test_folds_over_a_csr(C, degrees):
    rng = np.random.RandomState(len(degrees))
    flat, start = _csr(degrees, rng)
    P, S = int(start[-1]), len(degrees)
    xy = rng.uniform(-50, 50, 2 * P).astype(np.float32)
    if P:
        # pin_pos backward: sequential float sums in CSR order, 3 nodes past the last with pins
        pos = torch.zeros(2 * (S + 3), device="cuda")
        got = C.pin_pos_backward(_t(xy), pos, _t(flat), _t(start), S).cpu().numpy()
        for axis in range(2):
            want = np.zeros(S + 3, np.float32)
            for i in range(S):
                s = np.float32(0)
                for k in range(start[i], start[i + 1]):
                    s = np.float32(s + xy[axis * P + flat[k]])
                want[i] = s
            assert np.array_equal(got[axis * (S + 3):(axis + 1) * (S + 3)], want)
    # HPWL: masked and empty nets count nothing
    mask = (rng.uniform(size=S) < 0.8).astype(np.uint8) * (np.array(degrees) >= 2).astype(np.uint8)
    w = rng.uniform(0.5, 2, S).astype(np.float32)
    total = 0.0
    for i in np.nonzero(mask)[0]:
        px, py = xy[:P][flat[start[i]:start[i + 1]]], xy[P:][flat[start[i]:start[i + 1]]]
        h = np.float32(np.float32(np.float32(px.max() - px.min()) + py.max()) - py.min())
        total += float(np.float32(h * w[i]))
    if P:
        args = (_t(xy), _t(flat), _t(start), _t(w), _t(mask))
        got = C.hpwl_forward(*args)[0].item()
        assert abs(got - total) <= 1e-13 * max(total, 1.0) * max(S, 1)  # fp64 sums in two orders
        assert C.hpwl_forward_f32(*args).item() == np.float32(got)


@pytest.mark.parametrize("pins", [1, 255, (1 << 20) - 1, 1 << 20, (1 << 20) + 77])
def test_pin_positions(C, pins):
    rng = np.random.RandomState(1)
    n = 3001
    pos, off = _t(rng.uniform(0, 9e3, 2 * n).astype(np.float32)), _t(rng.uniform(-9, 9, 2 * pins).astype(np.float32))
    p2n = _t(rng.randint(0, n, pins).astype(np.int32))
    got = C.pin_pos_forward(pos, off[:pins].contiguous(), off[pins:].contiguous(), p2n)
    i = p2n.long()
    assert torch.equal(got, torch.cat([off[:pins] + pos[i], off[pins:] + pos[n + i]]))


def test_wa_value_with_gamma_and_preconditioner(C):
    from dreamplace_b200.weighted_average_wirelength import PinLanes
    rng = np.random.RandomState(3)
    flat, start = _csr([2, 3, 5, 9, 40, 8, 1] * 37, rng)
    P, S = int(start[-1]), len(start) - 1
    lanes = PinLanes(_t(flat), _t(start))
    pos = _t(rng.uniform(0, 900, 2 * P).astype(np.float32))
    w, mask, gamma = _t(rng.uniform(0.5, 2, S).astype(np.float32)), torch.ones(S, dtype=torch.uint8, device="cuda"), \
        torch.tensor(7.3, device="cuda")
    plan = (lanes.group_deg, lanes.group_base, lanes.group_net, lanes.ln_pin, w, mask)
    a, b = (torch.zeros(2 * lanes.num_slots, device="cuda") for _ in range(2))
    wl64 = torch.empty(1280, dtype=torch.float64, device="cuda")
    C.wa_pins_forward(pos, *plan, (1.0 / gamma).reshape(1), wl64, a)
    value = C.wa_pins_value(pos, *plan, gamma, b)
    assert torch.equal(a, b) and value.item() == wl64[0].float().item()
    for n in (1, 257, 5000):
        g, pws, area = (_t(rng.uniform(0, 3, k).astype(np.float32)) for k in (2 * n, n, n))
        lam = torch.tensor([0.37], device="cuda")
        want = g.view(2, n) / (pws + 1.0 * lam * area).clamp(min=1.0)
        assert C.precondition(g, pws, area, lam, 1.0)
        assert torch.equal(g, want.reshape(-1))


@pytest.mark.parametrize("nm,nf,fixed", [(1, 0, 0), (300, 0, 7), (513, 200, 3), (0, 90, 5)])
def test_force_in_node_order(C, nm, nf, fixed):
    rng = np.random.RandomState(nm)
    n, count, b = nm + fixed + nf, nm + nf, 64
    order = _t(np.concatenate([rng.permutation(nm), n - nf + rng.permutation(nf)]).astype(np.int32))
    xy = _t(rng.uniform(0, 60, 2 * count).astype(np.float32))
    rec = _t(np.tile(np.array([1.5, 2.5, -0.1, 0.2], np.float32), count))
    ratio = _t(rng.uniform(0.5, 1, count).astype(np.float32))
    ex, ey = (_t(rng.normal(size=b * b).astype(np.float32)) for _ in range(2))
    g = torch.tensor([0.7], device="cuda")
    force_o = torch.empty(2 * count, device="cuda")
    C.electric_force_ordered(g, ex, ey, xy, rec, ratio, count, 0.0, 0.0, 1.0, 1.0, b, b, -1.0, force_o)
    want = C.scatter_pairs_to_nodes(force_o, order, count, n)
    got = C.electric_force_nodes(g, ex, ey, xy, order, rec, ratio, nm, nf, n, 0.0, 0.0, 1.0, 1.0, b, b, -1.0)
    assert torch.equal(got, want)


def test_precondition_takes_what_the_tensor_expression_takes(C):
    """Operands the kernel has no form for (a strided or fp64 node area, a pin
    weight sum of another type, a lambda on the host) go through the tensor
    expression; both count as a change of the gradient in place."""
    from types import SimpleNamespace
    from dreamplace_b200.place_obj import PreconditionOp
    rng = np.random.RandomState(5)
    n = 777
    pws, area, g0 = (_t(rng.uniform(0, 3, k).astype(np.float32)) for k in (n, n, 2 * n))
    lam = torch.tensor([0.37], device="cuda")
    wide = torch.zeros(2 * n, device="cuda")
    wide[::2] = area
    want = (g0.view(2, n) / (pws + 1.0 * lam * area).clamp(min=1.0)).reshape(-1)
    forms = {"kernel": (pws, area, lam, 0), "strided area": (pws, wide[::2], lam, 0),
             "fp64 area": (pws, area.double(), lam, 1e-6), "fp64 pin weights": (pws.double(), area, lam, 1e-6),
             "strided pin weights": (torch.stack([pws, pws], 1)[:, 0], area, lam, 0),
             "host lambda": (pws, area, torch.tensor(0.37), 0)}
    for name, (p, a, w, tol) in forms.items():
        op = PreconditionOp(SimpleNamespace(num_nodes=n), SimpleNamespace(node_areas=a, net_weights=None),
                            SimpleNamespace(pws_op=lambda _: p))
        g = g0.clone()
        version = g._version
        assert op(g, w) is g and op.iteration == 1
        assert g._version > version, name
        assert float((g - want).abs().max()) <= tol * float(want.abs().max()), name


def test_folds_read_only_the_segments_they_are_given(C):
    """Segment i is [start[i], start[i + 1]), empty where the second is not above
    the first, also for a start array that does not ascend; and a masked net's
    entries are not read, however many it has."""
    rng = np.random.RandomState(11)
    P, n = 640, 45
    xy = rng.uniform(-50, 50, 2 * P).astype(np.float32)
    flat = rng.permutation(P).astype(np.int32)
    for start in (np.array([5, 8, 0, 5], np.int32), rng.randint(0, P, n + 1).astype(np.int32)):
        S = len(start) - 1
        got = C.pin_pos_backward(_t(xy), torch.zeros(2 * S, device="cuda"), _t(flat), _t(start), S).cpu().numpy()
        want, total = np.zeros(2 * S, np.float32), 0.0
        mask = start[1:] > start[:-1]
        for i in range(S):
            px, py = (xy[a + flat[start[i]:max(start[i + 1], start[i])]] for a in (0, P))
            for k in range(len(px)):
                want[i] = np.float32(want[i] + px[k])
                want[S + i] = np.float32(want[S + i] + py[k])
            if mask[i]:
                total += float(np.float32(np.float32(np.float32(px.max() - px.min()) + py.max()) - py.min()))
        assert np.array_equal(got, want)
        h = C.hpwl_forward(_t(xy), _t(flat), _t(start), torch.empty(0, device="cuda"), _t(mask.astype(np.uint8)))
        assert abs(h[0].item() - total) <= 1e-13 * S * max(total, 1.0)  # fp64 sums in two orders
    # one masked net of 8M entries among small ones: a warp that walks them needs
    # 64k dependent rounds of L2 reads (over 30 ms), the rest of the call microseconds
    big = 8 << 20
    start = np.concatenate([np.arange(0, 80, 4), [big], big + np.arange(4, 44, 4)]).astype(np.int32)
    flat = torch.arange(int(start[-1]), dtype=torch.int32, device="cuda") % 1000
    mask = np.diff(start) < 100
    args = (_t(rng.uniform(0, 9, 2 * int(start[-1])).astype(np.float32)), flat, _t(start),
            torch.empty(0, device="cuda"), _t(mask.astype(np.uint8)))
    C.hpwl_forward(*args)
    t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    t0.record()
    C.hpwl_forward(*args)
    t1.record()
    t1.synchronize()
    assert t0.elapsed_time(t1) < 5.0


def test_trial_start_zeroes_large_maps_of_few_nodes(C):
    """The zeroed ranges are whole words, ragged ones included, and take the whole
    GPU also where the nodes need one block only: 256 MB are 45 us at the HBM
    rate, and over 10 ms from a block or two."""
    n = 100
    nodes = [torch.rand(2 * n, device="cuda") for _ in range(6)]
    size = torch.ones(n, device="cuda")
    state = torch.zeros(8 + 2 * 1280, dtype=torch.float64, device="cuda")
    big = torch.ones((64 << 20) + 3, dtype=torch.int32, device="cuda")
    small = torch.ones(5, device="cuda")
    cells = torch.ones(4, dtype=torch.float64, device="cuda")

    def start():
        C.trial_start(None, [1.0] * 5, None, *nodes, state, size, size, 0.0, 0.0, 10.0, 10.0, n, 0, None, None,
                      [big, small], cells[0:1], cells[2:3])
    start()
    assert not big.any() and not small.any() and cells.tolist() == [0.0, 1.0, 0.0, 1.0]
    t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    t0.record()
    start()
    t1.record()
    t1.synchronize()
    assert t0.elapsed_time(t1) < 2.0


def test_backward_serves_the_cells_of_its_forward(C):
    """The filler count is an attribute that a program may set between calls (a
    visiting order is kept for each): a backward still writes the force of the
    cells that its own forward scattered."""
    from dreamplace_b200 import synthetic
    from dreamplace_b200.electric_potential import ElectricPotential
    d = synthetic.scaled(2000, num_bins=64, seed=5)
    centers = [_t(d.bin_centers(lo, hi, size)) for lo, hi, size in ((d.xl, d.xh, d.bin_size_x),
                                                                    (d.yl, d.yh, d.bin_size_y))]
    m = d.num_movable_nodes
    op = ElectricPotential(_t(d.node_size_x), _t(d.node_size_y), *centers, d.target_density, d.xl, d.yl, d.xh, d.yh,
                           d.bin_size_x, d.bin_size_y, m, d.num_terminals, d.num_filler_nodes, 0, True,
                           _t(np.argsort(d.node_size_x[:m], kind="stable").astype(np.int32)), precision="fp32")
    pos = _t(np.random.RandomState(2).uniform(0, d.xh * 0.9, 2 * d.num_nodes).astype(np.float32)).requires_grad_(True)
    want, = torch.autograd.grad(op(pos), pos)
    energy, fillers = op(pos), op.num_filler_nodes
    op.num_filler_nodes = 0
    got, = torch.autograd.grad(energy, pos)
    assert fillers > 0 and torch.equal(got, want)
