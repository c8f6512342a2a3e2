"""Cases that stand for the work users of dreamplace_b200 have it do, for timing it.

The framework runs one path, global placement, at three levels that programs
call: iterations of the graph engine (``GPEngine.step``), one evaluation of the
objective and its gradient through the drop-in modules (``PlaceObj``), and the
modules themselves (``ElectricPotential``, ``WeightedAverageWirelength``,
``HPWL`` / ``ElectricOverflow``, the Poisson solve and the 2-D transforms).
Designs follow the synthetic generator's shapes: row height 12, log-uniform
widths, nets of degree 2 + Geometric(0.45), 70% of a net's pins from a
500-cell window, 70% utilisation; they are made on the GPU so that many states
can be prepared quickly.  ``spread`` is how far placement has come: cells near
the die centre early (0.01 .. 0.1), over the whole die late (1).
"""
import functools
import math

import numpy as np
import torch

from dreamplace_b200 import dct2_fft2, electric_potential, synthetic
from dreamplace_b200.nonlinear_place import NonLinearPlace
from dreamplace_b200.params import Params
from dreamplace_b200.place_obj import PlaceDataCollection, PlaceObj, build_ops
from dreamplace_b200.placement_ops import HPWL, PinPos
from dreamplace_b200.weighted_average_wirelength import WeightedAverageWirelength

DEVICE = "cuda"
ROW = 12.0
PRECISIONS = ("split_bf16", "fp32")


def listed():
    return [
        # placement of a small block: the batch of small designs and the 10k-cell test design; bound by launches
        {"name": "gp 10k cells", "kind": "gp", "cells": 10000, "bins": 128, "spread": 0.05, "iterations": 32,
         "precision": "split_bf16", "deterministic": True},
        # a mid-size block late in placement, an odd number of cells, fp32 density atomics
        {"name": "gp 200k cells", "kind": "gp", "cells": 200003, "bins": 512, "spread": 1.0, "iterations": 16,
         "precision": "split_bf16", "deterministic": False},
        # the headline design: iterations of the 2.1M-cell placement
        {"name": "gp 2.1M cells", "kind": "gp", "cells": 2100000, "bins": 1024, "spread": 0.5, "iterations": 8,
         "precision": "split_bf16", "deterministic": False},
        # one objective + gradient evaluation of the autograd loop (the reference's own loop over the drop-in modules)
        {"name": "objective 50k cells", "kind": "objective", "cells": 50000, "bins": 256, "spread": 0.5,
         "precision": "split_bf16", "deterministic": False},
        # the density operator alone, forward and backward: smallest, ordinary on a ragged grid, largest
        {"name": "density 2k cells", "kind": "density", "cells": 2000, "bins": 64, "spread": 1.0,
         "precision": "split_bf16", "deterministic": True},
        {"name": "density 130k cells ragged", "kind": "density", "cells": 130001, "bins": 360, "spread": 0.3,
         "precision": "fp32", "deterministic": True},
        {"name": "density 2.1M cells", "kind": "density", "cells": 2100000, "bins": 1024, "spread": 1.0,
         "precision": "split_bf16", "deterministic": False},
        # the wirelength operator alone, pin positions to node gradient
        {"name": "wirelength 10k cells", "kind": "wirelength", "cells": 10007, "spread": 0.1},
        {"name": "wirelength 2.1M cells", "kind": "wirelength", "cells": 2100000, "spread": 1.0},
        # the per-iteration evaluation of a loop outside the engine: HPWL and density overflow
        {"name": "metrics 500k cells", "kind": "metrics", "cells": 500009, "bins": 512, "spread": 1.0,
         "deterministic": True},
        # the four 2-D transforms as modules
        {"name": "transforms 512", "kind": "transforms", "bins": 512, "bins_y": 512, "precision": "fp32"},
        # the Poisson solve of the largest grid
        {"name": "poisson 4096", "kind": "poisson", "bins": 4096, "bins_y": 4096, "precision": "split_bf16"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gp", "density", "density", "wirelength", "objective", "metrics", "transforms", "poisson"])
    case = {"kind": kind}
    if kind in ("transforms", "poisson"):
        # grids are powers of two, as placers choose them, or ragged (sides a multiple of 8, as bf16 operands need)
        for side in ("bins", "bins_y"):
            n = _log_uniform(rng, 64, 2048)
            case[side] = 2 ** round(math.log2(n)) if rng.random() < 0.7 else max(8 * (n // 8), 64)
        case["precision"] = rng.choice(PRECISIONS + (("tf32", "bf16") if kind == "transforms" else ()))
        return case
    case["cells"] = _log_uniform(rng, 2000, 1500000)
    case["spread"] = round(rng.choice([rng.uniform(0.02, 0.2), rng.uniform(0.2, 1.0), 1.0]), 3)
    if kind == "wirelength":
        return case
    side = 2 ** round(math.log2(math.sqrt(case["cells"])))
    case["bins"] = min(max(side, 64), 1024)
    if kind in ("density", "metrics") and rng.random() < 0.3:
        case["bins"] = 8 * rng.randint(8, 100)
    case["deterministic"] = rng.random() < 0.5
    if kind == "metrics":
        return case
    case["precision"] = rng.choice(PRECISIONS)
    if kind == "gp":
        case["iterations"] = 8
        case["cells"] = min(case["cells"], 600000)
    return case


# ---------------------------------------------------------------- designs
def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device=DEVICE, dtype=torch.float64)


def _design(cells, bins, gen):
    """A design of the synthetic generator's shapes (dreamplace_b200.synthetic.Design), made on the GPU."""
    m = cells
    macros = max(round(m * 1000 / 2.1e6), 1)
    width = torch.exp(_rand(gen, m) * math.log(40.0)).round().clamp(min=1.0)
    mac = torch.floor(60 + 241 * _rand(gen, 2, macros))
    mov_area = float(width.sum()) * ROW
    mac_area = float((mac[0] * mac[1]).sum())
    side = math.ceil(math.sqrt(mov_area / 0.7 + mac_area) / ROW) * ROW
    # macros apart from one another: one per tile of a square tiling
    tiles = math.ceil(math.sqrt(macros))
    pitch = side / tiles
    at = torch.arange(macros, device=DEVICE)
    corner = torch.stack([at // tiles, at % tiles]) * pitch
    mac_xy = (corner + _rand(gen, 2, macros) * (pitch - mac).clamp(min=0.0)).floor()
    physical = m + macros
    # fillers: as many as PlaceDB's mean-width fillers would be, filling the free space exactly
    fillers = round(0.47 * m)
    filler_w = (side * side - mac_area - mov_area) / (fillers * ROW)
    size_x = torch.cat([width, mac[0], torch.full((fillers,), filler_w, device=DEVICE, dtype=torch.float64)]).float()
    size_y = torch.cat([torch.full((m,), ROW, device=DEVICE, dtype=torch.float64), mac[1],
                        torch.full((fillers,), ROW, device=DEVICE, dtype=torch.float64)]).float()
    # nets
    nets = round(m * 2.2 / 2.1)
    degree = (2 + torch.floor(torch.log(1 - _rand(gen, nets)) / math.log(1 - 0.45))).clamp(max=50).long()
    start = torch.zeros(nets + 1, device=DEVICE, dtype=torch.int64)
    torch.cumsum(degree, 0, out=start[1:])
    pins = int(start[-1])
    net_of_pin = torch.repeat_interleave(torch.arange(nets, device=DEVICE), degree)
    window = min(500, physical)
    centre = torch.floor(_rand(gen, nets) * (physical - window + 1)).long()
    near = centre[net_of_pin] + torch.floor(_rand(gen, pins) * window).long()
    anywhere = torch.floor(_rand(gen, pins) * physical).long()
    pin2node = torch.where(_rand(gen, pins) < 0.7, near, anywhere)
    offset = (_rand(gen, 2, pins) * torch.stack([size_x, size_y])[:, pin2node].double()).float()
    node2pin = torch.argsort(pin2node, stable=True)
    node_start = torch.zeros(physical + 1, device=DEVICE, dtype=torch.int64)
    torch.cumsum(torch.bincount(pin2node, minlength=physical), 0, out=node_start[1:])
    f32 = lambda t: t.float().cpu().numpy()  # noqa: E731
    i32 = lambda t: t.int().cpu().numpy()  # noqa: E731
    node_x = torch.cat([torch.zeros(m, device=DEVICE, dtype=torch.float64), mac_xy[0]])
    node_y = torch.cat([torch.zeros(m, device=DEVICE, dtype=torch.float64), mac_xy[1]])
    return synthetic.Design(
        name="cells%d" % m, xl=0.0, yl=0.0, xh=float(side), yh=float(side), row_height=ROW, site_width=1.0,
        num_movable_nodes=m, num_terminals=macros, num_filler_nodes=fillers, node_size_x=f32(size_x),
        node_size_y=f32(size_y), node_x=f32(node_x), node_y=f32(node_y), pin_offset_x=f32(offset[0]),
        pin_offset_y=f32(offset[1]), pin2node_map=i32(pin2node), pin2net_map=i32(net_of_pin),
        flat_net2pin_map=np.arange(pins, dtype=np.int32), flat_net2pin_start_map=i32(start),
        flat_node2pin_map=i32(node2pin), flat_node2pin_start_map=i32(node_start),
        net_weights=np.ones(nets, dtype=np.float32), num_bins_x=bins, num_bins_y=bins, target_density=1.0,
        total_movable_node_area=mov_area, total_fixed_node_area=mac_area,
        total_space_area=side * side - mac_area, movable_macro_mask=np.zeros(m, dtype=bool), seed=0)


def _positions(d, spread, gen):
    """[x(n) | y(n)]: movable cells along a serpentine of strips (cells near in
    index are near in space, as their nets draw them together), scaled towards
    the die centre by ``spread``, fixed cells at their places, fillers anywhere."""
    m, n, nf = d.num_movable_nodes, d.num_nodes, d.num_filler_nodes
    strips = max(round(math.sqrt(m / 200)), 1)
    t = torch.arange(m, device=DEVICE, dtype=torch.float64) * (strips / m)
    strip = torch.floor(t)
    along = t - strip
    along = torch.where(strip % 2 == 1, 1 - along, along)
    x = along * d.width + torch.randn(m, generator=gen, device=DEVICE, dtype=torch.float64) * (d.width / strips)
    y = (strip + _rand(gen, m)) * (d.height / strips)
    xy = torch.stack([x, y])
    xy = d.width / 2 + spread * (xy - d.width / 2)
    size = torch.from_numpy(np.stack([d.node_size_x, d.node_size_y])).to(DEVICE).double()
    fixed = torch.from_numpy(np.stack([d.node_x, d.node_y])).to(DEVICE).double()[:, m:]
    fill = _rand(gen, 2, nf) * d.width
    pos = torch.cat([xy, fixed, fill], dim=1)
    free = torch.ones(n, dtype=torch.bool, device=DEVICE)
    free[m:n - nf] = False
    pos = torch.where(free, torch.minimum(pos.clamp(min=0.0), d.width - size), pos)
    return pos.reshape(-1).float().contiguous()


@functools.lru_cache(maxsize=2)
def _inputs(cells, bins, spread, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    d = _design(cells, bins, gen)
    return d, _positions(d, spread, gen)


# ---------------------------------------------------------------- states
def _params(case):
    return Params(target_density=1.0, stop_overflow=0.07, dct_precision=case.get("precision", "split_bf16"),
                  deterministic_flag=int(case.get("deterministic", False)))


def _pin_pos(d, data):
    return PinPos(data.pin_offset_x, data.pin_offset_y, data.pin2node_map, data.flat_node2pin_map,
                  data.flat_node2pin_start_map, d.num_physical_nodes)


def _bin_geometry(d, bins):
    size = d.width / bins
    centers = torch.from_numpy(d.bin_centers(d.xl, d.xh, size)).to(DEVICE)
    return dict(bin_center_x=centers, bin_center_y=centers, target_density=d.target_density, xl=d.xl, yl=d.yl,
                xh=d.xh, yh=d.yh, bin_size_x=size, bin_size_y=size, num_movable_nodes=d.num_movable_nodes,
                num_terminals=d.num_terminals)


def _map(case, seed):
    """A normalised density map: clusters of cells over a noisy floor."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    M, N = case["bins"], case["bins_y"]
    u = torch.arange(M, device=DEVICE, dtype=torch.float64)[:, None] / M
    v = torch.arange(N, device=DEVICE, dtype=torch.float64)[None, :] / N
    rho = 0.6 + 0.3 * _rand(gen, M, N)
    for a, b, s, h in _rand(gen, 12, 4).tolist():
        rho += (0.5 + 2 * h) * torch.exp(-((u - a) ** 2 + (v - b) ** 2) / (2 * (0.02 + 0.1 * s) ** 2))
    return rho.float().contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("transforms", "poisson"):
        state = {"case": case, "map": _map(case, seed)}
        if kind == "transforms":
            M, N = case["bins"], case["bins_y"]
            expk = [dct2_fft2.get_exact_expk(n, torch.float32, DEVICE) for n in (M, N)]
            state["modules"] = [cls(expk[0], expk[1], precision=case["precision"]) for cls in
                                (dct2_fft2.DCT2, dct2_fft2.IDCT2, dct2_fft2.IDCT_IDXST, dct2_fft2.IDXST_IDCT)]
        return state
    bins = case.get("bins", 64)
    d, pos = _inputs(case["cells"], bins, case["spread"], seed)
    params = _params(case)
    state = {"case": case, "design": d, "pos": torch.nn.Parameter(pos.clone())}
    if kind == "gp":
        placer = NonLinearPlace(params, d, DEVICE)
        placer.pos[0].data.copy_(pos)
        placer(params, d, max_iterations=3)
        engine = placer.stepper.eng
        saved = engine.state_dict()
        # the checkpoint stays on the GPU, as a program that tries several continuations keeps it
        state["engine"] = engine
        state["saved"] = {k: [t.to(DEVICE) for t in v] if isinstance(v, list) else
                          v.to(DEVICE) if isinstance(v, torch.Tensor) else v for k, v in saved.items()}
        return state
    data = PlaceDataCollection(torch.nn.ParameterList([state["pos"]]), params, d, torch.device(DEVICE))
    if kind == "objective":
        stage = dict(params.global_place_stages[0])
        state["model"] = PlaceObj(1e-3, params, d, data, build_ops(params, d, data), stage).to(DEVICE)
    elif kind == "density":
        state["op"] = electric_potential.ElectricPotential(
            data.node_size_x, data.node_size_y, num_filler_nodes=d.num_filler_nodes, padding=0,
            deterministic_flag=case["deterministic"], sorted_node_map=data.sorted_node_map,
            precision=case["precision"], **_bin_geometry(d, bins))
    elif kind == "wirelength":
        state["pin_pos"] = _pin_pos(d, data)
        state["op"] = WeightedAverageWirelength(
            flat_netpin=data.flat_net2pin_map, netpin_start=data.flat_net2pin_start_map, pin2net_map=data.pin2net_map,
            net_weights=data.net_weights, net_mask=data.net_mask_ignore_large_degrees,
            pin_mask=data.pin_mask_ignore_fixed_macros, gamma=_gamma(case, d), algorithm="merged")
    else:  # metrics
        state["pin_pos"] = _pin_pos(d, data)
        state["hpwl"] = HPWL(data.flat_net2pin_map, data.flat_net2pin_start_map, data.pin2net_map, data.net_weights,
                             data.net_mask_all)
        state["op"] = electric_potential.ElectricOverflow(
            data.node_size_x, data.node_size_y, num_filler_nodes=0, padding=0,
            deterministic_flag=case["deterministic"], sorted_node_map=data.sorted_node_map,
            **_bin_geometry(d, bins))
    return state


def _gamma(case, d):
    """The schedule's gamma between early and late placement: 4 bin sizes of a grid of about one cell a bin."""
    return torch.tensor(8.0 * d.width / math.sqrt(case["cells"]), dtype=torch.float32, device=DEVICE)


def run(state):
    kind = state["case"]["kind"]
    if kind == "gp":
        engine = state["engine"]
        engine.load_state_dict(state["saved"])
        history = [engine.step() for _ in range(state["case"]["iterations"])]
        return {"pos": engine.current_position(), "grad": engine.G[engine.slot],
                "hpwl": [h[0] for h in history[-4:]], "overflow": [h[1] for h in history[-4:]]}
    if kind == "transforms":
        return [op(state["map"]) for op in state["modules"]]
    if kind == "poisson":
        ex, ey, energy = electric_potential.poisson_solve(state["map"], 1.0, 1.0, state["case"]["precision"])
        return {"field_x": ex, "field_y": ey, "energy": energy}
    pos = state["pos"]
    if kind == "metrics":
        with torch.no_grad():
            overflow, max_density = state["op"](pos)
            return {"hpwl": state["hpwl"](state["pin_pos"](pos)), "overflow": overflow, "max_density": max_density}
    if kind == "objective":
        obj, grad = state["model"].obj_and_grad_fn(pos)
        return {"objective": obj, "grad": grad}
    pos.grad = None
    value = state["op"](pos) if kind == "density" else state["op"](state["pin_pos"](pos))
    value.backward()
    return {"value": value, "grad": pos.grad}


# ---------------------------------------------------------------- what a pass cannot do without
def _sizes(case):
    """(nodes, scattered cells, pins, nets, bins) of a case, from the generator's means."""
    m = case["cells"]
    n = 1.47 * m
    return n, n, 3.22 * m * 2.2 / 2.1, m * 2.2 / 2.1, case.get("bins", 0) ** 2


def _solve_flops(M, N, transforms):
    """Fast transforms of real M x N maps: 2.5 MN log2(MN) operations each."""
    return transforms * 2.5 * M * N * math.log2(M * N)


def work(case):
    kind = case["kind"]
    if kind == "transforms":
        mn = case["bins"] * case["bins_y"]
        return {"bytes": 4 * (4 + 1) * mn, "flops": _solve_flops(case["bins"], case["bins_y"], 4)}
    if kind == "poisson":
        mn = case["bins"] * case["bins_y"]
        return {"bytes": 4 * 3 * mn, "flops": _solve_flops(case["bins"], case["bins_y"], 3)}
    n, ns, pins, nets, bins = _sizes(case)
    # density: position, size and gradient of each cell, the initial map; 9 bins a cell each way
    density = {"bytes": 24 * ns + 4 * bins, "flops": 9 * 12 * ns}
    if bins:
        density["flops"] += _solve_flops(case["bins"], case["bins"], 3)
    # wirelength: node and pin offset (12 B) of each pin, net starts, weights and masks, position and gradient of each node
    wirelength = {"bytes": 12 * pins + 9 * nets + 16 * n, "flops": 60 * pins}
    if kind == "density":
        return density
    if kind == "wirelength":
        return wirelength
    if kind == "metrics":
        return {"bytes": 16 * case["cells"] + 4 * bins + 12 * pins + 9 * nets, "flops": 9 * 6 * case["cells"] + 8 * pins}
    both = {k: density[k] + wirelength[k] - (16 * n if k == "bytes" else 0) for k in ("bytes", "flops")}
    both["bytes"] += 8 * n  # the preconditioner's pin weights and areas
    if kind == "objective":
        return both
    # an iteration also reads v, g, u and writes u', v', g' (about 1.05 evaluations each)
    return {"bytes": case["iterations"] * (both["bytes"] + 32 * n), "flops": case["iterations"] * both["flops"]}


def tolerance(case):
    """About four times what fp32 against split-BF16 solves, fp32 atomics against
    fixed-point sums, or either against 64 bits were seen to differ by."""
    kind, precision = case["kind"], case.get("precision", "fp32")
    if kind in ("transforms", "poisson"):
        # seen: fp32 1e-6 (4e-6 at 4096^2), hi + lo bf16 8e-6 (5e-5 at 4096^2), tf32 1.4e-3, bf16 2.9e-3
        return {"rel": {"fp32": 1.6e-5, "split_bf16": 2e-4, "tf32": 6e-3, "bf16": 1.2e-2}[precision]}
    if kind == "wirelength":
        return {"rel": 2e-5, "max": 4e-4}  # seen: 4e-6, 9e-5
    if kind == "metrics":
        return {"rel": 1.2e-4}  # seen: the overflow 3e-5 from 64 bits, by the rounding of positions far from the origin
    if kind in ("density", "objective"):
        # the field of a nearly even density is a small difference, and positions lose bits as bins get smaller
        # beside the die: seen 6e-6 at 64 bins, 2e-5 at 256, 2.6e-4 at 792, 4e-4 to 2e-3 at 1024
        rel = max(5e-5, 4e-9 * case["bins"] ** 2)
        return {"rel": rel, "max": 10 * rel}
    # a change of rounding travels through the iterations that follow: seen 4e-4 and 8e-2
    return {"rel": 2e-3, "max": 0.4}


# ---------------------------------------------------------------- the same in 64 bits
def _cos_matrix(n):
    k = torch.arange(n, dtype=torch.float64, device=DEVICE)
    return torch.cos(math.pi * k[:, None] * (2 * k[None, :] + 1) / (2 * n))


def _icos_matrix(n):
    m = _cos_matrix(n).T.clone()
    m[:, 0] *= 0.5
    return m


def _isin_matrix(n):
    k = torch.arange(n, dtype=torch.float64, device=DEVICE)
    return torch.sin(math.pi * k[None, :] * (2 * k[:, None] + 1) / (2 * n))


def _solve64(rho, aspect=1.0):
    M, N = rho.shape
    a = 4.0 / (M * N) * (_cos_matrix(M) @ rho @ _cos_matrix(N).T)
    wu = (torch.arange(M, dtype=torch.float64, device=DEVICE) * (2 * math.pi / M))[:, None]
    wv = (torch.arange(N, dtype=torch.float64, device=DEVICE) * (2 * math.pi / N) * aspect)[None, :]
    sq = wu ** 2 + wv ** 2
    sq[0, 0] = 1.0
    inv = 1.0 / sq
    inv[0, 0] = 0.0
    ex = 4.0 * (_isin_matrix(M) @ (a * wu * inv / 2) @ _icos_matrix(N).T)
    ey = 4.0 * (_icos_matrix(M) @ (a * wv * inv / 2) @ _isin_matrix(N).T)
    phi = 4.0 * (_icos_matrix(M) @ (a * inv) @ _icos_matrix(N).T)
    return ex, ey, (phi * rho).sum()


def _windows(d, pos, bins, cells):
    """(bin indices, x overlap, y overlap) of each stretched cell with its window of bins, in 64 bits."""
    n, m = d.num_nodes, d.num_movable_nodes
    size = d.width / bins
    node = torch.cat([torch.arange(m, device=DEVICE), torch.arange(n - (cells - m), n, device=DEVICE)])
    out = [node]
    for axis, sizes in enumerate((d.node_size_x, d.node_size_y)):
        s = torch.from_numpy(sizes).to(DEVICE).double()[node]
        stretched = s.clamp(min=math.sqrt(2) * size)
        lo = pos[axis * n + node] + (s - stretched) / 2
        first = torch.floor(lo / size).long()
        span = int(math.ceil(float(stretched.max()) / size)) + 1
        bin_ = first[:, None] + torch.arange(span, device=DEVICE)[None, :]
        overlap = torch.minimum(lo[:, None] + stretched[:, None], (bin_ + 1) * size) - torch.maximum(lo[:, None], bin_ * size)
        overlap = torch.where((bin_ >= 0) & (bin_ < bins), overlap.clamp(min=0.0), torch.zeros_like(overlap))
        out += [bin_.clamp(0, bins - 1), overlap, s / stretched]
    return out


def _density64(d, pos, bins, cells):
    """Density map (area) of the fixed cells and the first ``cells`` movable and filler cells."""
    m, n, size = d.num_movable_nodes, d.num_nodes, d.width / bins
    edge = torch.arange(bins + 1, dtype=torch.float64, device=DEVICE) * size
    sides = []
    for axis, sizes in enumerate((d.node_size_x, d.node_size_y)):
        lo = pos[axis * n + m:axis * n + m + d.num_terminals]
        hi = lo + torch.from_numpy(sizes[m:m + d.num_terminals]).to(DEVICE).double()
        sides.append((torch.minimum(hi[:, None], edge[1:]) - torch.maximum(lo[:, None], edge[:-1])).clamp(min=0.0))
    out = (sides[0].T @ sides[1]).clamp(max=size * size) * d.target_density
    w = _windows(d, pos, bins, cells)
    _, bx, ox, rx, by, oy, ry = w
    flat = out.reshape(-1)
    for i in range(bx.shape[1]):
        for j in range(by.shape[1]):
            flat.index_add_(0, bx[:, i] * bins + by[:, j], ox[:, i] * oy[:, j] * (rx * ry))
    return flat.view(bins, bins), w


def _density_grad64(d, pos, bins):
    """(energy, gradient [x | y]) of the electrostatic energy: the field force over each stretched cell."""
    cells = d.num_movable_nodes + d.num_filler_nodes
    density, w = _density64(d, pos, bins, cells)
    size = d.width / bins
    ex, ey, energy = _solve64(density / (size * size))
    node, bx, ox, rx, by, oy, ry = w
    grad = torch.zeros(2, d.num_nodes, dtype=torch.float64, device=DEVICE)
    for i in range(bx.shape[1]):
        for j in range(by.shape[1]):
            area = ox[:, i] * oy[:, j] * (rx * ry)
            at = bx[:, i] * bins + by[:, j]
            grad[0, node] -= area * ex.reshape(-1)[at]
            grad[1, node] -= area * ey.reshape(-1)[at]
    return energy, grad.reshape(-1)


def _pins64(d, pos):
    node = torch.from_numpy(d.pin2node_map).to(DEVICE).long()
    x = pos[node] + torch.from_numpy(d.pin_offset_x).to(DEVICE).double()
    y = pos[d.num_nodes + node] + torch.from_numpy(d.pin_offset_y).to(DEVICE).double()
    return node, x, y


def _wirelength64(d, pos, gamma):
    """(weighted-average wirelength, its gradient on the movable nodes)."""
    leaf = pos.clone().requires_grad_(True)
    node, *pins = _pins64(d, leaf)
    fixed = node >= d.num_movable_nodes
    net = torch.from_numpy(d.pin2net_map).to(DEVICE).long()
    degree = torch.bincount(net, minlength=d.num_nets)
    live = (degree >= 2) & (degree < 100)
    total = torch.zeros((), dtype=torch.float64, device=DEVICE)
    for p in pins:
        p = torch.where(fixed, p.detach(), p)
        for sign in (1.0, -1.0):
            top = torch.full((d.num_nets,), -math.inf, dtype=torch.float64, device=DEVICE)
            top.scatter_reduce_(0, net, (sign * p).detach(), "amax")
            e = torch.exp((sign * p - top[net]) / gamma)
            zero = torch.zeros(d.num_nets, dtype=torch.float64, device=DEVICE)
            wa = zero.index_add(0, net, p * e) / zero.index_add(0, net, e)
            total = total + sign * torch.where(live, wa, torch.zeros_like(wa)).sum()
    total.backward()
    return total.detach(), leaf.grad


def exact(case, seed):
    kind = case["kind"]
    if kind == "gp":
        return None  # a trajectory: its steps are the other kinds
    if kind in ("transforms", "poisson"):
        rho = _map(case, seed).double()
        if kind == "poisson":
            ex, ey, energy = _solve64(rho)
            return {"field_x": ex, "field_y": ey, "energy": energy.reshape(1)}
        M, N = rho.shape
        pairs = [(_cos_matrix(M), _cos_matrix(N), 4.0 / (M * N)), (_icos_matrix(M), _icos_matrix(N), 4.0),
                 (_icos_matrix(M), _isin_matrix(N), 4.0), (_isin_matrix(M), _icos_matrix(N), 4.0)]
        return [s * (a @ rho @ b.T) for a, b, s in pairs]
    bins = case.get("bins", 64)
    d, pos = _inputs(case["cells"], bins, case["spread"], seed)
    pos = pos.double()
    if kind == "density":
        energy, grad = _density_grad64(d, pos, bins)
        return {"value": energy, "grad": grad}
    if kind == "wirelength":
        value, grad = _wirelength64(d, pos, float(_gamma(case, d)))
        return {"value": value, "grad": grad}
    if kind == "metrics":
        _, x, y = _pins64(d, pos)
        net = torch.from_numpy(d.pin2net_map).to(DEVICE).long()
        hpwl = torch.zeros((), dtype=torch.float64, device=DEVICE)
        for p in (x, y):
            for sign in (1.0, -1.0):
                top = torch.full((d.num_nets,), -math.inf, dtype=torch.float64, device=DEVICE)
                hpwl = hpwl + top.scatter_reduce_(0, net, sign * p, "amax").sum()
        area = (d.width / bins) ** 2
        density, _ = _density64(d, pos, bins, d.num_movable_nodes)
        over = (density - d.target_density * area).clamp(min=0.0).sum()
        return {"hpwl": hpwl, "overflow": over.reshape(1), "max_density": (density.max() / area).reshape(1)}
    # objective: wirelength + 1e-3 density, the gradient over max(1, pin weights + 1e-3 area)
    lam = float(np.float32(1e-3))
    gamma = float(torch.tensor(10 * 4.0 * 2 * d.width / bins, dtype=torch.float32))
    energy, grad = _density_grad64(d, pos, bins)
    wl, wl_grad = _wirelength64(d, pos, gamma)
    weight = torch.zeros(d.num_nodes, dtype=torch.float64, device=DEVICE)
    node = torch.from_numpy(d.pin2node_map).to(DEVICE).long()
    weight.index_add_(0, node, torch.ones(node.numel(), dtype=torch.float64, device=DEVICE))
    area = torch.from_numpy(d.node_size_x).to(DEVICE).double() * torch.from_numpy(d.node_size_y).to(DEVICE).double()
    scale = (weight + lam * area).clamp(min=1.0)
    return {"objective": wl + lam * energy, "grad": ((wl_grad + lam * grad).view(2, -1) / scale).reshape(-1)}
