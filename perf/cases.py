"""The work a user of the placer has it do, as measurable cases.

Every case goes through the public Python entry points (Design, FluxionEngine's stages) on
seeded synthetic netlists with the repository's own shapes: 1.2 nets per gate, a die side of
1.2 sqrt(gates), density bins near sqrt(gates) in steps of 128, the serving and benchmark
congestion grids. Sizes run from the smallest serving job (5,000 gates) to the 1M-gate
benchmark, odd ones among them.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "neon-physics-fluxion_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import fluxion_b200 as fx  # noqa: E402

_PRECISION = {"i8": fx.FX_DCT_I8, "simt": fx.FX_DCT_SIMT}


def listed():
    return [
        # one iteration of the smallest serving design: a host loop that edits positions
        # between calls; launches and latency count
        {"name": "step_5k", "kind": "iterate", "gates": 5003, "iters": 1, "bins": 128,
         "grid": 256, "precision": "simt", "walk": "fast"},
        # the reproducible run of the small configuration: 10,000 gates, no density term,
        # 200 iterations in one call, exact walk
        {"name": "plain_10k", "kind": "iterate", "gates": 10000, "iters": 200, "bins": 0,
         "grid": 64, "precision": "simt", "walk": "exact"},
        # a mid-size ECO: a few iterations of a resident design with the serving defaults
        {"name": "eco_100k", "kind": "iterate", "gates": 99991, "iters": 4, "bins": 256,
         "grid": 256, "precision": "simt", "walk": "fast"},
        # the benchmark's step at full size with the default density precision
        {"name": "step_1m", "kind": "iterate", "gates": 1000000, "iters": 2, "bins": 1024,
         "grid": 512, "precision": "i8", "walk": "fast"},
        # the density force alone, default precision: the grid of a 400k-gate design
        {"name": "density_640", "kind": "density", "gates": 400003, "bins": 640,
         "precision": "i8"},
        # and the large grid of the precision study
        {"name": "density_2048", "kind": "density", "gates": 200000, "bins": 2048,
         "precision": "i8"},
        # Barnes-Hut forces alone of an ordinary design
        {"name": "bh_300k", "kind": "barnes_hut", "gates": 300007, "walk": "fast"},
        # batched leaf placement, bit-exact arithmetic: the leaves of a mid-size design
        {"name": "leaves_ieee", "kind": "leaves", "clusters": 2053, "max_size": 128,
         "iters": 300, "precision": "ieee"},
        # and the serving arithmetic on the full leaf batch
        {"name": "leaves_fast", "kind": "leaves", "clusters": 16384, "max_size": 128,
         "iters": 50, "precision": "fast"},
        # the hierarchy of a placement job (serving mode: FP64 norms, 30 power iterations)
        {"name": "partition_100k", "kind": "partition", "gates": 100003},
        # the refinement loop that ends a placement job
        {"name": "refine_50k", "kind": "refine", "gates": 50021, "grid": 256},
        # congestion and wirelength of host positions, as an external placer asks for them
        {"name": "congestion_500k", "kind": "congestion", "gates": 500009, "grid": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bins(n):
    return min(1024, max(128, int(round(math.sqrt(n) / 128.0)) * 128))


def draw(rng):
    kind = rng.choice(["iterate", "iterate", "iterate", "density", "density", "barnes_hut",
                       "barnes_hut", "leaves", "leaves", "partition", "refine", "congestion"])
    if kind == "iterate":
        n = _log(rng, 5000, 1000000)
        g = _bins(n)
        # longer runs of the contracting iteration amplify rounding; two iterations at most
        # on the larger designs
        return {"kind": kind, "gates": n, "iters": rng.randint(1, 4 if n <= 150000 else 2),
                "bins": g, "grid": rng.choice([64, 200, 256, 512]),
                "precision": "i8" if g >= 1024 else rng.choice(["i8", "simt"]),
                "walk": rng.choice(["fast", "fast", "exact"])}
    if kind == "density":
        return {"kind": kind, "gates": _log(rng, 5000, 400000),
                "bins": 128 * _log(rng, 1, 16), "precision": "i8"}
    if kind == "barnes_hut":
        return {"kind": kind, "gates": _log(rng, 5000, 1000000),
                "walk": rng.choice(["fast", "fast", "exact"])}
    if kind == "leaves":
        return {"kind": kind, "clusters": _log(rng, 64, 4096),
                "max_size": rng.choice([32, 64, 100, 128]),
                "iters": rng.choice([50, 100, 300]), "precision": rng.choice(["ieee", "fast"])}
    if kind == "partition":
        return {"kind": kind, "gates": _log(rng, 5000, 200000)}
    if kind == "refine":
        return {"kind": kind, "gates": _log(rng, 5000, 100000), "grid": rng.choice([64, 128, 256])}
    return {"kind": kind, "gates": _log(rng, 5000, 1000000), "grid": rng.choice([64, 300, 512, 1024])}


def _leaf_batch(case, seed):
    """Independent leaf clusters of log-uniform 16..max_size gates (the same sizes for every
    seed), 1.5 nets a gate of degree 2-8 inside a cluster, unit regions, as the leaf benchmark's."""
    k, most = case["clusters"], case["max_size"]
    u = np.random.RandomState(k).uniform(math.log(16), math.log(most + 1), k)
    sizes = np.clip(np.exp(u).astype(np.int64), 16, most)
    start = np.zeros(k + 1, np.int64)
    np.cumsum(sizes, out=start[1:])
    n = int(start[-1])
    rng = np.random.RandomState(seed + 1)
    cluster = np.repeat(np.arange(k), (3 * sizes + 1) // 2)
    m = len(cluster)
    degree = np.minimum(1 + rng.geometric(0.5, m), 8)
    # eight distinct members of the cluster: a start and gaps that cannot wrap onto it
    gap = 1 + (rng.random_sample((m, 8)) * ((sizes[cluster] - 1) // 7)[:, None]).astype(np.int64)
    gap[:, 0] = rng.randint(0, 1 << 30, m)
    member = start[cluster][:, None] + np.cumsum(gap, axis=1) % sizes[cluster][:, None]
    net_gate = member[np.arange(8)[None, :] < degree[:, None]].astype(np.int32)
    net_ptr = np.zeros(m + 1, np.int32)
    np.cumsum(degree, out=net_ptr[1:])
    w = (1 + rng.randint(0, 4, n)).astype(np.float32)
    circuit = fx.Circuit(n, net_ptr, net_gate, w, np.ones(n, np.float32), 1.0, 1.0)
    region = np.tile(np.array([0.5, 0.5, 1.0, 1.0], np.float32), k)
    zero = np.zeros(n, np.float32)
    return fx.Synth(circuit, fx.Placement(zero, zero.copy()), start.astype(np.int32), region)


def _synth(case, seed):
    if case["kind"] == "leaves":
        return _leaf_batch(case, seed)
    n = case["gates"]
    return fx.synth_plain(seed + 1, n, int(1.2 * n), 1.2 * math.sqrt(n))


def _density_weight():
    return float(fx.iter_cfg().density_weight)


def prepare(case, seed):
    syn = _synth(case, seed)
    ctx = fx.default_context()
    design = fx.Design(ctx, syn.circuit)
    p = syn.placement
    state = {"case": case, "design": design}
    kind = case["kind"]
    if kind in ("iterate", "density", "barnes_hut"):
        design.set_positions(p.gate_x, p.gate_y)
    if kind == "iterate":
        design.save_state()
        state["cfg"] = fx.iter_cfg(
            density_bins=case["bins"], dct_precision=_PRECISION[case["precision"]],
            cong_cols=case["grid"], cong_rows=case["grid"],
            bh_walk=fx.FX_BH_EXACT if case["walk"] == "exact" else fx.FX_BH_FAST)
    elif kind == "leaves":
        state["leaf_ptr"] = syn.leaf_ptr
        state["leaf_gate"] = np.arange(syn.circuit.num_gates, dtype=np.int32)
        state["region"] = syn.region
        state["cfg"] = fx.leaf_cfg(
            force_iterations=case["iters"],
            precision=fx.FX_LEAF_FAST if case["precision"] == "fast" else fx.FX_LEAF_IEEE)
    elif kind in ("partition", "refine"):
        part = fx.part_cfg(mode=fx.FX_PART_FP64, power_iterations=30, tol=0.0)
        state["cfg"] = part
        if kind == "refine":
            tree = design.partition(part)
            x, y, _ = design.place_leaves(tree["leaf_ptr"], tree["leaf_gate"], tree["region"],
                                          fx.leaf_cfg(precision=fx.FX_LEAF_IEEE))
            state["x"], state["y"] = x, y
            state["cfg"] = fx.refine_cfg(grid_cols=case["grid"], grid_rows=case["grid"])
    elif kind == "congestion":
        state["x"], state["y"] = p.gate_x, p.gate_y
    ctx.synchronize()
    return state


def run(state):
    case, d = state["case"], state["design"]
    kind = case["kind"]
    if kind == "iterate":
        d.restore_state()
        st = d.force_iterate(state["cfg"], case["iters"])
        x, y = d.get_positions()
        return {"x": x, "y": y, "hpwl": float(st.hpwl), "overflow": float(st.total_overflow)}
    if kind == "density":
        return d.density(case["bins"], 0.7, _density_weight(), _PRECISION[case["precision"]])
    if kind == "barnes_hut":
        f = d.barnes_hut(walk=fx.FX_BH_EXACT if case["walk"] == "exact" else fx.FX_BH_FAST)
        return dict(zip(("fx", "fy", "keys", "perm", "root"), f))
    if kind == "leaves":
        x, y, _ = d.place_leaves(state["leaf_ptr"], state["leaf_gate"], state["region"],
                                 state["cfg"])
        return {"x": x, "y": y}
    if kind == "partition":
        t = d.partition(state["cfg"])
        return {k: t[k] for k in ("leaf_ptr", "leaf_gate", "region", "leaf_depth")}
    if kind == "refine":
        x, y = state["x"].copy(), state["y"].copy()
        st = d.refine(state["cfg"], x, y)
        return {"x": x, "y": y, "iterations": int(st.iterations), "moves": int(st.moves),
                "hpwl": float(st.hpwl)}
    counts, hpwl, total, most = d.congestion(case["grid"], case["grid"], state["x"], state["y"])
    return {"counts": counts, "hpwl": hpwl, "total": total, "max": most}


def work(case):
    kind = case["kind"]
    if kind == "leaves":
        m = case["max_size"]
        # sizes are log-uniform in 16..m: mean and mean square
        span = math.log(m / 16.0)
        mean, square = (m - 16) / span, (m * m - 256) / 2.0 / span
        pairs = case["clusters"] * (square - mean) / 2.0
        gates = case["clusters"] * mean
        # 17 operations a pair and iteration; ids, regions and adjacency in, positions out
        return {"bytes": 40.0 * gates, "flops": 17.0 * pairs * case["iters"]}
    n = case["gates"]
    pins, adj = 3.12 * n, 11.1 * n
    if kind == "iterate":
        g, c = case["bins"], case["grid"]
        # adjacency, state in and out, net pins, areas, grids; about 272 Barnes-Hut terms of
        # 12 operations a gate, 3 a neighbour and axis, three 2-D fast transforms of the grid
        nbytes = 4 * adj + 4 * n + 4 * pins + 4.8 * n + 36 * n + 4 * g * g + 4 * c * c
        flops = 272 * 12 * n + 6 * adj + (3 * 5 * g * g * math.log2(g) if g else 0)
        return {"bytes": nbytes * case["iters"], "flops": flops * case["iters"]}
    if kind == "density":
        g = case["bins"]
        return {"bytes": 12.0 * n + 8.0 * n + 4.0 * g * g, "flops": 15.0 * g * g * math.log2(g)}
    if kind == "barnes_hut":
        return {"bytes": 8.0 * n + 16.0 * n, "flops": 272 * 12.0 * n}
    if kind == "partition":
        levels = max(1.0, math.log2(n / 64.0))
        return {"bytes": levels * 30 * (4 * adj / levels * 2 + 12 * n), "flops": levels * 60 * adj / 4}
    if kind == "refine":
        g = case["grid"]
        # at least one pass: nets and positions in, grid counted, positions out
        return {"bytes": 4 * pins + 4.8 * n + 16 * n + 4 * g * g, "flops": 8 * pins}
    g = case["grid"]
    return {"bytes": 4 * pins + 4.8 * n + 8 * n + 4 * g * g, "flops": 8.0 * pins + 4.0 * g * g}


def _density_exact(case, seed):
    """The DCT-Poisson field of the binned areas in 64 bits, with dense cosine matrices."""
    syn = _synth(case, seed)
    c, p, g = syn.circuit, syn.placement, case["bins"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    w, h = np.float32(c.chip_width), np.float32(c.chip_height)
    bw, bh = w / np.float32(g), h / np.float32(g)

    def bins(v, b):  # the bin is chosen in single precision, as the entry point defines it
        return np.clip(np.nan_to_num(v / b), 0, g - 1).astype(np.int64)

    col, row = bins(p.gate_x, bw), bins(p.gate_y, bh)
    area = (c.gate_widths * c.gate_heights).astype(np.float64)
    rho = np.bincount(row * g + col, weights=area, minlength=g * g).reshape(g, g)
    rho = rho / (float(bw) * float(bh)) - float(np.float32(0.7))
    k = torch.arange(g, dtype=torch.float64, device=dev)
    cm = torch.cos(math.pi * (2 * k[None, :] + 1) * k[:, None] / (2 * g)) * math.sqrt(2.0 / g)
    cm[0] *= math.sqrt(0.5)
    hat = cm @ torch.from_numpy(rho).to(dev) @ cm.T
    wx, wy = 1.0 / float(bw), 1.0 / float(bh)
    ax, ay = wx * torch.cos(math.pi * k / g) - wx, wy * torch.cos(math.pi * k / g) - wy
    lam = ay[:, None] ** 2 + ax[None, :] ** 2
    lam[0, 0] = 1.0
    hat = -hat / lam
    hat[0, 0] = 0.0
    phi = cm.T @ hat @ cm

    def slope(f, s):  # centred inside, one-sided at the edges, along the last axis
        e = torch.empty_like(f)
        e[:, 1:-1] = -(f[:, 2:] - f[:, :-2]) * (s * 0.5)
        e[:, 0] = -(f[:, 1] - f[:, 0]) * s
        e[:, -1] = -(f[:, -1] - f[:, -2]) * s
        return e

    ex, ey = slope(phi, wx).cpu().numpy(), slope(phi.T.contiguous(), wy).T.cpu().numpy()
    weight, ph = float(np.float32(_density_weight())), phi.cpu().numpy()
    return {"fx": area * ex[row, col] * weight, "fy": area * ey[row, col] * weight,
            "energy": float((0.5 * area * ph[row, col]).sum() * weight)}


def exact(case, seed):
    if case["kind"] == "density":
        return _density_exact(case, seed)
    if case["kind"] == "congestion":
        # the crossing counts are whole numbers; the wirelength is a 64-bit sum
        syn = _synth(case, seed)
        c, p = syn.circuit, syn.placement
        at = c.net_ptr[:-1][np.diff(c.net_ptr) > 0]
        span = 0.0
        for v in (p.gate_x, p.gate_y):
            q = v[c.net_gate].astype(np.float64)
            span += float((np.maximum.reduceat(q, at) - np.minimum.reduceat(q, at)).sum())
        return {"counts": None, "hpwl": span, "total": None, "max": None}
    # forces of the opening-angle tree, contracted positions and hierarchies are defined by
    # single-precision decisions: no 64-bit value of their own
    return None
