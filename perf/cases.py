"""The work that users of this placer have it do, as timed cases.

A case names a kind of call and its sizes; `prepare` makes what a program
holds before the call (a design, a handle, starting positions), `run` is one
pass through the public entry points, `work` the bytes and operations it
cannot do without, and `exact` the same results in 64 bits where they are
plain numbers.

  loop       Placer: some iterations of a placement, then the positions and the
             readout, as a program that shows or judges its progress has it;
             a placement that has reached its target starts over
  host_step  Placer.step_host: one iteration on the caller's pinned arrays
  batch      BatchPlacer: trial steps of many designs at once
  stages     the four stage calls in the order of a program that runs its own
             loop: wirelength gradient, density map, field, node forces
  field      one field solve of a density map in host memory
  device_field  one field solve on the caller's device buffers
  forward, gradient  the surrogate network's inference and training gradient
"""
import ctypes
import math

import numpy as np
import torch

import aieplace_gb300 as ap
from aieplace_gb300._lib import check, lib

DESIGN_SEED = 1  # the netlists are those of the benchmark and the tests; positions and maps come from the case's seed
MIN_BINS_MIXED = 128  # the mixed-precision solver takes bins from here on


def listed():
    return [
        # the smallest design of the tests: 576 unit cells, launches and latency
        dict(name="loop_576", kind="loop", cells=576, bins=32, solver="fp32", start="spread", iterations=10),
        # the tests' 20k-cell design on the mixed solver's smallest grid
        dict(name="loop_20k_mixed", kind="loop", cells=20_000, bins=128, solver="bf16x3", start="centre", iterations=10),
        # a block-sized design, default solver
        dict(name="loop_200k", kind="loop", cells=200_000, bins=512, solver="fp32", start="centre", iterations=10),
        # the benchmark's design with the default solver, from the clustered start of a fresh placement
        dict(name="loop_2m", kind="loop", cells=2_000_000, bins=1024, solver="fp32", start="centre", iterations=10),
        # the same in mixed precision, continued from a spread placement
        dict(name="loop_2m_mixed", kind="loop", cells=2_000_000, bins=1024, solver="bf16x3", start="spread",
             iterations=10),
        # the benchmark's end-to-end call: a host program that owns the positions
        dict(name="host_step_2m_mixed", kind="host_step", cells=2_000_000, bins=1024, solver="bf16x3"),
        # the batched form over uneven designs
        dict(name="batch_32", kind="batch", instances=32, lo=5_000, hi=150_000, trials=10),
        # a program with its own loop, on a die that is not square
        dict(name="stages_200k", kind="stages", cells=200_003, bins=512, solver="fp32", aspect=1.5),
        # the field alone, as the reference's doFFT is called
        dict(name="field_1024_mixed", kind="field", bins=1024, solver="bf16x3", aspect=1.0),
        # the smallest call: a host framework's own device buffers
        dict(name="device_field_96", kind="device_field", bins=96, aspect=1.0),
        # the surrogate: inference on a coarse grid, and a training batch's gradient
        dict(name="forward_256", kind="forward", factor=4, batch=1, res=256),
        dict(name="gradient_64", kind="gradient", factor=2, batch=8, res=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bins_for(cells, lo):
    """About four cells a bin, as the designs of the benchmark and the tests have."""
    return min(1024, max(lo, 2 ** math.ceil(math.log2(math.sqrt(cells / 4.0)))))


def draw(rng):
    kind = rng.choice(["loop", "loop", "loop", "host_step", "batch", "stages", "field", "device_field", "surrogate"])
    solver = rng.choice(["fp32", "bf16x3"])
    if kind == "loop":
        cells = _log_int(rng, 500, 2_000_000)
        return dict(kind=kind, cells=cells, bins=_bins_for(cells, 32 if solver == "fp32" else MIN_BINS_MIXED),
                    solver=solver, start=rng.choice(["centre", "spread"]),
                    iterations=rng.randint(4, 10))
    if kind == "host_step":
        cells = _log_int(rng, 500, 2_000_000)
        return dict(kind=kind, cells=cells, bins=_bins_for(cells, 32 if solver == "fp32" else MIN_BINS_MIXED),
                    solver=solver)
    if kind == "batch":
        return dict(kind=kind, instances=rng.randint(3, 32), lo=_log_int(rng, 500, 6_000),
                    hi=_log_int(rng, 8_000, 150_000), trials=rng.randint(4, 10))
    if kind == "stages":
        cells = _log_int(rng, 500, 250_000)
        return dict(kind=kind, cells=cells, bins=_bins_for(cells, 32 if solver == "fp32" else MIN_BINS_MIXED),
                    solver=solver, aspect=rng.choice([1.0, 1.5, 0.7]))
    if kind == "field":
        return dict(kind=kind, bins=rng.choice([32, 64, 128, 256, 512, 1024] if solver == "fp32" else
                                               [128, 256, 512, 1024]), solver=solver,
                    aspect=rng.choice([1.0, 1.5, 0.7]))
    if kind == "device_field":
        return dict(kind=kind, bins=32 * rng.randint(1, 8), aspect=round(rng.uniform(0.5, 2.0), 3))
    if rng.random() < 0.5:
        return dict(kind="forward", factor=rng.choice([1, 2, 4]), batch=rng.randint(1, 4), res=16 * rng.randint(2, 16))
    return dict(kind="gradient", factor=rng.choice([1, 2, 4]), batch=rng.randint(1, 8), res=16 * rng.randint(2, 6))


# ---- inputs -----------------------------------------------------------------
_designs = {}


def _design(cells, bins, aspect=1.0):
    """A design of the benchmark's statistics (fewer than 2000 cells: the unit-cell statistics of the smallest)."""
    key = (cells, bins, aspect)
    if key not in _designs:
        if cells < 2_000:
            spec = dict(num_cells=cells, num_nets=max(1, round(cells * 640 / 576)), num_macros=0, num_pads=24,
                        unit_cells=1, degree_mix=0, locality=0.0, window=64, target_density=1.0,
                        die_side=float(math.ceil(math.sqrt(cells))), bins=bins)
        else:
            spec = dict(num_cells=cells, num_nets=round(1.05 * cells),
                        num_macros=max(1, cells // (100 if cells > 500_000 else 50)), num_pads=0, unit_cells=0,
                        degree_mix=1, locality=0.8, window=64, target_density=0.8 if cells > 500_000 else 0.7,
                        die_side=0.0, bins=bins)
        nl = ap.synth.generate(spec, seed=DESIGN_SEED)
        if aspect != 1.0:  # a die higher (or wider) than the square one, the same cells on it
            die = nl["die"].copy()
            die[3 if aspect > 1.0 else 2] *= np.float32(max(aspect, 1.0 / aspect))
            nl["die"] = die
        _designs.clear()  # one design in memory at a time
        _designs[key] = nl
    return _designs[key]


def _positions(nl, start, seed):
    """Starting positions: `centre`, a fresh placement's cluster at the die
    centre; `spread`, a placement under way -- cells along a space-filling curve
    in netlist order (nets connect near indices) with some noise."""
    rng = np.random.default_rng(seed)
    mov = nl["node_fixed"] == 0
    n = int(mov.sum())
    w, h = float(nl["die"][2] - nl["die"][0]), float(nl["die"][3] - nl["die"][1])
    if start == "centre":
        px = 0.5 * w + rng.standard_normal(n)
        py = 0.5 * h + rng.standard_normal(n)
    else:
        code = (np.arange(n, dtype=np.uint64) * np.uint64((1 << 40) // n))
        cx, cy = np.zeros(n, np.uint64), np.zeros(n, np.uint64)
        for b in range(20):  # de-interleave the bits
            cx |= ((code >> np.uint64(2 * b)) & np.uint64(1)) << np.uint64(b)
            cy |= ((code >> np.uint64(2 * b + 1)) & np.uint64(1)) << np.uint64(b)
        noise = 2.0 * w / nl["bins"]
        px = cx * (w / (1 << 20)) + noise * rng.standard_normal(n)
        py = cy * (h / (1 << 20)) + noise * rng.standard_normal(n)
    x, y = nl["node_x"].copy(), nl["node_y"].copy()
    x[mov] = np.clip(px, 0.0, np.maximum(w - nl["node_w"][mov], 0.0)).astype(np.float32)
    y[mov] = np.clip(py, 0.0, np.maximum(h - nl["node_h"][mov], 0.0)).astype(np.float32)
    return x, y


def _map(bins, seed):
    """A density map as the loop meets them: nearly full bins, a crowded region, an empty one."""
    rng = np.random.default_rng(seed)
    d = (0.8 + 0.1 * rng.standard_normal((bins, bins))).astype(np.float32)
    a = int(rng.integers(bins // 8, bins // 2))
    d[a: a + bins // 4, bins // 4: bins // 2] += np.float32(rng.uniform(1.0, 3.0))
    d[bins // 8: bins // 5, a: a + bins // 8] = 0.0
    return d


def _field_design(aspect):
    """A small design whose handle serves the field call at any bin count."""
    return _design(576, 32, aspect)


def _net(case, seed):
    net = ap.Surrogate(factor=case["factor"], kernels=(3, 1, 1, 1), width=32, seed=1)
    rng = np.random.default_rng(seed)
    params = (0.15 * rng.standard_normal(net.num_params)).astype(np.float32)
    net.set_params(params)
    x = rng.standard_normal((case["batch"], net.cin, case["res"], case["res"])).astype(np.float32)
    t = rng.standard_normal((case["batch"], net.cout, case["res"], case["res"])).astype(np.float32)
    return net, params, x, t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        specs = ap.synth.batch_specs(case["instances"], seed=DESIGN_SEED, lo=case["lo"], hi=case["hi"])
        b = ap.BatchPlacer([ap.synth.generate(s, seed=DESIGN_SEED + i) for i, s in enumerate(specs)])
        b.initialize_placement(seed=seed, sigma=1.0)
        return dict(case=case, batch=b, seed=seed, trials=0)
    if kind in ("loop", "host_step", "stages"):
        nl = _design(case["cells"], case["bins"], case.get("aspect", 1.0))
        x, y = _positions(nl, case.get("start", "spread"), seed)
        pl = ap.Placer(nl, bins=case["bins"], field_solver=case["solver"])
        if kind == "stages":
            return dict(case=case, placer=pl, x=x, y=y, die=nl["die"])
        pl.initialize_placement(x, y)
        pinned = [torch.empty(len(x), dtype=torch.float32, pin_memory=True) for _ in range(4)]
        pinned[0].copy_(torch.from_numpy(x))
        pinned[1].copy_(torch.from_numpy(y))
        return dict(case=case, placer=pl, arrays=[t.numpy() for t in pinned], pinned=pinned, done=False)
    if kind == "field":
        pl = ap.Placer(_field_design(case["aspect"]), bins=case["bins"], field_solver=case["solver"])
        return dict(case=case, placer=pl, map=_map(case["bins"], seed))
    if kind == "device_field":
        m = case["bins"]
        d = torch.from_numpy(_map(m, seed)).cuda()
        return dict(case=case, d=d, ex=torch.empty_like(d), ey=torch.empty_like(d))
    net, _, x, t = _net(case, seed)
    return dict(case=case, net=net, x=x, t=t)


# ---- one pass ---------------------------------------------------------------
READOUT = ("iteration", "hpwl", "wa", "overflow", "overflow_abs", "gamma")
TARGET, MOST_ITERATIONS = 0.1, 3000  # a placement ends at 10% overflow, or after this many iterations
GAMMA, LAMBDA = 2.0, 0.05  # the stage calls' smoothing (in bins) and density weight


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("loop", "host_step"):
        pl = state["placer"]
        xi, yi, xo, yo = state["arrays"]
        if state["done"]:
            pl.initialize_placement(xi, yi)
        if kind == "loop":
            pl.perform_iteration(case["iterations"] - 1)
            s = pl.step_host(None, None, xo, yo)
            state["done"] = s["overflow"] < TARGET or s["iteration"] >= MOST_ITERATIONS
        else:
            s = pl.step_host(xi, yi, xo, yo)
            state["done"] = s["iteration"] >= MOST_ITERATIONS
        return dict(x=xo, y=yo, **{k: s[k] for k in READOUT})
    if kind == "batch":
        b = state["batch"]
        if state["trials"] >= MOST_ITERATIONS:
            b.initialize_placement(seed=state["seed"], sigma=1.0)
            state["trials"] = 0
        b.step(case["trials"])
        state["trials"] += case["trials"]
        at = [b.positions(i) for i in range(b.n)]
        stats = [b.stats(i) for i in range(b.n)]
        return dict(x=np.concatenate([a[0] for a in at]), y=np.concatenate([a[1] for a in at]),
                    iteration=np.array([s["iteration"] for s in stats]),
                    hpwl=np.array([s["hpwl"] for s in stats], np.float32),
                    overflow=np.array([s["overflow"] for s in stats], np.float32))
    if kind == "stages":
        pl, x, y, m = state["placer"], state["x"], state["y"], case["bins"]
        bw, bh = float(state["die"][2]) / m, float(state["die"][3]) / m
        gx, gy, wa, hpwl = pl.compute_all_partials(x, y, GAMMA * bw)
        rho = pl.compute_overlaps(x, y)
        ex, ey = pl.compute_electric_fields(rho * (2.0 ** -32 / (bw * bh)))
        fx, fy, px, py = pl.compute_node_forces(x, y, ex, ey, gamma=GAMMA * bw, lam=LAMBDA)
        return dict(gx=gx, gy=gy, wa=wa, hpwl=hpwl, rho=rho, ex=ex, ey=ey, fx=fx, fy=fy, px=px, py=py)
    if kind == "field":
        ex, ey = state["placer"].compute_electric_fields(state["map"])
        return dict(ex=ex, ey=ey)
    if kind == "device_field":
        check("ap_field_solve_noalloc", lib().ap_field_solve_noalloc(
            ctypes.c_void_p(state["d"].data_ptr()), ctypes.c_void_p(state["ex"].data_ptr()),
            ctypes.c_void_p(state["ey"].data_ptr()), case["bins"], ctypes.c_float(case["aspect"]),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return dict(ex=state["ex"], ey=state["ey"])
    if kind == "forward":
        return dict(y=state["net"].forward(state["x"]))
    loss, grad = state["net"].gradient(state["x"], state["t"], 1)
    return dict(loss=loss, grad=grad)


# ---- what a pass cannot do without ------------------------------------------
def _field_flops(m):
    """Three 2-D real transforms (one forward, two inverse) by fast algorithms: 2 x 2.5 m^2 log2(m) each."""
    return 15.0 * m * m * math.log2(m)


def _counts(cells):
    """Nodes, nets and pins of a design (expected pins a net of the degree mixes)."""
    if cells < 2_000:
        return cells + 24, round(cells * 640 / 576), 2.4 * cells * 640 / 576
    return 1.02 * cells, 1.05 * cells, 1.05 * cells * 4.475


def _iteration(cells, bins):
    """Bytes and operations of one iteration: the netlist once, the optimiser
    state (accepted and trial positions, gradients) read and written, sizes and
    positions read, the fixed map read, the density and the field once each."""
    nodes, nets, pins = _counts(cells)
    return (4 * nets + 4 * pins + 8 * nodes + 56 * cells + 20 * bins * bins,
            _field_flops(bins) + 60.0 * pins + 60.0 * cells)


def work(case):
    kind = case["kind"]
    if kind == "loop":
        b, f = _iteration(case["cells"], case["bins"])
        n = case["iterations"]
        return dict(bytes=n * b + 8 * case["cells"], flops=n * f)
    if kind == "host_step":
        b, f = _iteration(case["cells"], case["bins"])
        return dict(bytes=b + 16 * case["cells"], flops=f)
    if kind == "batch":
        total_b = total_f = 0.0
        for s in ap.synth.batch_specs(case["instances"], seed=DESIGN_SEED, lo=case["lo"], hi=case["hi"]):
            b, f = _iteration(s["num_cells"], s["bins"])
            total_b, total_f = total_b + case["trials"] * b, total_f + case["trials"] * f
        return dict(bytes=total_b, flops=total_f)
    if kind == "stages":
        nodes, nets, pins = _counts(case["cells"])
        m = case["bins"]
        # positions in, gradients, forces and preconditioned gradients out, the map and the field out and in
        return dict(bytes=8 * nodes + 24 * nodes + 4 * nets + 4 * pins + 28 * m * m,
                    flops=_field_flops(m) + 60.0 * pins + 60.0 * nodes)
    if kind in ("field", "device_field"):
        m = case["bins"]
        return dict(bytes=12 * m * m, flops=_field_flops(m))
    f, b, r = case["factor"], case["batch"], case["res"]
    cin, cout = f * f + 2, 2 * f * f
    macs = b * r * r * (9 * cin * 32 + 2 * 32 * 32 + 32 * cout)
    if kind == "forward":
        return dict(bytes=4.0 * b * r * r * (cin + cout), flops=2.0 * macs)
    return dict(bytes=4.0 * b * r * r * (cin + cout), flops=6.0 * macs)


# ---- the same in 64 bits ----------------------------------------------------
def _cosines(m, dev):
    k = torch.arange(m, dtype=torch.float64, device=dev)
    t = torch.outer(k, k + 0.5) * (math.pi / m)
    return torch.cos(t), torch.sin(t)


def _exact_field(d, m, ratio, dev):
    """phi_uv = a_uv / (wx^2 + wy^2), a the 2-D DCT-II with halved edges; the
    field by the sine-cosine and cosine-sine inverse transforms."""
    c, s = _cosines(m, dev)
    w = torch.arange(m, dtype=torch.float64, device=dev) * (math.pi / m)
    wx, wy = w[:, None], w[None, :] * ratio
    a = c @ d.to(torch.float64) @ c.T * (4.0 / m ** 2)
    a[0, :] *= 0.5
    a[:, 0] *= 0.5
    den = wx ** 2 + wy ** 2
    den[0, 0] = 1.0
    phi = a / den
    phi[0, 0] = 0.0
    return s.T @ (phi * wx) @ c, c.T @ (phi * wy) @ s


def _exact_wirelength(nl, x, y, gamma, dev):
    ptr = torch.from_numpy(nl["net_ptr"].astype(np.int64)).to(dev)
    deg = ptr[1:] - ptr[:-1]
    net = torch.repeat_interleave(torch.arange(len(deg), device=dev), deg)
    pin = torch.from_numpy(nl["pin_node"].astype(np.int64)).to(dev)
    keep = deg[net] >= 2
    net, pin = net[keep], pin[keep]
    live = deg >= 2
    grads, wa, hpwl = [], 0.0, 0.0
    for p in (x, y):
        v = p[pin]
        hi = torch.full((len(deg),), -math.inf, dtype=v.dtype, device=dev).scatter_reduce(0, net, v, "amax")
        lo = torch.full((len(deg),), math.inf, dtype=v.dtype, device=dev).scatter_reduce(0, net, v, "amin")
        zero = torch.zeros(len(deg), dtype=v.dtype, device=dev)
        ap_, am = torch.exp((v - hi[net]) / gamma), torch.exp((lo[net] - v) / gamma)
        bp, bm = zero.index_add(0, net, ap_), zero.index_add(0, net, am)
        wp = zero.index_add(0, net, ap_ * (v - hi[net])) / bp + hi  # the weighted averages
        wm = zero.index_add(0, net, am * (v - lo[net])) / bm + lo
        g = ap_ / bp[net] * (1 + (v - wp[net]) / gamma) - am / bm[net] * (1 - (v - wm[net]) / gamma)
        grads.append(torch.zeros(len(p), dtype=v.dtype, device=dev).index_add(0, pin, g))
        wa = wa + (wp - wm)[live].sum()
        hpwl = hpwl + (hi - lo)[live].sum()
    pins = torch.zeros(len(x), dtype=x.dtype, device=dev).index_add(0, pin, torch.ones_like(v))
    return grads[0], grads[1], wa, hpwl, pins


def _exact_stages(case, seed):
    dev = "cuda"
    m = case["bins"]
    nl = _design(case["cells"], m, case["aspect"])
    x, y = (torch.from_numpy(p).to(dev, torch.float64) for p in _positions(nl, "spread", seed))
    w, h = (torch.from_numpy(nl[k]).to(dev, torch.float64) for k in ("node_w", "node_h"))
    gamma = GAMMA * float(nl["die"][2]) / m
    gx, gy, wa, hpwl, pins = _exact_wirelength(nl, x, y, gamma, dev)
    # the grid's bin size is a multiple of 2^-16
    bw, bh = (round(float(np.float32(v) / np.float32(m)) * 65536.0) / 65536.0 for v in nl["die"][2:4])
    small = (w * h) <= bw * bh / 16  # such a node counts whole in its own bin
    c0 = torch.clamp(torch.floor(x / bw), 0, m - 1).long()
    r0 = torch.clamp(torch.floor(y / bh), 0, m - 1).long()
    moving = torch.from_numpy(nl["node_fixed"] == 0).to(dev)

    def weights(at):
        """(nodes, bin, overlap area) for every bin of the nodes `at`."""
        nc = int(torch.ceil(w[at].max() / bw)) + 1
        nr = int(torch.ceil(h[at].max() / bh)) + 1
        for j in range(nc):
            c = c0[at] + j
            ow = torch.minimum(x[at] + w[at], (c + 1) * bw) - torch.maximum(x[at], c * bw)
            for k in range(nr):
                r = r0[at] + k
                oh = torch.minimum(y[at] + h[at], (r + 1) * bh) - torch.maximum(y[at], r * bh)
                area = ow.clamp(min=0) * oh.clamp(min=0)
                area = torch.where(small[at], w[at] * h[at] if j == k == 0 else torch.zeros_like(area), area)
                fits = (c < m) & (r < m) & (area > 0)
                yield at[fits], (c * m + r)[fits], area[fits]

    index = torch.arange(len(x), device=dev)
    order = torch.argsort(w * h)  # nodes of like sizes together: few bins a group
    rho = torch.zeros(m * m, dtype=torch.float64, device=dev)
    for at in torch.chunk(index[order], 8):
        for _, b, area in weights(at):
            rho.index_add_(0, b, area)
    ratio = float(np.float32(np.float32(nl["die"][3] / m) / np.float32(nl["die"][2] / m)))
    ex, ey = (e.reshape(-1) for e in _exact_field((rho / (bw * bh)).reshape(m, m), m, ratio, dev))
    fx, fy = torch.zeros_like(x), torch.zeros_like(x)
    for at in torch.chunk(order[moving[order]], 8):
        for i, b, area in weights(at):
            fx.index_add_(0, i, area / (bw * bh) * ex[b])
            fy.index_add_(0, i, area / (bw * bh) * ey[b])
    hd = torch.clamp(pins + LAMBDA * w * h / (bw * bh), min=1.0)
    px = torch.where(moving, (gx - LAMBDA * fx) / hd, torch.zeros_like(x))
    py = torch.where(moving, (gy - LAMBDA * fy) / hd, torch.zeros_like(x))
    return dict(gx=gx, gy=gy, wa=wa, hpwl=hpwl, rho=None, ex=ex, ey=ey, fx=fx, fy=fy, px=px, py=py)


def _exact_net(params, x, case):
    f = case["factor"]
    y = x
    at = 0
    for layer, k in enumerate((3, 1, 1, 1)):
        cin = f * f + 2 if layer == 0 else 32
        cout = 2 * f * f if layer == 3 else 32
        weight = params[at: at + cout * cin * k * k].reshape(cout, cin, k, k)
        at += cout * cin * k * k
        y = torch.nn.functional.conv2d(y, weight, params[at: at + cout], padding=k // 2)
        at += cout
        if layer < 3:
            y = torch.relu(y)
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind in ("loop", "host_step", "batch"):
        return None  # many steps of a loop that amplifies rounding
    if kind == "stages":
        return _exact_stages(case, seed)
    if kind == "field":
        m, die = case["bins"], _field_design(case["aspect"])["die"]
        ratio = float(np.float32(np.float32(die[3] / m) / np.float32(die[2] / m)))
        ex, ey = _exact_field(torch.from_numpy(_map(m, seed)).cuda(), m, ratio, "cuda")
        return dict(ex=ex.reshape(-1), ey=ey.reshape(-1))
    if kind == "device_field":
        m = case["bins"]
        ex, ey = _exact_field(torch.from_numpy(_map(m, seed)).cuda(), m, float(np.float32(case["aspect"])), "cuda")
        return dict(ex=ex, ey=ey)
    net, params, x, t = _net(case, seed)
    net.close()
    p = torch.from_numpy(params).cuda().double().requires_grad_(kind == "gradient")
    y = _exact_net(p, torch.from_numpy(x).cuda().double(), case)
    if kind == "forward":
        return dict(y=y)
    inner = slice(1, case["res"] - 1)
    loss = ((y - torch.from_numpy(t).cuda().double())[:, :, inner, inner] ** 2).mean()
    loss.backward()
    return dict(loss=loss.detach(), grad=p.grad)
