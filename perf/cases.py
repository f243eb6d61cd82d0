"""The routing work that users of this framework have it do, as cases to be timed.

A case is one operation of ``lue_gb300.framework`` on one raster:

- ``accu``, ``accu_threshold``, ``accu_fraction``, ``accu_capacity`` and ``accu_trigger`` over a kept flow
  direction array (its topology and layouts are there, as in a model that routes many inputs over it);
- ``kinematic_wave``: ``steps`` time steps, through ``kinematic_wave`` for one step and
  ``kinematic_wave_steps`` for more;
- ``ensemble``: the same, over several catchments of different sizes packed into one atlas;
- ``new_raster``: ``d8_flow_direction`` of an elevation raster, then ``accu`` over the new array, so the
  topology is built within the pass, as in a script that routes over a raster once;
- ``neighbours``: ``upstream`` and ``downstream`` of one material.

Rasters are fractal terrain (halving amplitude per octave, the longest wavelength a quarter of the larger
side) on a plane tilted by 1 % to the south.  Pits are opened by carving the lowest way out of each basin,
so every cell drains off the array and the main channels are longer than the raster's side.  ``catchment``
keeps the cells that drain over the southern edge and makes the others no-data, as in a river basin clipped
from a larger raster.  ``new_raster`` keeps its pits, as raw elevation models have them.
"""
import math

import torch
import torch.nn.functional as F

from lue_gb300 import ensemble
from lue_gb300 import framework as lfr

CELL_SIZE = 10.0
TILT = 0.01
BETA, TIME_STEP, CHANNEL_LENGTH = 0.6, 3600.0, 100.0
DEVICE = "cuda"

# D8 codes in the order in which the steepest descent takes its candidates, with their offsets.
D8 = ((8, -1, 0), (4, 0, -1), (6, 0, 1), (2, 1, 0), (7, -1, -1), (9, -1, 1), (1, 1, -1), (3, 1, 1))

TWO_OUTPUT = ("accu_threshold", "accu_fraction", "accu_capacity", "accu_trigger")


def _case(name, op, rows, cols, dtype="float32", steps=1, catchment=False, material="lognormal", partition=0,
          amplitude=200.0):
    return {"name": name, "op": op, "rows": rows, "cols": cols, "dtype": dtype, "steps": steps,
            "catchment": catchment, "material": material, "partition": partition, "amplitude": amplitude}


def listed():
    return [
        # the smallest request that the server takes: launches and latency
        _case("accu_256", "accu", 256, 256),
        # plain accu on one small raster in 256 x 256 partitions, as on one CPU node
        _case("accu_1k", "accu", 1024, 1024, material="uniform", partition=256, amplitude=50.0),
        # the headline raster: long main channels, 268 M cells
        _case("accu_16k", "accu", 16384, 16384, partition=2048),
        # the double instantiation, on a river basin of odd extents
        _case("accu_f64_basin", "accu", 3001, 2777, dtype="float64", catchment=True),
        # infiltration per cell on the headline raster
        _case("threshold_16k", "accu_threshold", 16384, 16384, partition=2048),
        # losses along the flow, on a river basin of odd extents
        _case("fraction_basin", "accu_fraction", 2311, 1501, catchment=True),
        # a storage that spills once it is full, ordinary size
        _case("trigger_1500", "accu_trigger", 1500, 1500),
        # one time step per call: a model that changes its rain every step
        _case("wave_2k_1", "kinematic_wave", 2048, 2048, dtype="float64"),
        # a season of steps in one call on a large raster
        _case("wave_8k_100", "kinematic_wave", 8192, 8192, dtype="float64", steps=100, partition=1024),
        # scenarios of catchments of uneven size, all steps in one call
        _case("ensemble_48", "ensemble", 1600, 1600, dtype="float64", steps=48),
        # a script: elevation to flow direction to accumulated flow, once
        _case("new_raster_2k", "new_raster", 2048, 2048),
        # one-hop operations on a large raster with a ragged width
        _case("neighbours_8k", "neighbours", 8192, 8191),
    ]


def draw(rng):
    op = rng.choice(["accu", "accu", "accu_threshold", "accu_fraction", "accu_capacity", "accu_trigger",
                     "kinematic_wave", "kinematic_wave", "ensemble", "new_raster", "neighbours"])
    most = 2.0 ** (22 if op in ("ensemble", "new_raster", "accu_trigger") else 26)
    cells = math.exp(rng.uniform(math.log(2.0 ** 15), math.log(most)))
    ratio = math.exp(rng.uniform(math.log(0.5), math.log(2.0)))
    rows, cols = max(64, round(math.sqrt(cells * ratio))), max(64, round(math.sqrt(cells / ratio)))
    if rng.random() < 0.5:  # half of them of the round sizes that models like
        rows, cols = max(64, rows // 64 * 64), max(64, cols // 64 * 64)
    steps = 1
    if op in ("kinematic_wave", "ensemble"):
        steps = int(math.exp(rng.uniform(0.0, math.log(min(100.0, max(2.0, 2.0 ** 30 / cells))))))
    double = op in ("kinematic_wave", "ensemble") or (op == "accu" and cells < 2.0 ** 24 and rng.random() < 0.4)
    c = _case("", op, rows, cols, dtype="float64" if double else "float32", steps=steps,
              catchment=op in ("accu",) + TWO_OUTPUT and rng.random() < 0.4,
              material=rng.choice(["lognormal", "uniform"]), amplitude=rng.choice([50.0, 200.0]))
    del c["name"]
    return c


# --- terrain ----------------------------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def elevation(rows, cols, amplitude, g):
    """Float32 fractal terrain on a tilted plane."""
    z = torch.zeros(1, 1, rows, cols, device=DEVICE)
    wavelength, height = max(rows, cols) / 4.0, 1.0
    for _ in range(10):
        if wavelength < 4.0:
            break
        lattice = (int(rows / wavelength) + 3, int(cols / wavelength) + 3)
        noise = torch.rand(1, 1, *lattice, device=DEVICE, generator=g) - 0.5
        fine = F.interpolate(noise, scale_factor=wavelength, mode="bicubic", align_corners=False,
                             recompute_scale_factor=False)
        off = int(wavelength)
        z += height * fine[:, :, off:off + rows, off:off + cols]
        del fine
        wavelength, height = wavelength / 2.0, height / 2.0
    south = torch.arange(rows - 1, -1, -1, device=DEVICE, dtype=torch.float32)[:, None]
    return z[0, 0] * amplitude + south * (CELL_SIZE * TILT) + (2.0 * amplitude + 1.0)


def steepest_descent(z):
    """D8 codes of an elevation raster: the first of the largest drops, 5 without one; the ground outside the
    array lies lower than any cell."""
    rows, cols = z.shape
    padded = F.pad(z, (1, 1, 1, 1), value=torch.finfo(z.dtype).tiny)
    code = torch.full((rows, cols), 5, dtype=torch.uint8, device=z.device)
    drop = torch.zeros_like(z)
    for value, dr, dc in D8:
        d = z - padded[1 + dr:1 + dr + rows, 1 + dc:1 + dc + cols]
        better = d > drop
        drop = torch.where(better, d, drop)
        code.masked_fill_(better, value)
    return code


def downstream_index(code):
    """Flat index of each cell's downstream cell; the cell itself where flow ends or leaves the array."""
    rows, cols = code.shape
    down = torch.arange(rows * cols, device=code.device).view(rows, cols)
    step = torch.zeros(256, dtype=torch.int64, device=code.device)
    for value, dr, dc in D8:
        step[value] = dr * cols + dc
    off = torch.zeros_like(code, dtype=torch.bool)
    for r, c, leaving in ((0, slice(None), (7, 8, 9)), (-1, slice(None), (1, 2, 3)), (slice(None), 0, (7, 4, 1)),
                          (slice(None), -1, (9, 6, 3))):
        for value in leaving:
            off[r, c] |= code[r, c] == value
    down += step[code.long()].masked_fill_(off, 0)
    return down.view(-1)


def _ends(down):
    """Where each cell's flow ends, by pointer jumping."""
    while True:
        further = down[down]
        if torch.equal(further, down):
            return down
        down = further


def carve(z, code):
    """`code` with every pit opened: the way from its basin over the lowest pass into a basin that drains, along
    a minimum spanning tree of the basins; the flow from the pass back to the pit is reversed."""
    rows, cols = z.shape
    n = rows * cols
    down = downstream_index(code)
    end = _ends(down)
    pits = torch.nonzero((code == 5).view(-1)).view(-1)
    if pits.numel() == 0:
        return code
    basin_of = torch.zeros(n, dtype=torch.int32, device=z.device)  # 0: drains off the array
    basin_of[pits] = torch.arange(1, pits.numel() + 1, device=z.device, dtype=torch.int32)
    basin = basin_of[end].view(rows, cols)
    del end, basin_of
    # the passes between adjacent basins: two cells and the height of the higher one
    a, b, height = [], [], []
    for dr, dc in ((0, 1), (1, 0), (1, 1), (1, -1)):
        r0, c0 = slice(0, rows - dr), slice(max(0, -dc), cols - max(0, dc))
        r1, c1 = slice(dr, rows), slice(max(0, dc), cols - max(0, -dc))
        at = torch.nonzero(basin[r0, c0] != basin[r1, c1])
        u = at[:, 0] * cols + at[:, 1] + max(0, -dc)
        v = u + dr * cols + dc
        a.append(u)
        b.append(v)
        height.append(torch.maximum(z.reshape(-1)[u], z.reshape(-1)[v]))
    a, b, height = torch.cat(a), torch.cat(b), torch.cat(height)
    order = torch.argsort(height)
    a, b = a[order], b[order]  # a pass's rank is its key: all are different
    del height, order
    basin = basin.reshape(-1)
    nb = pits.numel() + 1
    ba, bb = basin[a].long(), basin[b].long()
    parent = torch.arange(nb, device=z.device)  # basin that a basin spills into
    leave = torch.full((nb,), -1, dtype=torch.int64, device=z.device)  # its cell at the pass
    enter = torch.full((nb,), -1, dtype=torch.int64, device=z.device)  # the cell beyond
    ids = torch.arange(nb, device=z.device)
    while True:  # each connected part of the tree takes its lowest pass to another one
        part = _ends(parent)
        between = torch.nonzero(part[ba] != part[bb]).view(-1)
        if between.numel() == 0:
            break
        a, b, ba, bb = a[between], b[between], ba[between], bb[between]
        rank = torch.arange(a.numel(), device=z.device)
        best = torch.full((nb,), a.numel(), dtype=torch.int64, device=z.device)
        best.scatter_reduce_(0, part[ba], rank, "amin")
        best.scatter_reduce_(0, part[bb], rank, "amin")
        chooser = torch.nonzero((best < a.numel()) & (ids != part[0])).view(-1)
        e = best[chooser]
        forth = part[ba[e]] == chooser
        u, v = torch.where(forth, a[e], b[e]), torch.where(forth, b[e], a[e])
        other = torch.where(forth, part[bb[e]], part[ba[e]])
        # two parts that chose the same pass: one of them stays
        keep = ~((best[other] == e) & (other != part[0]) & (chooser < other))
        u, v = u[keep], v[keep]
        start = basin[u].long()
        # from the pass's basin to the root of its part, the tree turns round
        marked = torch.zeros(nb, dtype=torch.bool, device=z.device)
        marked[start] = True
        jump = parent.clone()
        for _ in range(nb.bit_length()):
            hit = jump[marked]
            marked[hit] = True
            jump = jump[jump]
        turned = torch.nonzero(marked & (parent != ids)).view(-1)
        p, l, t = parent[turned], leave[turned], enter[turned]
        parent[p], leave[p], enter[p] = turned, t, l
        parent[start], leave[start], enter[start] = basin[v].long(), u, v
    # every basin's flow from its pass back to its pit is turned round
    cur, prev = leave[1:], enter[1:]
    while cur.numel():
        following = down[cur]
        down[cur] = prev
        on = following != cur
        cur, prev = following[on], cur[on]
    step = (down - torch.arange(n, device=z.device)).view(rows, cols)
    carved = code.clone()
    for value, dr, dc in D8:
        carved.masked_fill_(step == dr * cols + dc, value)
    return carved


def flow_direction(rows, cols, amplitude, catchment, g):
    z = elevation(rows, cols, amplitude, g)
    code = carve(z, steepest_descent(z))
    if catchment:
        end = _ends(downstream_index(code)).view(rows, cols)
        code.masked_fill_(end < (rows - 1) * cols, 255)
    return code


# --- inputs -----------------------------------------------------------------------------------------------


def _lognormal(shape, dtype, g):
    return torch.empty(shape, dtype=dtype, device=DEVICE).log_normal_(0.0, 1.0, generator=g)


def _uniform(shape, dtype, lo, hi, g):
    return torch.rand(shape, dtype=dtype, device=DEVICE, generator=g) * (hi - lo) + lo


def _rain(rows, cols, g):
    """Lateral inflow (m3/s per metre) of rain blobs of 0-20 mm/h."""
    r = torch.arange(rows, device=DEVICE, dtype=torch.float32)[:, None]
    c = torch.arange(cols, device=DEVICE, dtype=torch.float32)[None, :]
    rain = torch.zeros(rows, cols, device=DEVICE)
    blobs = torch.rand(12, 4, device=DEVICE, generator=g).cpu().tolist()
    for x, y, size, peak in blobs:
        s = (0.05 + 0.2 * size) * max(rows, cols)
        rain += (0.2 + 0.8 * peak) * 20.0 * (torch.exp(-(r - x * rows) ** 2 / (2 * s * s)) *
                                             torch.exp(-(c - y * cols) ** 2 / (2 * s * s)))
    return rain.clamp_(max=20.0) * (CELL_SIZE / 1000.0 / 3600.0)


# Sides of an ensemble's catchments, as shares of the largest.
MEMBERS = (1.0, 0.82, 0.67, 0.55, 0.45, 0.37)


def _members(case):
    return [(max(24, int(case["rows"] * s)), max(24, int(case["cols"] * s))) for s in MEMBERS]


def _inputs(case, seed):
    """What the user has: plain tensors."""
    g = _generator(seed)
    op, rows, cols = case["op"], case["rows"], case["cols"]
    dtype = getattr(torch, case["dtype"])
    x = {}
    if op == "ensemble":
        x["members"] = _members(case)
        x["codes"] = [flow_direction(h, w, case["amplitude"], False, g) for h, w in x["members"]]
        atlas = ensemble.Atlas(x["members"])
        x["code"] = atlas.pack(x["codes"], 255, torch.uint8, DEVICE)
        x["discharge"] = atlas.pack([_uniform(m, torch.float64, 0.0, 1.0, g) for m in x["members"]], 0.0,
                                    torch.float64, DEVICE)
        x["rain"] = atlas.pack([_rain(h, w, g) for h, w in x["members"]], 0.0, torch.float32, DEVICE)
        x["alpha"] = atlas.pack([_uniform(m, torch.float32, 1.0, 5.0, g) for m in x["members"]], 1.0, torch.float32,
                                DEVICE)
        return x
    if op == "new_raster":
        x["elevation"] = elevation(rows, cols, case["amplitude"], g)
    else:
        x["code"] = flow_direction(rows, cols, case["amplitude"], case["catchment"], g)
    if op == "kinematic_wave":
        x["discharge"] = _uniform((rows, cols), torch.float64, 0.0, 1.0, g)
        x["rain"] = _rain(rows, cols, g)
        x["alpha"] = _uniform((rows, cols), torch.float32, 1.0, 5.0, g)
        return x
    x["material"] = (_lognormal((rows, cols), dtype, g) if case["material"] == "lognormal" else
                     _uniform((rows, cols), dtype, 0.0, 1.0, g))
    if case["catchment"]:  # no material outside the river basin
        x["material"].masked_fill_(x["code"] == 255, float("nan"))
    if op == "accu_threshold":
        x["other"] = _uniform((rows, cols), dtype, 0.0, 0.5, g)
    elif op == "accu_fraction":
        x["other"] = _uniform((rows, cols), dtype, 0.0, 1.0, g)
    elif op == "accu_capacity":
        x["other"] = 50.0 * _lognormal((rows, cols), dtype, g)
    elif op == "accu_trigger":
        x["other"] = 2.0 * _lognormal((rows, cols), dtype, g)
    return x


def prepare(case, seed):
    op = case["op"]
    x = _inputs(case, seed)
    x.pop("codes", None)
    members = x.pop("members", None)
    ps = case["partition"] or None
    ps = (ps, ps) if ps else None
    state = {"op": op, "steps": case["steps"], "partition": ps}
    if members:
        state["atlas"] = ensemble.Atlas(members)
    for k, v in x.items():
        state[k] = lfr.PartitionedArray(v, ps)
    if "code" in state and op != "neighbours":
        # the flow direction array that the program keeps has been routed over before
        fd = state["code"]
        fd.topology()
        if op in TWO_OUTPUT:
            getattr(lfr, op)(fd, 1.0, 0.5)
        elif op == "accu":
            lfr.accu(fd, torch.tensor(1.0, dtype=getattr(torch, case["dtype"])))
        elif case["steps"] == 1:
            lfr.kinematic_wave(fd, 0.5, state["rain"], 1.0, BETA, TIME_STEP, CHANNEL_LENGTH)
        else:
            lfr.kinematic_wave_steps(fd, 0.5, state["rain"], 1.0, BETA, TIME_STEP, CHANNEL_LENGTH, 2)
    return state


def run(state):
    op = state["op"]
    if op == "accu":
        return lfr.accu(state["code"], state["material"]).data
    if op in TWO_OUTPUT:
        out, rest = getattr(lfr, op)(state["code"], state["material"], state["other"])
        return [out.data, rest.data]
    if op in ("kinematic_wave", "ensemble"):
        wave = (state["code"], state["discharge"], state["rain"], state["alpha"], BETA, TIME_STEP, CHANNEL_LENGTH)
        if state["steps"] == 1:
            out = lfr.kinematic_wave(*wave)
        else:
            out = lfr.kinematic_wave_steps(*wave, state["steps"])
        return out.data
    if op == "new_raster":
        fd = lfr.d8_flow_direction(state["elevation"])
        return [fd.data, lfr.accu(fd, state["material"]).data]
    return [lfr.upstream(state["code"], state["material"]).data, lfr.downstream(state["code"], state["material"]).data]


def work(case):
    n = float(case["rows"] * case["cols"])
    size = 8 if case["dtype"] == "float64" else 4
    op = case["op"]
    if op == "accu":  # direction, material; outflow
        return {"bytes": n * (1 + 2 * size), "flops": n}
    if op in TWO_OUTPUT:  # direction, material, the rule's parameter; two results
        return {"bytes": n * (1 + 4 * size), "flops": 4 * n}
    if op in ("kinematic_wave", "ensemble"):
        # direction, discharge, rain, alpha; discharge.  A step is three Newton steps of about ten operations, in
        # the fifth root of the discharge, and the sum of what flows in.
        if op == "ensemble":
            n = float(sum(h * w for h, w in _members(case)))
        return {"bytes": n * (1 + 8 + 4 + 4 + 8), "flops": n * case["steps"] * 35}
    if op == "new_raster":  # elevation, material; directions, outflow
        return {"bytes": n * (4 + 4 + 1 + 4), "flops": 17 * n}
    return {"bytes": n * (1 + 3 * size), "flops": n}


# --- what comes out, in 64 bits ---------------------------------------------------------------------------


class Sweep:
    """The cells of a flow direction raster by decreasing distance to where their flow ends: what drains into a
    cell lies one group before it."""

    def __init__(self, code):
        self.shape = code.shape
        flat = code.reshape(-1)
        down = downstream_index(code)
        valid = flat != 255
        distance = (down != torch.arange(down.numel(), device=code.device)).int()
        # flow into no-data ends there
        distance.masked_fill_(~valid | ~valid[down], 0)
        jump = torch.where(distance > 0, down, torch.arange(down.numel(), device=code.device))
        ends = distance == 0
        while True:
            more = distance[jump]
            if not bool(more.any()):
                break
            distance = distance + more
            jump = jump[jump]
        del jump
        cells = torch.nonzero(valid).view(-1)
        distance = distance[cells]
        self.distance, order = torch.sort(distance, descending=True)
        self.cells = cells[order]
        del cells, order, distance
        n = self.cells.numel()
        self.n = n
        place = torch.full((down.numel(),), n, dtype=torch.int32, device=code.device)
        place[self.cells] = torch.arange(n, device=code.device, dtype=torch.int32)
        to = place[down[self.cells]].long()
        self.to = to.masked_fill_(ends[self.cells], n)  # n: nowhere
        self.most = int(self.distance[0]) if n else 0
        counts = torch.bincount(self.distance.long(), minlength=self.most + 1).flip(0) if n else torch.zeros(1)
        self.first = [0] + torch.cumsum(counts, 0).cpu().tolist()

    def by_group(self, x):
        return x.reshape(-1)[self.cells].double()

    def raster(self, values):
        out = torch.full((self.shape[0] * self.shape[1],), float("nan"), dtype=torch.float64, device=values.device)
        out[self.cells] = values
        return out.view(self.shape)


def _rule(op, total, other):
    if op == "accu":
        return total.clone(), None
    if op == "accu_threshold":
        return (total - other).clamp_(min=0.0), torch.minimum(total, other)
    if op == "accu_fraction":
        flux = other * total
        return flux, total - flux
    if op == "accu_capacity":
        return torch.minimum(total, other), (total - other).clamp_(min=0.0)
    stays = total < other
    return total.masked_fill(stays, 0.0), total.masked_fill(~stays, 0.0)


def _route(op, code, material, other):
    s = Sweep(code)
    m = s.by_group(material)
    o = s.by_group(other) if other is not None else None
    total = torch.cat([m, m.new_zeros(1)])
    out, rest = torch.empty_like(m), torch.empty_like(m) if o is not None else None
    for k in range(s.most + 1):
        at = slice(s.first[k], s.first[k + 1])
        flux, stay = _rule(op, total[at], None if o is None else o[at])
        out[at] = flux
        if rest is not None:
            rest[at] = stay
        total.index_add_(0, s.to[at], flux)
    return s.raster(out), None if rest is None else s.raster(rest)


def _discharge(k, alpha, known):
    """The root of k Q + alpha Q^(3/5) = known, by Newton's method on y = Q^(1/5) from above."""
    y = torch.minimum((known / k) ** 0.2, (known / alpha) ** (1.0 / 3.0))
    for _ in range(8):
        y2 = y * y
        f = y * y2 * (k * y2 + alpha) - known
        df = y2 * (5.0 * k * y2 + 3.0 * alpha)
        y = y - torch.where(df > 0.0, f / df, torch.zeros_like(f))
    return y ** 5


def _wave(code, discharge, rain, alpha, steps):
    """All steps at once: a cell does a step one round after the cells that drain into it."""
    s = Sweep(code)
    k = TIME_STEP / CHANNEL_LENGTH
    q, gain, al = s.by_group(discharge), TIME_STEP * s.by_group(rain), s.by_group(alpha)
    # what has flowed in, for even and odd steps
    inflow = torch.zeros(2 * (s.n + 1), dtype=torch.float64, device=q.device)
    for r in range(s.most + steps):
        at = slice(s.first[max(0, r - steps + 1)], s.first[min(s.most, r) + 1])
        odd = ((r - s.most + s.distance[at]) & 1).long() * (s.n + 1)
        place = odd + torch.arange(at.start, at.stop, device=q.device)
        up = inflow[place]
        inflow[place] = 0.0
        q[at] = _discharge(k, al[at], k * up + al[at] * q[at] ** BETA + gain[at])
        inflow.index_add_(0, odd + s.to[at], q[at])
    return s.raster(q)


def _neighbours(code, material):
    rows, cols = code.shape
    down = downstream_index(code)
    here = torch.arange(rows * cols, device=code.device)
    m = material.reshape(-1).double()
    moves = down != here
    up = torch.zeros_like(m).index_add_(0, down[moves], m[moves])
    return up.view(rows, cols), torch.where(moves, m[down], torch.zeros_like(m)).view(rows, cols)


def exact(case, seed):
    op = case["op"]
    n = case["rows"] * case["cols"]
    if op in ("kinematic_wave", "ensemble") and (n * case["steps"] > 2 ** 28 or n > 2 ** 24):
        return None  # minutes
    x = _inputs(case, seed)
    if op in ("kinematic_wave", "ensemble"):
        return _wave(x["code"], x["discharge"], x["rain"], x["alpha"], case["steps"])
    if op == "neighbours":
        return list(_neighbours(x["code"], x["material"]))
    if op == "new_raster":
        return [None, _route("accu", steepest_descent(x["elevation"]), x["material"], None)[0]]
    out, rest = _route(op, x["code"], x["material"], x.get("other"))
    return out if rest is None else [out, rest]
