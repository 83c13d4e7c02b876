"""Performance cases of the curvelet engine: edge maps through its public entry points.

A case is one call (or one short sequence of calls) that a program of this
framework makes, on seeded synthetic edge maps: circular arcs and straight
segments sampled once per pixel with position and orientation noise, and uniform
clutter. Image sizes and densities are those of the benchmark's workloads.

  call "run"       Engine.run: a host array of edges in, curvelets in host memory out
  call "device"    Engine.run_device: edges a producer left on the GPU, curvelets kept there
  call "batch"     Engine.run_batch on a resident ragged batch, each map's curvelets taken out
  call "maps"      Engine.run_maps: many maps, host to host
  call "contours"  Engine.run_contours: curvelets, link graph, fragments and polyarcs
  call "staged"    build_neighbor_csr_graph, then CurveletGPU's two stages
"""
import math

import numpy as np
import torch

import curvelet_construction_on_gpu_b200 as cvl

# image sizes of the ragged mixes, and the smallest one
IMAGES = ((640, 480), (1280, 720), (1920, 1080), (3840, 2160))
PI = cvl.M_PI

# Means over these generators' maps, for work(): curvelets and neighbour pairs per edge.
CURVELETS_PER_EDGE = 2.2
PAIRS_PER_EDGE = 9.5


def _case(name, call, edges, width, height, **more):
    c = {"name": name, "call": call, "edges": edges, "width": width, "height": height, "maps": 1, "clutter": 0.2,
         "short_arcs": 0.0, "group_max_sz": 4, "scalar": "double"}
    c.update(more)
    return c


def listed():
    return [
        # one crop of an image, as an interactive tool or a tracker asks for it: latency only
        _case("tiny_run", "run", 517, 120, 90, clutter=0.1),
        # one small image from host to host, the command line's everyday map
        _case("small_run", "run", 4454, 480, 320, clutter=0.1),
        # one 1920x1080 map from host to host
        _case("hd_run", "run", 242059, 1920, 1080),
        # the same in the --float mode
        _case("hd_run_float", "run", 242059, 1920, 1080, scalar="float"),
        # a detector on the same GPU hands its edges over, a GPU consumer takes the curvelets
        _case("hd_device", "device", 242059, 1920, 1080),
        # the same with longer chains than the default (group_max_sz 7)
        _case("hd_device_chains7", "device", 180001, 1920, 1080, group_max_sz=7),
        # a dense 3840x2160 map: short high-curvature arcs and much clutter
        _case("dense4k_device", "device", 734971, 3840, 2160, clutter=0.4, short_arcs=0.5),
        # the largest single maps of the ragged mix
        _case("large4k_device", "device", 3650003, 3840, 2160),
        # a stream of small images, resident as one ragged batch
        _case("small_batch", "batch", 187003, 640, 480, maps=30, clutter=0.1),
        # the ragged mix (image sizes and densities vary over the maps), host to host
        _case("mixed_maps", "maps", 8000003, 0, 0, maps=24),
        # the downstream stages along with the curvelets
        _case("hd_contours", "contours", 242059, 1920, 1080),
        # the reference's template API, stage by stage
        _case("mid_staged", "staged", 30011, 960, 540, clutter=0.1),
    ]


def draw(rng):
    """One more case: a call, an image and a size of the listed ranges."""
    call = rng.choice(("run", "run", "device", "device", "device", "batch", "maps", "contours", "staged"))
    lo, hi = {"run": (300, 400000), "device": (2000, 3600000), "batch": (20000, 900000), "maps": (300000, 6000000),
              "contours": (4000, 300000), "staged": (4000, 60000)}[call]
    edges = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    maps = rng.randint(2, 30) if call in ("batch", "maps") else 1
    # curve pixels per image pixel: 0.02 to 0.44, as over the ragged mix
    width, height = 0, 0
    if call != "maps":
        area = edges / maps / math.exp(rng.uniform(math.log(0.03), math.log(0.4)))
        width = max(40, int(math.sqrt(area * rng.uniform(1.2, 1.8))))
        height = max(30, int(area / width))
    return {"call": call, "edges": edges, "width": width, "height": height, "maps": maps,
            "clutter": rng.choice((0.1, 0.2, 0.4)), "short_arcs": rng.choice((0.0, 0.0, 0.5)),
            "group_max_sz": rng.choice((4, 4, 4, 5, 7)),
            "scalar": "float" if call == "run" and rng.random() < 0.25 else "double"}


# ---------------------------------------------------------------------------
# edge maps
# ---------------------------------------------------------------------------
def _shape(case):
    """(edges, width, height) of each map. The ragged mix takes the image sizes in
    turn and a density factor between 1/4 and 4, spread evenly over its logarithm."""
    n, total = case["maps"], case["edges"]
    if case["call"] != "maps":
        cut = [total * k // n for k in range(n + 1)]
        return [(cut[k + 1] - cut[k], case["width"], case["height"]) for k in range(n)]
    sizes = [IMAGES[k % 4] for k in range(n)]
    weight = [w * h * 4.0 ** (2.0 * ((k * 0.6180339887498949 + 0.5) % 1.0) - 1.0) for k, (w, h) in enumerate(sizes)]
    ends = np.floor(np.cumsum(weight) * (total / sum(weight)) + 0.5).astype(int)
    ends[-1] = total
    counts = np.diff(np.concatenate([[0], ends]))
    return [(int(c), w, h) for c, (w, h) in zip(counts, sizes)]


def _edge_map(n, width, height, clutter, short_arcs, gen, dev):
    """n edges of one map: rows x, y, theta, strength (float64)."""
    def uni(lo, hi, k):
        return torch.rand(k, generator=gen, device=dev, dtype=torch.float64) * (hi - lo) + lo

    def normal(k, sigma):
        return torch.randn(k, generator=gen, device=dev, dtype=torch.float64) * sigma

    on_curves = n - int(round(n * clutter / (1.0 + clutter)))
    longest = min(400.0, 0.9 * max(width, height))
    k = max(4, int(2.2 * on_curves / (20.0 + longest)) * 2 + 4)  # curves: more samples than needed
    radius = torch.exp(uni(math.log(4.0), math.log(longest), k))
    length = uni(min(20.0, longest / 2), longest, k)
    kind = uni(0.0, 1.0, k)
    short = kind < short_arcs
    radius = torch.where(short, uni(3.0, 15.0, k), radius)
    length = torch.where(short, uni(10.0, 60.0, k), length)
    straight = kind > 1.0 - 0.2 * (1.0 - short_arcs)
    length = torch.where(straight, length, torch.minimum(length, 2.0 * PI * radius)).floor().clamp_(min=2.0)
    cx, cy, phi = uni(0.0, width, k), uni(0.0, height, k), uni(0.0, 2.0 * PI, k)
    sense = torch.where(uni(0.0, 1.0, k) < 0.5, -1.0, 1.0).to(torch.float64)
    reps = length.to(torch.int64)
    at = torch.repeat_interleave(torch.arange(k, device=dev), reps)
    s = torch.arange(at.numel(), device=dev, dtype=torch.float64) - (torch.cumsum(reps, 0) - reps)[at].to(torch.float64)
    off, turn = normal(at.numel(), 0.1), normal(at.numel(), 0.03)
    a = phi[at] + sense[at] * s / radius[at]
    r = radius[at] + off
    line = straight[at]
    c0, s0 = torch.cos(phi[at]), torch.sin(phi[at])
    x = cx[at] + torch.where(line, s * c0 - off * s0, r * torch.cos(a))
    y = cy[at] + torch.where(line, s * s0 + off * c0, r * torch.sin(a))
    th = torch.where(line, phi[at], a + sense[at] * (PI / 2.0)) + turn
    keep = torch.nonzero((x >= 0) & (x < width) & (y >= 0) & (y < height)).squeeze(1)[:on_curves]
    m = n - keep.numel()
    x = torch.cat([x[keep], uni(0.0, width, m)])
    y = torch.cat([y[keep], uni(0.0, height, m)])
    th = torch.cat([th[keep], uni(-PI, PI, m)])
    strength = torch.cat([uni(2.0, 20.0, keep.numel()), uni(1.0, 5.0, m)])
    return torch.stack([x, y, th, strength], dim=1)


def _placed(e, width, height, gen, scalar, call):
    """The map turned by quarter turns, mirrored or not, moved by whole pixels, its rows
    starting anywhere: the same scene in another frame. Neighbourhoods and bundles are
    symmetric under these, so every seed of a case has as many curvelets (arrays of one
    shape), with other coordinates, angles, ids and rows. Two cases take a part of it:
    32-bit rounding is symmetric under no move, and the contours' fragments and polyarcs
    follow the order of the rows and the axes."""
    turns, mirror, dx, dy = (int(torch.randint(0, k, (1,), generator=gen)) for k in (4, 2, 512, 512))
    first = int(torch.randint(0, e.shape[0], (1,), generator=gen))
    x, y, th, strength = e.unbind(1)
    if call != "contours":
        if mirror:
            x, th = width - x, PI - th
        for _ in range(turns):  # (x, y) -> (height - y, x)
            x, y, th, width, height = height - y, x, th + PI / 2.0, height, width
    th = PI - torch.remainder(PI - th, 2.0 * PI)  # (-pi, pi]
    if scalar == "double":
        e = torch.stack([x + dx, y + dy, th, strength], dim=1)
    else:
        e = torch.stack([e[:, 0], e[:, 1], PI - torch.remainder(PI - e[:, 2], 2.0 * PI), strength], dim=1)
    return e if call == "contours" else torch.roll(e, first, 0)


def _inputs(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    scene = torch.Generator(device=dev)
    scene.manual_seed(case["edges"] * 64 + case["maps"])
    place = torch.Generator()
    place.manual_seed(int(seed))
    return [_placed(_edge_map(n, w, h, case["clutter"], case["short_arcs"], scene, dev), w, h, place,
                    case["scalar"], case["call"]) for n, w, h in _shape(case)]


def prepare(case, seed):
    maps = _inputs(case, seed)
    state = {"case": case, "engine": cvl.default_engine(), "params": cvl.CurveletParams(group_max_sz=case["group_max_sz"])}
    counts = np.array([m.shape[0] for m in maps], np.int32)
    if case["call"] == "device":
        state["edges"] = maps[0].contiguous()
        state["ready"] = torch.cuda.Event()
        state["ready"].record()
        return state
    host = torch.cat(maps).cpu().numpy()
    if case["call"] == "batch":
        state["batch"] = state["engine"].upload_ragged(host, counts)
    elif case["call"] == "maps":
        # a program that streams maps keeps them in page-locked memory
        state["edges"], state["counts"] = torch.from_numpy(host).pin_memory().numpy(), counts
    else:
        state["edges"] = host.astype(np.float32) if case["scalar"] == "float" else host
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
class _OnDevice:
    """A device buffer of the engine, for torch.as_tensor."""

    def __init__(self, ptr, shape, kind):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 3}


def run(state):
    case, eng, params = state["case"], state["engine"], state["params"]
    call = case["call"]
    if call == "run":
        r = eng.run(state["edges"], params, scalar=case["scalar"])
        return {"chains": r.chains, "info": r.info, "valid_pairs": r.valid_pairs}
    if call == "device":
        e = state["edges"]
        eng.run_device(e.data_ptr(), e.shape[0], e.shape[1], params, ready_event=state["ready"].cuda_event, to_host=False)
        d = eng.device_results()
        c, w = d["num_curvelets"], d["chain_width"]
        if c == 0:
            return {"curvelets": 0}
        # (a consumer waits for d["done_event"] on its own stream)
        return {"chains": torch.as_tensor(_OnDevice(d["chains"], (c, w), "<i4"), device="cuda"),
                "info": torch.as_tensor(_OnDevice(d["info"], (c, 10), "<f8"), device="cuda")}
    if call == "batch":
        b = eng.run_batch(state["batch"], params)
        taken = [b.take_map(m) for m in range(case["maps"])]
        return {"maps": [{"chains": r.chains, "info": r.info} for r in taken]}
    if call == "maps":
        got = eng.run_maps(state["edges"], params, counts=state["counts"])
        return {"maps": [{"chains": r.chains, "info": r.info} for r in got]}
    if call == "contours":
        r, c = eng.run_contours(state["edges"], params, cvl.ContourParams(fit_polyarcs=True))
        return {"chains": r.chains, "info": r.info, "links": c.links, "frag_offsets": c.frag_offsets,
                "frag_ids": c.frag_ids, "poly_offsets": c.poly_offsets, "poly_ids": c.poly_ids, "poly_info": c.poly_info}
    e = state["edges"]
    graph = cvl.GPUNeighborGraph()
    cvl.build_neighbor_csr_graph(e.shape[0], e.shape[1], e, params.nrad, 3, params.max_candidates, 1, graph, engine=eng)
    cur = cvl.CurveletGPU(e.shape[0], e.shape[1], graph, params.dx, params.dt_deg / 180.0 * PI, params.sx, params.st,
                          params.max_k, params.group_max_sz, 1, e, params.nrad, engine=eng)
    formed = cvl.CurveletFormationResult()
    cur.form_pairwise_bundles(formed)
    cur.build_curvelets_greedy()
    return {"offsets": graph.neighbor_offsets, "ids": graph.neighbor_ids, "dist2": graph.neighbor_dist2,
            "valid_pairs": formed.valid_pairs, "chains": cur._edge_chain_final, "info": cur.curvelet_info_rows}


def work(case):
    """Edges in (32 B), curvelets out (10 doubles and a chain row); and the arithmetic of
    the pairwise bundles, 20 operations for each of a pair's 63 cells."""
    n = case["edges"]
    edge = 16 if case["scalar"] == "float" else 32
    return {"bytes": n * edge + CURVELETS_PER_EDGE * n * (80 + 4 * (case["group_max_sz"] + 1)),
            "flops": PAIRS_PER_EDGE * n * 63 * 20.0}


# ---------------------------------------------------------------------------
# the same in 64-bit torch operations
# ---------------------------------------------------------------------------
def _neighbours(e, nrad=3.5, w=3):
    """CSR of one map: (offsets, ids, d2), each list by (distance, window-scan order)."""
    n = e.shape[0]
    x, y = e[:, 0], e[:, 1]
    cx, cy = torch.round(x).to(torch.int64), torch.round(y).to(torch.int64)
    cx, cy = cx - cx.min() + w, cy - cy.min() + w
    stride = int(cx.max()) + w + 2
    key, order = torch.sort(cy * stride + cx, stable=True)
    anchors, others = [], []
    me = torch.arange(n, device=e.device)
    for dy in range(-w, w + 1):
        base = (cy + dy) * stride + cx
        lo, hi = torch.searchsorted(key, base - w), torch.searchsorted(key, base + w, right=True)
        cnt = hi - lo
        a = torch.repeat_interleave(me, cnt)
        k = torch.arange(a.numel(), device=e.device) - (torch.cumsum(cnt, 0) - cnt)[a] + lo[a]
        anchors.append(a)
        others.append(order[k])
    a, b = torch.cat(anchors), torch.cat(others)
    d2 = (x[a] - x[b]) * (x[a] - x[b]) + (y[a] - y[b]) * (y[a] - y[b])
    keep = (a != b) & (d2 <= nrad * nrad)
    a, b, d2 = a[keep], b[keep], d2[keep]
    o = torch.sort(d2, stable=True)[1]  # (anchor, distance); the scan order stays where both are equal
    o = o[torch.sort(a[o], stable=True)[1]]
    a, b, d2 = a[o], b[o], d2[o]
    off = torch.zeros(n + 1, dtype=torch.int64, device=e.device)
    off[1:] = torch.cumsum(torch.bincount(a, minlength=n), 0)
    return off, a, b, d2


def _to_2pi(t):
    return torch.remainder(t, 2.0 * PI)


def _curvelets(e, p, chunk=20000):
    """(offsets, ids, d2, valid pairs, chains, info) of one map; None where a list is cut."""
    dev = e.device
    off, pa, pb, d2 = _neighbours(e, p.nrad)
    n = e.shape[0]
    if int((off[1:] - off[:-1]).max()) >= p.max_candidates:
        return None
    dt = p.dt_deg / 180.0 * PI
    P, Q = 2 * math.floor(p.dx / p.sx + 0.5) + 1, 2 * math.floor(dt / p.st + 0.5) + 1
    gi = torch.arange(P, device=dev, dtype=torch.float64).repeat_interleave(Q)
    gj = torch.arange(Q, device=dev, dtype=torch.float64).repeat(P)
    ox, ot = p.sx * (gi - (P - 1) / 2.0), p.st * (gj - (Q - 1) / 2.0)
    rank = torch.argsort(torch.argsort(ox * ox + ot * ot, stable=True))
    gms, inf = p.group_max_sz, float("inf")
    valid_pairs, rows, infos = 0, [], []
    for a0 in range(0, n, chunk):
        a1 = min(n, a0 + chunk)
        lo, hi = int(off[a0]), int(off[a1])
        a, b = pa[lo:hi], pb[lo:hi]
        DX, DY = (e[a, 0] - e[b, 0])[:, None], (e[a, 1] - e[b, 1])[:, None]
        T2, T0 = e[a, 2][:, None], e[b, 2][:, None]
        tm, tp = T0 - dt, T0 + dt
        R2 = DX * DX + DY * DY
        close = R2 < 4 * p.dx * p.dx
        first = DX * torch.cos(T2) + DY * torch.sin(T2) < 0
        T2t = T2 + ot
        tt = torch.sin(T2t) * DX - torch.cos(T2t) * DY
        eq = R2 - 2.0 * ox * tt - p.dx * p.dx + ox * ox
        k_lo, k_hi = 2.0 * (tt - ox - p.dx) / eq, 2.0 * (tt - ox + p.dx) / eq
        sm, sp = torch.sin(T2t - tm), torch.sin(T2t - tp)
        km = sm / (-sm * ox + torch.cos(tm) * DX + torch.sin(tm) * DY)
        kp = sp / (-sp * ox + torch.cos(tp) * DX + torch.sin(tp) * DY)
        # (fmax and fmin: a 0/0 bounds nothing)
        bmin = torch.fmax(torch.fmax(torch.full_like(k_lo, -p.max_k), k_lo), torch.where(first, km, kp))
        bmax = torch.fmin(torch.fmin(torch.full_like(k_hi, p.max_k), k_hi), torch.where(first, kp, km))
        bmin, bmax = torch.where(close, -p.max_k, bmin), torch.where(close, p.max_k, bmax)
        valid = (bmax > bmin).any(1) | close[:, 0]
        valid_pairs += int(valid.sum())
        ahead = torch.cos(torch.atan2(-DY, -DX) - T2)[:, 0]
        pick = torch.nonzero(valid & (ahead != 0)).squeeze(1)
        # lists: (anchor, ahead first); a stable sort keeps the neighbour order within a list
        lid, o = torch.sort(2 * (a[pick] - a0) + (ahead[pick] < 0).to(torch.int64), stable=True)
        pick = pick[o]
        cnt = torch.bincount(lid, minlength=2 * (a1 - a0))
        start = (torch.cumsum(cnt, 0) - cnt)[lid]
        ns, pos = cnt[lid], torch.arange(pick.numel(), device=dev) - start
        cmin, cmax = bmin[pick].clone(), bmax[pick].clone()
        length = torch.ones_like(pos)
        chain = torch.full((pick.numel(), gms), -1, dtype=torch.int64, device=dev)
        for r in range(int(ns.max()) if ns.numel() else 0):
            on = torch.nonzero((r < ns) & (length < gms)).squeeze(1)
            if not on.numel():
                break
            q = pick[start[on] + r]
            lo_, hi_ = torch.maximum(cmin[on], bmin[q]), torch.minimum(cmax[on], bmax[q])
            own = pos[on] == r
            take = own | (hi_ > lo_).any(1)
            upd = take & ~own
            cmin[on[upd]], cmax[on[upd]] = lo_[upd], hi_[upd]
            at = on[take]
            chain[at, length[at]] = r
            length[at] += 1
        # first of equal chains of a list, longer than two edges
        code = lid.clone()
        for z in range(1, gms):
            code = torch.unique(code * 1025 + chain[:, z] + 1, return_inverse=True)[1]
        seen = torch.full((int(code.max()) + 1 if code.numel() else 1,), pick.numel(), dtype=torch.int64, device=dev)
        me = torch.arange(pick.numel(), device=dev)
        seen.scatter_reduce_(0, code, me, reduce="amin")
        got = torch.nonzero((seen[code] == me) & (length > 2)).squeeze(1)
        anchor, ln = a[pick[got]], length[got]
        ids = torch.full((got.numel(), gms), -1, dtype=torch.int64, device=dev)
        ids[:, 0] = anchor
        for z in range(1, gms):
            c = chain[got, z]
            ids[:, z] = torch.where(c >= 0, b[pick[(start[got] + c.clamp(min=0)).clamp(max=max(pick.numel() - 1, 0))]], -1)
        rows.append(torch.cat([anchor[:, None] + 1, ids + 1], 1))
        best = torch.where(cmax[got] > cmin[got], rank, rank.numel()).argmin(1) if got.numel() else got
        kmax, kmin = cmax[got, best], cmin[got, best]
        th = e[anchor, 2]
        theta = _to_2pi(th + ot[best])
        px, py = e[anchor, 0] - ox[best] * torch.sin(theta), e[anchor, 1] + ox[best] * torch.cos(theta)
        dist = torch.zeros_like(th)
        for z in range(gms - 1):
            u, v = ids[:, z], ids[:, z + 1].clamp(min=0)
            step = torch.sqrt((e[u, 0] - e[v, 0]) ** 2 + (e[u, 1] - e[v, 1]) ** 2)
            dist = dist + torch.where(ids[:, z + 1] >= 0, step, torch.zeros_like(step))
        quality = torch.where(dist > 0, 2.0 / (p.nrad / dist + dist / ln), torch.zeros_like(dist))
        fwd = (lid[got] % 2 == 0).to(torch.float64)
        infos.append(torch.stack([fwd, kmax, kmin, th, px, py, theta, (kmax + kmin) / 2.0, dist, quality], 1))
    return (off, pb, d2, valid_pairs, torch.cat(rows).to(torch.int32).cpu().numpy().view(np.uint32), torch.cat(infos).cpu().numpy())


def exact(case, seed):
    """What run() returns, from the formulas in 64 bits. The float mode's decisions are
    float decisions, so its rows have no 64-bit counterpart; the large maps take too
    long; the contours' links and ids are whole numbers, and polyarcs follow the
    sequential tracing of the fragments."""
    if case["scalar"] == "float" or case["edges"] > 400000:
        return None
    params = cvl.CurveletParams(group_max_sz=case["group_max_sz"])
    got = [_curvelets(e, params) for e in _inputs(case, seed)]
    if any(g is None for g in got):
        return None
    call = case["call"]
    if call in ("batch", "maps"):
        return {"maps": [{"chains": g[4], "info": g[5]} for g in got]}
    off, ids, d2, valid, chains, info = got[0]
    if call == "run":
        return {"chains": chains, "info": info, "valid_pairs": valid}
    if call == "device":
        return {"chains": chains.view(np.int32), "info": info} if len(chains) else {"curvelets": 0}
    if call == "contours":
        return {"chains": chains, "info": info, "links": None, "frag_offsets": None, "frag_ids": None,
                "poly_offsets": None, "poly_ids": None, "poly_info": None}
    return {"offsets": off.to(torch.int32).cpu().numpy(), "ids": ids.to(torch.int32).cpu().numpy(), "dist2": d2.cpu().numpy(),
            "valid_pairs": valid, "chains": chains, "info": info}
