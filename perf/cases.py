"""The framework's work as its users have it done, as cases to be timed.

A case is a dict of plain values; ``prepare`` makes what a program has in hand
before the call (snapshots on the device or in pinned host memory, output
buffers, a context), ``run`` is one pass through the public entry points, and
``exact`` gives the same outputs in 64 bits from plain torch.

The snapshots have the statistics the path meets: mean particle separation 2,
a uniform background with Plummer spheres or NFW halos in it, and a periodic
buffer shell of 8 units.  What a pass returns of each particle is what it
gives for the box's own particles, which come first in every snapshot.
"""
import ctypes
import math

import numpy as np
import torch

from asmooth_gb300 import api

K = 33  # neighbours that set the smoothing length, the particle itself among them
EXACT_MAX = 420_000  # particles up to which the all-pairs search of exact() stays within seconds
_CONTEXT = []


def listed():
    return [
        # a host program that may not allocate: one small sub-volume's smoothing lengths
        {"name": "noalloc_4k", "path": "noalloc", "n": 4099, "model": "uniform"},
        # a sub-volume of a test run: launches and host waits are most of it
        {"name": "step_16", "path": "step", "n": 16 ** 3, "model": "plummer", "ncs": "8,16"},
        # the 64^3 snapshot of Plummer spheres, side 128, in one piece
        {"name": "step_64", "path": "step", "n": 64 ** 3, "model": "plummer", "ncs": "32,64"},
        # a node-cube of side 256 whose periodic shell is built on the device
        {"name": "shell_step_128", "path": "shell_step", "n": 128 ** 3, "model": "nfw",
         "ncs": "32,64,128"},
        # the 256^3 snapshot of NFW halos, side 512: the whole step
        {"name": "step_256", "path": "step", "n": 256 ** 3, "model": "nfw", "ncs": "64,128,256"},
        # smoothing onto the periodic global mesh, with mesh sizes that no tile divides
        {"name": "global_100", "path": "global", "n": 1_000_003, "model": "nfw", "ncs": "50,101"},
        # density alone on one fine mesh
        {"name": "density_80", "path": "density", "n": 511_997, "model": "plummer", "ncs": "160"},
        # positions as 16-bit offsets from host memory, smoothed in one call
        {"name": "mixed_128", "path": "mixed", "n": 128 ** 3, "model": "nfw", "ncs": "32,64,128"},
        # particle records from host memory and back, halo particles marked
        {"name": "records_70", "path": "records", "n": 343_001, "model": "nfw", "ncs": "35,70"},
        # friends-of-friends groups and their catalogue
        {"name": "fof_128", "path": "fof", "n": 128 ** 3, "model": "nfw"},
        # a zipped snapshot from host memory: decode, shell, smoothing lengths
        {"name": "zip_64", "path": "zip", "n": 64 ** 3, "model": "plummer"},
        # several uneven cubes in one batch, new positions in every pass
        {"name": "batch_5", "path": "batch", "n": 48 ** 3, "items": 5, "model": "nfw",
         "ncs": "16,48"},
    ]


def draw(rng):
    path = rng.choice(["noalloc", "step", "step", "shell_step", "shell_step", "global", "density",
                       "mixed", "records", "fof", "zip", "batch"])

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if path == "noalloc":
        return {"path": path, "n": log_int(64, 32768), "model": rng.choice(["uniform", "plummer"])}
    top = {"step": 6_000_000, "shell_step": 4_000_000, "batch": 250_000}.get(path, 2_200_000)
    low = {"fof": 100_000, "mixed": 20_000}.get(path, 4096)
    c = {"path": path, "n": log_int(low, top), "model": rng.choice(["plummer", "nfw", "nfw"])}
    if path in ("fof", "zip"):
        return c
    side = c["n"] ** (1.0 / 3.0)
    fine = max(5, int(round(side * rng.uniform(0.6, 1.3))))  # cells of 1.5 to 3.3 units
    sizes = {fine}
    if path == "density":
        sizes = {int(fine * rng.choice([1, 2]))}
    else:
        for _ in range(rng.randrange(3)):
            sizes.add(max(4, int(fine * rng.uniform(0.2, 0.8))))
    c["ncs"] = ",".join(str(s) for s in sorted(sizes))
    if path == "batch":
        c["items"] = rng.randrange(2, 8)
    return c


# ---- snapshots ------------------------------------------------------------------


def _halo_sizes(n, model, rng):
    """Members of each halo and each halo's scale: Plummer spheres with half of
    the particles, NFW halos with 70% of them."""
    if model == "plummer":
        k = max(2, round(200 * n / 64 ** 3))
        members = rng.multinomial(n // 2, np.full(k, 1.0 / k))
        return members, np.exp(rng.uniform(np.log(0.5), np.log(4.0), k))
    k = max(4, round(5000 * n / 256 ** 3))
    mass = np.exp(rng.uniform(np.log(1e2), np.log(1e5), k))
    members = np.floor(mass / mass.sum() * 0.7 * n).astype(np.int64)
    return members, rng.uniform(4.0, 12.0, k)  # the NFW concentrations


def _snapshot(n, model, seed):
    """n particles of a periodic box: x in [0, box)^3 and v on the device, the
    box side, and the halos' centres and radii."""
    box = float(np.float32(2.0 * n ** (1.0 / 3.0)))
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    f64 = {"dtype": torch.float64, "device": "cuda", "generator": g}
    centre, radius = np.zeros((0, 3)), np.zeros(0)
    parts = []
    if model != "uniform":
        members, scale = _halo_sizes(n, model, rng)
        centre = rng.uniform(0.0, box, (len(members), 3))
        owner = torch.repeat_interleave(torch.as_tensor(members)).cuda()
        u = torch.rand(owner.numel(), **f64)
        s = torch.as_tensor(scale).cuda()[owner]
        if model == "plummer":
            r = s / torch.sqrt(u.clamp(1e-12, 1.0 - 1e-9) ** (-2.0 / 3.0) - 1.0)
            radius = 2.0 * scale
        else:
            radius = (3.0 * members / (4.0 * np.pi * 25.0)) ** (1.0 / 3.0)  # 200 x the mean, 1/8
            want = u * (torch.log1p(s) - s / (1.0 + s))
            lo, hi = torch.zeros_like(s), s.clone()
            for _ in range(40):  # the enclosed mass, inverted by bisection
                mid = 0.5 * (lo + hi)
                below = torch.log1p(mid) - mid / (1.0 + mid) < want
                lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
            r = 0.5 * (lo + hi) * torch.as_tensor(radius).cuda()[owner] / s
        d = torch.randn((owner.numel(), 3), **f64)
        d /= torch.linalg.norm(d, dim=1, keepdim=True)
        parts.append(torch.as_tensor(centre).cuda()[owner] + d * r[:, None])
    rest = n - sum(p.shape[0] for p in parts)
    parts.append(torch.rand((rest, 3), **f64) * box)
    x = torch.remainder(torch.cat(parts), box).float()
    x = x[torch.randperm(n, device="cuda", generator=g)]  # files are in no particular order
    x[x >= box] = 0.0
    v = torch.randn((n, 3), dtype=torch.float32, device="cuda", generator=g)
    return x.contiguous(), v, box, centre, radius


def _buffer(box):
    return min(8.0, box / 4.0)


def _with_shell(x, v, box, buf):
    """The particles and their periodic images within buf of the box."""
    xs, vs = [x], [v]
    for k in range(27):
        d = torch.tensor([k % 3 - 1, k // 3 % 3 - 1, k // 9 - 1], device=x.device)
        if k == 13:
            continue
        y = x - d.to(x.dtype) * box
        keep = ((y > -buf) & (y < box + buf)).all(1)
        xs.append(y[keep])
        vs.append(v[keep])
    return torch.cat(xs).contiguous(), torch.cat(vs).contiguous()


def _context():
    """The one context that a program keeps and gives its snapshots to."""
    if not _CONTEXT:
        _CONTEXT.append(api.Context(0))
    return _CONTEXT[0]


def _ncs(case):
    return [int(t) for t in case.get("ncs", "").split(",") if t]


def _zip_arrays(x, v, box, cells, v_r2i):
    """A snapshot as the four arrays of a zipped file: bytes within cells of
    side box/cells, velocities in units of 1/v_r2i, counts per cell."""
    rel = x.double() / (box / cells)
    c = rel.floor().clamp(0, cells - 1)
    off = ((rel - c) * 256.0).floor().clamp(0, 255).to(torch.uint8)
    c = c.to(torch.int64)
    cell = (c[:, 2] * cells + c[:, 1]) * cells + c[:, 0]
    cell, order = torch.sort(cell, stable=True)
    counts = torch.bincount(cell, minlength=cells ** 3)
    vq = (v[order].double() * v_r2i).round().clamp(-32768, 32767).to(torch.int16)
    return (off[order].cpu().numpy(), vq.cpu().numpy(),
            counts.clamp(max=255).to(torch.uint8).cpu().numpy(),
            counts[counts >= 255].to(torch.int32).cpu().numpy())


def _zip_geometry(n):
    cells = max(16, int(round(n ** (1.0 / 3.0))))
    return cells, 2, 64.0  # cells per dimension, their side, velocity units


# ---- a case's state ---------------------------------------------------------------


def prepare(case, seed):
    path, n = case["path"], case["n"]
    s = {"path": path, "ncs": _ncs(case)}
    if path == "batch":
        return _prepare_batch(case, seed, s)
    s["ctx"] = _context()
    x, v, box, centre, radius = _snapshot(n, case["model"], seed)
    if path == "noalloc":
        s.update(x=x, right=box, rk=torch.empty(n, device="cuda"), dens=torch.empty(n, device="cuda"))
        return s
    if path == "zip":
        cells, side, v_r2i = _zip_geometry(n)
        x = (x * ((cells * side) / box)).clamp(max=float(np.nextafter(np.float32(cells * side), np.float32(0))))
        box = float(cells * side)
        s.update(zip=_zip_arrays(x, v, box, cells, v_r2i), cells=cells, side=side, v_r2i=v_r2i)
    buf = _buffer(box)
    s.update(n=n, box=box, buf=buf, factor=buf / box, left=-buf,
             right=float(np.float32(box) + np.float32(buf)))
    xs, vs = _with_shell(x, v, box, buf)
    m = xs.shape[0]
    if path in ("shell_step", "zip"):
        room = m + n // 64 + 4096  # the shell's size comes out of the call
        s.update(x=x, v=v, rk=torch.empty(room, device="cuda"), dens=torch.empty(room, device="cuda"))
        return s
    x, v = xs, vs
    if path in ("step", "global", "density"):
        s.update(x=x, v=v, rk=torch.empty(m, device="cuda"), dens=torch.empty(m, device="cuda"))
    elif path == "fof":
        room = n // 100 + 64  # groups of 20 or more
        s.update(x=x, v=v, igrp=torch.empty(m, dtype=torch.int32, device="cuda"),
                 cat={"x": np.zeros((room, 3), np.float32), "v": np.zeros((room, 3), np.float32),
                      "nfof": np.zeros(room, np.int32)})
    elif path == "mixed":
        s.update(_quantised(x, s["left"], s["right"]))
        s["v"] = api.host_array((m, 3))
        s["v"][:] = v.cpu().numpy()
        s["rk"], s["dens"] = api.host_array(m), api.host_array(m)
        s["meshes"] = [api.host_array(6 * nc ** 3) for nc in s["ncs"]]
    elif path == "records":
        s["p"] = api.host_array(m, api.PARTICLE_DTYPE)
        s["p"]["x"], s["p"]["v"] = x.cpu().numpy(), v.cpu().numpy()
        s["out"] = api.host_array(m, api.PARTICLE_DTYPE)
        s["halos"] = api.make_halos(centre, radius, np.maximum(radius, 1.0) ** 3 * 200.0)
    else:
        raise ValueError(path)
    return s


def _quantised(x, left, right):
    """16-bit offsets in cells of 4 units, in pinned host memory."""
    size = 4.0
    grid = int(math.ceil((right - left) / size))
    while np.float32(left) + np.float32(size) * np.float32(grid) < np.float32(right):
        grid += 1
    rel = (x.double() - left) / size
    c = rel.floor().clamp(0, grid - 1)
    off = ((rel - c) * 65536.0).floor().clamp(0, 65535).to(torch.int32)
    c = c.to(torch.int64)
    cell = api.host_array(x.shape[0], np.int32)
    cell[:] = ((c[:, 2] * grid + c[:, 1]) * grid + c[:, 0]).cpu().numpy()
    o = api.host_array(tuple(x.shape), np.uint16)
    o[:] = off.cpu().numpy().astype(np.uint16)
    return {"cell": cell, "off": o, "grid": grid, "size": size}


class _Item:
    """What Batch needs to know of one cube."""

    def __init__(self, x, v, n_local, box, buf):
        self.x, self.v, self.n, self.n_local, self.boxsize = x, v, x.shape[0], n_local, box
        self.left, self.right = -buf, float(np.float32(box) + np.float32(buf))


def _batch_items(case, seed):
    """Uneven cubes: particle counts within a quarter of the case's n, as the
    clustering of neighbouring node-cubes makes them."""
    items = []
    for i in range(case["items"]):
        n = int(case["n"] * (0.75 + 0.5 * ((0.31 + 0.618034 * i) % 1.0)))
        x, v, box, _, _ = _snapshot(n, case["model"], seed * 64 + i)
        x, v = _with_shell(x, v, box, _buffer(box))
        items.append((x, v, n, box, _buffer(box)))
    return items


def _prepare_batch(case, seed, s):
    items = _batch_items(case, seed)
    s["ctx"] = api.Context(0)  # a batch has its context to itself
    s["items"] = [(x, v) for x, v, *_ in items]
    s["n"] = [n for _, _, n, _, _ in items]
    s["batch"] = api.Batch(s["ctx"], [_Item(x.cpu().numpy(), v.cpu().numpy(), n, box, buf)
                                      for x, v, n, box, buf in items], s["ncs"], -1)
    s["rk"] = [api.host_array(x.shape[0]) for x, _ in s["items"]]
    s["dens"] = [api.host_array(x.shape[0]) for x, _ in s["items"]]
    s["meshes"] = [[api.host_array(6 * nc ** 3) for nc in s["ncs"]] for _ in items]
    s["totals"] = [np.zeros(2 * len(s["ncs"])) for _ in items]
    return s


# ---- one pass ----------------------------------------------------------------------


class _DeviceArray:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (ptr, False),
                                         "version": 3}


def _meshes(ctx, ncs, channels=6):
    return [torch.as_tensor(_DeviceArray(ctx.mesh_device_ptr(k), channels * nc ** 3), device="cuda")
            for k, nc in enumerate(ncs)]


def run(state):
    return _RUN[state["path"]](state)


def _run_noalloc(s):
    s["dens"].zero_()
    rc = s["ctx"].lib.asg_neighbor_search_noalloc(
        ctypes.c_void_p(s["x"].data_ptr()), s["x"].shape[0], 0.0, s["right"],
        ctypes.c_void_p(s["rk"].data_ptr()), ctypes.c_void_p(s["dens"].data_ptr()), None)
    if rc:
        raise RuntimeError(f"asg_neighbor_search_noalloc: {rc}")
    return {"rk": s["rk"], "dens": s["dens"]}


def _smooth_loaded(s, **how):
    ctx = s["ctx"]
    ctx.run_neighbor_search()
    totals = ctx.run_deposit(s["box"], s["ncs"], -1, **how)
    ctx.store_fields_device(s["rk"].data_ptr(), s["dens"].data_ptr())
    return {"rk": s["rk"][:s["n"]], "dens": s["dens"][:s["n"]], "totals": totals,
            "meshes": _meshes(ctx, s["ncs"], 1 if how.get("density_only") else 6)}


def _load_device(s):
    s["ctx"].load_particles_device(s["x"].data_ptr(), s["x"].shape[0], s["left"], s["right"],
                                   s["v"].data_ptr())


def _run_step(s):
    _load_device(s)
    return _smooth_loaded(s)


def _run_global(s):
    _load_device(s)
    return _smooth_loaded(s, periodic=True)


def _run_density(s):
    _load_device(s)
    return _smooth_loaded(s, density_only=True)


def _run_shell_step(s):
    m, kept = s["ctx"].load_periodic_cube_device(s["x"].data_ptr(), s["n"], s["box"], s["factor"],
                                                 s["v"].data_ptr())
    _check_room(s, m)
    return {"n": m, "kept": kept, **_smooth_loaded(s)}


def _check_room(s, m):
    if m > s["rk"].shape[0]:
        raise RuntimeError("the shell is larger than the buffers for its results")


def _run_mixed(s):
    rk, dens, meshes, totals = s["ctx"].smooth_quantised(
        s["cell"], s["off"], s["v"], s["left"], s["right"], s["size"], s["grid"], s["box"],
        s["ncs"], -1, s["meshes"], s["rk"], s["dens"])
    return {"rk": rk[:s["n"]], "dens": dens[:s["n"]], "meshes": meshes, "totals": totals}


def _run_records(s):
    ctx = s["ctx"]
    ctx.load_particles(s["p"], s["left"], s["right"])
    ctx.run_neighbor_search()
    np_halo, m_halo = ctx.run_mark_halos(s["halos"])
    totals = ctx.run_deposit(s["box"], s["ncs"], -1)
    p = ctx.store_particles(s["out"])[:s["n"]]
    return {"rk": p["rk"], "dens": p["dens"], "igrp": p["igrp"], "np_halo": np_halo,
            "m_halo": m_halo, "totals": totals, "meshes": _meshes(ctx, s["ncs"])}


def _run_fof(s):
    ctx = s["ctx"]
    _load_device(s)
    groups = ctx.run_fof(0.4)
    halos = ctx.run_remove_small_groups(groups)
    cat = ctx.run_fof_halos(halos, s["box"])
    ctx.store_fields_device(0, 0, s["igrp"].data_ptr())
    for k, a in s["cat"].items():
        a[:len(cat)] = cat[k]
    return {"groups": groups, "halos": halos, "igrp": s["igrp"][:s["n"]], **s["cat"]}


def _run_zip(s):
    ctx = s["ctx"]
    z0, z1, z2, z3 = s["zip"]
    ctx.decode_zip(z0, z1, z2, z3, len(z0), s["cells"], s["side"], s["v_r2i"])
    m, kept = ctx.load_decoded_periodic(s["box"], s["factor"])
    _check_room(s, m)
    ctx.run_neighbor_search()
    ctx.store_fields_device(s["rk"].data_ptr(), s["dens"].data_ptr())
    return {"n": m, "kept": kept, "rk": s["rk"][:s["n"]], "dens": s["dens"][:s["n"]]}


def _run_batch(s):
    b, lib = s["batch"], s["ctx"].lib
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    host = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    for i, (x, v) in enumerate(s["items"]):
        if lib.asg_batch_set_item(b.h, i, ptr(x), ptr(v), 1):
            raise RuntimeError("asg_batch_set_item")
    b.run()
    for i in range(len(s["items"])):
        meshes = (ctypes.c_void_p * len(s["ncs"]))(*[m.ctypes.data for m in s["meshes"][i]])
        if lib.asg_batch_get(b.h, i, host(s["rk"][i]), host(s["dens"][i]), meshes,
                             host(s["totals"][i])):
            raise RuntimeError("asg_batch_get")
    return {"rk": [a[:n] for a, n in zip(s["rk"], s["n"])],
            "dens": [a[:n] for a, n in zip(s["dens"], s["n"])],
            "meshes": s["meshes"], "totals": s["totals"]}


_RUN = {"noalloc": _run_noalloc, "step": _run_step, "shell_step": _run_shell_step,
        "global": _run_global, "density": _run_density, "mixed": _run_mixed,
        "records": _run_records, "fof": _run_fof, "zip": _run_zip, "batch": _run_batch}


# ---- what a pass cannot do without ----------------------------------------------------


def work(case):
    path, n = case["path"], case["n"]
    count = case.get("items", 1)
    box = 2.0 * n ** (1.0 / 3.0)
    with_shell = n * (1.0 + 2.0 * _buffer(box) / box) ** 3
    m = n if path == "noalloc" else with_shell
    # the particles an exact search looks at: those in the cube that encloses
    # the sphere of the 33 nearest; 8 operations each, 14 for a kernel weight
    search = m * (8 * K * 6 / math.pi + 14 * (K - 1))
    read = {"noalloc": 12 * n, "shell_step": 24 * n, "mixed": 22 * m, "records": 36 * m,
            "zip": 9 * n + n}.get(path, 24 * m)
    if path == "fof":
        # a pair test with every friend, of which the linking length leaves a
        # handful at the mean density and about ten in a halo
        return {"bytes": read + 4 * m, "flops": 8 * 10 * m}
    wrote = 36 * m if path == "records" else 8 * m
    cells = sum(nc ** 3 for nc in _ncs(case))
    meshes = 4 * cells * (1 if path == "density" else 6)
    # at least one cell per particle and mesh: 12 operations for its channels
    deposit = m * len(_ncs(case)) * (2 if path == "density" else 12)
    return {"bytes": count * (read + wrote + meshes), "flops": count * (search + deposit)}


# ---- the same outputs in 64 bits --------------------------------------------------------


def _knn64(x):
    """Smoothing length and density of every particle, from all pairs: the 33
    nearest by (distance, index), the 32 nearest given the tent weight."""
    n = x.shape[0]
    x = x.double()
    rk = torch.empty(n, dtype=torch.float64, device=x.device)
    dens = torch.zeros(n, dtype=torch.float64, device=x.device)
    step = max(1, 200_000_000 // n)
    for a in range(0, n, step):
        q = x[a:a + step]
        d2 = torch.zeros((q.shape[0], n), dtype=torch.float64, device=x.device)
        for k in range(3):
            t = q[:, k:k + 1] - x[None, :, k]
            d2.addcmul_(t, t)
        del t
        d, i = torch.topk(d2, min(n, K + 31), dim=1, largest=False, sorted=True)
        del d2
        # ties in index order
        i, at = torch.sort(i, dim=1)
        d = torch.gather(d, 1, at)
        d, at = torch.sort(d, dim=1, stable=True)
        i = torch.gather(i, 1, at)[:, :K - 1]
        h = d[:, K - 1].sqrt()
        rk[a:a + step] = h
        w = (1.0 - (x[i] - q[:, None, :]).abs() / h[:, None, None]).prod(2) / h[:, None] ** 3
        dens.index_add_(0, i.reshape(-1), w.reshape(-1))
    return rk, dens


def _tent(t):
    """The integral of the unit tent from -inf to t, less a half."""
    t = t.clamp(-1.0, 1.0)
    return t - 0.5 * t * t.abs()


def _mesh64(x, v, dens, h, halo, box, nc, periodic=False, density_only=False):
    """Every particle's tent kernel integrated over the cells it reaches:
    n | halo | c | v of the mesh, and the sums of n and halo."""
    x, v = x.double(), v.double()
    if periodic:
        inside = ((x >= 0) & (x < box)).all(1)
        x, v, dens, h, halo = x[inside], v[inside], dens[inside], h[inside], halo[inside]
    dx = box / nc
    first = ((x - h[:, None]) / dx).floor().long()
    last = ((x + h[:, None]) / dx).floor().long()
    if not periodic:
        first, last = first.clamp(min=0), last.clamp(max=nc - 1)
    out = torch.zeros((6, nc ** 3), dtype=torch.float64, device=x.device)
    # particles by the widest of their ranges, so that each goes through its own cells
    span = (last - first + 1).clamp(min=0)
    live = (span > 0).all(1)
    wide = span.max(1).values
    lo = 0
    for hi in (1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 128, 256, 512):
        s = torch.nonzero(live & (wide > lo) & (wide <= hi)).flatten()
        lo = hi
        if not s.numel():
            continue
        for part in s.split(max(1, 40_000_000 // hi ** 3)):
            ws, cs = [], []
            for a in range(3):
                c = first[part, a, None] + torch.arange(hi, device=x.device)
                e = (c * dx - x[part, a, None]) / h[part, None]
                w = _tent(e + dx / h[part, None]) - _tent(e)
                w = torch.where(c <= last[part, a, None], w, torch.zeros_like(w))
                ws.append(w)
                cs.append(c.remainder(nc) if periodic else c.clamp(0, nc - 1))
            w = (ws[2][:, :, None, None] * ws[1][:, None, :, None] * ws[0][:, None, None, :]).flatten()
            c = ((cs[2][:, :, None, None] * nc + cs[1][:, None, :, None]) * nc
                 + cs[0][:, None, None, :]).flatten()
            k = hi ** 3
            hal = halo[part].double().repeat_interleave(k)
            m = w * (1.0 - hal)
            out[0].index_add_(0, c, m)
            if density_only:
                continue
            out[1].index_add_(0, c, w * hal)
            out[2].index_add_(0, c, m * dens[part].repeat_interleave(k))
            for a in range(3):
                out[3 + a].index_add_(0, c, m * v[part, a].repeat_interleave(k))
    totals = torch.stack([out[0].sum(), out[1].sum()])
    if density_only:
        return out[0], totals
    return torch.cat([out[:3].reshape(-1), out[3:].T.reshape(-1)]), totals


def _meshes64(x, v, dens, h, halo, box, ncs, **how):
    got = [_mesh64(x, v, dens, h, halo, box, nc, **how) for nc in ncs]
    return [m for m, _ in got], torch.stack([t for _, t in got])


def _shell64(x, box, buf):
    """The particles, then their images grouped by (bin of the particle, which
    face, edge or corner it is sent across), in the order of the interior."""
    b = (x >= buf).long() + (x > box - buf).long()
    b = b[:, 0] + 3 * b[:, 1] + 9 * b[:, 2]
    parts, source = [x], [torch.arange(x.shape[0], device=x.device)]
    for i in range(27):
        s = torch.nonzero(b == i).flatten()
        for j in range(27):
            to = [j % 3, j // 3 % 3, j // 9]
            at = [i % 3, i // 3 % 3, i // 9]
            if 13 in (i, j) or not all(t in (1, a) for t, a in zip(to, at)):
                continue
            parts.append(x[s] - (torch.tensor(to, device=x.device).double() - 1.0) * box)
            source.append(s)
    x, source = torch.cat(parts), torch.cat(source)
    keep = ((x > -buf) & (x < box + buf)).all(1)
    return x[keep], source[keep], int(keep[:b.shape[0]].sum())


def exact(case, seed):
    path, n, ncs = case["path"], case["n"], _ncs(case)
    box = 2.0 * n ** (1.0 / 3.0)
    m = n if path == "noalloc" else n * (1.0 + 2.0 * _buffer(box) / box) ** 3
    if path == "fof" or m > EXACT_MAX or (path == "batch" and m * m * case["items"] > EXACT_MAX ** 2):
        return None
    if path == "batch":
        out = {"rk": [], "dens": [], "meshes": [], "totals": []}
        for x, v, own, b, _ in _batch_items(case, seed):
            rk, dens = _knn64(x)
            meshes, totals = _meshes64(x, v, dens, rk, torch.zeros_like(rk), b, ncs)
            for k, o in (("rk", rk[:own]), ("dens", dens[:own]), ("meshes", meshes),
                         ("totals", totals.reshape(-1))):
                out[k].append(o)
        return out
    s = prepare(case, seed)
    if path == "noalloc":
        rk, dens = _knn64(s["x"])
        return {"rk": rk, "dens": dens}
    if path == "zip":
        z0, z1, z2, z3 = s["zip"]
        counts = torch.as_tensor(z2).cuda().long()
        counts[counts == 255] = torch.as_tensor(z3).cuda().long()
        cell = torch.repeat_interleave(torch.arange(counts.numel(), device="cuda"), counts)
        c = torch.stack([cell % s["cells"], cell // s["cells"] % s["cells"], cell // s["cells"] ** 2], 1)
        x = s["side"] * ((torch.as_tensor(z0).cuda().double() + 0.5) / 256.0 + c)
        x, _, kept = _shell64(x, s["box"], s["buf"])
        rk, dens = _knn64(x)
        return {"n": x.shape[0], "kept": kept, "rk": rk[:n], "dens": dens[:n]}
    out = {}
    if path == "shell_step":
        x, source, kept = _shell64(s["x"].double(), s["box"], s["buf"])
        x, v, out = x, s["v"][source], {"n": x.shape[0], "kept": kept}
    elif path == "mixed":
        cell = torch.as_tensor(s["cell"]).cuda().long()
        c = torch.stack([cell % s["grid"], cell // s["grid"] % s["grid"], cell // s["grid"] ** 2], 1)
        off = torch.as_tensor(s["off"].astype(np.int32)).cuda().double()
        x = s["left"] + s["size"] * (c + off / 65536.0)
        v = torch.as_tensor(s["v"]).cuda()
    elif path == "records":
        x = torch.as_tensor(np.ascontiguousarray(s["p"]["x"])).cuda().double()
        v = torch.as_tensor(np.ascontiguousarray(s["p"]["v"])).cuda()
    else:
        x, v = s["x"], s["v"]
    rk, dens = _knn64(x)
    halo = torch.zeros_like(rk)
    if path == "records":
        igrp = torch.zeros(x.shape[0], dtype=torch.int32, device="cuda")
        count, mass = 0, 0.0
        for h in s["halos"]:
            if not all(s["left"] < t < s["right"] for t in h["x"]):
                continue
            near = ((x - torch.as_tensor(h["x"]).cuda().double()) ** 2).sum(1) < float(h["r"]) ** 2
            igrp[near] = -1
            count, mass = count + int(near.sum()), mass + float(h["mass"]) / 8.0
        halo = (igrp < 0).double()
        out = {"igrp": igrp[:n], "np_halo": count, "m_halo": mass}
    how = {"periodic": True} if path == "global" else {"density_only": True} if path == "density" else {}
    meshes, totals = _meshes64(x, v, dens, rk, halo, s["box"], ncs, **how)
    return {"rk": rk[:n], "dens": dens[:n], "meshes": meshes, "totals": totals, **out}
