"""Measured cases of the ray tracer: what its users have it do, through the public Python API
(optixsoltracedemos_gb300.native), over the sizes, scenes and options of the repository's workloads.

A case is one pass of one of these programs:

  trace    Tracer.run() of a kept scene; the records stay on the device (a zero-copy consumer)
  window   Tracer.trace_into() of a ray window into the caller's tensor on the caller's stream
  compact  Tracer.run_to_host_compact_ptr() into pinned host memory (write_output-style consumers)
  track    one step of a tracking loop: new poses and sun, update(), run(), flux_map()
  batch    Batch.run(): instances with their own poses, suns and ray counts, flux maps out
  serve    Server: a burst of requests submitted and waited for

listed() / draw(rng) give the cases, prepare / run one pass of them, work() the bytes and operations
a pass cannot do without, exact() its records in 64 bits.
"""
import math

import numpy as np
import torch

from optixsoltracedemos_gb300 import native, scenes

RECORD_BYTES = 80   # five float4 slots of a ray
ELEMENT_BYTES = scenes.ELEMENT_DTYPE.itemsize
FLUX_BINS = 100     # bins per axis of a flux map
PAIR_LIMIT = 5e9    # ray-element pairs above which exact() takes too long


def listed():
    return [
        # a design loop or a unit check: the smallest trace, where the launch and its latency are the cost
        _trace("three_10k", "three", rays=10_000),
        # the reference's three-heliostat demo at its ordinary size, with element ids recorded
        _trace("three_1m_ids", "three", rays=1 << 20, ids=True),
        # the single parabolic heliostat study: 16M rays, Gaussian sun
        _trace("parabolic_16m", "parabolic", sun="gaussian", rays=1 << 24),
        # a progressive consumer: a slice of a long run into a tensor of its own
        dict(_trace("parabolic_window_200k", "parabolic", sun="gaussian", rays=200_003), kind="window",
             first=5_000_000),
        # records to the host for a CSV or another post-processor
        dict(_trace("parabolic_compact_4m", "parabolic", sun="gaussian", rays=1 << 22), kind="compact"),
        # the large plain field trace: 10,000 flat heliostats, records of 64M rays (5.4 GB)
        _trace("field_10k_64m", "field", heliostats=10_000, rays=1 << 26),
        # a medium field in the morning: 1,000 focused heliostats, the accurate arithmetic, ids, an odd count
        _trace("field_1k_low_sun", "field", heliostats=1_000, curved=True, accurate=True, elevation=15.0,
               azimuth=-70.0, rays=3_000_017, ids=True),
        # heliostats on a steep slope (as at a solar furnace): not a planar field, so traversed by the BVH
        _trace("hillside_600", "hillside", heliostats=600, sun="gaussian", elevation=40.0, azimuth=20.0,
               rays=1_234_567),
        # one step of the plain per-scene loop: the field re-aimed, traced and its receiver flux read
        dict(_trace("track_field_10k", "field", heliostats=10_000, rays=1 << 22), kind="track"),
        # a day of sun positions of the large field, uneven ray counts, one batch
        _many("batch_field_16", "batch", heliostats=10_000, count=16, rays_min=1 << 20, rays_max=1 << 24),
        # a parameter sweep of a small scene: many short instances
        _many("batch_three_64", "batch", heliostats=3, count=64, rays_min=1 << 16, rays_max=1 << 20),
        # a burst of mixed requests to the server: fields of 3, 1,000 and 10,000, flat and parabolic
        _many("serve_mix_24", "serve", heliostats=0, count=24, rays_min=1 << 20, rays_max=1 << 24),
    ]


def _trace(name, scene, *, rays, heliostats=0, curved=False, sun="pillbox", accurate=False, elevation=45.0,
           azimuth=0.0, ids=False):
    return {"name": name, "kind": "trace", "scene": scene, "heliostats": heliostats, "curved": curved, "sun": sun,
            "accurate": accurate, "elevation": elevation, "azimuth": azimuth, "rays": rays, "ids": ids, "first": 0}


def _many(name, kind, *, heliostats, count, rays_min, rays_max):
    return {"name": name, "kind": kind, "heliostats": heliostats, "count": count, "rays_min": rays_min,
            "rays_max": rays_max}


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["trace", "trace", "trace", "trace", "window", "compact", "track", "batch", "batch", "serve"])
    if kind in ("batch", "serve"):
        lo = log_int(1 << 16, 1 << 20)
        small = kind == "batch" and rng.random() < 0.5
        c = _many("", kind, heliostats=0 if kind == "serve" else 3 if small else log_int(50, 10_000),
                  count=rng.randint(2, 64 if small else 16), rays_min=lo, rays_max=lo * rng.randint(2, 16))
    else:
        scene = {"window": "parabolic", "compact": "parabolic", "track": "field"}.get(kind) or rng.choice(
            ["three", "parabolic", "field", "field", "hillside"])
        many = scene in ("field", "hillside")
        most = {"window": 1 << 22, "compact": 1 << 22, "track": 1 << 22}.get(kind, (1 << 25) if many else 1 << 24)
        c = dict(_trace("", scene, heliostats=log_int(20, 2_000 if scene == "hillside" else 10_000) if many else 0,
                        curved=many and rng.random() < 0.4, sun=rng.choice(["pillbox", "gaussian"]),
                        accurate=rng.random() < 0.3, elevation=rng.uniform(12.0, 80.0),
                        azimuth=rng.uniform(-120.0, 120.0),
                        rays=log_int(4_000, most) if not many else log_int(30_000, most),
                        ids=rng.random() < 0.3), kind=kind)
        if kind == "window":
            c["first"] = rng.randrange(0, 1 << 28)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------ scenes ---
def _scene(case, seed):
    """(elements, sun direction, sun shape, sun parameter) of a single-scene case: the positions, poses
    and the sun follow the seed."""
    rng = np.random.default_rng(seed)
    elev, azim = case["elevation"] + rng.uniform(-1, 1), case["azimuth"] + rng.uniform(-1, 1)
    if case["scene"] == "three":
        sc = scenes.three_heliostats(num_rays=1)
        e, sun = sc.elements, np.array([rng.uniform(-0.1, 0.1), -1.0, rng.uniform(0.9, 1.1)])
        e["aim_point"][:3] = scenes.bisector_aim(e["origin"][:3], sun, e["origin"][3])
    elif case["scene"] == "parabolic":
        sc = scenes.single_parabolic(num_rays=1)
        e, sun = sc.elements, np.array([rng.uniform(-0.1, 0.1), rng.uniform(-0.1, 0.1), 1.0])
        e["aim_point"][:1] = scenes.bisector_aim(e["origin"][:1], sun, e["origin"][1])
    else:
        sun = scenes.sun_vector(elev, azim)
        e = _field(case["heliostats"], case["curved"], sun, seed, slope=0.6 if case["scene"] == "hillside" else 0.0)
    gaussian = case["sun"] == "gaussian"
    shape = (scenes.SUN_GAUSSIAN if gaussian else scenes.SUN_PILLBOX) | (scenes.SUN_ACCURATE if case["accurate"] else 0)
    return e, sun, shape, 2.5e-3 if gaussian else 4.65e-3


def _field(n, curved, sun, seed, slope=0.0):
    """A radial-stagger field of n heliostats around a 200 m tower; slope: the ground rises by that
    much per metre northwards, the tower with it."""
    e = scenes.large_field(n_heliostats=n, sun=sun, num_rays=1, seed=seed, parabolic=curved).elements
    if slope:
        e["origin"][:, 2] += slope * e["origin"][:, 1]
        e["aim_point"][:, 2] += slope * e["origin"][:, 1]
        e = scenes.reaim(e, sun)
    return e


class _DeviceArray:
    """Zero-copy view of a tracer's device buffer; keeps the tracer alive with it."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3,
                                         "strides": None}


# ------------------------------------------------------------------------------------ one pass -
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "serve":
        return _prepare_serve(case, seed)
    elements, sun, shape, param = _scene(case, seed)
    n = case["rays"]
    t = native.Tracer(0, 1 if kind == "window" else n)
    t.set_elements(elements)
    t.set_sun_vector(sun)
    t.set_sun_shape(shape, param)
    t.set_seed(seed, 0)
    t.set_record_ids(case["ids"])
    t.initialize()
    s = {"kind": kind, "tracer": t}
    if kind == "trace":
        hits, ids = t.device_buffers()
        s["out"] = [torch.as_tensor(_DeviceArray(t, hits, (n, native.MAX_DEPTH, 4), "<f4"), device="cuda")]
        if case["ids"]:
            s["out"].append(torch.as_tensor(_DeviceArray(t, ids, (n, native.MAX_DEPTH), "<i4"), device="cuda"))
    elif kind == "window":
        s["out"] = torch.empty(n, native.MAX_DEPTH, 4, device="cuda")
        s["ids"] = torch.empty(n, native.MAX_DEPTH, device="cuda", dtype=torch.int32) if case["ids"] else None
        s["stream"] = torch.cuda.Stream()
        s["range"] = (case["first"], n)
    elif kind == "compact":
        s["points"] = torch.empty(n, 3, pin_memory=True)
        s["counts"] = torch.empty(n, dtype=torch.uint8, pin_memory=True)
        s["records"] = torch.zeros(4 * n, 4, pin_memory=True)
    elif kind == "track":
        # the step's new poses: the field re-aimed for the sun a few minutes later
        s["sun"] = scenes.sun_vector(case["elevation"] + 1.5, case["azimuth"] + 2.0 + (seed % 97) * 1e-3)
        s["poses"] = scenes.reaim(elements, s["sun"])
    torch.cuda.synchronize()
    return s


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    b = native.Batch(0, FLUX_BINS, FLUX_BINS)
    if case["heliostats"] <= 8:
        base = scenes.three_heliostats(num_rays=1).elements
    else:
        base = _field(case["heliostats"], False, scenes.sun_vector(45.0, 0.0), seed)
    sid = b.add_scene(base)
    for k, rays in enumerate(_counts(case, rng)):
        # the three-heliostat receiver faces the mirrors to the north: its suns stand in the south
        sun = (np.array([rng.uniform(-0.4, 0.4), -1.0, rng.uniform(0.6, 1.4)]) if case["heliostats"] <= 8
               else scenes.sun_vector(rng.uniform(10.0, 80.0), rng.uniform(-120.0, 120.0)))
        b.add_instance(sid, sun, scenes.SUN_PILLBOX, 4.65e-3, rays, seed=seed + k, instance=k,
                       poses=scenes.reaim(base, sun))
    return {"kind": "batch", "batch": b, "count": case["count"]}


def _prepare_serve(case, seed):
    rng = np.random.default_rng(seed)
    server = native.Server(0, memory_budget=2 << 30, max_active=64)
    sun0 = scenes.sun_vector(45.0, 0.0)
    fields = [scenes.three_heliostats(num_rays=1).elements] + [
        _field(n, curved, sun0, seed) for n in (1_000, 10_000) for curved in (False, True)]
    ids = [server.add_scene(f) for f in fields]
    jobs = []
    for k, rays in enumerate(_counts(case, rng)):
        which = k % len(fields)
        sun = (np.array([rng.uniform(-0.4, 0.4), -1.0, rng.uniform(0.6, 1.4)]) if which == 0
               else scenes.sun_vector(rng.uniform(10.0, 80.0), rng.uniform(-120.0, 120.0)))
        jobs.append((ids[which], sun, rays, seed + k, k, scenes.reaim(fields[which], sun)))
    return {"kind": "serve", "server": server, "jobs": jobs}


def _counts(case, rng):
    """Log-uniform ray counts of the instances or requests."""
    lo, hi = math.log(case["rays_min"]), math.log(case["rays_max"])
    return [int(math.exp(x)) for x in rng.uniform(lo, hi, case["count"])]


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        b.run()
        return {"counts": np.stack([b.counts(i) for i in range(state["count"])]),
                "stats": np.stack([b.stats(i) for i in range(state["count"])]).astype(np.int64)}
    if kind == "serve":
        server = state["server"]
        requests = [server.submit(scene, sun, scenes.SUN_PILLBOX, 4.65e-3, rays, seed=seed, instance=inst, poses=poses)
                    for scene, sun, rays, seed, inst, poses in state["jobs"]]
        done = [server.wait(r) for r in requests]
        return {"counts": np.stack([d[0] for d in done]), "stats": np.stack([d[1] for d in done]).astype(np.int64)}
    t = state["tracer"]
    if kind == "trace":
        t.run()
        return state["out"]
    if kind == "window":
        first, n = state["range"]
        ids = state["ids"]
        t.trace_into(state["out"].data_ptr(), ids.data_ptr() if ids is not None else None, first, n,
                     state["stream"].cuda_stream)
        return [state["out"]] if ids is None else [state["out"], ids]
    if kind == "compact":
        nr = t.run_to_host_compact_ptr(state["points"].data_ptr(), state["counts"].data_ptr(),
                                       state["records"].data_ptr(), state["records"].shape[0])
        return {"points": state["points"], "counts": state["counts"], "records": state["records"], "used": nr}
    t.set_elements(state["poses"])
    t.set_sun_vector(state["sun"])
    t.update()
    t.run()
    counts, flux = t.flux_map(FLUX_BINS, FLUX_BINS)
    return {"counts": counts, "flux": flux}


def work(case):
    """Bytes: the records (or flux maps, or compact records) written once and the element list read once.
    Operations: the sun-plane point of every ray (Halton sums and two scaled axes), and a direction, a
    closest hit, the reflection and the next closest hit for the share of them that meets an element."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        mean = (case["rays_max"] - case["rays_min"]) / math.log(case["rays_max"] / case["rays_min"])
        rays, maps = mean * case["count"], case["count"]
        heliostats = case["heliostats"] or 4_400  # mean of the server's five scenes
        return {"bytes": maps * (FLUX_BINS * FLUX_BINS * 4.0 + heliostats * ELEMENT_BYTES),
                "flops": rays * (40 + 0.5 * 400)}
    rays = case["rays"]
    meet = 0.5 if case["scene"] in ("field", "hillside") else 0.1
    out = RECORD_BYTES + (20 if case["ids"] else 0)
    if kind == "compact":
        out = 12 + 1 + 16 * 2 * meet
    elif kind == "track":
        out = 0
    return {"bytes": rays * out + max(case["heliostats"], 2) * ELEMENT_BYTES, "flops": rays * (40 + meet * 400)}


# ------------------------------------------------------------------------------------ 64 bits --
def exact(case, seed):
    """The records of a trace in 64 bits: every element tested by every ray.  Element ids, counts and
    flux maps are whole numbers (or scaled from them)."""
    if case["kind"] not in ("trace", "window", "compact"):
        return None
    elements, sun, shape, param = _scene(case, seed)
    if case["rays"] * float(len(elements)) > PAIR_LIMIT:
        return None
    frame = _sun_frame(elements, sun, shape, param)
    chunk = 1 << 21
    hits = torch.cat([_trace64(elements, frame, shape, case["first"] + k, min(chunk, case["rays"] - k), seed)
                      for k in range(0, case["rays"], chunk)])
    if case["kind"] == "compact":
        return {"points": hits[:, 0, 1:], "counts": None, "records": None, "used": None}
    return [hits, None] if case["ids"] else [hits]


def _axes(e):
    """World axes of an element's local frame: z towards the aim point, yaw and pitch, then the roll."""
    n = np.asarray(e["aim_point"]) - np.asarray(e["origin"])
    n = n / np.linalg.norm(n)
    a, b, g = math.atan2(n[0], n[2]), math.asin(n[1]), math.radians(float(e["zrot_deg"]))
    ca, sa, cb, sb, cg, sg = math.cos(a), math.sin(a), math.cos(b), math.sin(b), math.cos(g), math.sin(g)
    return np.array([[ca * cg + sa * sb * sg, -cb * sg, -sa * cg + ca * sb * sg],
                     [ca * sg - sa * sb * cg, cb * cg, -sa * sg - ca * sb * cg], [sa * cb, sb, ca * cb]])


def _box(e):
    """Axis-aligned box of an element: of its rectangle, or of the box around its cylinder."""
    half = np.array([e["width"] / 2, e["height"] / 2, e["width"] / 2 if e["surface"] == scenes.SURFACE_CYLINDER else 0])
    reach = np.abs(_axes(e).T) @ half
    return np.asarray(e["origin"]) - reach, np.asarray(e["origin"]) + reach


def _sun_frame(elements, sun, shape, param):
    s = np.asarray(sun, float) / np.linalg.norm(sun)
    boxes = [_box(e) for e in elements]
    corners = np.array([[(lo, hi)[k >> a & 1][a] for a in range(3)] for lo, hi in boxes for k in range(8)])
    depth = np.abs(corners @ s)
    su = np.cross([1.0, 0, 0] if abs(s[0]) < 0.9 else [0, 1.0, 0], s)
    su /= np.linalg.norm(su)
    sv = np.cross(s, su)
    pad = depth * math.tan(5 * param if shape & scenes.SUN_GAUSSIAN else param)
    u, v = corners @ su, corners @ sv
    v0 = (u - pad).min() * su + (v - pad).min() * sv + depth.max() * s
    cu = np.cross([0, 1.0, 0] if abs(s[0]) > 0.99 else [1.0, 0, 0], -s)
    cu /= np.linalg.norm(cu)
    return {"v0": v0, "e1": ((u + pad).max() - (u - pad).min()) * su, "e2": ((v + pad).max() - (v - pad).min()) * sv,
            "w": -s, "cu": cu, "cv": np.cross(-s, cu), "param": param, "boxes": boxes}


def _philox(ray, bounce, block, seed):
    """Philox-4x32-10 (Salmon et al., SC'11) of counter (ray, bounce << 4 | block, instance 0) under the
    seed, as uniforms (x >> 8 + 1) 2^-24."""
    mask = 0xFFFFFFFF

    def mul(m, x):  # 32 x 32 -> (high, low) from 16-bit halves: int64 holds every partial product
        lo, hi = m * (x & 0xFFFF), m * (x >> 16)
        t = hi + (lo >> 16)
        return t >> 16, (t << 16 | lo & 0xFFFF) & mask

    c = [ray & mask, ray >> 32, torch.full_like(ray, bounce << 4 | block), torch.zeros_like(ray)]
    k0, k1 = seed & mask, seed >> 32 & mask
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return [((x >> 8) + 1).double() * 2.0 ** -24 for x in c]


def _halton(i, base):
    r, f = torch.zeros_like(i, dtype=torch.float64), 1.0
    while int(i.max()) > 0:
        f /= base
        r += f * (i % base)
        i = i // base
    return r


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _normals(u1, u2):
    r, a = torch.sqrt(-2 * torch.log(u1)), 2 * math.pi * u2
    return r * torch.cos(a), r * torch.sin(a)


def _tilt(n, sigma, g1, g2):
    t = torch.zeros_like(n)
    steep = n[:, 0].abs() > 0.9
    t[:, 0], t[:, 1] = (~steep).double(), steep.double()
    t1 = _unit(torch.linalg.cross(t, n))
    t2 = torch.linalg.cross(n, t1)
    return _unit(n + (sigma * g1)[:, None] * t1 + (sigma * g2)[:, None] * t2)


def _hit(e, axes, o, d, tmin):
    """(distance or inf, normal) of every ray on one element's surface."""
    l, m = (o - torch.as_tensor(e["origin"].copy(), device=o.device)) @ axes.T, d @ axes.T
    inf = torch.full_like(l[:, 0], math.inf)
    hw, hh = float(e["width"]) / 2, float(e["height"]) / 2
    if e["surface"] == scenes.SURFACE_CYLINDER:
        a = m[:, 0] ** 2 + m[:, 2] ** 2
        tm = -(l[:, 0] * m[:, 0] + l[:, 2] * m[:, 2]) / a
        q = torch.sqrt((hw * hw - (l[:, 0] + tm * m[:, 0]) ** 2 - (l[:, 2] + tm * m[:, 2]) ** 2) / a)
        t = inf
        for side in (tm + q, tm - q):
            t = torch.where((side > tmin) & ((l[:, 1] + side * m[:, 1]).abs() <= hh), side, t)
        for cap in (-hh, hh):
            c = (cap - l[:, 1]) / m[:, 1]
            on = (c > tmin) & ((l[:, 0] + c * m[:, 0]) ** 2 + (l[:, 2] + c * m[:, 2]) ** 2 <= hw * hw)
            t = torch.where(on, torch.minimum(t, c), t)
        return t, d
    cx, cy = (float(e["curv_x"]), float(e["curv_y"])) if e["surface"] == scenes.SURFACE_PARABOLIC else (0.0, 0.0)
    a = 0.5 * (cx * m[:, 0] ** 2 + cy * m[:, 1] ** 2)
    b = cx * l[:, 0] * m[:, 0] + cy * l[:, 1] * m[:, 1] - m[:, 2]
    c = 0.5 * (cx * l[:, 0] ** 2 + cy * l[:, 1] ** 2) - l[:, 2]
    q = torch.sqrt(b * b - 4 * a * c)
    t1, t2 = (-b - q) / (2 * a), (-b + q) / (2 * a)
    t = torch.where(a.abs() < 1e-12, -c / b, torch.where((t1 > 0) & (t1 < t2), t1, t2))
    x, y = l[:, 0] + t * m[:, 0], l[:, 1] + t * m[:, 1]
    t = torch.where((t > tmin) & (x.abs() <= hw) & (y.abs() <= hh), t, inf)
    n = _unit(torch.stack([-cx * x, -cy * y, torch.ones_like(x)], 1)) @ axes
    return t, n


def _trace64(elements, frame, shape, first, count, seed):
    dev = "cuda"
    vec = {k: torch.as_tensor(v, device=dev) for k, v in frame.items() if isinstance(v, np.ndarray)}
    ray = torch.arange(first, first + count, device=dev)
    hits = torch.zeros(count, native.MAX_DEPTH, 4, device=dev, dtype=torch.float64)
    o = vec["v0"] + _halton(ray, 2)[:, None] * vec["e1"] + _halton(ray, 3)[:, None] * vec["e2"]
    hits[:, 0, 1:] = o
    u = _philox(ray, 0, 0, seed)
    if shape & scenes.SUN_GAUSSIAN:
        g1, g2 = _normals(u[0], u[1])
        d = vec["w"] + (frame["param"] * g1)[:, None] * vec["cu"] + (frame["param"] * g2)[:, None] * vec["cv"]
    else:
        omz = 2 * math.sin(frame["param"] / 2) ** 2 * (1 - u[1])
        r, phi = torch.sqrt(omz * (2 - omz)), 2 * math.pi * u[0]
        d = ((r * torch.cos(phi))[:, None] * vec["cu"] + (r * torch.sin(phi))[:, None] * vec["cv"]
             + (1 - omz)[:, None] * vec["w"])
    d, row, tmin = _unit(d), torch.arange(count, device=dev), 1e-3
    mats = [torch.as_tensor(_axes(e), device=dev) for e in elements]
    optics = torch.as_tensor(np.stack([elements[k] for k in ("slope_error", "specularity_error", "reflectivity")], 1),
                             device=dev)
    for depth in range(1, native.MAX_DEPTH):
        best, which, normal = torch.full_like(o[:, 0], math.inf), torch.zeros_like(row), torch.zeros_like(o)
        inv = 1 / d
        for k, e in enumerate(elements):
            lo, hi = (torch.as_tensor(b, device=dev) for b in frame["boxes"][k])
            t0, t1 = (lo - o) * inv, (hi - o) * inv
            meets = torch.minimum(t0, t1).amax(1).clamp(min=tmin) <= torch.maximum(t0, t1).amin(1)
            sel = meets.nonzero()[:, 0]
            if not len(sel):
                continue
            t, n = _hit(e, mats[k], o[sel], d[sel], tmin)
            closer = t < best[sel]
            sel = sel[closer]
            best[sel], which[sel], normal[sel] = t[closer], k, n[closer]
        at = (best < math.inf).nonzero()[:, 0]
        if not len(at):
            break
        o, d, row, which, normal = o[at] + best[at, None] * d[at], d[at], row[at], which[at], normal[at]
        receiver = which == len(elements) - 1
        one_sided = receiver if elements["surface"][-1] == scenes.SURFACE_FLAT else receiver & False
        seen = ~one_sided | ((normal * d).sum(1) < 0)
        stage = 1.0 + receiver.double()
        hits[row[seen], depth] = torch.cat([stage[:, None], o], 1)[seen]
        o, d, row, which, normal = (x[~receiver] for x in (o, d, row, which, normal))
        op, facing = optics[which], torch.where(((normal * d).sum(1) <= 0)[:, None], normal, -normal)
        ua, ub = _philox(row + first, depth, 0, seed), _philox(row + first, depth, 1, seed)
        tilted = _tilt(facing, op[:, 0], *_normals(ua[1], ua[2]))
        facing = torch.where((op[:, 0] > 0)[:, None], tilted, facing)
        d = d - 2 * (facing * d).sum(1, keepdim=True) * facing
        d = torch.where((op[:, 1] > 0)[:, None], _tilt(_unit(d), op[:, 1], *_normals(ub[0], ub[1])), d)
        kept = ua[0] <= op[:, 2]
        o, d, row, tmin = o[kept], d[kept], row[kept], 1e-2
    return hits
