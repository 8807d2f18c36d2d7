"""The work that users of this framework have it do, as cases to be timed.

A renderer that guides its paths does three things over and over: it turns the
segments of its paths into samples, it trains the field with a frame of
samples (Update), and it asks the field for directions (guided queries).  Each
case below is one of these through the public entry points, on inputs of the
shapes the tests and the benchmark of this repository use, made on the GPU.
"""

import math

import numpy as np
import torch

import openpgl_gb300 as pgl

# name: what it stands for
_LISTED = [
    # the first frame of a low-resolution preview: one region, latency counts
    dict(name="update_preview", kind="update", field="parallax", scene="cube", frames=1, samples=4099, volume=0.0,
         leaf=32000, source="pageable"),
    # one Update with a million samples that the renderer left in page-locked host memory
    dict(name="update_single", kind="update", field="parallax", scene="cube", frames=1, samples=1048576, volume=0.0,
         leaf=32000, source="pinned"),
    # a progressive render: eight frames of two million samples, a quarter of them in a volume
    dict(name="update_frames", kind="update", field="parallax", scene="cube", frames=8, samples=2097152, volume=0.25,
         leaf=32000, source="device"),
    # a scene with thousands of small light clusters and heavy-tailed weights, finer regions
    dict(name="update_clusters", kind="update", field="parallax", scene="clusters", frames=2, samples=4194304,
         volume=0.25, leaf=16000, source="device"),
    # the field type without parallax compensation, odd frame size, small regions
    dict(name="update_plain_vmm", kind="update", field="vmm", scene="cube", frames=3, samples=262147, volume=0.25,
         leaf=8000, source="device"),
    # the directional quadtree field type
    dict(name="update_quadtree", kind="update", field="quadtree", scene="cube", frames=2, samples=1048576, volume=0.25,
         leaf=32000, source="device"),
    # one wavefront of surface vertices: a cosine product and one sample each
    dict(name="query_surface", kind="query", field="parallax", scene="cube", mode="surface", queries=1048576,
         leaf=8000),
    # the last vertices of a wavefront: a launch that hardly fills the chip
    dict(name="query_small", kind="query", field="parallax", scene="cube", mode="surface", queries=777, leaf=8000),
    # volume vertices with the phase function's product
    dict(name="query_volume_hg", kind="query", field="parallax", scene="cube", mode="volume_hg", queries=262147,
         leaf=8000),
    # path vertices that draw four directions each, on many small regions
    dict(name="query_vertices", kind="query", field="parallax", scene="clusters", mode="vertices", queries=1000003,
         leaf=4000),
    # surface vertices on a quadtree field
    dict(name="query_quadtree", kind="query", field="quadtree", scene="cube", mode="surface", queries=1048576,
         leaf=8000),
    # the samples of a tile's paths, made on the device
    dict(name="path_samples", kind="paths", paths=131072, length=12),
]

# frames that train the field of a query case
_TRAIN_FRAMES, _TRAIN_SAMPLES = 4, 524288


def listed():
    return [dict(c) for c in _LISTED]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update", "update", "update", "query", "query", "query", "paths"])
    if kind == "update":
        frames = rng.randint(1, 8)
        return dict(kind="update", field=rng.choice(["parallax", "parallax", "vmm", "quadtree"]),
                    scene=rng.choice(["cube", "clusters"]), frames=frames,
                    samples=_log_uniform(rng, 1000, min(2097152, 8388608 // frames)),
                    volume=rng.choice([0.0, 0.25, 0.5]), leaf=rng.choice([4000, 8000, 16000, 32000]),
                    source=rng.choice(["pageable", "pinned", "device", "device"]))
    if kind == "query":
        mode = rng.choice(["surface", "surface", "volume", "volume_hg", "vertices"])
        fields = ["parallax", "parallax", "vmm"] if mode == "volume_hg" else ["parallax", "parallax", "vmm", "quadtree"]
        return dict(kind="query", field=rng.choice(fields), scene=rng.choice(["cube", "clusters"]), mode=mode,
                    queries=_log_uniform(rng, 500, 1048576), leaf=rng.choice([4000, 8000, 16000]))
    return dict(kind="paths", paths=_log_uniform(rng, 1000, 131072), length=rng.randint(2, 12))


# ---------------------------------------------------------------- inputs


def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _uniform(g, *shape):
    return torch.rand(shape, generator=g, device="cuda")


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda")


def _sphere(g, *shape):
    return torch.nn.functional.normalize(_normal(g, *shape, 3), dim=-1)


def _running(w):
    """Running sums of each row, in one order on every run."""
    return torch.cumsum(w.cpu().double(), 1).float().cuda()


def _lobes(g, n, kmax, kappa_lo, kappa_hi, all_lobes):
    """n mixtures of up to kmax lobes: means, concentrations, cumulative weights."""
    w = -torch.log(_uniform(g, n, kmax) + 1e-9)
    if not all_lobes:
        used = 1 + torch.floor(_uniform(g, n) * kmax)
        w = torch.where(torch.arange(kmax, device="cuda")[None, :] < used[:, None], w, torch.zeros_like(w))
    kappa = kappa_lo * torch.exp(_uniform(g, n, kmax) * math.log(kappa_hi / kappa_lo))
    return _sphere(g, n, kmax), kappa, _running(w / w.sum(1, keepdim=True))


def _directions(g, model, which):
    """One direction per sample from mixture which[i]."""
    mu, kappa, cdf = model
    lobe = (cdf[which] < _uniform(g, len(which))[:, None]).sum(1).clamp_(max=mu.shape[1] - 1)
    d = mu[which, lobe] + _normal(g, len(which), 3) / kappa[which, lobe].sqrt()[:, None]
    return torch.nn.functional.normalize(d, dim=-1)


class _Scene:
    """cube: positions on the faces of the unit cube, three lobes per octant
    (volume samples: inside it, one lobe).  clusters: 4096 Gaussian clusters of
    Zipf masses with one to six lobes each and heavy-tailed weights."""

    def __init__(self, kind, g):
        self.clusters = kind == "clusters"
        if self.clusters:
            n = 4096
            self.centre = _uniform(g, n, 3)
            self.sigma = 1e-3 * torch.exp(_uniform(g, n) * math.log(50.0))
            mass = torch.arange(1, n + 1, device="cuda", dtype=torch.float64) ** -1.1
            mass = mass[torch.randperm(n, generator=g, device="cuda")]
            self.cdf = torch.cumsum((mass / mass.sum()).cpu(), 0).cuda()
            self.model = _lobes(g, n, 6, 2.0, 1000.0, False)
        else:
            self.model = _lobes(g, 8, 3, 5.0, 200.0, True)
            self.fog = _sphere(g, 1)

    def _cluster(self, g, n):
        u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
        return torch.searchsorted(self.cdf, u).clamp_(max=len(self.cdf) - 1)

    def positions(self, g, n):
        if not self.clusters:
            return _uniform(g, n, 3)
        c = self._cluster(g, n)
        return self.centre[c] + self.sigma[c][:, None] * _normal(g, n, 3)

    def samples(self, g, n, volume):
        """n sample records (PGLSampleData) as a float32 tensor [n, 10]."""
        inside = _uniform(g, n) < volume
        if self.clusters:
            c = self._cluster(g, n)
            pos = self.centre[c] + self.sigma[c][:, None] * _normal(g, n, 3)
            direction = _directions(g, self.model, c)
            weight = torch.exp(2.0 * _normal(g, n))
        else:
            pos = _uniform(g, n, 3)
            axis = torch.floor(_uniform(g, n, 1) * 3).long().clamp_(max=2)
            face = pos.scatter(1, axis, torch.floor(_uniform(g, n, 1) * 2).clamp_(max=1))
            pos = torch.where(inside[:, None], pos, face)
            octant = ((pos >= 0.5).long() * torch.tensor([4, 2, 1], device="cuda")).sum(1)
            fog = torch.nn.functional.normalize(self.fog + _normal(g, n, 3) / math.sqrt(20.0), dim=-1)
            direction = torch.where(inside[:, None], fog, _directions(g, self.model, octant))
            weight = torch.exp(_normal(g, n))
        r = torch.empty(n, 10, device="cuda")
        r[:, 0:3] = pos
        r[:, 3:6] = direction
        r[:, 6] = weight
        r[:, 7] = 1.0 / (4.0 * math.pi)
        r[:, 8] = 0.05 + 1.95 * _uniform(g, n)
        r.view(torch.int32)[:, 9] = torch.where(inside, 2, 0).int()
        return r


_DEVICE = None


def _device():
    global _DEVICE
    if _DEVICE is None:
        _DEVICE = pgl.Device()
    return _DEVICE


def _new_field(case):
    return pgl.Field(_device(), pgl.FieldConfig(deterministic=True, max_samples_per_leaf=case["leaf"],
                                                parallax=case["field"] != "vmm", dqt=case["field"] == "quadtree"))


def _below_one(t):
    return t.clamp_(max=0.99999994)


def _query_records(case, scene, g):
    """Queries (PGLGuidedQuery, [n, 9]) or vertices (PGLGuidedVertex, [n, 19])."""
    n, vertices = case["queries"], case["mode"] == "vertices"
    q = torch.empty(n, 19 if vertices else 9, device="cuda")
    q[:, 0:3] = scene.positions(g, n)
    q[:, 3:6] = _sphere(g, n)
    if vertices:
        q[:, 6:9] = _sphere(g, n)
        q[:, 9] = _uniform(g, n)
        q[:, 10:] = _below_one(_uniform(g, n, 9))
    else:
        q[:, 6:] = _below_one(_uniform(g, n, 3))
    return q


def _segments(paths, length, g):
    """Random walks of 1 to `length` segments (PGLPathSegmentData, 34 words
    each) with the mix of vertices a path tracer records, and where each path
    begins."""
    lens = 1 + torch.floor(_uniform(g, paths) * length).long().clamp_(max=length - 1)
    begin = torch.zeros(paths + 1, dtype=torch.int64, device="cuda")
    begin[1:] = torch.cumsum(lens, 0)
    n = int(begin[-1])
    owner = torch.repeat_interleave(torch.arange(paths, device="cuda"), lens)
    step = (_uniform(g, n, 3) - 0.5) * 3.0
    walk = torch.cumsum((step.double() * 2.0 ** 30).long(), 0).double() * 2.0 ** -30
    start = torch.rand(paths, 3, generator=g, device="cuda", dtype=torch.float64) * 10.0
    u = [_uniform(g, n) for _ in range(14)]
    s = torch.zeros(n, 34, device="cuda")
    words = s.view(torch.int32)
    s[:, 0:3] = (start[owner] + walk - walk[begin[:-1]][owner]).float()
    s[:, 3:6] = _sphere(g, n)
    s[:, 6:9] = _sphere(g, n)
    s[:, 9:12] = _sphere(g, n)
    words[:, 12] = (u[0] < 0.2).int()  # volume scatter
    s[:, 13] = 0.01 * torch.exp(u[1] * math.log(1000.0))  # pdf of the direction
    words[:, 14] = (u[2] < 0.1).int()  # delta
    s[:, 15:18] = _uniform(g, n, 3) * 1.2  # scattering weight
    s[:, 18:21] = 0.5 + 0.5 * _uniform(g, n, 3)  # transmittance
    s[:, 21:24] = _uniform(g, n, 3) * 2.0 * (u[3] >= 0.5)[:, None]  # direct contribution
    s[:, 24] = u[4]  # multiple-importance weight
    s[:, 25:28] = _uniform(g, n, 3) * (u[5] >= 0.8)[:, None]  # scattered contribution
    s[:, 28] = torch.where(u[6] < 0.5, 1.0, torch.where(u[6] < 0.6, 0.0, u[7]))  # Russian roulette
    s[:, 29] = torch.where(u[8] < 0.7, 1.0, 1.0 + u[9])  # eta
    s[:, 30] = u[10] * torch.where(u[11] < 0.2, 0.01, 1.0)  # roughness
    return s, begin.int()


def _train_query_field(case, seed):
    g = _rng(seed)
    scene = _Scene(case["scene"], g)
    field, storage = _new_field(case), pgl.SampleStorage()
    for _ in range(_TRAIN_FRAMES):
        frame = scene.samples(g, _TRAIN_SAMPLES, 0.25)
        torch.cuda.synchronize()
        storage.clear()
        storage.add_samples_device(frame.data_ptr(), len(frame))
        field.update(storage)
    storage.release()
    return field, scene, g


class _State:
    """Releases the library's objects with it."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for name in ("field", "storage"):
            o = self.__dict__.get(name)
            if o is not None:
                o.release()


def prepare(case, seed):
    if case["kind"] == "update":
        g = _rng(seed)
        scene = _Scene(case["scene"], g)
        frames = [scene.samples(g, case["samples"], case["volume"]) for _ in range(case["frames"])]
        if case["source"] != "device":
            frames = [f.cpu().pin_memory() if case["source"] == "pinned" else f.cpu() for f in frames]
            frames = [f.numpy().view(pgl.PGL_SAMPLE_DTYPE).reshape(-1) for f in frames]
        s = _State(case=case, field=_new_field(case), storage=pgl.SampleStorage(), frames=frames,
                   saved=np.zeros(_save_bytes(case), np.uint8))
    elif case["kind"] == "query":
        field, scene, g = _train_query_field(case, seed)
        n = case["queries"]
        s = _State(case=case, field=field, q=_query_records(case, scene, g),
                   out=torch.zeros(n, 19 if case["mode"] == "vertices" else 8, device="cuda"))
        if case["mode"] == "volume_hg":
            s.g = 1.8 * _uniform(g, n) - 0.9
    else:
        seg, begin = _segments(case["paths"], case["length"], _rng(seed))
        room = case["paths"] * case["length"]
        s = _State(case=case, seg=seg, begin=begin, out=torch.zeros(room, 10, device="cuda"),
                   sample_begin=torch.zeros(len(begin), dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------- one pass


def _save_bytes(case):
    """Room for the saved field: some 3 KB per region, and a quadtree region
    by its nodes."""
    regions = 64 + 4 * case["samples"] * case["frames"] // case["leaf"]
    return regions * (24576 if case["field"] == "quadtree" else 3200)


def _save(s):
    """The trained field as the bytes of its file, in the program's own buffer."""
    n = s.field.lib.pglFieldStoreToBuffer(s.field.h, s.saved.ctypes.data_as(pgl.ctypes.c_char_p), s.saved.nbytes)
    if not 0 < n <= s.saved.nbytes:
        raise RuntimeError("no room for the field: %d bytes" % n)
    return s.saved


def run(s):
    case = s.case
    if case["kind"] == "update":  # a render from its first frame on, then the field is saved
        s.field.reset()
        for f in s.frames:
            s.storage.clear()
            if case["source"] == "device":
                s.storage.add_samples_device(f.data_ptr(), len(f))
            else:
                s.storage.add_samples(f)
            s.field.update(s.storage)
        return _save(s)
    if case["kind"] == "query":
        n, mode = case["queries"], case["mode"]
        if mode == "vertices":
            s.field.sample_vertices_device(s.q.data_ptr(), n, s.out.data_ptr())
            return {"region": s.out.view(torch.int32)[:, :2], "sample": s.out[:, 2:]}
        if mode == "volume_hg":
            s.field.sample_batch_hg_device(s.q.data_ptr(), s.g.data_ptr(), n, s.out.data_ptr())
        else:
            s.field.sample_batch_device(s.q.data_ptr(), n, s.out.data_ptr(), volume=mode == "volume")
        return {"region": s.out.view(torch.int32)[:, :2], "rest1d": s.out[:, 2], "direction": s.out[:, 3:6],
                "pdf": s.out[:, 6:]}
    pgl.path_samples_device(s.seg.data_ptr(), s.begin.data_ptr(), case["paths"], 100.0, s.out.data_ptr(),
                            s.sample_begin.data_ptr())
    return {"begin": s.sample_begin, "flags": s.out.view(torch.int32)[:, 9], "record": s.out[:, :9]}


def work(case):
    if case["kind"] == "update":
        n = case["samples"] * case["frames"]
        # the records once, the saved field once (about 3 KB per region, a region
        # for every `leaf` samples); the fit's operations per sample: the first
        # frame's EM takes tens of passes over some sixteen lobes, a later
        # frame's a few over eight, at 21 operations per lobe and pass (a
        # quadtree: one descent and splat)
        first, later = (100, 100) if case["field"] == "quadtree" else (40 * 16 * 21, 5 * 8 * 21)
        return {"bytes": 40 * n + 3000 * (1 + n // case["leaf"]),
                "flops": case["samples"] * (first + later * (case["frames"] - 1))}
    if case["kind"] == "query":
        n = case["queries"]
        if case["field"] == "quadtree":  # some eight levels down for a sample, as many for its pdf
            samples, size = (4, 152) if case["mode"] == "vertices" else (1, 68)
            return {"bytes": size * n, "flops": n * samples * 200}
        if case["mode"] == "vertices":
            return {"bytes": 152 * n, "flops": n * (8 * 62 + 50 + 4 * (8 * 12 + 64))}
        if case["mode"] == "volume_hg":
            return {"bytes": 72 * n, "flops": n * (3 * (8 * 62 + 50) + 4 * 8 * 12 + 64)}
        return {"bytes": 68 * n, "flops": n * (8 * 62 + 50 + 8 * 24 + 64)}
    seg = case["paths"] * (1 + case["length"]) / 2
    return {"bytes": seg * 136 + 0.5 * seg * 40 + 8 * case["paths"], "flops": seg * 20 * case["length"]}


# ---------------------------------------------------------------- 64-bit values


def exact(case, seed):
    """In 64 bits: the samples of paths, and guided queries of mixture fields
    (the trained mixtures are the queries' weights, read back from the field).
    A fit has no such value: its splits, merges and stopping are decisions on
    sums that rounding turns, so a fit in 64 bits is another fit.  None too for
    the phase function's product (the framework's own fits) and for quadtrees
    (decisions down the tree)."""
    if case["kind"] == "paths":
        return _exact_paths(case, seed)
    if case["kind"] == "query" and case["mode"] != "volume_hg" and case["field"] != "quadtree":
        return _exact_queries(case, seed)
    return None


_REGION = np.dtype([("valid", "u1"), ("vmm", "<f4", (4, 9, 8)), ("K", "<u8"), ("pivot", "<f4", (3,)),
                    ("bounds", "<f4", (6,)), ("suff", "<f4", (163,)), ("suffK", "<u8"), ("normalized", "u1"),
                    ("split", "<f4", (288,)), ("splitK", "<u8"), ("after", "<u8", (2,)), ("stats", "<f4", (13,)),
                    ("splitFlag", "u1"), ("range", "<u8", (2,))])


def _read_field(b, volume):
    """kd bounds, kd nodes and regions of one half of a saved mixture field."""
    o = 44  # header, types, iteration, samples per pixel
    for half in range(2):
        o += 65 + 77 + 24 + 1  # configuration
        bounds = np.frombuffer(b, "<f4", 6, o)
        n = int(np.frombuffer(b, "<u8", 1, o + 24)[0])
        nodes = np.frombuffer(b, np.dtype([("split", "<f4"), ("bits", "<u4")]), n, o + 32)
        o += 32 + 8 * n
        r = int(np.frombuffer(b, "<u8", 1, o)[0])
        regions = np.frombuffer(b, _REGION, r, o + 8)
        o += 8 + r * _REGION.itemsize
        if half == int(volume):
            return bounds, nodes, regions
        o += 2 + ((4 + 16 * r) if b[o + 1] else 0)


def _f64(x):
    return torch.as_tensor(np.array(x, dtype=np.float64), device="cuda")


def _rows(v):
    return _f64(v.reshape(len(v), -1))


def _dot(a, b):
    return (a * b).sum(-1)


def _frame_times(n, d):
    """d in the frame around n (z along n), with the framework's choice of x."""
    z = torch.zeros_like(n[:, 0])
    x0, x1 = torch.stack([z, n[:, 2], -n[:, 1]], 1), torch.stack([-n[:, 2], z, n[:, 0]], 1)
    x = torch.where((_dot(x0, x0) > _dot(x1, x1))[:, None], x0, x1)
    x = x / x.norm(dim=1, keepdim=True)
    y = torch.linalg.cross(n, x)
    y = y / y.norm(dim=1, keepdim=True)
    return d[:, 0:1] * x + d[:, 1:2] * y + d[:, 2:3] * n


class _Mixture:
    """Weights, concentrations, means [n, 32(, 3)] of n mixtures."""

    def __init__(self, w, kappa, mu):
        self.w, self.kappa, self.mu = w, kappa, mu

    def norm(self):
        k = torch.where(self.kappa > 0, self.kappa, torch.ones_like(self.kappa))
        return torch.where(self.kappa > 0, k / (2 * math.pi * -torch.expm1(-2 * k)),
                           torch.full_like(k, 1 / (4 * math.pi)))

    def pdf(self, d):
        c = (_dot(self.mu, d[:, None, :]) - 1).clamp(max=0)
        return (self.w * self.norm() * torch.exp(self.kappa * c)).sum(1)

    def times_cosine(self, n):
        kc = 2.18853
        nc = kc / (2 * math.pi * -math.expm1(-2 * kc))
        m = self.mu * self.kappa[..., None] + (n * kc)[:, None, :]
        k = m.norm(dim=-1)
        m = m / k[..., None]
        p = _Mixture(self.w, k, m)
        e = self.kappa * (_dot(self.mu, m) - 1) + kc * (_dot(n[:, None, :], m) - 1)
        p.w = self.w * self.norm() * nc / p.norm() * torch.exp(e)
        p.w = p.w / p.w.sum(1, keepdim=True)
        return p

    def sample(self, count, ux, uy):
        cum = torch.cumsum(self.w, 1)
        i = torch.minimum((cum < uy[:, None]).sum(1), count - 1)[:, None]
        w = self.w.gather(1, i)[:, 0]
        u1 = ((uy - (cum.gather(1, i)[:, 0] - w)) / w).clamp(max=1 - 2.0 ** -23)
        k = self.kappa.gather(1, i)[:, 0]
        mu = self.mu.gather(1, i[..., None].expand(-1, 1, 3))[:, 0]
        ks = torch.where(k > 0, k, torch.ones_like(k))
        ct = torch.where(k > 0, 1 + torch.log1p(torch.expm1(-2 * ks) * ux) / ks, 1 - 2 * u1).clamp(-1, 1)
        phi = 2 * math.pi * torch.where(k > 0, u1, ux)
        st = (1 - ct * ct).clamp(min=0).sqrt()
        return _frame_times(mu, torch.stack([st * phi.cos(), st * phi.sin(), ct], 1))


def _exact_queries(case, seed):
    field, scene, g = _train_query_field(case, seed)
    q = _query_records(case, scene, g).double()
    bounds, nodes, regions = _read_field(field.field_bytes(), case["mode"] == "volume")
    field.release()
    parts = []
    for a in range(0, len(q), 1 << 17):
        parts.append(_exact_part(case, q[a:a + (1 << 17)], bounds, nodes, regions))
    return {k: None if parts[0][k] is None else torch.cat([p[k] for p in parts]) for k in parts[0]}


def _exact_part(case, q, bounds, nodes, regions):
    n, vertices = len(q), case["mode"] == "vertices"
    pos, normal, s1d = q[:, 0:3], q[:, 3:6], q[:, 10 if vertices else 6]
    lo, hi = _f64(bounds[:3]), _f64(bounds[3:])
    ok = ((pos >= lo) & (pos <= hi)).all(1)
    # the leaf, then one of its nearest regions by the one-dimensional number
    split, bits = _f64(nodes["split"]), torch.as_tensor(nodes["bits"].astype(np.int64), device="cuda")
    at = torch.zeros(n, dtype=torch.int64, device="cuda")
    while True:
        dim, child = bits[at] >> 30, bits[at] & 0x3FFFFFFF
        inner = dim != 3
        if not bool(inner.any()):
            break
        c = pos.gather(1, dim.clamp(max=2)[:, None])[:, 0]
        at = torch.where(inner, child + (c >= split[at]).long(), at)
    leaf = child
    means = _f64(regions["stats"][:, 0:3])
    near = torch.cdist(means, means, compute_mode="donot_use_mm_for_euclid_dist").topk(min(8, len(means)), largest=False)[1]
    size = min(4, near.shape[1])
    sel = torch.floor(s1d * size)
    rest = torch.where(ok, (s1d - sel / size) * size, s1d)
    ids = near[leaf]
    order = (means[ids] - pos[:, None, :]).square().sum(-1).argsort(1)
    reg = ids.gather(1, order.gather(1, sel.long().clamp(max=size - 1)[:, None]))[:, 0]
    ok &= torch.as_tensor(regions["valid"].astype(bool), device="cuda")[reg]
    # the region's mixture as seen from the query point
    v = regions["vmm"].transpose(0, 2, 1, 3).reshape(len(regions), 9, 32)
    w, kappa, dist = _f64(v[:, 0])[reg], _f64(v[:, 1])[reg], _f64(v[:, 8])[reg]
    mu = _f64(v[:, 2:5].transpose(0, 2, 1))[reg]
    if case["field"] == "parallax":
        moved = mu * dist[..., None] + (_f64(regions["pivot"])[reg] - pos)[:, None, :]
        moved = moved / moved.norm(dim=-1, keepdim=True)
        mu = torch.where((dist > 0)[..., None], moved, mu)
    count = torch.as_tensor(regions["K"].astype(np.int64), device="cuda")[reg]
    seen = _Mixture(w, kappa, mu)
    used = seen if case["mode"] == "volume" else seen.times_cosine(normal)
    if vertices:
        cols = [rest[:, None]]
        for k in range(4):
            d = used.sample(count, q[:, 11 + 2 * k], q[:, 12 + 2 * k])
            cols.append(torch.where(ok[:, None], torch.cat([d, used.pdf(d)[:, None]], 1), torch.zeros(1, device="cuda").double()))
        return {"region": None, "sample": torch.cat(cols, 1)}
    d = used.sample(count, q[:, 7], q[:, 8])
    zero = torch.zeros(1, device="cuda", dtype=torch.float64)
    return {"region": None, "rest1d": rest, "direction": torch.where(ok[:, None], d, zero),
            "pdf": torch.where(ok[:, None], torch.stack([used.pdf(d), seen.pdf(d)], 1), zero)}


def _exact_paths(case, seed):
    seg, begin = _segments(case["paths"], case["length"], _rng(seed))
    paths, length = case["paths"], case["length"]
    lens = (begin[1:] - begin[:-1]).long()
    slot = torch.arange(length, device="cuda")
    there = slot[None, :] < lens[:, None]
    at = (begin[:-1].long()[:, None] + slot[None, :]).clamp(max=len(seg) - 1)
    s = seg.double()[at]  # [paths, length, 34]
    words = seg.view(torch.int32)[at]
    delta, volume = (words[..., 14] & 1) != 0, (words[..., 12] & 1) != 0
    f32 = lambda x: float(np.float32(x))  # noqa: E731
    last = torch.zeros(paths, dtype=torch.float64, device="cuda")
    record = torch.zeros(paths, length, 9, dtype=torch.float64, device="cuda")
    made = torch.zeros(paths, length, dtype=torch.bool, device="cuda")
    for i in range(length - 2, -1, -1):
        cur, have = s[:, i], there[:, i + 1]
        d = ((s[:, i + 1, 0:3] - cur[:, 0:3]).norm(dim=1) + last).clamp(max=200.0)
        stops = ~delta[:, i] & (cur[:, 30] >= f32(0.3))
        bent = d * (_dot(cur[:, 9:12], cur[:, 6:9]) / (_dot(cur[:, 9:12], cur[:, 3:6]) * cur[:, 29])).abs()
        step = torch.where(stops, torch.zeros_like(d), torch.where(cur[:, 29] != 1.0, bent, d))
        last = torch.where(have, step, last)
        t = torch.ones(paths, 3, dtype=torch.float64, device="cuda")
        c = torch.zeros_like(t)
        for j in range(i + 1, length):
            p, x, on = s[:, j - 1], s[:, j], there[:, j][:, None]
            t = torch.where(on, t * p[:, 18:21], t)
            ct = t.clamp(max=10.0)
            add = ct * x[:, 25:28]
            if j > i + 1:  # light at the next vertex itself is not guided to
                add = add + ct * x[:, 24:25] * x[:, 21:24]
            c = torch.where(on, c + add, c)
            rr = x[:, 28:29]
            t = torch.where(on, torch.where(rr > 0, t * x[:, 15:18] / torch.where(rr > 0, rr, torch.ones_like(rr)),
                                            torch.zeros_like(t)), t)
        pdf = cur[:, 13].clamp(min=f32(0.1))
        made[:, i] = have & ~delta[:, i] & (cur[:, 30] > f32(0.01)) & (c > 0).any(1) & (d > 0)
        record[:, i] = torch.cat([cur[:, 0:6], (c.sum(1) / 3 / pdf)[:, None], pdf[:, None], d[:, None]], 1)
    made, record, volume = made.flip(1), record.flip(1), volume.flip(1)  # the last vertex's sample comes first
    out = torch.zeros(paths * length, 9, dtype=torch.float64, device="cuda")
    rows = record[made]
    out[:len(rows)] = rows
    return {"begin": None, "flags": None, "record": out}
