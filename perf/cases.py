"""The workloads that this framework is timed on: builds, the batched queries on point and box trees,
collisions, forests and bulk insert, through the Python binding (octree_gb300) as a program with its
data on the GPU calls it; the smallest workload takes host arrays and gives host arrays back.

A case is a dict: "op" names the workload, the other values its sizes and types. Entities follow the
distributions of bench.py (uniform points, points with a noisy sphere shell, uniform and clustered
boxes); domains grow with the entity count, so that densities stay those of the named workloads.
"""
import ctypes
import math

import numpy as np
import torch

import octree_gb300 as otg

_TORCH = {"f64": torch.float64, "f32": torch.float32}
_NUMPY = {"f64": np.float64, "f32": np.float32}


def listed():
    return [
        # the smallest use: a few hundred host points, a handful of queries, answers on the host
        {"name": "small_points", "op": "small", "n": 777, "nq": 5, "k": 4, "dtype": "f64"},
        # the headline build (16M points, depth 10, 20 per node), handed on as static linear arrays
        {"name": "rebuild_points_16m", "op": "rebuild", "n": 16_000_000, "depth": 10, "elems": 20, "dtype": "f64"},
        # points arriving in a bulk at a tree that is built anew, then asked about
        {"name": "grow_points_4m", "op": "grow", "n": 4_000_000, "add": 262_144, "nq": 4096, "dtype": "f64"},
        # 10k range boxes on 1M uniform points
        {"name": "range_points_1m", "op": "range_points", "n": 1_000_000, "nq": 10_000, "dtype": "f64"},
        # k = 8 neighbours of 10k points on 1M uniform points
        {"name": "knn_1m_k8", "op": "knn", "n": 1_000_000, "nq": 10_000, "kmin": 8, "kmax": 8, "shell": False, "dtype": "f64"},
        # a million neighbour queries of uneven k on 16M points with a dense shell
        {"name": "knn_16m_uneven", "op": "knn", "n": 16_000_000, "nq": 1_000_000, "kmin": 1, "kmax": 64, "shell": True, "dtype": "f64"},
        # overlap range search and picking on single-precision boxes, odd counts
        {"name": "range_pick_boxes", "op": "range_boxes", "n": 500_009, "nq": 30_011, "dtype": "f32"},
        # all and first hits of rays through double-precision boxes
        {"name": "rays_1m", "op": "rays", "n": 1_000_000, "nq": 30_000, "dtype": "f64"},
        # camera frusta and planes over double-precision boxes
        {"name": "frustum_planes_1m", "op": "frustum", "n": 1_000_000, "nq": 64, "dtype": "f64"},
        # self collision of 4M boxes, half of them in clusters
        {"name": "self_collision_4m", "op": "self_collision", "n": 4_000_000, "depth": 12, "elems": 32, "dtype": "f64"},
        # one step of two scenes: the moving boxes' tree built anew, then its pairs with the static tree
        {"name": "pair_step_16m_8m", "op": "pair_step", "na": 16_000_000, "nb": 8_000_000, "dtype": "f64"},
        # one step of many small trees: one forest build, then ranges, rays and a frustum per tree
        {"name": "forest_step_4096", "op": "forest", "trees": 4096, "per_tree": 256, "dtype": "f32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["small", "rebuild", "grow", "range_points", "knn", "range_boxes", "rays", "frustum", "self_collision", "pair_step", "forest"])
    dtype = rng.choice(["f64", "f64", "f32"])
    if op == "small":
        return {"op": op, "n": _log(rng, 20, 20_000), "nq": _log(rng, 1, 200), "k": rng.randint(1, 20), "dtype": dtype}
    if op == "rebuild":
        return {"op": op, "n": _log(rng, 10_000, 16_000_000), "depth": rng.randint(7, 12), "elems": rng.choice([8, 16, 20, 32]), "dtype": dtype}
    if op == "grow":
        n = _log(rng, 20_000, 8_000_000)
        return {"op": op, "n": n, "add": max(1, n // rng.randint(8, 64)), "nq": _log(rng, 64, 20_000), "dtype": dtype}
    if op == "range_points":
        return {"op": op, "n": _log(rng, 50_000, 8_000_000), "nq": _log(rng, 50, 200_000), "dtype": dtype}
    if op == "knn":
        n = _log(rng, 50_000, 16_000_000)
        k = rng.randint(1, 64)
        return {"op": op, "n": n, "nq": _log(rng, 50, 500_000), "kmin": rng.choice([1, k]), "kmax": k, "shell": rng.random() < 0.5, "dtype": dtype}
    if op == "range_boxes":
        return {"op": op, "n": _log(rng, 20_000, 4_000_000), "nq": _log(rng, 50, 100_000), "dtype": dtype}
    if op == "rays":
        return {"op": op, "n": _log(rng, 20_000, 2_000_000), "nq": _log(rng, 50, 40_000), "dtype": dtype}
    if op == "frustum":
        return {"op": op, "n": _log(rng, 20_000, 2_000_000), "nq": _log(rng, 1, 128), "dtype": dtype}
    if op == "self_collision":
        return {"op": op, "n": _log(rng, 20_000, 4_000_000), "depth": rng.randint(8, 12), "elems": rng.choice([16, 20, 32]), "dtype": dtype}
    if op == "pair_step":
        na = _log(rng, 50_000, 16_000_000)
        return {"op": op, "na": na, "nb": max(1000, na // rng.randint(2, 9)), "dtype": dtype}
    return {"op": op, "trees": _log(rng, 8, 3000), "per_tree": rng.randint(16, 256), "dtype": "f32"}


# ---------------------------------------------------------------------------- inputs
class _Draws:
    """Seeded random arrays on the GPU, drawn in double precision."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def uniform(self, *shape):
        return torch.rand(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def integers(self, lo, hi, n):
        return torch.randint(lo, hi, (n,), generator=self.g, device="cuda")

    def directions(self, n):
        d = self.normal(n, 3)
        return d / d.norm(dim=1, keepdim=True)

    def permuted(self, a):
        return a[torch.randperm(len(a), generator=self.g, device="cuda")]

    def shell_points(self, n):
        """70% uniform in [0,1)^3, 30% on a sphere shell r = 0.4, radius noise 0.005 (bench.py: shell_points)."""
        s = int(n * 0.3)
        shell = 0.5 + self.directions(s) * (0.4 + 0.005 * self.normal(s, 1))
        return self.permuted(torch.cat([self.uniform(n - s, 3), shell]))

    def boxes_around(self, centre, half):
        return torch.cat([centre - half, centre + half], 1)

    def uniform_boxes(self, n, side):
        """Half-extents uniform in [0.05, 1] (bench.py: many_trees)."""
        return self.boxes_around(self.uniform(n, 3) * side, 0.05 + 0.95 * self.uniform(n, 3))

    def lognormal_boxes(self, n, side):
        """Half-extents lognormal(ln 1, 0.8) (bench.py: two_tree_boxes)."""
        return self.boxes_around(self.uniform(n, 3) * side, torch.exp(0.8 * self.normal(n, 3)))

    def clustered_boxes(self, n, side):
        """Half uniform, half in 64 Gaussian clusters; half-extents lognormal(ln 0.5, 0.6) (bench.py: cluster_boxes)."""
        h = n // 2
        heart = self.uniform(64, 3) * side
        c = torch.cat([self.uniform(h, 3) * side, heart[self.integers(0, 64, n - h)] + 0.01 * side * self.normal(n - h, 3)])
        return self.boxes_around(c, 0.5 * torch.exp(0.6 * self.normal(n, 3)))

    def range_boxes(self, n, side):
        """Edge lengths uniform in [0.5, 5] (bench.py: c1_workload)."""
        return self.boxes_around(self.uniform(n, 3) * side, 0.25 + 2.25 * self.uniform(n, 3))

    def rays(self, n, side):
        return torch.cat([self.uniform(n, 3) * side, self.directions(n)], 1)

    def planes(self, n, side):
        """Normalised planes through points of the domain: {origo distance, normal}."""
        nrm = self.directions(n)
        return torch.cat([(nrm * self.uniform(n, 3) * side).sum(1, keepdim=True), nrm], 1)

    def frusta(self, n, side):
        """Six planes per view, normals inwards: a 60 degree pyramid from a point of the domain, near and far plane."""
        eye, f = self.uniform(n, 3) * side, self.directions(n)
        up = torch.linalg.cross(f, self.directions(n))
        up = up / up.norm(dim=1, keepdim=True)
        right = torch.linalg.cross(f, up)
        s, c = math.sin(math.radians(30)), math.cos(math.radians(30))
        out = []
        for nrm, at in ((s * f + c * right, eye), (s * f - c * right, eye), (s * f + c * up, eye), (s * f - c * up, eye),
                        (f, eye + 0.01 * side * f), (-f, eye + 0.6 * side * f)):
            out.append(torch.cat([(nrm * at).sum(1, keepdim=True), nrm], 1))
        return torch.stack(out, 1)


def _tree_sizes(trees):
    """The quantiles of lognormal(ln 8000, 1.2), clipped to [1000, 200000] (bench.py: many_trees)."""
    u = (torch.arange(trees, device="cuda", dtype=torch.float64) + 0.5) / trees
    return torch.exp(math.log(8000.0) + 1.2 * math.sqrt(2.0) * torch.erfinv(2 * u - 1)).clamp(1000, 200_000).to(torch.int64)


def _side(n, of=1_000_000, side=100.0):
    """Edge of the domain that holds n entities at the density of `of` entities in a cube of edge `side`."""
    return side * (n / of) ** (1.0 / 3.0)


def _inputs(case, seed):
    """The arrays of a case on the GPU in its scalar type ("small": also there; prepare() takes them to the host)."""
    g, t, op = _Draws(seed), _TORCH[case["dtype"]], case["op"]
    if op == "small":
        s = {"points": g.uniform(case["n"], 3) * 10, "ranges": g.range_boxes(case["nq"], 10.0), "queries": g.uniform(case["nq"], 3) * 10}
    elif op == "rebuild":
        s = {"points": g.shell_points(case["n"])}
    elif op == "grow":
        s = {"points": g.shell_points(case["n"]), "add": g.shell_points(case["add"]), "queries": g.shell_points(case["nq"]),
             "space": torch.tensor([[-0.01] * 3 + [1.01] * 3], device="cuda", dtype=torch.float64)}
    elif op == "range_points":
        side = _side(case["n"])
        s = {"points": g.uniform(case["n"], 3) * side, "ranges": g.range_boxes(case["nq"], side)}
    elif op == "knn":
        make = g.shell_points if case["shell"] else lambda n: g.uniform(n, 3) * _side(case["n"])
        s = {"points": make(case["n"]), "queries": make(case["nq"])}
        if case["kmin"] != case["kmax"]:
            s["k"] = g.integers(case["kmin"], case["kmax"] + 1, case["nq"]).to(torch.int32)
    elif op == "range_boxes":
        side = _side(case["n"])
        s = {"boxes": g.uniform_boxes(case["n"], side), "ranges": g.range_boxes(case["nq"], side), "queries": g.uniform(case["nq"], 3) * side}
    elif op == "rays":
        side = _side(case["n"])
        s = {"boxes": g.uniform_boxes(case["n"], side), "rays": g.rays(case["nq"], side)}
    elif op == "frustum":
        side = _side(case["n"])
        s = {"boxes": g.uniform_boxes(case["n"], side), "frusta": g.frusta(case["nq"], side), "planes": g.planes(case["nq"], side),
             "halves": g.planes(max(1, case["nq"] // 8), side)}
    elif op == "self_collision":
        s = {"boxes": g.clustered_boxes(case["n"], _side(case["n"], 4_000_000, 1000.0))}
    elif op == "pair_step":
        side = _side(case["na"], 16_000_000, 4096.0)
        s = {"static": g.lognormal_boxes(case["na"], side), "moving": g.lognormal_boxes(case["nb"], side)}
    else:
        off = np.concatenate([[0], np.cumsum(g.permuted(_tree_sizes(case["trees"])).cpu().numpy())]).astype(np.uint64)
        nq = case["trees"] * case["per_tree"]
        lo, hi = g.uniform(case["trees"], 3) * 40, 60 + g.uniform(case["trees"], 3) * 40
        pl = torch.zeros(case["trees"], 6, 4, device="cuda", dtype=torch.float64)
        for a in range(3):
            pl[:, 2 * a, 0], pl[:, 2 * a, 1 + a] = lo[:, a], 1.0
            pl[:, 2 * a + 1, 0], pl[:, 2 * a + 1, 1 + a] = -hi[:, a], -1.0
        s = {"boxes": g.uniform_boxes(int(off[-1]), 100.0), "ranges": g.range_boxes(nq, 100.0), "rays": g.rays(nq, 100.0), "planes": pl}
        return {k: v.to(t).contiguous() for k, v in s.items()} | {"off": off}
    return {k: (v if k == "k" else v.to(t).contiguous()) for k, v in s.items()}


def prepare(case, seed):
    s, dt, op = _inputs(case, seed), _NUMPY[case["dtype"]], case["op"]
    s["op"], s["kept"] = op, _keep(case)
    if op == "small":
        for k in ("points", "ranges", "queries"):
            s[k] = s[k].cpu().numpy()
        s["tree"], s["k"] = otg.Tree("points", dt), case["k"]
    elif op == "rebuild":
        s["tree"], s["depth"], s["elems"] = otg.Tree("points", dt), case["depth"], case["elems"]
    elif op == "grow":
        s["tree"] = otg.Tree("points", dt)
    elif op in ("range_points", "knn"):
        s["tree"] = otg.Tree("points", dt).create(s.pop("points"), max_depth=10, max_elements=20)
        s.setdefault("k", case.get("kmax", 0))
    elif op in ("range_boxes", "rays", "frustum"):
        s["tree"] = otg.Tree("boxes", dt).create(s.pop("boxes"))
    elif op == "self_collision":
        s["tree"] = otg.Tree("boxes", dt).create(s.pop("boxes"), max_depth=case["depth"], max_elements=case["elems"])
    elif op == "pair_step":
        s["tree"], s["other"] = otg.Tree("boxes", dt).create(s.pop("static")), otg.Tree("boxes", dt)
    else:
        s["forest"] = otg.Forest("boxes", dt)
        s["query_off"] = np.arange(case["trees"] + 1, dtype=np.uint64) * np.uint64(case["per_tree"])
        s["view_off"] = np.arange(case["trees"] + 1, dtype=np.uint64)
    if "tree" in s and op in ("range_points", "knn", "range_boxes", "rays", "frustum", "self_collision", "pair_step"):
        s["tree"].sync()
    return s


# ---------------------------------------------------------------------------- one pass
class _Kept:
    """The arrays that a program keeps for one query's results: offsets, and room for `room` ids and
    distances; on the GPU, or on the host."""

    def __init__(self, nq, room, dist=False, host=False):
        self.room, self.host = room, host
        if host:
            self.arrays = [np.zeros(nq + 1, np.uint64), np.zeros(room, np.uint32)] + ([np.zeros(room)] if dist else [])
        else:
            z = lambda n, t: torch.zeros(n, device="cuda", dtype=t)
            self.arrays = [z(nq + 1, torch.int64), z(room, torch.int32)] + ([z(room, torch.float64)] if dist else [])

    def take(self, result):
        """The result into these arrays."""
        if self.host:
            for kept, got in zip(self.arrays, result):
                kept[: len(got)] = got
            return tuple(self.arrays)
        if result.sizes()[1] > self.room:
            raise ValueError("more results than there is room for: %d > %d" % (result.sizes()[1], self.room))
        p = [ctypes.c_void_p(t.data_ptr()) for t in self.arrays] + [None]
        if otg.library().otg_result_copy(result.h, p[0], p[1], p[2], otg.MEM_DEVICE, None) != otg.OTG_OK:
            raise otg.OtgError("copying a result")
        return tuple(self.arrays)


class _DeviceArray:
    """A device array owned by the framework, for torch to read in place."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr or 0, False), "version": 3}


def _static(tree, kept):
    """The tree as static linear arrays, into the program's own arrays."""
    lay = otg.StaticLayout()
    if otg.library().otg_tree_export_static(tree.h, ctypes.byref(lay), None) != otg.OTG_OK:
        raise otg.OtgError("static export")
    m, f = lay.node_count, "<f%d" % lay.scalar_bytes
    if m > len(kept["depths"]):
        raise ValueError("more nodes than there is room for: %d" % m)
    for name, ptr, shape, typestr in (("child_begins", lay.child_begins, (m + 1,), "<i4"), ("segments", lay.entity_segments, (m, 2), "<i4"),
                                      ("depths", lay.depth_ids, (m,), "|u1"), ("entities", lay.entity_storage, (lay.entity_count,), "<i4"),
                                      ("geometry", lay.geometry, (m, lay.geometry_per_node), f)):
        kept[name][: shape[0]].copy_(torch.as_tensor(_DeviceArray(ptr, shape, typestr), device="cuda"))
    return {k: kept[k] for k in ("child_begins", "segments", "depths", "entities", "geometry")}


def _room(mean, spread, nq):
    """Room for the results of nq queries with `mean` results each, `spread` their standard deviation."""
    return int(mean * nq + 8 * spread * math.sqrt(nq)) + 1024


def _keep(case):
    """The arrays that the program keeps for a case's results."""
    op, nq = case["op"], case.get("nq", 0)
    if op == "small":
        return {"range": _Kept(nq, nq * case["n"], host=True), "knn": _Kept(nq, nq * min(case["k"], case["n"]), dist=True, host=True)}
    if op == "rebuild":
        m, z = int(0.6 * case["n"]) + 64, lambda *a: torch.zeros(*a[:-1], device="cuda", dtype=a[-1])
        return {"child_begins": z(m + 1, torch.int32), "segments": z(m, 2, torch.int32), "depths": z(m, torch.uint8),
                "entities": z(case["n"], torch.int32), "geometry": z(m, 3, _TORCH[case["dtype"]])}
    if op == "grow":
        return {"knn": _Kept(nq, nq * 8, dist=True)}
    if op == "range_points":
        return {"range": _Kept(nq, _room(20.8, 20, nq))}
    if op == "knn":
        return {"knn": _Kept(nq, nq * case["kmax"] + 64, dist=True)}
    side = _side(case.get("n", 0))
    if op == "range_boxes":
        return {"range": _Kept(nq, _room(56, 40, nq)), "pick": _Kept(nq, _room(1.3, 1.5, nq))}
    if op == "rays":
        return {"all": _Kept(nq, _room(0.85 * side, 0.6 * side + 10, nq), dist=True), "first": _Kept(nq, 8 * nq + 1024, dist=True)}
    if op == "frustum":
        halves = max(1, nq // 8)
        return {"frustum": _Kept(nq, int(0.16 * case["n"] * nq) + 4096), "plane": _Kept(nq, int(3 * side * side * nq) + 4096),
                "half": _Kept(halves, halves * case["n"])}
    if op == "self_collision":
        return {"pairs": _Kept(1, int(6.5 * case["n"]) + 4096)}
    if op == "pair_step":
        return {"pairs": _Kept(1, int(0.12 * case["nb"]) + 4096)}
    nq, n = case["trees"] * case["per_tree"], int(_tree_sizes(case["trees"]).sum())
    return {"range": _Kept(nq, nq // 2 + 8192), "rays": _Kept(nq, 2 * nq + 8192, dist=True), "frustum": _Kept(case["trees"], n)}


def run(s):
    op, kept = s["op"], s["kept"]
    if op == "small":
        t = s["tree"].create(s["points"])
        return {"range": kept["range"].take(t.range_search(s["ranges"])[:2]), "knn": kept["knn"].take(t.knn(s["queries"], s["k"]))}
    if op == "rebuild":
        return _static(s["tree"].create(s["points"], max_depth=s["depth"], max_elements=s["elems"]), kept)
    if op == "grow":
        t = s["tree"].create(s["points"], max_depth=10, box=s["space"], max_elements=20)
        t.insert(s["add"])
        return {"knn": kept["knn"].take(t.knn(s["queries"], 8, raw=True))}
    t = s.get("tree")
    if op == "range_points":
        return {"range": kept["range"].take(t.range_search(s["ranges"], raw=True))}
    if op == "knn":
        return {"knn": kept["knn"].take(t.knn(s["queries"], s["k"], raw=True))}
    if op == "range_boxes":
        return {"range": kept["range"].take(t.range_search(s["ranges"], mode=otg.RANGE_OVERLAP, raw=True)),
                "pick": kept["pick"].take(t.pick_search(s["queries"], raw=True))}
    if op == "rays":
        return {"all": kept["all"].take(t.ray_all(s["rays"], raw=True)), "first": kept["first"].take(t.ray_first(s["rays"], raw=True))}
    if op == "frustum":
        return {"frustum": kept["frustum"].take(t.frustum_culling(s["frusta"], raw=True)), "plane": kept["plane"].take(t.plane_search(s["planes"], raw=True)),
                "half": kept["half"].take(t.plane_positive_segmentation(s["halves"], raw=True))}
    if op == "self_collision":
        return {"pairs": kept["pairs"].take(t.collision_self(raw=True))}
    if op == "pair_step":
        s["other"].create(s["moving"])
        return {"pairs": kept["pairs"].take(t.collision_pair(s["other"], raw=True))}
    f = s["forest"].create(s["boxes"], s["off"])
    return {"range": kept["range"].take(f.range_search(s["ranges"], s["query_off"], raw=True)),
            "rays": kept["rays"].take(f.ray_all(s["rays"], s["query_off"], raw=True)),
            "frustum": kept["frustum"].take(f.frustum_culling(s["planes"], s["view_off"], raw=True))}


# ---------------------------------------------------------------------------- work and exact values
def work(case):
    """Bytes: the entities or the part of them that is in the results, the queries and the results, once
    each. Flops: the comparisons and arithmetic of the accepted tests alone (a box or distance test about 12)."""
    w, op = {"f64": 8, "f32": 4}[case["dtype"]], case["op"]
    if op == "small":
        hits = case["nq"] * (1 + 20.8 * case["n"] / 1000.0 + case["k"])
        return {"bytes": case["n"] * 3 * w + case["nq"] * (9 * w + 16) + hits * 12, "flops": hits * 12}
    if op == "rebuild":
        # entities in, ids and the nodes (about one per five entities: begins, segment, depth, min point) out
        return {"bytes": case["n"] * (3 * w + 4) + case["n"] / 5 * (13 + 3 * w), "flops": case["n"] * 12}
    if op == "grow":
        return {"bytes": (case["n"] + case["add"]) * (3 * w + 4) + case["nq"] * (3 * w + 8 + 8 * 12), "flops": case["n"] * 12}
    if op == "range_points":
        hits = case["nq"] * 20.8
        return {"bytes": min(hits, case["n"]) * 3 * w + case["nq"] * (6 * w + 8) + hits * 4, "flops": hits * 12}
    if op == "knn":
        hits = case["nq"] * (case["kmin"] + case["kmax"]) / 2
        return {"bytes": min(hits, case["n"]) * 3 * w + case["nq"] * (3 * w + 12) + hits * 12, "flops": hits * 12}
    if op == "range_boxes":
        hits = case["nq"] * (55.0 + 1.2)
        return {"bytes": min(hits, case["n"]) * 6 * w + case["nq"] * (9 * w + 16) + hits * 4, "flops": hits * 12}
    if op == "rays":
        hits = case["nq"] * 1.65 * 0.5 * _side(case["n"])
        return {"bytes": min(hits, case["n"]) * 6 * w + case["nq"] * (6 * w + 16) + hits * 12, "flops": hits * 24}
    if op == "frustum":
        hits = case["nq"] * case["n"] * 0.03 + max(1, case["nq"] // 8) * case["n"] * 0.5
        return {"bytes": case["n"] * 6 * w + case["nq"] * (28 * w + 16) + hits * 4, "flops": hits * 36}
    if op == "self_collision":
        return {"bytes": case["n"] * (6 * w + 20), "flops": case["n"] * 30}
    if op == "pair_step":
        return {"bytes": (case["na"] + case["nb"]) * 6 * w + case["nb"] * 4, "flops": case["nb"] * 30}
    n, nq = case["trees"] * 15_500, case["trees"] * case["per_tree"]
    hits = nq * (0.5 + 0.8) + n * 0.2
    return {"bytes": n * 7 * w + nq * (12 * w + 16) + hits * 4, "flops": n * 12 + hits * 12}


def _near(points, queries, k):
    """The k smallest distances of each query, ascending, in double precision."""
    p, out = points.double(), []
    step = max(1, 100_000_000 // len(p))
    for q in queries.double().split(step):
        d2 = torch.zeros(len(q), len(p), device=p.device, dtype=torch.float64)
        for a in range(3):
            d2 += (q[:, a : a + 1] - p[None, :, a]).square_()
        out.append(d2.topk(k, dim=1, largest=False).values.sort(dim=1).values.sqrt_())
    return torch.cat(out)


def _ray_hits(boxes, rays, tol):
    """Enter distances of every (ray, box) hit, by ray and distance, in double precision."""
    b, out = boxes.double(), []
    for r in rays.double().split(max(1, 50_000_000 // len(b))):
        enter = torch.full((len(r), len(b)), -math.inf, device=b.device, dtype=torch.float64)
        leave = torch.full_like(enter, math.inf)
        for a in range(3):
            x = (b[None, :, a] - r[:, a : a + 1]) / r[:, 3 + a : 4 + a]
            y = (b[None, :, 3 + a] - r[:, a : a + 1]) / r[:, 3 + a : 4 + a]
            enter = torch.maximum(enter, torch.minimum(x, y))
            leave = torch.minimum(leave, torch.maximum(x, y))
        hit = (enter - 0.5 * tol < leave + 0.5 * tol) & (leave + 0.5 * tol > 0)
        q = hit.nonzero()[:, 0]
        d = (enter[hit] - 0.5 * tol).clamp_(min=0)
        d, at = d.sort()
        out.append(d[q[at].sort(stable=True).indices])
    return torch.cat(out)


def _padded(values, room):
    return torch.cat([values, values.new_zeros(room - len(values))])


def exact(case, seed):
    op = case["op"]
    if op == "small":
        s = _inputs(case, seed)
        d = _near(s["points"], s["queries"], min(case["k"], case["n"])).reshape(-1).cpu().numpy()
        return {"range": (None, None), "knn": (None, None, d)}
    if op == "grow" and (case["n"] + case["add"]) * case["nq"] <= 5e10:
        s = _inputs(case, seed)
        return {"knn": (None, None, _near(torch.cat([s["points"], s["add"]]), s["queries"], 8).reshape(-1))}
    if op == "knn" and case["n"] * case["nq"] <= 5e10:
        s = _inputs(case, seed)
        d = _near(s["points"], s["queries"], case["kmax"])
        if "k" in s:
            d = d[torch.arange(case["kmax"], device=d.device)[None, :] < s["k"][:, None]]
        return {"knn": (None, None, _padded(d.reshape(-1), case["nq"] * case["kmax"] + 64))}
    if op == "rays" and case["dtype"] == "f64" and case["n"] * case["nq"] <= 5e10:
        s = _inputs(case, seed)
        return {"all": (None, None, _padded(_ray_hits(s["boxes"], s["rays"], 100 * 2.0**-52), _keep(case)["all"].room)), "first": (None, None, None)}
    return None
