"""Performance cases of the BVH builder: what a program has it do, over the range of sizes.

Every case goes through the package's public entry points, in one of these forms:

* ``call``    -- ``build_bvh8`` / ``build_bvh2`` with metrics: the reference-shaped call, which
  allocates its outputs, returns with the stream drained and reports the trees' SAH costs;
* ``builder`` -- ``Builder.build`` (resident workspace, new output tensors) and the SAH cost of the
  BVH8 (``nxb_eval_bvh8_cost``), by which a program decides whether to keep a tree;
* ``frame``   -- ``Builder.enqueue``: everything resident, nothing allocated, nothing waited for
  (a frame loop);
* ``batch``   -- ``Batch.build`` of many meshes;
* ``server``  -- a burst of requests submitted to a ``Server``, waited for and released;
* ``sort``    -- ``nxb_stage_radix_sort``, for callers that keep their own keys.

The order of BVH8 nodes in memory depends on scheduling (a node's index is the order in which its
parent was finished), so the node array of two builds of the same input is not the same sequence of
bytes.  What is returned of a BVH8 is therefore what does not depend on that order: its node and
leaf counts and, where the form has it, its cost over all nodes.  The BVH2's numbering is
deterministic: its nodes come back whole, byte for byte.
"""
import ctypes
import math
import random

import numpy as np
import torch

import nexusbvh_gb300 as nxb

_LARGEST = 12_582_912  # the benchmark's largest plain mesh


def listed():
    def plain(name, form, scene, n, bits, prim="triangle", radius=8, auction=False, wide=True):
        return {"name": name, "form": form, "scene": scene, "n": n, "bits": bits, "prim": prim, "radius": radius,
                "auction": auction, "wide": wide}

    return [
        # a single small object through the reference-shaped call: latency, launches
        plain("call-soup-1021", "call", "soup", 1021, 30),
        # instance boxes of a scene rebuilt every frame (63-bit codes, boxes, odd size)
        plain("frame-boxes-16411", "frame", "clustered", 16_411, 63, prim="box"),
        # the configuration's small plain mesh rebuilt every frame
        plain("frame-soup-65536", "frame", "soup", 65_536, 30),
        # BVH2 only, boxes of an ordinary mesh, odd size
        plain("call-bvh2-boxes-500009", "call", "clustered", 500_009, 63, prim="box", wide=False),
        # quality options on an ordinary mesh: auction slot assignment
        plain("builder-auction-1m", "builder", "sphere", 1_048_576, 30, auction=True),
        # the widest search radius
        plain("builder-radius16-3m", "builder", "clustered", 3_000_017, 63, radius=16),
        # the configuration's displaced sphere, a connected surface mesh
        plain("builder-sphere-4m", "builder", "sphere", 4_194_304, 63),
        # the headline mesh
        plain("builder-clustered-12m", "builder", "clustered", _LARGEST, 63),
        # many small objects at once: a scene's dynamic meshes
        {"name": "batch-200-small", "form": "batch", "meshes": 200, "lo": 16, "hi": 4096, "counts_seed": 7},
        # the configuration's batch
        {"name": "batch-1024", "form": "batch", "meshes": 1024, "lo": 256, "hi": 262_144, "counts_seed": 3},
        # the configuration's burst of small requests
        {"name": "server-burst-96", "form": "server", "requests": 96, "lo": 1024, "hi": 65_536, "counts_seed": 21},
        # a caller's own 64-bit keys, every bit of them in use
        {"name": "sort-64bit-5m", "form": "sort", "n": 5_000_011, "bits": 64},
    ]


def _log_u(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng: random.Random):
    form = rng.choices(["call", "builder", "frame", "batch", "server", "sort"], [3, 4, 3, 2, 1, 1])[0]
    if form == "batch":
        lo = _log_u(rng, 16, 256)
        return {"form": form, "meshes": _log_u(rng, 8, 900), "lo": lo, "hi": _log_u(rng, 4 * lo, 200_000),
                "counts_seed": rng.randrange(1 << 30)}
    if form == "server":
        return {"form": form, "requests": rng.randrange(16, 129), "lo": 1024, "hi": _log_u(rng, 8192, 65_536),
                "counts_seed": rng.randrange(1 << 30)}
    if form == "sort":
        return {"form": form, "n": _log_u(rng, 2000, 8_000_000), "bits": rng.choice([32, 64])}
    return {"form": form, "scene": rng.choice(["soup", "sphere", "clustered"]), "n": _log_u(rng, 300, 10_000_000),
            "bits": rng.choice([30, 63]), "prim": rng.choice(["triangle", "triangle", "box"]),
            "radius": rng.choice([8, 8, 8, 4, 16]), "auction": rng.random() < 0.15,
            "wide": form != "call" or rng.random() < 0.75}


# ---------------------------------------------------------------- scenes
# The distributions of nexusbvh_gb300.scenes, generated on the GPU.

def _gen(seed):
    return torch.Generator("cuda").manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _soup(n, g):
    return (_rand(g, n, 1, 3) + (_rand(g, n, 3, 3) - 0.5) * 0.01).reshape(n, 9)


def _sphere(n, g):
    """Triangles of a (2 nv x nv) grid on a displaced unit sphere, the first n of 4 nv^2."""
    nv = max(2, math.ceil(math.sqrt(n / 4)))
    nu = 2 * nv
    a = torch.randint(1, 65, (8,), generator=g, device="cuda")
    b = torch.randint(1, 65, (8,), generator=g, device="cuda")
    psi = _rand(g, 8).double() * (2 * math.pi)
    theta = torch.linspace(0.0, math.pi, nv + 1, dtype=torch.float64, device="cuda")[:, None]
    phi = (2 * math.pi / nu) * torch.arange(nu, dtype=torch.float64, device="cuda")[None, :]
    r = torch.ones(nv + 1, nu, dtype=torch.float64, device="cuda")
    for k in range(8):
        r += (0.02 / (k + 1)) * torch.sin(a[k] * theta + b[k] * phi + psi[k])
    st = torch.sin(theta)
    v = torch.stack([r * st * torch.cos(phi), r * st * torch.sin(phi), r * torch.cos(theta)], dim=-1).float()
    w = torch.roll(v, -1, dims=1)
    t1 = torch.cat([v[:-1], v[1:], w[1:]], dim=-1)
    t2 = torch.cat([v[:-1], w[1:], w[:-1]], dim=-1)
    return torch.stack([t1, t2], dim=2).reshape(-1, 9)[:n].contiguous()


def _clustered(n, g, components=256):
    means = _rand(g, components, 3)
    sigma = torch.exp(_rand(g, components, 3) * math.log(50.0) + math.log(0.001))
    weights = -torch.log(_rand(g, components).clamp_min(1e-12)).double()
    edges = torch.cumsum(weights / weights.sum(), 0)
    out = torch.empty(n, 9, device="cuda")
    for at in range(0, n, 1 << 22):
        m = min(1 << 22, n - at)
        comp = torch.searchsorted(edges, _rand(g, m).double()).clamp_max(components - 1)
        c = means[comp] + torch.randn(m, 3, generator=g, device="cuda") * sigma[comp]
        out[at:at + m, 0:3] = c
        for k in (1, 2):
            d = torch.randn(m, 3, generator=g, device="cuda")
            d /= d.norm(dim=1, keepdim=True).clamp_min(1e-12)
            length = torch.exp(torch.randn(m, 1, generator=g, device="cuda") - 6.0)
            out[at:at + m, 3 * k:3 * k + 3] = c + length * d
    return out


def _boxes(tris):
    v = tris.view(-1, 3, 3)
    return torch.cat([v.amin(1), v.amax(1)], dim=1).contiguous()


def _prims(case, seed):
    t = {"soup": _soup, "sphere": _sphere, "clustered": _clustered}[case["scene"]](case["n"], _gen(seed))
    return _boxes(t) if case["prim"] == "box" else t


def _counts(case, how_many):
    rng = np.random.default_rng(case["counts_seed"])
    lo, hi = case["lo"], case["hi"]
    return np.floor(np.exp(rng.uniform(np.log(lo), np.log(hi + 1), size=how_many))).astype(np.int64).clip(lo, hi)


def _batch_prims(counts, seed):
    """Meshes end to end: uniform soups, each in a box of its own."""
    g = _gen(seed)
    m = len(counts)
    origin = (_rand(g, m, 1, 3) - 0.5) * 200.0
    extent = torch.exp(_rand(g, m, 1, 3) * math.log(100.0) + math.log(0.1))
    mesh = torch.repeat_interleave(torch.arange(m, device="cuda"), torch.from_numpy(counts).cuda())
    soup = _soup(int(counts.sum()), g).view(-1, 3, 3)
    return (origin[mesh] + soup * extent[mesh]).reshape(-1, 9)


# ---------------------------------------------------------------- cases
class _DeviceArray:
    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3,
                                         "strides": None}


def _config(case):
    return nxb.BuildConfig(prioritize_speed=case["bits"] == 30, search_radius=case["radius"],
                           auction=case["auction"])


def prepare(case, seed):
    form = case["form"]
    s = {"case": case}
    if form == "batch":
        counts = _counts(case, case["meshes"])
        s["prims"] = _batch_prims(counts, seed)
        s["batch"] = nxb.Batch(counts)
        a = s["batch"].arrays()
        s["bvh2"] = torch.as_tensor(_DeviceArray(a.bvh2_nodes, (a.bvh2_node_capacity, 8), "<i4", s["batch"]),
                                    device="cuda")
        s["bvh2"].owner = s["batch"]  # the nodes are the batch's memory: it lives as long as they are looked at
        s["bvh2"].zero_()  # the arrays have one unused node between two meshes
        return s
    if form == "server":
        counts = _counts(case, case["requests"])
        s["meshes"] = [t.contiguous() for t in torch.split(_batch_prims(counts, seed), counts.tolist())]
        s["server"] = nxb.Server()
        s["config"] = nxb.BuildConfig(prioritize_speed=True)
        torch.cuda.synchronize()  # the server reads device inputs on streams of its own
        return s
    if form == "sort":
        n, kb = case["n"], case["bits"] // 8
        lib = nxb.load()
        s["keys"] = torch.randint(-2 ** 31, 2 ** 31, (n, kb // 4), generator=_gen(seed), device="cuda",
                                  dtype=torch.int64).to(torch.int32).view(torch.int64 if kb == 8 else torch.int32).view(n)
        s["out_keys"] = torch.empty_like(s["keys"])
        s["out_vals"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["scratch"] = torch.empty(lib.nxb_sort_scratch_bytes(n, kb, 0, 8 * kb), dtype=torch.uint8, device="cuda")
        s["err"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        return s
    n = case["n"]
    s["prims"] = _prims(case, seed)
    s["config"] = _config(case)
    if form == "builder":
        s["builder"] = nxb.Builder()
    if form == "frame":
        s["builder"] = nxb.Builder()
        z = s["builder"].sizes(n, s["config"])
        s["ws"] = s["builder"].workspace(z.workspace_bytes)
        s["bvh2"] = torch.empty((z.bvh2_node_count, 32), dtype=torch.uint8, device="cuda")
        s["bvh8"] = torch.empty((z.bvh8_node_capacity, 80), dtype=torch.uint8, device="cuda")
        s["prim_idx"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["result"] = torch.zeros(ctypes.sizeof(nxb.CResult), dtype=torch.uint8, device="cuda")
    return s


def run(s):
    case = s["case"]
    form = case["form"]
    if form == "frame":
        s["builder"].enqueue(s["prims"], case["n"], s["config"], s["ws"], s["bvh2"], s["bvh8"], s["prim_idx"],
                             s["result"])
        return {"bvh2": s["bvh2"].view(torch.int32), "result": s["result"].view(torch.int32)}
    if form == "builder":
        b8 = s["builder"].build(s["prims"], s["config"])
        # the root's box is the last BVH2 node's first 24 bytes
        cost = torch.empty(1, dtype=torch.float32, device="cuda")
        nxb.check(nxb.load().nxb_eval_bvh8_cost(b8.nodes.data_ptr(), b8.node_count, b8.bvh2.nodes[-1].data_ptr(),
                                                cost.data_ptr(), int(torch.cuda.current_stream().cuda_stream)),
                  "nxb_eval_bvh8_cost")
        return {"bvh2": b8.bvh2.nodes.view(torch.int32), "bvh8_nodes": b8.node_count, "bvh8_cost": cost,
                "bounds": np.asarray(b8.bounds, dtype=np.float32)}
    if form == "call":
        m = nxb.BVHBuildMetrics()
        if case["wide"]:
            b = nxb.build_bvh8(s["prims"], s["config"], m)
            return {"bvh8_nodes": b.node_count, "bounds": np.asarray(b.bounds, dtype=np.float32),
                    "bvh2_cost": m.bvh2_cost, "bvh8_cost": m.bvh8_cost, "children": m.average_child_per_node}
        b = nxb.build_bvh2(s["prims"], s["config"], m)
        return {"bvh2": b.nodes.view(torch.int32), "bounds": np.asarray(b.bounds, dtype=np.float32),
                "bvh2_cost": m.bvh2_cost}
    if form == "batch":
        meshes = s["batch"].build(s["prims"])
        return {"bvh2": s["bvh2"], "meshes": np.frombuffer(bytes(b"".join(bytes(x) for x in meshes)), dtype=np.int32)}
    if form == "server":
        server = s["server"]
        tickets = [server.submit(p, s["config"]) for p in s["meshes"]]
        counts, bounds = [], []
        for t in tickets:
            r = server.wait(t)
            counts.append(r.bvh8.node_count)
            bounds.append(tuple(r.bvh8.bounds.bmin) + tuple(r.bvh8.bounds.bmax))
            server.release(t)
        return {"bvh8_nodes": np.asarray(counts, dtype=np.int64), "bounds": np.asarray(bounds, dtype=np.float32)}
    kb = case["bits"] // 8
    nxb.check(nxb.load().nxb_stage_radix_sort(kb, s["keys"].data_ptr(), s["out_keys"].data_ptr(), None,
                                              s["out_vals"].data_ptr(), case["n"], 0, 8 * kb, s["scratch"].data_ptr(),
                                              s["scratch"].numel(), s["err"].data_ptr(),
                                              int(torch.cuda.current_stream().cuda_stream)), "nxb_stage_radix_sort")
    return {"keys": s["out_keys"], "values": s["out_vals"]}


def exact(case, seed):
    """The scene boxes in 64 bits.  Node arrays, counts and sorted keys are whole numbers; the costs sum over trees
    that no other code builds."""
    form = case["form"]
    if form in ("call", "builder"):
        p = _prims(case, seed).double().view(case["n"], -1, 3)
        bounds = torch.stack([p.amin((0, 1)), p.amax((0, 1))]).cpu().numpy()
        if form == "builder":
            return {"bvh2": None, "bvh8_nodes": None, "bvh8_cost": None, "bounds": bounds}
        if case["wide"]:
            return {"bvh8_nodes": None, "bounds": bounds, "bvh2_cost": None, "bvh8_cost": None, "children": None}
        return {"bvh2": None, "bounds": bounds, "bvh2_cost": None}
    if form == "server":
        counts = _counts(case, case["requests"])
        rows = []
        for t in torch.split(_batch_prims(counts, seed).double(), counts.tolist()):
            v = t.view(-1, 3)
            rows.append(torch.cat([v.amin(0), v.amax(0)]))
        return {"bvh8_nodes": None, "bounds": torch.stack(rows).cpu().numpy()}
    return None


def work(case):
    """Input primitives read once, the outputs of the form written once (BVH2 nodes 32 bytes, BVH8 nodes 80 bytes,
    about one per five primitives, and the primitive order)."""
    form = case["form"]
    if form == "sort":
        return {"bytes": case["n"] * (2 * case["bits"] // 8 + 4), "flops": 0}
    bvh8 = 80 / 5 + 4
    if form == "batch":
        return {"bytes": float(_counts(case, case["meshes"]).sum()) * (36 + 64 + bvh8), "flops": 0}
    if form == "server":
        return {"bytes": float(_counts(case, case["requests"]).sum()) * (36 + bvh8), "flops": 0}
    per = 36 if case["prim"] == "triangle" else 24
    if form == "call":
        per += bvh8 if case["wide"] else 64
    else:
        per += 64 + bvh8
    return {"bytes": float(case["n"]) * per, "flops": 0}
