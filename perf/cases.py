"""The work that users of this package have it do, as a list of measurable cases.

A case is one call (or the few calls that belong together) on the package's
public entry points, with inputs that stand for a real use: label-tree solves
of small to large volumes, batches, gradients for training, graph solves, the
filter facade on host images, the vote and energy of a labelling, and the
data-term producers that precede a solve.

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  inputs and the solver a program keeps, made from the seed
  run(state)           one pass through the public entry points
  work(case)           bytes and operations one pass cannot do without
  exact(case, seed)    the same outputs in double precision with plain torch

Volumes are float32 [VZ, VY, VX].  Phantoms are painted ellipsoids with
Gaussian noise, data terms the Gaussian negative log-likelihood of each class,
smoothness images 0.2 * exp(-|grad I|^2 / 0.01): the distributions of
robartsvtk_gb300/synthetic.py, made on the GPU.  Trees are written as parent
lists ("-1 0 0": a root with two leaves), graphs as edge lists ("0>1 0>2").
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

FLAT3 = "-1 0 0 0"
FLAT4 = "-1 0 0 0 0"
TREE4 = "-1 0 1 1 0 4 4"                               # root -> 2 branches -> 2 leaves each
TREE5 = "-1 0 1 1 1 0 0"                               # a branch of three leaves beside two leaves
TREE8 = "-1 0 0 1 1 2 2 3 3 4 4 5 5 6 6"               # root -> 2 -> 4 -> 8
DAG4 = "0>1 1>2 1>3 0>4 4>5 4>6 4>3"                   # TREE4 with leaf 3 under both branches
TREES = (FLAT3, FLAT4, TREE4, TREE5, "-1 0 0", "-1 0 1 1 0", "-1 0 0 0 0 0 0", "-1 0 1 1 0 4 4 0 7 7", TREE8)
GRAPHS = (DAG4, "0>1 0>2 1>3 1>4 2>4 2>5", "0>1 0>2 0>3 1>4 2>4")
STEP, CC = 0.1, 0.25                                   # the reference's defaults


def listed():
    return [
        # a region of interest re-segmented while a user edits it: small, so latency and launches count
        dict(name="solve_roi", kind="solve", vx=40, vy=36, vz=28, tree=FLAT3, smooth="none", iterations=100,
             semantics="cuda"),
        # a brain-sized volume, odd in every axis, uneven tree, two smoothness images
        dict(name="solve_odd", kind="solve", vx=181, vy=217, vz=181, tree=TREE5, smooth="two", iterations=100,
             semantics="cuda"),
        # the two-level 4-leaf tree at 256^3 (the benchmark's volume) with the default iteration count
        dict(name="solve_tree4", kind="solve", vx=256, vy=256, vz=256, tree=TREE4, smooth="shared", iterations=100,
             semantics="cuda"),
        # the largest: a CT-like volume with a three-level 8-leaf tree
        dict(name="solve_large", kind="solve", vx=512, vy=512, vz=384, tree=TREE8, smooth="shared", iterations=20,
             semantics="cuda"),
        # the CPU class's semantics, for users who switch from it
        dict(name="solve_ref_cpu", kind="solve", vx=192, vy=160, vz=144, tree=FLAT4, smooth="none", iterations=200,
             semantics="cpu"),
        # a study: uneven volumes that share one tree, solved together
        dict(name="batch", kind="batch", count=20, lo=48, hi=192, tree=FLAT3, iterations=100),
        # a training step: loss and gradients of the data terms and smoothness weights, states checkpointed
        dict(name="adjoint_flat", kind="adjoint", vx=128, vy=128, vz=128, tree=FLAT4, smooth="none", iterations=300,
             every=30),
        # a training step on a patch with a hierarchical tree, every state kept
        dict(name="adjoint_tree", kind="adjoint", vx=96, vy=88, vz=72, tree=TREE4, smooth="shared", iterations=60,
             every=0),
        # labels on a directed acyclic graph
        dict(name="dag", kind="dag", vx=192, vy=180, vz=160, graph=DAG4, smooth="shared", iterations=60),
        # the filter facade on host images, inputs and outputs copied (a VTK pipeline's update)
        dict(name="filter_host", kind="filter", vx=128, vy=112, vz=96, tree=FLAT3, iterations=100),
        # the vote over a labelling and its energy
        dict(name="vote_energy", kind="post", vx=256, vy=256, vz=256, tree=TREE4, smooth="shared"),
        # data terms of four classes, and a log-likelihood from four raters' label maps
        dict(name="data_terms", kind="terms", vx=256, vy=256, vz=192, classes=4, maps=4),
    ]


def _sides(rng, lo, hi):
    base = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return [max(12, int(base * rng.uniform(0.75, 1.33))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["solve"] * 5 + ["batch", "adjoint", "dag", "filter", "post", "terms"])
    if kind == "batch":
        lo = rng.randint(24, 64)
        return dict(kind=kind, count=rng.randint(4, 20), lo=lo, hi=rng.randint(lo + 8, 176), tree=FLAT3,
                    iterations=rng.randint(20, 100))
    vx, vy, vz = _sides(rng, 20, {"solve": 330, "dag": 220, "filter": 140, "adjoint": 100, "post": 280,
                                  "terms": 280}[kind])
    c = dict(kind=kind, vx=vx, vy=vy, vz=vz)
    if kind == "terms":
        return dict(c, classes=rng.randint(2, 5), maps=rng.randint(2, 6))
    if kind == "dag":
        c["graph"] = rng.choice(GRAPHS)
        n = 1 + max(int(v) for v in c["graph"].replace(">", " ").split())
    else:
        c["tree"] = rng.choice(TREES[:8] if kind != "solve" else TREES)
        n = len(c["tree"].split())
    if kind != "filter":
        c["smooth"] = rng.choice(["none", "shared", "two"])
    if kind == "post":
        return c
    # at most a third of the largest listed case's voxel-vertex-iterations
    cap = 9.0e9 / (vx * vy * vz * (n - 1)) / (8 if kind == "adjoint" else 1)
    c["iterations"] = max(3, min(int(math.exp(rng.uniform(math.log(20), math.log(250)))), int(cap)))
    if kind == "solve":
        c["semantics"] = rng.choice(["cuda"] * 5 + ["cpu"])
        if c["semantics"] == "cuda" and rng.random() < 0.15:
            c["log"] = True  # the convergence log, read after the solve
    if kind == "adjoint":
        c["every"] = rng.choice([0, max(2, c["iterations"] // 10)])
    return c


# ---- the problems ----------------------------------------------------------

def _parent(case):
    return [int(p) for p in case["tree"].split()]


def _edges(case):
    return [tuple(int(v) for v in e.split(">")) for e in case["graph"].split()]


def _leaves_of(parent):
    """Leaves in depth-first pre-order."""
    out, stack = [], [parent.index(-1)]
    while stack:
        v = stack.pop()
        kids = [w for w, p in enumerate(parent) if p == v]
        if not kids:
            out.append(v)
        stack.extend(reversed(kids))
    return out


def _graph_leaves(edges):
    """Leaves of a graph by vertex id (every graph here numbers them so)."""
    n = 1 + max(max(e) for e in edges)
    return [v for v in range(n) if not any(p == v for p, _ in edges)]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _phantom(dims, classes, seed, sigma):
    """(class map, noisy image, class means) of painted ellipsoids."""
    vx, vy, vz = dims
    r = np.random.default_rng(int(seed) + 1)
    truth = torch.zeros((vz, vy, vx), dtype=torch.int32, device="cuda")
    z, y, x = (torch.arange(n, dtype=torch.float32, device="cuda") for n in (vz, vy, vx))
    for k in range(classes):
        c = r.uniform(0, 1, 3) * np.array([vx, vy, vz])
        rad = r.uniform(0.08, 0.32, 3) * min(vx, vy, vz) + 1.0
        inside = ((((x - c[0]) / rad[0]) ** 2)[None, None, :] + (((y - c[1]) / rad[1]) ** 2)[None, :, None]
                  + (((z - c[2]) / rad[2]) ** 2)[:, None, None]) <= 1.0
        truth[inside] = k
        del inside
    means = (np.arange(classes) + r.uniform(0.2, 0.8, classes)) / classes * 0.8 + 0.1
    img = torch.tensor(means, dtype=torch.float32, device="cuda")[truth.long()]
    img += sigma * torch.randn(img.shape, generator=_generator(seed), device="cuda")
    return truth, img, means


def _costs(img, means, sigma):
    return [(0.5 * ((img - float(m)) / sigma) ** 2).contiguous() for m in means]


def _edge_smoothness(img, scale):
    g2 = torch.zeros_like(img)
    for axis in range(3):
        g2 += torch.gradient(img, dim=axis)[0] ** 2
    return (scale * torch.exp(-g2 / 0.01)).contiguous()


def _smooth_images(case, img, vertices, leaves):
    if case.get("smooth", "none") == "none":
        return {}
    S = _edge_smoothness(img, 0.2)
    if case["smooth"] == "shared":
        return {v: S for v in vertices}
    S2 = _edge_smoothness(img, 0.1)
    return {v: (S if v in leaves else S2) for v in vertices}


def _alpha(case, vertices):
    """Smoothness weight per vertex: 1 with an image, as the benchmark's, else about 0.1."""
    return {v: 1.0 if case.get("smooth", "none") != "none" else 0.1 + 0.01 * (v % 3) for v in vertices}


def _problem(case, seed):
    dims = (case["vx"], case["vy"], case["vz"])
    if case["kind"] == "dag":
        edges = _edges(case)
        n, leaves = 1 + max(max(e) for e in edges), _graph_leaves(edges)
        root = next(v for v in range(n) if not any(c == v for _, c in edges))
    else:
        parent = _parent(case)
        n, leaves, root = len(parent), _leaves_of(parent), parent.index(-1)
    vertices = [v for v in range(n) if v != root]
    truth, img, means = _phantom(dims, len(leaves), seed, 0.08)
    return {"dims": dims, "leaves": leaves, "truth": truth, "img": img,
            "data": dict(zip(leaves, _costs(img, means, 0.08))),
            "smooth": _smooth_images(case, img, vertices, leaves), "alpha": _alpha(case, vertices)}


def _batch_dims(case, seed):
    # sizes belong to the case, not to the inputs: every seed has the same work
    r = np.random.default_rng(case["count"] * 100003 + case["lo"] * 1009 + case["hi"])
    return [tuple(int(v) for v in r.integers(case["lo"], case["hi"] + 1, 3)) for _ in range(case["count"])]


def _label_maps(truth, count, seed):
    """Raters' maps: the truth with 10 % of the voxels relabelled at random."""
    g = _generator(seed + 1)
    maps = []
    for _ in range(count):
        flip = torch.rand(truth.shape, generator=g, device="cuda") < 0.1
        other = torch.randint(0, 4, truth.shape, generator=g, device="cuda", dtype=torch.int32)
        maps.append(torch.where(flip, other, truth).contiguous())
    return maps


def _labelling(p, seed):
    """Leaf labels as a solve leaves them: near one-hot, in [0, 1], summing to 1."""
    logits = torch.stack([-0.25 * p["data"][v] for v in p["leaves"]])
    u = torch.softmax(logits, 0)
    return {v: u[j].contiguous() for j, v in enumerate(p["leaves"])}


def prepare(case, seed):
    import robartsvtk_gb300 as rv
    from robartsvtk_gb300.segmentation import DAGSolver, HMFBatchSolver

    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        dims, parent = _batch_dims(case, seed), _parent(case)
        s = HMFBatchSolver(dims, parent)
        outs = []
        for b, d in enumerate(dims):
            _, img, means = _phantom(d, len(s.leaves), seed * 64 + b, 0.08)
            for leaf, cost in zip(s.leaves, _costs(img, means, 0.08)):
                s.set_data(b, leaf, cost)
            outs.append([torch.empty((d[2], d[1], d[0]), device="cuda") for _ in s.leaves])
        for v in range(1, len(parent)):
            s.set_smoothness_scalar(v, 0.15)
        s.set_params(case["iterations"], STEP, CC)
        st.update(solver=s, outs=outs)
        return st
    if kind == "terms":
        dims = (case["vx"], case["vy"], case["vz"])
        truth, img, means = _phantom(dims, case["classes"], seed, 0.05)
        intensity = (img * 800.0).contiguous()  # scanner units for the histogram
        st.update(img=img, means=[float(m) for m in means], intensity=intensity,
                  maps=_label_maps(truth, case["maps"], seed))
        return st
    p = _problem(case, seed)
    shape = tuple(p["truth"].shape)
    if kind == "post":
        st.update(dims=p["dims"], parent=_parent(case), data=p["data"], smooth=p["smooth"] or None,
                  labels=_labelling(p, seed), leaves=p["leaves"])
        return st
    if kind == "filter":
        f = rv.HierarchicalMaxFlowSegmentation()
        f.SetStructure(_parent(case))
        for v, d in p["data"].items():
            f.SetDataInputDataObject(v, d.cpu().numpy())
        for v, a in p["alpha"].items():
            f.AddSmoothnessScalar(v, a)
        f.SetNumberOfIterations(case["iterations"])
        st.update(filter=f, leaves=p["leaves"])
        return st
    if kind == "dag":
        edges = _edges(case)
        s = DAGSolver(p["dims"], 1 + max(max(e) for e in edges), edges)
    else:
        semantics = rv.REF_CPU if case.get("semantics") == "cpu" else rv.REF_CUDA
        s = rv.HMFSolver(p["dims"], _parent(case), semantics)
    for v, a in p["alpha"].items():
        s.set_smoothness_scalar(v, a)
    for v, S in p["smooth"].items():
        s.set_smoothness(v, S)
    s.set_params(case["iterations"], STEP, CC)
    if kind == "adjoint":
        data = torch.stack([p["data"][v] for v in s.leaves]).requires_grad_(True)
        alpha = torch.tensor([p["alpha"].get(v, 0.0) for v in range(len(s.parent))], dtype=torch.float64,
                             requires_grad=True)
        rank = {v: j for j, v in enumerate(s.leaves)}
        truth = torch.tensor([rank[v] for v in p["leaves"]], dtype=torch.int32, device="cuda")[p["truth"].long()]
        st.update(solver=s, data=data, alpha=alpha, truth=truth.contiguous())
        return st
    for v, d in p["data"].items():
        s.set_data(v, d)
    if case.get("log"):
        s.set_convergence_log(True)
    st.update(solver=s, leaves=p["leaves"], outs=[torch.empty(shape, device="cuda") for _ in p["leaves"]])
    return st


def run(state):
    import robartsvtk_gb300 as rv

    case = state["case"]
    kind = case["kind"]
    stream = torch.cuda.current_stream()
    if kind in ("solve", "dag"):
        s = state["solver"]
        s.solve(stream)
        for leaf, out in zip(state["leaves"], state["outs"]):
            s.labels(leaf, out=out, stream=stream)
        if case.get("log"):
            c = s.convergence()
            return {"labels": state["outs"], "max": c["max"], "mean": c["mean"]}
        return {"labels": state["outs"]}
    if kind == "batch":
        s = state["solver"]
        s.solve(stream)
        for b, outs in enumerate(state["outs"]):
            for leaf, out in zip(s.leaves, outs):
                s.labels(b, leaf, out=out, stream=stream)
        return {"labels": state["outs"]}
    if kind == "adjoint":
        from robartsvtk_gb300.autograd import hmf_loss

        state["data"].grad = state["alpha"].grad = None
        loss = hmf_loss(state["solver"], state["data"], state["alpha"], state["truth"],
                        checkpoint_every=case["every"])
        loss.backward()
        return {"loss": loss, "d_data": state["data"].grad, "d_alpha": state["alpha"].grad}
    if kind == "filter":
        f = state["filter"]
        if f.Update() != 1:
            raise RuntimeError(f.GetLastError())
        return {"labels": [f.GetOutputDataObject(v) for v in state["leaves"]]}
    if kind == "post":
        votes = rv.vote([state["labels"][v] for v in state["leaves"]], values=state["leaves"], stream=stream)
        f0, f = rv.decomposition_energy(state["dims"], state["parent"], state["data"], state["labels"],
                                        state["smooth"], stream=stream)
        return {"votes": votes, "f0": f0, "f": f}
    from robartsvtk_gb300 import dataterm as dt

    terms = [dt.data_term(dt.GAUSSIAN, state["img"], k1=0.05, c1=m, entropy=True, normalize=True, stream=stream)
             for m in state["means"]]
    member = dt.data_term(dt.LOGISTIC, state["img"], k1=12.0, c1=state["means"][-1], entropy=True, stream=stream)
    like = dt.log_likelihood(state["intensity"], state["maps"], label_id=1, resolution=1.0, required_agreement=0.7,
                             stream=stream)
    return {"terms": terms, "member": member, "likelihood": like}


def work(case):
    """Bytes and operations of one pass.  An iteration of a solve updates the
    whole state: each vertex's three flows, sink and label and its parent's
    view of them read and written once, each data term and distinct
    smoothness image read once, 4 V (12 N + L + S + 2) bytes (the divergence
    included); a volume whose state stays on chip can go below that."""
    kind = case["kind"]
    if kind == "batch":
        vox = float(sum(a * b * c for a, b, c in _batch_dims(case, 0)))
    else:
        vox = float(case["vx"] * case["vy"] * case["vz"])
    if kind == "terms":
        k, m = case["classes"], case["maps"]
        return {"bytes": 4.0 * vox * ((k + 1) * 2 + 2 + m), "flops": vox * (8.0 * k + 40.0 + 2.0 * m)}
    if kind == "dag":
        edges = _edges(case)
        n, leaves = max(max(e) for e in edges), len(_graph_leaves(edges))
    else:
        parent = _parent(case)
        n, leaves = len(parent) - 1, len(_leaves_of(parent))
    images = {"none": 0, "shared": 1, "two": 2}[case.get("smooth", "none")]
    if kind == "post":
        return {"bytes": 4.0 * vox * (leaves + 1) + 4.0 * vox * (2 * leaves + images),
                "flops": vox * (2.0 * leaves + 14.0 * n)}
    its = case["iterations"]
    ends = 4.0 * vox * 2 * leaves + (4.0 * vox * 2 * leaves if kind == "filter" else 0.0)
    if case.get("semantics") == "cpu":  # a voxel's iterations need nothing but its own leaf values
        return {"bytes": ends, "flops": 6.0 * vox * leaves * its}
    arrays = 12 * n + leaves + images + 2 + (2 * n if kind == "dag" else 0)
    step_bytes, step_flops = 4.0 * vox * arrays, vox * (64.0 * n)
    if kind == "adjoint":  # per reverse step: the state read, its adjoint read and written, gradients accumulated
        back = 4.0 * vox * (5 * n + 1 + 2 * (5 * n + 1) + 4 * leaves + images)
        return {"bytes": its * (step_bytes + back) + ends, "flops": its * step_flops * 3.0}
    return {"bytes": its * step_bytes + ends, "flops": its * step_flops}


# ---- double precision, plain torch -------------------------------------------

def _low(a, axis):
    """a at the lower neighbour along `axis`, zero on the low face."""
    pad = [0, 0, 0, 0, 0, 0]
    pad[2 * (2 - axis)] = 1
    return F.pad(a.narrow(axis, 0, a.shape[axis] - 1), pad)


def _high(a, axis):
    """a at the upper neighbour along `axis`, zero on the high face."""
    pad = [0, 0, 0, 0, 0, 0]
    pad[2 * (2 - axis) + 1] = 1
    return F.pad(a.narrow(axis, 1, a.shape[axis] - 1), pad)


def _not_low_face(a, axis):
    pad = [0, 0, 0, 0, 0, 0]
    pad[2 * (2 - axis)] = 1
    return F.pad(a.narrow(axis, 1, a.shape[axis] - 1), pad)


def _flow_step(p, div, sink, inc, label, limit, step, icc):
    """One vertex: new flows (x, y, z order of axes 2, 1, 0) and divergence."""
    g = step * (((sink + div) - inc) - label * icc)
    q = {a: _not_low_face(p[a] - (g - _low(g, a)), a) for a in p}
    h = None
    for a in q:
        t = q[a] * q[a] + _high(q[a] * q[a], a)
        h = t if h is None else h + t
    h = 0.5 * h
    over = h > limit * limit
    m = torch.where(over, limit / torch.sqrt(torch.where(over, h, torch.ones_like(h))), torch.ones_like(h))
    new = {a: q[a] * 0.5 * (m + _low(m, a)) for a in q}
    d = None
    for a in new:
        t = new[a] - _high(new[a], a)
        d = t if d is None else d + t
    return new, d


def _saturate(u):
    return torch.where(u <= 0, torch.zeros_like(u), torch.where(u >= 1, torch.ones_like(u), u))


def _capacity(v, cap):
    v = torch.where(v < 0, torch.zeros_like(v), v)
    return torch.where(v > cap, cap, v)


def _tree_init(parent, leaves, data):
    order = _post_order(parent)
    m = torch.stack([data[v] for v in leaves]).min(0).values
    hit = {v: (data[v] == m).to(m.dtype) for v in leaves}
    total = sum(hit.values())
    u = {}
    for v in order:
        if v in hit:
            u[v] = hit[v] / total
        elif parent[v] >= 0:
            u[v] = sum(u[w] for w, q in enumerate(parent) if q == v)
    sink = {v: m for v in range(len(parent))}
    zero = torch.zeros_like(m)
    return {"u": u, "s": sink, "p": {v: {2: zero, 1: zero, 0: zero} for v in u}, "d": {v: zero for v in u}}


def _post_order(parent):
    out = []

    def visit(v):
        for w, q in enumerate(parent):
            if q == v:
                visit(w)
        out.append(v)

    visit(parent.index(-1))
    return out


def _f32(x):
    return float(np.float32(x))


def _tree_iteration(st, parent, data, limit, step, cc):
    icc = 1.0 / cc
    root = parent.index(-1)
    p, d = {}, {}
    for v in st["u"]:
        p[v], d[v] = _flow_step(st["p"][v], st["d"][v], st["s"][v], st["s"][parent[v]], st["u"][v], limit[v], step, icc)
        st["p"][v] = None  # the old flows are read by their own vertex only
    s = dict(st["s"])
    u = st["u"]
    for v in _post_order(parent):
        kids = [w for w, q in enumerate(parent) if q == v]
        if not kids:
            s[v] = _capacity(s[parent[v]] - d[v] + u[v] * icc, data[v])
            continue
        w = sum(s[k] + d[k] - u[k] * icc for k in kids)
        s[v] = (icc + w) / len(kids) if v == root else (w + s[parent[v]] - d[v] + u[v] * icc) / (len(kids) + 1)
    new = {v: _saturate(u[v] + cc * (s[parent[v]] - d[v] - s[v])) for v in u}
    return {"u": new, "s": s, "p": p, "d": d}


def _limits(p):
    vertices = p["alpha"]
    return {v: _f32(a) * p["smooth"][v].double() if v in p["smooth"]
            else torch.tensor(_f32(a), dtype=torch.float64, device="cuda") for v, a in vertices.items()}


def _exact_tree(case, p, parent, iterations):
    data = {v: d.double() for v, d in p["data"].items()}
    limit = _limits(p)
    st = _tree_init(parent, p["leaves"], data)
    change = {"max": [], "mean": []}
    for _ in range(iterations):
        old = st["u"]
        st = _tree_iteration(st, parent, data, limit, _f32(STEP), _f32(CC))
        if case.get("log"):
            diff = [(st["u"][v] - old[v]).abs() for v in old]
            change["max"].append(max(float(t.max()) for t in diff))
            change["mean"].append(float(sum(t.sum() for t in diff)) / (len(diff) * diff[0].numel()))
    return st, change


def _exact_ref_cpu(case, p):
    data = {v: d.double() for v, d in p["data"].items()}
    st = _tree_init(_parent(case), p["leaves"], data)
    m, out = st["s"][0], []
    for v in p["leaves"]:
        u = st["u"][v]
        for _ in range(case["iterations"]):
            s = m + u / _f32(CC)
            s = torch.where(s > data[v], data[v], s)
            u = u + _f32(CC) * (m - s)
        out.append(u)
    return {"labels": out}


def _exact_dag(case, p):
    edges = _edges(case)
    n = 1 + max(max(e) for e in edges)
    step, cc = _f32(STEP), _f32(CC)
    icc = 1.0 / cc
    parents = {v: [a for a, b in edges if b == v] for v in range(n)}
    kids = {v: [b for a, b in edges if a == v] for v in range(n)}
    root = next(v for v in range(n) if not parents[v])
    order, todo = [], {v: len(parents[v]) for v in range(n)}
    ready = [root]
    while ready:
        v = ready.pop(0)
        order.append(v)
        for k in kids[v]:
            todo[k] -= 1
            if not todo[k]:
                ready.append(k)
    share = {v: 1.0 / max(1, len(parents[v])) for v in range(n)}
    weight = {v: sum(share[k] ** 2 for k in kids[v]) for v in range(n)}
    data = {v: d.double() for v, d in p["data"].items()}
    limit = _limits(p)
    m = torch.stack([data[v] for v in p["leaves"]]).min(0).values
    hit = {v: (data[v] == m).to(m.dtype) for v in p["leaves"]}
    total = sum(hit.values())
    u = {}
    for v in reversed(order):
        if v in hit:
            u[v] = hit[v] / total
        elif v != root:
            u[v] = sum(share[k] * u[k] for k in kids[v])
    s = {v: m for v in range(n)}
    inc = {v: m for v in u}
    zero = torch.zeros_like(m)
    flow = {v: {2: zero, 1: zero, 0: zero} for v in u}
    div = {v: zero for v in u}
    its = case["iterations"]
    for it in range(its):
        for v in u:
            flow[v], div[v] = _flow_step(flow[v], div[v], s[v], inc[v], u[v], limit[v], step, icc)
        s[root] = s[root] + 1.0 / (cc * weight[root])
        for v in order:
            if v in hit:
                s[v] = _capacity(inc[v] - div[v] + u[v] * icc, data[v])
                u[v] = _saturate(u[v] + cc * (inc[v] - div[v] - s[v]))
            elif v != root:
                k = 1.0 / (weight[v] + 1.0)
                s[v] = (1.0 - k) * s[v] + k * (inc[v] - div[v] + u[v] * icc)
        if it == its - 1:
            break
        for v in reversed(order):
            if v == root:
                continue
            push = s[v] - inc[v] + div[v] - u[v] * icc
            for q in parents[v]:
                s[q] = s[q] + share[v] / (weight[q] if q == root else weight[q] + 1.0) * push
            if v not in hit:
                u[v] = _saturate(u[v] + cc * (inc[v] - div[v] - s[v]))
        for v in u:
            inc[v] = sum(share[v] * s[q] for q in parents[v])
    return {"labels": [u[v] for v in p["leaves"]]}


def _exact_adjoint(case, p):
    """Reverse mode by hand over stored states: torch differentiates one iteration at a time."""
    parent, its = _parent(case), case["iterations"]
    leaves = p["leaves"]
    step, cc = _f32(STEP), _f32(CC)
    data = {v: p["data"][v].double().requires_grad_(True) for v in leaves}
    alpha = {v: torch.tensor(_f32(a), dtype=torch.float64, device="cuda", requires_grad=True)
             for v, a in p["alpha"].items()}
    vertices = list(alpha)

    def flat(st):
        return ([st["u"][v] for v in vertices] + [st["s"][v] for v in range(len(parent))]
                + [st["d"][v] for v in vertices] + [st["p"][v][a] for v in vertices for a in (2, 1, 0)])

    def nest(x):
        k, n = len(vertices), len(parent)
        return {"u": dict(zip(vertices, x[:k])), "s": dict(enumerate(x[k:k + n])),
                "d": dict(zip(vertices, x[k + n:2 * k + n])),
                "p": {v: dict(zip((2, 1, 0), x[2 * k + n + 3 * j:2 * k + n + 3 * j + 3])) for j, v in enumerate(vertices)}}

    def advance(x, dat, al):
        limit = {v: al[v] * p["smooth"][v].double() if v in p["smooth"] else al[v] for v in vertices}
        return flat(_tree_iteration(nest(x), parent, dat, limit, step, cc))

    keep = 20
    with torch.no_grad():
        x = flat(_tree_init(parent, leaves, data))
        saved = {0: x}
        for t in range(its):
            x = advance(x, data, alpha)
            if (t + 1) % keep == 0:
                saved[t + 1] = x
    truth = p["truth"].long()
    final = [y.detach().requires_grad_(True) for y in x]
    lab = torch.stack([nest(final)["u"][v] for v in leaves])
    picked = lab.gather(0, truth[None])[0]
    loss = -torch.log(torch.where(picked > 1e-6, picked, torch.full_like(picked, 1e-6))).sum() / picked.numel()
    bar = torch.autograd.grad(loss, final, allow_unused=True)
    bar = [torch.zeros_like(y) if b is None else b for b, y in zip(bar, final)]
    dd = {v: torch.zeros_like(data[v]) for v in leaves}
    da = {v: 0.0 for v in vertices}
    wrt = [data[v] for v in leaves] + [alpha[v] for v in vertices]

    def collect(grads):
        for v, g in zip(leaves, grads):
            if g is not None:
                dd[v] += g
        for v, g in zip(vertices, grads[len(leaves):]):
            if g is not None:
                da[v] += float(g)

    for first in range((its - 1) // keep * keep if its else 0, -1, -keep):
        with torch.no_grad():
            states = [saved[first]]
            for t in range(first, min(first + keep, its) - 1):
                states.append(advance(states[-1], data, alpha))
        while states:
            here = [y.detach().requires_grad_(True) for y in states.pop()]
            nxt = advance(here, data, alpha)
            pairs = [(y, b) for y, b in zip(nxt, bar) if y.requires_grad]
            g = torch.autograd.grad([y for y, _ in pairs], here + wrt, [b for _, b in pairs], allow_unused=True)
            bar = [torch.zeros_like(y) if b is None else b for b, y in zip(g, here)]
            collect(g[len(here):])
    start = flat(_tree_init(parent, leaves, data))
    pairs = [(y, b) for y, b in zip(start, bar) if y.requires_grad]
    collect(torch.autograd.grad([y for y, _ in pairs], wrt, [b for _, b in pairs], allow_unused=True))
    return {"loss": loss.detach(), "d_data": torch.stack([dd[v] for v in leaves]),
            "d_alpha": torch.tensor([da.get(v, 0.0) for v in range(len(parent))], dtype=torch.float64)}


def _exact_post(case, p, seed):
    parent, leaves = _parent(case), p["leaves"]
    lab = {v: t.double() for v, t in _labelling(p, seed).items()}
    f0 = float(sum((p["data"][v].double() * lab[v]).sum() for v in leaves))
    f = np.zeros(len(parent))
    for v in _post_order(parent):
        if parent[v] < 0:
            continue
        if v not in lab:
            lab[v] = sum(lab[w] for w, q in enumerate(parent) if q == v)
        g2 = 0.0
        for a in range(3):
            n = lab[v].shape[a]
            up = torch.cat([lab[v].narrow(a, 1, n - 1), lab[v].narrow(a, n - 1, 1)], a)
            dn = torch.cat([lab[v].narrow(a, 0, 1), lab[v].narrow(a, 0, n - 1)], a)
            g2 = g2 + (up - dn) ** 2
        term = 0.5 * torch.sqrt(g2)
        if v in p["smooth"]:
            term = p["smooth"][v].double() * term
        f[v] = float(term.sum())
    return {"votes": None, "f0": f0, "f": f}


def _exact_terms(case, seed):
    dims = (case["vx"], case["vy"], case["vz"])
    truth, img, means = _phantom(dims, case["classes"], seed, 0.05)
    maps = _label_maps(truth, case["maps"], seed)
    x = img.double()
    lo, hi = float(x.min()), float(x.max())
    terms = []
    for m in (float(v) for v in means):
        e = 0.5 * ((x - m) / 0.05) ** 2
        ends = [0.5 * ((r - m) / 0.05) ** 2 for r in (lo, hi)]
        least = 0.0 if lo < m < hi else min(ends)
        terms.append((e - least) / (max(ends) - least))
    member = torch.log1p(torch.exp(-12.0 * (x - float(means[-1]))))
    # the bin of a voxel is part of the definition (float32 arithmetic); its cost is in double
    intensity = img * 800.0
    agree = sum((k == 1).to(torch.int32) for k in maps)
    seeds = agree.double() >= 0.7 * case["maps"]
    if not bool(seeds.any()):
        return {"terms": terms, "member": member, "likelihood": torch.ones_like(x)}
    first, last = intensity[seeds].min(), intensity[seeds].max()
    bins = int(last - first) + 1
    size = int(torch.clamp(last, min=0.0) - first) + 1
    at = (intensity - first).to(torch.int64)
    hist = torch.bincount(at[seeds], minlength=max(bins, size)).double()
    cost = -torch.log(hist / float(seeds.sum()) + 1e-10)
    outside = (intensity < first) | (at >= size)
    like = torch.where(outside, torch.full_like(x, -math.log(1e-10)), cost[torch.where(outside, 0, at)])
    return {"terms": terms, "member": member, "likelihood": like}


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "terms":
            return _exact_terms(case, seed)
        if kind == "batch":
            parent, out = _parent(case), []
            for b, d in enumerate(_batch_dims(case, seed)):
                leaves = _leaves_of(parent)
                _, img, means = _phantom(d, len(leaves), seed * 64 + b, 0.08)
                p = {"leaves": leaves, "data": dict(zip(leaves, _costs(img, means, 0.08))), "smooth": {},
                     "alpha": {v: 0.15 for v in range(1, len(parent))}}
                st, _ = _exact_tree(case, p, parent, case["iterations"])
                out.append([st["u"][v] for v in leaves])
            return {"labels": out}
        p = _problem(case, seed)
        if kind == "post":
            return _exact_post(case, p, seed)
        if kind == "dag":
            return _exact_dag(case, p)
        if case.get("semantics") == "cpu":
            return _exact_ref_cpu(case, p)
        if kind != "adjoint":
            st, change = _exact_tree(case, p, _parent(case), case["iterations"])
            out = {"labels": [st["u"][v] for v in p["leaves"]]}
            return dict(out, **{k: np.array(v) for k, v in change.items()}) if case.get("log") else out
    return _exact_adjoint(case, p)
