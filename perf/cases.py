"""The workloads this library is timed on: what its users call, over the sizes they call it with.

listed() names them, draw() makes more of the same kinds, prepare() builds what a program holds
before the call (the resident tree, the queries, the parameters), run() is one call through the
public entry points (`sbh_capi`, `sbh_torch`), work() the bytes and operations one call cannot
do without, and exact() the answer in 64 bits where the method is exact summation.

Kinds of case ("what"):
  eval    one evaluation: brute force, Barnes-Hut, warp-vote Barnes-Hut or stochastic Barnes-Hut
          of gravity, winding number, smooth distance or Plummer; on device buffers
          (`GpuTree.eval_device`) or host arrays (`GpuTree.eval`, blocking, with counts)
  grad    values and query gradients forward and backward through `sbh_torch.evaluate`
  batch   many problems evaluated at their own points in one `eval_batch`, own terms excluded
  serve   a stream of requests on resident trees through `Server.submit` / `Request.wait`
  build   a tree from new host points (`GpuTree.build`) and one evaluation on it
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "stochastic-barnes-hut_b200"))

import sbh_capi as C  # noqa: E402
import sbh_torch  # noqa: E402
import sbh_workloads as W  # noqa: E402

KERNELS = {"gravity": C.GRAVITY, "wn": C.WINDING_NUMBER, "smooth": C.SMOOTH_DIST,
           "plummer": C.PLUMMER}
METHODS = {"brute_force": C.BRUTE_FORCE, "barnes_hut": C.BARNES_HUT,
           "barnes_hut_vote": C.BARNES_HUT_VOTE, "stochastic": C.STOCHASTIC}
ALPHA = 100.0  # smooth distance, as the serving and differentiation workloads use it
EPS = 1e-3     # Plummer softening


def listed():
    return [
        # A probe of the field at a few positions: the smallest call, all latency and launches.
        dict(name="bh_gravity_64q", what="eval", method="barnes_hut", kernel="gravity", dim=3,
             source="gauss", n=10000, nq=64, dsl=1, leaf=1, beta=2.0, host=False),
        # An ordinary request of the sampler from a host program, counts read as well.
        dict(name="sbh_gravity_host_1500q", what="eval", method="stochastic", kernel="gravity",
             dim=3, source="gauss", n=100000, nq=1500, dsl=2, leaf=1, budget=256, host=True),
        # An ordinary distance request on a large scan: the serving workload's exact summation.
        dict(name="bf_smooth_997q", what="eval", method="brute_force", kernel="smooth", dim=3,
             source="sphere", n=1000003, nq=997, dsl=1, leaf=1, host=False),
        # The plain method's small workload: all pairs, and Barnes-Hut with 8 points a leaf.
        dict(name="bf_plummer_65k", what="eval", method="brute_force", kernel="plummer", dim=3,
             source="gauss", n=65536, nq=65536, dsl=1, leaf=8, host=False),
        dict(name="bh_plummer_leaf8_65k", what="eval", method="barnes_hut", kernel="plummer",
             dim=3, source="gauss", n=65536, nq=65536, dsl=1, leaf=8, beta=2.0, host=False),
        # Inside/outside of a surface on a dense grid of positions: the largest calls.
        dict(name="bh_wn_4m", what="eval", method="barnes_hut", kernel="wn", dim=3, source="torus",
             n=1 << 20, nq=1 << 22, dsl=1, leaf=1, beta=2.0, host=False),
        dict(name="sbh_wn_4m", what="eval", method="stochastic", kernel="wn", dim=3,
             source="torus", n=1 << 20, nq=1 << 22, dsl=2, leaf=1, budget=256, host=False),
        # Fitting positions to a surface: exact gradients of a modest set ...
        dict(name="grad_bf_smooth_4001q", what="grad", method="brute_force", kernel="smooth", dim=2,
             source="circle", n=262144, nq=4001, dsl=1, leaf=1),
        # ... and stochastic gradients of a million positions (training-sized forward + backward).
        dict(name="grad_sbh_smooth_1m", what="grad", method="stochastic", kernel="smooth", dim=3,
             source="torus", n=524288, nq=1 << 20, dsl=2, leaf=1, budget=128),
        # Potentials of many particle systems at their own particles in one call.
        dict(name="batch_gravity_32", what="batch", problems=32, n_lo=1024, n_hi=1 << 17, budget=128),
        # Requests of mixed sizes and kernels arriving at a server with resident trees.
        dict(name="serve_48", what="serve", trees=6, requests=48, n_lo=10000, n_hi=500000,
             nq_hi=100000),
        # A moving point set: the tree is built again for every step, then evaluated.
        dict(name="build_1m", what="build", kernel="wn", dim=3, source="torus", n=1 << 20, nq=65536,
             dsl=2, leaf=1, beta=2.0),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.999))))


# What drawn cases may ask for: pairs of an all-pairs case, positions of a walk, sampled paths.
MAX_PAIRS, MAX_WALKS, MAX_PATHS = 1 << 31, 1 << 19, 1 << 25


def draw(rng):
    what = rng.choice(["eval", "eval", "eval", "eval", "grad", "grad", "batch", "serve", "build"])
    if what == "batch":
        return dict(what=what, problems=rng.randint(2, 40), n_lo=1024, n_hi=_log(rng, 8192, 1 << 17),
                    budget=rng.choice([64, 128, 256]))
    if what == "serve":
        return dict(what=what, trees=rng.randint(2, 6), requests=rng.randint(4, 56), n_lo=10000,
                    n_hi=_log(rng, 20000, 500000), nq_hi=_log(rng, 100, 100000))
    dim = rng.choice([2, 3])
    c = dict(what=what, dim=dim, dsl=rng.choice([1, 1, 2, 2, 3]),
             source=rng.choice(["gauss", "circle"] if dim == 2 else ["gauss", "torus", "sphere"]))
    if what == "build":
        return dict(c, kernel=rng.choice(list(KERNELS)), n=_log(rng, 1000, 1 << 20),
                    nq=_log(rng, 32, 65536), leaf=1, beta=2.0)
    method = rng.choice(["brute_force", "barnes_hut", "stochastic", "barnes_hut_vote"]
                        if what == "eval" else ["brute_force", "barnes_hut", "stochastic"])
    kernel = rng.choice(list(KERNELS) if what == "eval" else ["gravity", "smooth", "plummer"])
    n = _log(rng, 1000, 2000000)
    leaf = rng.choice([1, 1, 1, 8]) if n <= 200000 else 1
    c.update(method=method, kernel=kernel, n=n, leaf=leaf)
    if method == "brute_force":
        cap = MAX_PAIRS if what == "eval" else MAX_PAIRS // 4
        c["nq"] = _log(rng, 1, max(2, min(65536, cap // n)))
    elif method == "stochastic":
        c["budget"] = rng.choice([64, 128, 256])
        c["dsl"] = rng.choice([1, 2])
        c["nq"] = _log(rng, 1, MAX_PATHS // c["budget"])
    else:
        c["beta"] = rng.choice([1.25, 2.0, 2.0, 3.0])
        c["nq"] = _log(rng, 1, MAX_WALKS)
    if what == "eval":
        c["host"] = rng.random() < 0.4
    return c


# ---- inputs ---------------------------------------------------------------------------------

def _points(source, n, dim, seed):
    if source == "gauss":
        return W.gaussian_mixture(n, seed, dim=dim)
    return {"torus": W.torus_surface, "sphere": W.sphere_surface,
            "circle": W.circle_points}[source](n, seed)


def _tree(pts, nrm, m, dsl, leaf):
    lo, hi = W.padded_box(pts)
    return C.GpuTree.build(pts, nrm, m, lo, hi, alpha=ALPHA, dim_split_log=dsl, leaf_size=leaf)


def _queries(case, seed, lo, hi):
    """(dim, nq) float32 positions on the host, uniform in the sources' surroundings."""
    rng = np.random.default_rng([seed, 1])
    pad = 0.25 * float(np.max(hi - lo))
    q = rng.random((case["dim"], case["nq"]), dtype=np.float32)
    return ((lo - pad)[:, None] + q * (hi - lo + 2 * pad)[:, None]).astype(np.float32)


def _params(case, tree, seed):
    samples = W.samples_for_budget(case.get("budget", 1), tree.info.root_children)
    return C.params(method=METHODS[case["method"]], kernel=KERNELS[case["kernel"]],
                    beta=case.get("beta", 2.0), samples_per_subdomain=samples, seed=seed % 1000,
                    eps=EPS)


def _batch_problems(case, seed):
    """Sizes log-spaced from n_lo to n_hi in a mixed order; the points are the seed's."""
    k = case["problems"]
    sizes = [int(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** ((i + 0.5) / k)) for i in range(k)]
    order = np.random.default_rng([k, 2]).permutation(k)
    return [dict(n=sizes[i], seed=seed * 1000 + int(i)) for i in order]


# The operating points of the serving workload: median relative error of 1e-3 or better.
SERVED = {"gravity": ("barnes_hut", 2.0), "wn": ("barnes_hut", 5.0), "smooth": ("brute_force", 2.0)}


def _serve_plan(case, seed):
    """The resident trees' (source, n, dim, seed) and the requests' (tree, kernel, positions, seed):
    sizes log-spaced over their ranges, the same for every seed; contents are the seed's."""
    rng = np.random.default_rng([case["requests"], 3])
    trees, reqs = [], []
    for i in range(case["trees"]):
        dim = 3 if i % 2 == 0 else 2
        source = ("gauss", "torus", "sphere")[i % 3] if dim == 3 else ("gauss", "circle")[i // 2 % 2]
        f = (i + 0.5) / case["trees"]
        trees.append((source, int(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** f), dim, seed + i))
    for r in range(case["requests"]):
        f = (r + 0.5) / case["requests"]
        t = int(rng.integers(case["trees"]))
        reqs.append((t, tuple(SERVED)[r % 3], max(1, int(case["nq_hi"] ** f)), seed * 1000 + r))
    order = rng.permutation(len(reqs))
    return trees, [reqs[i] for i in order]


def prepare(case, seed):
    what = case["what"]
    if what == "batch":
        problems, keep = [], []
        for b in _batch_problems(case, seed):
            pts, nrm, m = W.gaussian_mixture(b["n"], b["seed"])
            tree = _tree(pts, nrm, m, 2, 1)
            q = torch.from_numpy(np.ascontiguousarray(pts.T)).cuda()
            mass, out = torch.from_numpy(m).cuda(), torch.empty(b["n"], device="cuda")
            p = C.params(method=C.STOCHASTIC, kernel=C.GRAVITY, seed=b["seed"] % 1000,
                         samples_per_subdomain=W.samples_for_budget(case["budget"],
                                                                    tree.info.root_children))
            problems.append((tree, p, q.data_ptr(), b["n"], out.data_ptr(), 0, mass.data_ptr()))
            keep.append((q, mass, out))
        return dict(what=what, problems=problems, keep=keep)
    if what == "serve":
        trees, reqs = _serve_plan(case, seed)
        server = C.Server(slots=3, slot_queries=1 << 20)
        boxes, ids = [], []
        for source, n, dim, s in trees:
            pts, nrm, m = _points(source, n, dim, s)
            boxes.append(W.padded_box(pts))
            ids.append(server.add_tree(_tree(pts, nrm, m, 1, 1)))
        stream = []
        for t, kernel, nq, s in reqs:
            lo, hi = boxes[t]
            q = np.random.default_rng(s).uniform(lo, hi, (nq, len(lo))).astype(np.float32)
            method, beta = SERVED[kernel]
            p = C.params(method=METHODS[method], kernel=KERNELS[kernel], beta=beta)
            stream.append((ids[t], np.asfortranarray(q), p))
        return dict(what=what, server=server, stream=stream)
    pts, nrm, m = _points(case["source"], case["n"], case["dim"], seed)
    lo, hi = W.padded_box(pts)
    q = _queries(case, seed, lo, hi)
    if what == "build":
        p = C.params(method=C.BARNES_HUT, kernel=KERNELS[case["kernel"]], beta=case["beta"], eps=EPS)
        return dict(what=what, pts=pts, nrm=nrm, m=m, lo=lo, hi=hi, q=q.T, p=p, dsl=case["dsl"],
                    leaf=case["leaf"])
    tree = _tree(pts, nrm, m, case["dsl"], case["leaf"])
    if what == "grad":
        x = torch.from_numpy(np.ascontiguousarray(q.T)).cuda().requires_grad_(True)
        samples = W.samples_for_budget(case.get("budget", 1), tree.info.root_children)
        return dict(what=what, tree=tree, x=x, gout=torch.ones(case["nq"], device="cuda"),
                    kw=dict(kernel=case["kernel"], method=case["method"], beta=case.get("beta", 2.0),
                            samples_per_subdomain=samples, seed=seed % 1000, eps=EPS))
    p = _params(case, tree, seed)
    if case["host"]:
        return dict(what="host", tree=tree, q=q.T, p=p)
    return dict(what="device", tree=tree, q=torch.from_numpy(q).cuda(), p=p,
                out=torch.empty(case["nq"], device="cuda"))


# ---- one call -------------------------------------------------------------------------------

def run(s):
    what = s["what"]
    if what == "device":
        s["tree"].eval_device(s["q"].data_ptr(), s["q"].shape[1], s["out"].data_ptr(), s["p"],
                              stream=torch.cuda.current_stream().cuda_stream)
        return s["out"]
    if what == "host":
        values, _, counts = s["tree"].eval(s["q"], s["p"], contribs=True)
        return values, counts
    if what == "grad":
        s["x"].grad = None
        d = sbh_torch.evaluate(s["tree"], s["x"], **s["kw"])
        d.backward(s["gout"])
        return d.detach(), s["x"].grad
    if what == "batch":
        C.eval_batch(s["problems"], stream=torch.cuda.current_stream().cuda_stream)
        return [out for _, _, out in s["keep"]]
    if what == "serve":
        pending = [s["server"].submit(t, q, p) for t, q, p in s["stream"]]
        return [r.wait() for r in pending]
    tree = C.GpuTree.build(s["pts"], s["nrm"], s["m"], s["lo"], s["hi"], alpha=ALPHA,
                           dim_split_log=s["dsl"], leaf_size=s["leaf"])
    values, _ = tree.eval(s["q"], s["p"])
    return values, tree.info.num_nodes, tree.info.depth


# ---- what a call cannot do without ----------------------------------------------------------

# Floating-point operations of one term of each kernel (3D; roots, reciprocals and exponentials
# counted as one), and about how many terms a query's walk adds for each level of its tree.
TERM_FLOPS = {"gravity": 12, "wn": 18, "smooth": 11, "plummer": 11}


def _terms(method, n, beta=2.0, budget=0):
    if method == "brute_force":
        return n
    levels = max(1.0, math.log2(n) / 3)
    if method == "stochastic":
        return min(n, 1024) + 4 * budget
    return min(n, 8 * beta * beta * levels)


def work(case):
    what = case["what"]
    if what == "batch":
        mean = (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])
        n = case["problems"] * mean
        return dict(bytes=n * (32 + 12 + 4 + 4),
                    flops=n * _terms("stochastic", mean, budget=case["budget"]) * TERM_FLOPS["gravity"])
    if what == "serve":
        trees, reqs = _serve_plan(case, 0)
        nbytes = sum(32 * n for _, n, _, _ in trees)
        flops = 0.0
        for t, kernel, nq, _ in reqs:
            method, beta = SERVED[kernel]
            nbytes += 16 * nq
            flops += nq * _terms(method, trees[t][1], beta) * TERM_FLOPS[kernel]
        return dict(bytes=nbytes, flops=flops)
    n, nq, dim = case["n"], case["nq"], case["dim"]
    point = 4 * (dim + 1 + (dim if case["kernel"] == "wn" else 0))
    if what == "build":
        # the host arrays once in, the device image (points, codes, nodes) once out
        nodes = 1.4 * n
        nbytes = n * 4 * (2 * dim + 1) + n * (32 + 8) + nodes * (80 + 8 * max(1, 2 ** (dim * case["dsl"]) // 64))
        return dict(bytes=nbytes + nq * 4 * (dim + 1),
                    flops=nq * _terms("barnes_hut", n, case["beta"]) * TERM_FLOPS[case["kernel"]])
    terms = _terms(case["method"], n, case.get("beta", 2.0), case.get("budget", 0))
    flops = nq * terms * TERM_FLOPS[case["kernel"]]
    nbytes = n * point + nq * 4 * (dim + 1)
    if what == "grad":
        return dict(bytes=nbytes + nq * 4 * (2 * dim + 1), flops=2 * flops)
    return dict(bytes=nbytes, flops=flops)


# ---- 64-bit answers of exact summation --------------------------------------------------------

def _sum64(kernel, pts, nrm, m, q, grad=False):
    """Sums over all sources in float64 (dim, nq) -> values, or (values, gradients)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    pts, nrm, m, q = (torch.from_numpy(np.ascontiguousarray(a)).to(dev).double()
                      for a in (pts, nrm, m, q.T))
    n, dim = pts.shape
    values, grads = [], []
    for c in q.split(max(1, (1 << 25) // n)):
        d = [pts[None, :, k] - c[:, k, None] for k in range(dim)]
        r2 = sum(x * x for x in d)
        r = r2.sqrt()
        if kernel == "smooth" and grad:
            t = -ALPHA * r
            top = t.max(dim=1, keepdim=True).values
            w = (t - top).exp()
            s = w.sum(1)
            values.append(-(top[:, 0] + s.log()) / ALPHA)
            u = w / torch.where(r > 0, r, torch.ones_like(r))
            grads.append(torch.stack([-(u * x).sum(1) / s for x in d], 1))
            continue
        if kernel == "gravity":
            f = -m / (r + 0.1)
            g = torch.where(r > 0, -m / (r * (r + 0.1) ** 2), torch.zeros_like(r)) if grad else None
        elif kernel == "plummer":
            e2 = float(np.float32(EPS) * np.float32(EPS))
            f = m * (r2 + e2).rsqrt()
            g = m * (r2 + e2) ** -1.5 if grad else None
        elif kernel == "smooth":
            f = (-ALPHA * r).exp()
        else:
            dot = sum(nrm[None, :, k] * x for k, x in enumerate(d))
            pi = float(np.float32(math.pi))
            f = m * dot / (4 * pi * (r2 * r + 1e-5) if dim == 3 else 2 * pi * (r2 + 1e-5))
        values.append(f.sum(1))
        if grad:
            grads.append(torch.stack([(g * x).sum(1) for x in d], 1))
    v = torch.cat(values).cpu()
    return (v, torch.cat(grads).cpu()) if grad else v


def exact(case, seed):
    """Barnes-Hut and the sampler approximate the sums by construction (which nodes they open is
    decided in FP32), so they have no 64-bit value of their own; exact summation has."""
    what = case["what"]
    if what == "serve":
        trees, reqs = _serve_plan(case, seed)
        points = [_points(*t) for t in trees]
        out = []
        for t, kernel, nq, s in reqs:
            if SERVED[kernel][0] != "brute_force" or nq * trees[t][1] > 1 << 31:
                out.append(None)
                continue
            lo, hi = W.padded_box(points[t][0])
            q = np.random.default_rng(s).uniform(lo, hi, (nq, len(lo))).astype(np.float32)
            out.append(_sum64(kernel, *points[t], q.T))
        return out
    if what not in ("eval", "grad") or case["method"] != "brute_force":
        return None
    pts, nrm, m = _points(case["source"], case["n"], case["dim"], seed)
    q = _queries(case, seed, *W.padded_box(pts))
    if what == "grad":
        return _sum64(case["kernel"], pts, nrm, m, q, grad=True)
    v = _sum64(case["kernel"], pts, nrm, m, q)
    return (v, None) if case["host"] else v
