"""Performance cases of the framework: what a user's program has it do, through
the public Python interface (`amrlbm.AmrLbm`, `amrlbm.Net`).

A case is a dict of plain values. Its "kind" says what one pass is:

  loop     a solver run between two outputs: `steps` iterations of the main loop
           (regrids inside), then every leaf's fields and the diagnostics on the host
  coupled  a host code that owns the fields (the Fortran driver's arrays): upload of
           every leaf, `steps` iterations, download of every leaf and the diagnostics
  calls    the reference driver's Main_Loop through its separate call sites, `steps`
           times, then the fields on the host
  batch    `count` uneven problems in one pool, `steps` iterations, then every
           instance's diagnostics and the fields C, P, Ux, Uy on the host
  train    `steps` Adam steps of the refine-flag forecaster on minibatches of `count`
  infer    the forecaster's logits of `count` blocks

Fields go to page-locked arrays of a fixed capacity, allocated once (the mesh
changes, so the leaf count does); the part past the current leaves stays zero.

Time loops go on from the state that the pass before left, as a run does.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..",
                                "amr-lbm-openmp-2d_b200"))
import amrlbm  # noqa: E402

FIELDS = ("h", "g", "C", "P", "Ux", "Uy")
MACRO = ("C", "P", "Ux", "Uy")


# ---------------------------------------------------------------------------
# the cases

def listed():
    def mesh(name, kind, nbx, nby, levels, radius, **kw):
        c = dict(name=name, kind=kind, nx=16, ny=16, nbx=nbx, nby=nby, levels=levels, min_levels=0,
                 radius=radius, ratio=10.0, visc=10.0, bo=10.0, ar=archimedes(10.0, 1e-3), gy=5e-6,
                 w=4.0, m0=0.02, tol=1e-3, every=10, steps=100, precision="fp64", bubbles=1,
                 forecast=False)
        c.update(kw)
        return c

    # a sixteenth of the workloads' gravity at their relaxation times (a quarter
    # of their Archimedes number): over the thousands of steps that repeated
    # passes add up to, the bubble stays where it is and the mesh about as large
    large = dict(ratio=1000.0, visc=100.0, ar=archimedes(10.0, 1e-5) / 4, gy=2.5e-7 / 16)
    many = dict(ratio=1000.0, visc=100.0, bo=20.0, ar=40.0 / 4, tol=3e-4, bubbles=8,
                gy=5e-6 * 51.2 ** 3 / 128.0 ** 3 / 16)
    return [
        # the reference's own compile-time configuration: 8x8 blocks, a regrid
        # after every step. A mesh of a few dozen blocks: launches and latency
        mesh("reference_8x8_fp64", "loop", 1, 3, 5, 25.6, nx=8, ny=8, min_levels=1, ratio=1000.0,
             visc=100.0, bo=40.0, ar=40.0, w=5.0, m0=0.03, tol=2e-3, every=1, steps=32),
        # the small validation bubble (64x128 base, density ratio 10), regrid every step
        mesh("small_every_step_fp64", "loop", 4, 8, 2, 32.0, every=1, steps=64),
        # the same in 16-bit storage with the usual interval
        mesh("small_bf16", "loop", 4, 8, 2, 32.0, precision="bf16"),
        # the headline workload (256x512 base, 3 levels, density ratio 1000)
        mesh("large_fp64", "loop", 16, 32, 3, 128.0, **large),
        mesh("large_fp16", "loop", 16, 32, 3, 128.0, precision="fp16", **large),
        # the headline workload driven by a code that keeps the fields on the host
        mesh("coupled_fp64", "coupled", 16, 32, 3, 128.0, steps=10, **large),
        # ... and by the reference's driver through its separate call sites
        mesh("call_sites_fp64", "calls", 16, 32, 3, 128.0, steps=4, **large),
        # blocks that are neither square nor a power of two, an odd base grid
        mesh("ragged_12x10_fp64", "loop", 13, 27, 2, 96.0, nx=12, ny=10, tol=3e-4,
             gy=1e-7, ar=archimedes(10.0, 1e-3) / 4),
        # eight bubbles (radius 32 to 128), regrids every 32 steps with the forecaster attached
        mesh("bubbles_forecast_fp64", "loop", 32, 64, 3, 64.0, every=32, steps=96, forecast=True,
             **many),
        # a parameter study: uneven problems advanced together
        dict(name="batch_fp64", kind="batch", count=48, precision="fp64", every=10, steps=30),
        dict(name="batch_fp16", kind="batch", count=48, precision="fp16", every=10, steps=30),
        # training the forecaster: minibatches of the size that the training loop uses
        dict(name="train_512", kind="train", count=512, steps=4),
    ]


def draw(rng):
    """One more case of the ranges that the listed ones span."""
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    kind = rng.choice(("loop", "loop", "loop", "loop", "coupled", "calls", "batch", "train",
                       "infer"))
    if kind == "train":
        return dict(kind=kind, count=int(log(33, 512)), steps=rng.randint(1, 4))
    if kind == "infer":
        return dict(kind=kind, count=int(log(65, 4096)), steps=1)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(8, 40), every=rng.choice((8, 10, 32)),
                    precision=rng.choice(("fp64", "fp16", "bf16")), steps=rng.randint(10, 30))
    nx, ny = rng.choice(((16, 16), (16, 16), (16, 16), (8, 8), (12, 10), (10, 14), (20, 8)))
    precision = rng.choice(("fp64", "fp64", "fp16", "bf16")) if nx == ny else "fp64"
    levels = rng.randint(2, 3)
    nbx = int(log(3, 24))
    nby = int(nbx * rng.uniform(1.6, 2.4)) + 1
    side = min(nx * nbx, ny * nby / 2.0) * 2 ** levels
    radius = side * rng.uniform(0.12, 0.22)
    ratio = log(10, 1000)
    eo = rng.uniform(2, 40)
    # gravity for a velocity scale sqrt(gy D) and relaxation times of the
    # heavy phase that the lattice carries (tau between about 0.05 and 0.6)
    scale, tau = 0.0015, log(0.06, 0.4)
    gy = scale ** 2 / (2 * radius)
    muh = tau / 3.0
    ar = math.sqrt(gy * (1 - 1 / ratio) * (2 * radius) ** 3) / muh
    every = rng.choice((1, 4, 10, 32))
    steps = rng.randint(2, 4) if kind == "calls" else rng.randint(5, 40) if kind == "coupled" else \
        rng.randint(20, 100)
    return dict(kind=kind, nx=nx, ny=ny, nbx=nbx, nby=nby, levels=levels, min_levels=0,
                radius=radius, ratio=ratio, visc=min(ratio, 100.0), bo=eo, ar=ar, gy=gy, w=4.0,
                m0=0.02, tol=1e-3, every=every, steps=steps, precision=precision,
                bubbles=1, forecast=nx == ny == 16 and rng.random() < 0.2)


def archimedes(eo, mo):
    return (eo ** 3 / mo) ** 0.25


# ---------------------------------------------------------------------------
# what a program has in hand before the call

def refined_blocks(c):
    """Blocks that the interface refines, all levels together (measured on the
    listed meshes: 2 to 3 blocks across it)."""
    n, total = (c["nx"] + c["ny"]) / 2.0, 0.0
    for j in range(1, c["levels"] + 1):
        total += 2.4 * c["bubbles"] * 2 * math.pi * c["radius"] / (n * 2 ** j)
    return total


def pool_blocks(c):
    """Pool size of a mesh case: twice what the mesh starts with, or so, since
    it moves and the disturbed band widens."""
    base = c["nbx"] * c["nby"]
    full = sum(base * 4 ** lv for lv in range(c["levels"] + 1))
    return min(full, base + 4 * int(2.5 * refined_blocks(c) + 16))


def mesh_params(c, rng):
    """Solver parameters; the seed moves the bubble by a few cells and changes
    its size by a few per cent."""
    D = 2 ** c["levels"]
    width, height = c["nx"] * c["nbx"] * D, c["ny"] * c["nby"] * D
    radius = c["radius"] * rng.uniform(0.98, 1.02)
    return amrlbm.Params(
        nx=c["nx"], ny=c["ny"], nbx=c["nbx"], nby=c["nby"], dx0=D, min_levels=c["min_levels"],
        max_levels=c["levels"], max_blks=pool_blocks(c), regrid_every=c["every"],
        rho_l=1.0 / c["ratio"], rho_h=1.0, visc_ratio=c["visc"], bo=c["bo"], ar=c["ar"], gy=c["gy"],
        w=c["w"], m0=c["m0"], radius=radius, xc=width / 2.0 + rng.uniform(-6, 6),
        yc=height / 4.0 + rng.uniform(-6, 6), refin_tol=c["tol"], deref_tol=c["tol"] / 2,
        hydrostatic_start=1)


def host_arrays(sim, capacity, fields):
    size = dict(h=np.prod(sim.hshape), g=np.prod(sim.hshape), C=np.prod(sim.cshape),
                P=np.prod(sim.pshape), Ux=np.prod(sim.pshape), Uy=np.prod(sim.pshape))
    return {k: torch.zeros(capacity, int(size[k]), dtype=torch.float64, pin_memory=True).numpy()
            for k in fields}


def net_weights(seed):
    """Weights of the forecaster as a training run starts from: He-scaled."""
    g = np.random.default_rng(seed)
    out = []
    for fan, n in ((36, 32), (288, 32), (288, 32)):
        out += [g.normal(0, math.sqrt(2.0 / fan), fan * n), np.zeros(n)]
    out += [g.normal(0, math.sqrt(1.0 / 32), 32), np.zeros(1)]
    return np.concatenate(out).astype(np.float32)


def net_samples(count, seed):
    """Samples as `block_features` gives them, of planar interfaces through the
    block at random places and angles: C, the logarithm of the error term, the
    flow; labels of about one in four."""
    g = np.random.default_rng(seed)
    y, x = np.meshgrid(np.arange(18) - 8.5, np.arange(18) - 8.5, indexing="ij")
    ang, off = g.uniform(0, 2 * np.pi, (count, 1, 1)), g.uniform(-24, 24, (count, 1, 1))
    dist = x * np.cos(ang) + y * np.sin(ang) - off
    C = 0.5 + 0.5 * np.tanh(dist / 2.0)
    e = 0.25 / np.cosh(dist / 2.0) ** 2
    out = np.zeros((count, 4, 18, 18), np.float32)
    out[:, 0], out[:, 1] = C, np.log1p(e / 1e-3)
    for k in (2, 3):
        out[:, k, 1:17, 1:17] = g.normal(0, 0.05, (count, 1, 1)) + g.normal(0, 0.005, (count, 16, 16))
    return out, (g.random(count) < np.where(np.abs(off.ravel()) < 10, 0.45, 0.05)).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "infer"):
        net = amrlbm.Net(seed=seed, max_batch=512)
        net.set_params(net_weights(seed))
        x, y = net_samples(case["count"] * case["steps"], seed)
        return dict(case=case, net=net, x=x, y=y)
    rng = random.Random(seed)
    if kind == "batch":
        inst = amrlbm.batch_instances(case["count"], seed=seed)
        base = sum(i.nbx * i.nby for i in inst)
        pool = base + 1000 * len(inst)
        capacity = 400 * len(inst) + 2000
        sim = amrlbm.AmrLbm(amrlbm.batch_params(max_blks=pool, regrid_every=case["every"]),
                            instances=inst)
        fields = MACRO
    else:
        p = mesh_params(case, rng)
        base = p.nbx * p.nby
        capacity = base + 3 * (p.max_blks - base) // 4 + 1  # all that the pool can hold
        sim = amrlbm.AmrLbm(p)
        if case["bubbles"] > 1:
            width = case["nx"] * case["nbx"] * 2 ** case["levels"]
            height = case["ny"] * case["nby"] * 2 ** case["levels"]
            # the several-bubble workload's own layout, each a little elsewhere
            xyr = amrlbm.random_bubbles(case["bubbles"], case["radius"] / 2, case["radius"] * 2,
                                        width, height, 20261205)
            sim.set_bubbles([[x + rng.uniform(-1.5, 1.5), y + rng.uniform(-1.5, 1.5),
                              r * rng.uniform(0.98, 1.0)] for x, y, r in xyr])
        fields = FIELDS
    sim.initialize_rising_bubble()
    sim.set_precision(case["precision"])
    state = dict(case=case, sim=sim, out=host_arrays(sim, capacity, fields), fields=fields, net=None)
    if case.get("forecast"):
        state["net"] = amrlbm.Net(seed=seed, max_batch=512)
        state["net"].set_params(net_weights(seed))
        # a threshold that a trained forecaster's confident flags pass
        sim.set_regrid_net(state["net"], horizon=16.0, threshold=0.999999)
    if kind == "coupled":
        state["ids"], state["now"] = download(state)
    return state


# ---------------------------------------------------------------------------
# one pass

def download(state):
    """Every leaf's fields into the page-locked arrays; the leaves' ids."""
    sim, out = state["sim"], state["out"]
    ids = sim.leaves()
    part = {k: v[:len(ids)] for k, v in out.items()}
    if state["fields"] is FIELDS:
        sim.download_fields(ids, out=part)
    else:
        # the wrapper of a whole-block download always takes h and g too:
        # the C interface takes any of the fields
        import ctypes as ct
        ids = np.ascontiguousarray(ids, dtype=np.int32)
        ptr = [part[k].ctypes.data_as(ct.POINTER(ct.c_double)) if k in part else None
               for k in FIELDS]
        status = sim.lib.amrlbm_download_fields(
            sim.ctx, len(ids), ids.ctypes.data_as(ct.POINTER(ct.c_int32)), *ptr)
        if status:
            raise amrlbm.AmrLbmError(status, "download")
    for v in out.values():
        v[len(ids):state.get("filled", 0)] = 0.0
    state["filled"] = len(ids)
    return ids, part


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "infer":
        return {"logits": state["net"].forward(state["x"])}
    if kind == "train":
        net, n, losses = state["net"], case["count"], []
        for i in range(case["steps"]):
            losses.append(net.train_step(state["x"][i * n:(i + 1) * n], state["y"][i * n:(i + 1) * n],
                                         lr=2e-3, pos_weight=3.0))
        return {"losses": np.array(losses, np.float32), "weights": net.params()}
    sim = state["sim"]
    if kind == "coupled":
        sim.upload_fields(state["ids"], state["now"])
    if kind == "calls":
        for _ in range(case["steps"]):
            sim.determine_min_max_levels()
            sim.fill_ghost_cells_c2()
            sim.phase_field_lbm_h_g()
            sim.macroscopic_values_h()
            sim.fill_ghost_cells_c()
            sim.macroscopic_values_g()
            sim.refine_derefine_mesh()
    else:
        sim.main_loop(case["steps"])
    ids, part = download(state)
    if kind == "coupled":
        state["ids"], state["now"] = ids, part
    diag = [sim.output()] if kind != "batch" else sim.output_instances()
    return {"leaves": len(ids), "fields": state["out"],
            "diagnostics": np.array([[d[k] for k in sorted(d)] for d in diag])}


# ---------------------------------------------------------------------------

def work(case):
    """Bytes: per update of a leaf cell every population, C, P, Ux and Uy read
    and written once (352 bytes in FP64, 104 in 16-bit storage), and the
    fields that go to and from the host. Operations: those of the formulas."""
    kind = case["kind"]
    if kind in ("train", "infer"):
        n = case["count"] * case["steps"]
        flops = 2.0 * 324 * 32 * (36 + 288 + 288) * n
        return dict(bytes=n * 4 * 324 * 4.0 + 4 * 20801.0 * 8 * (kind == "train"),
                    flops=flops * (3 if kind == "train" else 1))
    per = 352 if case["precision"] == "fp64" else 104
    if kind == "batch":
        cells, host = 330 * case["count"] * 256.0, (400.0 / 256 + 3) * 8
    else:
        cells = (case["nbx"] * case["nby"] + 3 * refined_blocks(case)) * case["nx"] * case["ny"]
        host = (18 * (1 + 2.0 / case["nx"]) * (1 + 2.0 / case["ny"]) + 5) * 8
        host *= 2 if kind == "coupled" else 1
    return dict(bytes=cells * (per * case["steps"] + host), flops=cells * 700.0 * case["steps"])


# ---------------------------------------------------------------------------
# 64-bit values

def exact(case, seed):
    """The forecaster in 64 bits with torch. The mesh cases have none here: the
    adaptive time loop (quadtree with its id allocation, interpolated ghost
    rings, regrids) in plain numpy would be a second solver."""
    if case["kind"] not in ("train", "infer"):
        return None
    n, steps = case["count"], case["steps"]
    x, y = net_samples(n * steps, seed)
    w = torch.from_numpy(net_weights(seed).astype(np.float64)).requires_grad_()

    def logits(xb):
        at, a = 0, torch.from_numpy(xb.astype(np.float64))
        for cin in (4, 32, 32):
            k = w[at:at + 9 * cin * 32].reshape(3, 3, cin, 32).permute(3, 2, 0, 1)
            b = w[at + 9 * cin * 32:at + 9 * cin * 32 + 32]
            at += 9 * cin * 32 + 32
            a = torch.relu(torch.nn.functional.conv2d(a, k, b, padding=1))
        return a.amax(dim=(2, 3)) @ w[at:at + 32] + w[at + 32]

    if case["kind"] == "infer":
        with torch.no_grad():
            return {"logits": torch.cat([logits(x[i:i + 512]) for i in range(0, n, 512)])}
    m1, m2, losses = torch.zeros_like(w), torch.zeros_like(w), []
    for i in range(steps):
        yb = torch.from_numpy(y[i * n:(i + 1) * n].astype(np.float64))
        z = logits(x[i * n:(i + 1) * n])
        loss = torch.nn.functional.binary_cross_entropy_with_logits(
            z, yb, pos_weight=torch.tensor(3.0, dtype=torch.float64))
        g, = torch.autograd.grad(loss, w)
        losses.append(loss.item())
        with torch.no_grad():
            m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
            w -= 2e-3 * (m1 / (1 - 0.9 ** (i + 1))) / ((m2 / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
    return {"losses": np.array(losses), "weights": w.detach()}
