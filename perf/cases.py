"""Performance cases: what programs call this framework for, through its public entry points, over the sizes they use.

The engine's work is one voxel solve per foot and surgical action (``solve_cn``: operator and hierarchy set-up, CG,
displacements and reactions), the single-connectivity block solve (``solve``), batches of small feet, and the pieces
of those that a program keeps a handle for (``Problem.solve`` for another load, ``Problem.precondition``,
``Problem.apply``), the stress recovery after a solve, and the layers of the warm-start network, forward and
backward.  Sizes follow the repository's configurations: feet from 24x18x16 cells (tests) over 96x64x48 (training
grid) to 160x112x96 (5M dofs), blocks around 48x32x24, network layers of the 96x64x48 network.

A foot's geometry comes from ``synth.hindfoot_problem`` (case field ``foot``: the geometry's seed); the seed of
``prepare`` draws the patient: tissue stiffnesses, ground and ligament stiffness, the load and the vectors.
"""
import ctypes as C
import functools

import numpy as np
import torch

from comech_b200 import _lib, batch, engine, synth, warmnet
from comech_b200.grid import lame

KINDS = {"conv3": _lib.GATHER_SHIFT, "down": _lib.GATHER_DOWN, "up": _lib.GATHER_ONE}
TAPS = {"conv3": 27, "down": 8, "up": 8}


def listed():
    return [
        # the smallest solve a program makes: a test-sized foot from host arrays, launch- and host-bound
        dict(name="foot 24x18x16 mixed", op="foot", nx=24, ny=18, nz=16, foot=1, action="none", precision="mixed",
             tol=1e-10, warm=False),
        # the two-material block, plain FP64, from host arrays
        dict(name="block 48x32x24 fp64", op="block", nx=48, ny=32, nz=24, precision="fp64", tol=1e-10),
        # one foot of the training-set size with an osteotomy, the whole engine call with the learned start
        dict(name="foot 96x64x48 mixed warm", op="foot", nx=96, ny=64, nz=48, foot=2, action="osteotomy",
             precision="mixed", tol=1e-10, warm=True),
        # the 5M-dof foot from device arrays: set-up, solve, displacements and stress (the headline workload)
        dict(name="foot 160x112x96 device", op="device", nx=160, ny=112, nz=96, foot=0, action="none",
             precision="mixed", tol=1e-9, warm=True),
        # a bank of uneven feet and actions solved together
        dict(name="batch of 6 feet", op="batch", nx=40, ny=30, nz=25, foot=3, count=6, precision="mixed", tol=1e-10),
        # another load on a foot whose handle is kept: odd sizes, plain FP64
        dict(name="solve 64x45x38 fp64", op="solve", nx=64, ny=45, nz=38, foot=4, action="fusion", precision="fp64",
             tol=1e-10),
        # the preconditioner alone, as a caller's own Krylov loop uses it
        dict(name="vcycle 96x64x48 fp64", op="vcycle", nx=96, ny=64, nz=48, foot=5, action="resection"),
        # the operator alone: K u in FP64 at the largest grid, in FP32 at an odd one
        dict(name="apply 160x112x96 fp64", op="apply", nx=160, ny=112, nz=96, foot=0, action="none", prec="fp64"),
        dict(name="apply 97x67x58 fp32", op="apply", nx=97, ny=67, nz=58, foot=6, action="interposition",
             prec="fp32"),
        # the widest layer at the network's full resolution (f0a), forward
        dict(name="conv 64-32 96x64x48", op="conv", kind="conv3", nx=96, ny=64, nz=48, ci=64, co=32),
        # a full-resolution layer's backward pass (f0b): data, weight and bias gradients
        dict(name="conv grad 32-32 96x64x48", op="grad", kind="conv3", nx=96, ny=64, nz=48, ci=32, co=32),
        # the bottleneck layer: few voxels, many channels
        dict(name="conv 256-256 12x8x6", op="conv", kind="conv3", nx=12, ny=8, nz=6, ci=256, co=256),
    ]


def draw(rng):
    """One more case: the operation, then sizes spread over the logarithm of its range, seldom round."""
    op = rng.choice(["foot", "block", "device", "solve", "vcycle", "apply", "conv", "grad", "conv", "grad", "batch",
                     "stress"])

    def log(a, b):
        return int(round(a * (b / a) ** rng.random()))

    def foot_dims(a, b):
        nx = log(a, b)
        return dict(nx=nx, ny=int(nx * rng.uniform(0.66, 0.74)), nz=int(nx * rng.uniform(0.56, 0.64)),
                    foot=rng.randrange(8))

    act = rng.choice(synth.ACTIONS)
    if op == "block":
        return dict(op=op, nx=log(14, 64), ny=log(12, 48), nz=log(10, 40), precision=rng.choice(["fp64", "mixed"]),
                    tol=1e-10)
    if op == "foot":
        return dict(op=op, **foot_dims(24, 90), action=act, precision=rng.choice(["fp64", "mixed", "mixed", "refine"]),
                    tol=1e-10, warm=rng.random() < 0.4)
    if op == "device":
        return dict(op=op, **foot_dims(48, 140), action=act, precision=rng.choice(["fp64", "mixed"]), tol=1e-10,
                    warm=rng.random() < 0.5)
    if op == "solve":
        return dict(op=op, **foot_dims(24, 110), action=act, precision=rng.choice(["fp64", "mixed"]), tol=1e-10)
    if op == "vcycle":
        return dict(op=op, **foot_dims(24, 140), action=act)
    if op == "apply":
        return dict(op=op, **foot_dims(24, 140), action=act, prec=rng.choice(["fp64", "fp32"]))
    if op == "batch":
        return dict(op=op, **foot_dims(24, 44), count=rng.randrange(4, 8), precision=rng.choice(["fp64", "mixed"]),
                    tol=1e-10)
    if op == "stress":
        return dict(op=op, **foot_dims(24, 140), action=act)
    kind = rng.choice(["conv3", "conv3", "conv3", "down", "up"])
    l = rng.randrange(4 if kind == "conv3" else 3)
    s = [(96, 64, 48)[d] * rng.uniform(0.7, 1.0) / 2 ** l for d in range(3)]
    nx, ny, nz = (max(4, int(v)) if kind == "conv3" else max(4, 2 * int(v / 2)) for v in s)
    w = warmnet.WIDTHS[l]
    ci, co = {"conv3": (rng.choice([w, w, 2 * w]) if l < 3 else w, w), "down": (w, 2 * w),
              "up": (2 * w, w)}[kind]
    return dict(op=op, kind=kind, nx=nx, ny=ny, nz=nz, ci=ci, co=co)


# ---------------------------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=16)
def _geometry(nx, ny, nz, foot, action):
    P = synth.hindfoot_problem(nx, ny, nz, h=80.0 / nx, seed=foot, action=action)
    P["tissue"] = np.unique(np.stack([P["E"], P["nu"]], 1), axis=0, return_inverse=True)
    return P


def _foot(nx, ny, nz, foot, action, seed):
    """Inputs of solve_cn for one patient: the foot's geometry with drawn stiffnesses and load."""
    G = _geometry(nx, ny, nz, foot, action)
    rng = np.random.default_rng([seed, nx, foot])
    kinds, which = G["tissue"]
    E = (kinds[:, 0] * rng.uniform(0.7, 1.4, len(kinds)))[which.ravel()]
    lam, mu = lame(E, kinds[:, 1][which.ravel()])
    s = G["extra"]
    springs = synth.SpringSet(s.pair_a, s.pair_b, s.pair_k * rng.uniform(0.7, 1.4), s.line_a, s.line_b, s.line_d,
                              s.line_k * rng.uniform(0.7, 1.4, len(s.line_k)))
    fn, fa = G["fixed"]
    (ln, la, lt), = G["loads"]
    t = lt * rng.uniform(0.6, 1.6) + np.linalg.norm(lt) * np.array([*rng.uniform(-0.15, 0.15, 2), 0.0])
    return dict(grid=G["grid"], lam=lam, mu=mu, active=G["active"], cn=G["cn"], orig=G["orig"],
                fixed=(fn, fa * rng.uniform(0.7, 1.4)), loads=[(ln, la, t)], extra=springs,
                node_groups=G["node_groups"])


def _block(case, seed):
    P = synth.block_problem(case["nx"], case["ny"], case["nz"], seed=seed)
    return dict(grid=P["grid"], lam=P["lam"], mu=P["mu"], active=P["active"], springs=P["springs"], loads=P["loads"])


def _case_foot(case, seed):
    return _foot(case["nx"], case["ny"], case["nz"], case["foot"], case["action"], seed)


def _batch_items(case, seed):
    out = []
    for i in range(case["count"]):
        f = 1.0 + 0.25 * i / (case["count"] - 1)
        out.append(_foot(int(case["nx"] * f), int(case["ny"] * f), int(case["nz"] * f), case["foot"] + i,
                         synth.ACTIONS[1 + i % 5], seed + i))
    return out


def _on_device(P):
    """The operator's big arrays on the device, the small ones on the host (as Problem takes them)."""
    fn, fa = P["fixed"]
    nr, cr, nc, cc, v = P["extra"].node_coo()
    (ln, la, lt), = P["loads"]
    groups = P["node_groups"]
    return dict(mat=torch.from_numpy(np.concatenate([P["lam"], P["mu"]])).cuda(),
                active=torch.from_numpy(P["active"].astype(np.uint8)).cuda(),
                cn=torch.from_numpy(np.ascontiguousarray(P["cn"], np.int64)).cuda(),
                orig=torch.from_numpy(np.ascontiguousarray(P["orig"], np.int64)).cuda(),
                cells=torch.from_numpy(np.flatnonzero(P["active"])).cuda(),
                pen_node=fn, pen_k=np.repeat((fa * engine.K_GROUND)[:, None], 3, axis=1),
                extra=(3 * nr + cr, 3 * nc + cc, v), g_off=np.r_[0, np.cumsum([len(x) for x in groups])],
                g_nodes=torch.from_numpy(np.concatenate(groups)).cuda(), l_nodes=torch.from_numpy(ln).cuda(),
                l_vals=torch.from_numpy(la[:, None] * lt[None, :]).cuda(), load_nodes=ln, load_z=la * lt[2])


def _problem(P, d, precision, tol):
    return engine.Problem(P["grid"], _lib.MAT_ISO_SRI, d["mat"], d["active"], cn=d["cn"], orig=d["orig"],
                          pen_node=d["pen_node"], pen_k=d["pen_k"], extra_coo=d["extra"], precision=precision, tol=tol)


def _field(n, seed, dtype=torch.float64):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, generator=g, device="cuda", dtype=torch.float64).to(dtype)


def _rows(x, y, z):
    return (x + 2) * (y + 2) * (z + 2)


def _inside(x, y, z, dev="cuda"):
    m = torch.zeros(x + 2, y + 2, z + 2, dtype=torch.bool, device=dev)
    m[1:-1, 1:-1, 1:-1] = True
    return m.reshape(-1)


def _activations(dims, c, g, signed):
    """A layer's activations (after ReLU) or their gradients: BF16 rows of the padded grid with a zero shell."""
    a = torch.randn(_rows(*dims), c, generator=g, device="cuda")
    a = a if signed else a.clamp_(min=0)
    return (a * _inside(*dims)[:, None]).to(torch.bfloat16)


def _layer(case, seed):
    """Input, output gradient, weights [taps][co][ci] and bias of one layer.  nx, ny, nz: the finer grid."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    fine = (case["nx"], case["ny"], case["nz"])
    coarse = tuple(v // 2 for v in fine)
    kind, ci, co = case["kind"], case["ci"], case["co"]
    src, dst = {"conv3": (fine, fine), "down": (fine, coarse), "up": (coarse, fine)}[kind]
    W = torch.randn(TAPS[kind], co, ci, generator=g, device="cuda")
    W *= (2.0 / (ci * (1 if kind == "up" else TAPS[kind]))) ** 0.5
    return dict(src=src, dst=dst, fine=fine, coarse=coarse, x=_activations(src, ci, g, False),
                gy=_activations(dst, co, g, True), W=W, b=0.1 * torch.randn(co, generator=g, device="cuda"))


def prepare(case, seed):
    op = case["op"]
    s = dict(case=case)
    if op == "foot":
        s["P"] = _case_foot(case, seed)
        s["net"] = warmnet.default_net() if case["warm"] else None
    elif op == "block":
        s["P"] = _block(case, seed)
    elif op == "batch":
        s["items"] = _batch_items(case, seed)
    elif op == "device":
        s["P"] = _case_foot(case, seed)
        s["d"] = _on_device(s["P"])
        s["net"] = warmnet.default_net() if case["warm"] else None
    elif op in ("solve", "vcycle", "apply"):
        P = _case_foot(case, seed)
        d = _on_device(P)
        s["pr"] = _problem(P, d, case.get("precision", "fp64"), case.get("tol", 1e-8))
        s["pr"].set_rigid_groups(d["g_nodes"], offsets=d["g_off"])
        n = 3 * len(P["orig"])
        if op == "solve":
            s["f"] = s["pr"].rhs([(d["l_nodes"], d["l_vals"])])
        elif op == "vcycle":
            s["r"] = _field(n, seed) * s["pr"].used_mask()[0].repeat_interleave(3)
            s["pr"].precondition(s["r"])
        else:
            s["u"] = _field(n, seed, torch.float64 if case["prec"] == "fp64" else torch.float32)
    elif op == "stress":
        P = _case_foot(case, seed)
        s["P"], s["d"] = P, _on_device(P)
        s["U"] = 1e-3 * _field(3 * len(P["orig"]), seed)
    else:
        s.update(_layer(case, seed))
        flip = 1 if case["kind"] == "conv3" else 0
        t, co, ci = s["W"].shape
        s["fwd"], s["bwd"] = (torch.empty(t * co * ci, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        _lib.check(_lib.load().feb_net_weights(engine._ptr(s["W"]), t, co, ci, engine._ptr(s["fwd"]),
                                               engine._ptr(s["bwd"]), flip, engine._stream()))
        s["y"] = torch.zeros(_rows(*s["dst"]), co, dtype=torch.bfloat16, device="cuda")
        s["gx"] = torch.zeros(_rows(*s["src"]), ci, dtype=torch.bfloat16, device="cuda")
        s["status"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    return s


# ---------------------------------------------------------------------------------------------- passes
def _conv(s, gather, grid, fine, src, wt, n, dst, bias=None, relu=0, mask=None, scatter_c=0):
    c = _lib.FebConv()
    c.gather, c.scatter = gather, 1 if scatter_c else 0
    c.grid, c.fine = _lib.FebNetGrid(*grid), _lib.FebNetGrid(*fine)
    setattr(c, "in", src.data_ptr())
    c.in_ld, c.kc, c.n, c.wt = src.shape[1], src.shape[1], n, wt.data_ptr()
    c.out, c.out_ld, c.scatter_c, c.relu = dst.data_ptr(), dst.shape[1], scatter_c, relu
    c.bias = bias.data_ptr() if bias is not None else None
    if mask is not None:
        c.mask, c.mask_ld = mask.data_ptr(), mask.shape[1]
    c.status = s["status"].data_ptr()
    _lib.check(_lib.load().feb_net_conv(C.byref(c), engine._stream()))


def _forward(s):
    """The layer with bias and ReLU (feb_net_conv), as the network's forward pass calls it."""
    kind, co = s["case"]["kind"], s["case"]["co"]
    grid = s["coarse"] if kind != "conv3" else s["fine"]
    _conv(s, KINDS[kind], grid, s["fine"], s["x"], s["fwd"], 8 * co if kind == "up" else co, s["y"], bias=s["b"],
          relu=1, scatter_c=co if kind == "up" else 0)
    return s["y"]


def _backward(s):
    """Data gradient (masked by the input's ReLU), weight gradient and bias gradient of the layer."""
    kind, ci, co = s["case"]["kind"], s["case"]["ci"], s["case"]["co"]
    grid = s["coarse"] if kind != "conv3" else s["fine"]
    gather = {"conv3": _lib.GATHER_SHIFT, "down": _lib.GATHER_ONE, "up": _lib.GATHER_DOWN}[kind]
    _conv(s, gather, grid, s["fine"], s["gy"], s["bwd"], 8 * ci if kind == "down" else ci, s["gx"], mask=s["x"],
          scatter_c=ci if kind == "down" else 0)
    dw, db = torch.zeros_like(s["W"]), torch.zeros_like(s["b"])
    w = _lib.FebWgrad()
    w.mode = {"conv3": _lib.GATHER_SHIFT, "down": _lib.GATHER_DOWN, "up": _lib.GATHER_UP}[kind]
    w.grid, w.fine = _lib.FebNetGrid(*grid), _lib.FebNetGrid(*s["fine"])
    w.p, w.p_ld, w.na, w.q, w.q_ld, w.nb = s["gy"].data_ptr(), co, co, s["x"].data_ptr(), ci, ci
    w.dw = dw.data_ptr()
    lib, st = _lib.load(), engine._stream()
    _lib.check(lib.feb_net_wgrad(C.byref(w), st))
    _lib.check(lib.feb_net_colsum(engine._ptr(s["gy"]), s["gy"].shape[0], co, 0, co, engine._ptr(db), st))
    return s["gx"], dw, db


def _stress(grid, mat, U, cells, cn):
    """Cell stress, von Mises and element forces on the device (feb_cell_stress, feb_element_forces)."""
    n = len(cells)
    sig, vm, eps, f = (torch.empty(k * n, dtype=torch.float64, device="cuda") for k in (6, 1, 6, 24))
    gs = engine._grid_struct(grid)
    lib, p, st = _lib.load(), engine._ptr, engine._stream()
    _lib.check(lib.feb_cell_stress(C.byref(gs), _lib.MAT_ISO_SRI, p(mat), p(U), n, p(cells), p(cn), 1, p(sig), p(vm),
                                   p(eps), st))
    _lib.check(lib.feb_element_forces(C.byref(gs), p(mat), p(U), n, p(cells), p(cn), p(f), st))
    return sig, vm, eps, f


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "foot":
        P = s["P"]
        U, _, R = engine.solve_cn(P["grid"], P["lam"], P["mu"], P["active"], P["cn"], P["orig"], P["fixed"], P["loads"],
                                  P["extra"], P["node_groups"], tol=case["tol"], precision=case["precision"],
                                  warm_start=s["net"])
        return U, R
    if op == "block":
        P = s["P"]
        U, _ = engine.solve(P["grid"], P["lam"], P["mu"], P["active"], P["springs"], P["loads"], method="gmg",
                            tol=case["tol"], precision=case["precision"])
        return U
    if op == "batch":
        return [(U, R) for U, _, R in batch.solve_batch(s["items"], precision=case["precision"], tol=case["tol"])]
    if op == "device":
        P, d = s["P"], s["d"]
        pr = _problem(P, d, case["precision"], case["tol"])
        try:
            pr.set_rigid_groups(d["g_nodes"], offsets=d["g_off"])
            f = pr.rhs([(d["l_nodes"], d["l_vals"])])
            x0, nc = None, len(P["lam"])
            if s["net"] is not None:
                x0 = s["net"].predict_x0(P["grid"], d["mat"][:nc], d["mat"][nc:], d["active"], P["orig"],
                                         P["fixed"][0], d["load_nodes"], d["load_z"], len(P["orig"]),
                                         orig_dev=d["orig"])
            x, _ = pr.solve(f, x0)
            U = pr.export(x)
            return (U, *_stress(P["grid"], d["mat"], U, d["cells"], d["cn"])[:2])
        finally:
            pr.close()
    if op == "solve":
        return s["pr"].solve(s["f"])[0]
    if op == "vcycle":
        return s["pr"].precondition(s["r"])
    if op == "apply":
        return s["pr"].apply(s["u"])
    if op == "stress":
        return _stress(s["P"]["grid"], s["d"]["mat"], s["U"], s["d"]["cells"], s["d"]["cn"])
    return _forward(s) if op == "conv" else _backward(s)


# ---------------------------------------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass at the least: inputs read once and outputs written once; iterative paths
    count their products of the operator (8 per iteration: two Chebyshev-3 smoothers with their residuals, the CG
    product and the coarser levels), each reading and writing its vectors once, for 50 iterations."""
    op = case["op"]
    x, y, z = case["nx"], case["ny"], case["nz"]
    if op in ("conv", "grad"):
        fine, coarse = x * y * z, (x // 2) * (y // 2) * (z // 2)
        kind, ci, co = case["kind"], case["ci"], case["co"]
        src, dst = {"conv3": (fine, fine), "down": (fine, coarse), "up": (coarse, fine)}[kind]
        flops = 2 * (fine if kind == "conv3" else coarse) * TAPS[kind] * ci * co
        nw = TAPS[kind] * ci * co
        if op == "conv":
            return {"bytes": 2 * (src * ci + dst * co + nw), "flops": flops}
        return {"bytes": 2 * (2 * src * ci + dst * co + nw) + 4 * nw, "flops": 2 * flops}
    cells, nodes = x * y * z, (x + 1) * (y + 1) * (z + 1)
    if op == "stress":
        return {"bytes": cells * (16 + 8 + 64 + 37 * 8) + nodes * 24, "flops": cells * 1400}
    if op == "apply":
        s = 8 if case["prec"] == "fp64" else 4
        return {"bytes": nodes * 6 * s + cells, "flops": cells * 300}
    if op == "vcycle":
        return {"bytes": 7 * nodes * 12 * 8, "flops": 7 * cells * 350}
    s = 4 if case["precision"] != "fp64" else 8
    solve = {"bytes": 50 * (7 * nodes * 12 * s + nodes * 20 * 8), "flops": 50 * 8 * cells * 350}
    if op == "batch":
        return {k: v * 1.4 * case["count"] for k, v in solve.items()}
    return solve


# ---------------------------------------------------------------------------------------------- 64-bit values
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


CORNER = np.array([[l & 1, l >> 1 & 1, l >> 2 & 1] for l in range(8)])


def _strain(pt, h):
    """Strain-displacement matrix (6, 24) of the trilinear hexahedron of edge h at the local point pt in [-1, 1]^3."""
    s = 2.0 * CORNER - 1.0
    B = np.zeros((6, 8, 3))
    for ax in range(3):
        a, b = (k for k in range(3) if k != ax)
        d = s[:, ax] * (1 + s[:, a] * pt[a]) * (1 + s[:, b] * pt[b]) / (4 * h)
        B[ax, :, ax] = d
        for row, (p, q) in ((3, (0, 1)), (4, (1, 2)), (5, (0, 2))):
            if ax in (p, q):
                B[row, :, q if ax == p else p] = d
    return B.reshape(6, 24)


def _element(h, sri):
    """lambda and mu parts (24, 24) of the element stiffness of a cube: mu with 2x2x2 points, lambda at the centre
    (sri) or with 2x2x2 points."""
    DL, DM = np.zeros((6, 6)), np.diag([2.0, 2, 2, 1, 1, 1])
    DL[:3, :3] = 1
    g = 3 ** -0.5
    Bs = [_strain([a, b, c], h) for a in (-g, g) for b in (-g, g) for c in (-g, g)]
    KM = sum(B.T @ DM @ B for B in Bs) * h ** 3 / 8
    B0 = _strain([0, 0, 0], h)
    KL = B0.T @ DL @ B0 * h ** 3 if sri else sum(B.T @ DL @ B for B in Bs) * h ** 3 / 8
    return KL, KM


class _Operator:
    """K u of a foot or a block in plain torch, 64 bits."""

    def __init__(self, P, sri):
        dev, g = _dev(), P["grid"]
        t = functools.partial(torch.as_tensor, device=dev)
        act = np.flatnonzero(P["active"])
        cn = P["cn"][act] if "cn" in P else g.cell_nodes[act]
        self.n = len(P["orig"]) if "orig" in P else (g.nx + 1) * (g.ny + 1) * (g.nz + 1)
        self.cn, self.lam, self.mu = t(cn), t(P["lam"][act])[:, None], t(P["mu"][act])[:, None]
        self.KL, self.KM = (t(K) for K in _element(float(g.xe[1] - g.xe[0]), sri))
        self.diag = torch.zeros(self.n, 3, dtype=torch.float64, device=dev)
        if "fixed" in P:
            fn, fa = P["fixed"]
            self.diag.index_add_(0, t(fn), t(np.repeat((fa * engine.K_GROUND)[:, None], 3, 1)))
            nr, cr, nc, cc, v = P["extra"].node_coo()
            self.row, self.col, self.val = t(3 * nr + cr), t(3 * nc + cc), t(v)
        else:
            for nodes, area, k in P["springs"]:
                self.diag.index_add_(0, t(nodes), t(area)[:, None] * t(k)[None])
            self.row = None
        self.used = torch.zeros(self.n, dtype=torch.bool, device=dev)
        self.used[self.cn.reshape(-1)] = True
        self.diag *= self.used[:, None]

    def __call__(self, u):
        u = u.reshape(self.n, 3)
        y = self.diag * u
        for c in range(0, len(self.cn), 1 << 19):
            cn = self.cn[c:c + (1 << 19)]
            ue = u[cn].reshape(-1, 24)
            f = self.lam[c:c + (1 << 19)] * (ue @ self.KL) + self.mu[c:c + (1 << 19)] * (ue @ self.KM)
            y.index_add_(0, cn.reshape(-1), f.reshape(-1, 3))
        y = y.reshape(-1)
        if self.row is not None:
            y.index_add_(0, self.row, self.val * u.reshape(-1)[self.col])
        return y

    def diagonal(self):
        d = self.diag.clone()
        e = self.lam * self.KL.diagonal()[None] + self.mu * self.KM.diagonal()[None]
        d.index_add_(0, self.cn.reshape(-1), e.reshape(-1, 3))
        d = d.reshape(-1)
        if self.row is not None:
            on = self.row == self.col
            d.index_add_(0, self.row[on], self.val[on])
        return d


def _exact_solution(P, sri):
    """Displacements by Jacobi-preconditioned CG in 64 bits to a residual of 1e-13; NaN on unused nodes."""
    K = _Operator(P, sri)
    dev = _dev()
    f = torch.zeros(K.n, 3, dtype=torch.float64, device=dev)
    for nodes, area, t in P["loads"]:
        f.index_add_(0, torch.as_tensor(nodes, device=dev),
                     torch.as_tensor(np.asarray(area)[:, None] * np.asarray(t)[None], device=dev))
    f = f.reshape(-1)
    d = K.diagonal()
    m = torch.where(d > 0, 1 / d, torch.zeros_like(d))
    x, r = torch.zeros_like(f), f.clone()
    z = m * r
    p, rz, stop = z.clone(), r @ z, 1e-13 * f.norm()
    for it in range(20000):
        q = K(p)
        a = rz / (p @ q)
        x += a * p
        r -= a * q
        if it % 50 == 0 and r.norm() < stop:
            break
        z = m * r
        rz, old = r @ z, rz
        p = z + (rz / old) * p
    U = x.reshape(-1, 3)
    return torch.where(K.used[:, None], U, torch.full_like(U, float("nan"))).cpu().numpy()


def _exact_layer(case, seed):
    s = _layer(case, seed)
    op, kind, ci, co = case["op"], case["kind"], case["ci"], case["co"]
    dev = s["x"].device
    x, gy = s["x"].double(), s["gy"].double()
    W = s["W"].to(torch.bfloat16).double()
    X = x.reshape(*(v + 2 for v in s["src"]), ci)[1:-1, 1:-1, 1:-1]
    G = gy.reshape(*(v + 2 for v in s["dst"]), co)[1:-1, 1:-1, 1:-1]
    k = 3 if kind == "conv3" else 2
    taps = [(t // (k * k), t // k % k, t % k) for t in range(k ** 3)]

    def pad(v, dims, c):
        out = torch.zeros(*(d + 2 for d in dims), c, dtype=torch.float64, device=dev)
        out[1:-1, 1:-1, 1:-1] = v
        return out.reshape(-1, c)

    def window(v, t, dims):
        """v's cells that tap t pairs with each cell of the other side (a view of the fine or zero-padded grid)."""
        if kind == "conv3":
            return v.reshape(*(d + 2 for d in dims), -1)[tuple(slice(t[a], t[a] + dims[a]) for a in range(3))]
        return v[t[0]::2, t[1]::2, t[2]::2]

    if op == "conv":
        if kind == "up":
            y = torch.zeros(*s["dst"], co, dtype=torch.float64, device=dev)
            for i, t in enumerate(taps):
                window(y, t, None).copy_(X @ W[i].T)
        else:
            y = sum(window(x if kind == "conv3" else X, t, s["dst"]) @ W[i].T for i, t in enumerate(taps))
        return pad((y + s["b"].double()).clamp(min=0), s["dst"], co)
    gx = torch.zeros(*s["src"], ci, dtype=torch.float64, device=dev)
    dw = torch.zeros_like(s["W"], dtype=torch.float64)
    for i, t in enumerate(taps):
        if kind == "conv3":
            gx += window(gy, [2 - v for v in t], s["src"]) @ W[i]
            a, b = G, window(x, t, s["src"])
        elif kind == "down":
            window(gx, t, None).copy_(G @ W[i])
            a, b = G, window(X, t, None)
        else:
            gx += window(G, t, None) @ W[i]
            a, b = window(G, t, None), X
        dw[i] = a.reshape(-1, co).T @ b.reshape(-1, ci)
    return pad(gx * (X > 0), s["src"], ci), dw, gy.sum(0)


def exact(case, seed):
    op = case["op"]
    if op in ("conv", "grad"):
        return _exact_layer(case, seed)
    if op == "apply":
        P = _case_foot(case, seed)
        K = _Operator(P, True)
        u = _field(3 * K.n, seed, torch.float64 if case["prec"] == "fp64" else torch.float32).double().to(_dev())
        return K(u)
    if op == "block" and case["nx"] * case["ny"] * case["nz"] <= 60000:
        return _exact_solution(_block(case, seed), False)
    if op == "foot" and case["nx"] <= 40:
        return _exact_solution(_case_foot(case, seed), True), None
    if op == "stress":
        P = _case_foot(case, seed)
        act = np.flatnonzero(P["active"])
        U = (1e-3 * _field(3 * len(P["orig"]), seed)).to(_dev()).reshape(-1, 3)
        t = functools.partial(torch.as_tensor, device=_dev())
        lam, mu, h = t(P["lam"][act])[:, None], t(P["mu"][act])[:, None], 80.0 / case["nx"]
        u = U[t(P["cn"][act])].reshape(-1, 24)
        eps = u @ t(_strain([0, 0, 0], h)).T
        sig = mu * eps * t([2.0, 2, 2, 1, 1, 1])
        sig[:, :3] += lam * eps[:, :3].sum(1, keepdim=True)
        a, b, c = sig[:, 0], sig[:, 1], sig[:, 2]
        vm = (0.5 * ((a - b) ** 2 + (b - c) ** 2 + (c - a) ** 2) + 3 * (sig[:, 3:] ** 2).sum(1)).sqrt()
        KL, KM = (t(K) for K in _element(h, True))
        return sig.reshape(-1), vm, eps.reshape(-1), (lam * (u @ KL) + mu * (u @ KM)).reshape(-1)
    return None
