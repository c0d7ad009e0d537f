"""What is timed when this framework is made faster: the work its users have it do.

Every case goes through the package's public entry points on synthetic speckle frames (the
package's own renderer), sized as the repository's benchmark workloads, tests and baseline
configurations are.  ``listed()`` names the fixed cases, ``draw()`` gives further ones of the
same ranges, ``prepare()`` makes what a program holds before the call, ``run()`` is one pass,
``work()`` the bytes and operations a pass cannot do without, and ``exact()`` the same outputs
in 64-bit torch arithmetic where they have such values.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "3d-stereo-aldic_b200"))

import aldic_b200 as A  # noqa: E402
from aldic_b200 import learned as L  # noqa: E402
from aldic_b200 import synth_gpu, train_net  # noqa: E402

F64 = dict(dtype=torch.float64, device="cuda")


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # One camera, small frames: the 512 x 512 temporal pass (subset 31, 900 subsets), whose
        # kernels are short enough that launches and latency count.
        dict(name="temporal512", kind="pass", M=512, N=512, bits=8, w=30, step=16, search=10, tol=1e-3, quad=False,
             host=False),
        # A MATLAB-style caller with host arrays: 1920 x 1200 frames, subset 33, step 32 (the
        # reference's regression pipeline), a (step, subset) pair without a tile kernel.
        dict(name="host1920x1200", kind="pass", M=1920, N=1200, bits=8, w=32, step=32, search=20, tol=1e-3, quad=True,
             host=True),
        # One temporal frame with the search's initial guess: 2048 x 2048, subset 33, step 16.
        dict(name="frame2048", kind="pass", M=2048, N=2048, bits=8, w=32, step=16, search=16, tol=1e-3, quad=True,
             host=False),
        # The stereo match's initial guess: whole-field search of radius 70 on 16-bit frames,
        # bad-point removal and Init.
        dict(name="stereo_guess2048", kind="search", M=2048, N=2048, bits=16, w=40, step=10, search=70),
        # The stereo match's IC-GN: 40 000 subsets of 41 x 41 from a search's rounded guess, with
        # the Hessians that the ALDIC steps read.
        dict(name="icgn2048", kind="icgn", M=2048, N=2048, bits=16, w=40, step=10, tol=1e-3, quad=True, F0=False),
        # A plate with a hole on its quadtree mesh (masked subsets, nodes 4 to 16 px apart).
        dict(name="icgn_plate2048", kind="plate", M=2048, N=2048, w=32, step=16, hole=300, tol=1e-2),
        # The same plate's ALDIC local step (Subpb1) and global step (Subpb2).
        dict(name="subpb1_plate2048", kind="subpb1", M=2048, N=2048, w=32, step=16, hole=300, tol=1e-2),
        dict(name="subpb2_plate2048", kind="subpb2", M=2048, N=2048, w=32, step=16, hole=300, order=2, beta=1e-2),
        # One frame through the learned initial guess (network prediction, IC-GN from it, the
        # ZNCC judgement, the integer search where it fails).
        dict(name="learned2048", kind="learned", M=2048, N=2048, w=32, step=16, search=16, tol=1e-3),
        # Training the proposal network: Adam steps of 256 samples.
        dict(name="train256", kind="train", batch=256, steps=8),
        # One frame of a stereo sequence at 4096 x 3000: both cameras' IC-GN from extrapolated
        # guesses on 119 475 subsets each, then triangulation.
        dict(name="sequence4096", kind="sequence", M=4096, N=3000, bits=16, w=40, step=10, tol=1e-2),
    ]


def draw(rng):
    def logi(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["pass", "pass", "search", "icgn", "icgn", "plate", "subpb1", "subpb2", "learned", "train",
                       "sequence"])
    if kind in ("pass", "search"):
        while True:
            c = dict(kind=kind, M=logi(256, 2048), N=logi(256, 2048), bits=rng.choice([8, 16]),
                     w=2 * rng.randint(10, 24), step=rng.randint(8, 32), search=logi(4, 70))
            if rng.random() < 0.4:  # the window and step pairs of the usual set-ups
                c["step"], c["w"] = rng.choice([(10, 40), (16, 30), (16, 32), (12, 20), (8, 32)])
            n = (c["M"] // c["step"]) * (c["N"] // c["step"])
            if min(c["M"], c["N"]) > c["w"] + 2 * c["step"] + 2 * c["search"] + 8 \
                    and n * (2.0 * c["search"] + 3) ** 2 * (c["w"] + 1) ** 2 < 5e10:
                break
        if kind == "pass":
            c.update(tol=rng.choice([1e-2, 1e-3]), quad=rng.random() < 0.6, host=rng.random() < 0.3)
        return c
    if kind == "icgn":
        return dict(kind=kind, M=logi(300, 2048), N=logi(300, 2048), bits=rng.choice([8, 16]),
                    w=2 * rng.randint(10, 30), step=rng.randint(8, 24), tol=rng.choice([1e-2, 1e-3]),
                    quad=rng.random() < 0.6, F0=rng.random() < 0.4)
    if kind in ("plate", "subpb1", "subpb2"):
        M = 16 * rng.randint(40, 112)
        c = dict(kind=kind, M=M, N=16 * rng.randint(40, 112), w=rng.choice([16, 20, 24, 32, 40]), step=16,
                 hole=rng.randint(60, M // 8))
        if kind == "subpb2":
            c.update(order=rng.choice([2, 2, 3]), beta=rng.choice([1e-3, 1e-2, 1e-1]))
        else:
            c["tol"] = rng.choice([1e-2, 1e-3])
        return c
    if kind == "learned":
        return dict(kind=kind, M=4 * rng.randint(100, 512), N=4 * rng.randint(100, 512), w=32,
                    step=4 * rng.randint(3, 8), search=16, tol=rng.choice([1e-2, 1e-3]))
    if kind == "train":
        return dict(kind=kind, batch=8 * rng.randint(4, 64), steps=rng.choice([4, 8]))
    return dict(kind=kind, M=logi(1024, 4096), N=logi(768, 3000), bits=16, w=2 * rng.randint(12, 20),
                step=rng.randint(10, 20), tol=1e-2)


# --------------------------------------------------------------------------------- inputs
def _pair(seed, M, N, umax, bits=8):
    """A speckle pair under a smooth field, as flat CUDA tensors, x fastest."""
    p = synth_gpu.field_pair(seed, M=M, N=N, umax=umax, gmax=0.05)
    if bits == 16:
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed + 1)
        p.ref, p.deff = [(im.to(torch.int32) * 200 + torch.randint(0, 200, im.shape, generator=gen, device="cuda",
                                                                   dtype=torch.int32)).to(torch.uint16)
                         for im in (p.ref, p.deff)]
    return p


def _grid(M, N, w, step):
    """The search grid's subset centres ((2, n), x fastest) and its size."""
    return L.search_nodes([1, M], [1, N], w, step)


@functools.lru_cache(maxsize=1)
def _the_stream():
    return torch.cuda.Stream()


def _stream(ctx):
    """The one stream a program runs its frames on, in order."""
    ctx.set_stream(_the_stream().cuda_stream)
    return _the_stream()


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _icgn_out(n, H=True, mark=True):
    b = {"U": torch.empty(2 * n, **F64), "F": torch.empty(4 * n, **F64),
         "conv": torch.empty(n, dtype=torch.int32, device="cuda")}
    if H:
        b["H"] = torch.empty(21 * n, **F64)
    if mark:
        b["mark"] = torch.empty(n, dtype=torch.uint8, device="cuda")
    return b


def _load(ctx, s, both=True):
    M, N = s["M"], s["N"]
    ctx.load_image_raw(0, s["ref"], [1, M], [1, N], want_stats=False, shape=(M, N))
    if both:
        ctx.load_image_raw(1, s["deff"], [1, M], [1, N], want_stats=False, shape=(M, N))
    ctx.compute_gradients()


@functools.lru_cache(maxsize=4)
def _plate_mesh(M, N, w, step, hole):
    """The plate's mask and quadtree mesh, which a program makes once for a specimen."""
    x, y = np.meshgrid(np.arange(1, M + 1), np.arange(1, N + 1), indexing="ij")
    mask = np.ones((M, N))
    mask[(x - M / 2) ** 2 + (y - N / 2) ** 2 < hole ** 2] = 0
    nodes, nx, ny = _grid(M, N, w, step)
    X, Y = (c.reshape(ny, nx) for c in nodes)
    mesh = A.MeshSetUp(X, Y, {"winstepsize": step, "ImgSize": [M, N]})
    mesh["elementMinSize"] = 4
    q, _, _ = A.GenerateQuadtreeMesh(np.zeros(2 * nodes.shape[1]), None, mask, mesh, {"winstepsize": step, "winsize": w})
    return mask, q["coordinatesFEM"], q["elementsFEM"], np.asarray(q["dirichlet"])


def prepare(case, seed):
    c = dict(case)
    s = dict(c)
    rng = np.random.default_rng(seed)
    kind = c["kind"]
    if kind in ("pass", "search"):
        p = _pair(seed, c["M"], c["N"], 0.8 * c["search"], c["bits"])
        nodes, nx, ny = _grid(c["M"], c["N"], c["w"], c["step"])
        n = nx * ny
        s.update(ctx=A.Context(0), nx=nx, ny=ny, ref=p.ref, deff=p.deff)
        s["stream"] = _stream(s["ctx"])
        if c.get("host"):
            s.update(ref=p.ref.cpu().numpy().reshape(c["M"], c["N"], order="F"),
                     deff=p.deff.cpu().numpy().reshape(c["M"], c["N"], order="F"), coords=nodes.T.copy())
        else:
            s.update(coords=_dev(nodes), U0=torch.empty(2 * n, **F64), out=_icgn_out(n),
                     grid={k: torch.empty(n, **F64) for k in ("x", "y", "u", "v", "phi")})
        if kind == "search":
            _load(s["ctx"], s)
    elif kind == "icgn":
        p = _pair(seed, c["M"], c["N"], 12.0, c["bits"])
        nodes, _, _ = _grid(c["M"], c["N"], c["w"], c["step"])
        n = nodes.shape[1]
        u, v = p.field.disp(nodes[0], nodes[1])
        U0 = np.stack([u, v], 1).ravel() + rng.uniform(-0.1, 0.1, 2 * n)  # a search's guess: to 1e-3 px
        F0 = p.field.grad(nodes[0], nodes[1]).ravel() + rng.normal(0, 0.003, 4 * n)
        s.update(ctx=A.Context(0), ref=p.ref, deff=p.deff, coords=_dev(nodes), U0=_dev(np.round(U0, 3)),
                 F0=_dev(F0) if c["F0"] else None, out=_icgn_out(n))
        if c["F0"]:
            s["out"]["zncc"] = torch.empty(n, **F64)
        s["stream"] = _stream(s["ctx"])
        _load(s["ctx"], s)
    elif kind in ("plate", "subpb1", "subpb2"):
        mask, crd, elements, dirichlet = _plate_mesh(c["M"], c["N"], c["w"], c["step"], c["hole"])
        n = crd.shape[0]
        p = synth_gpu.field_pair(seed, M=64, N=64) if kind == "subpb2" else _pair(seed, c["M"], c["N"], 6.0)
        u, v = p.field.disp(crd[:, 0], crd[:, 1])
        F = p.field.grad(crd[:, 0], crd[:, 1])
        U = np.stack([u, v], 1).ravel()
        s.update(ctx=A.Context(0), n=n, coords=_dev(crd.T))
        s["stream"] = _stream(s["ctx"])
        if kind == "subpb2":
            s["ctx"].subpb2_set_mesh(n, elements, dirichlet)
            s.update(U=_dev(U + rng.normal(0, 0.01, 2 * n)), F=_dev((F + rng.normal(0, 1e-3, F.shape)).ravel()),
                     out=torch.empty(2 * n, **F64), mu=1e-3, beta=c["beta"] * c["step"] ** 2 * 1e-3)
        else:
            md = _dev(mask.ravel(order="F"))
            s.update(ref=(p.ref * md).to(torch.uint8), deff=p.deff, mask=md)
            ctx = s["ctx"]
            ctx.load_image_raw(0, s["ref"], [1, c["M"]], [1, c["N"]], want_stats=False, shape=(c["M"], c["N"]))
            ctx.load_image_raw(1, s["deff"], [1, c["M"]], [1, c["N"]], want_stats=False, shape=(c["M"], c["N"]))
            ctx.set_mask(md)
            ctx.compute_gradients()
            if kind == "plate":
                s.update(U0=_dev(np.round(U + rng.uniform(-0.1, 0.1, 2 * n), 3)), out=_icgn_out(n))
            else:
                s.update(U=_dev(U + rng.normal(0, 0.02, 2 * n)), F=_dev((F + rng.normal(0, 1e-3, F.shape)).ravel()),
                         vdual=_dev(rng.normal(0, 1e-3, 2 * n)),
                         wl=torch.full((2 * n,), c["w"], dtype=torch.int32, device="cuda"),
                         out={"U": torch.empty(2 * n, **F64), "conv": torch.empty(n, dtype=torch.int32, device="cuda")})
    elif kind == "learned":
        p = _pair(seed, c["M"], c["N"], 12.0)
        gx, gy = [21, c["M"] - 20], [21, c["N"] - 20]
        n = L.search_nodes(gx, gy, c["w"], c["step"])[0].shape[1]
        net = L.ProposalNet(0, max_batch=min(16384, (n + 7) // 8 * 8))
        net.set_params(np.load(train_net.DEFAULT_WEIGHTS))
        s.update(ctx=A.Context(0), net=net, ref=p.ref, deff=p.deff)
        s["li"] = L.LearnedInit(net, s["ctx"], c["search"], gx, gy, c["w"], c["step"], c["tol"],
                                stream=_the_stream())
    elif kind == "train":
        k, b = c["steps"], c["batch"]
        net = L.ProposalNet(0, max_batch=b, seed=seed % 1000)
        g = int(math.ceil(math.sqrt(k * b)))
        M = 12 * g + 80
        p = _pair(seed, M, M, 12.0)
        nodes = L.grid_nodes(M, M, 32, 12)[:, :k * b]
        ctx = A.Context(0)
        _load(ctx, dict(M=M, N=M, ref=p.ref, deff=p.deff))
        X = torch.empty((k * b, 72, 72, 2), dtype=torch.bfloat16, device="cuda")
        ctx.net_extract(_dev(nodes), X)
        ctx.synchronize()
        T = np.concatenate([np.stack(p.field.disp(nodes[0], nodes[1]), 1), p.field.grad(nodes[0], nodes[1])], 1)
        order = torch.randperm(k * b, generator=torch.Generator().manual_seed(seed)).cuda()
        X, T = X[order], _dev((T * L.SCALE).astype(np.float32))[order]
        net.set_stream(_the_stream().cuda_stream)
        s.update(net=net, stream=_the_stream(), X=list(X.split(b)), T=list(T.split(b)))
    elif kind == "sequence":
        nodes, _, _ = _grid(c["M"], c["N"], c["w"], c["step"])
        n = nodes.shape[1]
        f = 4000.0
        K = np.array([[f, 0, (c["M"] + 1) / 2.0], [0, f, (c["N"] + 1) / 2.0], [0, 0, 1.0]])
        a = math.atan(0.15) * 2
        R = np.array([[math.cos(a), 0, math.sin(a)], [0, 1, 0], [-math.sin(a), 0, math.cos(a)]])
        s.update(n=n, cams=[], K=K, R=R, T=np.array([-300.0, 0.0, 45.0]), pairs=torch.empty((4, n), **F64),
                 xyz={"xyz": torch.empty(3 * n, **F64), "err": torch.empty(n, **F64)})
        for k in range(2):
            p = _pair(2 * seed + k, c["M"], c["N"], 10.0, c["bits"])
            crd = nodes if k == 0 else nodes + rng.uniform(-3, 3, nodes.shape)  # the matched points: not on a grid
            u, v = p.field.disp(crd[0], crd[1])
            cam = dict(ctx=A.Context(0), M=c["M"], N=c["N"], ref=p.ref, deff=p.deff, coords=_dev(crd),
                       U0=_dev(np.stack([u, v], 1).ravel() + rng.normal(0, 0.05, 2 * n)),
                       out=_icgn_out(n, H=False, mark=False))
            s["stream"] = _stream(cam["ctx"])
            s.setdefault("main", cam["ctx"])
            _load(cam["ctx"], cam, both=False)
            s["cams"].append(cam)
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------- one pass
def _guess(s):
    """The whole-field search, the bad-point removal and Init, device-resident."""
    ctx, g = s["ctx"], s["grid"]
    ctx.integer_search([s["search"]] * 2, [1, s["M"]], [1, s["N"]], s["w"], s["step"], out=g)
    u, v = g["u"].view(s["nx"], s["ny"]), g["v"].view(s["nx"], s["ny"])
    ctx.remove_outliers(u, v, 100.0)
    ctx.init_u0(u, v, out=s["U0"])


def run(s):
    kind = s["kind"]
    if kind == "pass" and s["host"]:
        ctx = s["ctx"]
        _load(ctx, s)
        g = ctx.integer_search([s["search"]] * 2, [1, s["M"]], [1, s["N"]], s["w"], s["step"])
        u, v = ctx.remove_outliers(g["u"], g["v"], 100.0)
        U0 = ctx.init_u0(u, v)
        r = ctx.local_icgn(int(s["quad"]), s["coords"], U0, s["w"], s["tol"])
        return {"phi": g["phi"], "u": u, "v": v, "U": r["U"], "F": r["F"], "conv": r["conv"], "H": r["H"]}
    if kind == "pass":
        with torch.cuda.stream(s["stream"]):
            _load(s["ctx"], s)
            _guess(s)
            b = s["ctx"].local_icgn(int(s["quad"]), s["coords"], s["U0"], s["w"], s["tol"], out=s["out"])
        g = s["grid"]
        return {"phi": g["phi"], "u": g["u"], "v": g["v"], "U": b["U"], "F": b["F"], "conv": b["conv"], "H": b["H"]}
    if kind == "search":
        with torch.cuda.stream(s["stream"]):
            _guess(s)
        return {"phi": s["grid"]["phi"], "u": s["grid"]["u"], "v": s["grid"]["v"], "U0": s["U0"]}
    if kind in ("icgn", "plate"):
        with torch.cuda.stream(s["stream"]):
            F0 = s.get("F0")
            b = s["ctx"].local_icgn(int(s.get("quad", True)), s["coords"], s["U0"], s["w"], s["tol"], out=s["out"],
                                    F0=F0, want_zncc=F0 is not None)
        r = {k: b[k] for k in ("U", "F", "conv", "H")}
        if F0 is not None:
            r["zncc"] = b["zncc"]
        return r
    if kind == "subpb1":
        with torch.cuda.stream(s["stream"]):
            b = s["ctx"].subpb1(1, s["coords"], s["U"], s["F"], s["vdual"], 1e-3, s["tol"], winsize=s["w"],
                                winsize_list=s["wl"], out=s["out"])
        return {"U": b["U"], "conv": b["conv"]}
    if kind == "subpb2":
        with torch.cuda.stream(s["stream"]):
            s["ctx"].subpb2(s["coords"], None, s["order"], s["beta"], s["mu"], s["U"], s["F"], out=s["out"])
        return {"U": s["out"]}
    if kind == "learned":
        li = s["li"]
        with torch.cuda.stream(li.stream):
            _load(s["ctx"], s)
        li.run()
        return {k: li.buf[k] for k in ("U0", "F0", "U", "F", "conv", "zncc")}
    if kind == "train":
        with torch.cuda.stream(s["stream"]):
            for X, T in zip(s["X"], s["T"]):
                s["net"].train_step(X, T, 1e-4)
        return {"params": s["net"].get_params()}
    # sequence: the next frame of both cameras, then the points in space
    with torch.cuda.stream(s["stream"]):
        for cam in s["cams"]:
            cam["ctx"].load_image_raw(1, cam["deff"], [1, s["M"]], [1, s["N"]], want_stats=False,
                                      shape=(s["M"], s["N"]))
            cam["ctx"].local_icgn(1, cam["coords"], cam["U0"], s["w"], s["tol"], out=cam["out"])
        s["pairs"].copy_(torch.cat([cam["coords"] + cam["out"]["U"].view(-1, 2).t() for cam in s["cams"]], 0))
        s["main"].triangulate(s["pairs"], s["K"], s["K"], s["R"], s["T"], out=s["xyz"])
    return {"xyz": s["xyz"]["xyz"], "err": s["xyz"]["err"],
            "cams": [{k: cam["out"][k] for k in ("U", "F", "conv")} for cam in s["cams"]]}


# ----------------------------------------------------------------------------------- work
ITER = 4  # Gauss-Newton iterations a subset needs from a good guess


def _icgn_work(n, w, H):
    px = n * (w + 1) ** 2
    return (n * 8 * (4 + 6 + (21 if H else 0)), px * (92.0 * ITER + 50.0))


def _search_work(M, N, w, step, r):
    """Products and sums of the cross-correlation at every shift: the window products formed
    once per image position and shift, and per window one addition, one subtraction and the
    normalisation (the windows of a row overlap), or the windows apart where they do not."""
    nodes = max((M - w - step) // step, 1) * max((N - w - step) // step, 1)
    shifts = (2.0 * r + 3) ** 2
    share = min(float((w + 1) ** 2), 2.0 * step * step)
    return nodes * shifts * (2.0 * share + 8.0), nodes * 5 * 8


def work(case):
    c = case
    kind = c["kind"]
    if kind == "train":  # forward and backward (3x) of the network, per sample ~2.1 M + its windows' convolutions
        macs = 18 * 18 * 9 * 32 * 1.3 + (256 + 64) * 288 * 32 + 64 * 81 * 32 + 16 * 729 * 64 + 16 * 576 * 64 + 1024 * 128
        return {"bytes": c["steps"] * (c["batch"] * 72 * 72 * 2 * 2 + 227152 * 4 * 6.0),
                "flops": c["steps"] * c["batch"] * 6.0 * macs}
    M, N, w, step = c["M"], c["N"], c["w"], c["step"]
    px = float(M) * N
    if kind in ("plate", "subpb1", "subpb2"):
        n = M * N / step ** 2 + 2 * math.pi * c["hole"] / 4 * 10  # the grid, and the nodes along the hole's edge
        if kind == "subpb2":  # K_e once; a preconditioned CG of some 30 steps on x and y
            return {"bytes": n * 8 * 10, "flops": n * (8 * 4 * 120.0 + 30 * (4 * 32 * 2 + 20))}
        b, f = _icgn_work(n, w, kind == "plate")
        return {"bytes": px * 17 + b, "flops": f if kind == "plate" else f * 0.8}
    if kind == "sequence":
        n = (M // step - w // step) * (N // step - w // step)
        b, f = _icgn_work(n, w, False)
        return {"bytes": 2 * (px * (c["bits"] // 8 + 12) + b) + n * 64, "flops": 2 * f + n * 600.0}
    n = max((M - w - step) // step, 1) * max((N - w - step) // step, 1)
    b, f = _icgn_work(n, w, True)
    if kind == "icgn":
        return {"bytes": px * 16 + b, "flops": f}
    if kind == "learned":
        net = 2 * (px / 4 * 9 * 32 + px / 16 * 288 * 32) * 2 + n * 2.0 * (64 * 81 * 32 + 16 * 729 * 64 + 16 * 576 * 64
                                                                         + 1024 * 128)
        return {"bytes": 2 * px + b, "flops": f + net}
    sf, sb = _search_work(M, N, w, step, c["search"])
    if kind == "search":
        return {"bytes": px * 8 + sb, "flops": sf}
    return {"bytes": 2 * px * c["bits"] / 8 + b + sb, "flops": f + sf}


# ---------------------------------------------------------------------- the same in 64 bits
def _normal64(img, M, N):
    x = img.to(torch.int32).double().view(N, M).t()  # [x, y]
    return (x - x.mean()) / x.std()


def _grad64(f):
    """7-tap central differences (1/60 [-1 9 -45 0 45 -9 1]), valid part: (M-6) x (N-6)."""
    k = [-1, 9, -45, 0, 45, -9, 1]
    M, N = f.shape
    gx = sum(k[i] * f[i:M - 6 + i, 3:N - 3] for i in range(7)) / 60
    gy = sum(k[i] * f[3:M - 3, i:N - 6 + i] for i in range(7)) / 60
    return gx, gy


def _weights64(t):
    return [(t * (t * (-24 * t + 57) - 33)) / 56, (t * (t * (64 * t - 117) - 3) + 56) / 56,
            (t * (t * (-64 * t + 75) + 45)) / 56, (t * (t * (24 * t - 15) - 9)) / 56]


def _icgn64(ref, deff, M, N, coords, U0, F0, w, tol, quad, want_H):
    """First-order IC-GN (Gauss-Newton, the reference's stopping rules) of unmasked windows, all
    subsets of a chunk at once.  None where a window has pixels the reference treats apart."""
    f, g = _normal64(ref, M, N), _normal64(deff, M, N)
    gx, gy = _grad64(f)
    if bool((f == 0).any()) or bool((gx == 0).sum() > 0.02 * gx.numel()):
        return None
    n = coords.shape[1]
    U, F = torch.full((n, 2), math.nan, **F64), torch.full((n, 4), math.nan, **F64)
    H21 = torch.zeros((21, n), **F64)
    conv = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    zn = torch.full((n,), math.nan, **F64)
    crd = coords.t()
    if quad:
        crd = torch.floor(crd + 0.5)
    h, size = w // 2, torch.tensor([M, N], device="cuda")
    ok = ((crd == torch.floor(crd)) & (crd - h - 3 >= 1) & (crd + h - 3 <= size - 6)).all(1)
    todo = torch.nonzero(ok)[:, 0]
    d = torch.arange(-h, h + 1, **F64)
    dx, dy = (m.reshape(-1) for m in torch.meshgrid(d, d, indexing="ij"))
    tri = [(i, j) for i in range(6) for j in range(i, 6)]
    for at in todo.split(max(1, 4_000_000 // dx.numel())):
        c0 = crd[at]
        ix = (c0[:, :1] - 1 + dx).long()
        iy = (c0[:, 1:] - 1 + dy).long()
        fw, gxw, gyw = f[ix, iy], gx[ix - 3, iy - 3], gy[ix - 3, iy - 3]
        J = torch.stack([gxw * dx, gyw * dx, gxw * dy, gyw * dy, gxw, gyw], 1)
        H = J @ J.transpose(1, 2)
        mf = fw.mean(1, keepdim=True)
        bf = ((fw - mf) ** 2).sum(1, keepdim=True).sqrt()
        fn = (fw - mf) / bf
        P = torch.zeros((at.numel(), 6), **F64)
        if F0 is not None:
            P[:, :4] = F0.view(-1, 4)[at]
        P[:, 4:] = U0.view(-1, 2)[at]
        code = torch.full((at.numel(),), 101, dtype=torch.int32, device="cuda")
        z = torch.full((at.numel(),), math.nan, **F64)
        live = torch.arange(at.numel(), device="cuda")
        first = torch.zeros(at.numel(), **F64)
        for it in range(1, 102):
            p, cc = P[live], c0[live]
            lx = cc[:, :1] + p[:, 4:5] + (1 + p[:, :1]) * dx + p[:, 2:3] * dy
            ly = cc[:, 1:] + p[:, 5:] + p[:, 1:2] * dx + (1 + p[:, 3:4]) * dy
            inside = ((lx.amin(1) >= 3) & (lx.amax(1) <= M - 2) & (ly.amin(1) >= 3) & (ly.amax(1) <= N - 2))
            live, p, lx, ly = live[inside], p[inside], lx[inside], ly[inside]
            if live.numel() == 0:
                break
            fx, fy = torch.floor(lx), torch.floor(ly)
            wx, wy = _weights64(lx - fx), _weights64(ly - fy)
            kx, ky = fx.long() - 2, fy.long() - 2
            gw = sum(wy[b] * sum(wx[a] * g[kx + a, ky + b] for a in range(4)) for b in range(4))
            mg = gw.mean(1, keepdim=True)
            bg = ((gw - mg) ** 2).sum(1, keepdim=True).sqrt()
            gn = (gw - mg) / bg
            z[live] = (fn[live] * gn).sum(1)
            b = ((fn[live] - gn).unsqueeze(1) * J[live]).sum(2) * bf[live]
            norm = torch.linalg.vector_norm(b, dim=1)
            if it == 1:
                first[live] = norm
            f1 = first[live]
            done = (torch.where(f1 > tol, norm / f1, torch.zeros_like(norm)) < tol) | (norm < tol)
            code[live[done]] = it
            live, p, b = live[~done], p[~done], b[~done]
            if live.numel() == 0 or it == 101:
                break
            q = -torch.linalg.solve(H[live], b.unsqueeze(2))[:, :, 0]
            W = torch.zeros((live.numel(), 3, 3), **F64)
            D = torch.zeros_like(W)
            for m, r in ((W, p), (D, q)):
                m[:, 0, 0], m[:, 0, 1], m[:, 0, 2] = 1 + r[:, 0], r[:, 2], r[:, 4]
                m[:, 1, 0], m[:, 1, 1], m[:, 1, 2] = r[:, 1], 1 + r[:, 3], r[:, 5]
                m[:, 2, 2] = 1
            W = W @ torch.linalg.inv(D)
            P[live] = torch.stack([W[:, 0, 0] - 1, W[:, 1, 0], W[:, 0, 1], W[:, 1, 1] - 1, W[:, 0, 2], W[:, 1, 2]], 1)
        code[code > 100] = 101
        U[at], F[at], conv[at], zn[at] = P[:, 4:], P[:, :4], code, z
        H21[:, at] = torch.stack([H[:, i, j] for i, j in tri])
    r = {"U": U.reshape(-1), "F": F.reshape(-1), "conv": None}
    if want_H:
        r["H"] = H21.reshape(-1)
    return r, zn


def _phi64(s):
    """findpeak's peak value (ny x nx, column-major) of each grid subset's normalised
    cross-correlation over its border-clamped search region."""
    M, N, w, r = s["M"], s["N"], s["w"], s["search"]
    ref, deff = (torch.from_numpy(x.ravel(order="F").copy()).cuda() if isinstance(x, np.ndarray) else x
                 for x in (s["ref"], s["deff"]))
    f, g = _normal64(ref, M, N), _normal64(deff, M, N)
    nodes, nx, ny = _grid(M, N, s["w"], s["step"])
    st = (_dev(nodes) - w / 2).long()  # (2, n): the windows' first pixels, 1-based
    K, W1 = w + 3 + 2 * r, w + 1
    P = 1 << (K - 1).bit_length() if K > 96 else K
    size = torch.tensor([[M], [N]], device="cuda")
    lo = torch.where(st - r < 1, st - 1, torch.full_like(st, r))
    hi = torch.where(st + w + r > size, size - st - w - 1, torch.full_like(st, r)).clamp_min(0)
    k, kw = torch.arange(K, device="cuda"), torch.arange(W1, device="cuda")
    phi = torch.empty(nodes.shape[1], **F64)
    for at in torch.arange(nodes.shape[1], device="cuda").split(max(1, 12_000_000 // (P * P))):
        def rows(ax):
            q = st[ax, at][:, None] - 1 - r - 1 + k
            keep = (q >= (st[ax, at] - lo[ax, at] - 1)[:, None]) & (q <= (st[ax, at] + w + hi[ax, at] - 1)[:, None])
            a = k[:-w] - (r - lo[ax, at])[:, None]
            crop = (a >= 0) & (a <= (lo[ax, at] + hi[ax, at] + 2)[:, None])
            return q.clamp(0, (M, N)[ax] - 1), keep, crop
        qx, okx, cx = rows(0)
        qy, oky, cy = rows(1)
        D = g[qx[:, :, None], qy[:, None, :]] * (okx[:, :, None] & oky[:, None, :])
        T = f[st[0, at][:, None, None] - 1 + kw[:, None], st[1, at][:, None, None] - 1 + kw]
        T = T - T.mean((1, 2), keepdim=True)
        num = torch.fft.irfft2(torch.fft.rfft2(D, (P, P)) * torch.fft.rfft2(T, (P, P)).conj(), (P, P))[:, :K - w, :K - w]

        def box(x):
            x = torch.nn.functional.pad(x.cumsum(1).cumsum(2), (1, 0, 1, 0))
            return x[:, W1:, W1:] - x[:, :-W1, W1:] - x[:, W1:, :-W1] + x[:, :-W1, :-W1]
        den = (box(D * D) - box(D) ** 2 / W1 ** 2).clamp_min(0).sqrt() * T.square().sum((1, 2)).sqrt()[:, None, None]
        keep = cx[:, :, None] & cy[:, None, :]
        ncc = torch.where(keep & (den > 1e-6), num / den, torch.zeros_like(num))
        best = torch.where(keep, ncc, torch.full_like(ncc, -2)).transpose(1, 2).reshape(at.numel(), -1).argmax(1)
        pb, pa = best // (K - w), best % (K - w)
        pad = torch.nn.functional.pad(ncc, (1, 1, 1, 1))
        i = torch.arange(at.numel(), device="cuda")
        c = {(b, a): pad[i, pa + 1 + a, pb + 1 + b] for a in (-1, 0, 1) for b in (-1, 0, 1)}  # (column, row) offsets
        S, Sx, Sy = sum(c.values()), sum(q[0] * v for q, v in c.items()), sum(q[1] * v for q, v in c.items())
        S2x, S2y = sum(v for q, v in c.items() if q[0]), sum(v for q, v in c.items() if q[1])
        A2, A3, A5, A6 = Sx / 6, Sy / 6, S2x / 2 - S / 3, S2y / 2 - S / 3
        A1, A4 = (5 * S - 3 * (S2x + S2y)) / 9, (c[1, 1] - c[1, -1] - c[-1, 1] + c[-1, -1]) / 4
        dd = A4 * A4 - 4 * A5 * A6
        xo, yo = (-A3 * A4 + 2 * A6 * A2) / dd, -(A4 * A2 - 2 * A5 * A3) / dd
        inner = (cx[i, pa] & cx[i, (pa - 1).clamp_min(0)] & cx[i, (pa + 1).clamp_max(K - w - 1)] & (pa > 0)
                 & (pa < K - w - 1) & cy[i, (pb - 1).clamp_min(0)] & cy[i, (pb + 1).clamp_max(K - w - 1)] & (pb > 0)
                 & (pb < K - w - 1) & (xo.abs() <= 1) & (yo.abs() <= 1))
        xo, yo = torch.round(1000 * xo) / 1000, torch.round(1000 * yo) / 1000
        phi[at] = torch.where(inner, A1 + A2 * xo + A3 * yo + A4 * xo * yo + A5 * xo * xo + A6 * yo * yo, c[0, 0])
    return phi.view(ny, nx).t().reshape(-1)


def _global64(case, s):
    """The global step's system assembled element by element and solved by conjugate gradients
    until the residual no longer falls."""
    _, crd, E, dirichlet = _plate_mesh(case["M"], case["N"], case["w"], case["step"], case["hole"])
    n, E = crd.shape[0], _dev(E.astype(np.int64))
    on = (E > 0).double()
    xy = torch.cat([_dev(crd), torch.zeros((1, 2), **F64)])[torch.where(E > 0, E - 1, torch.full_like(E, n))]
    d5, d6, d7, d8 = on[:, 4:].t()
    g = {2: ([-3 ** -0.5, 3 ** -0.5], [1.0, 1.0]), 3: ([0.0, 0.6 ** 0.5, -0.6 ** 0.5], [8 / 9, 5 / 9, 5 / 9])}[case["order"]]
    sg = np.sign
    idx = (E - 1).clamp_min(0)
    ue, Fe = s["U"].view(n, 2)[idx] * on[..., None], s["F"].view(n, 4)[idx]
    Ke = torch.zeros((E.shape[0], 8, 8), **F64)
    be = torch.zeros((E.shape[0], 8, 2), **F64)
    for a, wa in zip(*g):
        for e, we in zip(*g):
            n5, n6 = d5 * 0.5 * (1 + a) * (1 - abs(e)), d6 * 0.5 * (1 + e) * (1 - abs(a))
            n7, n8 = d7 * 0.5 * (1 - a) * (1 - abs(e)), d8 * 0.5 * (1 - e) * (1 - abs(a))
            k5, e5 = d5 * 0.5 * (1 - abs(e)), d5 * 0.5 * (1 + a) * sg(-e)
            k6, e6 = d6 * 0.5 * (1 + e) * sg(-a), d6 * 0.5 * (1 - abs(a))
            k7, e7 = -d7 * 0.5 * (1 - abs(e)), d7 * 0.5 * (1 - a) * sg(-e)
            k8, e8 = d8 * 0.5 * (1 - e) * sg(-a), -d8 * 0.5 * (1 - abs(a))
            Nn = torch.stack([(1 - a) * (1 - e) * 0.25 - 0.5 * (n7 + n8), (1 + a) * (1 - e) * 0.25 - 0.5 * (n8 + n5),
                              (1 + a) * (1 + e) * 0.25 - 0.5 * (n5 + n6), (1 - a) * (1 + e) * 0.25 - 0.5 * (n6 + n7),
                              n5, n6, n7, n8], 1)
            dk = torch.stack([-0.25 * (1 - e) - 0.5 * (k7 + k8), 0.25 * (1 - e) - 0.5 * (k8 + k5),
                              0.25 * (1 + e) - 0.5 * (k5 + k6), -0.25 * (1 + e) - 0.5 * (k6 + k7), k5, k6, k7, k8], 1)
            de = torch.stack([-0.25 * (1 - a) - 0.5 * (e7 + e8), -0.25 * (1 + a) - 0.5 * (e8 + e5),
                              0.25 * (1 + a) - 0.5 * (e5 + e6), 0.25 * (1 - a) - 0.5 * (e6 + e7), e5, e6, e7, e8], 1)
            j = torch.stack([(dk[..., None] * xy).sum(1), (de[..., None] * xy).sum(1)], 1)
            det = torch.linalg.det(j)
            D = torch.linalg.solve(j, torch.stack([dk, de], 1))  # (elements, 2, 8)
            Dn = D.transpose(1, 2)
            jw = (det * wa * we)[:, None, None]
            NN = Nn[:, :, None] * Nn[:, None, :]
            Ke += jw * (s["beta"] * Dn @ D + s["mu"] * NN)
            be += jw * (s["mu"] * NN @ ue + s["beta"] * torch.stack(
                [Dn[..., 0] * Fe[..., 0] + Dn[..., 1] * Fe[..., 2], Dn[..., 0] * Fe[..., 1] + Dn[..., 1] * Fe[..., 3]], 2))
    Ke, be = Ke * on[:, :, None] * on[:, None, :], be * on[..., None]
    flat = idx.reshape(-1)

    def gather(x):
        return torch.zeros((n, x.shape[-1]), **F64).index_add_(0, flat, x.reshape(-1, x.shape[-1]))

    free = torch.zeros(n, dtype=torch.bool, device="cuda")
    free[torch.unique(E)[1:] - 1] = True
    x = torch.zeros((n, 2), **F64)
    dn = _dev(np.unique(dirichlet).astype(np.int64) - 1)
    free[dn] = False
    x[dn] = s["U"].view(n, 2)[dn]
    free = free[:, None].double()
    diag = gather(torch.diagonal(Ke, dim1=1, dim2=2)[..., None]) + (1 - free)

    def K(v):
        return gather(Ke @ (v[idx] * on[..., None]))

    r = (gather(be) - K(x)) * free
    z = r / diag
    p, rz, r0 = z.clone(), (r * z).sum(), float((r * r).sum())
    for _ in range(2000):
        q = K(p) * free
        al = rz / (p * q).sum()
        x, r = x + al * p, r - al * q
        if float((r * r).sum()) <= 1e-30 * r0:
            break
        z = r / diag
        rn = (r * z).sum()
        p, rz = z + rn / rz * p, rn
    return x.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("plate", "subpb1", "learned", "train"):
        # masked windows follow flood-filled regions, the network rounds its activations to 16
        # bits: their outputs have no 64-bit value of their own
        return None
    s = prepare(case, seed)
    if kind in ("pass", "search"):
        # u and v are rounded to 1e-3 px inside findpeak and IC-GN starts from them; the peak
        # value is the computed number
        phi = _phi64(s)
        none = ("u", "v", "U", "F", "conv", "H") if kind == "pass" else ("u", "v", "U0")
        return {"phi": phi.view(s["nx"], s["ny"]).t().contiguous() if case.get("host") else phi, **dict.fromkeys(none)}
    if kind == "subpb2":
        return {"U": _global64(case, s)}
    if kind == "icgn":
        got = _icgn64(s["ref"], s["deff"], s["M"], s["N"], s["coords"], s["U0"], s["F0"], s["w"], s["tol"], s["quad"], True)
        if got is None:
            return None
        r, zn = got
        return dict(r, zncc=zn) if s["F0"] is not None else r
    cams = []
    for cam in s["cams"]:
        got = _icgn64(cam["ref"], cam["deff"], s["M"], s["N"], cam["coords"], cam["U0"], None, s["w"], s["tol"], True, False)
        if got is None:
            return None
        cams.append(got[0])
    p = torch.cat([cam["coords"] + r["U"].view(-1, 2).t() for cam, r in zip(s["cams"], cams)], 0).t()
    K, R, T = (_dev(s[k]) for k in ("K", "R", "T"))
    PL = torch.cat([K, torch.zeros((3, 1), **F64)], 1)
    PR = K @ torch.cat([R, T[:, None]], 1)
    xyz, err = torch.full((s["n"], 3), math.nan, **F64), torch.full((s["n"],), math.nan, **F64)
    ok = torch.isfinite(p).all(1)
    p = p[ok]
    m = torch.stack([p[:, :1] * PL[2] - PL[0], p[:, 1:2] * PL[2] - PL[1], p[:, 2:3] * PR[2] - PR[0],
                     p[:, 3:] * PR[2] - PR[1]], 1).cpu().numpy()
    X = _dev(np.linalg.svd(m)[2][:, 3])
    X = X / X[:, 3:]
    xyz[ok] = X[:, :3]
    l, r = X @ PL.t(), X @ PR.t()
    err[ok] = (torch.hypot(l[:, 0] / l[:, 2] - p[:, 0], l[:, 1] / l[:, 2] - p[:, 1])
               + torch.hypot(r[:, 0] / r[:, 2] - p[:, 2], r[:, 1] / r[:, 2] - p[:, 3])) / 2
    return {"xyz": xyz.t().reshape(-1), "err": err, "cams": cams}
