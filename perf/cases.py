"""The work that users of this framework have it do, as cases that can be timed.

Each case is one call sequence of a user's program through the public entry
points (windtunnel.AeroEngine / AeroBatch / Viewer, the warm-start network of
windtunnel.surrogate and its operators in windtunnel.net):

    edit    a setup change in the interactive viewer: re-voxelize the car into the
            running flow, one frame, the force readout and the streamline pass
    loop    the headless loop: frames of 8 collide-stream steps and 2 heat passes
            with a force readout each, then the coarse field
    run     a study's chunk of collide-stream steps: per-step force history and
            the coarse field (what windtunnel.warmstart.run_cases does per chunk)
    box     an external box mesh given as flags, advanced from a perturbed state,
            and the whole field read back
    batch   the batched aero map: lattices of uneven sizes in one launch per step
    viewer  a whole viewer frame, read back as an image
    predict the warm-start network's field for new cars (committed weights)
    train   one training step of that network
    conv    one convolution layer of such a network, forward and backward
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "f1-wind-tunnel_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

WEIGHTS = os.path.join(PKG, "windtunnel", "data", "warmstart_f1.npz")
SIM = dict(u_in=0.08, tau0=0.51, smag=0.1, sponge_cells=16.0)  # the benchmark workloads' parameters
TUNNEL_X = 11.52    # length of the half tunnel the F1 workloads span, m
GRID = (64, 24, 24)  # x, y, z of the network's padded grid
COARSE = (64, 24, 20)


# ------------------------------------------------------------------------- cases
def listed():
    return [
        # the reference's lowest quality: the interactive loop's smallest lattice, where launches and latency count
        dict(name="edit_low", kind="edit", nx=168, ny=50, nz=38),
        # the headless loop at the reference's medium quality, default engine settings
        dict(name="loop_medium", kind="loop", nx=232, ny=68, nz=52, storage="f32", frames=16),
        # the benchmark's lattice (generic F1 at 4.5 cm), frames with a force readout each
        dict(name="loop_f1", kind="loop", nx=256, ny=96, nz=80, storage="f32", frames=16),
        # the same lattice in half-precision storage, as the study runs it
        dict(name="run_f1_f16", kind="run", nx=256, ny=96, nz=80, storage="f16", steps=256),
        # the precision-sweep lattice (2.25 cm), the largest of the repository
        dict(name="run_large_f16", kind="run", nx=512, ny=192, nz=160, storage="f16", steps=64),
        # the plain FP32 cube configuration: 1000 steps, then the field
        dict(name="box_cube", kind="box", nx=128, ny=64, nz=64, edge=22, storage="f32", steps=1000),
        # rows that no warp or block divides, in the other 16-bit storage
        dict(name="box_ragged_bf16", kind="box", nx=203, ny=77, nz=61, edge=25, storage="bf16", steps=250),
        # a quarter of the aero map: lattices of uneven sizes advanced together
        dict(name="batch_aeromap", kind="batch", count=8, nx_min=128, nx_max=256, storage="f16", steps=64),
        # the headless check's hero shot as a frame of the viewer
        dict(name="viewer_hero", kind="viewer", width=1280, height=720, flow="streamlines"),
        # the warm start of one car: latency of the whole network
        dict(name="predict_one", kind="predict", batch=1),
        # the training step that the network was made with
        dict(name="train_16", kind="train", batch=16),
        # one layer on an odd grid with odd channel counts
        dict(name="conv_ragged", kind="conv", batch=3, d=11, h=21, w=37, cin=40, cout=64, taps=27),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("edit", "loop", "run", "box", "batch", "viewer", "predict", "train", "conv"))
    if kind == "edit":
        nx = rng.randint(120, 296)
        return dict(kind=kind, nx=nx, ny=max(30, nx * 3 // 10 + rng.randint(-3, 3)), nz=max(24, nx * 9 // 40 + rng.randint(-3, 3)))
    if kind == "loop":
        nx = _log_int(rng, 96, 384)
        return dict(kind=kind, nx=nx, ny=max(24, nx * 3 // 8 + rng.randint(-4, 4)), nz=max(20, nx * 5 // 16 + rng.randint(-4, 4)),
                    storage=rng.choice(("f32", "f32", "f16", "bf16")), frames=rng.randint(2, 24))
    if kind == "run":
        nx = _log_int(rng, 96, 512)
        return dict(kind=kind, nx=nx, ny=max(24, nx * 3 // 8 + rng.randint(-4, 0)), nz=max(20, nx * 5 // 16 + rng.randint(-4, 0)),
                    storage=rng.choice(("f32", "f16", "bf16")), steps=2 * rng.randint(8, 32))
    if kind == "box":
        nx = rng.randint(64, 224)
        ny, nz = rng.randint(32, 96), rng.randint(24, 80)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, edge=rng.randint(5, min(26, ny // 2, nz // 2)),
                    storage=rng.choice(("f32", "f16", "bf16")), steps=2 * rng.randint(4, 200))
    if kind == "batch":
        lo = rng.randint(96, 160)
        return dict(kind=kind, count=rng.randint(2, 12), nx_min=lo, nx_max=rng.randint(lo, 256),
                    storage=rng.choice(("f32", "f16", "bf16")), steps=2 * rng.randint(4, 48))
    if kind == "viewer":
        h = rng.randint(180, 720)
        return dict(kind=kind, width=h * 16 // 9 + rng.randint(0, 7), height=h,
                    flow=rng.choice(("streamlines", "smoke", "vortices", "none")))
    if kind == "predict":
        return dict(kind=kind, batch=rng.randint(2, 50))
    if kind == "train":
        return dict(kind=kind, batch=rng.randint(2, 15))
    return dict(kind=kind, batch=rng.randint(1, 16), d=rng.randint(3, 24), h=rng.randint(3, 24), w=rng.randint(5, 64),
                cin=8 * rng.randint(1, 16), cout=rng.choice((8, 16, 32, 64, 128)), taps=rng.choice((27, 27, 27, 1)))


# --------------------------------------------------------------------- the inputs
def _f1_engine(case, seed):
    import windtunnel as wt
    dims = (case["nx"], case["ny"], case["nz"])
    e = wt.AeroEngine(dims=dims, origin=(wt.ORIGIN_X, 0.0, 0.0), h=TUNNEL_X / dims[0],
                      sim=wt.make_sim(storage=case["storage"], **SIM))
    e.set_shape_raw(wt.config_f1_shape(seed))
    return e


def _setup(rng):
    """A car setup as the viewer's panels give it: wing angles and ride heights."""
    from windtunnel import ShapeKind, ShapeParams
    return ShapeParams(kind=ShapeKind.F1, frontFlapDeg=float(rng.uniform(-4, 8)), rearFlapDeg=float(rng.uniform(-6, 8)),
                       rideH=float(rng.uniform(0.06, 0.12)), rearRideH=float(rng.uniform(0.08, 0.16)))


def _flow_view(flow):
    from windtunnel.viewer import FlowMode, ViewParams
    return ViewParams(flow_mode={"streamlines": FlowMode.Streamlines, "smoke": FlowMode.Smoke,
                                 "vortices": FlowMode.Vortices, "none": FlowMode.None_}[flow])


def _cube_flags(case):
    """Flags of a cube of `edge` cells on the floor, cut by the symmetry plane, about a third of the way in."""
    nx, ny, nz, e = case["nx"], case["ny"], case["nz"], case["edge"]
    solid = np.zeros((nz, ny, nx), np.uint32)
    x0 = max(4, nx * 5 // 16 - e // 2)
    solid[: (e + 1) // 2, :e, x0:x0 + e] = 1
    return solid


_C = np.array([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [-1, -1, 0],
               [1, -1, 0], [-1, 1, 0], [1, 0, 1], [-1, 0, -1], [1, 0, -1], [-1, 0, 1], [0, 1, 1], [0, -1, -1],
               [0, 1, -1], [0, -1, 1]])
_W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


def _start_populations(case, seed):
    """Inlet equilibrium with a small random disturbance: float32 [19, nz, ny, nx]."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = SIM["u_in"]
    cu = _C[:, 0] * u
    feq = torch.tensor(_W * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * u * u), dtype=torch.float32, device="cuda")
    noise = torch.randn((19, case["nz"], case["ny"], case["nx"]), generator=g, device="cuda")
    return (feq.view(19, 1, 1, 1) * (1 + 1e-3 * noise)).cpu().numpy()


def _network_input(batch, seed):
    """[batch, 24, 24, 64, 8] BF16: tanh of a distance to a car-sized body per sample, then the six scalar features."""
    r = np.random.default_rng(seed)
    x, y, z = GRID
    gx, gy, gz = np.meshgrid((np.arange(x) + 0.5) * 0.18 - 2.4, (np.arange(y) + 0.5) * 0.18, (np.arange(z) + 0.5) * 0.18, indexing="ij")
    out = np.zeros((batch, z, y, x, 8), np.float32)
    mask = np.zeros((batch, z, y, x), np.float32)
    for b in range(batch):
        c, s = r.uniform((2.3, 0.3, -0.1), (2.9, 0.6, 0.1)), r.uniform((2.3, 0.3, 0.6), (2.7, 0.5, 0.95))
        q = np.stack([np.abs(gx - c[0]) - s[0], np.abs(gy - c[1]) - s[1], np.abs(gz - c[2]) - s[2]])
        d = np.linalg.norm(np.maximum(q, 0), axis=0) + np.minimum(q.max(0), 0)
        d = np.transpose(d, (2, 1, 0))
        out[b, ..., 0] = 1.0
        out[b, :20, ..., 0] = np.tanh(d[:20] / 0.3)
        out[b, ..., 1:7] = r.uniform(-1, 1, 6)
        mask[b, :20] = d[:20] > 0
    return torch.tensor(out, device="cuda").to(torch.bfloat16), torch.tensor(mask, device="cuda")


def _network(seed=0):
    from windtunnel.surrogate import Surrogate
    m = Surrogate(seed=seed)
    with np.load(WEIGHTS) as z:
        m.load_state({k: z[k] for k in z.files})
    return m


def _conv_tensors(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = (case["batch"], case["d"], case["h"], case["w"])
    k = case["taps"] * case["cin"]
    r = lambda *shape: torch.randn(shape, generator=g, device="cuda")  # noqa: E731
    x = torch.relu(r(*s, case["cin"])).to(torch.bfloat16)
    w = (r(case["cout"], case["taps"], case["cin"]) * (2.0 / k) ** 0.5).to(torch.bfloat16)
    b = r(case["cout"]) * 0.1
    dy = (r(*s, case["cout"]) * 1e-3).to(torch.bfloat16)
    return x, w, b, dy


def prepare(case, seed):
    import windtunnel as wt
    kind = case["kind"]
    if kind == "edit":
        rng = np.random.default_rng(seed)
        e = wt.AeroEngine(dims=(case["nx"], case["ny"], case["nz"]))
        from windtunnel.viewer import Viewer
        v = Viewer(e, 64, 36, particles=1)
        setups = [_setup(rng) for _ in range(4)]
        e.set_shape(setups[0])
        e.reset()
        for _ in range(4):
            e.frame(8)
        e.read_forces()
        return dict(kind=kind, e=e, viewer=v, setups=setups, next=1)
    if kind in ("loop", "run"):
        e = _f1_engine(case, seed)
        e.frame(8)
        e.read_forces_raw()
        return dict(case, e=e)
    if kind == "box":
        dims = (case["nx"], case["ny"], case["nz"])
        e = wt.AeroEngine(dims=dims, origin=(0.0, 0.0, 0.0), h=0.045, sim=wt.make_sim(storage=case["storage"], **SIM))
        e.set_solid(_cube_flags(case), np.zeros(e.n, np.float32))
        e.write_state(f=_start_populations(case, seed))
        return dict(case, e=e)
    if kind == "batch":
        grids = []
        for k in range(case["count"]):
            nx = case["nx_min"] + (case["nx_max"] - case["nx_min"]) * k // max(1, case["count"] - 1)
            grids.append(((nx, max(24, nx * 3 // 8), max(20, nx * 5 // 16)), (wt.ORIGIN_X, 0.0, 0.0), TUNNEL_X / nx))
        b = wt.AeroBatch(grids, wt.make_sim(storage=case["storage"], **SIM))
        rng = np.random.default_rng(seed)
        for e in b.lattices:
            e.set_shape_raw(wt.config_f1_shape(seed, ride=float(rng.uniform(0.01, 0.06)), rear_ride=float(rng.uniform(0.01, 0.06))))
        return dict(case, b=b)
    if kind == "viewer":
        from windtunnel.viewer import Viewer, orbit
        rng = np.random.default_rng(seed)
        e = wt.AeroEngine("medium")
        v = Viewer(e, case["width"], case["height"])
        v.set_view(_flow_view(case["flow"]))
        e.set_shape(_setup(rng))
        e.reset()
        v.reset_particles()
        e.step(160, 2, 4.0)
        cam = orbit(dict(yaw=float(rng.uniform(0.4, 2.7)), pitch=float(rng.uniform(0.1, 0.35)),
                         distance=float(rng.uniform(5.5, 8.0))), case["width"] / case["height"])
        return dict(kind=kind, e=e, viewer=v, cam=cam)
    if kind == "predict":
        return dict(kind=kind, m=_network(), x=_network_input(case["batch"], seed)[0])
    if kind == "train":
        x, mask = _network_input(case["batch"], seed)
        g = torch.Generator(device="cuda").manual_seed(seed)
        target = torch.randn((*x.shape[:4], 4), generator=g, device="cuda") * 0.1
        return dict(kind=kind, m=_network(), x=x, target=target, mask=mask)
    from windtunnel.net import Ops
    ops = Ops()
    x, w, b, dy = _conv_tensors(case, seed)
    dev = dict(device="cuda")
    cin, cout, taps = case["cin"], case["cout"], case["taps"]
    ws = torch.empty(max(1, ops.workspace_bytes(x.shape, cin, cout, taps) // 4), **dev)
    return dict(kind=kind, ops=ops, x=x, w=w, b=b, dy=dy, taps=taps, ws=ws,
                wt=torch.empty((cin, taps, cout), dtype=torch.bfloat16, **dev),
                y=torch.empty((*x.shape[:4], cout), dtype=torch.bfloat16, **dev),
                dx=torch.empty((*x.shape[:4], cin), **dev), dw=torch.empty((cout, taps, cin), **dev),
                db=torch.empty(cout, **dev))


# ------------------------------------------------------------------------ one pass
def _forces(f):
    return [np.array(f.raw[:], np.int32), np.array(f.sum[:], np.float64), float(f.mass), int(f.guarded)]


def run(state):
    kind = state["kind"]
    if kind == "edit":
        e = state["e"]
        e.set_shape(state["setups"][state["next"] % 4])
        state["next"] += 1
        e.frame(8)
        lines = e.streamlines(state["viewer"].stream_params(), state["viewer"].view_uniform())
        f = e.read_forces()
        return dict(lines=lines, raw=f.raw, sum64=f.sum64, drag=f.dragN, down=f.downforceN, mass=f.mass)
    if kind == "loop":  # forces of frame k are collected while frame k + 1 runs, as the engine maps them
        e, readings, ticket = state["e"], [], None
        for _ in range(state["frames"]):
            e.frame(8)
            queued = e.read_forces_async()
            if ticket is not None:
                readings.append(_forces(e.collect_forces(ticket)))
            ticket = queued
        readings.append(_forces(e.collect_forces(ticket)))
        return dict(raw=np.stack([r[0] for r in readings]), sum64=np.stack([r[1] for r in readings]),
                    mass=np.array([r[2] for r in readings]), coarse=e.read_coarse(*_coarse(e)))
    if kind == "run":
        e = state["e"]
        e.step(state["steps"])
        return dict(history=e.force_history(state["steps"]), coarse=e.read_coarse(*_coarse(e)))
    if kind == "box":
        e = state["e"]
        e.step(state["steps"])
        d = e.debug_read()
        return dict(fields=d["fields"], solid=d["solid"].astype(np.int32), history=e.force_history(state["steps"]))
    if kind == "batch":
        b = state["b"]
        b.step(state["steps"])
        return [dict(history=e.force_history(state["steps"]), coarse=e.read_coarse(*_coarse(e))) for e in b.lattices]
    if kind == "viewer":
        state["viewer"].frame(state["cam"], 8)
        return state["viewer"].image()
    if kind == "predict":
        return state["m"].forward(state["x"])
    if kind == "train":
        m = state["m"]
        loss, _ = m.train_step(state["x"], state["target"], state["mask"], 2e-3)
        return dict(loss=loss, weights={n: [c.w, c.b] for n, c in m.L.items()}, grads={n: [c.gw, c.gb] for n, c in m.L.items()})
    o = state["ops"]
    o.weight_transpose(state["w"], state["wt"])
    o.conv_forward(state["x"], state["w"], state["b"], state["y"], True)
    o.conv_backward_data(state["dy"], state["wt"], state["dx"], state["w"].shape[2], state["w"].shape[0], state["taps"])
    o.conv_backward_weight(state["x"], state["dy"], state["dw"], state["ws"], state["taps"])
    o.bias_grad(state["dy"], state["db"])
    return dict(y=state["y"], dx=state["dx"], dw=state["dw"], db=state["db"])


def _coarse(e):
    return tuple(min(c, d) for c, d in zip(COARSE, e.dims))


# ----------------------------------------------------------------- what it cannot do without
def _step_bytes(storage):
    return 19 * 2 * (4 if storage == "f32" else 2) + 4


HEAT_BYTES = 28
# operations of one collide-stream update (moments, equilibria, stress, relaxation)
STEP_FLOPS = 420


def _layers(b):
    d = {0: 24 * 24 * 64, 1: 12 * 12 * 32, 2: 6 * 6 * 16, 3: 3 * 3 * 8}
    chain = [(0, 8, 16), (0, 16, 16), (1, 16, 32), (1, 32, 32), (2, 32, 64), (2, 64, 64), (3, 64, 128), (3, 128, 128),
             (2, 128, 64), (2, 64, 64), (1, 64, 32), (1, 32, 32), (0, 32, 16), (0, 16, 16)]
    return [(b * d[lv], ci, co, 27) for lv, ci, co in chain] + [(b * d[0], 16, 8, 1)]


def work(case):
    kind = case["kind"]
    if kind == "conv":
        m = case["batch"] * case["d"] * case["h"] * case["w"]
        k = case["taps"] * case["cin"] * case["cout"]
        return dict(bytes=m * (2 * case["cin"] + 2 * 2 * case["cout"] + 4 * case["cin"]) + k * (2 + 4), flops=6.0 * m * k)
    if kind in ("predict", "train"):
        layers = _layers(case["batch"])
        macs = sum(m * ci * co * t for m, ci, co, t in layers)
        par = sum(ci * co * t + co for _, ci, co, t in layers)
        io = case["batch"] * 24 * 24 * 64
        if kind == "predict":
            return dict(bytes=io * 32 + par * 2, flops=2.0 * macs)
        first = layers[0][0] * layers[0][1] * layers[0][2] * layers[0][3]
        return dict(bytes=io * (16 + 16 + 4) + par * (4 * 7 + 2), flops=2.0 * (3 * macs - first))
    if kind == "viewer":  # one medium frame of 8 steps and 2 heat passes, then the render targets once each
        n, px = 232 * 68 * 52, case["width"] * case["height"]
        return dict(bytes=n * (8 * _step_bytes("f32") + 2 * HEAT_BYTES) + px * (8 * 4 + 4 + 4), flops=8.0 * n * STEP_FLOPS)
    if kind == "edit":
        n = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=n * (8 * _step_bytes("f32") + 2 * HEAT_BYTES + 9) + 90 * 360 * 16, flops=8.0 * n * STEP_FLOPS)
    if kind == "batch":
        n = 0
        for k in range(case["count"]):
            nx = case["nx_min"] + (case["nx_max"] - case["nx_min"]) * k // max(1, case["count"] - 1)
            n += nx * max(24, nx * 3 // 8) * max(20, nx * 5 // 16)
    else:
        n = case["nx"] * case["ny"] * case["nz"]
    steps = 8 * case["frames"] if kind == "loop" else case["steps"]
    heat = 2 * case["frames"] * HEAT_BYTES if kind == "loop" else 0
    return dict(bytes=n * (steps * _step_bytes(case["storage"]) + heat + 16), flops=float(n) * steps * STEP_FLOPS)


# ------------------------------------------------------------------ the same in 64 bits
def _conv64(x, w):
    """[b, d, h, w, ci] by [co, taps, ci], zero padding, float64."""
    if w.shape[1] == 1:
        return x @ w[:, 0].T
    b, d, h, ww, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = torch.zeros((b, d, h, ww, w.shape[0]), dtype=torch.float64, device=x.device)
    for t in range(27):
        z, r, c = t // 9, t // 3 % 3, t % 3
        y += p[:, z:z + d, r:r + h, c:c + ww] @ w[:, t].T
    return y


def _exact_conv(case, seed):
    x, w, b, dy = (t.double() for t in _conv_tensors(case, seed))
    y = torch.relu(_conv64(x, w) + b)
    dx = _conv64(dy, w.flip(1).permute(2, 1, 0))
    if case["taps"] == 1:
        dw = torch.einsum("bdhwi,bdhwo->oi", x, dy)[:, None]
    else:
        _, d, h, ww, _ = x.shape
        p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        dw = torch.stack([dy.reshape(-1, dy.shape[-1]).T @ p[:, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + ww].reshape(-1, x.shape[-1])
                          for t in range(27)], 1)
    return dict(y=y, dx=dx, dw=dw, db=dy.sum((0, 1, 2, 3)))


def _exact_predict(case, seed):
    """The network without any rounding of its activations, on its BF16 weights."""
    a = _network_input(case["batch"], seed)[0].double()
    with np.load(WEIGHTS) as z:
        p = {k: torch.tensor(z[k], device="cuda") for k in z.files}

    def conv(n, v, act=True):
        v = _conv64(v, p[n + ".w"].to(torch.bfloat16).double()) + p[n + ".b"].double()
        return torch.relu(v) if act else v

    def pool(v):
        b, d, h, w, c = v.shape
        return v.view(b, d // 2, 2, h // 2, 2, w // 2, 2, c).mean((2, 4, 6))

    def up(v):
        return v.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    s0 = conv("e0b", conv("e0a", a))
    s1 = conv("e1b", conv("e1a", pool(s0)))
    s2 = conv("e2b", conv("e2a", pool(s1)))
    q = conv("e3b", conv("e3a", pool(s2)))
    q = conv("d2b", conv("d2a", up(q)) + s2)
    q = conv("d1b", conv("d1a", up(q)) + s1)
    q = conv("d0b", conv("d0a", up(q)) + s0)
    return conv("head", q, False)


def _exact_box(case, seed):
    """The half tunnel of the engine (D3Q19, regularized collision, Smagorinsky, boundary precedence inlet, outlet,
    moving floor, far field, symmetry plane / solid) around a cube, in float64."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev, u0 = "cuda", SIM["u_in"]
    solid = torch.tensor(_cube_flags(case).astype(bool), device=dev)
    f = torch.tensor(_start_populations(case, seed), device=dev).double()
    w = torch.tensor(_W, device=dev)
    cu = torch.tensor(_C[:, 0] * u0, device=dev, dtype=torch.float64)
    feq_in = w * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * u0 * u0)
    opp = [0] + [i + 1 if i & 1 else i - 1 for i in range(1, 19)]
    zmir = [int(np.flatnonzero((_C == c * (1, 1, -1)).all(1))[0]) for c in _C]
    xs = torch.arange(nx, device=dev, dtype=torch.float64)

    def smooth(lo, hi):
        t = ((xs - lo) / (hi - lo)).clamp(0, 1)
        return t * t * (3 - 2 * t)

    tau0 = SIM["tau0"] + 0.4 * smooth(nx - SIM["sponge_cells"], nx - 1) + 0.25 * (1 - smooth(0.0, 10.0))
    # belt speed under the floor cells: 0 next to the body's contact patch
    belt = torch.full((nz, nx), u0, device=dev, dtype=torch.float64)
    s = solid[:, 0]
    near = solid[:, 1].clone()
    near[:, :-2] |= s[:, 2:]
    near[:, 2:] |= s[:, :-2]
    near[:-1] |= s[1:]
    near[1:] |= s[:-1]
    belt[near] = 0.0
    pu = torch.zeros((3, nz, ny), device=dev, dtype=torch.float64)  # velocity of the outlet column
    pu[0] = u0
    ks2 = 18 * math.sqrt(2.0) * SIM["smag"] ** 2
    for _ in range(case["steps"]):
        g = torch.empty_like(f)
        g[0] = f[0]
        for i in range(1, 19):
            cx, cy, cz = (int(v) for v in _C[i])
            g[i] = torch.roll(f[i], (cz, cy, cx), (0, 1, 2))
            hit = torch.roll(solid, (cz, cy, cx), (0, 1, 2))
            if cz > 0:
                g[i, 0] = torch.roll(f[zmir[i], 0], (cy, cx), (0, 1))
                hit[0] = torch.roll(solid[0], (cy, cx), (0, 1))
            g[i] = torch.where(hit, f[opp[i]], g[i])
            if cy < 0:
                g[i, :, -1] = feq_in[i]
            if cz < 0:
                g[i, -1] = feq_in[i]
            if cy > 0:
                g[i, :, 0] = f[opp[i], :, 0] + 6 * w[i] * cx * belt
            if cx < 0:
                c = cx * pu[0] + cy * pu[1] + cz * pu[2]
                g[i, :, :, -1] = w[i] * (1 + 3 * c + 4.5 * c * c - 1.5 * (pu * pu).sum(0))
            if cx > 0:
                g[i, :, :, 0] = feq_in[i]
        rho = g.sum(0)
        C = torch.tensor(_C, device=dev, dtype=torch.float64)
        u = torch.einsum("ia,izyx->azyx", C, g) / rho
        uu = (u * u).sum(0)
        c = torch.einsum("ia,azyx->izyx", C, u)
        eq = w.view(19, 1, 1, 1) * rho * (1 + 3 * c + 4.5 * c * c - 1.5 * uu)
        ne = g - eq
        pi = torch.einsum("ia,ib,izyx->abzyx", C, C, ne)
        q = torch.sqrt((pi * pi).sum((0, 1)))
        tau = 0.5 * (tau0 + torch.sqrt(tau0 * tau0 + ks2 * q / rho))
        k = 4.5 * (1 - 1 / tau)
        qp = torch.einsum("ia,ib,abzyx->izyx", C, C, pi) - (pi[0, 0] + pi[1, 1] + pi[2, 2]) / 3
        f = eq + k * w.view(19, 1, 1, 1) * qp
        f = torch.where(solid, w.view(19, 1, 1, 1), f)
        pu = torch.where(solid[:, :, -1], pu, u[:, :, :, -1])
    fields = torch.cat([u, rho[None]])
    fields = torch.where(solid, torch.zeros_like(fields), fields)
    return dict(fields=fields.permute(1, 2, 3, 0).reshape(-1, 4), solid=None, history=None)


def exact(case, seed):
    if case["kind"] == "conv":
        return _exact_conv(case, seed)
    if case["kind"] == "predict":
        return _exact_predict(case, seed)
    if case["kind"] == "box" and case["nx"] * case["ny"] * case["nz"] * case["steps"] < 6e8:
        return _exact_box(case, seed)
    return None  # a car's flags come from its distance field, an image from the shaders: no plain restatement
