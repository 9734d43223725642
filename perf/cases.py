"""The calls that users of this framework make, as cases to be timed.

A case is a dict of plain values; `kind` says which entry points it goes through:

  run      one pore image: warm start from given fields, time steps with the
           residual of every step (Solver.run, the executable's loop), its
           observables and fields
  advance  one pore image: time steps without residual (Solver.advance_graph,
           the loop of a run to steady state), fields
  batch    several images stepped together (Batch.advance: training data), fields
  pore     local pore size and Knudsen number of an image (host arrays in and out)
  conv     one convolution layer of the warm-start network, forward and backward
  train    one training step of the network: forward, loss, backward, Adam
  predict  the network's forward pass on one image

The solver's images follow from the case (so that a case always has the same
cells); the Knudsen number and the starting fields follow from the seed.
Fields come back in the precision in which the solver holds its state (FP32),
the density as its deviation from the initial density, as
surrogate.steady_targets gives them to the network.
"""
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from mantiis_gb300 import native, surrogate

# lattice updates per pixel of the image and coarse step for 1, 2 and 3 quadtree
# levels, at porosity 0.6 (seeded images, disk radii of 6 to 40 pixels in 1024^2; three levels: 3 to 10 in 256^2)
UPDATES_PER_PIXEL = {1: 0.6, 2: 0.41, 3: 1.1}
WIDTHS = (32, 64, 128, 256, 256)  # the network's default


def listed():
    return [
        # the smallest ordinary run: a 128^2 single-block image, radii 4-10,
        # where launches and latency count
        dict(name="run 128", kind="run", image=3528, n=128, levels=1, steps=100, rmin=4, rmax=10, porosity=0.65,
             kn=0.1, sim="transport", collision=2, wall=2),
        # an odd side and the other collision and wall models (MRT, MDBB)
        dict(name="run 301 mrt mdbb", kind="run", image=4329, n=301, levels=1, steps=100, rmin=4, rmax=14,
             porosity=0.6, kn=0.2, sim="transport", collision=1, wall=1),
        # the reference's own depth limit at 1024^2 with its residual in every
        # step, from a warm start
        dict(name="run 1024 2 levels", kind="run", image=4337, n=1024, levels=2, steps=100, rmin=6, rmax=40,
             porosity=0.6, kn=0.02, sim="transport", collision=2, wall=2),
        # a 1024^2 single block on its way to the steady state
        dict(name="advance 1024", kind="advance", image=3953, n=1024, levels=1, steps=400, rmin=6, rmax=40,
             porosity=0.6, kn=0.05, sim="transport", collision=2, wall=2),
        # the headline benchmark's batch of four 1024^2 images, at the depth at
        # which the reference's scheme has a steady state
        dict(name="batch 4x1024 2 levels", kind="batch", image=4683, sides="1024,1024,1024,1024", levels="2,2,2,2",
             steps=100, porosity=0.6, kn=0.015),
        # training data: sides and depths mixed
        dict(name="batch uneven", kind="batch", image=4203, sides="128,512,1024,256,512,128", levels="1,2,2,3,1,2",
             steps=100, porosity=0.6, kn=0.02),
        # Shan-Chen adsorption at 512^2 with the exponential pseudopotential
        dict(name="adsorption 512", kind="run", image=4275, n=512, levels=1, steps=200, rmin=6, rmax=40, porosity=0.6,
             kn=0.1, sim="adsorption", psi_form=1),
        # the reference's Peng-Robinson pseudopotential on a small odd side
        dict(name="adsorption 190 PR", kind="run", image=4471, n=190, levels=1, steps=100, rmin=4, rmax=12,
             porosity=0.65, kn=0.1, sim="adsorption", psi_form=0),
        # what a user runs once per image before the solver
        dict(name="pore 1024", kind="pore", n=1024, rmin=6, rmax=40, porosity=0.6),
        # a middle layer of the network at its training size
        dict(name="conv 64-128 32", kind="conv", batch=8, cin=64, cout=128, n=32),
        # a training step at the size train() and train_mixed() batch to
        dict(name="train 8x128", kind="train", batch=8, n=128),
        # the prediction for one large image
        dict(name="predict 512", kind="predict", batch=1, n=512),
    ]


def _log_int(rng, a, b):
    return int(round(float(np.exp(rng.uniform(np.log(a), np.log(b))))))


def draw(rng):
    kind = rng.choice(["run", "run", "adsorption", "advance", "batch", "pore", "conv", "train", "predict"])
    porosity = round(rng.uniform(0.5, 0.7), 3)
    image = rng.randrange(10000)
    if kind in ("run", "advance"):
        levels = rng.choice([1, 1, 2, 3])
        # multi-block: sides are powers of two; larger Kn, the plain MRT and three
        # levels of larger images diverge at the coarse/fine exchange
        n = _log_int(rng, 100, 1100) if levels == 1 else 256 if levels == 3 else rng.choice([256, 512, 1024])
        options = [(2, 2), (2, 2), (2, 1), (2, 0), (0, 2)] + ([(1, 2), (1, 0), (1, 1)] if levels == 1 else [])
        collision, wall = rng.choice(options)
        kn = _log_int(rng, 10, 120 if levels == 1 else 20) / 1000.0
        return dict(kind=kind, image=image, n=n, levels=levels, steps=rng.randint(60, 130 if kind == "run" else 400),
                    rmin=max(3, n // 128), rmax=max(8, n // 25), porosity=porosity, kn=kn,
                    sim="transport", collision=collision, wall=wall)
    if kind == "adsorption":
        n = _log_int(rng, 64, 600)
        return dict(kind="run", image=image, n=n, levels=1, steps=rng.randint(60, 200 if n > 250 else 100),
                    rmin=max(3, n // 100), rmax=max(8, n // 18), porosity=porosity, kn=0.1, sim="adsorption",
                    psi_form=rng.choice([0, 1]))
    if kind == "batch":
        sides = [rng.choice([128, 256, 512, 1024]) for _ in range(rng.randint(2, 5))]
        levels = [rng.randint(1, 3 if n == 256 else 2) for n in sides]
        return dict(kind="batch", image=image, sides=",".join(map(str, sides)), levels=",".join(map(str, levels)),
                    steps=rng.randint(50, 100),
                    porosity=porosity, kn=_log_int(rng, 10, 20) / 1000.0)
    if kind == "pore":
        n = _log_int(rng, 100, 1500)
        return dict(kind="pore", n=n, rmin=max(3, n // 170), rmax=max(8, n // 25), porosity=porosity)
    if kind == "conv":
        n = _log_int(rng, 8, 140)
        most = max(8, min(256, 8 * 128 * 128 * 32 // (8 * n * n)))
        return dict(kind="conv", batch=rng.randint(1, 8), cin=_log_int(rng, 2, most), cout=_log_int(rng, 3, most), n=n)
    if kind == "train":
        n = 16 * rng.randint(2, 9)
        return dict(kind="train", batch=rng.randint(1, max(1, 8 * 128 * 128 // (n * n))), n=n)
    return dict(kind="predict", batch=1, n=16 * _log_int(rng, 4, 64))


# ---- inputs


def _image(n, rmin, rmax, porosity, kn, image, levels):
    # void x edges: solid pixels on the x-periodic seam leak mass in the reference's scheme
    pore = native.generate_disks(n, rmin, rmax, porosity, image, open_x_edges=True)
    locpore, kn_unit = native.pore_properties_gpu(pore, 1.0, 1.0)
    void = pore == 1
    mfp = native.units()["mfp"]
    dx = float(mfp * kn_unit[void].mean() / kn)
    return dict(pore=pore, kn=np.where(void, kn_unit * mfp / dx, 0.0), locpore=locpore, dx=dx, levels=levels)


def _smooth(rng, x, y, n, amplitude):
    """A field of a few long waves at the cells' places."""
    v = np.zeros(x.shape)
    for _ in range(4):
        kx, ky = rng.integers(1, 5, 2)
        v += rng.standard_normal() * np.cos(2 * np.pi * (kx * x + ky * y) / n + rng.uniform(0, 2 * np.pi))
    return amplitude * v


def _pinned(count):
    return torch.empty(count, dtype=torch.float64).pin_memory().numpy()


def _start(s, rho0, rng, noise=None):
    """Starting fields of a solver's cells, in pinned memory: the reference's
    adsorption start (at rest, uniform density noise), else a warm start's."""
    x, y, _ = s.cell_positions()
    start = [_pinned(s.n_cells) for _ in range(3)]
    if noise is not None:
        start[0][:] = rho0 + rng.uniform(-noise, noise, s.n_cells)
        start[1][:] = 0.0
        start[2][:] = 0.0
    else:
        start[0][:] = rho0 * (1.0 + _smooth(rng, x, y, s.n, 1e-6))
        start[1][:] = 1e-6 + _smooth(rng, x, y, s.n, 3e-7)
        start[2][:] = _smooth(rng, x, y, s.n, 3e-7)
    return start


def _solver(case, seed):
    levels = case["levels"]
    rng = np.random.default_rng(seed)
    kn = case["kn"] * rng.uniform(0.8, 1.25)
    d = _image(case["n"], case["rmin"], case["rmax"], case["porosity"], kn, case["image"], levels)
    if case["sim"] == "adsorption":
        p = native.default_params(simulation=native.SIM_ADSORPTION, dx=d["dx"], psi_form=case["psi_form"])
        if case["psi_form"] == 1:
            p.g_ff, p.g_fs, p.rho_psi, p.rho_init, p.fbody = -4.5 / 18, -1.5, 0.5, 0.5, 0.0
    else:
        p = surrogate.solver_params(d, collision=case["collision"], wall=case["wall"])
    s = native.Solver(d["pore"], d["kn"], d["locpore"], p)
    rho0 = p.rho_init if p.rho_init > 0 else s.info["rho_in"]
    noise = None if case["sim"] == "transport" else 1e-3 * min(1.0, 2.0 * rho0)
    start = _start(s, rho0, rng, noise)
    return dict(solver=s, start=start, rho0=rho0, out={k: _pinned(s.n_cells) for k in ("rho", "ux", "uy")})


def _weights(cin, cout, gen):
    w = torch.randn((cout, cin, 3, 3), generator=gen, dtype=torch.float32, device="cuda") * (2.0 / (9 * cin)) ** 0.5
    return w, torch.randn(cout, generator=gen, dtype=torch.float32, device="cuda") * 0.05


def _net_shapes():
    w = WIDTHS
    return ([(2, w[0]), (w[0], w[0])] + [(w[i - 1], w[i]) for i in range(1, 5)] +
            [(w[i + 1], w[i]) for i in range(3, -1, -1)] + [(w[0], 3)])


def _net_inputs(case, seed):
    """Weights of every layer, and inputs, targets and masks shaped like the
    network's: a void mask, scaled log Kn on the void, asinh-scaled fields."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    layers = [_weights(ci, co, gen) for ci, co in _net_shapes()]
    b, n = case["batch"], case["n"]
    coarse = torch.randn((b, 1, max(2, n // 16), max(2, n // 16)), generator=gen, device="cuda")
    mask = (torch.nn.functional.interpolate(coarse, size=(n, n), mode="bilinear") > -0.2).float()
    kn = torch.randn((b, 1, n, n), generator=gen, device="cuda") * 0.2 - 0.5
    x = torch.cat([mask, kn * mask], 1).contiguous()
    target = (torch.randn((b, 3, n, n), generator=gen, device="cuda") * mask).contiguous()
    return layers, x, target, mask[:, 0].contiguous()


def _conv_inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    w, b = _weights(case["cin"], case["cout"], gen)
    n = case["n"]
    x = torch.relu(torch.randn((case["batch"], case["cin"], n, n), generator=gen, device="cuda"))
    dy = torch.randn((case["batch"], case["cout"], n, n), generator=gen, device="cuda") / (n * n)
    return w, b, x, dy


def _load(layer, w, b):
    layer.w.copy_(w)
    layer.b.copy_(b)
    layer.sync_bf16()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "advance"):
        state = _solver(case, seed)
        if kind == "advance":
            state["solver"].set_equilibrium(*state["start"])
        return dict(state, kind=kind, steps=case["steps"])
    if kind == "batch":
        sides = [int(v) for v in case["sides"].split(",")]
        levels = [int(v) for v in case["levels"].split(",")]

        rng = np.random.default_rng(seed)
        kn = case["kn"] * rng.uniform(0.8, 1.25, len(sides))

        def make(i):
            n = sides[i]
            return _image(n, max(3, n // 170), max(8, n // 25), case["porosity"], kn[i], case["image"] + i, levels[i])

        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as ex:
            images = list(ex.map(make, range(len(sides))))
        solvers = surrogate.make_solvers(images)
        outs = [{k: _pinned(s.n_cells) for k in ("rho", "ux", "uy")} for s in solvers]
        for s in solvers:
            s.set_equilibrium(*_start(s, s.info["rho_in"], rng))
        return dict(kind=kind, batch=native.Batch(solvers), solvers=solvers, outs=outs, steps=case["steps"])
    if kind == "pore":
        pore = native.generate_disks(case["n"], case["rmin"], case["rmax"], case["porosity"], seed)
        return dict(kind=kind, pore=pore)
    if kind == "conv":
        w, b, x, dy = _conv_inputs(case, seed)
        layer = surrogate.Conv3x3(case["cin"], case["cout"], np.random.default_rng(0))
        _load(layer, w, b)
        return dict(kind=kind, layer=layer, x=x, dy=dy)
    layers, x, target, mask = _net_inputs(case, seed)
    net = surrogate.UNet(WIDTHS)
    for layer, (w, b) in zip(net.layers(), layers):
        _load(layer, w, b)
    return dict(kind=kind, net=net, x=x, target=target, mask=mask)


# ---- one pass


def _fields(solver, out, rho0):
    c = solver.cells(out=out)
    return dict(drho=(torch.from_numpy(c["rho"]) - rho0).float(), ux=torch.from_numpy(c["ux"]).float(),
                uy=torch.from_numpy(c["uy"]).float())


def run(state):
    kind = state["kind"]
    if kind == "run":
        s = state["solver"]
        s.set_equilibrium(*state["start"])
        s.run(state["steps"])
        observed = s.observables()  # mean velocity, permeability, mass and the last step's residual
        return dict(_fields(s, state["out"], state["rho0"]), **{k: float(v) for k, v in observed.items()})
    if kind == "advance":
        s = state["solver"]
        s.advance_graph(state["steps"])
        return _fields(s, state["out"], state["rho0"])
    if kind == "batch":
        state["batch"].advance(state["steps"])
        return [_fields(s, o, s.info["rho_in"]) for s, o in zip(state["solvers"], state["outs"])]
    if kind == "pore":
        locpore, kn, iterations = native.pore_properties_gpu(state["pore"], 1e-9, 5e-9, return_iterations=True)
        return dict(locpore=locpore, kn=kn, iterations=iterations)
    if kind == "conv":
        layer = state["layer"]
        layer.zero_grad()
        y = layer.forward(state["x"], True)
        dx = layer.backward(state["x"], state["dy"])
        return dict(y=y, dx=dx, dw=layer.dw, db=layer.db)
    net = state["net"]
    if kind == "predict":
        return net.forward(state["x"])
    net.zero_grad()
    loss, dp = surrogate.masked_loss(net.forward(state["x"], keep=True), state["target"], state["mask"])
    net.backward(dp)
    net.adam(1e-3)
    layers = net.layers()
    return dict(loss=loss, dw=[l.dw for l in layers], db=[l.db for l in layers], w=[l.w for l in layers],
                b=[l.b for l in layers])


# ---- what a pass cannot do without


def _conv_flops(cin, cout, pixels):
    return 2.0 * 9 * cin * cout * pixels


def _net_flops(case):
    flops = 0.0
    scale = [0, 0, 1, 2, 3, 4, 3, 2, 1, 0, 0]  # pooling level each layer runs at
    for (ci, co), s in zip(_net_shapes(), scale):
        flops += _conv_flops(ci, co, case["batch"] * (case["n"] >> s) ** 2)
    return flops


def work(case):
    kind = case["kind"]
    if kind in ("run", "advance"):
        n2 = case["n"] ** 2
        updates = UPDATES_PER_PIXEL[case["levels"]] * n2 * case["steps"]
        per = 80.0 if case["sim"] == "adsorption" else 72.0
        # 9 populations read and written per update (adsorption: the
        # pseudopotential too); FP64 fields of every cell in (run) and out
        cells = 0.6 * n2 * 24.0 * (2 if kind == "run" else 1)
        return dict(bytes=per * updates + cells, flops=250.0 * updates)
    if kind == "batch":
        updates = cells = 0.0
        for n, l in zip(case["sides"].split(","), case["levels"].split(",")):
            updates += UPDATES_PER_PIXEL[int(l)] * int(n) ** 2 * case["steps"]
            cells += 0.5 * int(n) ** 2 * 24.0
        return dict(bytes=72.0 * updates + cells, flops=250.0 * updates)
    if kind == "pore":
        return dict(bytes=(4.0 + 16.0) * case["n"] ** 2, flops=0.0)
    if kind == "conv":
        pixels = case["batch"] * case["n"] ** 2
        weights = 9.0 * case["cin"] * case["cout"]
        return dict(bytes=pixels * 4.0 * (2 * case["cin"] + 2 * case["cout"]) + weights * 6.0,
                    flops=3 * _conv_flops(case["cin"], case["cout"], pixels))
    pixels = case["batch"] * case["n"] ** 2
    weights = sum(9.0 * ci * co for ci, co in _net_shapes())
    if kind == "predict":
        return dict(bytes=pixels * 4.0 * 5 + weights * 2.0, flops=_net_flops(case))
    # Adam: weights and two moments read and written, the gradient read
    return dict(bytes=pixels * 4.0 * 6 + weights * 30.0, flops=3 * _net_flops(case))


# ---- the same in 64 bits, in plain torch


def _bf16(w):
    return w.to(torch.bfloat16).double()  # the convolutions take BF16 weights


def _net_exact(layers, x):
    import torch.nn.functional as F

    def conv(k, v, relu=True):
        y = F.conv2d(v, layers[k][0], layers[k][1], padding=1)
        return torch.relu(y) if relu else y

    e = [conv(1, conv(0, x))]
    for i in range(1, 5):
        e.append(conv(1 + i, F.avg_pool2d(e[-1], 2)))
    d = e[4]
    for k, i in enumerate(range(3, -1, -1)):
        d = conv(6 + k, F.interpolate(d, scale_factor=2, mode="nearest")) + e[i]
    return conv(10, d, relu=False)


def exact(case, seed):
    """The network's cases in FP64.  None for the others: the solver's need the
    reference's boundary tables, the pore properties its thinning and search."""
    kind = case["kind"]
    if kind == "conv":
        w, b, x, dy = _conv_inputs(case, seed)
        w, b, x, dy = _bf16(w), b.double(), x.double(), dy.double()
        y = torch.relu(torch.nn.functional.conv2d(x, w, b, padding=1))
        return dict(y=y, dx=torch.nn.grad.conv2d_input(x.shape, w, dy, padding=1),
                    dw=torch.nn.grad.conv2d_weight(x, w.shape, dy, padding=1), db=dy.sum((0, 2, 3)))
    if kind not in ("train", "predict"):
        return None
    layers, x, target, mask = _net_inputs(case, seed)
    if kind == "predict":
        return _net_exact([(_bf16(w), b.double()) for w, b in layers], x.double())
    leaves = [(_bf16(w).requires_grad_(), b.double().requires_grad_()) for w, b in layers]
    p = _net_exact(leaves, x.double())
    m = mask.double()[:, None]
    loss = (m * (p - target.double())).square().sum() / (3 * mask.double().sum())
    loss.backward()

    def adam(v, g):  # the first step: the moments' corrections cancel their factors
        return v.double() - 1e-3 * g / (g.abs() + 1e-8)

    dw, db = [w.grad for w, _ in leaves], [b.grad for _, b in leaves]
    return dict(loss=loss.detach().reshape(1), dw=dw, db=db, w=[adam(v, g) for (v, _), g in zip(layers, dw)],
                b=[adam(v, g) for (_, v), g in zip(layers, db)])
