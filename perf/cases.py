"""The work that users of this framework have it do, as measurable cases.

Each case is one pass through the public entry points (`Flac`, `Batch`,
`Surrogate`, `Fno`), on sizes of the package's own workloads:

* `block`: the main loop of a model in double precision, ten steps (one
  period of the frequency tests), the mesh-quality test and the state an
  output needs back on the host;
* `dropin`: one step through the per-subroutine calls of a host program that
  keeps the reference's structure, its clock and `cord` / `vel` copied back;
* `remesh`: the remesh event after a block of steps;
* `mixed`: ten mixed-precision steps and the fields sampled on the mesh;
* `ensemble`: ten steps of a parameter sweep and the surrogate's snapshot;
* `predict`: the surrogate's forecast of a sweep from its sampled fields;
* `train`: one training step of the surrogate's network.

A model's state moves on from pass to pass, as it does for a user.
"""
import ctypes as C
import functools
import os
import tempfile
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from geoflac_gb300 import bytes_model, capi, clone, inpgen, new_state
from geoflac_gb300.batch import Batch
from geoflac_gb300.flac import Flac
from geoflac_gb300.fno import Fno, FnoConfig
from geoflac_gb300.surrogate import CRUST_PHASE, NCH, Normaliser, Surrogate

STEPS = 10  # steps of a block: one period of the models' ifreq_* tests
WARM = 100  # steps that a model has behind it when a pass begins
STATE = capi.F_CORD | capi.F_VEL | capi.F_TEMP | capi.F_STRESS | capi.F_APS | capi.F_PHASE
FIELDS = ("cord", "vel", "temp", "stress0", "aps", "iphase")
GRID = FnoConfig()
CHANNELS = ("vx", "vz", "sxx", "szz", "sxz", "aps", "temp", "crust", "uz")


def listed():
    return [
        # the smallest configured model: launch latency and short kernels
        dict(name="block_extension_60x20", kind="block", model="extension", nex=60, nez=20, side=3),
        # a mid-sized model with odd sides, Winkler base and phase changes
        dict(name="block_convergence_241x61", kind="block", model="convergence", nex=241, nez=61, side=3),
        # the headline model with its 25 markers per element
        dict(name="block_extension_1000x300", kind="block", model="extension", nex=1000, nez=300, side=5),
        # the same loop with the magma sub-model and surface processes
        dict(name="block_magma_300x75", kind="block", model="magma", nex=300, nez=75, side=3),
        # a host program that calls routine by routine
        dict(name="dropin_convergence_600x150", kind="dropin", model="convergence", nex=600, nez=150, side=3),
        # the remesh event of a long run
        dict(name="remesh_extension_400x120", kind="remesh", model="extension", nex=400, nez=120, side=3),
        # mixed precision, the smallest and the headline size
        dict(name="mixed_extension_60x20", kind="mixed", model="extension", nex=60, nez=20, side=3),
        dict(name="mixed_extension_1000x300", kind="mixed", model="extension", nex=1000, nez=300, side=5),
        # a handful of small members, and a sweep over the whole range of meshes
        dict(name="ensemble_8_small", kind="ensemble", members=8, lo=80, hi=120, sweep=1),
        dict(name="ensemble_64", kind="ensemble", members=64, lo=80, hi=400, sweep=2),
        # the surrogate: a screening batch, and a training step
        dict(name="predict_64", kind="predict", members=64),
        dict(name="train_64", kind="train", batch=64, weighted=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("block", "block", "dropin", "remesh", "mixed", "mixed", "ensemble", "predict", "train"))
    if kind == "ensemble":
        lo = rng.randint(80, 120)
        return dict(kind=kind, members=_log_int(rng, 3, 48), lo=lo, hi=rng.randint(lo + 1, 400),
                    sweep=rng.randint(3, 999))
    if kind == "predict":
        return dict(kind=kind, members=_log_int(rng, 1, 64))
    if kind == "train":
        # the network trains on multiples of 8, with or without the topography rows' weight
        return dict(kind=kind, batch=8 * rng.randint(1, 8), weighted=rng.random() < 0.5)
    nex = _log_int(rng, 60, 400 if kind == "remesh" else 900)
    nez = max(15, int(nex * rng.uniform(0.25, 0.33)))
    model = "extension" if kind in ("mixed", "remesh") else rng.choice(("extension", "convergence"))
    return dict(kind=kind, model=model, nex=nex, nez=nez, side=3)


# ---------------------------------------------------------------- models
def _model(case):
    nex, nez = case["nex"], case["nez"]
    if case["model"] == "extension":
        edge = 5e3 * (60.0 / nex) ** 0.572  # 5 km elements at 60 columns, 1 km at 1000
        m = inpgen.two_phase_extension(nex, nez, nex * edge, max(nez * edge, 90e3), ny_rem=1)
    elif case["model"] == "convergence":
        m = inpgen.convergence(nex, nez)
    else:
        m = inpgen.magma_arc(nex, nez)
        m.prod_magma, m.prod_magma2 = 2e-15, 1e-13  # the reference's default rates
    m.ntest_rem = STEPS
    return m


def _seed_melting(p, s):
    """Melting of the arc model: a hot mantle column under the ocean and
    subducted basalt and sediment below the Moho, by fractions of the mesh."""
    nz1, nx1 = p.nz - 1, p.nx - 1

    def r(f):
        return int(round(f * nz1))

    def c(f):
        return int(round(f * nx1))

    temp, ids, nm, ph = s["temp"], s["mark_id_elem"], s["nmark_elem"], s["mark_phase"]
    temp[r(2 / 15):r(5 / 15), c(8 / 60):c(17 / 60)] = 1500.0
    for i in range(c(34 / 60), c(38 / 60)):
        for j in range(r(3 / 15), r(5 / 15)):
            marks = ids[:nm[j, i], j, i] - 1
            ph[marks] = 3 if i % 2 else 11
            count = np.bincount(ph[marks], minlength=p.nphase + 1)[1:p.nphase + 1]
            s["phase_ratio"][:, j, i] = count / nm[j, i]
            s["iphase"][j, i] = int(np.argmax(count)) + 1
    temp[r(3 / 15):r(6 / 15), c(34 / 60):c(39 / 60)] = 1100.0


def _start_up(model, side):
    with tempfile.TemporaryDirectory() as d:
        return new_state(model.write(os.path.join(d, "model.inp")), markers_per_side=side)


@functools.lru_cache(maxsize=2)
def _base(key):
    """A model's host state after its first steps (double precision)."""
    case = dict(key)
    p, c, s = _start_up(_model(case), case["side"])
    if case["model"] == "magma":
        _seed_melting(p, s)
        return p, c, s  # its first steps are the ones that melt
    with Flac(p, c, s, "fp64") as g:
        g.step(WARM)
        g.download()
    return p, c, s


def _perturb(p, s, seed):
    """What differs between two runs of one set-up: a degree or two of
    temperature inside, and random initial weakness in a tenth of the columns."""
    rng = np.random.default_rng(seed)
    s["temp"][1:-1, :] += rng.normal(0.0, 1.0, size=(p.nz - 2, p.nx))
    w = max(1, (p.nx - 1) // 10)
    i0 = int(rng.integers(0, p.nx - 1 - w + 1))
    s["aps"][:, i0:i0 + w] += rng.uniform(0.0, 0.05, size=(p.nz - 1, w))


def _flac(case, seed, mode):
    p, c, s = clone(*_base(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "kind")))))
    _perturb(p, s, seed)
    pinned = []

    def make(nbytes):
        pinned.append(torch.empty(nbytes, dtype=torch.uint8, pin_memory=True))
        return pinned[-1].numpy()

    if mode == "fp64":  # the arrays that come back to the host live in pinned memory
        s.rehome(["cord", "vel", "temp", "temp0", "stress0", "aps", "iphase", "phase_ratio", "jmoho"], make)
    return Flac(p, c, s, mode), pinned


@functools.lru_cache(maxsize=1)
def _sweep(members, lo, hi, sweep):
    scale = (lo, max(25, round(lo * 0.3)), hi, max(26, round(hi * 0.3)))
    models = [inpgen.ensemble_member(k, sweep, scale)[0] for k in range(members)]
    with ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 4)) as ex:
        return list(ex.map(lambda m: _start_up(m, 3), models))


# ---------------------------------------------------------------- surrogate
#: per channel: mean, spread, spread of the increments over a forecast (SI units)
_STATS = np.array([[0.0, 4e-10, 4e-11], [0.0, 2e-10, 3e-11], [-3e9, 2e9, 4e7], [-3e9, 2e9, 3e7], [0.0, 6e7, 5e6],
                   [0.05, 0.12, 0.01], [800.0, 450.0, 2.0], [0.3, 0.45, 0.01], [0.0, 900.0, 150.0]])


def _fields(n, seed):
    """Smooth random fields of the sampled channels' sizes, FP32 [n, H, W, 9]."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    h = torch.linspace(0.0, 1.0, GRID.H, device="cuda")[:, None]
    w = torch.linspace(0.0, 1.0, GRID.W, device="cuda")[None, :]
    out = torch.empty((n, GRID.H, GRID.W, NCH), device="cuda")
    out.normal_(0.0, 0.05, generator=g)
    for _ in range(6):
        a, kh, kw, ph = (torch.rand((4, n, 1, 1, NCH), generator=g, device="cuda") * 2 - 1)
        out += 0.5 * a * torch.sin(9 * kh * h[..., None] + 20 * kw * w[..., None] + 3.1 * ph)
    mean, std = (torch.tensor(_STATS[:, k], dtype=torch.float32, device="cuda") for k in (0, 1))
    return out * std + mean


def _network(seed):
    net = Fno(GRID, seed=seed % (1 << 31))
    for k, v in net.p.items():
        if k.startswith("R"):
            v *= 30.0  # spectral weights of a trained network's size
    return net


def _member_params(n, seed):
    rng = np.random.default_rng([seed, 7])
    lo, hi = np.array([10.0, 25.0, 400.0, -5.0]), np.array([35.0, 45.0, 800.0, 5.0])
    return (lo + (hi - lo) * rng.random((n, 4))).astype(np.float32)


def _stats():
    pm, ps = [22.5, 35.0, 600.0, 0.0], [7.2, 5.8, 115.0, 2.9]
    return Normaliser(torch.tensor(np.concatenate([_STATS[:, 0], _STATS[:, 1], pm, ps]), dtype=torch.float32).cuda(),
                      torch.tensor(np.concatenate([0 * _STATS[:, 2], _STATS[:, 2]]), dtype=torch.float32).cuda())


def _train_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["batch"]
    mean, std = (torch.tensor(_STATS[:, k], dtype=torch.float32, device="cuda") for k in (0, 1))
    x = torch.zeros((n, GRID.H, GRID.W, GRID.cin), device="cuda")
    x[..., :NCH] = (_fields(n, seed) - mean) / std
    x[..., NCH:NCH + 4] = torch.rand((n, 1, 1, 4), generator=g, device="cuda") * 3 - 1.5
    y = torch.zeros((n, GRID.H, GRID.W, GRID.cout), device="cuda")
    y[..., :NCH] = (_fields(n, seed + 1) - mean) / std
    weight = None
    if case["weighted"]:
        weight = torch.ones((GRID.H, GRID.W, GRID.cout), device="cuda")
        weight[:2, :, 8] = 64.0  # the topography rows
    return x.to(torch.bfloat16), y, weight


# ---------------------------------------------------------------- passes
def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind}
    if kind in ("block", "dropin", "remesh"):
        st["g"], st["pinned"] = _flac(case, seed, "fp64")
        if kind == "dropin":
            st["g"].set_sync(False)
    elif kind == "mixed":
        st["g"], _ = _flac(case, seed, "mixed")
        st["b"] = Batch([st["g"]])
        st["grid"] = torch.empty((1, case["nez"] + 1, case["nex"] + 1, NCH), dtype=torch.float32, device="cuda")
    elif kind == "ensemble":
        models = []
        for k, base in enumerate(_sweep(case["members"], case["lo"], case["hi"], case["sweep"])):
            p, c, s = clone(*base)
            _perturb(p, s, [seed, k])
            models.append(Flac(p, c, s, "mixed"))
        st["b"] = Batch(models)
        st["b"].set_config(threads=256, items_per_thread=2, ctas_per_sm=3, graph_steps=STEPS)
        st["grid"] = torch.empty((len(models), GRID.H, GRID.W, NCH), dtype=torch.float32, device="cuda")
    elif kind == "predict":
        st["sur"] = Surrogate(GRID, _stats())
        st["sur"].net = _network(seed)
        st["raw"] = _fields(case["members"], seed)
        st["prm"] = _member_params(case["members"], seed)
    else:
        st["net"] = _network(seed)
        st["x"], st["y"], st["weight"] = _train_inputs(case, seed)
    return st


def _host(g):
    return {f: g.state[f] for f in FIELDS}


def _channels(grid):
    return {name: grid[..., k] for k, name in enumerate(CHANNELS)}


def run(st):
    kind, g = st["kind"], st.get("g")
    if kind == "block":
        g.run(1)
        g.download(STATE)
        return _host(g)
    if kind == "dropin":
        p, k = g.params, g.clock
        g.fl_therm()
        if k.nloop % p.ifreq_rmasses == 0:
            g.change_phase()
        g.fl_rheol()
        g.fl_node()
        g.fl_move()
        if k.nloop % p.ifreq_rmasses == 0:
            g.rmasses()
        if k.nloop % p.ifreq_imasses == 0:
            g.dt_mass()
        g.download(capi.F_CORD | capi.F_VEL)
        k.nloop += 1  # the host program's own loop counter and time
        k.time += k.dt
        capi.check(g.lib.gf_set_clock(g.ctx, C.byref(k)), "gf_set_clock")
        return {"cord": g.state["cord"], "vel": g.state["vel"]}
    if kind == "remesh":
        g.step(STEPS)
        g.itest_mesh()
        g.remesh()
        g.download(STATE)
        return _host(g)
    if kind == "mixed":
        g.step(STEPS)
        st["b"].sample(st["grid"], st["grid"].shape[1], st["grid"].shape[2], CRUST_PHASE)
        return _channels(st["grid"])
    if kind == "ensemble":
        st["b"].step(STEPS)
        st["b"].sample(st["grid"], GRID.H, GRID.W, CRUST_PHASE)
        return _channels(st["grid"])
    if kind == "predict":
        return _channels(st["sur"].predict(st["raw"], st["prm"]))
    net = st["net"]
    out = net.forward(st["x"], train=True)
    _, dout = net.loss_grad(out, st["y"], st["weight"])
    grads = net.backward(dout)
    net.adam(lr=1e-4)
    return {"out": out, "grad": grads}


# ---------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind in ("predict", "train"):
        n, c = case.get("members") or case["batch"], GRID
        points = n * c.H * c.W
        dense = 2 * points * (c.cin * c.C + c.layers * c.C * c.C + c.C * c.P + c.P * c.cout)
        spectral = 2 * n * c.C * (c.H * c.W * 2 * c.m2 + c.H * 2 * c.m2 * 2 * c.Q + 4 * c.modes * c.C) * 2 * c.layers
        weights = 4 * c.layers * c.modes * c.C * c.C * 2
        if kind == "predict":
            return {"bytes": points * NCH * 8 + weights, "flops": dense + spectral}
        # inputs, targets and outputs once; weights, gradients and moments read and written by the optimiser
        return {"bytes": points * (2 * c.cin + 4 * c.cout + 4 * c.cout) + 7 * weights, "flops": 3 * (dense + spectral)}
    if kind == "ensemble":
        bases = [inpgen.ensemble_member(k, case["sweep"], (case["lo"], max(25, round(case["lo"] * 0.3)), case["hi"],
                                                           max(26, round(case["hi"] * 0.3))))[0]
                 for k in range(case["members"])]
        elems = sum(m.nex * m.nez for m in bases)
        out = case["members"] * GRID.H * GRID.W * NCH * 4
    else:
        elems = case["nex"] * case["nez"]
        out = elems * (4 * 8 if kind == "dropin" else NCH * 4 if kind == "mixed" else 25 * 8)
    mode = "mixed" if kind in ("mixed", "ensemble") else "fp64"
    steps = 1 if kind == "dropin" else STEPS
    # about a thousand operations per element and step, in the precision of the mode
    return {"bytes": elems * steps * bytes_model.step_bytes_per_element(mode, nphase=4) + out,
            "flops": 1000.0 * elems * steps}


# ---------------------------------------------------------------- 64 bits
def _fno64(p, x):
    """The network by its definition, in 64 bits (torch's FFT)."""
    c = GRID
    rows = torch.tensor([c.k1(q) for q in range(c.Q)], device=x.device)
    gelu = torch.nn.functional.gelu
    z = x @ p["lift_w"].T + p["lift_b"]
    for l in range(c.layers):
        f = torch.fft.rfft2(z, dim=(1, 2))[:, rows, :c.m2]  # [B, Q, m2, C]
        r = torch.view_as_complex(p[f"R{l}"].contiguous()).reshape(c.m2, c.Q, c.C, c.C)
        mixed = torch.einsum("bqki,kqio->bqko", f, r)
        full = torch.zeros((x.shape[0], c.H, c.W // 2 + 1, c.C), dtype=mixed.dtype, device=x.device)
        full = full.index_copy(1, rows, torch.nn.functional.pad(mixed, (0, 0, 0, c.W // 2 + 1 - c.m2)))
        s = torch.fft.irfft2(full, s=(c.H, c.W), dim=(1, 2))
        z = z @ p[f"w{l}"].T + p[f"b{l}"] + s
        if l < c.layers - 1:
            z = gelu(z)
    return gelu(z @ p["p1_w"].T + p["p1_b"]) @ p["p2_w"].T + p["p2_b"]


def exact(case, seed):
    """The surrogate's cases.  The models' cases have none: their outputs are
    the state after ten coupled steps (rheology, thermal update in the
    reference's serial order, marker phases), which plain array code takes
    minutes for at these sizes."""
    if case["kind"] == "predict":
        n = case["members"]
        p = {k: v.double() for k, v in _network(seed).p.items()}
        raw, prm = _fields(n, seed).double(), torch.from_numpy(_member_params(n, seed)).cuda().double()
        norm = _stats()
        st, sd = norm.stats.double(), norm.stats_d.double()
        x = torch.zeros((n, GRID.H, GRID.W, GRID.cin), dtype=torch.float64, device="cuda")
        x[..., :9] = (raw - st[:9]) / st[9:18]
        x[..., 9:13] = ((prm - st[18:22]) / st[22:26])[:, None, None, :]
        for ch, size, shape in ((13, GRID.W, (1, 1, -1)), (14, GRID.H, (1, -1, 1))):  # cell centres in [-1, 1]
            x[..., ch] = (2 * (torch.arange(size, dtype=torch.float64, device="cuda") + 0.5) / size - 1).view(shape)
        out = torch.cat([_fno64(p, x[i:i + 8]) for i in range(0, n, 8)])
        return _channels(raw + sd[:9] + sd[9:] * out[..., :9])
    if case["kind"] == "train":
        p = {k: v.double().requires_grad_() for k, v in _network(seed).p.items()}
        x, y, weight = _train_inputs(case, seed)
        w = 1.0 if weight is None else weight.double()
        outs = []
        for i in range(0, case["batch"], 8):
            out = _fno64(p, x[i:i + 8].double())
            ((out - y[i:i + 8].double()).square() * w).sum().div(y.numel()).backward()
            outs.append(out.detach())
        return {"out": torch.cat(outs), "grad": {k: v.grad for k, v in p.items()}}
    return None
