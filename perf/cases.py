"""The work a user of this framework has it do, as cases that can be timed and compared.

Each case is one whole call path through the public entry points:

run     a realisation with the run loop on the device (Simulation.run), `final` with every
        person's state copied back at its end
peak    the same loop at epidemic-peak load from the first timestep on
host    a realisation stepped from the host, from an uploaded start state to a
        downloaded final state (what a C host around the ABI does)
batch   realisations of one population stepped together (Batch.run), one scenario each
probs   UpdateProbs, the dense normaliser of the spatial sampler
setup   a synthetic population built on the device and copied to the host's buffers
train   minibatch steps of the scenario surrogate, weights read back at the end
screen  surrogate predictions for many scenarios

A population (its structure, parameter block and kernel tables) is what a program
keeps over its realisations, so it is made once per size and each prepared state is
a replica of it; the epidemic's seeds, start states and scenarios come from the seed.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "covid-sim_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from covidsim_b200 import abi, params as prm, population, sim, surrogate  # noqa: E402

DAYS, OUT = surrogate.DAYS, len(surrogate.OUTPUTS)
# weights [out, in] of the surrogate's layers: six linear, three convolutions (5 taps)
LAYERS = ((512, 8), (512, 512), (512, 512), (512, 512), (256, 512), (2944, 256), (64, 320), (32, 320), (4, 160))


def listed():
    return [
        # the scale of a first try and of the parity tests
        dict(name="run_20k_60d", kind="run", people=20_000, cx=12, cy=12, nmcl=4, days=60, seeds=20, policy="none",
             adunits=0, every_step=False, final=True),
        # a C host's realisation: one call per timestep, daily counters read back
        dict(name="host_200k_30d", kind="host", people=200_000, cx=120, cy=120, nmcl=10, days=30, seeds=400,
             policy="global", adunits=0),
        # 1 M people without interventions
        dict(name="run_1m_120d", kind="run", people=1_000_000, cx=240, cy=240, nmcl=10, days=120, seeds=100,
             policy="none", adunits=0, every_step=False, final=False),
        # an odd population on an oblong grid, staggered triggers per admin unit and the
        # reference's UpdateProbs test after every timestep
        dict(name="run_1m5_adunits_150d", kind="run", people=1_500_007, cx=340, cy=260, nmcl=5, days=150, seeds=317,
             policy="adunit", adunits=5, every_step=True, final=False),
        # the benchmark's default workload: a whole year of 10 M people with interventions
        dict(name="run_10m_365d", kind="run", people=10_000_000, cx=240, cy=240, nmcl=10, days=365, seeds=100,
             policy="global", adunits=0, every_step=False, final=False),
        # 10 M people on the finer grid, the sweeps under the largest load they meet
        dict(name="peak_10m_8d", kind="peak", people=10_000_000, cx=600, cy=600, nmcl=10, days=8, seeds=500_000),
        # a scenario sweep's batch
        dict(name="batch_16x1m_120d", kind="batch", people=1_000_000, cx=240, cy=240, nmcl=10, days=120, seeds=100,
             members=16),
        # the normaliser at the finer grid
        dict(name="probs_600x600", kind="probs", people=2_000_000, cx=600, cy=600, nmcl=10),
        # a new population
        dict(name="setup_1m", kind="setup", people=1_000_000, cx=240, cy=240, nmcl=10, blobs=0, adunits=0),
        # training as the scenario sweep's pipeline does it, and at a full (ragged) batch
        dict(name="train_64x16", kind="train", rows=64, steps=16),
        dict(name="train_250x8", kind="train", rows=250, steps=8),
        # screening a scenario sweep
        dict(name="screen_20000", kind="screen", rows=20_000, batch=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, cells):
    # an oblong grid of about `cells` cells, its sides multiples of 4 as the set-up makes them
    a = math.exp(rng.uniform(-0.4, 0.4))
    s = math.sqrt(cells)
    return tuple(min(600, max(8, 4 * int(round(v / 4)))) for v in (s * a, s / a))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "peak", "host", "batch", "batch", "probs", "setup", "train", "train", "screen"])
    if kind == "train":
        return dict(kind=kind, rows=_log(rng, 1, 500), steps=rng.randint(2, 16))
    if kind == "screen":
        return dict(kind=kind, rows=_log(rng, 1, 20_000), batch=rng.choice([64, 200, 256, 512]))
    if kind == "probs":
        cx, cy = _side(rng, _log(rng, 400, 300_000))
        return dict(kind=kind, people=_log(rng, 20_000, 1_500_000), cx=cx, cy=cy, nmcl=rng.randint(2, 8))
    people = _log(rng, 5_000, 300_000 if kind in ("host", "batch") else 3_000_000)
    cx, cy = _side(rng, people / math.exp(rng.uniform(math.log(8), math.log(150))))
    case = dict(kind=kind, people=people, cx=cx, cy=cy, nmcl=rng.randint(3, 10))
    if kind == "setup":
        blobs = rng.choice([0, 0, 7, 30])
        return dict(case, blobs=blobs, adunits=rng.choice([0, 3, 10]))
    case["days"] = _log(rng, 7, 120)
    if kind == "peak":
        return dict(case, days=rng.randint(4, 12), seeds=max(20, people // rng.randint(15, 60)))
    case["seeds"] = _log(rng, 10, max(20, people // 50))
    if kind == "batch":
        return dict(case, members=rng.randint(2, 16))
    policy = rng.choice(["none", "global", "adunit"])
    case.update(policy=policy, adunits=rng.randint(2, 10) if policy == "adunit" else 0)
    if kind == "host":
        return case
    return dict(case, every_step=rng.random() < 0.5, final=people < 300_000 and rng.random() < 0.5)


# ------------------------------------------------------------- populations
_bases = {}


def _cell_deg(case):
    # 1/120 degree as the 240 x 240 grid, finer where that would pass 2 degrees
    return min(1.0 / 120, 2.0 / max(case["cx"], case["cy"]))


def _grid(case):
    g = population.make_grid(nmcl=case["nmcl"])
    g.update(ncw=case["cx"], nch=case["cy"], cell_width=_cell_deg(case), cell_height=_cell_deg(case))
    return g


def _base(case):
    """The population of the case's size and a Simulation of it, made once."""
    key = tuple(case.get(k, 0) for k in ("people", "cx", "cy", "nmcl", "adunits"))
    if key not in _bases:
        if len(_bases) >= 6:   # bounded: a long list of drawn sizes
            _bases.pop(next(iter(_bases)))
        grid = _grid(case)
        pop = population.generate_on_device(case["people"], grid, adunit_grid=case.get("adunits") or None)
        P, lk, hr = prm.build_params(grid)
        P.LocalBeta, _ = sim.calibrate_local_beta(pop, P, 2.4, sample=min(20_000, case["people"]))
        _bases[key] = (sim.Simulation(pop, P, lk, hr), pop, P)
    return _bases[key]


def _policy(case):
    if case["policy"] == "none":
        return None
    units = max(1, case["adunits"]) ** 2
    return sim.InterventionPolicy(threshold=max(1, int(case["people"] * 1e-5 / units)), duration=60.0,
                                  per_adunit=case["policy"] == "adunit")


def _cells(s):
    """Every cell's counts, as a host's sample reads them."""
    n = s.pop.n_cells
    a = np.empty((5, n), np.int32)
    be = s.backend
    if be.lib.cs_gpu_get_cell_counts(be.ctx, *(a[k].ctypes.data for k in range(5))) != 0:
        raise abi.CovidSimError("cs_gpu_get_cell_counts")
    return a


# ---------------------------------------------------------------- surrogate
def _net_inputs(case, seed):
    rng = np.random.default_rng([seed, 7])
    w = []
    for o, i in LAYERS:
        lim = math.sqrt(6.0 / i)
        w += [rng.uniform(-lim, lim, o * i).astype(np.float32), rng.uniform(-0.05, 0.05, o).astype(np.float32)]
    x = rng.random((case["rows"], 8), dtype=np.float32)
    # smooth daily curves on the log1p scale of the outputs
    y = np.empty((0, DAYS, OUT), np.float32)
    if case["kind"] == "train":
        t = np.arange(DAYS, dtype=np.float32)[None, :, None]
        p = rng.random((case["rows"], 3, OUT), dtype=np.float32)
        y = (8.0 * p[:, :1] * np.exp(-((t - 40 - 280 * p[:, 1:2]) / (20 + 60 * p[:, 2:])) ** 2)).astype(np.float32)
    return np.concatenate(w), x, y


def _forward64(w, x):
    h = x
    for k in range(6):
        h = torch.relu(h @ w[2 * k].T + w[2 * k + 1])
    h = h.reshape(-1, 46, 64)
    for k in range(6, 9):
        cin = LAYERS[k][1] // 5
        h = h[:, :, :cin].repeat_interleave(2, dim=1)
        T = h.shape[1]
        h = torch.nn.functional.pad(h, (0, 0, 2, 2))
        h = torch.cat([h[:, j:j + T] for j in range(5)], dim=2) @ w[2 * k].T + w[2 * k + 1]
        if k < 8:
            h = torch.relu(h)
    return h[:, :DAYS]


def _weights64(flat):
    f, k, w = torch.from_numpy(flat).double().cuda(), 0, []
    for o, i in LAYERS:
        w += [f[k:k + o * i].reshape(o, i).clone(), f[k + o * i:k + o * i + o].clone()]
        k += o * i + o
    return w


LR, DECAY = 3e-4, 1e-4


# ------------------------------------------------------------------- cases
def _setup_buffers(case):
    """Host buffers a population's arrays are copied to, each as long as it can get,
    and the cs_setup_out pointing at them."""
    n, npt = case["people"], 4
    mcells = min(n, case["cx"] * case["cy"] * case["nmcl"] ** 2)
    cells = min(n, case["cx"] * case["cy"])
    spec = dict(person_hh=(n, "i4"), person_mcell=(n, "i4"), person_age=(n, "u1"), person_place=(npt * n, "i4"),
                person_group=(npt * n, "u2"), hh_first=(n, "i4"), hh_nh=(n, "u2"), hh_x=(n, "f4"), hh_y=(n, "f4"),
                mcell_cell=(mcells, "i4"), mcell_adunit=(mcells, "i4"), mcell_grid=(mcells, "i8"),
                cell_grid=(cells, "i4"), cell_start=(cells + 1, "i4"))
    out, arrs = abi.cs_setup_out(), {}
    for k, (size, dt) in spec.items():
        arrs[k] = np.zeros(size, {"u2": "i2"}.get(dt, dt))
        setattr(out, k, arrs[k].ctypes.data)
    for k in ("place_mcell", "place_x", "place_y", "place_member_ofs", "place_members", "place_group_ofs",
              "group_start", "group_size"):
        arrs[k] = [np.zeros(n + 1, "f4" if k[-2:] in ("_x", "_y") else "i4") for _ in range(npt)]
        for t in range(npt):
            getattr(out, k)[t] = arrs[k][t].ctypes.data
    return arrs, out


def _synthetic_cells(pop, seed):
    """S, L, I, R of every cell part way through an epidemic."""
    rng = np.random.default_rng([seed, 11])
    n = np.diff(pop.cell_start)
    S = np.floor(n * rng.random(len(n))).astype(np.int32)
    L = np.floor((n - S) * rng.random(len(n)) * 0.2).astype(np.int32)
    I = np.floor((n - S - L) * rng.random(len(n)) * 0.3).astype(np.int32)
    return n, S, L, I, (n - S - L - I).astype(np.int32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "setup":
        S, P, keep = population.setup_spec(case["people"], _grid(case), seed=seed, blobs=case["blobs"],
                                           blob_share=0.4, adunit_grid=case["adunits"] or None)
        arrs, out = _setup_buffers(case)
        return dict(kind=kind, spec=S, params=P, keep=keep, arrs=arrs, out=out, lib=abi.load_library())
    if kind in ("train", "screen"):
        w, x, y = _net_inputs(case, seed)
        net = surrogate.Surrogate(max_batch=case["rows"] if kind == "train" else case["batch"], params=w)
        return dict(kind=kind, net=net, w=w, x=x, y=y, steps=case.get("steps", 0))
    base, pop, P = _base(case)
    if kind == "batch":
        thetas = surrogate.sample_scenarios(case["members"], seed)
        sims, policies = [], []
        beta = P.LocalBeta
        for th in thetas:
            q, pol = surrogate.scenario_params(P, beta, th)
            sims.append(base.replica(q))
            policies.append(pol)
        return dict(kind=kind, batch=sim.Batch(sims), seeds=[seed + 7919 * k for k in range(len(sims))],
                    policies=policies, days=case["days"], n_seed=case["seeds"])
    s = base.replica()
    st = dict(kind=kind, sim=s, seed=seed, days=case.get("days", 0))
    if kind == "run":
        st.update(n_seed=case["seeds"], policy=_policy(case), every_step=case["every_step"], arrs={}, view=None)
        if case["final"]:
            st["arrs"], st["view"] = sim.state_arrays(pop.n_people, pop.n_cells)
    elif kind == "peak":
        st.update(people=s.choose_seeds(seed, case["seeds"]), policy=sim.run_policy(None, pop.num_place_types))
    elif kind == "host":
        arrs, view = sim.state_arrays(pop.n_people, pop.n_cells)
        out, view_out = sim.state_arrays(pop.n_people, pop.n_cells)
        s.backend.begin_run(seed, s.choose_seeds(seed, case["seeds"]))
        s.backend.download(view)
        st.update(arrs=arrs, view=view, out=out, view_out=view_out, policy=_policy(case))
    else:   # probs: the cells part way through an epidemic
        arrs, view = sim.state_arrays(pop.n_people, pop.n_cells)
        s.backend.begin_run(seed, s.choose_seeds(seed, 1))
        s.backend.download(view)
        _, arrs["cell_S"][:], arrs["cell_L"][:], arrs["cell_I"][:], arrs["cell_R"][:] = _synthetic_cells(pop, seed)
        s.backend.upload(seed, view)
        tot, s0 = np.empty(pop.n_cells, np.float64), np.empty(pop.n_cells, np.int32)
        some = abi.cs_state_view()
        some.cell_tot_prob, some.cell_S0 = tot.ctypes.data, s0.ctypes.data
        st.update(tot=tot, s0=s0, view=some)
    return st


def run(st):
    kind = st["kind"]
    if kind == "run":
        series, blocks = st["sim"].run(st["seed"], st["days"], n_seed=st["n_seed"], policy=st["policy"],
                                       probs_every_step=st["every_step"], blocks=True)
        if st["view"] is not None:
            st["sim"].backend.download(st["view"])
        return dict(st["arrs"], blocks=blocks, cells=_cells(st["sim"]))
    if kind == "peak":
        be = st["sim"].backend
        be.begin_run(st["seed"], st["people"])
        return dict(blocks=be.run_device(st["days"], st["policy"]), cells=_cells(st["sim"]))
    if kind == "host":
        s = st["sim"]
        series, blocks = s.run(st["seed"], st["days"], policy=st["policy"], initial_state=st["view"],
                               device_loop=False, blocks=True)
        s.backend.download(st["view_out"])
        return dict(st["out"], blocks=blocks)
    if kind == "batch":
        series, blocks = st["batch"].run(st["seeds"], st["days"], n_seed=st["n_seed"], policy=st["policies"],
                                         blocks=True)
        return blocks
    if kind == "probs":
        be = st["sim"].backend
        be.update_probs(0)
        be.download(st["view"])
        return dict(tot_prob=st["tot"], S0=st["s0"])
    if kind == "setup":
        lib, h = st["lib"], C.c_void_p()
        try:
            if lib.cs_gpu_setup_run(C.byref(st["spec"]), C.byref(st["params"]), 0, C.byref(h)) != 0 or \
                    lib.cs_gpu_setup_sizes(h, C.byref(st["out"])) != 0 or \
                    lib.cs_gpu_setup_download(h, C.byref(st["out"])) != 0:
                raise abi.CovidSimError(lib.cs_gpu_setup_last_error(h).decode())
        finally:
            lib.cs_gpu_setup_destroy(h)
        return st["arrs"]
    if kind == "train":
        net = st["net"]
        net.set_params(st["w"])
        losses = [net.train_step(st["x"], st["y"], LR, DECAY) for _ in range(st["steps"])]
        return dict(weights=net.get_params(), losses=np.array(losses, np.float32))
    return st["net"].predict(st["x"])


def work(case):
    kind = case["kind"]
    if kind in ("train", "screen"):
        # 2 flops per weight and row for the linear layers, per weight and time point for
        # the convolutions; a training step also forms both gradients of every product
        macs = sum(o * i for o, i in LAYERS[:6]) + sum(o * i * 92 * 2 ** k for k, (o, i) in enumerate(LAYERS[6:]))
        n = sum(o * i + o for o, i in LAYERS)
        if kind == "screen":
            return dict(flops=2 * macs * case["rows"], bytes=4 * n + case["rows"] * (32 + 4 * DAYS * OUT))
        # weights, both moments read and written each step; the minibatch's inputs and targets
        return dict(flops=6 * macs * case["rows"] * case["steps"],
                    bytes=case["steps"] * (24 * n + case["rows"] * (32 + 4 * DAYS * OUT)) + 8 * n)
    cells, people = case["cx"] * case["cy"], case["people"]
    if kind == "probs":   # every cell pair once; the cells' counts in, the quotients out
        return dict(flops=2 * cells * cells, bytes=28 * cells + 32 * people)
    if kind == "setup":   # the weights' draws and the arrays handed over
        return dict(flops=0, bytes=16 * cells * case["nmcl"] ** 2 + 45 * people)
    steps = 4 * case["days"] * case.get("members", 1)
    state, static = 57, 60   # bytes per person of dynamic state written and structure read
    infected = 0.5 if kind != "peak" else 0.3
    # the state's reset or upload, the structure and state around each infected person
    # (its household, places and contacts), every cell's counts once a timestep
    members = case.get("members", 1)
    extra = 2 * state * people if kind == "host" else 0
    return dict(flops=0, bytes=members * people * (state + int(infected * (static + 10 * 32))) + 16 * cells * steps + extra)


def exact(case, seed):
    """tot_prob, the surrogate's predictions and its trained weights in 64 bits; the other
    paths return whole numbers and random trajectories."""
    kind = case["kind"]
    if kind in ("train", "screen"):
        flat, x, y = _net_inputs(case, seed)
        w = _weights64(flat)
        x = torch.from_numpy(x).double().cuda()
        if kind == "screen":
            with torch.no_grad():
                return torch.cat([_forward64(w, b) for b in x.split(1000)]).cpu().numpy()
        y = torch.from_numpy(y).double().cuda()
        m, v, losses = [torch.zeros_like(p) for p in w], [torch.zeros_like(p) for p in w], []
        for k in range(1, case["steps"] + 1):
            w = [p.detach().requires_grad_() for p in w]
            loss = ((_forward64(w, x) - y) ** 2).mean()
            losses.append(float(loss))
            g = torch.autograd.grad(loss, w)
            with torch.no_grad():
                m = [0.9 * a + 0.1 * b for a, b in zip(m, g)]
                v = [0.999 * a + 0.001 * b * b for a, b in zip(v, g)]
                w = [p * (1 - LR * DECAY) - LR * (a / (1 - 0.9 ** k)) / ((b / (1 - 0.999 ** k)).sqrt() + 1e-8)
                     for p, a, b in zip(w, m, v)]
        return dict(weights=torch.cat([p.detach().reshape(-1) for p in w]).cpu().numpy(), losses=np.array(losses))
    if kind != "probs":
        return None
    _, pop, _ = _base(case)
    n, S, L, I, _ = _synthetic_cells(pop, seed)
    s0 = (S + L + I).astype(np.int32)
    cx, cy = case["cx"], case["cy"]
    dev = dict(dtype=torch.float64, device="cuda")
    grids = torch.zeros(2, cy, cx, **dev)
    gx, gy = torch.from_numpy(pop.cell_grid // cy).long().cuda(), torch.from_numpy(pop.cell_grid % cy).long().cuda()
    grids[0, gy, gx] = torch.from_numpy(s0).to(**dev)
    grids[1, gy, gx] = torch.from_numpy(n).to(**dev)
    # great-circle distances by the model's tables of sin, cos (degrees) and asin^2(sqrt(x))
    # at steps of 1/1000, linear between; the power-law kernel of those distances
    step = _cell_deg(case)
    deg = torch.arange(361, **dev) * 3.1415926535 / 180
    sin, cos = torch.sin(deg), torch.cos(deg)
    tab = torch.asin(torch.sqrt(torch.arange(1001, **dev) / 1000)) ** 2

    def at(table, v):
        k = v.floor().long()
        f = v - k
        return (1 - f) * table[k] + f * table[(k + 1).clamp(max=len(table) - 1)]
    y0 = pop.grid["bbox_bottom_left_y"]
    radius = 40003200 / 3.1415926535 / 2
    dx = torch.arange(cx, **dev)
    sx = at(sin, torch.clamp(dx - 1, min=0) * step / 2)
    rows = torch.arange(cy, **dev)
    size = 1 << (2 * cx - 1).bit_length()
    spec = torch.fft.rfft(grids, n=size)
    ratio = torch.empty(cy, cx, **dev)
    for yl in range(cy):
        ya = torch.where(rows > yl, torch.full_like(rows, yl + 1), torch.full_like(rows, yl))
        yb = torch.where(rows < yl, rows + 1, rows)
        sy = at(sin, (ya - yb).abs() * step / 2)
        ca, cb = at(cos, (ya * step + y0).abs()), at(cos, (yb * step + y0).abs())
        h = 1000 * (sy[:, None] ** 2 + (ca * cb)[:, None] * sx[None] ** 2)
        K = 1 / (1 + (4 * radius * radius * at(tab, h) / 4000.0 ** 2) ** 1.5)
        G = torch.zeros(cy, size, **dev)
        G[:, :cx] = K
        G[:, size - cx + 1:] = K[:, 1:].flip(1)
        AB = torch.fft.irfft((torch.fft.rfft(G)[None] * spec).sum(1), n=size)[:, :cx]
        ratio[yl] = AB[0] / AB[1]
    return dict(tot_prob=ratio[gy, gx].cpu().numpy(), S0=s0)
