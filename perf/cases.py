"""What the performance measurements of this framework run.

A case is a plain dict.  `path` names the work; the other keys are its size and options:

sweep      a block of Monte Carlo sweeps followed by what a run's save interval takes: the statistics and the
           configuration, copied into pinned host arrays (GBSystem.sweep / stats / download).  One system
           ("replicas" 1) or a batch of independent replicas of uneven size, temperature and pressure.
roundtrip  the drop-in seam: the caller's arrays and running energy go up, one sweep runs, the arrays come back.
energy     tot_ene, the FP64 total energy of a configuration.
fit        one call of Surrogate.fit (forward and backward passes and Adam on recorded volume-move samples).
predict    Surrogate.predict on many feature rows (forward only).
"""
import math

import numpy as np
import torch

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc
from parellel_mc_mpi_for_liquidcrystalsystems_b200 import _lib, da

SWEEP = dict(path="sweep", replicas=1, ensemble="nvt", precision="fp32", grid="even", density=0.30, temperature=0.9,
             pressure=2.0, colloid=0.0, screen="none")
HIDDEN = 128
RELAX = 20  # sweeps from the lattice start before a state is handed over


def listed():
    return [
        # the smallest system of use: the 1000-rod validation run in FP64, a parity check's size
        dict(SWEEP, name="nvt_fp64_1000", n=1000, precision="fp64", temperature=1.0, sweeps=4),
        # FP64 sweeps of a mid-size system: the mode results are validated with
        dict(SWEEP, name="nvt_fp64_8192", n=8192, precision="fp64", temperature=1.0, sweeps=4),
        # a small production system: many short launches per sweep, odd cell counts
        dict(SWEEP, name="nvt_fp32_4096", n=4096, grid="fine", density=0.32, temperature=0.8, sweeps=50),
        # colloid in a liquid crystal at constant pressure, plain volume moves
        dict(SWEEP, name="npt_colloid_32768", n=32768, ensemble="npt", colloid=5.0, sweeps=50),
        # the same physics at 262,144 rods, volume moves screened by the FP32-pair energy change
        dict(SWEEP, name="npt_screen_262144", n=262144, ensemble="npt", colloid=8.0, density=0.28, temperature=0.85,
             screen="fp32", sweeps=20),
        # ... and screened by the network (features, two GEMMs, exact energies for what passes)
        dict(SWEEP, name="npt_learned_262144", n=262144, ensemble="npt", colloid=8.0, density=0.28, temperature=0.85,
             screen="learned", sweeps=20),
        # the largest system: a million rods on the nematic side
        dict(SWEEP, name="nvt_fp32_1048576", n=1048576, density=0.32, temperature=0.8, sweeps=10),
        # a parameter scan: 64 independent replicas swept in one graph
        dict(SWEEP, name="batch_64", n=16384, replicas=64, ensemble="mixed", grid="fine", density=0.32,
             temperature=1.0, colloid=4.5, screen="fp32", sweeps=4),
        # a host program that keeps its own arrays and calls in for every sweep
        dict(SWEEP, path="roundtrip", name="roundtrip_1048576", n=1048576, density=0.32, temperature=0.8, sweeps=1),
        # the energy check of a million rods
        dict(path="energy", name="energy_1048576", n=1048576, density=0.30, colloid=0.0),
        # the screen's training on a run's recorded samples, and its use on many rows at once
        dict(path="fit", name="fit_2048", rows=2048, batch=256, epochs=1),
        dict(path="predict", name="predict_4096", rows=4096, batch=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, odd ones among them."""
    path = rng.choice(["sweep"] * 7 + ["batch", "roundtrip", "energy", "fit", "predict"])
    if path == "fit":
        batch = rng.choice([128, 200, 256, 512])
        return dict(path="fit", rows=batch * rng.randint(2, 8), batch=batch, epochs=1)
    if path == "predict":
        return dict(path="predict", rows=_log_int(rng, 64, 4096), batch=rng.choice([128, 512]))
    density, temperature = round(rng.uniform(0.28, 0.33), 4), round(rng.uniform(0.7, 1.3), 3)
    if path == "energy":
        return dict(path="energy", n=_log_int(rng, 2000, 1048576), density=density,
                    colloid=round(rng.uniform(2.0, 4.0), 2) if rng.random() < 0.5 else 0.0)
    if path == "roundtrip":
        return dict(SWEEP, path="roundtrip", n=_log_int(rng, 30000, 1048576), density=density, temperature=temperature,
                    sweeps=1)
    if path == "batch":
        return dict(SWEEP, n=_log_int(rng, 4000, 12000), replicas=rng.choice([8, 13, 24, 48]), ensemble="mixed",
                    grid="fine", density=density, temperature=temperature, colloid=round(rng.uniform(3.0, 5.0), 2),
                    screen=rng.choice(["none", "fp32"]), sweeps=4)
    kind = rng.choice(["fp64", "nvt", "nvt", "npt", "npt"])
    if kind == "fp64":
        return dict(SWEEP, n=_log_int(rng, 1000, 12000), precision="fp64", density=density, temperature=temperature,
                    grid=rng.choice(["even", "fine"]), sweeps=1)
    if kind == "nvt":
        n = _log_int(rng, 4000, 1000000)
        return dict(SWEEP, n=n, density=density, temperature=temperature, grid="fine" if n < 20000 else "even",
                    sweeps=10)
    n = _log_int(rng, 20000, 262144)
    return dict(SWEEP, n=n, ensemble="npt", density=density, temperature=temperature, colloid=round(rng.uniform(3, 8), 2),
                pressure=round(rng.uniform(1.5, 2.5), 2), grid="fine" if n < 30000 else "even",
                screen=rng.choice(["none", "fp32", "learned"]), sweeps=10)


# ---------------------------------------------------------------------------
# sweeps
# ---------------------------------------------------------------------------

def _params(case, seed):
    """The parameters of every replica of a case."""
    rng = np.random.default_rng(1000003 * (seed % 1000003) + case["n"])
    ps = []
    for r in range(case["replicas"]):
        n, T, rho, P, R = case["n"], case["temperature"], case["density"], case["pressure"], case["colloid"]
        npt = case["ensemble"] == "npt"
        if case["ensemble"] == "mixed":  # half NVT, half NPT, a third with a colloid, N over a factor of 16
            n = int(round(n * 4.0 ** ((r + 0.5) / case["replicas"] * 2.0 - 1.0)))
            T, rho, P = T * rng.uniform(0.75, 1.25), rho * rng.uniform(0.95, 1.03), P * rng.uniform(0.75, 1.25)
            R = R * rng.uniform(0.67, 1.33) if r % 3 == 0 else 0.0
            npt = r % 2 == 1
        ps.append(lcmc.default_params(
            mc_ensemble_type=2 if npt else 1, num_particles=n, system_density=rho, system_temperature=T,
            system_pressure=P, colloid_radius=R, colloid_wall_option=1 if R > 0 else 0, npt_max_dlnV=0.01,
            gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0, gb_nu_exponent=1.0, cutoff_radius=4.0,
            max_displacement=0.1, max_rotation=0.1, init_lattice=1, init_orientation_cone_deg=20.0,
            cell_grid=1 if case["grid"] == "fine" else 0, precision_mode=1 if case["precision"] == "fp32" else 0,
            rng_seed=seed * 4096 + r + 1))
    return ps


def _sweep(s, k):
    """k sweeps, going on over an energy-check notice (the chain is unchanged by it)."""
    try:
        s.sweep(k)
    except lcmc.LcmcError as e:
        if e.code != _lib.EDRIFT:
            raise
        s.clear_error_flags()


def _pinned(n):
    t = torch.empty(n, dtype=torch.float64, pin_memory=True)
    return t, t.numpy()


def _prepare_sweep(case, seed):
    ps = _params(case, seed)
    s = lcmc.GBSystem(ps)
    for r in range(len(ps)):
        s.get_initial_config(r)
    keep = None
    if case["screen"] == "fp32":
        s.set_fp32_screen(True)
    elif case["screen"] == "learned":
        keep = da.Surrogate(max_batch=128, seed=seed + 1)
        s.set_surrogate(keep)
    _sweep(s, RELAX)
    total = sum(p.num_particles for p in ps)
    own = [_pinned(total) for _ in range(6)]
    views, at = [], 0
    for p in ps:
        views.append([a[at:at + p.num_particles] for _, a in own])
        at += p.num_particles
    state = dict(case=case, system=s, own=own, views=views, keep=keep, box=None, energy=0.0)
    if case["path"] == "roundtrip":
        _, state["box"] = s.download(out=views[0])
        state["energy"] = s.stats()["energy"]
    return state


def _run_sweep(state):
    s, views = state["system"], state["views"]
    _sweep(s, state["case"]["sweeps"])
    boxes, energies, accepted = [], [], []
    for r in range(s.n_replicas):
        st = s.stats(r)
        _, box = s.download(replica=r, out=views[r])
        boxes.append(box)
        energies.append(st["energy"])
        accepted.append(st["accepted"])
    return {"arrays": [a for _, a in state["own"]], "box": np.array(boxes), "energy": np.array(energies),
            "accepted": np.array(accepted)}


def _run_roundtrip(state):
    s, arrays = state["system"], state["views"][0]
    s.upload(*arrays, state["box"], energy=state["energy"])
    _sweep(s, 1)
    _, state["box"] = s.download(out=arrays)
    st = s.stats()
    state["energy"] = st["energy"]
    return {"arrays": arrays, "energy": np.array([st["energy"]]), "accepted": np.array([st["accepted"]])}


# ---------------------------------------------------------------------------
# energy
# ---------------------------------------------------------------------------

def _configuration(case, seed):
    """A body-centred layered configuration with thermal disorder, made with torch alone: six arrays and the box edge.
    Layers 1.05 rod lengths apart along z, rods near z; with a colloid, the rods around it are left out."""
    n, R = case["n"], case["colloid"]
    L = (n / case["density"] + 4.0 / 3.0 * 3.1415926535898 * R ** 3) ** (1.0 / 3.0)
    nz = max(1, int(math.floor(L / 3.15)))
    na = 1
    while True:
        s = torch.arange(2 * na * na * nz, dtype=torch.int64)
        b, q = s & 1, s >> 1
        xyz = torch.stack([(q % na + 0.5 * b) * (L / na), ((q // na) % na + 0.5 * b) * (L / na),
                           (q // (na * na) + 0.5 * b) * (L / nz)])
        if R > 0:
            xyz = xyz[:, ((xyz - 0.5 * L).abs() ** 2).sum(0) > (R + 1.2) ** 2]
        if xyz.shape[1] >= n:
            break
        na = max(na + 1, int(math.sqrt(n / (2.0 * nz)) * 0.98))
    m = xyz.shape[1]
    f = torch.arange(m, dtype=torch.int64)
    xyz = xyz[:, ((f + 1) * n) // m > (f * n) // m].double()
    g = torch.Generator().manual_seed(seed)
    xyz = xyz + 0.04 * (2.0 * torch.rand(3, n, generator=g, dtype=torch.float64) - 1.0)
    xyz = torch.remainder(xyz, L).clamp_(0.0, L)
    ct = 1.0 - torch.rand(n, generator=g, dtype=torch.float64) * (1.0 - math.cos(math.radians(8.0)))
    ph = 2.0 * math.pi * torch.rand(n, generator=g, dtype=torch.float64)
    st = torch.sqrt(1.0 - ct * ct)
    return [t.contiguous().numpy() for t in (xyz[0], xyz[1], xyz[2], st * torch.cos(ph), st * torch.sin(ph), ct)], L


def _prepare_energy(case, seed):
    arrays, L = _configuration(case, seed)
    p = lcmc.default_params(num_particles=case["n"], system_density=case["density"], colloid_radius=case["colloid"],
                            colloid_wall_option=1 if case["colloid"] > 0 else 0, max_displacement=0.1, rng_seed=seed + 1)
    s = lcmc.GBSystem(p)
    s.upload(*arrays, np.array([L, L, L]), energy=0.0)
    return dict(case=case, system=s)


def _pair_sum(x, u, L, lo, hi, start, count, nc):
    """Sum of the Gay-Berne terms (kappa 3, kappa' 5, mu 2, nu 1, rc 4) of particles [lo, hi) of the cell-sorted arrays
    with every neighbour, each pair seen from both sides."""
    chi, chip = 0.8, (math.sqrt(5.0) - 1.0) / (math.sqrt(5.0) + 1.0)
    i = torch.arange(lo, hi, device=x.device)
    c = ((x[lo:hi] / (L / nc)).floor().long()).clamp_(0, nc - 1)
    total = torch.zeros((), dtype=torch.float64, device=x.device)
    width = int(count.max())
    seen = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                key = ((dx % nc), (dy % nc), (dz % nc))
                if key in seen:  # fewer than three cells per axis
                    continue
                seen.append(key)
                cell = ((c[:, 2] + dz) % nc * nc + (c[:, 1] + dy) % nc) * nc + (c[:, 0] + dx) % nc
                k = torch.arange(width, device=x.device)
                j = (start[cell][:, None] + k).clamp_(max=x.shape[0] - 1)
                on = (k < count[cell][:, None]) & (j != i[:, None])
                d = x[j] - x[lo:hi, None]
                d = d - L * torch.round(d / L)
                r2 = (d * d).sum(-1)
                a, b = torch.nonzero(on & (r2 < 16.0), as_tuple=True)
                d, r = d[a, b], torch.sqrt(r2[a, b])
                e1, e2 = u[lo:hi][a], u[j[a, b]]
                cc = (e1 * e2).sum(-1)
                p, q = (d * e1).sum(-1) / r, (d * e2).sum(-1) / r
                ps, ms = (p + q) ** 2, (p - q) ** 2
                eps = (1.0 - 0.5 * chip * (ps / (1.0 + chip * cc) + ms / (1.0 - chip * cc))) ** 2 / torch.sqrt(
                    1.0 - chi * chi * cc * cc)
                sig = 1.0 / torch.sqrt(1.0 - 0.5 * chi * (ps / (1.0 + chi * cc) + ms / (1.0 - chi * cc)))
                D = r - sig + 1.0
                w = (1.0 / D) ** 6
                total = total + torch.where(D < 0.001, torch.full_like(D, 1e9), 4.0 * eps * w * (w - 1.0)).sum()
    return 0.5 * total


def _exact_energy(case, seed):
    arrays, L = _configuration(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.tensor(np.stack(arrays[:3], 1), device=dev)
    u = torch.tensor(np.stack(arrays[3:], 1), device=dev)
    u = u / u.norm(dim=1, keepdim=True)
    nc = max(1, int(math.floor(L / 4.0)))
    c = ((x / (L / nc)).floor().long()).clamp_(0, nc - 1)
    cell = (c[:, 2] * nc + c[:, 1]) * nc + c[:, 0]
    order = torch.argsort(cell, stable=True)
    x, u, cell = x[order], u[order], cell[order]
    count = torch.bincount(cell, minlength=nc ** 3)
    start = torch.cumsum(count, 0) - count
    total = sum(_pair_sum(x, u, L, lo, min(lo + 65536, len(x)), start, count, nc) for lo in range(0, len(x), 65536))
    R = case["colloid"]
    if R > 0:  # rod of length 3 at a sphere of radius R in the box centre, cut 12 beyond its surface
        d = x - 0.5 * L
        r = d.norm(dim=1)
        d, r, v = d[r - R <= 12.0], r[r - R <= 12.0], u[r - R <= 12.0]
        s2 = 1.0 - ((d * v).sum(1) / r) ** 2
        chi, chip = 0.8, (math.sqrt(5.0) - 1.0) / (math.sqrt(5.0) + 1.0)
        eps = 5.0 * ((1.0 - chip) / (1.0 - chip * s2)) ** 2
        D = r - R - torch.sqrt((1.0 - chi * s2) / (1.0 - chi)) + 1.0
        w = eps * (1 / (45 * D ** 9) - 1 / (6 * D ** 3) - 1 / (40 * r * D ** 8) + 1 / (4 * r * D ** 2))
        total = total + torch.where(D <= 1e-10, torch.full_like(D, 1e8), w).sum()
    return {"energy": np.array([float(total)])}


# ---------------------------------------------------------------------------
# the volume-move surrogate
# ---------------------------------------------------------------------------

def _features(rows, seed):
    """Feature rows like those recorded in a run: 8 pooled channels of 8^3 cells around their bulk values, and |d ln V|."""
    g = torch.Generator().manual_seed(seed)
    mean = torch.tensor([1.0, 0.2, 0.0, 0.0, 0.2, 0.0, 0.35, 1.05]).repeat_interleave(512)
    x = torch.empty(rows, 4097)
    x[:, :4096] = mean + 0.1 * torch.randn(rows, 4096, generator=g)
    x[:, 4096] = torch.rand(rows, generator=g)
    slope = 40.0 * (x[:, :512].mean(1) - 1.0) + x[:, 4096] - 0.5 + 0.05 * torch.randn(rows, generator=g)
    return x.contiguous().numpy(), slope.double().numpy()


def _weights(seed):
    """All parameters of the network in the C ABI's order, W1 with its columns padded to 4224."""
    g = torch.Generator().manual_seed(seed + 77)
    def uniform(rows, cols):
        return math.sqrt(6.0 / (rows + cols)) * (2.0 * torch.rand(rows, cols, generator=g) - 1.0)
    W1 = torch.zeros(HIDDEN, 4224)
    W1[:, :4097] = uniform(HIDDEN, 4097)
    return [W1, 0.1 * uniform(HIDDEN, 1)[:, 0], uniform(HIDDEN, HIDDEN), 0.1 * uniform(HIDDEN, 1)[:, 0],
            uniform(1, HIDDEN)[0], torch.zeros(1)]


def _prepare_net(case, seed):
    net = da.Surrogate(max_batch=case["batch"], seed=seed + 1)
    w = torch.cat([t.reshape(-1) for t in _weights(seed)]).contiguous().numpy()
    for _ in range(2):  # the second call finds the weights in place, however the first one's copy was ordered
        _lib.check(_lib.lib().lcmc_mlp_set_params(net.handle, w.ctypes.data_as(_lib.FP)))
        torch.cuda.synchronize()
    x, slope = _features(case["rows"], seed)
    return dict(case=case, net=net, x=x, slope=slope, params=np.empty_like(w))


def _run_fit(state):
    net, case = state["net"], state["case"]
    loss = net.fit(state["x"], state["slope"], epochs=case["epochs"], batch=case["batch"])
    _lib.check(_lib.lib().lcmc_mlp_get_params(net.handle, state["params"].ctypes.data_as(_lib.FP)))
    return {"loss": np.array([loss], dtype=np.float32), "params": state["params"]}


def _exact_predict(case, seed):
    W1, b1, W2, b2, w3, b3 = [t.double() for t in _weights(seed)]
    x = torch.from_numpy(_features(case["rows"], seed)[0]).double()
    h = torch.nn.functional.silu(x @ W1[:, :4097].T + b1)
    h = torch.nn.functional.silu(h @ W2.T + b2)
    return {"slope": (h @ w3 + b3).numpy()}


# ---------------------------------------------------------------------------

def prepare(case, seed):
    if case["path"] == "energy":
        return _prepare_energy(case, seed)
    if case["path"] in ("fit", "predict"):
        return _prepare_net(case, seed)
    return _prepare_sweep(case, seed)


def run(state):
    path = state["case"]["path"]
    if path == "sweep":
        return _run_sweep(state)
    if path == "roundtrip":
        return _run_roundtrip(state)
    if path == "energy":
        return {"energy": np.array([state["system"].tot_ene()])}
    if path == "fit":
        return _run_fit(state)
    return {"slope": state["net"].predict(state["x"])}


def exact(case, seed):
    """Values in 64 bits without this package.  A sweep has none: its moves depend on every rounding before them."""
    if case["path"] == "energy":
        return _exact_energy(case, seed)
    if case["path"] == "predict":
        return _exact_predict(case, seed)
    return None


def work(case):
    """Bytes and operations of one pass: a configuration read and written once (48 bytes a rod); per attempt the pairs
    inside the cutoff, old and new state, 8 operations for the distance and 61 for the Gay-Berne term each; per volume
    move the pairs of both volumes."""
    if case["path"] in ("fit", "predict"):
        rows = case["rows"] * case.get("epochs", 1)
        weights = HIDDEN * 4097 + HIDDEN * HIDDEN
        steps = case["rows"] // case["batch"] * case.get("epochs", 0)
        return {"bytes": 4.0 * rows * 4097 + 16.0 * weights * steps,
                "flops": 2.0 * weights * rows * (2 if case["path"] == "fit" else 1)}
    n = float(case["n"])
    if case.get("ensemble") == "mixed":
        n = float(sum(p.num_particles for p in _params(case, 0)))
    pairs = case["density"] * 4.0 / 3.0 * math.pi * 64.0
    if case["path"] == "energy":
        return {"bytes": 48.0 * n, "flops": n * 0.5 * pairs * 69.0}
    volume = {"nvt": 0.0, "npt": 1.0, "mixed": 0.5}[case["ensemble"]]
    flops = n * case["sweeps"] * pairs * 69.0 * (2.0 + volume)
    return {"bytes": 96.0 * n, "flops": flops}
