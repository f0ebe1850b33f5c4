"""Performance cases of the engine: what a user's program asks of it, through
its public entry points, from one force evaluation of a small system to
batches of hundreds of replicas.

Four kinds of case:

  forces   one evaluation of every force and energy term on an uploaded state
           (a host program that keeps its own integrator)
  run      a block of MD steps of a batch of replicas, then the snapshot of
           every replica's in-domain atoms and energies: one output interval
           of a simulation
  window   the gradient harness: the ion-vapor objective of a window of MD
           steps and its derivatives by the interaction parameters
  place    the initial placement of the gas and vapor molecules
"""
import functools
import math

import numpy as np
import torch

from md_nucleation_b200 import abi, engine, generate, gradients
from md_nucleation_b200.system import KB, StateArrays, mb_sigma

CHECKED = abi.Q_ALL & ~abi.Q_BLIND_INSERT  # overlapping entries wait for the next rebuild
RI = 110.0                                 # radius of the effective domain with its shell (A)
V_DOMAIN = 4.0 / 3.0 * math.pi * RI ** 3
# chains that grow quickly: number of atoms -> generator seed
CHAINS = {50: 0, 100: 0, 150: 6, 200: 11, 250: 6, 300: 21, 500: 0}
GASES = ("He", "Ar", "N2", "N2monoatomic")
VAPOR_ATOMS = {"methanol": 6, "water": 3}


def listed():
    return [
        # a plugin host: forces and energies of a small cluster on its own coordinates
        dict(name="forces-small", kind="forces", chain=0, gas="N2", vapor="methanol", n_gas=3000, n_vap=40,
             box=260.0, fp64=False),
        # one MD step and its output, the interactive or coupled use: latency of a call
        run_case("step-one", chain=0, gas="He", vapor="methanol", n_gas=2000, n_vap=20, gas_in=135.0, steps=1),
        # an output interval of the smallest production system: Na4Cl3 in helium
        run_case("nacl-single", chain=0, gas="He", vapor="methanol", n_gas=2000, n_vap=20, gas_in=135.0, steps=100),
        # the 150-atom chain in 100,000 rigid N2 at 1e5 Pa
        run_case("chain-single", chain=150, gas="N2", rigid=True, vapor="methanol", n_gas=100_000, n_vap=100,
                 gas_in=135.0, steps=100),
        # the densest domain: 20,000 gas atoms around many vapor molecules
        run_case("dense-single", chain=300, gas="N2", vapor="methanol", n_gas=21_001, n_vap=200, gas_in=9900.0,
                 steps=50),
        # relaxation of a small batch: Nose-Hoover on the ion, energies of every step
        run_case("relax-16", replicas=16, mixed=True, steps=50, energy=2, nvt=abi.NVT_NH),
        # the production batch: 256 uneven replicas, launch tuned once
        run_case("batch-256", replicas=256, mixed=True, steps=100, tune=True),
        # FP64 pair arithmetic, the accuracy runs
        run_case("fp64-8", replicas=8, mixed=True, steps=25, fp64=True),
        # gas-gas LJ on beside the other terms
        run_case("gg-4", replicas=4, chain=50, gas="He", vapor="water", n_gas=2500, n_vap=50, gas_in=900.0, gg=True,
                 steps=50),
        # the large dilute system: 1,000,000 N2 and 1,000 water around a 500-atom chain, several replicas
        run_case("large-8", replicas=8, chain=500, gas="N2", vapor="water", n_gas=1_000_000, n_vap=1000,
                 gas_in=135.0, steps=100),
        # forward and backward of the gradient harness
        dict(name="window-400", kind="window", chain=150, gas="N2", n_gas=20_000, n_vap=20, near=8, steps=400, every=100),
        # the initial placement of the large system
        dict(name="place-large", kind="place", chain=500, n_gas=1_000_000, n_vap=1000, gas_in=135.0),
    ]


def run_case(name=None, replicas=1, mixed=False, chain=0, gas="He", rigid=False, vapor="methanol", n_gas=0, n_vap=0,
             gas_in=0.0, gg=False, fp64=False, steps=100, energy=1, nvt=abi.NVT_OFF, tune=False):
    """mixed: every replica draws its own species and sizes; else all share
    the given ones.  gas_in: gas molecules expected inside the domain, which
    sets the density and with it the box."""
    c = dict(kind="run", replicas=replicas, mixed=mixed, chain=chain, gas=gas, rigid=rigid, vapor=vapor, n_gas=n_gas,
             n_vap=n_vap, gas_in=gas_in, gg=gg, fp64=fp64, steps=steps, energy=energy, nvt=nvt, tune=tune)
    return dict(c, name=name) if name else c


def log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["forces", "single", "single", "batch", "batch", "batch", "gg", "large", "window", "place"])
    chain = rng.choice([0, 0] + list(CHAINS)[:6])
    gas, vapor = rng.choice(GASES), rng.choice(list(VAPOR_ATOMS))
    if kind == "forces":
        return dict(kind="forces", chain=chain, gas=gas, vapor=vapor, n_gas=round(log_uniform(rng, 1500, 12_000)),
                    n_vap=rng.randint(5, 90), box=rng.uniform(245.0, 320.0), fp64=rng.random() < 0.3)
    if kind == "single":
        n_gas = round(log_uniform(rng, 2000, 100_000))
        return run_case(chain=chain, gas=gas, rigid=gas == "N2" and rng.random() < 0.5, vapor=vapor, n_gas=n_gas,
                        n_vap=rng.randint(10, 300), gas_in=log_uniform(rng, 100, min(15_000, 0.45 * n_gas)),
                        steps=round(log_uniform(rng, 1, 120)), energy=rng.randint(0, 2),
                        nvt=rng.choice([abi.NVT_OFF, abi.NVT_OFF, abi.NVT_SCALE, abi.NVT_NH]))
    if kind == "batch":
        return run_case(replicas=round(log_uniform(rng, 2, 192)), mixed=True, steps=round(log_uniform(rng, 5, 80)),
                        energy=rng.randint(0, 2), fp64=rng.random() < 0.15,
                        nvt=rng.choice([abi.NVT_OFF, abi.NVT_OFF, abi.NVT_SCALE, abi.NVT_NH]))
    if kind == "gg":
        return run_case(replicas=rng.randint(1, 8), chain=rng.choice([0, 50, 100]), gas=gas, vapor=vapor,
                        n_gas=round(log_uniform(rng, 1500, 4000)), n_vap=rng.randint(5, 60),
                        gas_in=log_uniform(rng, 150, 700), gg=True, fp64=rng.random() < 0.3,
                        steps=round(log_uniform(rng, 10, 60)))
    if kind == "large":
        return run_case(replicas=rng.randint(1, 6), chain=rng.choice([150, 300, 500]), gas=gas, vapor=vapor,
                        n_gas=round(log_uniform(rng, 150_000, 1_000_000)), n_vap=rng.randint(200, 1000),
                        gas_in=log_uniform(rng, 100, 400), steps=round(log_uniform(rng, 10, 100)))
    if kind == "window":
        return dict(kind="window", chain=rng.choice([50, 100, 150, 200]), gas="N2", n_gas=rng.randint(2000, 30_000),
                    n_vap=rng.randint(8, 40), near=rng.randint(2, 8), steps=rng.randint(60, 400),
                    every=rng.choice([25, 50, 100]))
    return dict(kind="place", chain=chain, n_gas=round(log_uniform(rng, 2000, 1_000_000)), n_vap=rng.randint(10, 1000),
                gas_in=log_uniform(rng, 50, 400))


# --------------------------------------------------------------------------
# systems
# --------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def ion_species(chain):
    if not chain:
        return generate.nacl_cluster()
    return generate.chain(chain, 2.0 if chain >= 500 else 1.0, np.random.default_rng(CHAINS[chain]))


def vapor_species(name):
    return generate.methanol() if name == "methanol" else generate.water()


def box_of(n_gas, gas_in):
    """The edge at which the domain holds gas_in of n_gas molecules; at least
    2.2 domain radii, so that the sphere stays inside the periodic cell."""
    return max(2.2 * RI, (n_gas * V_DOMAIN / gas_in) ** (1.0 / 3.0))


def placer(box, ion_x, n_gas, n_vap, gas_sigma, vapor_sigma, seed, apart):
    """mdn_place, then vapor centres 8 A from each other and gas centres
    `apart` from the vapor (the engine's insertion tests the rest)."""
    sigma = [s * 1e5 for s in (gas_sigma, vapor_sigma)]  # m/s
    gx, gv, vx, vv = engine.place(box, ion_x, int(1.12 * n_gas) + 200, 3 * n_vap + 20, *sigma, seed)
    keep = []
    for i in range(len(vx)):
        if len(keep) < n_vap and (not keep or np.linalg.norm(vx[keep] - vx[i], axis=1).min() >= 8.0):
            keep.append(i)
    vx, vv = vx[keep], vv[keep]
    g = torch.from_numpy(gx).cuda()
    near = torch.zeros(len(gx), dtype=torch.bool, device="cuda")
    for c in torch.from_numpy(vx).cuda().split(64):
        near |= ((g[:, None, :] - c[None]) ** 2).sum(-1).min(dim=1).values < apart * apart
    ok = (~near).cpu().numpy()
    gx, gv = gx[ok][:n_gas], gv[ok][:n_gas]
    if len(gx) < n_gas or len(vx) < n_vap:
        raise RuntimeError("placement came out short")
    return gx, gv, vx, vv


def make_spec(c, seed):
    """One replica of the case."""
    rng = np.random.default_rng(seed)
    ion = ion_species(c["chain"])
    terms = generate.BASE_TERMS | abi.I_SHAKE | (abi.I_AMBER if c["chain"] else abi.I_BMH)
    box = c.get("box") or box_of(c["n_gas"], c["gas_in"])
    dens = c["n_gas"] / box ** 3
    kw = dict(gas_name=c["gas"], n_gas=c["n_gas"], n_vap=c["n_vap"], T=300.0, p=dens * 1e30 * KB * 300.0, dt=1.0,
              seed=int(seed) & 0xFFFFFFFF, shake_h=True, rng=rng, box=box)
    sp = (ion, generate.gas_species(c["gas"], rigid=c.get("rigid", False)), vapor_species(c["vapor"]))
    apart = min(10.0, 0.5 * dens ** (-1.0 / 3.0))
    if c.get("gg"):  # the gas molecules apart from each other too
        return generate.assemble(*sp, interactions=terms | abi.I_GG, min_dist=apart, gas_min_dist=4.0, **kw)
    return generate.assemble(*sp, interactions=terms, placer=functools.partial(placer, apart=apart), **kw)


def mixed_case(rng):
    """The draw of one replica of the production batch: gas, vapor, ion and
    sizes, 500 to 20,000 atoms inside the domain."""
    gas = GASES[int(rng.integers(0, 4))]
    chain = 0 if rng.integers(0, 2) == 0 else list(CHAINS)[int(rng.integers(0, 6))]
    n_gas = int(round(math.exp(rng.uniform(math.log(5000), math.log(100_000)))))
    atoms = math.exp(rng.uniform(math.log(500), math.log(20_000)))
    gas_in = max(50.0, (atoms - (chain or 7)) / (2 if gas == "N2" else 1))
    # the sphere must fit the box: a dense draw takes more molecules
    n_gas = max(n_gas, int(math.ceil(gas_in / V_DOMAIN * (2.2 * RI) ** 3)))
    return dict(chain=chain, gas=gas, vapor=("water", "methanol")[int(rng.integers(0, 2))], n_gas=n_gas,
                n_vap=int(rng.integers(10, 301)), gas_in=gas_in)


def replica_cases(c):
    """The species and sizes of the case's replicas: the same for every seed,
    which sets positions, orientations and velocities."""
    if not c["mixed"]:
        return [c] * c["replicas"]
    rng = np.random.default_rng([c["replicas"], 2])
    return [mixed_case(rng) for _ in range(c["replicas"])]


def rows_of(c):
    """Snapshot rows that hold one replica's domain with room to spare."""
    frac = min(1.0, V_DOMAIN / box_of(c["n_gas"], c["gas_in"]) ** 3)
    most = lambda n: 1.25 * n * frac + 6 * math.sqrt(n * frac) + 20
    return int((c["chain"] or 7) + most(c["n_gas"]) * (2 if c["gas"] == "N2" else 1) +
               most(c["n_vap"]) * VAPOR_ATOMS[c["vapor"]])


# --------------------------------------------------------------------------
# prepare / run
# --------------------------------------------------------------------------
def prepare(case, seed):
    return {"forces": prepare_forces, "run": prepare_run, "window": prepare_window,
            "place": prepare_place}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def prepare_run(c, seed):
    specs = [make_spec(k, 1000 * seed + r) for r, k in enumerate(replica_cases(c))]
    e = engine.Engine(specs, quirks=CHECKED, force_mode=int(c["fp64"]))
    if c["nvt"] != abi.NVT_OFF:
        e.set_nvt_batch(np.full(e.n, c["nvt"], np.int32), np.full(e.n, 300.0))
    if c["tune"]:
        e.tune_launch(40)
    buf = engine.SnapshotBuffer(e.n, sum(rows_of(k) for k in replica_cases(c)))
    for a in (buf.type, buf.x, buf.v):
        a[:] = 0
    return dict(run=run_run, engine=e, buf=buf, steps=c["steps"], energy=c["energy"])


def run_run(s):
    e, buf = s["engine"], s["buf"]
    e.step(s["steps"], s["energy"])
    off = e.snapshot(buf)
    return dict(offset=off, type=Rows.of(buf, buf.type), x=Rows.of(buf, buf.x), v=Rows.of(buf, buf.v), U=buf.U)


class Rows(np.ndarray):
    """The array of a snapshot buffer, keeping the buffer's page-locked memory."""

    @classmethod
    def of(cls, buf, a):
        a = a.view(cls)
        a.buf = buf
        return a


def prepare_window(c, seed):
    """`near` of the vapor molecules start close to the ion, and the list
    margin keeps the window free of a domain rebuild."""
    spec = make_spec(dict(c, vapor="methanol", rigid=True, gas_in=135.0), 1000 * seed)
    rng = np.random.default_rng([seed, 3])
    placed = []
    while len(placed) < c["near"]:
        d = rng.normal(size=3)
        p = d / np.linalg.norm(d) * rng.uniform(8.0, 28.0)
        if np.linalg.norm(spec.ion.x - p, axis=1).min() < 6.0:
            continue
        if placed and np.linalg.norm(np.array(placed) - p, axis=1).min() < 8.0:
            continue
        placed.append(p)
    spec.vapor_x[:c["near"]] = np.array(placed)
    spec.margin = 40.0
    theta, rows = gradients.parameters(spec)
    # the optimiser's current parameters, a few per cent off the start
    theta = theta * torch.from_numpy(1.0 + 0.02 * rng.standard_normal(len(theta)))
    return dict(run=run_window, spec=spec, rows=rows, theta=theta.requires_grad_(), steps=c["steps"], every=c["every"])


def run_window(s):
    J = gradients.window_objective(s["theta"], s["spec"], s["rows"], engine_options=dict(quirks=CHECKED),
                                   n_steps=s["steps"], checkpoint_every=s["every"])
    (g,) = torch.autograd.grad(J, s["theta"])
    return dict(J=J.detach(), grad=g)


def place_args(c, seed):
    rng = np.random.default_rng([seed, 4])
    q = rng.normal(size=(3, 3))
    ion = ion_species(c["chain"]).top.x @ np.linalg.qr(q)[0]
    m = [28.0 / 6.02e23 / 1000, 18.015 / 6.02e23 / 1000]
    sigma = [float(mb_sigma(300.0, k)) * 1e5 for k in m]
    return box_of(c["n_gas"], c["gas_in"]), np.ascontiguousarray(ion), sigma, int(rng.integers(0, 2 ** 62))


def prepare_place(c, seed):
    box, ion, sigma, key = place_args(c, seed)
    return dict(run=run_place, args=(box, ion, c["n_gas"], c["n_vap"], sigma[0], sigma[1], key))


def run_place(s):
    return list(engine.place(*s["args"]))


def forces_system(c, seed):
    """A spec and a state of it made here: every molecule whose centre lies
    in the domain is in, its atoms the template in a random orientation."""
    spec = make_spec(dict(c, rigid=False), 1000 * seed)
    rng = np.random.default_rng([seed, 5])
    s = StateArrays.for_spec(spec)
    s.ion_x[:], s.ion_v[:] = spec.ion.x, spec.ion_v
    ng = spec.n_gas
    s.mol_x[1:1 + ng], s.mol_v[1:1 + ng] = spec.gas_x, spec.gas_v
    s.mol_x[1 + ng:], s.mol_v[1 + ng:] = spec.vapor_x, spec.vapor_v
    m = spec.atom_mass[spec.ion.type]
    com = (spec.ion.x * m[:, None]).sum(0) / m.sum()
    s.mol_x[0] = com
    inside = ((s.mol_x - com) ** 2).sum(1) < RI ** 2
    s.region[:] = inside
    for x, centre, top in ((s.gas_ax, s.mol_x[1:1 + ng], spec.gas), (s.vap_ax, s.mol_x[1 + ng:], spec.vapor)):
        q = rng.normal(size=(len(centre), 3, 3))
        tm = spec.atom_mass[top.type]
        body = top.x - (top.x * tm[:, None]).sum(0) / tm.sum()
        # stretched a little, so that the bonds pull
        x[:] = 1.01 * np.einsum("aj,njk->nak", body, np.linalg.qr(q)[0]) + centre[:, None]
    r = np.linalg.norm(s.vap_ax - com, axis=2)
    s.vap_w[:] = np.where(r < 100, 1.0, np.where(r > RI, 0.0, np.cos(np.pi / 20 * (r - 95.0)) ** 2)).astype(np.float32)
    s.loop_update = 10
    return spec, s


def prepare_forces(c, seed):
    spec, s = forces_system(c, seed)
    e = engine.Engine([spec], quirks=CHECKED, force_mode=int(c["fp64"]))
    e.upload(0, s)
    return dict(run=run_forces, engine=e)


def run_forces(s):
    e = s["engine"]
    e.compute_forces()
    st = e.state(0)
    return dict(ion_f=st.ion_f, gas_f=st.gas_af, vapor_f=st.vap_af, U=e.energies())


# --------------------------------------------------------------------------
# work
# --------------------------------------------------------------------------
def replica_work(c, steps):
    """Bytes and operations of one replica: its in-domain state read and
    written once, its rows of the snapshot written; per step the kick, drift
    and bonds of every atom (30), each core pair (29) and each listed pair of
    a gas atom and a core atom (20), lists of 30 A."""
    ag, av = 2 if c["gas"] == "N2" else 1, VAPOR_ATOMS[c["vapor"]]
    box = c.get("box") or box_of(c["n_gas"], c["gas_in"])
    frac = min(1.0, V_DOMAIN / box ** 3)
    gas, vap = c["n_gas"] * frac, c["n_vap"] * frac
    core = (c["chain"] or 7) + vap * av
    atoms = core + gas * ag
    listed_pairs = c["n_gas"] / box ** 3 * 4.0 / 3.0 * math.pi * 30.0 ** 3 * ag * ((c["chain"] or 7) + vap * ag)
    flops = 30.0 * atoms + 29.0 * core * core / 2 + 20.0 * listed_pairs
    if c.get("gg"):
        flops += 10.0 * gas * ag * gas * ag / V_DOMAIN * 4.0 / 3.0 * math.pi * 30.0 ** 3
    return (144.0 + 52.0) * atoms, flops * steps


def work(case):
    c = case
    if c["kind"] == "place":
        n = c["n_gas"] + c["n_vap"]
        return dict(bytes=48.0 * n, flops=80.0 * n)
    if c["kind"] == "window":
        b, f = replica_work(dict(c, vapor="methanol", gas_in=135.0), c["steps"])
        pairs = 135.0 * 2 * c["chain"] * 0.2 + (c["chain"] + 6.0 * c["near"]) ** 2 / 2
        return dict(bytes=b + 144.0 * c["n_gas"], flops=f + 150.0 * pairs * c["steps"])
    if c["kind"] == "forces":
        b, f = replica_work(c, 1)
        return dict(bytes=b, flops=f)
    parts = [replica_work(k, c["steps"]) for k in replica_cases(c)]
    return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))


# --------------------------------------------------------------------------
# 64-bit values
# --------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "forces":
        return exact_forces(case, seed)
    if case["kind"] == "place":
        return exact_place(case, seed)
    # a trajectory with domain rebuilds, and the gradient of one, have no
    # short plain form
    return None


def philox(c, key):
    """Philox4x32-10 of counters c (four uint32 arrays)."""
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    c = [np.asarray(v, np.uint64) for v in c]
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        lo, sh = np.uint64(0xFFFFFFFF), np.uint64(32)
        c = [(b >> sh) ^ c[1] ^ np.uint64(k0), b & lo, (a >> sh) ^ c[3] ^ np.uint64(k1), a & lo]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return [(v.astype(np.float64) + 0.5) / 4294967296.0 for v in c]


def stream(n, purpose, key):
    i = np.arange(n, dtype=np.uint64)
    one = np.ones(n, np.uint64)
    return philox([i, 0 * i, one * np.uint64(purpose), one * np.uint64(0x706C6163)], key)


def exact_place(c, seed):
    box, ion, sigma, key = place_args(c, seed)
    out, started = [], False
    reach = np.linalg.norm(ion, axis=1).max() + 10.5
    for species, n in ((0, c["n_gas"]), (1, c["n_vap"])):
        x = (np.stack(stream(int(1.2 * n) + 4096, species, key)[:3], 1) - 0.5) * box
        r = np.linalg.norm(x, axis=1)
        ion_ok = np.ones(len(x), bool)
        for k in np.nonzero(r < reach)[0]:
            ion_ok[k] = np.linalg.norm(ion - x[k], axis=1).min() > 10.0
        ok = ion_ok & (r > 10.0)
        if not started:  # the very first molecule is tested against the ion alone
            ok[np.nonzero(ion_ok)[0][0]] = True
            started = True
        u = stream(n, 2 + species, key)
        z = [np.sqrt(-2 * np.log(u[0])) * f(2 * np.pi * u[1]) for f in (np.cos, np.sin)]
        z.append(np.sqrt(-2 * np.log(u[2])) * np.cos(2 * np.pi * u[3]))
        out += [x[ok][:n], sigma[species] * np.stack(z, 1) * 1e-5]
    return out


BORN = {  # rho A, 6 C, 8 D, sigma, rho (Tosi-Fumi NaCl)
    (0, 0): (25.4435, 101.1719, 48.1771, 2.340), (0, 1): (20.3548, 674.4793, 837.077, 2.755),
    (1, 0): (20.3548, 674.4793, 837.077, 2.755), (1, 1): (15.2661, 6985.6786, 14031.5785, 3.170)}


def bonded(x, top, spec):
    """Forces and (bond + angle, dihedral) energies of one molecule [n, 3] or
    many [m, n, 3] by automatic differentiation."""
    x = torch.from_numpy(np.array(x)).requires_grad_()
    at = lambda k, rows: x[..., torch.from_numpy(np.asarray(rows)[:, k].astype(np.int64)), :]
    zero = x.sum() * 0.0
    ea, ed = zero, zero
    if len(top.bonds):
        co = torch.from_numpy(spec.bond_coeff[top.bonds[:, 2]])
        ea = ea + (co[:, 0] * ((at(0, top.bonds) - at(1, top.bonds)).norm(dim=-1) - co[:, 1]) ** 2).sum()
    if len(top.angles):
        co = torch.from_numpy(spec.angle_coeff[top.angles[:, 3]])
        a, b = at(0, top.angles) - at(1, top.angles), at(2, top.angles) - at(1, top.angles)
        th = torch.acos((a * b).sum(-1) / (a.norm(dim=-1) * b.norm(dim=-1)))
        ea = ea + (co[:, 0] * (th - co[:, 1]) ** 2).sum()
    if len(top.dihedrals):
        d = top.dihedrals
        b1, b2, b3 = at(0, d) - at(1, d), at(2, d) - at(1, d), at(3, d) - at(2, d)
        a, b = torch.linalg.cross(b1, -b2), torch.linalg.cross(b3, -b2)
        phi = torch.atan2(b2.norm(dim=-1) * (a * b3).sum(-1), (a * b).sum(-1))
        for k in range(3):
            co = torch.from_numpy(spec.dihedral_coeff[d[:, 4], 5 * k:5 * k + 5])
            on = torch.from_numpy((spec.dihedral_multi[d[:, 4]] > k).astype(np.float64))
            ed = ed + (on * co[:, 0] * (1 + torch.cos(co[:, 1] * phi - co[:, 2] * math.pi / 180))).sum()
    (g,) = torch.autograd.grad(ea + ed, x)
    return -g.numpy(), float(ea.detach()), float(ed.detach())


def lj(spec, xa, ta, xb, tb, on, qa=None, qb=None, wa=None, wb=None):
    """LJ (+ Coulomb) of the marked pairs: forces on a, on b, energy.  The
    taper weights scale the force, not the energy."""
    eps = np.sqrt(np.outer(spec.atom_eps, spec.atom_eps))[np.ix_(ta, tb)]
    sig = (0.5 * (spec.atom_sigma[:, None] + spec.atom_sigma[None]))[np.ix_(ta, tb)]
    d = xa[:, None] - xb[None]
    r2 = np.where(on, (d ** 2).sum(-1), 1.0)
    s6 = (sig ** 2 / r2) ** 3
    f, e = 24 * eps * s6 * (2 * s6 - 1) / r2, 4 * eps * s6 * (s6 - 1)
    if qa is not None:
        kq = 1.602e-19 ** 2 / 4 / np.pi / 8.85e-12 * 6.02e23 * 1e10 / 4184 * np.outer(qa, qb) / np.sqrt(r2)
        f, e = f + kq / r2, e + kq
    f = np.where(on, f * (1.0 if wa is None else np.outer(wa, wb)), 0.0)
    F = f[..., None] * d
    return F.sum(1), -F.sum(0), float(np.where(on, e, 0.0).sum())


def exact_forces(c, seed):
    spec, s = forces_system(c, seed)
    ni, ng, ag, av = spec.ion.n, spec.n_gas, spec.gas.n, spec.vapor.n
    gin, vin = np.nonzero(s.region[1:1 + ng])[0], np.nonzero(s.region[1 + ng:])[0]
    X, G, V = s.ion_x, s.gas_ax[gin], s.vap_ax[vin]
    ti, tg, tv = spec.ion.type, spec.gas.type, spec.vapor.type
    ml2 = (spec.cutoff + spec.margin) ** 2
    U = np.zeros(8)
    fi, fg, fv = np.zeros_like(X), np.zeros_like(G), np.zeros_like(V)
    nv = len(vin)
    Vf, Tv, Qv, Wv = V.reshape(-1, 3), np.tile(tv, nv), np.tile(spec.vapor.charge, nv), s.vap_w[vin].reshape(-1)
    mol = np.repeat(np.arange(nv), av)
    gc, vc = s.mol_x[1 + gin], s.mol_x[1 + ng + vin]
    # gas with the ion: atoms of every gas molecule whose centre is near the ion atom
    near = ((gc[:, None] - X[None]) ** 2).sum(-1) < ml2
    for a in range(ag):
        f, r, e = lj(spec, G[:, a], np.full(len(G), tg[a]), X, ti, near)
        fg[:, a] += f
        fi += r
        U[abi.U_GI] += e
    # gas with the vapor: the partner loop runs over as many vapor atoms as a gas molecule has
    if nv:
        near = ((gc[:, None] - vc[None]) ** 2).sum(-1) < ml2
        for a in range(ag):
            for b in range(min(ag, av)):
                f, r, e = lj(spec, G[:, a], np.full(len(G), tg[a]), V[:, b], np.full(nv, tv[b]), near)
                fg[:, a] += f
                fv[:, b] += r
                U[abi.U_VG] += e
        f, r, e = lj(spec, X, ti, Vf, Tv, np.ones((ni, len(Vf)), bool), spec.ion.charge, Qv, np.ones(ni), Wv)
        fi += f
        fv += r.reshape(fv.shape)
        U[abi.U_VI] += e
        f, r, e = lj(spec, Vf, Tv, Vf, Tv, np.triu(mol[:, None] != mol[None]), Qv, Qv, Wv, Wv)
        fv += (f + r).reshape(fv.shape)
        U[abi.U_VV] += e
    # the ion
    if spec.interactions & abi.I_AMBER:
        ex = np.zeros((ni, ni), bool)
        for rows, k in ((spec.ion.bonds, 1), (spec.ion.rigid, 1), (spec.ion.angles, 2), (spec.ion.dihedrals, 3)):
            ex[rows[:, 0], rows[:, k]] = ex[rows[:, k], rows[:, 0]] = True
        q = spec.ion.charge
        f, r, e = lj(spec, X, ti, X, ti, np.triu(~ex, 1), q, q)
        fi += f + r
        fb, ea, ed = bonded(X, spec.ion, spec)
        fi += fb
        U[abi.U_ION] += e + ea + ed
    if spec.interactions & abi.I_BMH:
        kq = 1.602e-19 ** 2 / 4 / np.pi / 8.85e-12 * 6.02e23 * 1e10 / 4184
        for i in range(ni):
            for j in range(i + 1, ni):
                A, Cc, D, sg = BORN[int(spec.ion_bmh_type[i]), int(spec.ion_bmh_type[j])]
                d = X[i] - X[j]
                r = np.sqrt(d @ d)
                ex = math.exp(3.1546 * (sg - r))
                qq = kq * spec.ion.charge[i] * spec.ion.charge[j] / r
                f = (A * 3.1546 / 4.184 * 3.1546 * r * ex - (6 * Cc / r ** 6 + 8 * D / r ** 8) / 4.184 + qq) / r ** 2 * d
                fi[i] += f
                fi[j] -= f
                U[abi.U_ION] += qq + A * 3.1546 / 4.184 * ex - (Cc / r ** 6 + D / r ** 8) / 4.184
    # inside the gas and vapor molecules (vapor bonds and angles are booked
    # with the gas, vapor dihedrals with the ion)
    f, ea, _ = bonded(G, spec.gas, spec)
    fg += f
    U[abi.U_GAS] += ea
    if nv:
        f, ea, ed = bonded(V, spec.vapor, spec)
        fv += f
        U[abi.U_GAS] += ea
        U[abi.U_ION] += ed
    out = dict(ion_f=fi, gas_f=np.zeros_like(s.gas_ax), vapor_f=np.zeros_like(s.vap_ax), U=U[None])
    out["gas_f"][gin], out["vapor_f"][vin] = fg, fv
    return out
