"""Performance cases of the constant-pH Monte Carlo engine: what a program that uses the
library has it do, through its public entry points.

Systems are grafted weak-polyelectrolyte brushes in a slab (walls at 0 and H, box padded to
3 H), in the model of `configs.native_params`: WCA + FENE chains on a square lattice, explicit
ions, SPME.  Particle numbers, box sizes, meshes, salt, pH and move mixes span those of the
repository's configurations (16 chains of 20 beads to 144 chains of 50; 0.5k to 20k particles;
1 to 256 replicas).  Chains start as stretched helices about their graft points and ions on
free lattice sites, so that no pair overlaps.

Energies are handed back in single precision: the engine's pair and mesh terms are FP32 (its
FP64 is what they are added in), as are the energies of the programs that call it.  Positions
and charges are FP32, types, flags and counters whole numbers.
"""
import math

import numpy as np
import torch

from ph_brush_b200 import Engine, Surrogate, SystemArrays, _abi, configs

CHARGED, NEUTRAL, ANION, CATION, PERMANENT = 1, 0, 2, 3, 4
SITES = (1.0 / 1.2) ** 3  # lattice sites per sigma^3 that an ion may start on


def listed():
    return [
        # one small replica followed on its own, 16 chains of 20 beads: a trial's latency
        dict(name="chain_small", kind="run", replicas=1, side=4, spacing=4.0, length=20, permanent=0, height=40.0,
             salt=0.002, pH=7.5, swap=0.0, order=5, mesh=32, depth=128, tuned=0, trials=250),
        # one large replica without batching, 100 chains of 50 titratable beads, ~12k particles
        dict(name="chain_12k", kind="run", replicas=1, side=10, spacing=4.0, length=50, permanent=0, height=100.0,
             salt=0.0075, pH=6.5, swap=0.0, order=5, mesh=64, depth=384, tuned=0, trials=400),
        # the production sweep: 256 diblock replicas over pH and salt in one engine, tuned
        dict(name="sweep_256", kind="run", replicas=256, side=12, spacing=4.0, length=50, permanent=20, height=60.0,
             salt=0.012, pH=7.0, swap=0.0, order=5, tuned=1, trials=400),
        # a sweep of uneven replicas: several grafting densities, lengths and mesh depths, as created
        dict(name="sweep_uneven", kind="run", replicas=24, side=8, spacing=2.7, length=57, permanent=0, height=67.0,
             salt=0.006, pH=6.0, swap=0.0, order=5, tuned=0, trials=300),
        # reservoir salt swaps and titration with the learned first stage of delayed acceptance
        dict(name="reservoir_da", kind="run", replicas=8, side=10, spacing=4.0, length=50, permanent=0, height=100.0,
             salt=0.0075, pH=7.0, swap=0.05, order=5, mesh=64, depth=384, tuned=0, trials=200, surrogate=1),
        # states uploaded from pinned memory, a short run, states read back: a driver that
        # exchanges configurations between steps
        dict(name="exchange_64", kind="exchange", replicas=64, side=11, spacing=4.0, length=50, permanent=20,
             height=60.0, salt=0.012, pH=7.0, swap=0.0, order=5, tuned=1, trials=100),
        # energies of given configurations: one of 12k particles, and a batch of 64
        dict(name="energy_12k", kind="energy", replicas=1, side=10, spacing=4.0, length=50, permanent=0, height=100.0,
             salt=0.0075, pH=6.5, order=5, mesh=64, depth=384),
        dict(name="energy_batch", kind="energy", replicas=64, side=9, spacing=4.0, length=50, permanent=20,
             height=60.0, salt=0.006, pH=7.0, order=5),
        # many trial moves of one configuration judged at once (insertion scans, training data)
        dict(name="scan_512", kind="scan", replicas=1, side=10, spacing=4.0, length=50, permanent=0, height=100.0,
             salt=0.0075, pH=6.5, order=5, mesh=64, depth=384, trials=512),
        # a caller's own Monte Carlo loop: one trial judged, then committed, four times over
        dict(name="host_loop", kind="loop", replicas=1, side=4, spacing=4.0, length=20, permanent=0, height=40.0,
             salt=0.002, pH=7.5, order=5, mesh=32, depth=128, trials=4),
        # loss and gradient of the learned first stage on one training batch
        dict(name="surrogate_grad", kind="grad", samples=4096, hidden=128),
        # the swap phase of the reference's driver on the device, in its own model (no walls, LJ 3 sigma)
        dict(name="swap_phase", kind="phase2", replicas=1, side=10, spacing=4.0, length=50, permanent=0, height=100.0,
             salt=0.0075, pH=7.0, order=4, trials=100),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["run", "run", "batch", "batch", "exchange", "energy", "scan", "loop", "grad", "phase2"])
    if kind == "grad":
        return dict(kind="grad", samples=int(_log(rng, 96, 8192)) | 1, hidden=rng.choice([64, 128]))
    side = rng.randint(4, 11)
    length = rng.randint(20, 55)
    c = dict(kind=kind, replicas=1, side=side, spacing=round(rng.uniform(2.7, 4.5), 2), length=length,
             permanent=rng.choice([0, 0, min(20, length // 2)]), height=float(length + rng.randint(8, 30)),
             salt=round(_log(rng, 0.0005, 0.015), 5), pH=round(rng.uniform(5.0, 9.0), 2), order=rng.choice([5, 5, 5, 4, 6]))
    if kind in ("run", "batch", "exchange"):
        c["swap"] = rng.choice([0.0, 0.0, 0.05])
        c["tuned"] = 0
        if kind != "run":
            c["replicas"] = int(_log(rng, 3, 96))
            c["tuned"] = rng.randint(0, 1)
        c["trials"] = int(_log(rng, 20, 400)) | 1
        c["kind"] = "exchange" if kind == "exchange" else "run"
        if kind == "run" and rng.random() < 0.3:
            c["surrogate"] = 1
    elif kind == "energy":
        c["replicas"] = int(_log(rng, 1, 40))
    elif kind == "scan":
        c["trials"] = int(_log(rng, 5, 512))
    elif kind == "loop":
        c["trials"] = rng.randint(1, 6)
    else:
        c.update(order=4, permanent=0, trials=rng.randint(20, 120))
    return c


# ---------------------------------------------------------------------------
# systems
# ---------------------------------------------------------------------------
def _brush(rng, side_x, side_y, a, length, permanent, H, ion_frac, salt, spare=64):
    """Stretched chains on a side_x x side_y lattice of spacing a with counterions and salt pairs."""
    Lx, Ly, b = side_x * a, side_y * a, 0.97
    nch = side_x * side_y
    radius = min(0.75, 0.22 * a) * rng.uniform(0.7, 1.0, nch)
    rise = min(0.80, (H - 1.0) / length)
    k = np.arange(length)
    turn = 2.0 * np.arcsin(np.minimum(1.0, math.sqrt(b * b - rise * rise) / (2.0 * radius)))
    ph = rng.uniform(0, 2 * np.pi, nch)[:, None] + turn[:, None] * k
    gx = (np.arange(nch) % side_x + 0.5) * a
    gy = (np.arange(nch) // side_x + 0.5) * a
    x = gx[:, None] + radius[:, None] * np.cos(ph)
    y = gy[:, None] + radius[:, None] * np.sin(ph)
    z = np.broadcast_to(0.2 + rise * k, (nch, length))
    beads = np.stack([x.ravel() % Lx, y.ravel() % Ly, z.ravel()], 1)
    nb = len(beads)
    t = np.zeros((nch, length), np.int32)
    q = np.zeros((nch, length), np.float32)
    f = np.full((nch, length), _abi.F_MOBILE, np.int32)
    f[:, 0] = 0
    first = permanent if permanent else 0
    t[:, :first] = PERMANENT
    q[:, :first] = 1.0
    f[:, first:] |= _abi.F_TITRATABLE
    titr = np.arange(nb).reshape(nch, length)[:, first:].ravel()
    ion = rng.permutation(titr)[:int(round(ion_frac * len(titr)))]
    t.ravel()[ion] = CHARGED
    q.ravel()[ion] = 1.0
    # free sites of a lattice of ~1.2 sigma, none within 1 sigma of a bead
    n3 = [max(2, int(Lx / 1.2)), max(2, int(Ly / 1.2)), max(2, int((H - 0.6) / 1.2))]
    w = np.array([Lx / n3[0], Ly / n3[1], (H - 0.6) / n3[2]])
    free = np.ones(n3, bool)
    home = np.floor((beads - [0, 0, 0.3]) / w).astype(int)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                c = home + [dx, dy, dz]
                ok = (c[:, 2] >= 0) & (c[:, 2] < n3[2])
                c = c[ok]
                p = (c + 0.5) * w + [0, 0, 0.3]
                d = p - beads[ok]
                d[:, 0] -= Lx * np.round(d[:, 0] / Lx)
                d[:, 1] -= Ly * np.round(d[:, 1] / Ly)
                hit = c[(d * d).sum(1) < 1.0]
                free[hit[:, 0] % n3[0], hit[:, 1] % n3[1], hit[:, 2]] = False
    sites = np.argwhere(free)
    n_pos = int((q > 0).sum())
    n_salt = int(round(salt * Lx * Ly * H))
    n_salt = max(0, min(n_salt, (int(0.4 * np.prod(n3)) - n_pos) // 2))  # dense brushes leave less room for salt
    n_ion = n_pos + 2 * n_salt
    if n_ion > len(sites):
        raise ValueError("no room for the ions")
    # counterions mostly inside the brush, salt anywhere
    top = 0.2 + rise * length + 3.0
    key = rng.random(len(sites)) + np.where((sites[:, 2] + 0.5) * w[2] < top, 0.0, 0.5)
    near = np.argsort(key)
    pick = near[:n_pos]
    rest = rng.permutation(near[n_pos:])[:n_ion - n_pos]
    ions = (np.concatenate([sites[pick], sites[rest]]) + 0.5) * w + [0, 0, 0.3] + rng.uniform(-0.03, 0.03, (n_ion, 3))
    ti = np.concatenate([np.full(n_pos, ANION), np.tile([CATION, ANION], n_salt)]).astype(np.int32)
    qi = np.where(ti == CATION, 1.0, -1.0).astype(np.float32)
    fi = np.where(ti == CATION, _abi.F_MOBILE | _abi.F_CATION, _abi.F_MOBILE | _abi.F_ANION).astype(np.int32)
    P = np.concatenate([beads, ions]).astype(np.float32)
    P[:, 0] = np.where(P[:, 0] >= np.float32(Lx), 0, np.maximum(P[:, 0], 0))
    P[:, 1] = np.where(P[:, 1] >= np.float32(Ly), 0, np.maximum(P[:, 1], 0))
    i = np.arange(nb).reshape(nch, length)
    n_sites = nch * (length - first)
    return SystemArrays(P[:, 0].copy(), P[:, 1].copy(), P[:, 2].copy(), np.concatenate([q.ravel(), qi]),
                        np.concatenate([t.ravel(), ti]).astype(np.int32), np.concatenate([f.ravel(), fi]).astype(np.int32),
                        i[:, :-1].ravel().astype(np.int32), i[:, 1:].ravel().astype(np.int32), np.array([Lx, Ly, 3 * H]),
                        capacity=nb + n_ion + n_sites + spare, meta={"chains": nch, "n_sites": n_sites, "height": H})


def _mesh(case, side, a, H):
    if "mesh" in case:
        return case["mesh"], case["mesh"], case["depth"]
    n = configs.smooth_mesh(min(64, max(32, side * a / 0.75)))
    return n, n, configs.smooth_mesh(3 * H / 0.75)


def _systems(case, seed):
    """The case's replicas: pH and salt spread about the case's values over a sweep; a batch shares
    one starting structure per eight pH values, as titration curves are started.  Sizes follow from
    the case, places and charges from the seed."""
    rng, size = np.random.default_rng([seed, 11]), np.random.default_rng(case["replicas"])
    R = case["replicas"]
    systems, params = [], []
    for r in range(R):
        pH = case["pH"] if R == 1 else 5.0 + 4.0 * ((r * 5 + 3) % 16) / 15.0
        side, a, length, H = case["side"], case["spacing"], case["length"], case["height"]
        salt = case["salt"]
        if R > 8 and r % 8 == 0:
            uneven = case["permanent"] == 0
            side = max(4, side - int(size.integers(0, 5)))
            if uneven:
                length = max(20, length - int(size.integers(0, 25)))
                H = H - (case["length"] - length)
            salt = salt * math.exp(size.uniform(-2.0, 0.7))
        if r % 8 == 0:
            s = _brush(rng, side, side, a, length, case["permanent"], H, configs.ideal_alpha(case["pH"], 7.3), salt,
                       spare=64 if not case.get("swap") else 1024)
            mesh = _mesh(case, side, a, H)
            rsalt = salt
        p = configs.native_params(pH, 7.3, mesh, s.meta["height"], int(seed) * 1000 + r, salt_conc=rsalt, order=case["order"],
                                  p_disp=0.9 - case.get("swap", 0.0), p_titr=0.1, p_swap=case.get("swap", 0.0))
        systems.append(s)
        params.append(p)
    return systems, params


def _pinned(n):
    f = {k: torch.empty(n, dtype=torch.float32, pin_memory=True).numpy() for k in ("x", "y", "z", "q")}
    f.update({k: torch.empty(n, dtype=torch.int32, pin_memory=True).numpy() for k in ("type", "flags")})
    return f


def _moves(s, p, rng, n):
    """Trial moves of configuration s, a dict per changed particle: displacements, protonations with
    a counterion inserted, deprotonations with one removed, salt pairs inserted."""
    mobile = np.flatnonzero(s.flags & _abi.F_MOBILE)
    titr = (s.flags & _abi.F_TITRATABLE) != 0
    neutral, charged = np.flatnonzero(titr & (s.q == 0)), np.flatnonzero(titr & (s.q > 0))
    anions = np.flatnonzero(s.flags & _abi.F_ANION)
    Lx, Ly = np.float32(s.box[0]), np.float32(s.box[1])

    def spot():  # away from the other particles by more than 0.95 sigma
        for _ in range(200):
            v = np.array([rng.uniform(0, s.box[0]), rng.uniform(0, s.box[1]), rng.uniform(0.3, p.wall_hi - 0.3)]).astype(np.float32)
            d = np.stack([s.x, s.y, s.z], 1) - v
            d[:, 0] -= Lx * np.round(d[:, 0] / Lx)
            d[:, 1] -= Ly * np.round(d[:, 1] / Ly)
            if (d * d).sum(1).min() > 0.9 and v[0] < Lx and v[1] < Ly:
                break
        return v

    def there(i, v, q, t):
        return dict(index=int(i), x=float(v[0]), y=float(v[1]), z=float(v[2]), q=float(q), type=int(t))

    out = []
    for k in range(n):
        kind = ("disp", "disp", "prot", "deprot", "disp", "pair")[k % 6]
        if kind == "disp" or (kind == "prot" and not len(neutral)) or (kind == "deprot" and not (len(charged) and len(anions))):
            i = mobile[rng.integers(len(mobile))]
            v = np.array([s.x[i], s.y[i], s.z[i]], np.float32) + rng.uniform(-0.1, 0.1, 3).astype(np.float32)
            v[0] = v[0] + Lx if v[0] < 0 else (v[0] - Lx if v[0] >= Lx else v[0])
            v[1] = v[1] + Ly if v[1] < 0 else (v[1] - Ly if v[1] >= Ly else v[1])
            v = np.minimum(np.maximum(v, np.float32(0)), np.nextafter(np.array([Lx, Ly, p.wall_hi], np.float32), np.float32(0)))
            out.append([there(i, v, s.q[i], s.type[i])])
        elif kind == "prot":
            i = neutral[rng.integers(len(neutral))]
            out.append([there(i, (s.x[i], s.y[i], s.z[i]), 1.0, CHARGED), there(s.n, spot(), -1.0, ANION)])
        elif kind == "deprot":
            i, j = charged[rng.integers(len(charged))], anions[rng.integers(len(anions))]
            gone = there(j, (s.x[j], s.y[j], s.z[j]), -1.0, ANION)
            gone["present"] = 0
            out.append([there(i, (s.x[i], s.y[i], s.z[i]), 0.0, NEUTRAL), gone])
        else:
            a, b = spot(), spot()
            out.append([there(s.n, a, 1.0, CATION), there(s.n + 1, b, -1.0, ANION)])
    return out


def _loop_moves(case, seed, s, p):
    """Moves of the caller's own loop, each followed by its reverse: displacement out, protonation,
    displacement back, deprotonation, over 16 particles and sites."""
    rng = np.random.default_rng([seed, 13])
    out = []
    mv = _moves(s, p, rng, 96)
    for d, c in zip([m for m in mv if len(m) == 1][:16], [m for m in mv if len(m) == 2 and m[0]["type"] == CHARGED][:16]):
        i, j = d[0]["index"], c[0]["index"]
        gone = dict(c[1], present=0)
        back = dict(d[0], x=float(s.x[i]), y=float(s.y[i]), z=float(s.z[i]))
        was = dict(c[0], q=0.0, type=NEUTRAL)
        if i == j:  # the same bead is moved and protonated: its charge state follows
            back.update(q=1.0, type=CHARGED)
            c = [dict(c[0], x=d[0]["x"], y=d[0]["y"], z=d[0]["z"]), c[1]]
        out += [d, c, [back], [was, gone]]
    return out


def _samples(case, seed):
    """One training batch of the first stage: neighbour-shell counts, one-hot states, targets in kT."""
    g = torch.Generator().manual_seed(int(seed) * 7 + 5)
    n, R, K = case["samples"], _abi.SUR_ROWS, _abi.SUR_INPUTS
    x = torch.zeros(n, R, K)
    shell = torch.arange(16).repeat_interleave(4).float()
    x[:, :, :64] = torch.poisson((0.02 * (shell + 0.5) ** 2).expand(n, R, 64).contiguous(), generator=g)
    x[:, :, 64] = torch.rand(n, R, generator=g)
    state = torch.randint(0, 4, (n, R), generator=g)
    x[:, :, 65:69] = torch.nn.functional.one_hot(state, 4).float()
    x[:, :, 69] = (2 * torch.rand(n, 1, generator=g) - 1) * 2
    x[:, :, 70] = -2.0 + 0.5 * torch.randn(n, 1, generator=g)
    sign = torch.tensor([-1.0, 1.0, 1.0, 0.0]).repeat(n, 1)
    sign[:, 2] *= (torch.rand(n, generator=g) < 0.5).float()
    t = 3.0 * torch.randn(n, generator=g)
    mu, sd = x.reshape(-1, K).mean(0), x.reshape(-1, K).std(0)
    sd = torch.where(sd > 1e-3, sd, torch.ones_like(sd))
    return x.numpy(), sign.numpy(), t.numpy(), mu.numpy(), sd.numpy()


def _network(seed, hidden, mu, sd, scale):
    net = Surrogate(hidden=hidden, seed=int(seed) + 3)
    net.set_scaling(mu, sd, scale)
    return net


def _reference_system(case, seed):
    rng = np.random.default_rng([seed, 17])
    s = _brush(rng, case["side"], case["side"], case["spacing"], case["length"], 0, case["height"], 0.5, case["salt"])
    return configs.to_reference_semantics(s, n_w=s.meta["n_sites"], seed=int(seed) % (1 << 31), spacing=0.7)


# ---------------------------------------------------------------------------
# the measured passes
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "grad":
        x, sign, t, mu, sd = _samples(case, seed)
        st.update(x=x, sign=sign, t=t, net=_network(seed, case["hidden"], mu, sd, 3.0))
        return st
    if kind == "phase2":
        s, p = _reference_system(case, seed)
        nh_p, nh_n = np.flatnonzero(s.type == 4), np.flatnonzero(s.type == 3)
        w, cl = np.flatnonzero(s.type == 6), np.flatnonzero(s.type == 7)
        mt = np.zeros(625, np.uint32)
        mt[:624] = np.random.RandomState(int(seed) % (1 << 31)).get_state()[1]
        mt[624] = 624
        st.update(engine=Engine(s, p), mt=mt,
                  job=dict(replica=0, nh_n_type=3, nh_p_type=4, w_type=6, cl_type=7, q_nh_p=1.0, q_cl=-1.0, beta=1.0,
                           max_attempts=case["trials"], patience=1 << 20, energy_interval=50, nh_p=nh_p, nh_n=nh_n, w=w,
                           cl=cl, mt_state=mt))
        # the configuration that every phase starts from (a driver runs a phase on a given state)
        st["start"] = st["engine"].state(0)
        return st
    systems, params = _systems(case, seed)
    eng = Engine(systems, params)
    st["engine"] = eng
    if case.get("tuned"):  # a tuning found earlier with Engine.autotune
        eng.set_tuning(48, 256)
        if case["order"] == 5:
            eng.set_tile_shapes(cand_round=2, g_rows=21)
    if case.get("surrogate"):
        _, _, _, mu, sd = _samples({"samples": 512}, seed)
        net = _network(seed, 128, mu, sd, 1.0)
        eng.attach_surrogate(net)
        st["net"] = net
    if kind in ("run", "exchange"):
        st["out"] = _pinned(sum(eng.caps))
        if kind == "exchange":
            st["in"] = _pinned(sum(eng.caps))
            eng.state(-1, out=st["in"])
    elif kind == "scan":
        st["moves"] = _moves(systems[0], params[0], np.random.default_rng([seed, 19]), case["trials"])
    elif kind == "loop":
        st["moves"] = _loop_moves(case, seed, systems[0], params[0])
        st["at"] = 0
    return st


COMPONENTS = ("lj", "fene", "coul_real", "coul_recip", "self", "qcorr", "slab", "total")


def _columns(rows):
    return {k: np.array([r[k] for r in rows], np.float32) for k in COMPONENTS}


def _run_outputs(stats, out):
    # (the number of mesh rebuilds and the rounding drift are diagnostics, not results)
    r = dict(out)
    r["attempted"] = np.array([s["attempted"] for s in stats], np.int64)
    r["accepted"] = np.array([s["accepted"] for s in stats], np.int64)
    r["ions"] = np.array([[s["n_charged_sites"], s["n_cations"], s["n_anions"]] for s in stats], np.int64)
    r["energy"] = np.array([s["energy"] for s in stats], np.float32)
    return r


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "grad":
        loss, g = state["net"].gradient(state["x"], state["sign"], state["t"])
        return {"loss": np.float32(loss), "grad": g}
    eng = state["engine"]
    if kind == "run":
        return _run_outputs(eng.run(case["trials"]), eng.state(-1, out=state["out"]))
    if kind == "exchange":
        eng.set_state(state["in"], -1)
        return _run_outputs(eng.run(case["trials"]), eng.state(-1, out=state["out"]))
    if kind == "energy":
        return _columns(eng.energy())
    if kind == "scan":
        return _columns(eng.delta_energy_components(state["moves"]))
    if kind == "loop":
        rows = []
        for k in range(case["trials"]):
            m = state["moves"][(state["at"] + k) % len(state["moves"])]
            rows += eng.delta_energy_components([m])
            eng.commit(m)
        state["at"] += case["trials"]
        return _columns(rows)
    eng.set_state(state["start"])
    res, _ = eng.phase2([state["job"]])[0]
    after = eng.state(0)
    return {"q": after["q"], "type": after["type"], "mt": state["mt"].astype(np.int64),
            "counts": np.array([res["attempted"], res["accepted"], res["since_best"]], np.int64),
            "E": np.float32(res["E"]), "best_E": np.float32(res["best_E"])}


def work(case):
    """Bytes and operations that a pass cannot do without.  A trial reads the particles within the
    cutoff of its old and new places (20 B each) and the potential under two stencils, and does ~40
    operations a pair; a whole energy reads every particle once and does its pairs and one
    real-to-complex transform pair of the mesh."""
    kind = case["kind"]
    if kind == "grad":
        rows = case["samples"] * _abi.SUR_ROWS
        h, k = case["hidden"], _abi.SUR_INPUTS
        n_par = k * h + 2 * h * h + 4 * h + 1
        return {"bytes": 4.0 * (rows * (k + 1) + case["samples"] + 2 * n_par), "flops": 6.0 * rows * (k * h + 2 * h * h + h)}
    R, area, H = case["replicas"], (case["side"] * case["spacing"]) ** 2, case["height"]
    beads = case["side"] ** 2 * case["length"]
    n = R * (beads * (1.7 if kind != "phase2" else 2.5) + 2 * case["salt"] * area * H)
    rho = n / R / (area * H)
    pairs = 4.19 * 27.0 * rho  # neighbours within the 3 sigma cutoff
    P3 = case["order"] ** 3
    if kind == "energy":
        mesh = math.prod([float(v) for v in _mesh(case, case["side"], case["spacing"], H)])
        return {"bytes": n * 36.0 + R * 64.0, "flops": n * (20.0 * pairs + 4.0 * P3) + 5.0 * R * mesh * math.log2(mesh)}
    trials = R * case["trials"]
    per_b, per_f = 2 * pairs * 20.0 + 8.0 * P3, 2 * pairs * 40.0 + 4.0 * P3
    state = {"run": 24.0, "exchange": 48.0, "phase2": 48.0}.get(kind, 0.0) * n
    return {"bytes": trials * per_b + state, "flops": trials * per_f}


# ---------------------------------------------------------------------------
# energies in 64 bits, without the library's code
# ---------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Exact:
    """Energies of the native model in FP64: direct pair sums and SPME with torch's FFT."""

    def __init__(self, s, p):
        dev, f8 = _dev(), torch.float64
        pad = 2  # room for inserted ions
        z = np.zeros(pad, np.float32)
        self.pos = torch.tensor(np.stack([np.concatenate([v, z]) for v in (s.x, s.y, s.z)], 1), dtype=f8, device=dev)
        self.q = torch.tensor(np.concatenate([s.q, z]), dtype=f8, device=dev)
        self.here = torch.tensor(np.concatenate([(s.flags & _abi.F_GHOST) == 0, np.zeros(pad, bool)]), device=dev)
        self.L = torch.tensor(np.asarray(s.box, np.float32), dtype=f8, device=dev)
        self.p, self.n = p, s.n
        self.bi = torch.tensor(s.bond_i, dtype=torch.long, device=dev)
        self.bj = torch.tensor(s.bond_j, dtype=torch.long, device=dev)
        self.elf, self.alpha = 138.935458 / p.epsilon_r, p.ewald_alpha
        self.V = float(np.prod(np.asarray(s.box, np.float64)))
        self.mesh = tuple(p.mesh)
        k2, fac = [], []
        for ax in range(3):
            m = self.mesh[ax]
            j = torch.arange(m, device=dev)
            k = torch.where(j <= m // 2, j, j - m).to(f8) / float(self.L[ax])
            k2.append(k * k)
            fac.append(torch.exp(-(math.pi / self.alpha) ** 2 * k * k) / self._moduli(m))
        kk = k2[0][:, None, None] + k2[1][None, :, None] + k2[2][None, None, :]
        kk[0, 0, 0] = 1.0
        self.theta = self.elf / (math.pi * self.V) * fac[0][:, None, None] * fac[1][None, :, None] * fac[2][None, None, :] / kk
        self.theta[0, 0, 0] = 0.0

    def _moduli(self, m):
        P = self.p.order
        w = [self._spline(torch.zeros(1, dtype=torch.float64, device=_dev()))[:, j] for j in range(P)]
        j = torch.arange(P, dtype=torch.float64, device=_dev())
        k = torch.arange(m, dtype=torch.float64, device=_dev())
        ph = 2 * math.pi * k[:, None] * j[None, :] / m
        v = torch.cat(w)
        mod = (torch.cos(ph) @ v) ** 2 + (torch.sin(ph) @ v) ** 2
        near = 0.5 * (torch.roll(mod, 1) + torch.roll(mod, -1))
        return torch.where(mod < 1e-7, near, mod)

    def _spline(self, t):
        """Cardinal B-spline weights of the mesh points floor(g) + P/2 - P + 1 + j at fraction t."""
        P = self.p.order
        c = [t, 1.0 - t]
        for n in range(3, P + 1):
            up = []
            for i in range(n):
                a = c[i] if i < n - 1 else torch.zeros_like(t)
                b = c[i - 1] if i >= 1 else torch.zeros_like(t)
                up.append(((t + i) * a + (n - t - i) * b) / (n - 1))
            c = up
        return torch.stack(c[::-1], 1)

    def stencil(self, pos):
        P = self.p.order
        idx, w = [], []
        for ax in range(3):
            g = pos[:, ax] / self.L[ax] * self.mesh[ax]
            fl = torch.floor(g)
            w.append(self._spline(g - fl))
            base = fl.long() + P // 2 - P + 1
            idx.append((base[:, None] + torch.arange(P, device=pos.device)) % self.mesh[ax])
        flat = (idx[0][:, :, None, None] * self.mesh[1] + idx[1][:, None, :, None]) * self.mesh[2] + idx[2][:, None, None, :]
        ww = w[0][:, :, None, None] * w[1][:, None, :, None] * w[2][:, None, None, :]
        return idx, w, flat.reshape(len(pos), -1), ww.reshape(len(pos), -1)

    def spectrum(self):
        m = self.here & (self.q != 0)
        _, _, flat, w = self.stencil(self.pos[m])
        Q = torch.zeros(int(np.prod(self.mesh)), dtype=torch.float64, device=flat.device)
        Q.index_add_(0, flat.reshape(-1), (w * self.q[m][:, None]).reshape(-1))
        return torch.fft.fftn(Q.reshape(self.mesh))

    def _image(self, d):
        return d - self.L * torch.round(d / self.L)

    def pair(self, r2, qq):
        """(LJ, real-space Coulomb) of pairs at squared distance r2."""
        rc2 = 2.0 ** (1.0 / 3.0)
        s6 = 1.0 / torch.clamp(r2, min=1e-12) ** 3
        lj = torch.where(r2 <= rc2, 4.0 * (s6 * s6 - s6) + 1.0, torch.zeros_like(r2))
        r = torch.sqrt(r2)
        c = torch.where(r2 <= self.p.rc_coul ** 2, self.elf * qq * torch.erfc(self.alpha * r) / torch.clamp(r, min=1e-12), torch.zeros_like(r2))
        return lj, c

    def bond(self, r2):
        R2 = self.p.fene_r0 ** 2
        return torch.where(r2 < R2, -0.5 * self.p.fene_k * R2 * torch.log(torch.clamp(1.0 - r2 / R2, min=1e-300)), torch.full_like(r2, math.inf))

    def moments(self, q, z):
        return q.sum(), (q * q).sum(), (q * z).sum(), (q * z * z).sum()

    def long_range(self, mom):
        Q, Q2, M, S = mom
        own = -self.elf * self.alpha / math.sqrt(math.pi) * Q2
        net = -math.pi * self.elf / (2 * self.V * self.alpha ** 2) * Q * Q
        c = 2 * math.pi / self.V * self.elf
        slab = c * M * M
        if abs(float(Q)) > 1e-4:
            slab = slab - c * Q * (S + Q * self.L[2] ** 2 / 12.0)
        return own, net, slab

    def energy(self):
        i = torch.nonzero(self.here)[:, 0]
        pos, q = self.pos[i], self.q[i]
        lj = c = 0.0
        n = len(i)
        step = max(1, 12_000_000 // n)
        for a in range(0, n, step):
            d = self._image(pos[a:a + step, None] - pos[None, :])
            r2 = (d * d).sum(-1)
            near = torch.nonzero((r2 <= 9.0001) & (torch.arange(n, device=pos.device)[None, :] > torch.arange(a, min(n, a + step), device=pos.device)[:, None]))
            e = self.pair(r2[near[:, 0], near[:, 1]], q[a + near[:, 0]] * q[near[:, 1]])
            lj, c = lj + e[0].sum(), c + e[1].sum()
        d = self._image(self.pos[self.bi] - self.pos[self.bj])
        fene = self.bond((d * d).sum(-1)).sum()
        F = self.spectrum()
        rec = 0.5 * (self.theta * (F.real ** 2 + F.imag ** 2)).sum()
        own, net, slab = self.long_range(self.moments(q, pos[:, 2]))
        e = [lj, fene, c, rec, own, net, slab]
        return [float(v) for v in e] + [float(sum(e))]

    def change(self, move):
        """Apply a move: [(index, new position, new charge, present)]."""
        for ch in move:
            k = ch["index"]
            self.here[k] = bool(ch.get("present", 1))
            v = np.array([ch["x"], ch["y"], ch["z"]], np.float32)
            self.pos[k] = torch.tensor(v, dtype=torch.float64, device=self.pos.device)
            self.q[k] = float(ch["q"])

    def deltas(self, moves):
        """Energy changes of each move from the present configuration, by component."""
        F = self.spectrum()
        M = float(np.prod(self.mesh))
        phi = (torch.fft.ifftn(self.theta * F).real * M).reshape(-1)
        g = (torch.fft.ifftn(self.theta.to(torch.complex128)).real * M).reshape(-1)
        mom0 = self.moments(self.q[self.here], self.pos[self.here][:, 2])
        base = self.long_range(mom0)
        out = []
        for mv in moves:
            old, new = [], []  # (index, position, charge)
            for ch in mv:
                k = ch["index"]
                if bool(self.here[k]):
                    old.append((k, self.pos[k], self.q[k]))
                if ch.get("present", 1):
                    v = torch.tensor(np.array([ch["x"], ch["y"], ch["z"]], np.float32), dtype=torch.float64, device=self.pos.device)
                    new.append((k, v, torch.tensor(float(ch["q"]), dtype=torch.float64, device=self.pos.device)))
            rest = self.here.clone()
            for ch in mv:
                rest[ch["index"]] = False
            lj = c = fene = 0.0
            for sign, side in ((-1.0, old), (1.0, new)):
                for a, (k, v, qk) in enumerate(side):
                    d = self._image(self.pos - v)
                    r2 = (d * d).sum(-1)
                    ok = rest & (r2 <= 9.0001)
                    e = self.pair(r2[ok], self.q[ok] * qk)
                    lj, c = lj + sign * e[0].sum(), c + sign * e[1].sum()
                    for k2, v2, q2 in side[a + 1:]:
                        d2 = self._image(v - v2)
                        e = self.pair((d2 * d2).sum(-1, keepdim=True), (qk * q2)[None])
                        lj, c = lj + sign * e[0].sum(), c + sign * e[1].sum()
                    b = torch.cat([self.bj[self.bi == k], self.bi[self.bj == k]])
                    fene = fene + sign * self.bond(r2[b]).sum()
            pos = torch.stack([v for _, v, _ in old + new])
            w8 = torch.stack([-q for _, _, q in old] + [q for _, _, q in new])
            idx, _, flat, w = self.stencil(pos)
            rec = (w8 * (w * phi[flat]).sum(1)).sum()
            P = self.p.order
            for a in range(len(pos)):
                for b in range(len(pos)):
                    dd = [(idx[ax][a][:, None] - idx[ax][b][None, :]) % self.mesh[ax] for ax in range(3)]
                    at = ((dd[0][:, None, None, :, None, None] * self.mesh[1] + dd[1][None, :, None, None, :, None]) * self.mesh[2]
                          + dd[2][None, None, :, None, None, :]).reshape(P ** 3, P ** 3)
                    rec = rec + 0.5 * w8[a] * w8[b] * (w[a] @ (g[at] @ w[b]))
            zz = pos[:, 2]
            sq = torch.cat([-torch.ones(len(old)), torch.ones(len(new))]).to(pos.device).double()
            qq = torch.stack([q for _, _, q in old + new])
            mom = (mom0[0] + (sq * qq).sum(), mom0[1] + (sq * qq * qq).sum(), mom0[2] + (sq * qq * zz).sum(), mom0[3] + (sq * qq * zz * zz).sum())
            lr = [x - y for x, y in zip(self.long_range(mom), base)]
            e = [float(v) for v in (lj, fene, c, rec, *lr)]
            out.append(e + [sum(e)])
        return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        return _exact_gradient(case, seed)
    if kind not in ("energy", "scan", "loop"):
        return None  # a Markov chain's state has no value of its own in 64 bits
    systems, params = _systems(case, seed)
    if kind == "energy":
        rows = [_Exact(s, p).energy() for s, p in zip(systems, params)]
    elif kind == "scan":
        moves = _moves(systems[0], params[0], np.random.default_rng([seed, 19]), case["trials"])
        rows = _Exact(systems[0], params[0]).deltas(moves)
    else:
        ex, rows = _Exact(systems[0], params[0]), []
        moves = _loop_moves(case, seed, systems[0], params[0])
        for k in range(case["trials"]):
            rows += ex.deltas([moves[k % len(moves)]])
            ex.change(moves[k % len(moves)])
    return {k: np.array([r[i] for r in rows], np.float64) for i, k in enumerate(COMPONENTS)}


def _exact_gradient(case, seed):
    """Loss and gradient of the network in FP64 (weights as the network holds them)."""
    x, sign, t, mu, sd = _samples(case, seed)
    H, K, dev = case["hidden"], _abi.SUR_INPUTS, _dev()
    flat = torch.tensor(_network(seed, H, mu, sd, 3.0).params(), dtype=torch.float64, device=dev, requires_grad=True)
    sizes = [K * H, H, H * H, H, H * H, H, H, 1]
    w1, b1, w2, b2, w3, b3, w4, b4 = torch.split(flat, sizes)
    h = torch.tensor((x.astype(np.float64) - mu) / sd, device=dev).reshape(-1, K)
    gelu = torch.nn.functional.gelu
    h = gelu(h @ w1.reshape(K, H) + b1)
    h = gelu(h @ w2.reshape(H, H) + b2)
    h = gelu(h @ w3.reshape(H, H) + b3)
    y = (h @ w4 + b4).reshape(-1, _abi.SUR_ROWS)
    pred = (y * torch.tensor(sign, dtype=torch.float64, device=dev)).sum(1)
    target = torch.clamp(torch.tensor(t, dtype=torch.float64, device=dev), -25.0, 25.0) / 3.0
    loss = 0.5 * ((pred - target) ** 2).mean()
    (g,) = torch.autograd.grad(loss, flat)
    return {"loss": np.float64(loss.item()), "grad": g.cpu().numpy()}
