"""The work that users of parent_gb300 have it do, as cases that can be timed and compared.

A case is one call sequence of the Python interface on inputs a user's program has in hand:

  entropy    a trajectory's BAT columns -> the .par body and the MIST tree (PARENT.x, then get_PAR_MIST.x)
  batch      many small trajectories -> every body and tree in one call
  mist       a .par body read from a file -> its MIST tree (get_PAR_MIST.x alone)
  cartesian  decoded coordinates -> BAT columns on the device -> body and tree, with no .bat in between

DOFs = 3 * atoms - 6. "bins" is the bin count of every DOF type, or "b" / "a" / "d" give the 2D counts by type.
"""
import math

import numpy as np
import torch

import parent_gb300 as pg

TWO_PI = 2 * math.pi
_ENGINE = []


def _engine():
    # a program keeps one context for all its trajectories
    if not _ENGINE:
        _ENGINE.append(pg.Engine(0))
    return _ENGINE[0]


# ------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest call a user makes: a peptide, a short run, columns read from a file into host arrays
        dict(name="peptide_66dof_2k_f64", kind="entropy", atoms=24, frames=2000, prec=1, host=1, bins=50),
        # the plain configuration of the benchmark: 100 atoms, double precision, host arrays
        dict(name="plain_294dof_20k_f64", kind="entropy", atoms=100, frames=20000, prec=1, host=1, bins=50),
        # the benchmark's small system, columns already on the device (read there by the .bat reader)
        dict(name="small_603dof_50k", kind="entropy", atoms=203, frames=50000, prec=0, host=0, bins=50),
        # coordinates straight from a decoder, a ragged frame count, a bin count of its own for every DOF type
        dict(name="cartesian_400atoms_33333", kind="cartesian", atoms=400, frames=33333, prec=1, b=24, a=30, d=36),
        # the benchmark's precision path at the usual 50 bins, and as it is swept over the bin count: 30 and 10
        dict(name="protein_2994dof_100k", kind="entropy", atoms=1000, frames=100000, prec=0, host=0, bins=50),
        dict(name="protein_2994dof_100k_30bins", kind="entropy", atoms=1000, frames=100000, prec=0, host=0, bins=30),
        dict(name="protein_2994dof_100k_10bins", kind="entropy", atoms=1000, frames=100000, prec=0, host=0, bins=10),
        # finer bins than the usual 50, as a long run of a mid-sized system allows
        dict(name="fine_1194dof_60001_90bins", kind="entropy", atoms=400, frames=60001, prec=0, host=1, bins=90),
        # a long trajectory of a mid-sized domain: a million frames
        dict(name="long_894dof_1m", kind="entropy", atoms=300, frames=1000000, prec=0, host=0, bins=50),
        # the benchmark's protein dimer, at a fifth of its frames
        dict(name="dimer_7494dof_100k", kind="entropy", atoms=2500, frames=100000, prec=0, host=0, bins=50),
        # the benchmark's batch of independent systems of 50 to 800 atoms, a quarter of it
        dict(name="batch_16_systems", kind="batch", systems=16, atoms=800, frames=100000, prec=0, host=0, bins=50),
        # the tree of a body that was computed earlier and read back from its .par
        dict(name="mist_2994dof", kind="mist", atoms=1000),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _updates(case):
    """DOF pairs x frames."""
    if case["kind"] == "mist":
        return 0.0
    if case["kind"] == "batch":
        return sum(d * (d - 1) / 2 * f for d, f in ((3 * a - 6, f) for a, f in _systems(case)))
    D = 3 * case["atoms"] - 6
    return D * (D - 1) / 2 * case["frames"]


def draw(rng):
    kind = rng.choice(["entropy"] * 7 + ["batch", "mist", "cartesian"])
    while True:
        c = dict(kind=kind)
        if kind == "mist":
            c["atoms"] = _logint(rng, 24, 2500)
            return c
        c["atoms"] = _logint(rng, 24, 2500)
        c["frames"] = _logint(rng, 1000, 1000000)
        # converted columns stay in double precision: rounded to single, a dihedral just below 2 pi leaves its range
        c["prec"] = 1 if kind == "cartesian" else rng.randint(0, 1)
        if kind == "batch":
            c["atoms"], c["frames"], c["systems"] = min(c["atoms"], 800), min(c["frames"], 100000), rng.randint(2, 24)
            if c["atoms"] < 60 or c["frames"] < 6000:
                continue
        if kind != "cartesian":
            c["host"] = rng.randint(0, 1)
        if rng.random() < 0.25 or kind == "cartesian":
            c["b"], c["a"], c["d"] = (rng.randint(8, 50) for _ in range(3))
        else:
            c["bins"] = rng.choice([50, 50, rng.randint(8, 50), rng.randint(8, 50), rng.randint(51, 100)])
        top = max(_bins(c)[3:])
        values = (3 * c["atoms"] - 6) * c["frames"] * c.get("systems", 1)
        # no more than the largest listed case (2.8e12 updates); above 50 bins the listed one's size
        if _updates(c) <= (2.8e12 if top <= 50 else 1.0e11) and values <= 1.0e9:
            return c


def _bins(case):
    if "bins" in case:
        return (case["bins"],) * 6
    return (case["b"], case["a"], case["d"]) * 2


def _systems(case):
    """(atoms, frames) of every system of a batch: atoms uniform in 50..max, frames log-uniform in 5000..max."""
    out = []
    for k in range(case["systems"]):
        u, v = ((k * 0.754877666 + 0.31) % 1.0, (k * 0.569840291 + 0.67) % 1.0)
        out.append((int(50 + u * (case["atoms"] - 50)), int(5000 * (case["frames"] / 5000) ** v)))
    return out


def work(case):
    if case["kind"] == "mist":
        D = 3 * case["atoms"] - 6
        return {"bytes": 8.0 * D * (D - 1) / 2 + 8.0 * D + 32.0 * D, "flops": 2.0 * D * D}
    systems = _systems(case) if case["kind"] == "batch" else [(case["atoms"], case["frames"])]
    nbytes = 0.0
    for atoms, frames in systems:
        D = 3 * atoms - 6
        values = 3.0 * atoms * 4 if case["kind"] == "cartesian" else D * (8.0 if case["prec"] else 4.0)
        nbytes += values * frames + 8.0 * (D + D * (D - 1) / 2) + 32.0 * D
    # one increment per (pair, frame)
    return {"bytes": nbytes, "flops": _updates(case)}


# ------------------------------------------------------------------ inputs

def _columns(atoms, frames, prec, gen):
    """A linear chain's BAT columns as in the benchmark's synthetic systems: bonds ~ N(0.15, 0.005), angles around
    1.91, dihedrals of one to three states, all correlated through slow latents; a fifth of the dihedrals and a
    twentieth of the bonds switch slowly between two states."""
    dev = "cuda"
    nd = atoms - 3
    dt = torch.float64 if prec else torch.float32

    def rnd(*s):
        return torch.randn(*s, generator=gen, device=dev)

    def uni(*s):
        return torch.rand(*s, generator=gen, device=dev)

    taps = 0.95 ** torch.arange(128, device=dev, dtype=torch.float32).flip(0)
    lat = torch.nn.functional.conv1d(rnd(8, 1, frames + 127), taps.reshape(1, 1, -1) * math.sqrt(1 - 0.95 ** 2))[:, 0]
    slow = torch.nn.functional.avg_pool1d(rnd(8, 1, frames + 512), 513, 1)[:, 0] * math.sqrt(513.0)

    def block(n, kind):
        out = torch.empty(n, frames, dtype=dt, device=dev)
        step = max(1, int(4e7 // frames))
        for k in range(0, n, step):
            m = min(step, n - k)
            w = 0.3 * rnd(m, 8)
            z = (rnd(m, frames) + w @ lat) / (1 + (w * w).sum(1, keepdim=True)).sqrt()
            state = (slow[torch.randint(0, 8, (m,), generator=gen, device=dev)] > rnd(m, 1)).float()
            if kind == "b":
                x = 0.15 + 0.005 * z + 0.02 * state * (uni(m, 1) < 0.05)
            elif kind == "a":
                x = (1.91 + 0.158 * z).clamp(0.02, math.pi - 0.02)
            else:
                fast = uni(m, frames) * (1 + 2 * uni(m, 1))
                mode = torch.where(uni(m, 1) < 0.2, state, (fast > 0.7).float() + (fast > 1.6).float())
                mu, width = TWO_PI * uni(m, 3), 0.22 + 0.4 * uni(m, 3)
                x = torch.remainder(mu.gather(1, mode.long()) + width.gather(1, mode.long()) * z, TWO_PI)
            x = x.to(dt)
            if prec:  # the digits below single precision
                x += 1e-9 * uni(m, frames)
            out[k:k + m] = x.clamp_(max=6.28318) if kind == "d" else x
        return out

    return block(nd + 2, "b"), block(nd + 1, "a"), block(nd, "d")


def _coordinates(atoms, frames, gen):
    """Decoded coordinates (frames, atoms, 3) in nm of a fluctuating chain, and its dihedral table (atoms 1-based,
    type, parent): every third dihedral is taken relative to the one before it."""
    rng = np.random.default_rng(int(torch.randint(0, 1 << 30, (1,), generator=gen, device="cuda")))
    base = np.zeros((atoms, 3))
    for i in range(1, atoms):  # a helix-like backbone with irregular turns: bond angles stay well inside (0, pi)
        t = 1.7 * i + rng.normal(0, 0.25)
        base[i] = base[i - 1] + 0.15 * np.array([0.85 * math.cos(t), 0.85 * math.sin(t), 0.5])
    x = torch.randn(frames, atoms, 3, generator=gen, device="cuda") * 0.012
    xyz = (torch.as_tensor(base, device="cuda").float() + x).cpu().numpy()
    dih = np.zeros((atoms - 3, 6), np.int32)
    for i in range(atoms - 3):
        dih[i] = [i + 1, i + 2, i + 3, i + 4, 0, i if i % 3 == 1 else -1]
    return xyz, dih


def _body(atoms, gen):
    """A .par body whose mutual informations come from a few shared modes: S2 = S1 + S1 - MI."""
    n_dih = atoms - 3
    D, nb, na = 3 * n_dih + 3, n_dih + 2, n_dih + 1

    def rnd(*s):
        return torch.randn(*s, generator=gen, device="cuda", dtype=torch.float64)

    s1 = 1.5 + 0.8 * rnd(D)
    load = 0.35 * rnd(D, 6)
    load = load / (1 + (load * load).sum(1, keepdim=True)).sqrt()
    mi = -0.5 * torch.log1p(-(load @ load.T).square().clamp(max=0.99)) + 0.01 * torch.rand(D, D, generator=gen, device="cuda", dtype=torch.float64)
    mi = torch.triu(mi, 1)
    s2 = (s1[:, None] + s1[None, :] - mi).cpu()
    lo, n = {"b": 0, "a": nb, "d": nb + na}, {"b": nb, "a": na, "d": n_dih}
    blocks = {"s1_" + t: s1[lo[t]:lo[t] + n[t]].cpu().numpy() for t in "bad"}
    for p in ("bb", "ba", "bd", "aa", "ad", "dd"):
        q = s2[lo[p[0]]:lo[p[0]] + n[p[0]], lo[p[1]]:lo[p[1]] + n[p[1]]]
        if p[0] == p[1]:  # the pairs in reverse lexicographic order
            i, j = torch.triu_indices(n[p[0]], n[p[0]], 1)
            blocks[p] = q[i, j].flip(0).numpy().copy()
        else:
            blocks[p] = q.reshape(-1).numpy().copy()
    return pg.ParBody(n_dih, blocks)


def _body_buffer(n_dih):
    """A body to fill, and the one array that its blocks lie in."""
    sizes = pg.block_sizes(n_dih)
    flat = np.zeros(sum(sizes.values()))
    blocks, at = {}, 0
    for k, n in sizes.items():
        blocks[k] = flat[at:at + n]
        at += n
    return pg.ParBody(n_dih, blocks), flat


def _trajectory(cols, host):
    if host:
        return pg.Trajectory(*(c.cpu().numpy() for c in cols))
    b, a, d = cols
    return pg.BatView(d.shape[0], b.shape[1], int(b.dtype == torch.float64), 1, b.shape[1], b.data_ptr(), a.data_ptr(), d.data_ptr())


def _gen(seed):
    return torch.Generator("cuda").manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)


def prepare(case, seed):
    gen = _gen(seed)
    s = dict(kind=case["kind"], eng=_engine())
    if case["kind"] == "mist":
        s["body"] = _body(case["atoms"], gen)
    elif case["kind"] == "cartesian":
        s["xyz"], s["dih"] = _coordinates(case["atoms"], case["frames"], gen)
        s["prec"], s["bins"] = case["prec"], _bins(case)
        s["out"], s["flat"] = _body_buffer(case["atoms"] - 3)
    else:
        systems = _systems(case) if case["kind"] == "batch" else [(case["atoms"], case["frames"])]
        cols = [_columns(a, f, case["prec"], gen) for a, f in systems]
        s["trajs"] = [_trajectory(c, case["host"]) for c in cols]
        s["cols"] = None if case["host"] else cols
        outs = [_body_buffer(a - 3) for a, _ in systems]
        s["out"], s["flat"] = [o[0] for o in outs], [o[1] for o in outs]
        s["bins"] = _bins(case)
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run

def _tree(edges, totals):
    return {"t1": edges["t1"], "t2": edges["t2"], "i1": edges["i1"], "i2": edges["i2"], "left": edges["left"],
            "mi": edges["mi"], "totals": totals}


def run(s):
    eng = s["eng"]
    if s["kind"] == "mist":
        return _tree(*eng.mist(s["body"].n_dih, s["body"]))
    if s["kind"] == "batch":
        _, trees = eng.entropy_batch(s["trajs"], s["bins"], bodies=s["out"])
        return {"bodies": s["flat"], "edges": _tree(np.concatenate([e for e, _ in trees]), np.stack([t for _, t in trees]))}
    if s["kind"] == "cartesian":
        view = eng.bat_from_cartesian(s["xyz"], s["dih"], s["prec"])
        out, flat = s["out"], s["flat"]
    else:
        view, out, flat = s["trajs"][0], s["out"][0], s["flat"][0]
    eng.entropy(view, s["bins"], out=out)
    return {"body": flat, **_tree(*eng.mist(out.n_dih))}


# ------------------------------------------------------------------- exact

def _bat_columns(xyz, dih):
    """BAT_builder's conversion in 64 bits from the same single-precision coordinates."""
    x = (torch.as_tensor(xyz, device="cuda").double() * 10.0).float()

    def vec(a1, a0):
        return (x[:, a1] - x[:, a0]).double()

    at = torch.as_tensor(dih[:, :4].astype(np.int64) - 1, device="cuda")
    b1, b2, b3 = vec(at[:, 1], at[:, 0]), vec(at[:, 2], at[:, 1]), vec(at[:, 3], at[:, 2])
    bl, prev = b3.square().sum(-1).sqrt(), b2.square().sum(-1).sqrt()
    ang = torch.acos((b2 * b3).sum(-1) / bl / prev)
    A, B = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
    num = (torch.linalg.cross(A, B) * b2).sum(-1) / prev
    phi = torch.atan2(num, (A * B).sum(-1))
    for i in range(dih.shape[0]):
        if dih[i, 5] != -1:
            phi[:, i] -= phi[:, dih[i, 5] - 1]
    phi = phi + TWO_PI - ((phi + TWO_PI) / TWO_PI).trunc() * 2 * math.pi
    r0, r1 = b1[:, :1].square().sum(-1).sqrt(), prev[:, :1]
    ra = torch.acos((b1[:, 0] * b2[:, 0]).sum(-1) / r0[:, 0] / r1[:, 0])[:, None]
    return [torch.cat(v, 1).T.contiguous() for v in ([r0, r1, bl], [ra, ang], [phi])]


def _shifted(x):
    """A block of dihedral columns moved so that its emptiest stretch of 100 bins lies at the ends."""
    size = (TWO_PI + 0.000000005) / 100
    idx = (x / size).long()
    occ = torch.zeros(x.shape[0], 100, dtype=torch.int64, device=x.device).scatter_add_(1, idx, torch.ones_like(idx)).cpu().numpy()
    shift = []
    for h in occ:
        pos = 0
        if (h == 0).any():
            longest, cur, start, pos = 0, 0, 0, -1
            for k in range(200):
                if h[k % 100] == 0:
                    if cur == 0:
                        cur, start = 1, k
                    cur += 1
                elif cur > 0:
                    if cur > longest:
                        longest, pos = cur, start
                    cur = 0
        else:
            pos = int(np.argmin(h))
        shift.append(TWO_PI - (pos + 0.5) * size)
    y = x + torch.as_tensor(shift, dtype=torch.float64, device=x.device)[:, None]
    return y - TWO_PI * (y / TWO_PI).trunc()


def _dofs(cols, bins):
    """Per DOF: 2D bin of every frame, 1D entropy, the constant of its 2D entropies."""
    idx, s1, con = [], [], []
    for t, c in enumerate(cols):
        for k in range(0, c.shape[0], 256):
            x = c[k:k + 256].double()
            x = _shifted(x) if t == 2 else x
            F = x.shape[1]
            mn, mx = x.amin(1) - 0.000000005, x.amax(1) + 0.000000005
            mn = mn.clamp(min=0.0)
            mx = mx if t == 0 else mx.clamp(max=math.pi if t == 1 else TWO_PI)
            mx = torch.where(mx - mn < 1.0e-4, mx + 0.05, mx)
            for b in (bins[t], bins[3 + t]):
                size = (mx - mn) / b
                i = ((x - mn[:, None]) / size[:, None]).long()
                n = torch.zeros(x.shape[0], b, dtype=torch.float64, device=x.device).scatter_add_(1, i, torch.ones_like(x))
                mid = mn[:, None] + size[:, None] * (torch.arange(b, device=x.device, dtype=torch.float64) + 0.5)
                jac = mid * mid if t == 0 else torch.sin(mid) if t == 1 else torch.ones_like(mid)
                lnj = torch.where(n > 0, torch.log(jac), torch.zeros_like(jac))
                if b == bins[t] and len(s1) == len(con):
                    p = torch.xlogy(n / F, n / F).sum(1)
                    s1.append(-p + torch.log(size) + (n * lnj).sum(1) / F + ((n > 0).double().sum(1) - 1.0) / (2.0 * F))
                if b == bins[3 + t] and len(con) < len(s1):
                    last = torch.log(size) + (n * lnj).sum(1) / F
                    keep = i.to(torch.int16)
            con.append(last)
            idx.append(keep)
    return idx, torch.cat(s1), torch.cat(con)


def _pair_entropies(cols, bins):
    """The body of a trajectory, flat: the counts from products of one-hot matrices (exact in 32-bit floats below 2^24)."""
    F, n_dih = cols[0].shape[1], cols[2].shape[0]
    parts, s1, con = _dofs(cols, bins)
    nb, na = n_dih + 2, n_dih + 1
    tb = [bins[3]] * nb + [bins[4]] * na + [bins[5]] * n_dih
    idx = torch.cat(parts)
    D, B = idx.shape[0], max(bins[3:])
    S = torch.zeros(D, D, dtype=torch.float64, device=idx.device)
    blk = max(1, min(D, int(3e9 // (F * B * 4)), 4000 // B))
    one = torch.arange(B, device=idx.device, dtype=torch.int16)

    def hot(k):
        return (idx[k:k + blk, None, :] == one[None, :, None]).float().reshape(-1, F)

    old = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True  # zeros and ones: no digit is lost
    try:
        for r in range(0, D, blk):
            R = hot(r)
            for c in range(r, D, blk):
                C = R if c == r else hot(c)
                n = (R @ C.T).double().reshape(R.shape[0] // B, B, C.shape[0] // B, B)
                h = torch.xlogy(n, n).sum((1, 3))
                occ = (n > 0).double().sum((1, 3))
                S[r:r + blk, c:c + blk] = math.log(F) + con[r:r + blk, None] + con[None, c:c + blk] - h / F + (occ - 1.0) / (2.0 * F)
    finally:
        torch.backends.cuda.matmul.allow_tf32 = old
    assert len(tb) == D
    lo, n = {"b": 0, "a": nb, "d": nb + na}, {"b": nb, "a": na, "d": n_dih}
    flat = [s1]
    for p in ("bb", "ba", "bd", "aa", "ad", "dd"):
        q = S[lo[p[0]]:lo[p[0]] + n[p[0]], lo[p[1]]:lo[p[1]] + n[p[1]]]
        if p[0] == p[1]:
            i, j = torch.triu_indices(n[p[0]], n[p[0]], 1, device=S.device)
            flat.append(q[i, j].flip(0))
        else:
            flat.append(q.reshape(-1))
    S = torch.triu(S, 1)
    mi = torch.triu(s1[:, None] + s1[None, :] - S, 1)
    return torch.cat(flat).cpu().numpy(), s1.cpu().numpy(), (mi + mi.T).cpu().numpy()


def _exact_tree(n_dih, s1, M):
    """Prim's tree from bond 0: the MI of every edge in the order of joining, and the ten totals."""
    D, nb, na = 3 * n_dih + 3, n_dih + 2, n_dih + 1
    typ = np.array([0] * nb + [1] * na + [2] * n_dih)
    key, frm, out = M[0].copy(), np.zeros(D, int), np.ones(D, bool)
    out[0] = False
    mi, pair = [], np.zeros(6)
    for _ in range(D - 1):
        v = int(np.argmax(np.where(out, key, -np.inf)))
        mi.append(key[v])
        a, b = sorted((typ[frm[v]], typ[v]))
        pair[b if a == 0 else 2 + b if a == 1 else 5] += key[v]
        out[v] = False
        better = out & (M[v] > key)
        key[better], frm[better] = M[v][better], v
    s = [s1[:nb].sum(), s1[nb:nb + na].sum(), s1[nb + na:].sum()]
    return np.array(mi), np.array(s + list(pair) + [sum(s) - sum(mi)])


def exact(case, seed):
    gen = _gen(seed)
    none = dict.fromkeys(("t1", "t2", "i1", "i2", "left"))
    if case["kind"] == "mist":
        body = _body(case["atoms"], gen)
        n_dih = body.n_dih
        nb, na = n_dih + 2, n_dih + 1
        D, lo, n = 3 * n_dih + 3, {"b": 0, "a": nb, "d": nb + na}, {"b": nb, "a": na, "d": n_dih}
        s1 = np.concatenate([body.blocks["s1_" + t] for t in "bad"])
        S = np.zeros((D, D))
        for p in ("bb", "ba", "bd", "aa", "ad", "dd"):
            q = S[lo[p[0]]:lo[p[0]] + n[p[0]], lo[p[1]]:lo[p[1]] + n[p[1]]]
            if p[0] == p[1]:
                q[np.triu_indices(n[p[0]], 1)] = body.blocks[p][::-1]
            else:
                q[:] = body.blocks[p].reshape(n[p[0]], n[p[1]])
        mi = np.triu(s1[:, None] + s1[None, :] - S, 1)
        e, t = _exact_tree(n_dih, s1, mi + mi.T)
        return {**none, "mi": e, "totals": t}
    bins = _bins(case)
    systems = _systems(case) if case["kind"] == "batch" else [(case["atoms"], case["frames"])]
    # the one-hot products: over about 20 seconds there is no value
    if sum((3 * a - 6.0) ** 2 * max(bins[3:]) ** 2 * f for a, f in systems) > 3.0e15:
        return None
    if case["kind"] == "cartesian":
        cols = _bat_columns(*_coordinates(case["atoms"], case["frames"], gen))
        all_cols = [cols]
    else:
        all_cols = (_columns(a, f, case["prec"], gen) for a, f in systems)
    flats, edges, totals = [], [], []
    for (atoms, _), cols in zip(systems, all_cols):
        flat, s1, M = _pair_entropies(cols, bins)
        e, t = _exact_tree(atoms - 3, s1, M)
        flats.append(flat)
        edges.append(e)
        totals.append(t)
    if case["kind"] == "batch":
        return {"bodies": flats, "edges": {**none, "mi": np.concatenate(edges), "totals": np.stack(totals)}}
    return {"body": flats[0], **none, "mi": edges[0], "totals": totals[0]}
