"""The work that users of galaxy_b200 have it do, as cases that can be timed and checked.

A case is a dict of plain values. ``prepare`` makes what a program holds before the call
(a state and a handle), ``run`` is one pass through the public entry points, ``exact`` is
the same answer in 64 bits by plain torch (a Barnes-Hut walk over the same Morton tree,
direct sums for energies and for the SPH neighbour loops).

Ranges: gravity from 512 to 2,097,152 particles (the collision, Plummer and disk workloads
of the benchmark), opening angles 0.3 to 0.7, FP32 and FP64 walks, monopoles and
quadrupoles, 30-bit and 63-bit keys, resident and host-array stepping, active subsets,
batches of uneven systems, gas of 8,192 to 131,072 particles, energies up to 131,072.
"""

import math

import numpy as np
import torch

import galaxy_b200 as gb
from galaxy_b200 import ic, workloads

G = 1.0


def listed():
    base = dict(theta=0.5, eps=0.02, dt=5e-4, precision="f32", multipole="mono", morton63=False)
    return [
        # An interactive viewer: one step of a small cluster, the picture read back each time.
        dict(base, name="viewer 512", path="resident", ic="plummer", n=512, eps=0.05, dt=1e-3, steps=1),
        # The single Plummer sphere with quadrupole nodes (the plain configuration).
        dict(base, name="plummer 16384 quad", path="resident", ic="plummer", n=16384, eps=0.01, dt=1e-3,
             multipole="quad", steps=20),
        # The two-galaxy collision, 2 x 524,288: the headline workload, stepped resident.
        dict(base, name="collision 1048576", path="resident", ic="collision", n=1048576, ratio=1.0, steps=8),
        # The largest run: mass ratio 1:3, the widest opening angle (boxes are tested too), 63-bit keys.
        dict(base, name="collision 2097152 wide", path="resident", ic="collision", n=2097152, ratio=3.0,
             theta=0.7, morton63=True, steps=6),
        # The drop-in ForceSolver on host arrays, an odd size in the middle of the range.
        dict(base, name="force disk 200003", path="force", ic="disk", n=200003, eps=0.01),
        # The same call in the reference's own FP64 arithmetic: validation runs.
        dict(base, name="force f64 30011", path="force", ic="plummer", n=30011, eps=0.01, precision="f64"),
        # Block time steps: 2% of a galaxy's particles are due.
        dict(base, name="active 2% of 300007", path="active", ic="disk", n=300007, eps=0.01, share=0.02),
        # LeapfrogKdk on the caller's pinned arrays, a whole step end to end, small opening angle.
        dict(base, name="host step 262144", path="host", ic="collision", n=262144, ratio=2.0, theta=0.4, steps=1),
        # Many uneven systems stepped together (half Plummer spheres, half disks).
        dict(base, name="batch of 24", path="batch", ic="both", n=32768, eps=0.01, systems=24, morton63=True,
             steps=4),
        # Gas and stars stepped resident: gravity on all, density and hydro on the gas.
        dict(base, name="gas 65536+65536", path="gas", ic="mix", n=65536, stars=65536, eps=0.01, dt=1e-4,
             steps=2),
        # GravitySph on host arrays with an internal energy (adiabatic gas), odd sizes.
        dict(base, name="gas host 20011 adiabatic", path="gas_host", ic="mix", n=20011, stars=23017, eps=0.01),
        # Energy and angular momentum of a run, tracked by FP64 sums over all pairs.
        dict(base, name="energy 65537", path="energy", ic="disk", n=65537, eps=0.01),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["resident"] * 4 + ["force"] * 3 + ["active", "host", "batch", "gas", "gas_host", "energy"])
    c = dict(path=path, theta=round(rng.uniform(0.3, 0.7), 2), eps=rng.choice([0.01, 0.02, 0.05]),
             dt=rng.choice([1e-3, 5e-4]), precision="f32", multipole="mono", morton63=rng.random() < 0.4)
    if path in ("gas", "gas_host"):
        c.update(ic="mix", n=size(8192, 131072 if path == "gas" else 65536), dt=1e-4,
                 morton63=False)
        c["stars"] = int(c["n"] * rng.uniform(1.0, 2.0))
        if path == "gas":
            c["steps"] = rng.randint(1, 2)
    elif path == "batch":
        c.update(ic="both", n=size(8192, 65536), systems=rng.randint(3, 28), morton63=True, steps=rng.randint(1, 4),
                 theta=0.5)
    elif path == "energy":
        c.update(ic="disk", n=size(2048, 131072))
    else:
        c["ic"] = rng.choice(["collision", "disk", "plummer"])
        big = 32768 if c["ic"] == "plummer" and not c["morton63"] else 1048576 if path == "resident" else 524288
        c["n"] = size(512, big)
        if c["ic"] == "collision":
            c["ratio"] = round(rng.uniform(1.0, 10.0), 2)
        if path != "host" and rng.random() < 0.25:
            c["multipole"] = "quad"
        elif path == "force" and rng.random() < 0.3:
            c["precision"], c["n"] = "f64", size(512, 65536 if c["ic"] != "plummer" else 32768)
        if path == "active":
            c["share"] = round(math.exp(rng.uniform(math.log(0.002), math.log(0.5))), 4)
        if path in ("resident", "host"):
            c["steps"] = rng.randint(1, 6) if path == "resident" else 1
            c["steps"] = min(c["steps"], max(1, int(3e7 * c["theta"] ** 2 / c["n"])))
    return c


def _state(c, seed):
    if c["ic"] == "plummer":
        return ic.plummer(c["n"], seed)
    if c["ic"] == "disk":
        st = ic.disk_galaxy(c["n"], seed)
        if c["path"] == "energy":  # a galaxy on its way, so that the momentum sums are not zero
            st.pos += np.array([3.0, -2.0, 1.0])
            st.vel += np.array([0.3, -0.2, 0.1])
        return st
    if c["ic"] == "collision":
        return ic.collision(c["n"], seed, mass_ratio=c["ratio"], pericentre=4.0, incl1_deg=30.0, incl2_deg=60.0)
    st = workloads.gas_star_mix(c["n"], c["stars"], seed)
    st.u[:] = np.where(st.kind == 1, np.random.default_rng(seed + 1).uniform(0.5, 1.5, len(st)), 0.0)
    return st


def _systems(c, seed):
    """The batch: sizes from 1/8 of n to n, log-uniform (the case's own, whatever the seed),
    Plummer spheres and disks in turn."""
    rng = np.random.default_rng(c["n"])
    out = []
    for i in range(c["systems"]):
        n = int(math.exp(rng.uniform(math.log(c["n"] / 8), math.log(c["n"]))))
        st = ic.plummer(n, seed * 1009 + i) if i % 2 == 0 else ic.disk_galaxy(n, seed * 1009 + i)
        out.append((st, c["dt"] if (i // 2) % 2 == 0 else 2 * c["dt"]))
    return out


def _active(c, seed):
    k = max(1, int(c["share"] * c["n"]))
    return np.sort(np.random.default_rng(seed).choice(c["n"], k, replace=False)).astype(np.int64)


class _Held(np.ndarray):
    """A view that keeps the owner of its pinned memory alive."""

    owner = None


def _held(a, owner):
    v = a.view(_Held)
    v.owner = owner
    return v


def prepare(case, seed):
    c, path = case, case["path"]
    kw = dict(precision=c["precision"], multipole=c["multipole"], morton63=c["morton63"])
    s = {"case": c}
    if path == "batch":
        s["h"] = gb.Batch(**kw)
        s["ids"] = [s["h"].add(st, G, c["eps"], c["theta"], dt) for st, dt in _systems(c, seed)]
        return s
    st = s["state"] = _state(c, seed)
    if path in ("resident", "energy"):
        s["h"] = gb.GpuResidentLeapfrog(G, c["eps"], c["theta"], **kw)
        s["h"].upload(st)
    elif path == "gas":
        s["h"] = gb.GpuResidentLeapfrog.new_with_sph(G, c["eps"], c["theta"], **kw)
        s["h"].upload(st)
    elif path == "gas_host":
        s["h"] = gb.GpuGravitySph(G, c["eps"], c["theta"], sph=dict(eos="adiabatic", warm_start=0), **kw)
    else:
        s["h"] = gb.GpuLbvh(G, c["eps"], c["theta"], **kw)
        if path == "host":
            s["pinned"], s["primed"] = gb.PinnedState.from_state(st), False
        if path == "active":
            s["active"] = _active(c, seed)
    return s


def run(state):
    c, h = state["case"], state["h"]
    path = c["path"]
    if path in ("resident", "gas"):
        h.step_many(c["dt"], c["steps"])
        st = h.snapshot()
        out = {"pos": st.pos, "vel": st.vel}
        if path == "gas":
            d = h.snapshot_gas_density()
            out.update(rho=d.rho, h=d.h)
        return out
    if path == "force":
        return h.accelerations(state["state"])
    if path == "active":
        return h.accelerations_active(state["state"], state["active"])
    if path == "host":
        p = state["pinned"]
        state["primed"] = h.kdk_step_host(p, c["dt"], state["primed"])
        return {k: _held(getattr(p, k), p) for k in ("pos", "vel", "acc")}
    if path == "batch":
        h.step(c["steps"])
        out = [h.snapshot(i) for i in state["ids"]]
        return [(st.pos, st.vel) for st in out]
    if path == "gas_host":
        return h.accel_and_dudt(state["state"])
    d = h.diagnostics()
    return {"energies": np.array([d[k] for k in ("kinetic", "potential", "total")]), "momentum": d["momentum"],
            "angular_momentum": d["angular_momentum"]}


def _terms(n, theta):
    """Terms per particle of a walk (fits the counted walks of the collision and the disks)."""
    return min(n - 1.0, 19.0 * max(1.0, math.log2(n)) / theta ** 2)


def work(case):
    """Bytes: the state once in and once out per step (positions, velocities, masses,
    accelerations). Flops: 20 a monopole term, 55 with the quadrupole, 15 a pair of the
    energy's double sum; gas: about 60 neighbours in the density and in the force."""
    c, n = case, case["n"]
    path, steps = c["path"], c.get("steps", 1)
    per = 55 if c["multipole"] == "quad" else 20
    if path == "batch":
        n = int(c["systems"] * c["n"] * 0.42)  # mean of the log-uniform sizes
        return {"bytes": 152.0 * n * steps, "flops": float(per) * n * _terms(c["n"] / 2, c["theta"]) * steps}
    if path == "energy":
        return {"bytes": 56.0 * n, "flops": 7.5 * n * n}
    if path in ("gas", "gas_host"):
        t = n + c["stars"]
        return {"bytes": 152.0 * t * steps, "flops": steps * (20.0 * t * _terms(t, c["theta"]) + n * 60.0 * (12 * 15 + 60))}
    if path == "active":
        return {"bytes": 32.0 * n + 24.0 * n * c["share"], "flops": per * n * c["share"] * _terms(n, c["theta"])}
    if path == "force":
        return {"bytes": 56.0 * n, "flops": per * n * _terms(n, c["theta"])}
    return {"bytes": 152.0 * n * steps, "flops": per * n * _terms(n, c["theta"]) * steps}


def tolerance(case):
    """About four times what the paths were measured to be off ``exact`` (or more where other
    draws of the range are harder)."""
    path = case["path"]
    if path == "energy":
        return {"rel": 1e-11}  # FP64 sums of n^2 terms in another order
    if path == "gas_host":
        return {"rel": 2e-7, "max": 1e-4}  # FP32 gravity beside FP64 hydro
    if path in ("resident", "batch", "gas", "host") and case["precision"] == "f32":
        # an FP32 force moves an FP64 velocity by dt times its rounding; "host" returns the force too
        return {"rel": 1e-6, "max": 4e-5} if path == "host" else {"rel": 1e-8, "max": 1e-6}
    if case["precision"] == "f64":
        return {"rel": 1e-12, "max": 1e-10}
    return {"rel": 2e-6, "max": 4e-5}  # FP32 terms and sums


# ---- the same answers in 64 bits, in plain torch ----------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(_dev())


def _high_bit(x):
    hb = torch.zeros_like(x)
    for s in (32, 16, 8, 4, 2, 1):
        m = x >= (1 << s)
        hb += s * m
        x = torch.where(m, x >> s, x)
    return hb


def _tree(x, m, bits, quad):
    """The radix tree over the Morton order of x, folded: nodes 0..n-1 are the leaves in
    that order, node n + j is the split between leaves j and j + 1."""
    n, dev = x.shape[0], x.device
    lo, hi = x.min(0).values, x.max(0).values
    half = max(0.5 * float((hi - lo).max()), 1e-12) * (1.0 + 1e-9)
    side = 1 << bits
    lane = torch.floor((x - ((lo + hi) * 0.5 - half)) * (side / (2.0 * half))).clamp(0, side - 1).long()
    code = torch.zeros(n, dtype=torch.long, device=dev)
    for b in range(bits):
        for a in range(3):
            code |= ((lane[:, a] >> b) & 1) << (3 * b + a)
    code, order = torch.sort(code, stable=True)
    i = torch.arange(n, device=dev)
    j = i[:-1]
    cx = code[:-1] ^ code[1:]
    delta = torch.where(cx != 0, 63 - _high_bit(cx), 64 + 31 - _high_bit(j ^ (j + 1)))
    levels = torch.unique(delta).tolist()
    left, right = torch.zeros_like(j), torch.zeros_like(j)
    for d in levels:
        sep = delta < d
        before = torch.cummax(torch.where(sep, j, -1), 0).values
        after = torch.where(sep, j, n - 1).flip(0).cummin(0).values.flip(0)
        at = delta == d
        left[at], right[at] = before[at] + 1, after[at]
    big = torch.cat([torch.full((1,), -1, device=dev), delta, torch.full((1,), -1, device=dev)])
    kids = torch.zeros(n - 1, 2, dtype=torch.long, device=dev)
    for ids, l, r in ((i, i, i), (n + j, left, right)):
        dl, dr = big[l], big[r + 1]
        own = (dl >= 0) | (dr >= 0)  # the root has no parent
        isl = dr > dl
        kids[r[own & isl], 0] = ids[own & isl]
        kids[(l - 1)[own & ~isl], 1] = ids[own & ~isl]
    com = torch.zeros(2 * n - 1, 3, dtype=torch.float64, device=dev)
    mass = torch.zeros(2 * n - 1, dtype=torch.float64, device=dev)
    com[:n], mass[:n] = x[order], m[order]
    mn, mx = com.clone(), com.clone()
    q = torch.zeros(2 * n - 1, 6, dtype=torch.float64, device=dev) if quad else None
    for d in reversed(levels):
        g = torch.nonzero(delta == d).squeeze(1)
        a, b = kids[g, 0], kids[g, 1]
        u = n + g
        mass[u] = mass[a] + mass[b]
        mn[u], mx[u] = torch.minimum(mn[a], mn[b]), torch.maximum(mx[a], mx[b])
        com[u] = (com[a] * mass[a, None] + com[b] * mass[b, None]) / mass[u, None]
        if quad:
            for k in (a, b):
                e = com[k] - com[u]
                e2 = (e * e).sum(1)
                f = torch.stack([3 * e[:, 0] ** 2 - e2, 3 * e[:, 0] * e[:, 1], 3 * e[:, 0] * e[:, 2],
                                 3 * e[:, 1] ** 2 - e2, 3 * e[:, 1] * e[:, 2], 3 * e[:, 2] ** 2 - e2], 1)
                q[u] += q[k] + mass[k, None] * f
    root = int(n + torch.argmin(delta))
    ctr, hf = (mn + mx) * 0.5, (mx - mn) * 0.5
    off = torch.sqrt(((com - ctr) ** 2).sum(1))
    return dict(n=n, order=order, com=com, mass=mass, ctr=ctr, hf=hf, off=off, size=2 * hf.max(1).values, kids=kids,
                q=q, root=root)


def _gravity(x, m, c, rows=None):
    """Barnes-Hut accelerations (of the given rows) by the reference's opening rule."""
    if x.shape[0] < 2:
        return torch.zeros_like(x)
    t = _tree(x, m, 21 if c["morton63"] else 10, c["multipole"] == "quad" and c["precision"] == "f32")
    n, eps2, theta = t["n"], c["eps"] ** 2, c["theta"]
    inv = torch.empty_like(t["order"])
    inv[t["order"]] = torch.arange(n, device=x.device)
    slots = torch.arange(n, device=x.device) if rows is None else inv[rows]
    acc = torch.zeros(n, 3, dtype=torch.float64, device=x.device)
    xs = t["com"][:n]
    for k in range(0, slots.shape[0], 32768):
        i = slots[k:k + 32768]
        u = torch.full_like(i, t["root"])
        while i.numel():
            d = t["com"][u] - xs[i]
            d2 = (d * d).sum(1)
            leaf, mu = u < n, t["mass"][u]
            inside = ((xs[i] - t["ctr"][u]).abs() <= t["hf"][u]).all(1)
            far = ~inside & (theta * (torch.sqrt(d2) - t["off"][u]) >= t["size"][u])
            take = torch.where(leaf, u != i, far) & (mu > 0)
            a, r2 = i[take], d2[take] + eps2
            dt_, ut = d[take], u[take]
            r = torch.sqrt(r2)
            f = dt_ * (mu[take] / (r2 * r))[:, None]
            if t["q"] is not None:
                Q = t["q"][ut]
                Qd = torch.stack([(Q[:, :3] * dt_).sum(1),
                                  Q[:, 1] * dt_[:, 0] + Q[:, 3] * dt_[:, 1] + Q[:, 4] * dt_[:, 2],
                                  Q[:, 2] * dt_[:, 0] + Q[:, 4] * dt_[:, 1] + Q[:, 5] * dt_[:, 2]], 1)
                r5 = r2 * r2 * r
                f += (2.5 * (dt_ * Qd).sum(1) / (r5 * r2))[:, None] * dt_ - Qd / r5[:, None]
            acc.index_add_(0, a, f)
            go = ~leaf & ~take & (mu > 0)
            i = i[go].repeat_interleave(2)
            u = t["kids"][u[go] - n].reshape(-1)
    out = torch.zeros_like(acc)
    out[t["order"]] = acc
    return G * out


def _w(q):
    return torch.where(q < 1, 1 - 1.5 * q * q + 0.75 * q ** 3, torch.where(q < 2, 0.25 * (2 - q) ** 3, torch.zeros_like(q)))


def _dw(q):
    return torch.where(q < 1, -3 * q + 2.25 * q * q, torch.where(q < 2, -0.75 * (2 - q) ** 2, torch.zeros_like(q)))


_CHUNK = 1024


def _density(x, m, hint=None, n_ngb=48.0, tol=1e-3):
    """Adaptive smoothing lengths by the reference's bracket and bisection, and densities."""
    n = x.shape[0]
    ext = x.max(0).values - x.min(0).values
    diag = float(torch.sqrt((ext * ext).sum()))
    s_est = (float(ext.prod()) / n) ** (1.0 / 3.0)
    scale = (3.0 * n_ngb / (32.0 * math.pi)) ** (1.0 / 3.0)
    cap = max(64.0 * s_est * scale, 4.0 * diag)
    cell = torch.floor(x / (4.0 * s_est)).long()
    _, where, cnt = torch.unique(cell, dim=0, return_inverse=True, return_counts=True)
    seed = torch.clamp(4.0 * s_est / cnt[where].double() ** (1.0 / 3.0) * scale, max=cap)
    if hint is not None:
        seed = hint
    rho, hs = torch.zeros_like(m), torch.zeros_like(m)
    for k in range(0, n, _CHUNK):
        xi = x[k:k + _CHUNK]
        lo, hi = torch.clamp(seed[k:k + _CHUNK] / 2, max=cap), torch.clamp(seed[k:k + _CHUNK] * 2, max=cap)
        d2 = sum((xi[:, None, a] - x[None, :, a]) ** 2 for a in range(3))

        def pairs(radius):
            i, j = torch.nonzero(d2 <= (radius * radius)[:, None], as_tuple=True)
            return i, j, torch.sqrt(d2[i, j])

        def count(h, p):
            s = torch.zeros_like(h).index_add_(0, p[0], _w(p[2] / h[p[0]]))
            return 32.0 / 3.0 * s

        p = pairs(2 * hi)
        for _ in range(64):
            grow = (count(hi, p) < n_ngb) & (hi < cap)
            if not bool(grow.any()):
                break
            hi = torch.where(grow, torch.clamp(2 * hi, max=cap), hi)
            p = pairs(2 * hi)
        for _ in range(60):
            shrink = count(lo, p) > n_ngb
            if not bool(shrink.any()):
                break
            lo = torch.where(shrink, lo / 2, lo)
        at_hi = count(hi, p) < n_ngb
        at_lo = ~at_hi & (count(lo, p) > n_ngb)
        a, b = lo.clone(), hi.clone()
        for _ in range(64):
            go = (b - a > tol * b) & ~at_hi & ~at_lo
            if not bool(go.any()):
                break
            mid = 0.5 * (a + b)
            less = count(mid, p) < n_ngb
            a, b = torch.where(go & less, mid, a), torch.where(go & ~less, mid, b)
        h = torch.where(at_hi, hi, torch.where(at_lo, lo, 0.5 * (a + b)))
        w = m[p[1]] * _w(p[2] / h[p[0]]) / (math.pi * h[p[0]] ** 3)
        rho[k:k + _CHUNK] = torch.zeros_like(h).index_add_(0, p[0], w)
        hs[k:k + _CHUNK] = h
    return rho, hs


def _hydro(x, v, m, rho, h, u=None, c_s=1.0, gamma=5.0 / 3.0, alpha=1.0, beta=2.0, eps2=0.01):
    """Symmetric pressure and Monaghan viscosity forces, and du/dt."""
    n = x.shape[0]
    term = (gamma - 1) * u / rho if u is not None else c_s * c_s / rho
    cs = torch.sqrt(gamma * (gamma - 1) * u) if u is not None else torch.full_like(rho, c_s)
    acc, dudt = torch.zeros_like(x), torch.zeros_like(rho)
    for k in range(0, n, _CHUNK):
        xi, hk = x[k:k + _CHUNK], h[k:k + _CHUNK]
        d2 = sum((xi[:, None, a] - x[None, :, a]) ** 2 for a in range(3))
        hm = 2 * torch.maximum(hk[:, None], h[None, :])
        i, j = torch.nonzero((d2 < hm * hm) & (d2 > 0), as_tuple=True)
        i = i + k
        rv, vv = x[i] - x[j], v[i] - v[j]
        r = torch.sqrt((rv * rv).sum(1))
        g = sum(_dw(r / hh) / (math.pi * hh ** 4 * r) for hh in (h[i], h[j])) * 0.5
        grad = rv * g[:, None]
        vr = (vv * rv).sum(1)
        hb = 0.5 * (h[i] + h[j])
        mu = torch.where(vr < 0, hb * vr / (r * r + eps2 * hb * hb), torch.zeros_like(vr))
        visc = (-alpha * 0.5 * (cs[i] + cs[j]) * mu + beta * mu * mu) / (0.5 * (rho[i] + rho[j]))
        acc.index_add_(0, i, grad * (-m[j] * (term[i] + term[j] + visc))[:, None])
        dudt.index_add_(0, i, m[j] * (term[i] + 0.5 * visc) * (vv * grad).sum(1))
    return acc, dudt


def _kdk(st, dt, steps, force):
    x, v = _t(st.pos), _t(st.vel)
    a = force(x, v)
    for _ in range(steps):
        v = v + a * (0.5 * dt)
        x = x + v * dt
        a = force(x, v)
        v = v + a * (0.5 * dt)
    return x, v, a


def exact(case, seed):
    c, path = case, case["path"]
    if path == "batch":
        out = []
        for st, dt in _systems(c, seed):
            m = _t(st.mass)
            out.append(_kdk(st, dt, c["steps"], lambda x, v: _gravity(x, m, c))[:2])
        return out
    if path in ("resident", "host") and c["n"] * (c["steps"] + 1) / c["theta"] ** 2 > 6e7:
        return None
    st = _state(c, seed)
    x, v, m = _t(st.pos), _t(st.vel), _t(st.mass)
    if path == "energy":
        ke = 0.5 * float((m * (v * v).sum(1)).sum())
        pe = 0.0
        for k in range(0, len(st), _CHUNK):
            d2 = sum((x[k:k + _CHUNK, None, a] - x[None, :, a]) ** 2 for a in range(3)) + c["eps"] ** 2
            i = torch.arange(d2.shape[0], device=x.device)
            w = m[k:k + _CHUNK, None] * m[None, :] / torch.sqrt(d2)
            w[i, k + i] = 0.0
            pe -= 0.5 * G * float(w.sum())
        return {"energies": np.array([ke, pe, ke + pe]), "momentum": (m[:, None] * v).sum(0),
                "angular_momentum": (m[:, None] * torch.linalg.cross(x, v)).sum(0)}
    if path in ("gas", "gas_host"):
        g = _t(st.kind) > 0
        hint = [None]

        def force(x, v):
            a = _gravity(x, m, c)
            rho, h = _density(x[g], m[g], hint[0])
            hint[0] = h
            u = _t(st.u)[g] if path == "gas_host" else None
            ah, du = _hydro(x[g], v[g], m[g], rho, h, u)
            a[g] += ah
            return (a, rho, h, du)

        if path == "gas_host":
            a, _, _, du = force(x, v)
            dudt = torch.zeros_like(m)
            dudt[g] = du
            return a, dudt
        last = []

        def step(x, v):
            last[:] = force(x, v)
            return last[0]

        x, v, _ = _kdk(st, c["dt"], c["steps"], step)
        return {"pos": x, "vel": v, "rho": last[1], "h": last[2]}
    if path == "active":
        return _gravity(x, m, c, torch.from_numpy(_active(c, seed)).to(x.device))
    if path == "force":
        return _gravity(x, m, c)
    x, v, a = _kdk(st, c["dt"], c["steps"], lambda x, v: _gravity(x, m, c))
    return {"pos": x, "vel": v, "acc": a} if path == "host" else {"pos": x, "vel": v}
