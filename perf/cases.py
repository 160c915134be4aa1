"""Performance cases of the DMK energy library, each one pass through the
public Python interface (pdmk4mc_b200), with an FP64 Ewald value to hold the
outputs against.

A case is a dict of plain values:
  op         "energy", "trial", "moves", "candidates", "replicas", "potential"
  n          particles (replicas: the largest replica)
  digits     3, 6, 9 or 12
  precision  "fp64" or "mixed"
  layout     "uniform", or "clustered" (64 Gaussian clusters, sigma = L / 40,
             over a 20 % uniform background)
  leaf       n_per_leaf
  source     "host" or "device": where the positions of an energy lie
  count      moves, candidates, points or replicas of one pass
  step       largest displacement per axis of a trial move
The box has density one (L = n^(1/3)); charges are +1 and -1 in turn, an odd
system ends with a +2, -1, -1 triple so that every system is neutral.
"""
import math

import numpy as np
import torch

import pdmk4mc_b200 as P

MODES = {3: (4, 6), 6: (8, 12), 9: (13, 19), 12: (17, 26)}  # window and difference modes per half axis
PRECISION = {"fp64": P.PRECISION_FP64, "mixed": P.PRECISION_MIXED}


def case(name, op, n, digits, precision="fp64", layout="uniform", leaf=200, source="device", count=1, step=0.3):
    return dict(name=name, op=op, n=n, digits=digits, precision=precision, layout=layout, leaf=leaf, source=source,
                count=count, step=step)


def listed():
    return [
        # one energy of a small system from host arrays, as the example program does it: launches and host latency
        case("energy_1e3_d6", "energy", 1000, 6, leaf=10, source="host"),
        # the interface's default accuracy and leaf size at a size of the runtime benchmark, host arrays
        case("energy_128e3_d3", "energy", 128000, 3, source="host"),
        # the energy of an ordinary system at the 1e-8 setting, both precisions of the largest one after it
        case("energy_1e5_d9_mixed", "energy", 100000, 9, "mixed"),
        case("energy_1e6_d9_mixed", "energy", 1000000, 9, "mixed"),
        case("energy_1e6_d9_fp64", "energy", 1000000, 9, "fp64"),
        # an adaptive tree over a nonuniform system of odd size at the highest accuracy
        case("energy_clustered_d12_mixed", "energy", 200001, 12, "mixed", layout="clustered"),
        # the host's own Metropolis loop: one trial shift, and its update when it is accepted
        case("trial_1e3_d6", "trial", 1000, 6, leaf=10, step=0.5),
        # Metropolis sweeps on the device, ordinary and largest, the configuration read at the end of each
        case("moves_1e5_d9", "moves", 100000, 9, count=2000),
        case("moves_1e6_d9", "moves", 1000000, 9, "mixed", count=4000),
        # many candidates against one state (multiple-try and rejection-free schemes)
        case("candidates_1e6_d9", "candidates", 1000000, 9, "mixed", count=4096, step=0.5),
        # a set of uneven replicas: a full energy and 64 trial moves of each
        case("replicas_256_d9", "replicas", 50000, 9, "mixed", count=256),
        # potentials and fields at some of the particles (forces, reweighting)
        case("potential_1e5_d9", "potential", 100000, 9, count=4097),
    ]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["energy", "energy", "energy", "trial", "moves", "moves", "candidates", "replicas", "potential"])
    digits = rng.choice([3, 6, 9, 9, 12])
    precision = rng.choice(["fp64", "mixed"])
    layout = rng.choice(["uniform", "uniform", "clustered"]) if op != "replicas" else "uniform"
    # deep 12-digit trees and clustered ones hold many large expansion rows
    n = log_uniform(rng, 1000, 1000000 if digits < 12 and layout == "uniform" else 200001)
    if op == "replicas":
        n = log_uniform(rng, 4000, 50000)
    leaf = 200 if n >= 40000 else max(8, n // 128)
    count = {"energy": 1, "trial": 1, "moves": log_uniform(rng, 16, 4000), "candidates": log_uniform(rng, 1, 4096),
             "replicas": log_uniform(rng, 4, 64 if digits == 12 else 256), "potential": log_uniform(rng, 1, 4097)}[op]
    c = case("", op, n, digits, precision, layout, leaf, rng.choice(["host", "device"]), count,
             round(rng.uniform(0.1, 0.5), 2))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs


def box(n):
    return float(n) ** (1.0 / 3.0)


def charges(n):
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    if n % 2:
        q[-3:] = (2.0, -1.0, -1.0)
    return torch.from_numpy(q).cuda()


def system(n, layout, seed):
    """Positions [n, 3] in [0, L) and charges [n] on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    L = box(n)
    r = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64) * L
    if layout == "clustered":
        m = int(0.8 * n)
        centres = torch.rand((64, 3), generator=g, device="cuda", dtype=torch.float64) * L
        which = torch.randint(0, 64, (m,), generator=g, device="cuda")
        spread = torch.randn((m, 3), generator=g, device="cuda", dtype=torch.float64) * (L / 40)
        r[:m] = torch.remainder(centres[which] + spread, L)
    r[r >= L] = 0.0
    return r.contiguous(), charges(n)


def proposals(n, m, step, seed):
    rng = np.random.default_rng([int(seed), n, m])
    return rng.integers(0, n, m), rng.uniform(-step, step, (m, 3)), rng.uniform(0.0, 1.0, m)


def replica_sizes(c, seed):
    rng = np.random.default_rng([int(seed), 5])
    n = np.rint(np.exp(rng.uniform(math.log(2000), math.log(c["n"]), c["count"]))).astype(int)
    return [int(v) // 2 * 2 for v in n]


REPLICA_MOVES = 64
TRIALS = 512


def params(c, n, leaf):
    return P.HPDMKParams(n_per_leaf=leaf, digits=c["digits"], L=box(n), init=P.DIRECT)


def open_tree(c, n, leaf, r, q):
    return P.HPDMKPtTree(params(c, n, leaf), None, None, precision=PRECISION[c["precision"]],
                         device_inputs=(r.data_ptr(), q.data_ptr(), n))


def prepare(c, seed):
    if c["op"] == "replicas":
        trees, idx, disp, u = [], [], [], []
        for k, n in enumerate(replica_sizes(c, seed)):
            r, q = system(n, "uniform", seed * 1000 + k)
            torch.cuda.synchronize()
            trees.append(open_tree(c, n, max(8, n // 128), r, q))
            p = proposals(n, REPLICA_MOVES, c["step"], seed * 1000 + k)
            idx.append(p[0])
            disp.append(p[1])
            u.append(p[2])
        return dict(case=c, trees=trees, idx=np.stack(idx), disp=np.stack(disp), u=np.stack(u))
    r, q = system(c["n"], c["layout"], seed)
    torch.cuda.synchronize()
    if c["op"] == "energy":
        if c["source"] == "host":
            return dict(case=c, r=r.cpu().numpy().reshape(-1), q=q.cpu().numpy())
        return dict(case=c, r=r, q=q)
    tree = open_tree(c, c["n"], c["leaf"], r, q)
    tree.form_outgoing_pw()
    tree.form_incoming_pw()
    tree.synchronize()
    m = TRIALS if c["op"] == "trial" else c["count"]
    idx, disp, u = proposals(c["n"], m, c["step"], seed)
    return dict(case=c, tree=tree, idx=idx, disp=disp, u=u, at=0)


# ---------------------------------------------------------------------------
# one pass


def run(s):
    c = s["case"]
    op = c["op"]
    if op == "energy":
        # a full energy from raw positions: tree, outgoing and incoming expansions, the three parts
        if c["source"] == "host":
            tree = P.HPDMKPtTree(params(c, c["n"], c["leaf"]), s["r"], s["q"], precision=PRECISION[c["precision"]])
        else:
            tree = open_tree(c, c["n"], c["leaf"], s["r"], s["q"])
        tree.form_outgoing_pw()
        tree.form_incoming_pw()
        parts = tree.eval_energy_parts()
        tree.close()
        return {"energy": parts.sum(), "parts": parts}
    if op == "trial":
        k = s["at"]
        s["at"] = (k + 1) % TRIALS
        d = s["disp"][k]
        dE = s["tree"].eval_shift_energy(s["idx"][k], d[0], d[1], d[2])
        accepted = int(s["u"][k] < math.exp(min(0.0, -dE)))
        if accepted:
            s["tree"].update_shift(s["idx"][k], d[0], d[1], d[2])
        return {"dE": np.float64(dE), "accepted": accepted}
    if op == "moves":
        dE, accepted = s["tree"].mc_run(s["idx"], s["disp"], s["u"], 1.0)
        return {"dE": dE, "accepted": accepted, "positions": s["tree"].positions()}
    if op == "candidates":
        return {"dE": s["tree"].eval_shift_energy_batch(s["idx"], s["disp"])}
    if op == "replicas":
        energy = P.replicas_energy(s["trees"])
        dE, accepted = P.replicas_mc_run(s["trees"], s["idx"], s["disp"], s["u"], 1.0)
        return {"energy": energy, "dE": dE, "accepted": accepted}
    phi, field = s["tree"].potential(s["idx"])
    return {"phi": phi, "field": field}


# ---------------------------------------------------------------------------
# the work of one pass


def levels_of(n, leaf):
    """Levels that carry expansions in a uniform tree: 2 up to the leaves' parents' parents."""
    depth = 2
    while n / 8.0 ** depth > leaf:
        depth += 1
    return max(1, depth - 2)


def energy_work(n, digits, leaf):
    nw, nd = MODES[digits]
    lev = levels_of(n, leaf)
    modes = (2 * nw + 1) ** 3 + lev * (2 * nd + 1) ** 3  # real degrees of freedom of the half grids
    pairs = 0.5 * n * 4.2 * n / 8.0 ** (lev + 2)          # within one leaf size
    # an outgoing coefficient takes a product and a sum per particle, a pair a polynomial of 2 nd terms
    return 32.0 * n, 2.0 * n * modes + pairs * 2.0 * nd


def shift_work(n, digits, leaf):
    nw, nd = MODES[digits]
    lev = levels_of(n, leaf)
    modes = (2 * nw + 1) ** 3 / 2 + lev * (2 * nd + 1) ** 3 / 2
    # origin and target rows, one complex coefficient and its table value each, and the near field of both
    return 24.0 * modes + 64.0 * n / 8.0 ** (lev + 2), 2 * 8.0 * modes


def update_work(n, digits, leaf):
    nw, nd = MODES[digits]
    lev = levels_of(n, leaf)
    # the moved particle's own row of each level, read and written
    modes = (2 * nw + 1) ** 3 / 2 + lev * (2 * nd + 1) ** 3 / 2
    return 32.0 * modes, 2 * 8.0 * modes


def work(c):
    n, d, leaf = c["n"], c["digits"], c["leaf"]
    if c["op"] == "energy":
        b, f = energy_work(n, d, leaf)
    elif c["op"] == "replicas":
        b = f = 0.0
        steps = 32
        for k in range(steps):  # sizes are log-uniform
            m = 2000 * (c["n"] / 2000.0) ** ((k + 0.5) / steps)
            lf = max(8, m / 128)
            e, s, w = energy_work(m, d, lf), shift_work(m, d, lf), update_work(m, d, lf)
            b += (e[0] + REPLICA_MOVES * (s[0] + 0.75 * w[0])) * c["count"] / steps
            f += (e[1] + REPLICA_MOVES * (s[1] + 0.75 * w[1])) * c["count"] / steps
    else:
        b, f = shift_work(n, d, leaf)
        if c["op"] in ("trial", "moves"):
            w = update_work(n, d, leaf)
            b, f = b + 0.75 * w[0], f + 0.75 * w[1]
        b, f = b * c["count"], f * c["count"]
        if c["op"] in ("candidates", "potential"):
            # the candidates read one state: its incoming rows once
            rows = sum(8 ** l for l in range(2, 2 + levels_of(n, leaf)))
            b = min(b, 16.0 * rows * (2 * MODES[d][1] + 1) ** 3 / 2 + 32.0 * n)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# FP64 Ewald sums in plain torch


REACH = 5.6  # erfc(5.6) and exp(-5.6^2) are below 3e-14


def structure_factor(r, q, L, nk):
    """S(k) = sum_j q_j exp(i k.r_j) on the cube |m| <= nk, kz >= 0: [nk + 1, 2 nk + 1, 2 nk + 1]."""
    S = torch.zeros((nk + 1, 2 * nk + 1, 2 * nk + 1), dtype=torch.complex128, device=r.device)
    m = torch.arange(-nk, nk + 1, device=r.device, dtype=torch.float64) * (2 * math.pi / L)
    for at in range(0, r.shape[0], 200000):
        x, w = r[at:at + 200000], q[at:at + 200000]
        ex, ey = (torch.polar(torch.ones(1, dtype=torch.float64, device=r.device), x[:, a:a + 1] * m) for a in (0, 1))
        for kz in range(nk + 1):
            ez = torch.polar(torch.ones(1, dtype=torch.float64, device=r.device), x[:, 2] * (kz * 2 * math.pi / L)) * w
            S[kz] += (ey * ez[:, None]).T @ ex
    return S


def reciprocal_weights(nk, L, alpha, device):
    """(4 pi / V) exp(-k^2 / 4 alpha^2) / k^2 on the half cube, each mode standing for its mirror too."""
    m = torch.arange(-nk, nk + 1, device=device, dtype=torch.float64)
    z = torch.arange(0, nk + 1, device=device, dtype=torch.float64)
    k2 = (z[:, None, None] ** 2 + m[None, :, None] ** 2 + m[None, None, :] ** 2) * (2 * math.pi / L) ** 2
    w = torch.where(k2 > 0, torch.exp(-k2 / (4 * alpha ** 2)) / k2, torch.zeros_like(k2)) * (2 * math.pi / L ** 3)
    w[1:] *= 2
    return w


def screened(d2, alpha):
    """erfc(alpha r) / r from r^2, zero at r = 0."""
    r = torch.sqrt(d2)
    return torch.where(d2 > 0, torch.special.erfc(alpha * r) / r, torch.zeros_like(r))


def ewald_energy(r, q, L):
    n = r.shape[0]
    cells = 8 if n > 250000 else 1
    alpha = REACH * (2 if cells == 1 else cells) / L
    nk = math.ceil(REACH * alpha * L / math.pi)
    E = float((reciprocal_weights(nk, L, alpha, r.device) * structure_factor(r, q, L, nk).abs() ** 2).sum())
    E -= alpha / math.sqrt(math.pi) * float((q * q).sum())

    def pairs(xi, qi, xj, qj):
        t = 0.0
        rows = max(1, int(6e7 // max(1, xj.shape[0])))
        for at in range(0, xi.shape[0], rows):
            d2 = torch.zeros((min(rows, xi.shape[0] - at), xj.shape[0]), dtype=torch.float64, device=r.device)
            for a in range(3):
                d = xi[at:at + rows, a, None] - xj[None, :, a]
                d -= L * torch.round(d / L)
                d2 += d * d
            t += float(0.5 * (qi[at:at + rows] * (screened(d2, alpha) @ qj)).sum())
        return t

    if cells == 1:
        return E + pairs(r, q, r, q)
    cell = torch.clamp((r * (cells / L)).long(), max=cells - 1)
    key = (cell[:, 0] * cells + cell[:, 1]) * cells + cell[:, 2]
    order = torch.argsort(key)
    r, q, key = r[order], q[order], key[order]
    edge = torch.searchsorted(key, torch.arange(cells ** 3 + 1, device=r.device)).tolist()
    for b in range(cells ** 3):
        x, y, z = b // cells ** 2, b // cells % cells, b % cells
        near = [((x + i) % cells * cells + (y + j) % cells) * cells + (z + k) % cells
                for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)]
        xi = r[edge[b]:edge[b + 1]]
        if xi.shape[0]:
            E += pairs(xi, q[edge[b]:edge[b + 1]], torch.cat([r[edge[v]:edge[v + 1]] for v in near]),
                       torch.cat([q[edge[v]:edge[v + 1]] for v in near]))
    return E


class Shifts:
    """Ewald energy shifts of a set of systems, one move of each at a time (padded with zero charges)."""

    def __init__(self, systems):
        dev = systems[0][0].device
        top = max(r.shape[0] for r, _, _ in systems)
        R = len(systems)
        self.x = torch.zeros((R, top, 3), dtype=torch.float64, device=dev)
        self.q = torch.zeros((R, top), dtype=torch.float64, device=dev)
        self.L = torch.tensor([L for _, _, L in systems], dtype=torch.float64, device=dev)
        self.nk = nk = math.ceil(REACH * 2 * REACH / math.pi)
        self.alpha = 2 * REACH / self.L
        keep, self.w, self.S = None, [], []
        for k, (r, q, L) in enumerate(systems):
            self.x[k, :r.shape[0]] = r
            self.q[k, :r.shape[0]] = q
            w = reciprocal_weights(nk, L, 2 * REACH / L, dev).reshape(-1)
            if keep is None:
                keep = torch.nonzero(w > 1e-17 * w.max())[:, 0]
            self.w.append(w[keep])
            self.S.append(structure_factor(r, q, L, nk).reshape(-1)[keep])
        self.w, self.S = torch.stack(self.w), torch.stack(self.S)
        d = 2 * nk + 1
        self.m = torch.stack([keep % d - nk, keep // d % d - nk, keep // (d * d)]).double()

    def phases(self, x):
        k = (x * (2 * math.pi / self.L[:, None])) @ self.m
        return torch.polar(torch.ones_like(k), k)

    def near(self, x, i):
        L = self.L[:, None]
        d2 = torch.zeros_like(self.q)
        for a in range(3):
            d = x[:, a, None] - self.x[:, :, a]
            d -= L * torch.round(d / L)
            d2 += d * d
        v = self.q * screened(d2, self.alpha[:, None])
        v[self.all, i] = 0.0
        return v.sum(1)

    def shift(self, i, disp):
        """dE [R], the new positions and the change of S of moving particle i[k] of system k by disp[k]."""
        self.all = torch.arange(len(i), device=self.x.device)
        xo = self.x[self.all, i]
        L = self.L[:, None]
        xt = torch.remainder(xo + disp, L)
        xt = torch.where(xt >= L, torch.zeros_like(xt), xt)
        qi = self.q[self.all, i]
        dS = (self.phases(xt) - self.phases(xo)) * qi[:, None]
        dE = qi * (self.near(xt, i) - self.near(xo, i))
        dE = dE + (self.w * (2 * (self.S.conj() * dS).real + dS.abs() ** 2)).sum(1)
        return dE, xt, dS

    def metropolis(self, idx, disp, u):
        """Sequences [R, m] at beta = 1; dE, accepted and the final positions."""
        out, acc = [], []
        for c in range(idx.shape[1]):
            dE, xt, dS = self.shift(idx[:, c], disp[:, c])
            ok = u[:, c] < torch.exp(-dE)
            self.x[self.all, idx[:, c]] = torch.where(ok[:, None], xt, self.x[self.all, idx[:, c]])
            self.S += torch.where(ok[:, None], dS, torch.zeros_like(dS))
            out.append(dE)
            acc.append(ok)
        return torch.stack(out, 1), torch.stack(acc, 1).int(), self.x


def points(r, q, L, idx, x, mode):
    """Ewald potentials at points x [m, 3], particle idx[m] left out of the real-space sum but not of the reciprocal
    one; with the fields in mode "phi"."""
    n = r.shape[0]
    alpha = 2 * REACH / L
    nk = math.ceil(REACH * 2 * REACH / math.pi)
    w = reciprocal_weights(nk, L, alpha, r.device).reshape(-1)
    keep = torch.nonzero(w > 1e-17 * w.max())[:, 0]
    w, S = w[keep], structure_factor(r, q, L, nk).reshape(-1)[keep]
    d = 2 * nk + 1
    k = torch.stack([keep % d - nk, keep // d % d - nk, keep // (d * d)]).double() * (2 * math.pi / L)
    phi = torch.zeros(x.shape[0], dtype=torch.float64, device=r.device)
    field = torch.zeros_like(x)
    rows = max(1, int(6e7 // n))
    for at in range(0, x.shape[0], rows):
        xi, ii = x[at:at + rows], idx[at:at + rows]
        own = torch.arange(len(ii), device=r.device)
        dx = []
        d2 = torch.zeros((len(ii), n), dtype=torch.float64, device=r.device)
        for a in range(3):
            t = xi[:, a, None] - r[None, :, a]
            t -= L * torch.round(t / L)
            d2 += t * t
            dx.append(t)
        v = screened(d2, alpha)
        v[own, ii] = 0.0
        phi[at:at + rows] = v @ q
        if mode == "phi":
            g = v / d2 + (2 * alpha / math.sqrt(math.pi)) * torch.exp(-alpha * alpha * d2) / d2
            g[own, ii] = 0.0
            g *= q
            for a in range(3):
                field[at:at + rows, a] = (g * dx[a]).sum(1)
    for at in range(0, x.shape[0], 1024):
        e = torch.polar(torch.ones(1, dtype=torch.float64, device=r.device), x[at:at + 1024] @ k)
        t = S.conj() * e * (2 * w)
        phi[at:at + 1024] += t.real.sum(1)
        if mode == "phi":
            field[at:at + 1024] += t.imag @ k.T
    return phi, field


def exact(c, seed):
    """The pass's outputs from FP64 Ewald sums; the method's own parts of an energy have no such value."""
    n, L = c["n"], box(c["n"])
    dev = "cuda"
    if c["op"] == "replicas":
        systems, idx, disp, u = [], [], [], []
        for k, m in enumerate(replica_sizes(c, seed)):
            r, q = system(m, "uniform", seed * 1000 + k)
            systems.append((r, q, box(m)))
            p = proposals(m, REPLICA_MOVES, c["step"], seed * 1000 + k)
            idx.append(p[0])
            disp.append(p[1])
            u.append(p[2])
        energy = np.array([ewald_energy(r, q, l) for r, q, l in systems])
        dE, acc, _ = Shifts(systems).metropolis(*(torch.from_numpy(np.stack(v)).to(dev) for v in (idx, disp, u)))
        return {"energy": energy, "dE": dE, "accepted": acc}
    r, q = system(n, c["layout"], seed)
    if c["op"] == "energy":
        return {"energy": np.float64(ewald_energy(r, q, L)), "parts": None}
    m = TRIALS if c["op"] == "trial" else c["count"]
    idx, disp, u = (torch.from_numpy(v).to(dev) for v in proposals(n, m, c["step"], seed))
    if c["op"] == "trial":
        dE, acc, _ = Shifts([(r, q, L)]).metropolis(idx[None, :1], disp[None, :1], u[None, :1])
        return {"dE": np.float64(dE[0, 0].item()), "accepted": int(acc[0, 0])}
    if c["op"] == "moves":
        dE, acc, x = Shifts([(r, q, L)]).metropolis(idx[None], disp[None], u[None])
        return {"dE": dE[0], "accepted": acc[0], "positions": x[0].reshape(-1)}
    if c["op"] == "candidates":
        xo = r[idx]
        xt = torch.remainder(xo + disp, L)
        xt = torch.where(xt >= L, torch.zeros_like(xt), xt)
        po, pt = points(r, q, L, idx, xo, "dE")[0], points(r, q, L, idx, xt, "dE")[0]
        # |dS|^2, the particle's own share of the reciprocal sum's change
        alpha = 2 * REACH / L
        nk = math.ceil(REACH * 2 * REACH / math.pi)
        w = reciprocal_weights(nk, L, alpha, r.device).reshape(-1)
        keep = torch.nonzero(w > 1e-17 * w.max())[:, 0]
        d = 2 * nk + 1
        k = torch.stack([keep % d - nk, keep // d % d - nk, keep // (d * d)]).double() * (2 * math.pi / L)
        qi = q[idx]
        same = ((1 - torch.cos((xt - xo) @ k)) * w[keep]).sum(1)
        return {"dE": qi * (pt - po) + 2 * qi * qi * same}
    phi, field = points(r, q, L, idx, r[idx], "phi")
    # the particle's own Gaussian in the reciprocal sum
    phi = phi - q[idx] * (2 * (2 * REACH / L) / math.sqrt(math.pi))
    return {"phi": phi, "field": field}
