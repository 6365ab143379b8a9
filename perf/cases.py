"""Performance cases of the Swendsen-Wang engine: the calls its users make, over their range of sizes.

``listed()`` names the fixed cases, ``draw(rng)`` gives further ones from the same ranges, ``prepare`` builds what a
program holds before the call, ``run`` makes one pass through the public entry points and returns its outputs,
``work`` counts what a pass cannot do without, and ``exact`` replays a pass in plain torch (int64 and float64).

Kinds of case:

* ``sweep``   one ``sw_sweep`` call on host spins, the per-sweep API in a user's own loop: latency, launches, copies.
* ``single``  one ``run_single_realization`` task: one lattice, thermalisation and binned measurement.
* ``scan``    one ``run_temperature_scan`` call, disorder generation and jackknife included.
* ``batch``   a ``ChainSet`` of one size (realizations x temperatures) advanced by ``run_batched``.
* ``mix``     a ``ChainSet`` of uneven sizes advanced by ``run_batched``, as in finite-size scaling and serving.
* ``label``   ``label_and_wrap_many`` on frozen occupation masks held on the host.

Every chain of a ``batch`` or ``mix`` has been thermalised for a few sweeps by ``prepare``; each pass advances the
same chains further, so every pass is new work on new spins.
"""

from __future__ import annotations

import importlib
import math

import numpy as np
import torch

rb = importlib.import_module("rbim-fk-percolation_b200")

#: Sweeps that ``prepare`` runs before a pass on chain sets.
THERM = 12
#: Sizes of the uneven mix, and its disorder strengths.
MIX_L = (32, 48, 64, 96, 128, 192, 256, 512)
MIX_P = (0.02, 0.05, 0.08, 0.10)
#: Site-updates of a pass: the most that a drawn chain set, and a drawn single task or scan, may take.
MAX_BATCH, MAX_RUN = 5.0e8, 1.1e9


def listed():
    return [
        # A user's own loop over sw_sweep at the size of the README's scan: nothing but latency.
        {"name": "sweep_L32", "kind": "sweep", "L": 32, "p": 0.05, "T": 2.0},
        # One task of an odd size, whose tiles start inside rows (time series, quick looks at one realization).
        {"name": "single_L249", "kind": "single", "L": 249, "p": 0.08, "T": 1.8, "sweeps": 1000, "therm": 100,
         "bins": 10},
        # The large single lattice inside the percolating, non-magnetic window.
        {"name": "single_L1024", "kind": "single", "L": 1024, "p": 0.10, "T": 1.6, "sweeps": 1000, "therm": 100,
         "bins": 10},
        # The reference's headline scan, 32 realizations x 40 temperatures, with fewer sweeps.
        {"name": "scan_L32", "kind": "scan", "L": 32, "p": 0.05, "t_lo": 1.0, "t_hi": 3.0, "n_t": 40, "n_r": 32,
         "sweeps": 1000, "therm": 100, "bins": 10},
        # Many small lattices (serving requests, Binder crossings).
        {"name": "batch_L16", "kind": "batch", "L": 16, "p": 0.05, "t_lo": 1.0, "t_hi": 3.0, "n_t": 64, "n_r": 256,
         "sweeps": 50, "measure": True},
        # The uniform batch of 256 realizations x 64 temperatures.
        {"name": "batch_L64", "kind": "batch", "L": 64, "p": 0.05, "t_lo": 1.0, "t_hi": 3.0, "n_t": 64, "n_r": 256,
         "sweeps": 6, "measure": True},
        # An odd size, rows never aligned to words, during thermalisation (no measurement).
        {"name": "batch_L99_therm", "kind": "batch", "L": 99, "p": 0.08, "t_lo": 1.2, "t_hi": 2.4, "n_t": 32,
         "n_r": 128, "sweeps": 10, "measure": False},
        # A slice of the uneven-size configuration at the bench's headline size.
        {"name": "batch_L256", "kind": "batch", "L": 256, "p": 0.08, "t_lo": 1.2, "t_hi": 2.4, "n_t": 32, "n_r": 64,
         "sweeps": 4, "measure": True},
        # The same configuration at L = 512, beyond what one CTA holds.
        {"name": "batch_L512", "kind": "batch", "L": 512, "p": 0.05, "t_lo": 1.2, "t_hi": 2.4, "n_t": 32, "n_r": 16,
         "sweeps": 4, "measure": True},
        # The largest lattices that run many at a time.
        {"name": "batch_L1024", "kind": "batch", "L": 1024, "p": 0.10, "t_lo": 1.5, "t_hi": 1.7, "n_t": 32, "n_r": 4,
         "sweeps": 4, "measure": True},
        # Uneven sizes in one call: 1/64 of the finite-size-scaling configuration.
        {"name": "mix", "kind": "mix", "base": 64, "n_t": 32, "t_lo": 1.2, "t_hi": 2.4, "sweeps": 4, "measure": True},
        # Labelling of critical masks, host arrays in and out.
        {"name": "label_L256", "kind": "label", "L": 256, "n": 64, "q": 0.5},
    ]


def _log_int(rng, lo, hi):
    """An integer from lo to hi, uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("sweep", "single", "scan", "batch", "batch", "batch", "mix", "label"))
    p = round(rng.uniform(0.0, 0.12), 3)
    lo = round(rng.uniform(1.0, 1.6), 2)
    hi = round(rng.uniform(2.0, 3.0), 2)
    if kind == "sweep":
        return {"kind": kind, "L": _log_int(rng, 12, 512), "p": p, "T": round(rng.uniform(1.0, 3.0), 2)}
    if kind == "single":
        L = _log_int(rng, 16, 1024)
        sweeps = _log_int(rng, 200, max(200, min(1000, int(MAX_RUN / 1.1 / L**2))))
        return {"kind": kind, "L": L, "p": p, "T": round(rng.uniform(1.0, 3.0), 2), "sweeps": sweeps,
                "therm": sweeps // 10, "bins": 10}
    if kind == "scan":
        L, n_t, n_r = _log_int(rng, 12, 128), rng.randint(8, 40), rng.randint(4, 32)
        sweeps = max(20, min(1000, int(MAX_RUN / 1.1 / (L**2 * n_t * n_r))))
        return {"kind": kind, "L": L, "p": p, "t_lo": lo, "t_hi": hi, "n_t": n_t, "n_r": n_r, "sweeps": sweeps,
                "therm": sweeps // 10, "bins": 10}
    if kind == "batch":
        L, n_t = _log_int(rng, 12, 1024), rng.randint(8, 64)
        n_r = _log_int(rng, 2, max(2, min(256, int(1.3e8 / (L**2 * n_t)))))
        sweeps = _log_int(rng, 2, max(2, min(40, int(MAX_BATCH / (L**2 * n_t * n_r)))))
        return {"kind": kind, "L": L, "p": p, "t_lo": lo, "t_hi": hi, "n_t": n_t, "n_r": n_r, "sweeps": sweeps,
                "measure": rng.random() < 0.8}
    if kind == "mix":
        return {"kind": kind, "base": rng.randint(16, 64), "n_t": rng.randint(12, 32), "t_lo": lo, "t_hi": hi,
                "sweeps": rng.randint(2, 4), "measure": rng.random() < 0.8}
    L = _log_int(rng, 16, 512)
    n = _log_int(rng, 1, max(1, min(256, int(4.2e6 / L**2))))
    return {"kind": kind, "L": L, "n": n, "q": round(rng.uniform(0.35, 0.65), 2)}


# ---------------------------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------------------------


def _bonds(L, p, rng):
    """Bond-ordered couplings (bond 2n to x + 1, bond 2n + 1 to y + 1) of one +-J realization."""
    return np.where(rng.random(2 * L * L) < p, -1, 1).astype(np.int8)


def _groups(case):
    """(L, p, realizations) of each group of realizations of a chain set; every one runs at all temperatures."""
    if case["kind"] == "batch":
        return [(case["L"], case["p"], case["n_r"])]
    return [(L, p, max(1, round(case["base"] * (32 / L) ** 2))) for L in MIX_L for p in MIX_P]


def _chains(case, seed):
    """Couplings of a chain set's realizations, and (realization, L, beta, key) of its chains."""
    rng = np.random.default_rng([seed, 1])
    temps = np.linspace(case["t_lo"], case["t_hi"], case["n_t"])
    bonds, chains = [], []
    for L, p, n_r in _groups(case):
        base = len(bonds)
        bonds += [_bonds(L, p, rng) for _ in range(n_r)]
        keys = rng.integers(0, 2**63, size=(len(temps), n_r))
        chains += [(base + r, L, 1.0 / float(T), int(keys[i, r])) for i, T in enumerate(temps) for r in range(n_r)]
    return bonds, chains


def _run_length(case):
    """(n_therm, n_bins, sweeps_per_bin) of a chain set's chains: runs too long to end during the passes."""
    return (THERM if case["measure"] else 1 << 30, 4, 1 << 20)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "mix"):
        bonds, chains = _chains(case, seed)
        n_therm, n_bins, per_bin = _run_length(case)
        size = {r: L for r, L, _, _ in chains}
        packed = [rb.packing.pack_couplings(J, size[r]) for r, J in enumerate(bonds)]
        specs = [rb.ChainSpec(L=L, realization=r, key=key, beta=beta, n_therm=n_therm, n_bins=n_bins,
                              sweeps_per_bin=per_bin) for r, L, beta, key in chains]
        chain_set = rb.ChainSet(specs, packed)
        chain_set.init_spins(hot=True)
        chain_set.run_batched(THERM)
        return {"case": case, "chains": chain_set}
    if kind == "label":
        rng = np.random.default_rng([seed, 2])
        return {"case": case, "masks": rng.random((case["n"], 2 * case["L"] ** 2)) < case["q"]}
    state = {"case": case, "seed": seed}
    if kind == "single":
        state["J"] = _bonds(case["L"], case["p"], np.random.default_rng([seed, 3]))
    if kind == "sweep":
        rng = np.random.default_rng([seed, 4])
        L = case["L"]
        state.update(lattice=rb.build_lattice(L), J=_bonds(L, case["p"], rng), key=int(rng.integers(0, 2**63)),
                     spins=rng.integers(0, 2, size=L * L, dtype=np.int64) * 2 - 1, sweep=0)
    return state


# ---------------------------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("batch", "mix"):
        chain_set = state["chains"]
        chain_set.run_batched(case["sweeps"])
        return {"spins": chain_set.spin_pool, "sums": chain_set.acc_int, "moments": chain_set.acc_f64}
    if kind == "label":
        n, labels, wraps = rb.label_and_wrap_many(state["masks"], case["L"])
        return {"n": n, "labels": labels, "wraps": wraps}
    if kind == "sweep":
        r = rb.sw_sweep(state["spins"], state["lattice"], state["J"], 1.0 / case["T"], key=state["key"],
                        sweep=state["sweep"])
        state["sweep"] += 1
        return {"spins": state["spins"], "energy": r.energy, "magnetization": r.magnetization,
                "n_clusters": r.n_clusters, "largest_size": r.largest_size,
                "largest_abs_magnetization": r.largest_abs_magnetization, "second_size": r.second_size,
                "second_abs_magnetization": r.second_abs_magnetization, "wraps": [r.wraps_x, r.wraps_y]}
    if kind == "single":
        r = rb.run_single_realization(case["L"], state["J"], case["T"], n_sweeps=case["sweeps"],
                                      n_therm=case["therm"], n_bins=case["bins"], seed=state["seed"])
        return {"means": r.primitives, "bins": r.bin_primitives}
    r = rb.run_temperature_scan(case["L"], case["p"], np.linspace(case["t_lo"], case["t_hi"], case["n_t"]),
                                n_realizations=case["n_r"], n_sweeps=case["sweeps"], n_therm=case["therm"],
                                n_bins=case["bins"], seed=state["seed"])
    return r["observables"]


# ---------------------------------------------------------------------------------------------------------------
# The least work of a pass
# ---------------------------------------------------------------------------------------------------------------

#: Integer operations of one Philox4x32-10 block: ten rounds of two 32 x 32 -> 64 bit products (two operations each)
#: and four exclusive ors, and nine additions to each of the two key words.
PHILOX_OPS = 10 * 8 + 2 * 9


def _updates(case):
    """(site-updates of a pass, sites whose spins it reads and writes, sites of its realizations, chains)."""
    if case["kind"] == "sweep":
        n = case["L"] ** 2
        return n, n, n, 1
    if case["kind"] == "single":
        n = case["L"] ** 2
        return n * (case["sweeps"] + case["therm"]), n, n, 1
    if case["kind"] == "scan":
        n = case["L"] ** 2 * case["n_r"]
        return n * case["n_t"] * (case["sweeps"] + case["therm"]), n * case["n_t"], n, case["n_r"] * case["n_t"]
    sites = sum(L * L * n_r for L, _, n_r in _groups(case))
    reals = sum(n_r for _, _, n_r in _groups(case))
    return sites * case["n_t"] * case["sweeps"], sites * case["n_t"], sites, reals * case["n_t"]


def work(case):
    if case["kind"] == "label":
        n = case["n"] * case["L"] ** 2
        # Two occupation bytes read and one 64-bit label written a site; a compare a bond.
        return {"bytes": 10 * n, "flops": 2 * n}
    updates, spins, couplings, chains = _updates(case)
    # Spins (one bit) in and out, couplings (two bits) in, 14 sums of eight bytes a chain out.  The draws of a
    # site-update: a Philox block for the eight bonds of four sites, and one for 128 flip bits.
    return {"bytes": spins / 4 + couplings / 4 + 112 * chains, "flops": updates * PHILOX_OPS * (1 / 4 + 1 / 128)}


# ---------------------------------------------------------------------------------------------------------------
# The same pass in plain torch: int64 integers, float64 moments
# ---------------------------------------------------------------------------------------------------------------

_M32 = 0xFFFFFFFF
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _philox(block, sweep, stream, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) of counters (block, sweep, 0, stream) under keys (k0, k1), in int64."""
    c0, c1, c2, c3 = block, torch.full_like(block, sweep), torch.zeros_like(block), torch.full_like(block, stream)
    for _ in range(10):
        a, b = c0 * 0xD2511F53, c2 * 0xCD9E8D57  # the low 64 bits of each product are exact
        c0, c1, c2, c3 = ((b >> 32) & _M32) ^ c1 ^ k0, b & _M32, ((a >> 32) & _M32) ^ c3 ^ k1, a & _M32
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return torch.stack((c0, c1, c2, c3), dim=-1)


class _Replay:
    """Chains of one size: spins (n, L, L) as booleans (true: -1), advanced sweep by sweep."""

    def __init__(self, L, bonds, real, betas, keys):
        self.L, self.N, self.n = L, L * L, len(real)
        J = torch.from_numpy(np.stack(bonds)).to(_DEV).view(-1, L, L, 2) < 0
        real = torch.tensor(real, device=_DEV)
        self.neg_x, self.neg_y = J[..., 0][real], J[..., 1][real]
        self.k0 = torch.tensor([k & _M32 for k in keys], device=_DEV)[:, None]
        self.k1 = torch.tensor([(k >> 32) & _M32 for k in keys], device=_DEV)[:, None]
        thr = [int(math.floor(-math.expm1(-2.0 * b) * 4294967296.0)) for b in betas]
        self.thr = torch.tensor(thr, device=_DEV)[:, None]
        self.chunks = -(-self.N // 128)
        self.base = torch.arange(self.n, device=_DEV)[:, None] * self.N

    def _bits(self, sweep, stream):
        """Bit n & 127 of block n >> 7 of a stream for every site n, as booleans (n chains, N)."""
        block = torch.arange(self.chunks, device=_DEV)[None].expand(self.n, -1)
        words = _philox(block, sweep, stream, self.k0, self.k1).reshape(self.n, -1, 1)
        bits = (words >> torch.arange(32, device=_DEV)) & 1
        return bits.reshape(self.n, -1)[:, : self.N].bool()

    def hot(self):
        self.s = self._bits(0, 2).view(self.n, self.L, self.L)

    def _draws(self, sweep):
        """Whether each site's x and y bonds are drawn occupied, (n chains, N) booleans."""
        block = torch.arange(32 * self.chunks, device=_DEV)[None].expand(self.n, -1)
        w = _philox(block, sweep, 0, self.k0, self.k1)
        # Word s of lane i of a chunk's 32 blocks belongs to the chunk's site 32 s + i.
        w = w.view(self.n, self.chunks, 32, 4).transpose(2, 3).reshape(self.n, -1)[:, : self.N]
        out = []
        for half in (0, 16):
            u = (w >> half) & 0xFFFF
            yes = u < (self.thr >> 16)
            c, site = torch.nonzero(u == (self.thr >> 16), as_tuple=True)  # decided by 16 further bits
            if len(c):
                low = _philox(32 * (site >> 7) + (site & 31), sweep, 3, self.k0[c, 0], self.k1[c, 0])
                low = (low.gather(1, ((site >> 5) & 3)[:, None])[:, 0] >> half) & 0xFFFF
                yes[c, site] = low < (self.thr[c, 0] & 0xFFFF)
            out.append(yes.view(self.n, self.L, self.L))
        return out

    def _clusters(self, ox, oy):
        """Smallest site of each site's cluster (periodic in both directions), offset by chain."""
        label = (self.base + torch.arange(self.N, device=_DEV)).view(-1)
        far = torch.tensor(1 << 62, device=_DEV)
        bx, by = ox.roll(1, 1), oy.roll(1, 2)
        while True:
            g = label.view(self.n, self.L, self.L)
            m = g
            for o, there in ((ox, g.roll(-1, 1)), (oy, g.roll(-1, 2)), (bx, g.roll(1, 1)), (by, g.roll(1, 2))):
                m = torch.minimum(m, torch.where(o, there, far))
            new = label.scatter_reduce(0, label, m.reshape(-1), "amin")
            new = torch.minimum(new, m.reshape(-1))
            for _ in range(3):
                new = new[new]
            if torch.equal(new, label):
                return label.view(self.n, self.N) - self.base
            label = new

    def sweep(self, t, measure):
        """One sweep; measured: per chain E, M, clusters, S1, |M of the largest|, S2, |M of the second|."""
        dx, dy = self._draws(t)
        s = self.s
        ox = dx & ~(s ^ s.roll(-1, 1) ^ self.neg_x)
        oy = dy & ~(s ^ s.roll(-1, 2) ^ self.neg_y)
        root = self._clusters(ox, oy)
        self.s = s = s ^ self._bits(t, 1).gather(1, root).view_as(s)
        if not measure:
            return None
        unsat = (s ^ s.roll(-1, 1) ^ self.neg_x).sum((1, 2)) + (s ^ s.roll(-1, 2) ^ self.neg_y).sum((1, 2))
        spin = 1 - 2 * s.view(self.n, -1).long()
        size = torch.zeros_like(root).scatter_add_(1, root, torch.ones_like(root))
        # Among equal sizes the cluster with the smallest site comes first.
        top = (size * self.N + (self.N - 1 - torch.arange(self.N, device=_DEV))).topk(2, 1).values
        r1, r2 = (self.N - 1 - top % self.N).unbind(1)
        s1, s2 = (top // self.N).unbind(1)
        mc = [(spin * (root == r[:, None])).sum(1).abs() for r in (r1, r2)]
        return {"energy": 2 * unsat - 2 * self.N, "magnetization": spin.sum(1), "n_clusters": (size > 0).sum(1),
                "largest_size": s1, "largest_abs_mag": mc[0], "second_size": s2,
                "second_abs_mag": torch.where(s2 > 0, mc[1], 0)}


def _primitives(r):
    """The per-sweep primitives of a measured sweep in float64 (the wrapping ones left out)."""
    d = {k: v.double() for k, v in r.items()}
    m = d["magnetization"]
    return {"energy": d["energy"], "energy_sq": d["energy"] ** 2, "magnetization": m, "abs_magnetization": m.abs(),
            "magnetization_sq": m**2, "magnetization_4": m**4, "largest_size": d["largest_size"],
            "largest_abs_mag": d["largest_abs_mag"], "second_size": d["second_size"],
            "mag_ratio": d["largest_abs_mag"] / d["largest_size"], "n_clusters": d["n_clusters"]}


def _binned(replay, case):
    """{primitive: (chains, bins) means} of a run of thermalisation and binned measurement."""
    per = case["sweeps"] // case["bins"]
    for t in range(case["therm"]):
        replay.sweep(t, False)
    bins = []
    for b in range(case["bins"]):
        total = {}
        for k in range(per):
            for name, v in _primitives(replay.sweep(case["therm"] + b * per + k, True)).items():
                total[name] = total.get(name, 0) + v
        bins.append(total)
    return {name: (torch.stack([b[name] for b in bins], 1) / per).cpu().numpy() for name in bins[0]}


def _key(child):
    lo, hi = child.generate_state(2, dtype=np.uint32)
    return int(lo) | int(hi) << 32


def _observables(p, T, N):
    """Physical observables from primitive moments (arrays over temperatures and whatever follows)."""
    m2, m4 = p["magnetization_sq"] / N**2, p["magnetization_4"] / N**4
    return {"energy": p["energy"] / N, "specific_heat": (p["energy_sq"] - p["energy"] ** 2) / (T**2 * N),
            "magnetization": p["magnetization"] / N, "abs_magnetization": p["abs_magnetization"] / N,
            "susceptibility": (p["magnetization_sq"] - p["abs_magnetization"] ** 2) / (T * N),
            "binder": np.where(m2 > 0, 1 - m4 / (3 * np.where(m2 > 0, m2, 1) ** 2), 0.0),
            "p_infinity": p["largest_size"] / N, "largest_size": p["largest_size"],
            "largest_abs_magnetization": p["largest_abs_mag"], "cluster_magnetization_ratio": p["mag_ratio"],
            "second_size_fraction": p["second_size"] / N,
            "cluster_density_gap": (p["largest_size"] - p["second_size"]) / N,
            "n_clusters_per_site": p["n_clusters"] / N}


def _exact_scan(case, seed):
    """Disorder averages with the jackknife over realizations and the spread over bins."""
    L, n_t, n_r, nb = case["L"], case["n_t"], case["n_r"], case["bins"]
    temps = np.linspace(case["t_lo"], case["t_hi"], n_t)
    dseed, rseed = np.random.SeedSequence(seed).spawn(2)
    rng = np.random.default_rng(dseed)
    bonds = []
    for _ in range(n_r):
        jx, jy = (np.where(rng.random((L, L)) < case["p"], -1, 1) for _ in range(2))
        bonds.append(np.stack([jx, jy], -1).reshape(-1).astype(np.int8))
    keys = [_key(c) for c in rseed.spawn(n_t * n_r)]
    replay = _Replay(L, bonds, [k % n_r for k in range(n_t * n_r)], [1.0 / T for T in np.repeat(temps, n_r)], keys)
    replay.hot()
    bins = {k: v.reshape(n_t, n_r, nb) for k, v in _binned(replay, case).items()}
    mean = {k: v.mean(2) for k, v in bins.items()}
    value = _observables({k: v.mean(1) for k, v in mean.items()}, temps, L * L)
    left = _observables({k: (v.sum(1, keepdims=True) - v) / max(1, n_r - 1) for k, v in mean.items()},
                        temps[:, None], L * L)
    by_bin = _observables(bins, temps[:, None, None], L * L)
    out = {}
    for name in value:
        thermal = np.sqrt(np.mean(by_bin[name].std(2, ddof=1) ** 2 / nb, axis=1) / n_r)
        error = np.sqrt((n_r - 1) * left[name].var(1)) if n_r > 1 else thermal
        out[name] = {"value": value[name], "error": error, "thermal_error": thermal}
    return out | {name: None for name in ("wrap_x", "wrap_y", "wrap_any")}


def _exact_chains(case, seed):
    """The floating sums of a chain set: M^4 and |M of the largest cluster| / its size, per bin."""
    bonds, chains = _chains(case, seed)
    n_bins = _run_length(case)[1]
    moments = torch.zeros(len(chains) * n_bins, 2, dtype=torch.float64, device=_DEV)
    if case["measure"]:
        by_size = {}
        for i, c in enumerate(chains):
            by_size.setdefault(c[1], []).append(i)
        for L, members in by_size.items():
            some = max(1, (1 << 25) // L**2)
            for k in range(0, len(members), some):
                part = members[k: k + some]
                reals = sorted({chains[i][0] for i in part})
                replay = _Replay(L, [bonds[r] for r in reals], [reals.index(chains[i][0]) for i in part],
                                 [chains[i][2] for i in part], [chains[i][3] for i in part])
                replay.hot()
                at = torch.tensor(part, device=_DEV) * n_bins  # the first bin of each
                for t in range(THERM + case["sweeps"]):
                    r = replay.sweep(t, t >= THERM)
                    if r is not None:
                        d = _primitives(r)
                        moments[at] += torch.stack([d["magnetization_4"], d["mag_ratio"]], 1)
    return {"spins": None, "sums": None, "moments": moments}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "mix"):
        return _exact_chains(case, seed)
    if kind == "scan":
        return _exact_scan(case, seed)
    if kind == "label":
        return None  # whole numbers only
    if kind == "single":
        J = _bonds(case["L"], case["p"], np.random.default_rng([seed, 3]))
        replay = _Replay(case["L"], [J], [0], [1.0 / case["T"]], [_key(np.random.SeedSequence(seed))])
        replay.hot()
        bins = {k: v[0] for k, v in _binned(replay, case).items()}
        return {"means": {k: float(v.mean()) for k, v in bins.items()}, "bins": bins}
    rng = np.random.default_rng([seed, 4])
    L = case["L"]
    J, key = _bonds(L, case["p"], rng), int(rng.integers(0, 2**63))
    replay = _Replay(L, [J], [0], [1.0 / case["T"]], [key])
    replay.s = torch.from_numpy(rng.integers(0, 2, size=L * L, dtype=np.int64) == 0).to(_DEV).view(1, L, L)
    r = {k: float(v) for k, v in replay.sweep(0, True).items()}
    return {"spins": None, "energy": r["energy"], "magnetization": r["magnetization"], "n_clusters": None,
            "largest_size": None, "largest_abs_magnetization": r["largest_abs_mag"], "second_size": None,
            "second_abs_magnetization": r["second_abs_mag"], "wraps": [None, None]}
