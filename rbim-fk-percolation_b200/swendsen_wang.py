"""A single Swendsen-Wang update on the GPU (mirror of ``src/rbim/swendsen_wang.py``).

``sw_sweep`` runs one sweep of one lattice on the engine ``engine="auto"`` picks
for it and returns the reference's ``SweepResult``.  It is the per-sweep API; throughput
work goes through :class:`~.engine.ChainSet` and ``run_temperature_scan``,
which keep the state on the device across sweeps.
"""

from __future__ import annotations

import threading
from dataclasses import dataclass
from typing import Optional

import numpy as np

from .engine import ChainSet, ChainSpec, _torch, auto_engine, require_cuda, single_cta_threads
from .lattice import Lattice
from .packing import pack_couplings, pack_spins, threshold, unpack_spins, words_for

__all__ = [
    "SweepResult",
    "energy",
    "magnetization",
    "random_spins",
    "aligned_spins",
    "initial_spins",
    "sw_sweep",
]


@dataclass(frozen=True)
class SweepResult:
    """Observables of one sweep (reference ``swendsen_wang.py:24-53``).

    Every field is measured on the device in the sweep's record, including
    ``second_abs_magnetization`` (|M| of the second-largest cluster,
    reference ``swendsen_wang.py:151-154``).
    """

    energy: float
    magnetization: float
    n_clusters: int
    largest_size: int
    largest_abs_magnetization: float
    second_size: int
    second_abs_magnetization: float
    wraps_x: Optional[bool]
    wraps_y: Optional[bool]


def random_spins(n_sites: int, rng: np.random.Generator) -> np.ndarray:
    """Random ``+-1`` configuration (reference ``swendsen_wang.py:56-58``)."""
    return rng.integers(0, 2, size=n_sites, dtype=np.int64) * 2 - 1


def aligned_spins(n_sites: int) -> np.ndarray:
    """All spins up (reference ``swendsen_wang.py:61-63``)."""
    return np.ones(n_sites, dtype=np.int64)


def initial_spins(n_sites: int, rng: np.random.Generator, start: str = "hot") -> np.ndarray:
    """Hot or cold start (reference ``swendsen_wang.py:66-78``)."""
    if start == "hot":
        return random_spins(n_sites, rng)
    if start == "cold":
        return aligned_spins(n_sites)
    raise ValueError(f"start must be 'hot' or 'cold', got {start!r}")


def energy(spins: np.ndarray, lattice: Lattice, J: np.ndarray) -> float:
    """``-sum J s s`` over bonds (host helper, reference ``swendsen_wang.py:81-84``)."""
    ends = lattice.bonds
    return -float(np.sum(J * spins[ends[:, 0]] * spins[ends[:, 1]]))


def magnetization(spins: np.ndarray) -> float:
    """``sum s`` (host helper, reference ``swendsen_wang.py:87-89``)."""
    return float(np.sum(spins))


def sw_sweep(spins: np.ndarray, lattice: Lattice, J: np.ndarray, beta: float, rng=None, *, key: Optional[int] = None,
             sweep: int = 0, measure: bool = True, measure_percolation: bool = True,
             device=None) -> Optional[SweepResult]:
    """One Swendsen-Wang update of ``spins`` in place (reference ``swendsen_wang.py:103-172``).

    Randomness comes from the Philox stream of ``key`` at sweep counter
    ``sweep``; when ``key`` is omitted it is drawn from ``rng``.  The device
    buffers of L x L lattices are kept between calls (one chain set per device
    and L, used under a lock), so a loop over ``sw_sweep`` allocates device
    memory only on its first call; each call still copies the spins and
    couplings in and the spins and the record out, in one copy each way.
    """
    L = lattice.L
    if key is None:
        if rng is None:
            raise ValueError("sw_sweep needs a key or a numpy Generator")
        key = int(rng.integers(0, 2**63, dtype=np.int64))
    st = _sweep_state(L, device)
    with st.lock:
        # One chain whose only sweep is `sweep`: measured when n_therm == sweep.
        st.couplings[:] = pack_couplings(J, L)
        st.spins[:] = pack_spins(spins, L)
        d = st.desc
        d["key"], d["thr"], d["sweep"] = int(key) & (2**64 - 1), threshold(beta), sweep
        d["n_therm"] = sweep if measure else sweep + 1
        st.run()
        spins[...] = unpack_spins(st.spins, L, dtype=spins.dtype)
        if not measure:
            return None
        rec = st.record.copy()
    wx = bool(rec[7]) if measure_percolation else None
    wy = bool(rec[8]) if measure_percolation else None
    return SweepResult(energy=float(rec[0]), magnetization=float(rec[1]), n_clusters=int(rec[2]),
                       largest_size=int(rec[3]), largest_abs_magnetization=float(rec[4]), second_size=int(rec[5]),
                       second_abs_magnetization=float(rec[6]), wraps_x=wx, wraps_y=wy)


class _SweepState:
    """Device and host buffers of ``sw_sweep`` for L x L lattices on one device, used under ``lock``.

    The chain set's inputs (bin sums, couplings, descriptor, cleared status,
    spins) and its outputs (status, spins, record) lie in one device buffer,
    mirrored in one pinned host buffer, so that a call makes one copy in and
    one copy out.
    """

    def __init__(self, L: int, dev):
        torch = _torch()
        spec = ChainSpec(L=L, realization=0, key=0, beta=1.0, n_therm=0, n_bins=1, sweeps_per_bin=1, records=True)
        cs = ChainSet([spec], [np.zeros(2 * words_for(L), dtype="<u4")], device=dev)
        with torch.cuda.device(dev):
            self.engine = auto_engine([spec])
        self.lock = threading.Lock()
        self.chain_set, self.device, self.threads = cs, dev, single_cta_threads(L)
        at, end = {}, 0
        for name in ("acc_int", "acc_f64", "coupling_pool", "chains", "status", "spin_pool", "records"):
            t = getattr(cs, name)
            at[name] = (end, end + t.numel() * t.element_size())
            end = (at[name][1] + 15) & ~15
        device = torch.zeros(end, dtype=torch.uint8, device=dev)
        host = torch.zeros(end, dtype=torch.uint8, pin_memory=True)
        for name, (lo, hi) in at.items():
            t = getattr(cs, name)
            setattr(cs, name, device[lo:hi].view(t.dtype).view(t.shape))
        self._in = (device[: at["spin_pool"][1]], host[: at["spin_pool"][1]])
        self._out = (device[at["status"][0]:], host[at["status"][0]:])
        h = host.numpy()
        view = lambda name, dtype: h[slice(*at[name])].view(dtype)  # noqa: E731
        self.couplings, self.spins = view("coupling_pool", "<u4"), view("spin_pool", "<u4")
        self.record, self.status = view("records", np.int32), view("status", np.int32)
        self.desc = view("chains", cs.desc_host.dtype)
        self.desc[:] = cs.desc_host
        # The buffers are set up on this thread's stream; the next call may
        # come from another thread on another one.
        torch.cuda.current_stream(dev).synchronize()

    def run(self) -> None:
        """One sweep of the chain described by the host buffer; its spins, record and status come back there."""
        cs, stream = self.chain_set, _torch().cuda.current_stream(self.device)
        self.status[0] = 0  # the kernels only add bits: an earlier call's error is not this one's
        try:
            self._in[0].copy_(self._in[1], non_blocking=True)
            if self.engine == "grid":
                cs.run_grid(1)  # one cooperative launch over every SM
            elif self.engine == "batched":
                cs.run_batched(1, threads=self.threads)  # one resident CTA
            else:
                cs.run_plain(1)
            self._out[1].copy_(self._out[0], non_blocking=True)
        finally:
            stream.synchronize()  # the host buffer is free again, whatever happened
        if self.status[0]:
            cs.check_status()


_states_lock = threading.Lock()
_states = {}  # (device, L) -> _SweepState


def _sweep_state(L: int, device) -> _SweepState:
    """The state ``sw_sweep`` reuses for L x L lattices: one per (device, L), created on first use, so that a caller
    looping over ``sw_sweep`` does not allocate and free buffers every sweep."""
    dev = require_cuda(device)
    key = (str(dev), int(L))
    with _states_lock:
        state = _states.get(key)
        if state is None:
            state = _states[key] = _SweepState(L, dev)
        return state
