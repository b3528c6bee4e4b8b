"""solve(M, Q, B0, r, B) -> Carmichael hits: the exchange meet-in-the-middle join on one B200.

A candidate is S = (B0 \\ D) u I with D an r-subset of the base B0 and I an
r-subset of INS = Q \\ B0.  Because every prime q of the pool Q = Q(M) has
(q-1) | M, prod(S) == 1 (mod M) makes S Carmichael by Korselt
(src/mitm64.cpp:12-16).  The congruence is the residue join

    prod(I) == prod(D) * (prod B0)^-1   (mod M)

(the reference matches P0 * prod(I) == prod(D), gpu/mitm_gpu_mstar_driver.py:214-237;
both sides here carry the constant on the D side, so the large I side needs no
multiplier).  Device pipeline of the default ("fused") strategy, queued on one
stream by one native call (cf_solve):

  1. class join (csrc/cf_class.cu) where the probing side has 2^22 records or more:
     lists of prefixes and suffixes by residue class, one shared-memory filter per
     class, every probe record tested there, survivors matched exactly;
     else a table of the smaller side in L2 and a fused generate-and-probe of the
     other (csrc/cf_dtab.cuh, csrc/cf_fused.cu)
  2. k_check_pairs  : recompute residues, fp64 size screen, exact size, Korselt

The "partition" strategy materialises both sides (k_gen_part, k_join_part) instead;
the "bounded" one prunes them by the size bound (bsolve.py).

then one synchronisation, a copy of the (rare) checked pairs, and host
certification of every hit by ``certify.verify_certificate``.
"""
from __future__ import annotations

import ctypes as C
import math
import struct
from dataclasses import dataclass, field

import numpy as np

from . import _lib
from .certify import verify_certificate
from .tables import DeviceTables, ncomb, split_modulus, unrank_lex, wide_modulus

RESULT_DTYPE = np.dtype([("flags", "<u4"), ("r", "<u4"), ("d_idx", "<u2", (16,)), ("i_idx", "<u2", (16,))])

# One modulus of the batched kernels (CfBatchMod, cf_batch_mod_bytes() bytes); the
# single-modulus solve uses a one-row array of it for the partitioned table build.
MOD_DTYPE = np.dtype([
    ("poolD", "<u8"), ("tailD", "<u8"), ("poolI", "<u8"), ("tailI", "<u8"), ("screen", "<u8"),
    ("fpw", "<u8"), ("side", "<u8"), ("fill", "<u8"), ("bloom", "<u8"),
    ("nD", "<u8"), ("i_lo", "<u8"), ("nI", "<u8"),
    ("bbits", "<i4"), ("fbits", "<i4"), ("r", "<i4"), ("swap", "<i4"),
    ("pkw", "<u8"), ("psd", "<u8"), ("pcnt", "<u8"), ("pcap", "<u4"), ("plb", "<u4")])


def part_shape(n_build: int, bbits: int, lb: int, sigma: float, max_ranges: int) -> tuple[int, int] | None:
    """(bucket ranges, records per range) of the partitioned table build of n_build
    records into 2^bbits buckets, or None when the table has too many ranges."""
    nparts = 1 << max(0, bbits - lb)
    if nparts > max_ranges:
        return None
    mean = n_build / nparts
    cap = int(math.ceil(mean + sigma * math.sqrt(mean) + 32))
    return nparts, (cap + 3) // 4 * 4
ALL_FLAGS = (_lib.HIT_KEY_EQUAL | _lib.HIT_SCREEN | _lib.HIT_SIZE_EXACT | _lib.HIT_KORSELT | _lib.HIT_DISJOINT)


@dataclass(frozen=True)
class Hit:
    """One Carmichael number found by the join."""
    D: tuple[int, ...]        # deleted base primes (ascending)
    I: tuple[int, ...]        # inserted primes (ascending)
    n: int                    # prod(S)
    factors: tuple[int, ...]  # S, ascending


@dataclass
class SolveResult:
    hits: list[Hit]
    n_D: int                  # D-side records (C(|B0|, r))
    n_I: int                  # I-side records (C(|INS|, r))
    residue_pairs: int        # equal-residue (D, I) pairs (join_sorted's pair count)
    screened: int             # pairs surviving the fp64 log-size screen
    above_bound: int          # equal-residue pairs with prod(S) > B
    rejected: int             # pairs failing the device or host checks (0 unless a bug)
    device_ms: float | None = None
    plan: dict = field(default_factory=dict)
    pairs: list = field(default_factory=list)   # every equal-residue (D primes, I primes) pair
    launches: int = 0                           # kernels of this library launched by the solve

    @property
    def records(self) -> int:
        return self.n_D + self.n_I


@dataclass
class Tuning:
    """Launch shape of the partitioned join (chosen by autotune.py when tuned)."""
    d_per_part: int = 7000          # target D records per partition
    max_pbits: int = 12             # at most 2^12 partitions
    gen_shape: int = 1              # cf_gen_part launch shape (threads x records per thread)
    max_sbits: int = 14             # shared table of 2^sbits slots (4 B) per CTA
    isplit: int = 0                 # CTAs per partition in the join (0 = automatic)
    i_chunk_records: int = 1 << 31  # I-side records per generation/join chunk
    pair_capacity: int = 1 << 14    # initial candidate-pair buffer (grown on overflow)
    sigma: float = 6.0              # partition capacity = mean + sigma*sqrt(mean) + 16
    strategy: str = "fused"         # "fused": table + generate-and-probe; "partition": materialised join;
                                    # "bounded": size-bound-pruned sides + record join; "auto": bounded
                                    # where the bound prunes, else fused
    dtab_load: float = 5.0          # fused: minimum average D records per 16-slot bucket (up to 2x this)
    fused_grid: int = 0             # fused probe CTAs (0 = one per 16384 records)
    l2_table_bytes: int = 72 << 20  # fingerprint arrays above this get a Bloom-filter first level
    max_fbits: int = 21             # Bloom filter at most 2^21 blocks of 32 bytes (64 MB)
    max_nodes: int = 1 << 27        # bounded strategy: frontier nodes per block of first indices
    part_build: bool = True         # fused: partitioned table build for tables of part_min_buckets or more
    part_min_buckets: int = 1 << 21 # smaller tables stay in L2 while built alone: built in place
    part_lb: int = 10               # log2 buckets per range of the partitioned build (9 or 10)
    part_sigma: float = 8.0         # bucket-range capacity = mean + sigma*sqrt(mean) + 32
    class_join: bool = True         # fused: join by residue classes (csrc/cf_class.cu) where it applies
    class_ws_bytes: int = 36 << 30  # ... and its workspace is at most this, a fifth of the device (half of it for each
                                    # of a list's two)
    class_min_probe: int = 1 << 22  # ... and the probing side has this many records or more (see class_least)


def class_least(r: int, n_build: int, tu: Tuning) -> int:
    """Least probing side of a class join at radius r, n_build records on the other side.  Its lists and plan cost
    0.13 ms whatever the sides; a table probe costs more per record at larger radii.  Whole solves, class join
    against table join, ms: r = 3, 6.5e6 records .227 / .203, 1.2e7 .228 / .236, 2.9e7 .266 / .337; r = 4, 4.2e6 .212 / .198, 8.2e6
    .220 / .213, 1.5e7 .243 / .278; r = 5, 4.2e6 .190 / .189 (nD = 1.4e5) and .247 / .289 (7.6e6), 2.4e7
    .290 / .451; r = 6, 4.5e6 .197 / .219; r = 7, 5.4e6 .189 / .288; r = 8, 5.9e6 .226 / .364.  A table of few
    records is probed at the same few sectors: r = 3, 4.5e6 against 1,140 records .194 / .245, against 10,000
    .222 / .210; r = 4, 4.6e6 against 495 .183 / .266, against 27,405 .198 / .171."""
    return tu.class_min_probe * (3 if r < 5 and n_build >= 4096 else 1)


def dtab_shape(nD: int, tu: Tuning) -> tuple[int, int]:
    """(bbits, fbits) of the D table for nD records: 2^bbits buckets of 16 slots at an
    average load between dtab_load and 2*dtab_load (never above 12), and a Bloom-filter
    first level (about 8 bits per D record, at most 2^max_fbits blocks of 32 bytes) when
    the fingerprint array would not stay in L2 -- and none when that cap leaves fewer than
    6 bits per record."""
    bbits = max(4, int(math.floor(math.log2(max(nD / tu.dtab_load, 2.0)))),
                math.ceil(math.log2(max(nD / 12.0, 2.0))))
    fbits = 0
    if (1 << bbits) * 32 > tu.l2_table_bytes:
        fbits = min(tu.max_fbits, max(4, math.ceil(math.log2(max(nD / 32.0, 2.0)))))
        if (256 << fbits) < 6 * nD:      # under 6 filter bits per record the filter passes nearly everything
            fbits = 0
    return bbits, fbits


def _i_window(inst: "Instance", plan: dict) -> int:
    """Number of I ranks joined: the window [plan["i_lo"], plan["i_limit"]) of [0, C(|INS|, r)), where
    i_lo defaults to 0 and i_limit to C(|INS|, r)."""
    nI = ncomb(len(inst.INS), inst.r)
    lim = plan.get("i_limit")
    hi = nI if lim is None else min(nI, int(lim))
    return max(0, hi - _i_lo(plan))


def _i_lo(plan: dict) -> int:
    """First I rank of the window joined."""
    return int(plan.get("i_lo") or 0)


_PLAN_HEAD = struct.Struct("<8x4IQ")


def plan_head(cp) -> tuple[int, int, int, int, int]:
    """(ok, class modulus, filter modulus, classes, workspace bytes) of a class plan."""
    return _PLAN_HEAD.unpack_from(cp)


def _ws_bytes(cp: bytes) -> int:
    """Workspace bytes of a class plan."""
    return _PLAN_HEAD.unpack_from(cp)[4]


def make_class_plan(lib, M: int, nB: int, nINS: int, r: int, i_lo: int, n_I: int, swap: bool) -> tuple[bytes | None, int]:
    """cf_class_plan: (plan, workspace bytes), or (None, 0) where the class join does not apply."""
    cp = C.create_string_buffer(lib.cf_class_plan_bytes())
    _lib.check(lib.cf_class_plan(split_modulus(M)[0], nB, nINS, r, i_lo, n_I, int(swap), C.addressof(cp), len(cp)),
               "cf_class_plan")
    ok, _d, _mp, _phi, ws = plan_head(cp)
    return (cp.raw, ws) if ok else (None, 0)


def _pow2ceil(x: int) -> int:
    return 1 if x <= 1 else 1 << (x - 1).bit_length()


def class_pairs(nD: int, nI: int, M: int, tu: "Tuning") -> int:
    """Pair capacity of a class join: room for the pairs a modulus with few units has (8 nD nI / M)."""
    return max(tu.pair_capacity, min(1 << 22, _pow2ceil(8 * nD * nI // M)))


def _cap(mean: float, sigma: float) -> int:
    return int(math.ceil(mean + sigma * math.sqrt(max(mean, 1.0)) + 16))


@dataclass
class Instance:
    M: int
    B0: list[int]
    INS: list[int]
    r: int
    B: int
    P0: int

    @staticmethod
    def build(M: int, Q, B0, r: int, B: int) -> "Instance":
        M, r, B = int(M), int(r), int(B)
        if M < 2 or (M >> ((M & -M).bit_length() - 1)) >= 1 << 63:
            raise ValueError("M must be at least 2 with an odd part below 2^63")
        base = sorted(int(p) for p in B0)
        if len(set(base)) != len(base):
            raise ValueError("B0 has repeated primes")
        bset = set(base)
        ins = sorted(set(int(q) for q in Q) - bset)
        if not (0 <= r <= 10):
            raise ValueError("radius r must be 0..10")
        if len(base) > 1024 or len(ins) > 1024:
            raise ValueError("B0 and Q \\ B0 are limited to 1024 primes each")
        if B < 1:
            raise ValueError("size bound B must be >= 1")
        P0 = math.prod(base)
        if math.gcd(P0 * math.prod(ins), M) != 1:
            raise ValueError("every pool prime must be coprime to M (q does not divide M)")
        if (base and base[-1] >= 1 << 31) or (ins and ins[-1] >= 1 << 31):
            raise ValueError("pool primes must be below 2^31")
        if M % (1 << 33) == 0:
            raise ValueError("2^33 divides M: the solve path needs the 2-adic part of M below 2^33")
        return Instance(M, base, ins, r, B, P0)


def finish_rows(inst: Instance, res: np.ndarray, nD: int, nI: int, plan: dict, verify: bool) -> SolveResult:
    """SolveResult of one modulus from its checked candidate rows (RESULT_DTYPE).

    Rows without CF_HIT_KEY_EQUAL are fingerprint collisions of the fused join and
    are dropped; for the partition join, which compares full keys, they count as
    rejected.  Every hit is re-derived and, with verify, certified on the host."""
    r = inst.r
    hits, screened, above, rejected, pairs = [], 0, 0, 0, []
    bset = inst.B0
    fused = plan.get("strategy") == "fused"
    wide = wide_modulus(inst.M)                # keys taken mod 2^64: confirm every match exactly
    nres = 0
    for row in res:
        f = int(row["flags"])
        if not f & _lib.HIT_KEY_EQUAL:
            if not fused:
                rejected += 1
            continue
        di = [int(x) for x in row["d_idx"][:r]]
        ii = [int(x) for x in row["i_idx"][:r]]
        D = tuple(bset[i] for i in di)
        I = tuple(inst.INS[i] for i in ii)
        if wide and (inst.P0 * math.prod(I) - math.prod(D)) % inst.M:
            if not fused:                     # keys mod 2^64 matched, residues differ
                rejected += 1
            continue
        nres += 1
        pairs.append((D, I))
        if not f & _lib.HIT_SCREEN:
            above += 1
            continue
        screened += 1
        if not f & _lib.HIT_SIZE_EXACT:
            above += 1
            continue
        if (f & ALL_FLAGS) != ALL_FLAGS:
            rejected += 1
            continue
        dset = set(D)
        fac = tuple(sorted([p for p in bset if p not in dset] + list(I)))
        n = 1
        for p in fac:
            n *= p
        ok = n <= inst.B and (n - 1) % inst.M == 0
        if verify and ok:
            ok, n2, _why = verify_certificate(fac)
            ok = ok and n2 == n
        if not ok:
            rejected += 1
            continue
        hits.append(Hit(D, I, n, fac))
    hits.sort(key=lambda x: (x.n, x.D, x.I))
    pairs.sort()
    return SolveResult(hits=hits, n_D=nD, n_I=nI, residue_pairs=nres, screened=screened,
                       above_bound=above, rejected=rejected, plan=dict(plan), pairs=pairs)


class Solver:
    """Reusable device state for repeated solves on one device and stream."""

    READBACK_ROWS = 256

    def __init__(self, device=None, stream=None, tuning: Tuning | None = None):
        import torch
        self.torch = torch
        self.lib = _lib.load()
        self.device = torch.device(device if device is not None else "cuda")
        if self.device.type != "cuda":
            raise RuntimeError("the join runs on a CUDA device only")
        self.stream = stream
        self.tuning = tuning or Tuning()
        self.tables = DeviceTables(self.device, stream=stream, async_upload=True)
        self._bufs: dict[str, object] = {}
        self._rows = self.READBACK_ROWS  # checked rows that come back with a solve's counters
        self._pool = None                # solve_many: the caller's stream, from whose memory _buf allocates, so
                                         # that the next solver finds it again (its own streams are new ones)
        self._bufset = 0                 # which of two buffer sets the next enqueue uses (solve_many)
        self.d2h_bytes = 0               # bytes read back from the device by collect()
        self._pinned: dict = {}
        self._on: dict = {}              # buffer set -> raw stream of its last solve
        self._queued: dict = {}          # buffer set -> handle of the solve queued on it and not collected
        self._reserved: dict = {}        # buffer set -> bytes by name that lists have reserved
        self._class_cover = 0.0          # survivor estimate that the lists' class workspaces were reserved for
        self._bounded = None
        self.result_bytes = self.lib.cf_pair_result_bytes()
        assert self.result_bytes == RESULT_DTYPE.itemsize

    # -- buffers -----------------------------------------------------------
    def _buf(self, name: str, nbytes: int):
        key = (name, self._bufset)
        t = self._bufs.get(key)
        if t is None or t.numel() < nbytes:
            if t is not None:                  # a growing buffer grows by half (64 MB at most) at least, the old one
                nbytes = max(nbytes, min(t.numel() * 3 // 2, t.numel() + (64 << 20)))       # freed before it
                del self._bufs[key], t
            st = self._torch_stream()
            pool = self._pool or st
            with self.torch.cuda.stream(pool):
                t = self.torch.empty(max(nbytes, 16), dtype=self.torch.uint8, device=self.device)
            if st != pool:
                st.wait_stream(pool)               # what used the memory before, on the caller's stream
                t.record_stream(st)
            self._bufs[key] = t
        return t

    def _pinned_buf(self, name: str, nbytes: int, dev=None, sh: int = 0):
        """Page-locked host buffer of the current buffer set (rewritten only after the solve that
        last used it has been collected, see _leave_staging).
        dev: the device buffer that a native call on stream sh copies to or from it.  Torch, which hands freed
        page-locked memory out again, does not see such a copy, so one byte goes up through torch once per
        buffer and stream: the memory, once freed, then waits for that stream."""
        key = (name, self._bufset)
        t, streams = self._pinned.get(key) or (None, None)
        if t is None or t.numel() < nbytes:
            t, streams = self.torch.empty(max(nbytes, 64), dtype=self.torch.uint8, pin_memory=True), set()
            self._pinned[key] = t, streams
        if dev is not None and sh not in streams:
            with self.torch.cuda.stream(self._torch_stream()):
                dev[:1].copy_(t[:1], non_blocking=True)
            streams.add(sh)
        return t

    def _leave_staging(self):
        """Before a solve's tables are staged: page-locked buffers that a solve queued on this set and not
        collected may still read or write are left to it (freed, they wait for its stream)."""
        if self._queued.pop(self._bufset, None) is not None:
            for name in ("stage", "readback", "pdesc"):
                self._pinned.pop((name, self._bufset), None)

    def _sh(self):
        return _lib.stream_handle(self.stream)

    # -- planning ------------------------------------------------------------
    def plan(self, nD: int, nI: int, capD: int | None = None, capI: int | None = None,
             pairs: int | None = None) -> dict:
        tu = self.tuning
        pbits = min(tu.max_pbits, (_pow2ceil(-(-nD // tu.d_per_part))).bit_length() - 1)
        nparts = 1 << pbits
        chunk = min(nI, tu.i_chunk_records)
        cD = capD or _cap(nD / nparts, tu.sigma)
        cI = capI or _cap(chunk / nparts, tu.sigma)
        cD = min(cD, nD)
        cI = min(cI, chunk) if chunk else 1
        sbits = 4
        while sbits < tu.max_sbits and (1 << (sbits - 1)) < cD:
            sbits += 1
        isplit = tu.isplit or max(1, min(16, (2 * 148 * 2) // max(1, nparts)))
        bbits, fbits = dtab_shape(min(nD, nI), tu)     # the table holds the smaller side
        return dict(pbits=pbits, nparts=nparts, capD=max(cD, 1), capI=max(cI, 1), chunk=max(chunk, 1), sbits=sbits,
                    isplit=isplit, pairs=pairs or tu.pair_capacity, shape=tu.gen_shape, strategy=tu.strategy,
                    bbits=bbits, fbits=fbits, swap=nI < nD)

    # -- one solve -----------------------------------------------------------
    def _mark(self, marks, tag):
        if marks is not None:
            ev = self.torch.cuda.Event(enable_timing=True)
            ev.record(self._torch_stream())
            marks.append((tag, ev))

    def enqueue(self, inst: Instance, plan: dict, marks: list | None = None):
        """Queue the whole device pipeline for `inst` on the stream (no host sync).
        `marks` (optional list) receives (tag, CUDA event) pairs around every kernel."""
        if plan.get("strategy", "fused") == "fused":
            self._leave_staging()
            self._queued[self._bufset] = True      # also when a launch below fails
            sh = self._sh()
            if self._on.get(self._bufset) != sh:   # buffers made for another stream: kept until this one has passed too
                self._on[self._bufset] = sh
                for (_name, k), t in self._bufs.items():
                    if k == self._bufset:
                        t.record_stream(self._torch_stream())
            pshape = self._part_shape(inst, plan)
            h = self._enqueue_solve(inst, plan, marks, sh) if pshape is None \
                else self._enqueue_fused(inst, plan, pshape, marks)
            h["set"] = self._bufset
            self._queued[self._bufset] = h
            return h
        return self._enqueue_partition(inst, plan, marks)

    def _side_tables(self, inst: Instance, side: str):
        """(pool, tail) device tables of one side: D with multiplier (prod B0)^-1, I with 1."""
        M, r = inst.M, inst.r
        primes, mult = (inst.B0, pow(inst.P0, -1, M)) if side == "D" else (inst.INS, 1)
        pool = self.tables.pool(primes, r, M, mult)
        return pool, self.tables.tail(primes, r, M, mult, pool)

    def _tables_for(self, inst: Instance):
        poolD, tailD = self._side_tables(inst, "D")
        poolI, tailI = self._side_tables(inst, "I")
        screen = self.tables.screen(inst.P0, inst.B, 1e-6)
        return poolD, poolI, tailD, tailI, screen

    def _part_shape(self, inst: Instance, plan: dict) -> tuple | None:
        """(bucket ranges, range capacity) of a table join with the partitioned build, else None."""
        tu, lib = self.tuning, self.lib
        nb = 1 << plan["bbits"]
        if plan.get("class_plan") or not tu.part_build or plan.get("no_part") or nb < tu.part_min_buckets \
                or inst.r > lib.cf_batch_max_r():
            return None
        nD, nIt = ncomb(len(inst.B0), inst.r), _i_window(inst, plan)
        return part_shape(nIt if plan.get("swap") and nIt < nD else nD, plan["bbits"], tu.part_lb, tu.part_sigma,
                          lib.cf_batch_part_max_ranges())

    def _enqueue_solve(self, inst: Instance, plan: dict, marks: list | None, sh: int):
        """Class join, or table build in place and generate-and-probe, with tables, check and
        read-back: one cf_solve call.  Table by table from Python, k = 29, r = 2 took 235 us a
        solve against 184, and 24 portfolio moduli (11.0 ms against 8.3)"""
        lib, dp = self.lib, _lib.ptr
        r, M = inst.r, inst.M
        if inst.B < 1 or inst.B.bit_length() > 2048:
            raise ValueError("size bound B must be below 2^2048")
        nD, nIt = ncomb(len(inst.B0), r), _i_window(inst, plan)
        m, a = split_modulus(M)
        multD = pow(inst.P0, -1, M)
        cp = plan.get("class_plan")
        pD, pI = np.array(inst.B0, dtype=np.uint64), np.array(inst.INS, dtype=np.uint64)
        lb = np.frombuffer(inst.B.to_bytes((inst.B.bit_length() + 31) // 32 * 4, "little"), dtype=np.uint32)
        q = _lib.CfSolve(primesD=pD.ctypes.data, primesI=pI.ctypes.data, m=m, multD_odd=multD % m,
                         multD_2=multD & ((1 << a) - 1), n_D=nD, i_lo=_i_lo(plan), n_I=nIt, limbsB=lb.ctypes.data,
                         nlimbs=len(lb), lgP0=math.log2(inst.P0), lgB=math.log2(inst.B), eps=1e-6, nD=len(pD),
                         nI=len(pI), r=r, a=a, swap=int(bool(plan.get("swap")) and nIt < nD), bbits=plan["bbits"],
                         fbits=plan.get("fbits", 0), fused_grid=self.tuning.fused_grid)
        # in-place builds of tables of at most 2^20 buckets use compact side words (half the side area,
        # L2-resident while built); larger tables the wide entries
        q.side_format = 1 if q.bbits <= 20 else 0
        tb = lib.cf_solve_table_bytes(len(pD), len(pI), r)
        tabs = self._buf("tables", tb)
        stage = self._pinned_buf("stage", tb, tabs, sh)
        if cp:
            _ok, d, mp, _phi, q.ws_bytes = plan_head(cp)
            q.class_plan = C.cast(C.c_char_p(cp), C.c_void_p)
            q.multD_mp, q.multD_d = multD % mp, multD % d
            try:
                ws = self._buf("class", q.ws_bytes)
            except self.torch.OutOfMemoryError:    # a shared device: the table join needs less
                return self.enqueue(inst, self._replan(inst, dict(plan, no_class=True)), marks)
        else:
            q.ws_bytes = lib.cf_dtab_bytes2(q.bbits, q.fbits)
            ws = self._buf("dtab", q.ws_bytes)
            q.tails_bytes = lib.cf_solve_tail_bytes(len(pD), len(pI), r)
            q.tails = dp(self._buf("tails", q.tails_bytes))
        maxp = plan["pairs"]
        rb = self.result_bytes
        rows = max(0, min(self._rows, maxp))
        pairs, res, ctr = self._buf("pairs", maxp * 16), self._buf("res", maxp * rb), self._buf("ctr", 64)
        hm = self._pinned_buf("readback", 8 + rows * rb, ctr, sh)
        q.stage, q.tables, q.ws, q.pairs, q.results, q.misc = \
            stage.data_ptr(), dp(tabs), dp(ws), dp(pairs), dp(res), dp(ctr)
        q.max_pairs, q.rows, q.readback = maxp, rows, hm.data_ptr()
        if marks is not None:
            for j, tag in enumerate(("start", "gen_D", "probe", "check")):
                self._mark(marks, tag)             # makes the event; cf_solve records it again in its place
                q.events[j] = marks[-1][1].cuda_event
        _lib.check(lib.cf_solve(C.byref(q), sh), "cf_solve")
        ev = self.torch.cuda.Event()
        ev.record(self._torch_stream())
        return dict(misc=ctr[:64].view(self.torch.int32), dcnt=None, icnt=None, res=res, nD=nD, nI=nIt, plan=plan,
                    launches=9 if cp else 5, ev=ev, hread=hm, hrows=rows)

    def _enqueue_fused(self, inst: Instance, plan: dict, pshape: tuple, marks: list | None):
        """Table join with the partitioned build: D table, fused generate-and-probe, pair check."""
        torch, lib = self.torch, self.lib
        r = inst.r
        nD, nIt = ncomb(len(inst.B0), r), _i_window(inst, plan)
        bbits, fbits = plan["bbits"], plan.get("fbits", 0)
        tbytes = lib.cf_dtab_bytes2(bbits, fbits)
        tab = self._buf("dtab", tbytes)
        ctr = self._buf("ctr", 64)
        misc = ctr[:64].view(torch.int32)
        maxp = plan["pairs"]
        pairs = self._buf("pairs", maxp * 16)
        res = self._buf("res", maxp * self.result_bytes)
        sh = self._sh()
        dp = _lib.ptr
        ck = _lib.check
        misc.zero_()
        nb = 1 << bbits
        tab[: 32 * nb].zero_()                     # fingerprint sectors
        tab[160 * nb: tbytes].zero_()              # fill counters and Bloom filter
        # build on the smaller side (swap: the table holds the I window and the D side probes)
        swap = bool(plan.get("swap")) and nIt < nD
        pside = "D" if swap else "I"
        pn, pcount = (len(inst.B0), nD) if swap else (len(inst.INS), nIt)
        self._mark(marks, "start")
        ilo = _i_lo(plan)                          # first I rank of the window
        tables = self._tables_for(inst)
        self._part_build(inst, plan, pshape, tables, tab, nD, nIt, swap, misc)
        poolD, poolI, tailD, tailI, screen = tables
        ppool, ptail = (poolD, tailD) if pside == "D" else (poolI, tailI)
        ppool, ptail = dp(ppool), dp(ptail)
        self._mark(marks, "gen_D")
        ck(lib.cf_fused_probe3(ppool, ptail, pn, r, 0 if swap else ilo, pcount, dp(tab), bbits, fbits, 0,
                               ilo if swap else 0, int(swap), dp(pairs), maxp, dp(misc), dp(misc) + 4,
                               self.tuning.fused_grid, sh), "cf_fused_probe")
        self._mark(marks, "probe")
        ck(lib.cf_check_pairs(dp(poolD), dp(poolI), dp(screen), r, dp(pairs), dp(misc), maxp, dp(res),
                              dp(misc) + 4, sh), "cf_check_pairs")
        self._mark(marks, "check")
        return dict(misc=misc, dcnt=None, icnt=None, res=res, nD=nD, nI=nIt, plan=plan, launches=3)

    def _class_plan(self, inst: Instance, plan: dict) -> bytes | None:
        """The class join's plan for a fused solve (see cf_class_plan), or None where the table join
        is taken: a small probing side (class_least, or plan["class_least"]), a modulus without fitting
        divisors, a workspace above the limit, a run after an overflow."""
        tu, lib = self.tuning, self.lib
        nD, nI = ncomb(len(inst.B0), inst.r), _i_window(inst, plan)
        least = plan.get("class_least", class_least(inst.r, min(nD, nI), tu))
        if not tu.class_join or plan.get("no_class") or max(nD, nI) < least or not tu.l2_table_bytes:
            return None                       # (no L2 for tables: the caller wants the table join's filter level)
        if (inst.B0[-1] | inst.INS[-1]) >> 31:
            return None                       # the class join's kernels multiply 32-bit factors
        cp, ws = make_class_plan(lib, inst.M, len(inst.B0), len(inst.INS), inst.r, _i_lo(plan), nI,
                                 bool(plan.get("swap")))
        # k = 64: r = 5 54 to 210 MB, r = 6 0.8 to 13 GB, r = 7 1.3 to 40 GB (the table join 0.2, 1.3 and 10)
        sets = plan.get("sets") or (1 if self._pool is None else 2)
        return cp if ws * sets <= tu.class_ws_bytes else None

    def _part_build(self, inst: Instance, plan: dict, pshape: tuple, tables: tuple, tab, nD: int, nIt: int,
                    swap: bool, misc):
        """Partitioned table build (scatter by bucket range, shared-memory range build,
        overflow fix-up) through a one-modulus descriptor of the batched kernels."""
        torch, lib = self.torch, self.lib
        dp, ck, sh = _lib.ptr, _lib.check, self._sh()
        poolD, poolI, tailD, tailI, screen = tables
        bbits, fbits = plan["bbits"], plan.get("fbits", 0)
        nb = 1 << bbits
        nparts, cap = pshape
        n_build = nIt if swap else nD
        tile = lib.cf_batch_part_tile()
        # scratch: range counters, then the records of every range (4 + 8 bytes each)
        ocap = 1 << 12
        obytes = ocap * lib.cf_batch_ovf_bytes()
        up = lambda x: (x + 255) // 256 * 256
        scr = self._buf("pscratch", up(nparts * 4) + up(64) + up(obytes) + up(nparts * cap * 4) + nparts * cap * 8)
        base = dp(scr)
        pcnt, pmisc = base, base + up(nparts * 4)
        ovf = pmisc + up(64)
        pkw = ovf + up(obytes)
        psd = pkw + up(nparts * cap * 4)
        row = np.zeros(1, dtype=MOD_DTYPE)
        row["poolD"], row["tailD"], row["poolI"], row["tailI"] = dp(poolD), dp(tailD), dp(poolI), dp(tailI)
        row["screen"] = dp(screen)
        t0 = dp(tab)
        row["fpw"], row["side"], row["fill"] = t0, t0 + 32 * nb, t0 + 160 * nb
        row["bloom"] = t0 + 164 * nb if fbits else 0
        row["nD"], row["i_lo"], row["nI"] = nD, _i_lo(plan), nIt
        row["bbits"], row["fbits"], row["r"], row["swap"] = bbits, fbits, inst.r, int(swap)
        row["pkw"], row["psd"], row["pcnt"], row["pcap"], row["plb"] = pkw, psd, pcnt, cap, self.tuning.part_lb
        host = np.zeros(MOD_DTYPE.itemsize // 8 + 4, dtype=np.uint64)
        host[: MOD_DTYPE.itemsize // 8] = row.view(np.uint64)
        k = MOD_DTYPE.itemsize // 8
        host[k:k + 4] = (0, -(-n_build // tile), 0, nparts)        # scatter and range ticket prefix sums
        # pinned staging of this buffer set, rewritten only after its previous solve has been collected
        stage = self._pinned_buf("pdesc", host.nbytes)
        stage[: host.nbytes].numpy()[:] = host.view(np.uint8)
        hdev = self._buf("pdesc", host.nbytes)
        with torch.cuda.stream(self._torch_stream()):
            hdev[: host.nbytes].copy_(stage[: host.nbytes], non_blocking=True)
        self.h2d_desc_bytes = getattr(self, "h2d_desc_bytes", 0) + host.nbytes
        mods, tsS, tsP = dp(hdev), dp(hdev) + 8 * k, dp(hdev) + 8 * k + 16
        scr[: up(nparts * 4) + 64].zero_()
        err = dp(misc) + 4
        lb = self.tuning.part_lb
        ck(lib.cf_batch_part(0, mods, tsS, 1, pmisc, None, 0, pmisc + 24, err, lb, inst.r, 0, sh),
           "cf_batch_part(scatter)")
        ck(lib.cf_batch_part(1, mods, tsP, 1, pmisc + 8, ovf, ocap, pmisc + 24, err, lb, 0, 0, sh),
           "cf_batch_part(place)")
        ck(lib.cf_batch_part(2, mods, None, 1, None, ovf, ocap, pmisc + 24, err, lb, 0, 0, sh), "cf_batch_part(fix)")

    def _enqueue_partition(self, inst: Instance, plan: dict, marks: list | None):
        """Partitioned generation of both sides and the shared-memory partition join."""
        torch, lib = self.torch, self.lib
        r, M = inst.r, inst.M
        nD, nIt = ncomb(len(inst.B0), r), _i_window(inst, plan)
        P = plan["nparts"]
        pbits, shape = plan["pbits"], plan["shape"]
        multD = pow(inst.P0, -1, M)
        poolD = self.tables.pool(inst.B0, r, M, multD)
        poolI = self.tables.pool(inst.INS, r, M, 1)
        tailD = self.tables.tail(inst.B0, r, M, multD, poolD)
        tailI = self.tables.tail(inst.INS, r, M, 1, poolI)
        screen = self.tables.screen(inst.P0, inst.B, 1e-6)
        capD, capI, chunk = plan["capD"], plan["capI"], plan["chunk"]
        Dbuf = self._buf("D", P * capD * 16)
        Ibuf = self._buf("I", P * capI * 16)
        ctr = self._buf("ctr", (2 * P + 8) * 4)
        ctr_u32 = ctr[: (2 * P + 8) * 4].view(torch.int32)
        dcnt = ctr_u32[:P]
        icnt = ctr_u32[P:2 * P]
        misc = ctr_u32[2 * P:]          # [0] npairs, [1] err
        maxp = plan["pairs"]
        pairs = self._buf("pairs", maxp * 16)
        res = self._buf("res", maxp * self.result_bytes)
        sh = self._sh()
        dp = _lib.ptr
        ctr_u32.zero_()
        ck = _lib.check
        launches = 0
        self._mark(marks, "start")
        ck(lib.cf_gen_part(dp(poolD), dp(tailD), len(inst.B0), r, 0, nD, pbits, capD, dp(dcnt), dp(Dbuf),
                           dp(misc) + 4, shape, sh), "cf_gen_part(D)")
        launches += 1
        self._mark(marks, "gen_D")
        ilo = _i_lo(plan)
        for off in range(0, nIt, chunk):
            cnt = min(chunk, nIt - off)
            lo = ilo + off
            if off:
                icnt.zero_()
            ck(lib.cf_gen_part(dp(poolI), dp(tailI), len(inst.INS), r, lo, cnt, pbits, capI, dp(icnt), dp(Ibuf),
                               dp(misc) + 4, shape, sh), "cf_gen_part(I)")
            self._mark(marks, "gen_I")
            ck(lib.cf_join_part(dp(Dbuf), dp(dcnt), capD, dp(Ibuf), dp(icnt), capI, pbits, plan["sbits"],
                                plan["isplit"], 0, dp(pairs), maxp, dp(misc), dp(misc) + 4, sh),
               "cf_join_part")
            self._mark(marks, "join")
            launches += 2
        ck(lib.cf_check_pairs(dp(poolD), dp(poolI), dp(screen), r, dp(pairs), dp(misc), maxp, dp(res),
                              dp(misc) + 4, sh), "cf_check_pairs")
        launches += 1
        self._mark(marks, "check")
        return dict(misc=misc, dcnt=dcnt, icnt=icnt, res=res, nD=nD, nI=nIt, plan=plan, launches=launches)

    def collect(self, inst: Instance, h: dict, verify: bool = True) -> tuple[SolveResult | None, dict | None]:
        """Synchronise, read counters; returns (result, None) or (None, bigger plan) on overflow."""
        ev = h.get("ev")
        if ev is None:
            self._torch_stream().synchronize()
            misc = h["misc"][:2].cpu().numpy().view(np.uint32)
            self.d2h_bytes += 8
        else:                                      # staged by _stage_readback: wait for this solve only
            ev.synchronize()
            misc = h["hread"][:8].numpy().view(np.uint32).copy()
            self.d2h_bytes += 8 + h["hrows"] * self.result_bytes
        if self._queued.get(h.get("set")) is h:
            del self._queued[h["set"]]
        npairs, err = int(misc[0]), int(misc[1])
        plan = h["plan"]
        if err & _lib.ERR_TABLE_FULL:
            raise _lib.CfError(_lib.CF_EOVERFLOW, "solve", "D table full (internal error)")
        if err & (_lib.ERR_PART_OVERFLOW | _lib.ERR_PAIR_OVERFLOW):
            newp = dict(plan)
            if err & _lib.ERR_PART_OVERFLOW and h["dcnt"] is None:
                # fused: a survivor list of the class join, or a bucket range of the table build, ran out
                newp["no_class" if plan.get("class_plan") else "no_part"] = True
            elif err & _lib.ERR_PART_OVERFLOW:
                dmax = int(h["dcnt"].max().item())
                imax = int(h["icnt"].max().item())
                newp["capD"] = max(plan["capD"], dmax + 16)
                newp["capI"] = max(plan["capI"], imax + 16)
            if err & _lib.ERR_PAIR_OVERFLOW:
                newp["pairs"] = max(plan["pairs"] * 2, npairs + 16)
            return None, newp
        if err & _lib.ERR_SPIN_LIMIT:
            raise _lib.CfError(_lib.CF_ETIMEOUT, "solve", "a bounded device wait gave up")
        if err & 32:
            raise _lib.CfError(_lib.CF_EBADARG, "solve", "a kernel rejected its arguments (pool primes >= 2^31?)")
        if err & _lib.ERR_KEY_MISMATCH:
            raise _lib.CfError(_lib.CF_EBADARG, "solve", "checked pair with unequal residues (internal error)")
        nb = npairs * self.result_bytes
        if ev is not None and npairs <= h["hrows"]:
            res = np.frombuffer(h["hread"][8:8 + nb].numpy().tobytes(), dtype=RESULT_DTYPE)
        else:
            res = np.frombuffer(h["res"][:nb].cpu().numpy().tobytes(), dtype=RESULT_DTYPE)
            self.d2h_bytes += nb
        return self._finish(inst, h, res, verify), None

    def _finish(self, inst: Instance, h: dict, res: np.ndarray, verify: bool) -> SolveResult:
        return finish_rows(inst, res, h["nD"], h["nI"], h["plan"], verify)

    def _direct_plan(self, inst: Instance, i_limit: int | None, i_lo: int = 0, cp: bytes | None = None) -> dict | None:
        """The device plan of a fused or partition join of inst over the I ranks [i_lo, i_limit), or
        None when inst takes another path (radius 0, the bounded strategy, an empty window).  cp: the
        class plan of this instance and window where the caller has it."""
        if inst.r == 0:
            return None
        st = self.tuning.strategy
        if i_limit is None and not i_lo and (st == "bounded" or st == "auto"):
            from . import bsolve
            if bsolve.applicable(inst) and (st == "bounded" or bsolve.prunes(inst)):
                return None
        nD = ncomb(len(inst.B0), inst.r)
        nI = _i_window(inst, {"i_limit": i_limit, "i_lo": i_lo})
        if nI == 0 or nD == 0:
            return None
        plan = self.plan(nD, nI)
        plan["i_limit"] = i_limit
        plan["i_lo"] = int(i_lo)
        if min(nD, nI) >= 1 << 32:        # ranks in the fused table are 32-bit
            plan["strategy"] = "partition"
        if plan["strategy"] == "fused":
            plan["class_plan"] = cp or self._class_plan(inst, plan)
            if plan["class_plan"]:
                plan["pairs"] = class_pairs(nD, nI, inst.M, self.tuning)
        return plan

    def _replan(self, inst: Instance, newp: dict) -> dict:
        """The plan after an overflow: the capacities collect() asked for."""
        nD, nI = ncomb(len(inst.B0), inst.r), _i_window(inst, newp)
        plan = self.plan(nD, nI, newp["capD"], newp["capI"], newp["pairs"])
        plan["strategy"] = newp.get("strategy", plan["strategy"])
        plan["i_limit"] = newp.get("i_limit")
        plan["i_lo"] = _i_lo(newp)
        plan["no_part"] = newp.get("no_part", False)
        plan["no_class"] = newp.get("no_class", False)
        if plan["no_class"]:
            self._drop_class()
        if plan["strategy"] == "fused":
            plan["class_plan"] = self._class_plan(inst, plan)
        return plan

    def _drop_class(self):
        """Give the set's class workspace up: it is not held beside the other join's buffers."""
        self._bufs.pop(("class", self._bufset), None)
        self._reserved.get(self._bufset, {}).pop("class", None)
        self._class_cover = 0.0

    def solve_instance(self, inst: Instance, verify: bool = True, timed: bool = False,
                       marks: list | None = None, i_limit: int | None = None, i_lo: int = 0) -> SolveResult:
        """Join one instance.  i_lo, i_limit: join only the I ranks [i_lo, i_limit) (a bounded
        sample of the instance, or one device's share of it; every pair with such an I rank
        is found).  n_I of the result is the window's size."""
        if i_lo < 0 or (i_limit is not None and i_limit < 0):
            raise ValueError("the I-rank window must not start or end below 0")
        plan = self._direct_plan(inst, i_limit, i_lo)
        if plan is None:
            if inst.r == 0:
                return self._solve_r0(inst)
            st = self.tuning.strategy
            if i_limit is None and not i_lo and (st == "bounded" or st == "auto"):
                from . import bsolve
                if bsolve.applicable(inst) and (st == "bounded" or bsolve.prunes(inst)):
                    if self._bounded is None:
                        self._bounded = bsolve.BoundedSolve(self)
                    return self._bounded.solve(inst, verify)
            nD = ncomb(len(inst.B0), inst.r)
            return SolveResult([], nD, _i_window(inst, {"i_limit": i_limit, "i_lo": i_lo}), 0, 0, 0, 0)
        return self._run_plan(inst, plan, verify, timed, marks)

    def _run_plan(self, inst: Instance, plan: dict, verify: bool, timed: bool = False,
                  marks: list | None = None) -> SolveResult:
        """Enqueue, collect, and re-run with larger capacities while a buffer overflows."""
        for _attempt in range(6):
            ev0 = ev1 = None
            if timed:
                ev0 = self.torch.cuda.Event(enable_timing=True)
                ev1 = self.torch.cuda.Event(enable_timing=True)
                ev0.record(self._torch_stream())
            if marks is not None:
                marks.clear()
            h = self.enqueue(inst, plan, marks)
            if timed:
                ev1.record(self._torch_stream())
            out, newp = self.collect(inst, h, verify)
            if out is not None:
                if timed:
                    out.device_ms = ev0.elapsed_time(ev1)
                out.launches = h["launches"]
                return out
            plan = self._replan(inst, newp)
        raise _lib.CfError(_lib.CF_EOVERFLOW, "solve", "capacities kept overflowing")

    def _stage_readback(self, h: dict, rows: int):
        """Queue, behind a solve's kernels, the copy of its counters and of its first `rows`
        checked rows into page-locked memory, and an event after them: collect() then waits
        for this solve alone, not for work queued after it."""
        if h.get("ev") is not None:                # cf_solve has queued it
            return
        torch = self.torch
        rb = self.result_bytes
        rows = max(0, min(int(rows), int(h["plan"]["pairs"])))
        hm = self._pinned_buf("readback", 8 + rows * rb)
        st = self._torch_stream()
        with torch.cuda.stream(st):
            hm[:8].copy_(h["misc"][:2].view(torch.uint8), non_blocking=True)
            if rows:
                hm[8:8 + rows * rb].copy_(h["res"][: rows * rb], non_blocking=True)
        ev = torch.cuda.Event()
        ev.record(st)
        h.update(ev=ev, hread=hm, hrows=rows)

    def _reserve(self, insts: list, i_limit: int | None, i_lo: int, class_plans: list | None, use) -> dict:
        """The buffers of a list's fused solves, in both sets, at the sizes of its largest instances: grown
        solve by solve, a list of uneven pools met the device allocator (a millisecond of each of the first
        solves) between its kernels.  A class workspace is known by its plan only: unless one was reserved for
        longer survivor lists before, the instance whose lists should be the longest is planned here, and
        an eighth is added for the others' moduli.  Returns the plans made, by position."""
        tu, lib, plans = self.tuning, self.lib, {}
        if tu.strategy != "fused":
            return plans
        mb = mi = mr = small = 0
        by_class = []
        pairs = tu.pair_capacity
        for (nb, ni, r), i in {(len(x.B0), len(x.INS), x.r): i for i, x in enumerate(insts)}.items():
            nD, nI = ncomb(nb, r), ncomb(ni, r)
            nI = max(0, (nI if i_limit is None else min(nI, i_limit)) - i_lo)
            n, m = (nD, nI) if nD < nI else (nI, nD)
            if r == 0 or n == 0 or n >= 1 << 32:
                continue
            mb, mi, mr = max(mb, nb), max(mi, ni), max(mr, r)
            if not tu.class_join or m < class_least(r, n, tu):
                small = max(small, n)
                continue
            if nD * nI >> insts[i].M.bit_length() >= tu.pair_capacity >> 4:
                pairs = max(pairs, class_pairs(nD, nI, insts[i].M, tu))
            load = min(n / 140, 1e5) / 49152            # filter load, and passes of the filter, see cf_class_plan
            by_class.append((m * (load + load * load), i))
        if not mr:
            return plans
        mb, mi = max(mb, mr), max(mi, mr)
        need = dict(ctr=64, pairs=pairs * 16, res=pairs * self.result_bytes, tables=lib.cf_solve_table_bytes(mb, mi, mr))
        if small:
            need["dtab"] = lib.cf_dtab_bytes2(*dtab_shape(small, tu))
            need["tails"] = lib.cf_solve_tail_bytes(mb, mi, mr)
        if class_plans:
            need["class"] = max(map(_ws_bytes, class_plans))
        elif by_class:
            for est, i in sorted(by_class, reverse=True)[:3]:
                if est <= self._class_cover:
                    break
                plans[i] = self._direct_plan(insts[i], i_limit, i_lo)
                cp = plans[i].get("class_plan")
                if cp:
                    need["class"] = _ws_bytes(cp) * 9 // 8
                    self._class_cover = est
                    break
        rows = 8 + max(0, min(self._rows, tu.pair_capacity)) * self.result_bytes
        for k in range(min(2, len(insts))):
            have = self._reserved.setdefault(k, {})
            if rows <= have.get("rows", 0) and all([v <= have.get(name, 0) for name, v in need.items()]):
                continue
            with use(k):
                try:
                    for name, v in need.items():        # the workspace last: the rest is small
                        have[name] = self._buf(name, v).numel()
                except self.torch.OutOfMemoryError:
                    pass                                # the solves that do not fit find out one by one
                else:
                    self._pinned_buf("stage", need["tables"])
                    self._pinned_buf("readback", rows)
                    have["rows"] = rows
        return plans

    def solve_many(self, insts: list, verify: bool = True, marks_list: list | None = None,
                   i_limit: int | None = None, readback_rows: int = 256, streams: int = 2,
                   i_lo: int = 0, class_plans: list | None = None) -> list[SolveResult]:
        """Solve instances one after another, each with its own build, probe and check, while
        the host collects and certifies each one as the device runs the next: two buffer sets
        alternate, and every solve's counters and first checked rows come back behind its own
        kernels.  With streams = 2 the two buffer sets also have a CUDA stream each, so one
        solve's table build can run beside the previous solve's probe.  The results equal
        solve_instance's on each instance (i_lo, i_limit: the same I-rank window for every
        instance; class_plans: their class plans where the caller has them).  marks_list (optional
        list) receives one marks list per instance (see enqueue)."""
        torch = self.torch
        out: list = [None] * len(insts)
        base = self._torch_stream()
        saved = (self.stream, self.tables.stream)
        if getattr(self, "_many_streams", None) is None:
            self._many_streams = [torch.cuda.Stream(self.device), torch.cuda.Stream(self.device)]
        sts = self._many_streams[:2] if streams > 1 else [base]
        for st in sts:
            if st is not base:
                st.wait_stream(base)               # after everything queued before the call

        def use(k):
            self._bufset = k & 1
            st = sts[k & 1] if len(sts) > 1 else sts[0]
            self.stream = st
            self.tables.stream = st
            return torch.cuda.stream(st)

        pending = None
        self._rows = int(readback_rows)
        self._pool = base
        try:
            plans = self._reserve(insts, i_limit, i_lo, class_plans, use)
            for i in range(len(insts) + 1):
                cur = None
                if i < len(insts):
                    inst = insts[i]
                    marks = None
                    if marks_list is not None:
                        marks = []
                        marks_list.append(marks)
                    with use(i):                   # the set (and stream) the solve in flight does not use
                        plan = plans.get(i) or self._direct_plan(inst, i_limit, i_lo,
                                                                 class_plans[i] if class_plans else None)
                        if plan is None:
                            out[i] = self.solve_instance(inst, verify=verify, marks=marks, i_limit=i_limit,
                                                         i_lo=i_lo)
                        else:
                            h = self.enqueue(inst, plan, marks)
                            self._stage_readback(h, readback_rows)
                            cur = (i, h, marks)
                if pending is not None:
                    j, h, marks = pending
                    with use(j):
                        res, newp = self.collect(insts[j], h, verify)
                        if res is None:            # an overflow: run it again alone, larger
                            res = self._run_plan(insts[j], self._replan(insts[j], newp), verify, marks=marks)
                        else:
                            res.launches = h["launches"]
                    out[j] = res
                pending = cur
        finally:
            self._bufset = 0
            self._pool = None
            self._rows = self.READBACK_ROWS
            self.stream, self.tables.stream = saved
            for st in sts:
                if st is not base:
                    base.wait_stream(st)           # work queued after the call follows every solve
        return out

    def _torch_stream(self):
        return self.stream if self.stream is not None else self.torch.cuda.current_stream(self.device)

    def _solve_r0(self, inst: Instance) -> SolveResult:
        n = inst.P0
        hits = []
        if n % inst.M == 1 % inst.M and n <= inst.B:
            ok, _, _ = verify_certificate(inst.B0)
            if ok:
                hits.append(Hit((), (), n, tuple(inst.B0)))
        return SolveResult(hits, 1, 1, int(n % inst.M == 1 % inst.M), len(hits), 0, 0)

    def solve(self, M: int, Q, B0, r: int, B: int, verify: bool = True, timed: bool = False) -> SolveResult:
        return self.solve_instance(Instance.build(M, Q, B0, r, B), verify=verify, timed=timed)


_default_solvers: dict = {}


def solve(M: int, Q, B0, r: int, B: int, device=None, verify: bool = True, strategy: str = "fused") -> SolveResult:
    """Every Carmichael hit S = (B0 \\ D) u I with |D| = |I| = r, prod(S) == 1 (mod M), prod(S) <= B.

    Q is the eligible pool Q(M) (primes q with (q-1) | M and q not dividing M);
    INS = Q \\ B0.  Hits are certified on the host and returned ascending by n.
    strategy: "fused" (table + generate-and-probe), "partition" (materialised join), "bounded"
    (both sides pruned by the size bound, then a record join) or "auto" (bounded where the
    bound prunes, else fused).  Every strategy returns the same hits."""
    import torch
    dev = torch.device(device if device is not None else "cuda")
    key = (dev.type, dev.index, strategy)
    s = _default_solvers.get(key)
    if s is None:
        s = _default_solvers[key] = Solver(dev, tuning=Tuning(strategy=strategy))
    return s.solve(M, Q, B0, r, B, verify=verify)


def solve_many(instances, device=None, verify: bool = True, strategy: str = "fused") -> list[SolveResult]:
    """solve() over a list of (M, Q, B0, r, B) tuples (or objects with those attributes), in order:
    each instance is joined on its own on the device, while the host prepares the next one's
    tables and collects and certifies the previous one.  Returns one SolveResult per instance,
    equal to solve()'s."""
    import torch
    dev = torch.device(device if device is not None else "cuda")
    key = (dev.type, dev.index, strategy)
    s = _default_solvers.get(key)
    if s is None:
        s = _default_solvers[key] = Solver(dev, tuning=Tuning(strategy=strategy))
    xs = []
    for w in instances:
        M, Q, B0, r, B = (w.M, w.Q, w.B0, w.r, w.B) if hasattr(w, "M") else w
        xs.append(Instance.build(M, Q, B0, r, B))
    return s.solve_many(xs, verify=verify)


def decode_pair(inst: Instance, d_rank: int, i_rank: int):
    """(D primes, I primes) of a pair of lexicographic ranks."""
    di = unrank_lex(d_rank, len(inst.B0), inst.r)
    ii = unrank_lex(i_rank, len(inst.INS), inst.r)
    return tuple(inst.B0[i] for i in di), tuple(inst.INS[i] for i in ii)
