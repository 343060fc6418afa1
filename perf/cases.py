"""Measured cases: what users of the engine have it do, over the sizes they do it at.

Every case goes through the public entry points of ``awsemmd_b200.engine``
(and ``awsem_fragmem_noalloc`` of the C ABI, which takes device pointers):

* ``force``    one force call per MD step of a host code (``fix backbone/gpu``
               in LAMMPS): host positions in, host forces and energies out;
* ``md``       device-resident Langevin dynamics of one system;
* ``windows``  the same cut at output steps, where the input-script driver
               reads energies and the state;
* ``batch``    independent replicas advanced together;
* ``serve``    requests admitted to a serving handle, run and collected;
* ``fragmem``  the fragment-memory term alone on device buffers.

Systems are random AWSEM chains as the benchmark configurations describe
them (self-avoiding CA walks, 20 noisy memories per 9-residue window), made
here from the seed with torch.  ``exact`` evaluates the force field in 64 bits
from its published formulas with torch and automatic differentiation.
"""
import atexit
import ctypes
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from awsemmd_b200 import engine, synth

AA = "ARNDCQEGHILKMFPSTWYV"
GLY, PRO = AA.index("G"), AA.index("P")
WINDOW, MEMORIES, MIN_SEP = 9, 20, 3
MASS = (27.0, 28.0, 60.0, 2.0)  # CA, O, CB, H-beta
KT2V = 48.88821291 * 48.88821291
BOLTZ = 0.0019872067
DT, DAMP, TEMP = 2.0, 500.0, 300.0
PARAMS = os.path.join(os.path.dirname(os.path.abspath(engine.__file__)), "params")


def listed():
    return [
        # the smallest protein the project benchmarks (one chain of 100), as LAMMPS drives it: a call per step
        {"name": "force_100_fp64", "kind": "force", "chains": 1, "length": 100, "precision": "fp64"},
        # 8 chains of 250 (the single-system configuration), driven the same way in the mixed form
        {"name": "force_2000_mixed", "kind": "force", "chains": 8, "length": 250, "precision": "mixed"},
        # folding one small chain, state on the device
        {"name": "md_100_fp64", "kind": "md", "chains": 1, "length": 100, "precision": "fp64", "steps": 100},
        # the single-system configuration in the plain form and in the mixed form
        {"name": "md_2000_fp64", "kind": "md", "chains": 8, "length": 250, "precision": "fp64", "steps": 50},
        {"name": "md_2000_mixed", "kind": "md", "chains": 8, "length": 250, "precision": "mixed", "steps": 50},
        # the largest single system (160 chains of 250; cell-grid lists rebuilt every 10 steps)
        {"name": "md_40000_mixed", "kind": "md", "chains": 160, "length": 250, "precision": "mixed", "steps": 20,
         "neigh_every": 10},
        # an input script's run of an ordinary protein: output every 20 steps
        {"name": "windows_333_mixed", "kind": "windows", "chains": 1, "length": 333, "precision": "mixed", "steps": 100,
         "every": 20},
        # replica sampling in the plain form: 61 chains of 40 to 500 residues
        {"name": "batch_61_fp64", "kind": "batch", "replicas": 61, "lo": 40, "hi": 500, "precision": "fp64", "steps": 20},
        # the headline workload: 1,024 chains of 40 to 500 residues
        {"name": "batch_1024_mixed", "kind": "batch", "replicas": 1024, "lo": 40, "hi": 500, "precision": "mixed",
         "steps": 20},
        # structure-prediction requests of 30 to 1,000 residues served together, annealed 600 K -> 300 K
        {"name": "serve_24_mixed", "kind": "serve", "replicas": 24, "lo": 30, "hi": 1000, "precision": "mixed",
         "steps": 100},
        # the allocation-free fragment-memory call: one chain in the plain form, and near its size limit with
        # weighted memories
        {"name": "fragmem_250_fp64", "kind": "fragmem", "chains": 1, "length": 250, "precision": "fp64",
         "weighted": False},
        {"name": "fragmem_8000_mixed", "kind": "fragmem", "chains": 32, "length": 250, "precision": "mixed",
         "weighted": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["force", "md", "md", "windows", "batch", "batch", "serve", "fragmem"])
    precision = rng.choice(["fp64", "mixed", "mixed"])
    if kind in ("force", "md", "windows", "fragmem"):
        length = rng.randint(20, 400)
        most = {"force": 12000, "md": 24000, "windows": 4000, "fragmem": 8000}[kind]
        total = _log_int(rng, 40, most if precision == "mixed" else most // 3)
        case = {"kind": kind, "chains": max(1, total // length), "length": min(length, total), "precision": precision}
        if kind == "md":
            case["steps"] = rng.randint(15, 60)
            if rng.random() < 0.3:
                case["neigh_every"] = 10
        elif kind == "windows":
            case["steps"], case["every"] = 20 * rng.randint(2, 5), rng.choice([5, 10, 20])
        elif kind == "fragmem":
            case["weighted"] = rng.random() < 0.5
        return case
    if kind == "batch":
        replicas = _log_int(rng, 2, 400 if precision == "mixed" else 100)
        return {"kind": kind, "replicas": replicas, "lo": rng.randint(10, 60), "hi": rng.randint(100, 500),
                "precision": precision, "steps": rng.randint(10, 30)}
    return {"kind": kind, "replicas": _log_int(rng, 2, 32), "lo": rng.randint(12, 60), "hi": rng.randint(200, 1000),
            "precision": precision, "steps": rng.randint(20, 120)}


# --------------------------------------------------------------------------
# random systems

def _lengths(case):
    """Chain lengths and each chain's replica."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        g = np.random.default_rng(1000 * case["replicas"] + 10 * case["lo"] + case["hi"])  # the workload's lengths
        lo, hi, n = case["lo"], case["hi"], case["replicas"]
        if kind == "batch":
            ln = g.integers(lo, hi + 1, size=n)
        else:
            ln = np.exp(g.uniform(math.log(lo), math.log(hi), size=n)).round().astype(int)
        return [int(v) for v in ln], list(range(n))
    return [case["length"]] * case["chains"], [0] * case["chains"]


def _pick(mask, a, b):
    """a where the mask holds, else b, numbers taken in 64 bits."""
    a, b = (v if torch.is_tensor(v) else torch.full((), v, dtype=torch.float64, device=mask.device) for v in (a, b))
    return torch.where(mask, a, b)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True).clamp_min(1e-9)


def _walks(lengths, gen, dev):
    """Self-avoiding CA walks [chains][longest][3]: 3.8 A bonds, angles N(110, 10) degrees, of 24 proposals the first
    that stays 4 A from the chain (the farthest where none does)."""
    m, top, tries = len(lengths), max(max(lengths), 3), 24
    p = torch.zeros(m, top, 3, dtype=torch.float64, device=dev)
    p[:, 1, 0] = 3.8
    ang = torch.deg2rad(110 + 10 * torch.randn(m, top, tries, generator=gen, dtype=torch.float64, device=dev))
    tor = (2 * torch.rand(m, top, tries, generator=gen, dtype=torch.float64, device=dev) - 1) * math.pi
    p[:, 2] = p[:, 1] + 3.8 * torch.stack([-ang[:, 2, 0].cos(), ang[:, 2, 0].sin(), 0 * ang[:, 2, 0]], -1)
    order = sorted(range(m), key=lambda k: -lengths[k])
    still = torch.tensor([lengths[k] for k in order], device=dev)
    p = p[torch.tensor(order, device=dev)]
    counts = [int(v) for v in (torch.arange(top, device=dev)[:, None] < still[None]).sum(1).cpu()]
    for k in range(3, top):
        q = counts[k]  # the chains that reach this far: the first q
        bc = _unit(p[:q, k - 1] - p[:q, k - 2])
        nv = _unit(torch.linalg.cross(p[:q, k - 2] - p[:q, k - 3], bc))
        mv = torch.linalg.cross(nv, bc)
        th, ph = ang[:q, k, :, None], tor[:q, k, :, None]
        c = p[:q, k - 1, None] + 3.8 * (-th.cos() * bc[:, None] + th.sin() * ph.cos() * mv[:, None]
                                        + th.sin() * ph.sin() * nv[:, None])
        near = torch.cdist(c, p[:q, :k - 1], compute_mode="donot_use_mm_for_euclid_dist").amin(-1)
        ok = near >= 4.0
        best = torch.where(ok.any(1), ok.to(torch.int8).argmax(1), near.argmax(1))
        p[:q, k] = c[torch.arange(q, device=dev), best]
    out = torch.empty_like(p)
    out[torch.tensor(order, device=dev)] = p
    return [out[k, :n] for k, n in enumerate(lengths)]


def _beads(ca, first, last, gly):
    """O and CB / H-beta positions around a CA trace, CB on the L side."""
    prev = torch.where(first[:, None], 2 * ca - ca.roll(-1, 0), ca.roll(1, 0))
    nxt = torch.where(last[:, None], 2 * ca - ca.roll(1, 0), ca.roll(-1, 0))
    e1, e2 = _unit(ca - prev), _unit(nxt - ca)
    # a chain's ends have no bend: any normal will do there
    n = torch.linalg.cross(e1, e2)
    side = torch.linalg.cross(e1, _pick(e1[:, :1].abs() < 0.9, e1.new_tensor([1.0, 0, 0]), e1.new_tensor([0, 1.0, 0])))
    n = _unit(_pick(n.norm(dim=-1, keepdim=True) > 1e-6, n, side))
    u = e1 - e2
    u = _unit(_pick(u.norm(dim=-1, keepdim=True) > 1e-6, u, torch.linalg.cross(n, e1)))
    along = (2.40 ** 2 - 2.76 ** 2 + 3.8 ** 2) / 7.6
    perp = math.sqrt(2.40 ** 2 - along ** 2)
    sign = 1.0 - 2.0 * (torch.arange(len(ca), device=ca.device) % 2)[:, None]
    o = ca + along * e2 + perp * sign * n
    r = _pick(gly, 1.09, 1.53)[:, None]
    a = math.radians(52.0)
    cb = ca + r * (math.cos(a) * u - math.sin(a) * n)
    nv, cp = _virtual(ca, o)[0], _virtual(ca, o)[2]
    chi = (torch.linalg.cross(cp - ca, ca - nv) * (ca - cb)).sum(-1)
    flip = ((chi > 0) & ~first & ~last)[:, None]
    return o, torch.where(flip, cb + 2 * r * math.sin(a) * n, cb)


def _pack(parts, box, gen, dev):
    """A random rotation and place for each chain in the box, no two chains' CAs closer than about 4 A."""
    side = int(box + 400)
    taken = torch.zeros(side, side, side, dtype=torch.bool, device=dev)
    ball = torch.stack(torch.meshgrid(*[torch.arange(-4, 5, device=dev)] * 3, indexing="ij"), -1).reshape(-1, 3)
    ball = ball[(ball.double().norm(dim=1) <= 4.0)]
    moves = []
    for ca in parts:
        ca = ca - ca.mean(0)
        while True:
            n = 512
            q, _ = torch.linalg.qr(torch.randn(n, 3, 3, generator=gen, dtype=torch.float64, device=dev))
            q = q * torch.linalg.det(q)[:, None, None]
            at = (torch.rand(n, 1, 3, generator=gen, dtype=torch.float64, device=dev) - 0.5) * box
            cell = ((ca[None] @ q.transpose(1, 2) + at) + side / 2).long().clamp(0, side - 1)
            hit = taken[cell[..., 0], cell[..., 1], cell[..., 2]].any(1)
            good = (~hit).nonzero()
            if len(good):
                k = int(good[0])
                break
        moves.append((q[k], at[k]))
        mark = (cell[k][:, None] + ball[None]).clamp(0, side - 1).reshape(-1, 3)
        taken[mark[:, 0], mark[:, 1], mark[:, 2]] = True
    return moves


def _system(case, seed):
    """Everything about the case's chains, concatenated: torch tensors on the GPU (the CPU without one)."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    gen = torch.Generator(dev).manual_seed(int(seed) * 7919 + 17)
    lengths, rep = _lengths(case)
    n = sum(lengths)
    ln = torch.tensor(lengths, device=dev)
    chain = torch.repeat_interleave(torch.arange(len(lengths), device=dev), ln)
    start = torch.cumsum(ln, 0) - ln
    idx = torch.arange(n, device=dev)
    first, last = idx == start[chain], idx == (start + ln - 1)[chain]
    seq = torch.randint(0, 20, (n,), generator=gen, device=dev)
    walks = _walks(lengths, gen, dev)
    ca = torch.cat([w - w.mean(0) for w in walks])
    gly = seq == GLY
    o, cb = _beads(ca, first, last, gly)
    if len(set(rep)) < len(rep):  # several chains in one box: the configurations' density
        box = 150.0 * (n / 2000.0) ** (1 / 3) if n < 20000 else 320.0 * (n / 40000.0) ** (1 / 3)
        for k, (q, at) in enumerate(_pack(walks, max(box, 40.0), gen, dev)):
            s = slice(int(start[k]), int(start[k]) + lengths[k])
            ca[s], o[s], cb[s] = (v[s] @ q.T + at for v in (ca, o, cb))
    x = torch.stack([ca, o, cb], 1)
    mass = torch.tensor(MASS, dtype=torch.float64, device=dev)
    mass = torch.stack([mass[0].expand(n), mass[1].expand(n), torch.where(gly, mass[3], mass[2])], 1)
    v = torch.randn(n, 3, 3, generator=gen, dtype=torch.float64, device=dev) * (BOLTZ * TEMP / KT2V / mass).sqrt()[..., None]
    # helix / strand / coil segments of 4 to 12 residues
    cut = torch.randint(4, 13, (n,), generator=gen, device=dev).cumsum(0)
    kinds = torch.randint(0, 3, (n + 1,), generator=gen, device=dev)
    ss = kinds[torch.searchsorted(cut, idx, right=True)]
    # memories: noisy copies of every window of every chain
    w0 = idx[(idx + WINDOW - 1 < n) & (chain[(idx + WINDOW - 1).clamp(max=n - 1)] == chain)]
    at = w0[:, None] + torch.arange(WINDOW, device=dev)
    shape = (len(w0), MEMORIES, WINDOW, 3)
    mca = ca[at][:, None] + torch.randn(shape, generator=gen, dtype=torch.float64, device=dev)
    mcb = cb[at][:, None] + torch.randn(shape, generator=gen, dtype=torch.float64, device=dev)
    weight = torch.ones(len(w0), MEMORIES, dtype=torch.float64, device=dev)
    if case.get("weighted"):
        weight = 0.5 + torch.rand(weight.shape, generator=gen, dtype=torch.float64, device=dev)
    return {"lengths": lengths, "rep": rep, "chain": chain, "start": start, "end": start + ln - 1, "first": first,
            "last": last, "seq": seq, "gly": gly, "x": x, "v": v, "mass": mass, "ss": ss, "w0": w0, "mca": mca,
            "mcb": mcb, "weight": weight, "dev": dev}


def _descriptions(s):
    """The replicas as the engine takes them (host arrays, atoms CA, O, CB of each residue)."""
    x, v, seq = s["x"].cpu().numpy(), s["v"].cpu().numpy(), s["seq"].cpu().numpy()
    ss = s["ss"].cpu().numpy()
    w0, weight = s["w0"].cpu().numpy(), s["weight"].cpu().numpy()
    mca, mcb = s["mca"].cpu().numpy(), s["mcb"].cpu().numpy()
    letters = np.frombuffer(AA.encode(), np.uint8)[seq]
    out, chains, c0, r0 = [], s["lengths"], 0, 0
    while c0 < len(chains):
        c1 = c0
        while c1 < len(chains) and s["rep"][c1] == s["rep"][c0]:
            c1 += 1
        n = sum(chains[c0:c1])
        r = slice(r0, r0 + n)
        a, b = np.searchsorted(w0, [r0, r0 + n])
        m = (b - a) * MEMORIES
        here = w0[a:b]
        out.append({
            "n_res": n, "chain_len": np.array(chains[c0:c1], np.int32), "seq": letters[r].tobytes(),
            "ssweight": np.stack([ss[r] == 0, ss[r] == 1], 1).astype(np.float64),
            "x": np.ascontiguousarray(x[r]), "v": np.ascontiguousarray(v[r]), "n_mem": m,
            "mem_pos": np.repeat((here - r0).astype(np.int32), MEMORIES), "mem_len": np.full(m, WINDOW, np.int32),
            "mem_weight": np.ascontiguousarray(weight[a:b].reshape(-1)),
            "mem_seq": np.repeat(letters[here[:, None] + np.arange(WINDOW)][:, None], MEMORIES, 1).tobytes(),
            "mem_ca": mca[a:b].reshape(-1, 3), "mem_cb": mcb[a:b].reshape(-1, 3)})
        c0, r0 = c1, r0 + n
    return out


_FORCEFIELD = {}


def _forcefield():
    """The run directory with the force field's tables (one per process)."""
    if not _FORCEFIELD:
        d = tempfile.mkdtemp(prefix="awsem_")
        atexit.register(shutil.rmtree, d, True)
        _FORCEFIELD.update(synth.forcefield_dir(d))
    return _FORCEFIELD


def _seeds(n):
    return [101 + 7 * k for k in range(n)]


# --------------------------------------------------------------------------
# the measured calls

def prepare(case, seed):
    s = _system(case, seed)
    desc = _descriptions(s)
    st = {"case": case}
    if case["kind"] == "serve":
        records = sum(32 * -(-d["n_res"] // 32) * 6 * MEMORIES * 8 for d in desc)
        srv = engine.AwsemServer(_forcefield(), sum(32 * -(-d["n_res"] // 32) for d in desc) + 64, len(desc) + 2,
                                 records, precision=case["precision"], dt=DT, damp=DAMP)
        st["srv"], st["requests"] = srv, [srv.prepare(d, seed=k) for d, k in zip(desc, _seeds(len(desc)))]
        return st
    st["sys"] = sys_ = engine.AwsemBatch.from_arrays(_forcefield(), desc, precision=case["precision"],
                                                     seeds=_seeds(len(desc)))
    if case["kind"] == "fragmem":
        # the entry point's order: CA, CB, O of each residue, on the device
        st["x"] = s["x"][:, [0, 2, 1]].reshape(-1, 3).contiguous()
        st["f"], st["e"] = torch.empty_like(st["x"]), torch.empty(1, dtype=torch.float64, device=st["x"].device)
        fn = sys_.lib.awsem_fragmem_noalloc
        fn.argtypes = [ctypes.c_void_p] * 5
        st["fn"] = fn
        return st
    pin = torch.cuda.is_available()
    for key in ("x", "v"):  # page-locked host arrays, as a host code that moves state every call keeps them
        t = torch.empty(sys_.natoms, 3, dtype=torch.float64, pin_memory=pin)
        t.copy_(s[key].reshape(-1, 3))
        st[key] = t.numpy()
        st["new_" + key] = torch.empty(sys_.natoms, 3, dtype=torch.float64, pin_memory=pin).numpy()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "fragmem":
        rc = st["fn"](st["sys"].h, st["x"].data_ptr(), st["f"].data_ptr(), st["e"].data_ptr(),
                      torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("awsem_fragmem_noalloc failed")
        return {"f": st["f"], "e": st["e"]}
    if kind == "serve":
        srv = st["srv"]
        slots = [srv.admit(r, case["steps"], t_start=600.0, t_stop=300.0) for r in st["requests"]]
        srv.advance(case["steps"] + 1)
        got = [srv.collect(k) for k in slots]
        return {"x": np.concatenate([g[0] for g in got]), "v": np.concatenate([g[1] for g in got]),
                "energies": np.stack([g[2] for g in got])}
    sys_ = st["sys"]
    if kind == "force":
        f, e = sys_.compute(st["x"])
        return {"f": f, "energies": e}
    kw = {"dt": DT, "damp": DAMP, "t_start": TEMP, "t_stop": TEMP, "neigh_every": case.get("neigh_every", 0)}
    if kind == "batch":
        sys_.set_state_all(st["x"], st["v"])
        sys_.run(case["steps"], **kw)
        x, v = sys_.get_state_all(st["new_x"], st["new_v"])
        return {"x": x, "v": v, "energies": sys_.energies(0)}
    sys_.set_state(st["x"], st["v"])
    if kind == "md":
        sys_.run(case["steps"], **kw)
        x, v = sys_.get_state()
        return {"x": x, "v": v, "f": sys_.forces(), "energies": sys_.energies()}
    begin = sys_.step
    window = (begin, begin + case["steps"])
    sys_.run_window(0, window, False, **kw)
    frames, energies = [], [sys_.energies()]
    for at in range(0, case["steps"], case["every"]):
        sys_.run_window(min(case["every"], case["steps"] - at), window, True, **kw)
        energies.append(sys_.energies())
        frames.append(sys_.get_state())
    return {"x": np.stack([f[0] for f in frames]), "v": np.stack([f[1] for f in frames]), "energies": np.stack(energies)}


def work(case):
    """One pass's unavoidable traffic and arithmetic.  Per evaluation: every memory distance once, positions read,
    forces written (and, when integrating, positions and velocities read and written); about 12 operations per memory
    Gaussian, 60 per residue pair within 9.5 A (5 a residue) and 2,000 per residue for its backbone terms."""
    lengths, _ = _lengths(case)
    n, size = sum(lengths), 8 if case["precision"] == "fp64" else 4
    records = sum(max(ln - WINDOW + 1, 0) for ln in lengths) * MEMORIES * 21
    if case["kind"] == "fragmem":
        return {"bytes": records * (5 if case["weighted"] else 4) * size + n * 144, "flops": records * 48}
    evals = 1 if case["kind"] == "force" else case["steps"] + 1
    per = records * 4 * size + n * (144 if case["kind"] == "force" else 360)
    return {"bytes": evals * per, "flops": evals * (records * 48 + n * (5 * 60 + 2000))}


# --------------------------------------------------------------------------
# the force field in 64 bits

A_N, B_N, C_N = 0.483, 0.703, -0.186
A_P, B_P, C_P = 0.444, 0.235, 0.321
A_H, B_H, C_H = 0.841, 0.893, -0.734


def _dist(u, v):
    return ((u - v) ** 2).sum(-1).clamp_min(1e-20).sqrt()


def _virtual(ca, o):
    """N, H (of residues with a predecessor) and C' (with a successor)."""
    p, q, n = ca.roll(1, 0), o.roll(1, 0), ca.roll(-1, 0)
    return A_N * p + B_N * ca + C_N * q, A_H * p + B_H * ca + C_H * q, A_P * ca + B_P * n + C_P * o


def _table(name):
    with open(os.path.join(PARAMS, name)) as f:
        return np.array(f.read().split(), dtype=np.float64)


class _Field:
    """Energies of the default parameter file (with fragment memory, vexcluded 2 3.5 3.5 and the data file's harmonic
    bonds) over the concatenated chains of a _system."""

    def __init__(self, s):
        self.s, dev = s, s["dev"]
        t = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        g = _table("gamma.dat")[:840].reshape(2, 210, 2)
        up = np.triu_indices(20)
        water = np.zeros((2, 20, 20, 2))
        water[:, up[0], up[1]] = g
        water[:, up[1], up[0]] = g
        self.water, self.burial = t(water), t(_table("burial_gamma.dat")[:60].reshape(20, 3))
        two = lambda name: t(_table(name)[:800].reshape(2, 20, 20))  # noqa: E731
        self.ahb, self.anhb, self.phb = two("anti_HB"), two("anti_NHB"), two("para_HB")
        self.p1, self.a1 = t(_table("para_one")[:20]), t(_table("anti_one")[:20])
        self.h4 = t([0.77, 0.68, 0.07, 0.15, 0.23, 0.33, 0.27, 0.0, 0.06, 0.23, 0.62, 0.65, 0.50, 0.41, -3.0, 0.35, 0.11,
                     0.45, 0.17, 0.14])
        self.rep = torch.tensor(s["rep"], device=dev)[s["chain"]]
        self.pairs = None
        # memories: [windows][20][21 pairs][4 distances], 1e30 where glycine has no CB
        a, b = np.triu_indices(WINDOW, MIN_SEP)
        self.fa, self.fb = s["w0"][:, None] + torch.tensor(a, device=dev), s["w0"][:, None] + torch.tensor(b, device=dev)
        d = lambda u, v, i, j: (u[:, :, i] - v[:, :, j]).norm(dim=-1)  # noqa: E731
        m = torch.stack([d(s["mca"], s["mca"], a, b), d(s["mca"], s["mcb"], a, b), d(s["mcb"], s["mca"], a, b),
                         d(s["mcb"], s["mcb"], a, b)], -1)
        ga, gb = s["gly"][self.fa][:, None], s["gly"][self.fb][:, None]
        no = torch.stack([torch.zeros_like(ga), gb, ga, ga | gb], -1)
        self.mem = _pick(no, t(1e30), m)
        self.fm_var = t((b - a).astype(np.float64) ** 0.3)[:, None]

    def list_pairs(self, ca, reach=20.0):
        """Residue pairs i < j of one replica with CAs within reach."""
        n, out = len(ca), []
        for r in range(0, n, 2048):
            q = torch.cdist(ca[r:r + 2048], ca, compute_mode="donot_use_mm_for_euclid_dist") < reach
            q &= self.rep[r:r + 2048, None] == self.rep[None]
            i, j = q.nonzero(as_tuple=True)
            i = i + r
            out.append(torch.stack([i[j > i], j[j > i]]))
        self.pairs = torch.cat(out, 1)

    def energies(self, x):
        """(21 per-residue energy slots that carry forces, the sum to differentiate) at x [n][CA, O, CB][3]."""
        s = self.s
        ca, o, cb = x[:, 0], x[:, 1], x[:, 2]
        n, dev, seq, chain, gly, first, last = len(ca), s["dev"], s["seq"], s["chain"], s["gly"], s["first"], s["last"]
        N, H, CP = _virtual(ca, o)
        pro = seq == PRO
        idx = torch.arange(n, device=dev)
        E = {}
        add = lambda k, i, e: E.__setitem__(k, E.get(k, torch.zeros(n, dtype=torch.float64, device=dev)).index_add(0, i, e))  # noqa: E731
        dist = _dist
        # chain, chi
        for k, r0, u, v, m in ((10.0, 2.45798, N, cb, ~first & ~gly), (10.0, 2.50665, CP, cb, ~last & ~gly),
                               (30.0, 2.44973, N, CP, ~first & ~last)):
            add(1, idx[m], k * (dist(u[m], v[m]) - r0) ** 2)
        m = ~first & ~last & ~gly
        i = idx[m]
        a, b, c = CP[i] - ca[i], ca[i] - N[i], ca[i] - cb[i]
        chi = (torch.linalg.cross(a, b) * c).sum(-1) / (a.norm(dim=-1) * b.norm(dim=-1) * c.norm(dim=-1))
        add(3, i, 20.0 * (chi + 0.83) ** 2)
        # Ramachandran wells
        if len(i):
            def dihedral(a, b, c):
                dot = lambda u, v: (u * v).sum(-1)  # noqa: E731
                return torch.atan2(b.norm(dim=-1) * dot(c, torch.linalg.cross(b, a)),
                                   dot(a, b) * dot(b, c) - dot(b, b) * dot(a, c))
            phi = dihedral(CP[i] - ca[i], ca[i] - N[i], N[i] - CP[i - 1])
            psi = dihedral(N[i + 1] - CP[i], CP[i] - ca[i], ca[i] - N[i])
            wells = [(1.3149, 15.398, 0.15, 1.74, 0.65, -2.138), (1.32016, 49.0521, 0.25, 1.265, 0.45, 0.318),
                     (1.0264, 49.0954, 0.65, -1.041, 0.25, -0.78), (2.0, 419.0, 1.0, 0.995, 1.0, 0.820),
                     (2.0, 15.398, 1.0, 2.25, 1.0, -2.16)]
            prow = [(2.17, 105.52, 1.0, 1.153, 0.15, -2.4), (2.15, 109.09, 1.0, 0.95, 0.15, 0.218)]
            e = torch.zeros(len(i), dtype=torch.float64, device=dev)
            for k, (w, sg, fw, f0, sw, s0) in enumerate(wells + prow):
                on = (pro[i] if k >= 5 else ~pro[i]).double()
                scale = (s["ss"][i] == k - 3).double() if k in (3, 4) else 1.0
                e = e - 2.0 * w * on * scale * torch.exp(-sg * fw * ((phi + f0).cos() - 1) ** 2
                                                         - sg * sw * ((psi + s0).cos() - 1) ** 2)
            add(4, i, e)
        # residue pairs
        pi, pj = self.pairs
        other = chain[pi] != chain[pj]
        sep = pj - pi
        con = _pick(gly[:, None], ca, cb)
        rc = dist(con[pi], con[pj])

        def well(r, kappa, lo, hi):
            e = 0.25 * (1 + torch.tanh(kappa * (r - lo))) * (1 + torch.tanh(kappa * (hi - r)))
            span = 8.0 * 2.302585 / kappa
            return _pick((r > lo - span) & (r < hi + span), e, 0.0)

        far = other | (sep > 1)
        th0, th1, thh = (_pick(far, well(rc, k, lo, hi), 0.0) for k, lo, hi in ((5.0, 4.5, 6.5), (5.0, 6.5, 9.5),
                                                                                     (7.0, 4.5, 6.5)))
        zero = torch.zeros(n, dtype=torch.float64, device=dev)
        rho = zero.index_add(0, pi, th0).index_add(0, pj, th0)
        rho_h = zero.index_add(0, pi, thh).index_add(0, pj, thh)
        sig, sig_h = 0.5 * (1 - torch.tanh(7.0 * (rho - 2.6))), 0.5 * (1 - torch.tanh(7.0 * (rho_h - 3.0)))
        for k, lo, hi in ((0, 0.0, 3.0), (1, 3.0, 6.0), (2, 6.0, 9.0)):
            add(9, idx, -0.5 * self.burial[seq, k] * (torch.tanh(4.0 * (rho - lo)) + torch.tanh(4.0 * (hi - rho))))
        wide = other | (sep >= 10)
        for w, th in ((0, th0), (1, th1)):
            g = self.water[w, seq[pi], seq[pj]]
            sg = _pick((g[:, 0] - g[:, 1]).abs() < 1e-5, 0.5 * g.sum(-1),
                             g[:, 0] + (g[:, 1] - g[:, 0]) * sig[pi] * sig[pj])
            add(8, pi, _pick(wide, -sg * th, 0.0))
        # helical i, i + 4
        i = idx[:max(n - 4, 0)]
        i = i[chain[i] == chain[i + 4]]
        j = i + 4
        rn, rh = dist(o[i], N[j]), dist(o[i], H[j])
        prob = _pick(pro[i], self.h4[PRO], self.h4[seq[i]]) + self.h4[seq[j]]
        th = -1.5 * prob * torch.exp(-0.5 * (((rn - 2.98) / 0.68) ** 2 + ((rh - 2.06) / 0.76) ** 2))
        add(10, i, _pick(rn <= 6.0, (2.0 - 3.0 * sig_h[i] * sig_h[j]) * th, 0.0))
        # hydrogen bonds: acceptor O(i), donor N-H(j), both orders of each pair
        ai, dj = torch.cat([pi, pj]), torch.cat([pj, pi])
        keep = (chain[ai] != chain[dj]) | ((ai - dj).abs() > 2)
        keep &= ~pro[dj] & ~first[dj] & ~last[ai] & (dist(o[ai], N[dj]) < 7.0)
        self._dssp(add, ai[keep], dj[keep], ca, o, N, H, pro)
        # P_AP
        keep = (other | (sep >= min(5 + 8, 9))) & (dist(ca[pi], ca[pj]) < 8.0 + math.atanh(1 - 2e-12) / 7.0)
        self._pap(add, pi[keep], pj[keep], ca)
        # excluded volume: CA-CA, CA-CB, CB-CB (3.5 A in a chain below 5 residues apart, else 4.5) and O-O (3.5)
        rc = _pick(~other & (sep < 5), 3.5, 4.5)
        close = dist(ca[pi], ca[pj]) < 12.0
        pi2, pj2, rc2, bonded = pi[close], pj[close], rc[close], (~other & (sep == 1))[close]
        for u, v, m, r0 in ((ca, ca, ~bonded, rc2), (ca, cb, ~gly[pj2], rc2), (cb, ca, ~gly[pi2], rc2),
                            (cb, cb, ~gly[pi2] & ~gly[pj2], rc2), (o, o, rc2 > 0, torch.full_like(rc2, 3.5))):
            r = dist(u[pi2], v[pj2])
            m = m & (r < r0)
            add(18, pi2[m], 20.0 * (r[m] - r0[m]) ** 2)
        # harmonic bonds
        q = idx[~last]
        for u, v, r0, at in ((ca, o, 2.40, idx), (ca, cb, _pick(gly, 1.09, 1.53), idx)):
            add(19, at, 60.0 * (dist(u[at], v[at]) - r0) ** 2)
        add(19, q, 60.0 * (dist(ca[q], ca[q + 1]) - 3.816) ** 2 + 60.0 * (dist(o[q], ca[q + 1]) - 2.76) ** 2)
        total = sum(e.sum() for e in E.values())
        fm, surrogate = self.memory(ca, cb)
        E[12] = fm
        return E, total + surrogate

    def memory(self, ca, cb):
        """Fragment-memory energy per residue, and a scalar with its gradient."""
        s = self.s
        if not len(s["w0"]):
            z = torch.zeros(len(ca), dtype=torch.float64, device=s["dev"])
            return z, (ca * 0).sum()
        i, j = self.fa, self.fb
        r = torch.stack([(u[i] - v[j]).norm(dim=-1) for u in (ca, cb) for v in (ca, cb)], -1)  # [windows][21][4]
        with torch.no_grad():
            e, slope = torch.zeros_like(r), torch.zeros_like(r)
            for m in range(MEMORIES):
                d = r - self.mem[:, m]
                g = s["weight"][:, m, None, None] * torch.exp(-0.5 * d * d / self.fm_var)
                e -= g
                slope += _pick(g > 0, g * d / self.fm_var, 0.0)
            per = torch.zeros(len(ca), dtype=torch.float64, device=s["dev"]).index_add(0, i.reshape(-1), e.sum(-1).reshape(-1))
        return per, (slope * r).sum()

    def _dssp(self, add, i, j, ca, o, N, H, pro):
        s = self.s
        if not len(i):
            return
        seq, chain, first, last, top = s["seq"], s["chain"], s["first"], s["last"], len(s["seq"]) - 1
        ci, cj = chain[i], chain[j]
        rep_on = ~last[j] & ~pro[(j + 1).clamp(max=top)]
        ap_on = ~first[i] & ~last[j] & ~pro[i]
        p_on = (i < s["end"][ci] - 1) & ~last[j] & ~pro[(i + 2).clamp(max=top)]
        at = lambda k: k.clamp(0, top)  # noqa: E731
        same = ci == cj
        dij = (i - j).abs()
        cls = torch.where(same & (dij < 4), 0, torch.where(same & (dij < 18), 1, torch.where(same & (dij < 45), 2, 3)))
        tsa = [_pick(ap_on, 0.5 * self.ahb[k, seq[i], seq[j]], 0.0) for k in (0, 1)]
        tsn = [_pick(ap_on, 0.25 * (self.anhb[k, seq[at(i + 1)], seq[at(j - 1)]]
                                          + self.anhb[k, seq[at(i - 1)], seq[at(j + 1)]]), 0.0) for k in (0, 1)]
        tsp = _pick(p_on, self.phb[1, seq[at(i + 1)], seq[j]], 0.0)
        one, par = self.a1[seq[i]] + self.a1[seq[j]], self.p1[seq[at(i + 1)]] + self.p1[seq[j]]
        strand = (s["ss"][i] == 1) & (s["ss"][j] == 1)
        zero = torch.zeros_like(one)
        rows = []
        rows.append((zero, zero, zero, zero))
        rows.append((_pick(strand, -1.37, 0.0), zero,
                     _pick(strand, -3.49 - 1.30 * tsa[0] - 1.32 * tsn[0] - 1.22 * one, 0.0), zero))
        for a, b, c, d, e, f, g, h, k in ((1.36, 0.0, 3.50, 1.30, 1.32, 1.22, 3.47, 0.33, 1.01),
                                          (1.17, 0.0, 3.52, 1.30, 1.32, 1.22, 3.62, 0.33, 1.01)):
            rows.append((zero - a, zero - b, -c - d * tsa[1] - e * tsn[1] - f * one, -g - h * tsp - k * par))
        lam = [torch.stack([r[k] for r in rows]).gather(0, cls[None])[0] for k in range(4)]
        nus = []
        for c, ch, pref in ((i, ci, 1.0), (j, cj, 0.5)):
            use = (c - 2 >= s["start"][ch]) & (c + 2 <= s["end"][ch]) & (cls != 1)
            r = _dist(ca[at(c + 2)], ca[at(c - 2)])
            cut = abs(12.0 + math.atanh(2e-4 - 1) / pref)  # compared squared
            nu = _pick(r > cut, 0.5 * (1 + torch.tanh(pref * (r - 12.0))), 0.0)
            nus.append(_pick(use, nu, 1.0))
        gate = (nus[0] >= 1e-4) & (nus[1] >= 1e-4)
        th = []
        for acc, don, on in ((i, j, rep_on | True), (i, at(j + 1), rep_on), (j, i, ap_on), (j, at(i + 2), p_on)):
            rn, rh = _dist(o[acc], N[don]), _dist(o[acc], H[don])
            th.append(_pick(on, torch.exp(-0.5 * (((rn - 2.98) / 0.68) ** 2 + ((rh - 2.06) / 0.76) ** 2)), 0.0))
        e = th[0] * (lam[0] + lam[1] * th[1] + lam[2] * th[2] + lam[3] * th[3]) * nus[0] * nus[1]
        add(6, i[gate], e[gate])

    def _pap(self, add, i, j, ca):
        s = self.s
        if not len(i):
            return
        chain, top, dd, lo, hi = s["chain"], len(s["seq"]) - 1, 4, 5, 8
        ci, cj = chain[i], chain[j]
        ie, je = s["end"][ci] + 1, s["end"][cj] + 1
        same = ci == cj
        at = lambda k: k.clamp(0, top)  # noqa: E731

        def nu(a, b):
            r = _dist(ca[a], ca[b])
            span = float(int(8.0 * 2.302585 / 7.0) + 1)
            v = 0.5 * (1 + torch.tanh(7.0 * (8.0 - r)))
            return _pick(r > 8.0 + span, 0.0, _pick(r < 8.0 - span, 1.0, v))

        n0 = nu(i, j)
        med = same & (i < ie - (lo + 2 * dd)) & (j >= i + lo + 2 * dd) & (j <= torch.minimum(i + hi + 2 * dd, ie - 1))
        inside = (i + dd <= top) & (chain[at(i + dd)] == ci)
        lng = (same & (i < ie - (hi + 2 * dd + 1)) & (j >= i + hi + 2 * dd + 1) & (j < je)) | (
            ~same & inside & (j - dd >= 0) & (chain[at(j - dd)] == cj))
        par = (same & (i < ie - (hi + 1 + dd)) & (j >= i + hi + 1) & (j < ie - dd)) | (
            ~same & inside & (j + dd <= top) & (chain[at(j + dd)] == cj))
        beta = (s["ss"][i] == 1) & (s["ss"][j] == 1)
        factor = _pick(beta, 1.5, 1.0)
        gate = n0 >= 1e-12
        m = (med | lng) & gate
        k = med.double() + lng.double() * 0.4 * factor
        add(7, i[m], (-k * n0 * nu(at(i + dd), at(j - dd)))[m])
        m = par & gate
        add(7, i[m], (-0.4 * factor * n0 * nu(at(i + dd), at(j + dd)))[m])

    def forces(self, x):
        x = x.detach().requires_grad_(True)
        e, total = self.energies(x)
        (g,) = torch.autograd.grad(total, x)
        return -g, {k: v.detach() for k, v in e.items()}


def _mix(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _vector(e, rep, reps, kinetic=None):
    """The energies[21] rows of every replica."""
    out = np.zeros((reps, 21))
    for k, v in e.items():
        out[:, k] = torch.zeros(reps, dtype=torch.float64, device=v.device).index_add(0, rep, v).cpu().numpy()
    out[:, 0] = out[:, 1:18].sum(1)
    if kinetic is not None:
        out[:, 20] = torch.zeros(reps, dtype=torch.float64, device=rep.device).index_add(0, rep, kinetic).cpu().numpy()
    return out


def exact(case, seed):
    lengths, rep = _lengths(case)
    kind = case["kind"]
    evals = case.get("steps", 0) + 1
    if sum(lengths) * evals > 900000:
        return None
    s = _system(case, seed)
    field = _Field(s)
    x, reps = s["x"], max(rep) + 1
    if kind == "fragmem":
        x = x.detach().requires_grad_(True)
        e, surrogate = field.memory(x[:, 0], x[:, 2])
        (g,) = torch.autograd.grad(surrogate, x)
        return {"f": -g[:, [0, 2, 1]].reshape(-1, 3), "e": e.sum().reshape(1)}
    field.list_pairs(x[:, 0])
    if kind == "force":
        f, e = field.forces(x)
        return {"f": f.reshape(-1, 3), "energies": _vector(e, field.rep, reps)[0]}
    # velocity Verlet with Langevin forces, the noise keyed by (seed, step, atom id, component)
    dev, steps = s["dev"], case["steps"]
    t0, t1 = (600.0, 300.0) if kind == "serve" else (TEMP, TEMP)
    v, mass = s["v"].clone(), s["mass"][..., None]
    seeds = np.array(_seeds(reps), dtype=np.uint64)
    first = np.concatenate([[0], np.cumsum(np.bincount(field.rep.cpu().numpy(), minlength=reps))])
    rep_np = field.rep.cpu().numpy()
    tag = 3 * (np.arange(len(x)) - first[rep_np])[:, None] + np.arange(1, 4)
    key_at = (tag.astype(np.uint64)[..., None] * np.uint64(4)) + np.arange(3, dtype=np.uint64)
    drag = -mass / DAMP * KT2V
    kick = mass.sqrt() * math.sqrt(24.0 * BOLTZ / DAMP / DT / KT2V) * KT2V
    dtfm = 0.5 * DT / KT2V / mass
    frames, rows = [], []
    old = np.seterr(over="ignore")
    for step in range(steps + 1):
        if step % 10 == 0:
            field.list_pairs(x[:, 0])
        f, e = field.forces(x)
        key = _mix(seeds ^ _mix(np.array([step], dtype=np.uint64)))[rep_np]
        u = (_mix(key[:, None, None] ^ key_at) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
        temp = t0 + (step / steps) * (t1 - t0)
        f = f + drag * v + kick * math.sqrt(temp) * (torch.tensor(u, device=dev) - 0.5)
        if step:
            v = v + dtfm * f
        kinetic = 0.5 * KT2V * (mass * v * v).sum((1, 2))
        if kind == "windows" and (step % case["every"] == 0 or step == steps):
            rows.append(_vector(e, field.rep, reps, kinetic)[0])
            if step:
                frames.append((x.reshape(-1, 3), v.reshape(-1, 3)))
        if step < steps:
            v = v + dtfm * f
            x = x + DT * v
    np.seterr(**old)
    if kind == "windows":
        return {"x": torch.stack([q[0] for q in frames]), "v": torch.stack([q[1] for q in frames]),
                "energies": np.stack(rows)}
    energies = _vector(e, field.rep, reps, kinetic)
    out = {"x": x.reshape(-1, 3), "v": v.reshape(-1, 3), "energies": energies if kind == "serve" else energies[0]}
    if kind == "md":
        out["f"] = f.reshape(-1, 3)
    return out
