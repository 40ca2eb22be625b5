"""The work a program has this framework do, as cases that can be timed.

Every case goes through the public entry points (`mmc_ctypes`, the binding of
include/mmc.h): temperature stages of one lattice, of a batch of replicas and
of a parallel-tempering farm, the demag convolution on device buffers, the
energy gradient and the relaxation.  Sizes, materials and schedules are those
of the benchmark, the tests and the command line's example configuration, or
generic ones.  A stage case is what the anneal loop does between two outputs:
sweeps at one temperature, the observables, and the state read back.
"""
import atexit
import ctypes
import math
import os
import shutil
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "micromagnetic-gpu-monte-carlo_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import mmc_ctypes as M  # noqa: E402

# the material of the benchmark film (strong interfacial DMI) and of the slab
FILM = dict(dx=1e-9, dy=1e-9, dz=0.8e-9, ms=1.6e6, Aex=16e-12, Dind=6e-3, Ku1=2e6, anisUx=0.0, anisUy=0.0,
            anisUz=1.0, Bextx=0.0, Bexty=0.0, Bextz=0.3)
SLAB = dict(dx=2e-9, dy=2e-9, dz=1e-9, ms=1.1e6, Aex=15e-12, Dind=3e-3, Ku1=0.8e6, anisUx=0.0, anisUy=0.0,
            anisUz=1.0, Bextx=0.0, Bexty=0.0, Bextz=0.2)

_CACHE = None


def _cache_dir():
    """The tensor cache folder of this process (the library's own -tensorcache=
    feature): a program keeps the Newell tensor of a geometry."""
    global _CACHE
    if _CACHE is None:
        _CACHE = tempfile.mkdtemp(prefix="mmc_tensor_")
        atexit.register(shutil.rmtree, _CACHE, True)
    return _CACHE


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: a small film advanced a few sweeps between looks at
        # its observables (an interactive run, a short output period)
        dict(name="film32_f32_short", kind="stage", nx=32, ny=32, nz=1, pbc=20, precision=32, sweeps=10, T=300.0,
             material="film"),
        # the command line's example film in double precision: part of a stage
        dict(name="film64_f64_stage", kind="stage", nx=64, ny=64, nz=1, pbc=20, precision=64, sweeps=200, T=700.0,
             material="film"),
        # one 256 x 256 film, single precision: the usual single-lattice anneal
        dict(name="film256_f32_stage", kind="stage", nx=256, ny=256, nz=1, pbc=20, precision=32, sweeps=400, T=400.0,
             material="film"),
        # the same film in double precision, the reference-grade anneal
        dict(name="film256_f64_stage", kind="stage", nx=256, ny=256, nz=1, pbc=20, precision=64, sweeps=100, T=400.0,
             material="film"),
        # the benchmark's batch: 64 replicas of the 256 x 256 film, autotuned
        dict(name="batch64_256_f32", kind="batch", nx=256, ny=256, nz=1, pbc=20, precision=32, replicas=64,
             sweeps=1000, T=400.0, material="film", tune=True),
        # a seed ensemble of small films in double precision (the statistics
        # runs), launch shape as the library chooses it
        dict(name="batch32_64_f64", kind="batch", nx=64, ny=64, nz=1, pbc=20, precision=64, replicas=32, sweeps=100,
             T=300.0, material="film", tune=False),
        # replicas of an open rectangular film of odd sides (a patterned
        # element), launch shape as the library chooses it
        dict(name="batch8_151x89_open_f32", kind="batch", nx=151, ny=89, nz=1, pbc=0, precision=32, replicas=8,
             sweeps=200, T=150.0, material="film", tune=False),
        # parallel tempering: two batches (sides 128 and 256) of 32 replicas in
        # ladders of 16 temperatures, swaps every 10 sweeps, advanced as a farm
        dict(name="tempering_128_256_f32", kind="tempering", side0=128, side1=256, ladders=2, per_ladder=16,
             swap=10, sweeps=400, precision=32, pbc=20),
        # a thick film: eight layers, single precision
        dict(name="slab512x512x8_f32", kind="stage", nx=512, ny=512, nz=8, pbc=4, precision=32, sweeps=200, T=300.0,
             material="slab"),
        # the demag convolution alone on device buffers (a program with its own
        # time stepper), an open square element
        dict(name="demag512_open_f32", kind="demag", nx=512, ny=512, nz=1, pbc=0, precision=32, material="film"),
        # the energy gradient of an open film in double precision
        dict(name="grad256_open_f64", kind="grad", nx=256, ny=256, nz=1, pbc=0, precision=64, material="film"),
        # energy minimisation of a film in double precision, a bounded number
        # of steps
        dict(name="relax128_f64", kind="relax", nx=128, ny=128, nz=1, pbc=20, precision=64, steps=100,
             material="film"),
    ]


def _smooth(n):
    """Whether a periodic side has a transform: no prime factor above 31."""
    for f in range(2, 32):
        while n % f == 0:
            n //= f
    return n == 1


def _side(rng, lo, hi, periodic):
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if rng.random() < 0.5:  # half the sides as users like them
            n = max(8, 8 * round(n / 8))
        if not periodic or _smooth(n):
            return n


def draw(rng):
    kind = rng.choice(["stage", "stage", "stage", "batch", "batch", "batch", "tempering", "demag", "grad", "relax"])
    T = round(math.exp(rng.uniform(math.log(45.0), math.log(1400.0))), 1)
    if kind == "tempering":
        s = sorted([_side(rng, 64, 256, True), _side(rng, 64, 256, True)])
        return dict(kind=kind, side0=s[0], side1=s[1], ladders=rng.randint(1, 2), per_ladder=rng.choice([8, 12, 16]),
                    swap=rng.choice([5, 10, 20]), sweeps=rng.randrange(100, 400), precision=32,
                    pbc=rng.choice([2, 5, 20]))
    pbc = rng.choice([0, 0, 2, 5, 20])
    periodic = pbc != 0
    precision = rng.choice([32, 32, 64])
    if kind == "stage":
        nz = rng.choice([1, 1, 1, 2, 5, 8])
        hi = 384 if nz == 1 else 160
        nx, ny = _side(rng, 24, hi, periodic), _side(rng, 24, hi, periodic)
        most = 4e7 if precision == 32 else 8e6  # trials of a pass
        sweeps = int(max(5, min(500, rng.uniform(0.3, 1.0) * most / (nx * ny * nz))))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, pbc=min(pbc, 5) if nz > 1 else pbc, precision=precision,
                    sweeps=sweeps, T=T, material="film" if nz == 1 else "slab")
    if kind == "batch":
        R = rng.choice([2, 5, 8, 16, 24, 32, 64])
        nx, ny = _side(rng, 24, 256, periodic), _side(rng, 24, 256, periodic)
        most = 4e8 if precision == 32 else 1e7
        sweeps = int(max(5, min(500, rng.uniform(0.3, 1.0) * most / (R * nx * ny))))
        return dict(kind=kind, nx=nx, ny=ny, nz=1, pbc=pbc, precision=precision, replicas=R, sweeps=sweeps, T=T,
                    material="film", tune=rng.random() < 0.5)
    if kind == "demag":
        return dict(kind=kind, nx=_side(rng, 48, 512, False), ny=_side(rng, 48, 512, False), nz=1, pbc=0,
                    precision=precision, material="film")
    if kind == "grad":
        return dict(kind=kind, nx=_side(rng, 32, 256, False), ny=_side(rng, 32, 256, False), nz=1, pbc=0,
                    precision=precision, material="film")
    return dict(kind="relax", nx=_side(rng, 32, 192, periodic), ny=_side(rng, 32, 192, periodic), nz=1, pbc=pbc,
                precision=64, steps=rng.randint(40, 100), material="film")


# ------------------------------------------------------------------- prepare
def _config(case, seed, **kw):
    mat = FILM if case.get("material", "film") == "film" else SLAB
    d = dict(nx=case.get("nx"), ny=case.get("ny"), nz=case.get("nz", 1), pbc_x=case["pbc"], pbc_y=case["pbc"], pbc_z=0,
             precision=case["precision"], cal_demag_flag=1, use_random_init=1, randomseed=int(seed),
             Temperature_start=float(case.get("T", 300.0)), **mat)
    if case.get("nz", 1) > 1 and case["pbc"] > 0:
        d["tensor_far_radius"] = 32  # far images of a thick lattice by their expansion, as the benchmark's slab
    d.update(kw)
    return M.Config.defaults(**d)


def _random_m(n, seed, dtype):
    """Independent unit vectors, uniform on the sphere (3 x n, x block first)."""
    g = torch.Generator(device="cpu")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    z = 2 * torch.rand(n, generator=g, dtype=torch.float64) - 1
    a = 2 * math.pi * torch.rand(n, generator=g, dtype=torch.float64)
    r = torch.sqrt(1 - z * z)
    return torch.stack([r * torch.cos(a), r * torch.sin(a), z]).to(dtype).contiguous()


def _textured_m(case, seed):
    """A smooth texture with a little noise: the states that are relaxed and
    differentiated in earnest, float64 3 x n."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(int(seed) & 0x7FFFFFFF)
    x = 2 * np.pi * (np.arange(nx) / nx)[None, None, :]
    y = 2 * np.pi * (np.arange(ny) / ny)[None, :, None]
    p = rng.uniform(0, 2 * np.pi, 4)
    th = np.pi * (0.5 + 0.45 * np.sin(2 * x + p[0]) * np.cos(y + p[1])) + 0.02 * rng.standard_normal((nz, ny, nx))
    ph = 2 * np.sin(x + p[2]) + np.cos(2 * y + p[3]) + 0.02 * rng.standard_normal((nz, ny, nx))
    m = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)]).reshape(3, -1)
    return m / np.sqrt((m * m).sum(0))


def _pbatch(case, seed, side, bz, dind):
    """One batch of the tempering farm: `ladders` ladders of `per_ladder` temperatures."""
    R = case["ladders"] * case["per_ladder"]
    cfgs = []
    for r in range(R):
        k = r // case["per_ladder"]
        cfgs.append(_config(case, seed + r, nx=side, ny=side, nz=1, Bextz=bz[k], Dind=dind[k]))
    b = M.Batch(cfgs)
    b.build_demag(_cache_dir())
    T = np.geomspace(40.0, 1400.0, case["per_ladder"])
    b.set_ladders(np.arange(R, dtype=np.int32).reshape(case["ladders"], -1), np.tile(T, (case["ladders"], 1)),
                  case["swap"], seed % 100000)
    b.autotune(4)
    return b


def prepare(case, seed):
    seed = int(seed) % (1 << 40)
    kind = case["kind"]
    s = {"case": case}
    if kind == "stage":
        lat = M.Lattice(_config(case, seed))
        lat.build_demag(_cache_dir())
        s["lat"] = lat
    elif kind == "batch":
        b = M.Batch([_config(case, seed + r) for r in range(case["replicas"])])
        b.build_demag(_cache_dir())
        if case["tune"]:
            b.autotune(32)
        s["batches"] = [b]
    elif kind == "tempering":
        rng = np.random.default_rng(64)
        bz, dind = rng.uniform(0.1, 0.5, 4), rng.uniform(3e-3, 6e-3, 4)
        L = case["ladders"]
        s["batches"] = [_pbatch(case, seed, case["side0"], bz[:L], dind[:L]),
                        _pbatch(case, seed + 1000, case["side1"], bz[2:], dind[2:])]
        s["farm"] = M.Farm(s["batches"])
    elif kind == "demag":
        lat = M.Lattice(_config(case, seed))
        lat.build_demag()
        dt = torch.float32 if case["precision"] == 32 else torch.float64
        s["lat"] = lat
        s["m"] = _random_m(lat.n, seed, dt).cuda()
        s["h"] = torch.zeros_like(s["m"])
        s["bytes"] = lat.demag_scratch_bytes()
        s["scratch"] = torch.empty(s["bytes"], dtype=torch.uint8, device="cuda")
        s["stream"] = torch.cuda.Stream()
        s["ptr"] = [ctypes.c_void_p(s[k].data_ptr()) for k in ("m", "h", "scratch")]
        torch.cuda.synchronize()
    else:
        lat = M.Lattice(_config(case, seed))
        lat.build_demag(_cache_dir() if case["pbc"] else "")
        s["m0"] = _textured_m(case, seed)
        lat.set_m(s["m0"])
        s["lat"] = lat
    for b in s.get("batches", ()):  # where the states are read back to
        s.setdefault("out", []).append(np.zeros((b.R, 3, b.n)))
    return s


# ----------------------------------------------------------------------- run
def _observables(obs):
    e = np.array([[o.e_exchange, o.e_dmi, o.e_anisotropy, o.e_zeeman, o.e_demag, o.e_total] for o in obs])
    return {"energy": e, "m_avg": np.array([list(o.m) for o in obs]), "charge": np.array([o.q for o in obs]),
            "accepted": np.array([o.accepted for o in obs], dtype=np.int64)}


def _batch_state(b, out):
    L = M.lib()
    for r in range(b.R):
        M.check(L.mmc_batch_get_m(b.h, r, M.dptr(out[r, 0]), M.dptr(out[r, 1]), M.dptr(out[r, 2])))
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "stage":
        lat = state["lat"]
        lat.run_sweeps(case["T"], 0, 0, case["sweeps"])
        return dict(_observables([lat.energy()]), m=lat.get_m())
    if kind == "batch":
        b = state["batches"][0]
        b.run_sweeps(0, 0, case["sweeps"])
        return dict(_observables(b.energy()), m=_batch_state(b, state["out"][0]))
    if kind == "tempering":
        state["farm"].run_sweeps(0, 0, case["sweeps"])
        outs = []
        for b, out in zip(state["batches"], state["out"]):
            rep, counts = b.ladder_state()
            outs.append(dict(m=_batch_state(b, out), replicas=rep.astype(np.int64), counts=counts.astype(np.int64),
                             temperatures=b.temperatures()))
        return outs
    if kind == "demag":
        mp, hp, sp = state["ptr"]
        state["lat"].demag_apply(mp, hp, sp, state["bytes"], ctypes.c_void_p(state["stream"].cuda_stream))
        return state["h"]
    lat = state["lat"]
    if kind == "grad":
        g, dp = lat.grad()
        return {"dE_dm": g, "dE_dparams": [float(v) for v in dp]}
    lat.set_m(state["m0"])  # every pass minimises from the same state
    it, torque = lat.relax(torque_tol=1e-12, max_iter=case["steps"])
    return {"iterations": it, "torque": torque, "m": lat.get_m()}


# ---------------------------------------------------------------------- work
def _demag_work(nx, ny, nz, pbc, s):
    """(bytes of the tensor spectrum, flops) of one demag convolution: six real
    transforms of the zero-padded grid and the 3 x 3 real symmetric product."""
    px, py, pz = (nx, ny) + (nz,) if pbc else (2 * nx - 1, 2 * ny - 1, nz)
    pz = 2 * nz - 1
    N = px * py * pz
    return 6 * s * (px // 2 + 1) * py * pz, 6 * 2.5 * N * math.log2(max(N, 2)) + 30.0 * N / 2


def _sweep_work(nx, ny, nz, pbc, s, replicas, sweeps, evals=1):
    """Sweeps of `replicas` lattices and `evals` observables passes: each sweep
    reads and writes m and reads the tensor spectrum; a trial is a proposal, a
    local energy difference and a decision."""
    n = nx * ny * nz
    kb, df = _demag_work(nx, ny, nz, pbc, s)
    return {"bytes": sweeps * (kb + replicas * 6 * s * n) + evals * replicas * 3 * s * n + replicas * 24 * n,
            "flops": replicas * (sweeps * (df + 110.0 * n) + evals * (df + 150.0 * n))}


def work(case):
    s = case["precision"] // 8
    kind = case["kind"]
    if kind in ("stage", "batch"):
        return _sweep_work(case["nx"], case["ny"], case["nz"], case["pbc"], s, case.get("replicas", 1), case["sweeps"])
    if kind == "tempering":
        R = case["ladders"] * case["per_ladder"]
        w = [_sweep_work(a, a, 1, case["pbc"], s, R, case["sweeps"], case["sweeps"] // case["swap"])
             for a in (case["side0"], case["side1"])]
        return {k: w[0][k] + w[1][k] for k in w[0]}
    n = case["nx"] * case["ny"] * case["nz"]
    kb, df = _demag_work(case["nx"], case["ny"], case["nz"], case["pbc"], s)
    if kind == "demag":
        return {"bytes": kb + 6 * s * n, "flops": df}
    if kind == "grad":
        return {"bytes": kb + 3 * s * n + 24 * n, "flops": df + 150.0 * n}
    k = case["steps"]
    return {"bytes": (k + 1) * (kb + 6 * s * n + 48 * n) + 48 * n, "flops": (k + 1) * (df + 150.0 * n)}


# --------------------------------------------------------------------- exact
def _newell_nodes(n, d):
    """f(x,y,z), f(y,z,x), f(z,x,y), g(x,y,z), g(x,z,y), g(y,z,x) of Newell,
    Williams and Dunlop at the lattice nodes 0..n[a]."""
    X, Y, Z = np.meshgrid(*[np.arange(n[a] + 1) * d[a] for a in range(3)], indexing="ij")
    eps = 1e-200

    def f(x, y, z):
        R = np.sqrt(x * x + y * y + z * z)
        return (y / 2 * (z * z - x * x) * np.arcsinh(y / (np.sqrt(x * x + z * z) + eps))
                + z / 2 * (y * y - x * x) * np.arcsinh(z / (np.sqrt(x * x + y * y) + eps))
                - x * y * z * np.arctan(y * z / (x * R + eps)) + (2 * x * x - y * y - z * z) * R / 6)

    def g(x, y, z):
        R = np.sqrt(x * x + y * y + z * z)
        return (x * y * z * np.arcsinh(z / (np.sqrt(x * x + y * y) + eps))
                + y / 6 * (3 * z * z - y * y) * np.arcsinh(x / (np.sqrt(y * y + z * z) + eps))
                + x / 6 * (3 * z * z - x * x) * np.arcsinh(y / (np.sqrt(x * x + z * z) + eps))
                - z ** 3 / 6 * np.arctan(x * y / (z * R + eps)) - z * y * y / 2 * np.arctan(x * z / (y * R + eps))
                - z * x * x / 2 * np.arctan(y * z / (x * R + eps)) - x * y * R / 3)

    # xx, xy, xz, yy, yz, zz and each one's parity along x, y, z
    return [(f(X, Y, Z), (1, 1, 1)), (g(X, Y, Z), (-1, -1, 1)), (g(X, Z, Y), (-1, 1, -1)), (f(Y, Z, X), (1, 1, 1)),
            (g(Y, Z, X), (1, -1, -1)), (f(Z, X, Y), (1, 1, 1))]


def _open_tensor(n, d):
    """The six blocks of the open lattice's demag tensor at offsets
    -(n-1) .. n-1 per axis, laid out for circular convolution on 2n - 1."""
    out = []
    for F, par in _newell_nodes(n, d):
        for a in range(3):  # the second difference 2 F(o) - F(o - 1) - F(o + 1), o = 0 .. n-1, node -1 by parity
            F = np.moveaxis(F, a, 0)
            lo = np.concatenate([par[a] * F[1:2], F[:-2]])
            F = np.moveaxis(2 * F[:-1] - lo - F[1:], 0, a)
        for a in range(3):  # offsets n-1 .. 1 mirrored behind 0 .. n-1
            F = np.moveaxis(F, a, 0)
            F = np.moveaxis(np.concatenate([F, par[a] * F[:0:-1]]), 0, a)
        out.append(F / (-4 * np.pi * d[0] * d[1] * d[2]))
    return out


def _open_demag(case, d, m):
    """K * m for an open lattice: m and the result as 3 arrays [x][y][z]."""
    n = (case["nx"], case["ny"], case["nz"])
    p = tuple(2 * v - 1 for v in n)
    K = [np.fft.rfftn(k) for k in _open_tensor(n, d)]
    S = [np.fft.rfftn(c, p) for c in m]
    row = [(0, 1, 2), (1, 3, 4), (2, 4, 5)]
    return [np.fft.irfftn(sum(K[i] * s for i, s in zip(r, S)), p)[:n[0], :n[1], :n[2]] for r in row]


def _grid(case, m):
    return [c.reshape(case["nz"], case["ny"], case["nx"]).transpose(2, 1, 0) for c in m]


def _flat(f):
    return np.stack([c.transpose(2, 1, 0).reshape(-1) for c in f])


def _shift(c, a, s, edge):
    """c at the neighbour along axis a (s = +-1) of an open lattice; beyond the edge: the cell itself or 0."""
    c = np.moveaxis(c, a, 0)
    pad = c[-1:] if s > 0 else c[:1]
    pad = pad if edge else np.zeros_like(pad)
    return np.moveaxis(np.concatenate([c[1:], pad]) if s > 0 else np.concatenate([pad, c[:-1]]), 0, a)


def exact(case, seed):
    """The demag field and the gradient of open lattices from Newell's formulas
    and the energy's definition in 64 bits; sweeps are chains of random
    decisions and have no such value."""
    seed = int(seed) % (1 << 40)
    if case["kind"] not in ("demag", "grad") or case["pbc"]:
        return None
    mat = FILM if case["material"] == "film" else SLAB
    d = (mat["dx"], mat["dy"], mat["dz"])
    dt = torch.float32 if case["precision"] == 32 else torch.float64
    if case["kind"] == "demag":
        m = _random_m(case["nx"] * case["ny"] * case["nz"], seed, dt).double().numpy()
        return _flat(_open_demag(case, d, _grid(case, m)))
    m = _grid(case, torch.from_numpy(_textured_m(case, seed)).to(dt).double().numpy())
    h = _open_demag(case, d, m)
    mu0, ms, V = 4e-7 * math.pi, mat["ms"], d[0] * d[1] * d[2]
    # every axis open: a missing neighbour bonds to nothing
    ex = [sum((_shift(c, a, s, True) - c) / d[a] ** 2 for a in range(3) for s in (1, -1)) for c in m]

    def diff(c, a):
        return (_shift(c, a, 1, False) - _shift(c, a, -1, False)) / (2 * d[a])

    dm = [diff(m[2], 0), diff(m[2], 1), -(diff(m[0], 0) + diff(m[1], 1))]
    u = (mat["anisUx"], mat["anisUy"], mat["anisUz"])
    B = (mat["Bextx"], mat["Bexty"], mat["Bextz"])
    mu = sum(u[k] * m[k] for k in range(3))
    g = [-2 * V * (mat["Aex"] * ex[k] + mat["Dind"] * dm[k] + mat["Ku1"] * mu * u[k]) - ms * V * B[k]
         - mu0 * ms * ms * V * h[k] for k in range(3)]
    dot = [float((m[k] * h[k]).sum()) for k in range(3)]
    avg = [float(c.sum()) for c in m]
    e_ex = V * sum(float(((_shift(c, a, 1, True) - c) ** 2).sum()) / d[a] ** 2 for c in m for a in range(3))
    e_dm = -V * sum(float((m[k] * dm[k]).sum()) for k in range(3))
    dms = -V * sum(B[k] * avg[k] for k in range(3)) - mu0 * ms * V * sum(dot)
    return {"dE_dm": _flat(g),
            "dE_dparams": [e_ex, e_dm, -V * float((mu * mu).sum()), dms] + [-ms * V * a for a in avg]}
