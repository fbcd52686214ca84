"""Performance cases of the framework: what its users run, through the public Python entry points.

A case names an entry point ("what"), a geometry with its particle count, and the options that call takes:

* ``solve``: one right-hand side of a host-driven integrator -- set_states, solve, the rates read back -- as the drop-in
  class runs for the reference's own time stepper;
* ``rk4``: device-resident RK4 steps from a host state to a host state;
* ``batch``: RK4 steps of many ragged systems in one persistent launch per stage (graph-replayed);
* ``serve``: requests through the continuous-batching engine, submitted together and all fetched;
* ``noalloc``: the allocation-free solve on caller-owned device arrays;
* ``diagnose``: the conserved quantities of a running wake (FP64);
* ``columns`` / ``field``: the resolve path's influence-matrix columns, and one vorticity field (FP64).

Geometries are those of ``pawan_b200.geometry`` (single ring, coaxial ring pair, helical wake) and ``cloud``: particles
without spatial order and of mixed radii, which is what the workloads' tubes scramble into after a few steps, so that
every tile pair is a near one.  Particle counts are exact: a geometry made of whole stations is cut to ``n``.

Results of the FP32 pair path carry FP32 precision, and a program that asked for it keeps them as float32; results of
the FP64 paths are kept as float64.
"""
import math

import numpy as np
import torch

import pawan_b200 as pb
from pawan_b200 import geometry as g

_ctx = None


def _context():
    """One context for the whole program, as a user's program has."""
    global _ctx
    if _ctx is None:
        _ctx = pb.Context(0)
    return _ctx


# ------------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest system a host-driven time stepper solves: latency of the three calls
        dict(name="solve_ring_512", what="solve", geometry="ring", n=512, nu=0.0, precision="f32"),
        # the single-ring workload at its own size: ten device-resident steps
        dict(name="rk4_ring_2048", what="rk4", geometry="ring", n=2048, nu=0.0, precision="f32", steps=10, graph=False),
        # a scrambled wake with mixed radii and viscosity, an odd size: near tile pairs only
        dict(name="solve_cloud_20011", what="solve", geometry="cloud", n=20011, nu=1e-3, precision="f32"),
        # one right-hand side of the leapfrogging ring pair at its full size
        dict(name="solve_pair_131072", what="solve", geometry="pair", n=131072, nu=1e-4, precision="f32"),
        # the helical wake at its full size: four wakes, the largest configuration
        dict(name="solve_helix_262144", what="solve", geometry="helix", n=262144, nu=1e-3, precision="f32"),
        # ragged rings integrated together, graph-replayed
        dict(name="batch_48", what="batch", systems=48, lo=512, hi=16384, steps=2, graph=True),
        # serving: small and middling requests that arrive together
        dict(name="serve_24", what="serve", requests=24, lo=1024, hi=8192, steps=4),
        # FP64 for a run that is compared with the reference
        dict(name="solve_pair_16384_f64", what="solve", geometry="pair", n=16384, nu=1e-4, precision="f64"),
        # the Gaussian smoothing kernel
        dict(name="solve_pair_32000_gauss", what="solve", geometry="pair", n=32000, nu=1e-4, precision="f32",
             kernel="gaussian"),
        # the monitored quantities of a helical wake, taken every few steps of a run
        dict(name="diagnose_helix_65536", what="diagnose", geometry="helix", n=65536),
        # the influence matrix of the vring that is resolved by default: 25 columns, 3,950 particles
        dict(name="columns_25x3950", what="columns", geometry="ring", n=3950, columns=25),
        # an embedded caller that owns the device memory
        dict(name="noalloc_4096", what="noalloc", geometry="ring", n=4096, nu=1e-4),
    ]


def _size(rng, lo, hi):
    """Log-uniform, odd sizes among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["solve", "solve", "solve", "rk4", "rk4", "batch", "serve", "noalloc", "diagnose", "columns",
                       "field"])
    if what == "solve":
        precision = rng.choice(["f32", "f32", "f64"])
        kernel = rng.choice(["highorder", "highorder", "gaussian"])
        geometry = rng.choice(["ring", "pair", "helix", "cloud"])
        hi = {"ring": 32768, "pair": 131072, "helix": 262144, "cloud": 32768}[geometry]
        if precision == "f64" or kernel == "gaussian":
            hi = 32768
        return dict(what=what, geometry=geometry, n=_size(rng, 256, hi), nu=rng.choice([0.0, 1e-4, 1e-3]),
                    precision=precision, kernel=kernel)
    if what == "rk4":
        n = _size(rng, 512, 32768)
        return dict(what=what, geometry=rng.choice(["ring", "helix"]), n=n, nu=rng.choice([0.0, 1e-3]),
                    precision="f32", steps=rng.choice([1, 2, 4]), graph=rng.choice([False, True]))
    if what == "batch":
        return dict(what=what, systems=rng.randint(12, 48), lo=512, hi=_size(rng, 2048, 16384),
                    steps=rng.choice([1, 2]), graph=rng.choice([False, True]))
    if what == "serve":
        return dict(what=what, requests=rng.randint(4, 24), lo=1024, hi=_size(rng, 2048, 8192),
                    steps=rng.choice([2, 3, 4]))
    if what == "noalloc":
        return dict(what=what, geometry=rng.choice(["ring", "pair"]), n=_size(rng, 256, 16384),
                    nu=rng.choice([0.0, 1e-4]))
    if what == "diagnose":
        return dict(what=what, geometry="helix", n=_size(rng, 2048, 131072))
    if what == "columns":
        return dict(what=what, geometry=rng.choice(["ring", "pair"]), n=_size(rng, 1000, 12000),
                    columns=rng.choice([9, 25, 49, 121]))
    return dict(what=what, geometry=rng.choice(["ring", "helix", "cloud"]), n=_size(rng, 1000, 65536))


# ---------------------------------------------------------------------- inputs

def _particles(geometry, n, seed):
    """counts per wake and the union's (pos, vor, rad, vol), exactly n particles."""
    if geometry == "cloud":
        rng = np.random.default_rng(seed)
        counts = [n // 3, n // 5, n - n // 3 - n // 5]
        return counts, (rng.uniform(-1, 1, (n, 3)), rng.normal(0, 0.01, (n, 3)), rng.uniform(0.05, 0.2, n),
                        rng.uniform(1e-4, 2e-4, n))
    stations = {"ring": 1, "pair": 2, "helix": 4}[geometry] * g.N_CORE
    per = -(-n // stations)
    if geometry == "ring":
        sc = g.single_ring(n_stations=per, seed=seed)
    elif geometry == "pair":
        sc = g.ring_pair(n_stations=per, seed=seed)
    else:
        sc = g.helical_wake(n_stations=per, seed=seed)
    counts = list(sc.counts)
    counts[-1] -= sc.n - n
    return counts, tuple(np.ascontiguousarray(a[:n]) for a in sc.union())


def _batch(case, seed):
    scs = g.ragged_batch(n_solves=case["systems"], seed=11, n_lo=case["lo"], n_hi=case["hi"])
    rng = np.random.default_rng(seed)  # the sizes and rings of one batch; the seed moves every particle
    out = []
    for sc in scs:
        pos, vor, rad, vol = sc.union()
        out.append((sc.counts, (pos + rng.uniform(-g.JITTER, g.JITTER, pos.shape), vor, rad, vol), sc.nu, sc.dt))
    return out


def _requests(case, seed):
    rng = np.random.default_rng(13)  # the sizes of the requests; the seed moves their particles
    out = []
    for k in range(case["requests"]):
        n = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append((*_particles("pair" if k % 2 else "ring", n, seed * 1000 + k), 1e-4, 0.005))
    return out


def prepare(case, seed):
    what = case["what"]
    st = dict(case=case)
    if what == "noalloc":
        _, arrays = _particles(case["geometry"], case["n"], seed)
        st["arrays"] = [torch.from_numpy(a).cuda() for a in arrays]
        st["out"] = torch.empty((2, case["n"], 3), dtype=torch.float64, device="cuda")
        return st
    ctx = _context()
    if what == "batch":
        st["systems"], st["states"], st["dt"] = [], [], []
        for counts, arrays, nu, dt in _batch(case, seed):
            s = pb.System(ctx, counts, nu, "f32")
            s.set_particles(*arrays)
            s.checkpoint()
            st["systems"].append(s)
            st["dt"].append(dt)
        st["batch"] = pb.Batch(ctx, st["systems"])
        return st
    if what == "serve":
        st["requests"] = _requests(case, seed)
        st["server"] = pb.Server(ctx, budget_bytes=16 << 30)
        return st
    counts, arrays = _particles(case["geometry"], case["n"], seed)
    s = pb.System(ctx, counts, case.get("nu", 0.0), case.get("precision", "f32"))
    if case.get("kernel", "highorder") != "highorder":
        s.set_kernel(case["kernel"])
    s.set_particles(*arrays)
    st["system"] = s
    st["state"] = pb.union_to_state(counts, arrays[0], arrays[1])
    if what == "columns":
        st["alpha"] = np.random.default_rng(seed).standard_normal((case["columns"], case["n"], 3))
    return st


def _kept(case, a):
    return a.astype(np.float32) if case.get("precision", "f32") == "f32" else a


# ------------------------------------------------------------------- one pass

def run(st):
    case = st["case"]
    what = case["what"]
    if what == "solve":
        s = st["system"]
        s.set_states(st["state"])
        s.solve()
        rates = [s.wake_rates(w) for w in range(len(s.counts))]
        return {"velocity": [_kept(case, u) for u, _ in rates], "retvorcity": [_kept(case, da) for _, da in rates]}
    if what == "rk4":
        s = st["system"]
        s.set_states(st["state"])
        s.rk4({"ring": 0.01, "pair": 0.005, "helix": 0.002}[case["geometry"]], case["steps"], use_graph=case["graph"])
        return {"state": _kept(case, s.get_states())}
    if what == "batch":
        for s in st["systems"]:
            s.restore()
        st["batch"].rk4(st["dt"], case["steps"], use_graph=case["graph"])
        return {"states": [_kept(case, s.get_states()) for s in st["systems"]]}
    if what == "serve":
        srv = st["server"]
        ids = []
        for counts, arrays, nu, dt in st["requests"]:
            status, rid = srv.submit(counts, *arrays, nu, dt, case["steps"])
            if status:
                raise RuntimeError("request not accepted: status %d" % status)
            ids.append(rid)
        for rid in ids:
            srv.wait(rid)
        return {"states": [_kept(case, srv.fetch(rid)[0]) for rid in ids]}
    if what == "noalloc":
        pos, vor, rad, vol = st["arrays"]
        out = st["out"]
        status = pb.interact_noalloc(pos.data_ptr(), vor.data_ptr(), rad.data_ptr(), vol.data_ptr(), case["n"],
                                     case["nu"], out[0].data_ptr(), out[1].data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
        if status:
            raise RuntimeError("status %d" % status)
        kept = out.float()
        return {"velocity": kept[0], "retvorcity": kept[1]}
    if what == "diagnose":
        return st["system"].diagnose()
    if what == "columns":
        return {"fields": st["system"].influence_columns(st["alpha"])}
    return {"field": st["system"].influence()}


# ------------------------------------------------ what a pass cannot do without

def _sizes(case):
    if case["what"] == "batch":
        return [sc.n for sc in g.ragged_batch(n_solves=case["systems"], seed=11, n_lo=case["lo"], n_hi=case["hi"])]
    if case["what"] == "serve":
        rng = np.random.default_rng(13)
        return [int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
                for _ in range(case["requests"])]
    return [case["n"]]


def work(case):
    """Bytes: inputs and outputs once, in the caller's FP64.  Operations: the framework's own counts per interaction
    (96 with diffusion, 79 without), about 40 per ordered pair of the diagnostics, 20 per pair and 6 per column of the
    vorticity field."""
    what, sizes = case["what"], _sizes(case)
    n, n2 = sum(sizes), float(sum(s * s for s in sizes))
    if what == "diagnose":
        return {"bytes": 64.0 * n, "flops": 40.0 * n2}
    if what in ("columns", "field"):
        c = case.get("columns", 1)
        return {"bytes": (32.0 + 48.0 * c) * n, "flops": n2 * (20.0 + 6.0 * c)}
    per = 79.0 if case.get("nu", 1e-4) == 0.0 else 96.0
    return {"bytes": 112.0 * n, "flops": n2 * per * (4 * case.get("steps", 1) if what in ("rk4", "batch", "serve") else 1)}


# ------------------------------------------------------------- in 64 bits, plainly

_PAIRS = 1 << 24  # pairs in flight


def _tensors(arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).to("cuda" if torch.cuda.is_available() else "cpu")
            for a in arrays]


def _blocks(n):
    step = max(1, _PAIRS // n)
    for lo in range(0, n, step):
        yield lo, min(n, lo + step)


def _rates(pos, vor, rad, vol, nu, kernel="highorder"):
    """Velocity and vorticity rate of every particle: the smoothed Biot-Savart velocity, vortex stretching and particle
    strength exchange, summed over all other particles."""
    n = pos.shape[0]
    u, da = torch.empty_like(pos), torch.empty_like(pos)
    for lo, hi in _blocks(n):
        d = [pos[lo:hi, None, k] - pos[None, :, k] for k in range(3)]
        r2 = d[0] * d[0]
        r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        own = torch.arange(lo, hi, device=pos.device)
        r2[own - lo, own] = 1.0
        sig2 = 0.5 * (rad[lo:hi, None] ** 2 + rad[None, :] ** 2)
        rb2 = r2 / sig2
        sig3 = sig2 * sig2.sqrt()
        rb = rb2.sqrt()
        if kernel == "gaussian":
            z = torch.exp(-0.5 * rb2) / sig3 / (2 * math.pi) ** 1.5
            phi = torch.special.erf(rb * math.sqrt(0.5)) / (4 * math.pi) / sig3
        else:
            w = rb2 + 1.0
            w2 = w * w
            phi = (rb2 + 1.5) / w2 / sig3 / (4 * math.pi)
            z = 1.875 / math.pi / (w2 * w2 * w2 * w * w.sqrt()) / sig3
            del w, w2
        del sig3
        q = (phi / rb - z) / rb2
        del phi, rb, rb2
        f = (z - 3 * q) / r2
        e = z.mul_(2 * nu) / sig2
        del r2, sig2
        for m in (q, f, e):
            m[own - lo, own] = 0.0
        a, b = [vor[lo:hi, None, k] for k in range(3)], [vor[None, :, k] for k in range(3)]
        c = [a[(k + 1) % 3] * b[(k + 2) % 3] - a[(k + 2) % 3] * b[(k + 1) % 3] for k in range(3)]  # alpha_i x alpha_j
        t = d[0] * c[0]
        t.addcmul_(d[1], c[1]).addcmul_(d[2], c[2]).mul_(f)
        for k in range(3):
            i, j = (k + 1) % 3, (k + 2) % 3
            u[lo:hi, k] = (q * (b[i] * d[j] - b[j] * d[i])).sum(1)
            da[lo:hi, k] = (q * c[k]).addcmul_(t, d[k]).sum(1)
        if nu != 0.0:
            da[lo:hi] += vol[lo:hi, None] * (e @ vor) - vor[lo:hi] * (e @ vol)[:, None]
    return u, da


def _steps(arrays, nu, dt, steps):
    x, a, rad, vol = arrays
    for _ in range(steps):
        k1 = _rates(x, a, rad, vol, nu)
        k2 = _rates(x + k1[0] * (0.5 * dt), a + k1[1] * (0.5 * dt), rad, vol, nu)
        k3 = _rates(x + k2[0] * (0.5 * dt), a + k2[1] * (0.5 * dt), rad, vol, nu)
        k4 = _rates(x + k3[0] * dt, a + k3[1] * dt, rad, vol, nu)
        x = x + (k1[0] + 2 * k2[0] + 2 * k3[0] + k4[0]) * (dt / 6)
        a = a + (k1[1] + 2 * k2[1] + 2 * k3[1] + k4[1]) * (dt / 6)
    return x.cpu().numpy(), a.cpu().numpy()


def _fields(pos, rad, alpha):
    """alpha: (C, N, 3); the smoothed vorticity field of each column."""
    n, c = pos.shape[0], alpha.shape[0]
    cols = alpha.permute(1, 0, 2).reshape(n, 3 * c).contiguous()
    out = torch.empty_like(cols)
    for lo, hi in _blocks(n):
        r2 = sum((pos[lo:hi, None, k] - pos[None, :, k]) ** 2 for k in range(3))
        sig2 = 0.5 * (rad[lo:hi, None] ** 2 + rad[None, :] ** 2)
        z = (1.875 / math.pi) * (r2 / sig2 + 1.0) ** -7.5 / (sig2 * sig2.sqrt())
        out[lo:hi] = z @ cols
    return out.reshape(n, c, 3).permute(1, 0, 2).contiguous()


def _diagnostics(pos, vor, rad):
    a2 = (vor * vor).sum(1)
    rxa = torch.linalg.cross(pos, vor)
    ens = (5 / (4 * math.pi) * a2 / rad ** 3).sum()
    hel = torch.zeros_like(ens)
    n = pos.shape[0]
    for lo, hi in _blocks(n):
        x = [pos[None, :, k] - pos[lo:hi, None, k] for k in range(3)]
        r2 = x[0] * x[0]
        r2.addcmul_(x[1], x[1]).addcmul_(x[2], x[2])
        own = torch.arange(lo, hi, device=pos.device)
        r2[own - lo, own] = 1.0
        sig2 = 0.5 * (rad[lo:hi, None] ** 2 + rad[None, :] ** 2)
        a, b = [vor[lo:hi, None, k] for k in range(3)], [vor[None, :, k] for k in range(3)]
        w = (r2 + sig2) ** -3.5 / (8 * math.pi)
        e = w * (10 * sig2 * sig2 - 2 * r2 * r2 - 7 * sig2 * r2) * sum(a[k] * b[k] for k in range(3))
        e -= 15 * w * r2 * sum(a[k] * x[k] for k in range(3)) * sum(b[k] * x[k] for k in range(3))
        e[own - lo, own] = 0.0
        ens += e.sum()
        rb2 = r2 / sig2
        sig3 = sig2 * sig2.sqrt()
        z = (1.875 / math.pi) * (rb2 + 1.0) ** -7.5 / sig3
        q = ((rb2 + 1.5) / (rb2 + 1.0) ** 2 / sig3 / (4 * math.pi) / rb2.sqrt() - z) / rb2
        h = q * sum(x[k] * (a[(k + 1) % 3] * b[(k + 2) % 3] - a[(k + 2) % 3] * b[(k + 1) % 3]) for k in range(3))
        h[own - lo, own] = 0.0
        hel += h.sum()
    return {"total_vorticity": vor.sum(0).cpu().numpy(), "linear_impulse": (0.5 * rxa.sum(0)).cpu().numpy(),
            "angular_impulse": (torch.linalg.cross(pos, rxa).sum(0) / 3).cpu().numpy(), "enstrophy": float(ens),
            "helicity": float(hel)}


def exact(case, seed):
    what = case["what"]
    if what in ("batch", "serve"):
        states = []
        for counts, arrays, nu, dt in (_batch(case, seed) if what == "batch" else _requests(case, seed)):
            states.append(_state_vector(counts, *_steps(_tensors(arrays), nu, dt, case["steps"])))
        return {"states": states}
    counts, arrays = _particles(case["geometry"], case["n"], seed)
    pos, vor, rad, vol = _tensors(arrays)
    if what == "rk4":
        dt = {"ring": 0.01, "pair": 0.005, "helix": 0.002}[case["geometry"]]
        return {"state": _state_vector(counts, *_steps((pos, vor, rad, vol), case["nu"], dt, case["steps"]))}
    if what in ("solve", "noalloc"):
        u, da = (a.cpu().numpy() for a in _rates(pos, vor, rad, vol, case["nu"], case.get("kernel", "highorder")))
        if what == "noalloc":
            return {"velocity": u, "retvorcity": da}
        cut = np.cumsum(counts)[:-1]  # per wake
        return {"velocity": np.split(u, cut), "retvorcity": np.split(da, cut)}
    if what == "diagnose":
        return _diagnostics(pos, vor, rad)
    if what == "columns":
        alpha = np.random.default_rng(seed).standard_normal((case["columns"], case["n"], 3))
        return {"fields": _fields(pos, rad, _tensors([alpha])[0]).cpu().numpy()}
    return {"field": _fields(pos, rad, vor[None])[0].cpu().numpy()}


def _state_vector(counts, pos, vor):
    """Union arrays as a state vector: per wake, positions then strengths."""
    out, o = [], 0
    for c in counts:
        out += [pos[o:o + c].ravel(), vor[o:o + c].ravel()]
        o += c
    return np.concatenate(out)
