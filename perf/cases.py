"""The migration work that is timed: calls through the package's public entry points.

Each case is a dict of plain values; `prepare` makes what a user's program has in hand before
the call (a context with its geometry and Vrms, input traces), `run` is one call, `work` the
bytes and operations the call cannot do without, and `exact` the same result in 64 bits from
plain torch (masks as the operator defines them, in fp32; every value in fp64).

Kinds of call:
  device   Migrator.forward_device: traces and image in device memory (iterative solvers,
           pipelines that keep their cubes on the GPU)
  resident Migrator.forward_async on uploaded traces, fp32 or 16-bit storage, compensated or
           not (one upload, then repeated migrations)
  host     Migrator.forward_host: pinned host traces and Vrms in, image out, pipelined
  adjoint  Migrator.adjoint_device: demigration of an image in device memory
  lsm      Migrator.lsm_cg: least-squares migration, host in and out
  batch    Batch.run_async: velocity-scan panels over one cube and sub-volumes, one graph
  inline   MigrationKernel.kirchhoff_kernel_3d_with_padding: one output inline, host arrays
  job      SEG-Y records and a velocity table in, migrated image out (what one run of the
           command line does between its file reads and writes)
"""
import math

import numpy as np
import torch

from poststackmig3d_b200.migration import (Batch, MigrationKernel, Migrator, Problem,
                                           estimate_max_velocity, plan_geometry)

DEV = "cuda"

BASE = dict(dt=0.002, d_il=25.0, d_xl=25.0, angle=30.0, v0=2000.0, v1=2000.0, bump=0.0,
            amp=True, pad_il=0, pad_xl=0, precision="f32", compensated=False)


def _case(name=None, **kw):
    c = dict(BASE)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small target window, re-migrated interactively: launches and latency count
        _case("device_small", kind="device", n_il=31, n_xl=29, n_t=251, dt=0.004, pad_il=3,
              pad_xl=3, v0=1600.0, v1=2500.0, bump=0.05, angle=35.0),
        # one diffractor survey of 101 x 101 traces with 30 padded lines on every side, V const
        _case("device_padded", kind="device", n_il=101, n_xl=101, n_t=501, pad_il=30, pad_xl=30),
        # odd sizes, different bins along inline and crossline, no amplitude weight
        _case("device_ragged", kind="device", n_il=133, n_xl=87, n_t=733, d_il=25.0, d_xl=12.5,
              angle=40.0, v0=1600.0, v1=3100.0, bump=0.1, amp=False, pad_il=3, pad_xl=5),
        # a production cube: 401 x 401 traces, 2 s at 2 ms, Vrms 1500 -> 3500 m/s, 45 degrees
        _case("device_large", kind="device", n_il=401, n_xl=401, n_t=1001, angle=45.0,
              v0=1500.0, v1=3500.0, bump=0.05),
        # traces held in 16 bits (twice the cube per GPU), re-migrated from resident storage
        _case("resident_bf16", kind="resident", n_il=121, n_xl=121, n_t=876, angle=45.0,
              v0=1500.0, v1=3250.0, bump=0.05, precision="bf16"),
        # a whole call from pinned host memory and back, copies overlapped with the migration
        _case("host_cube", kind="host", n_il=151, n_xl=167, n_t=751, angle=40.0, v0=1500.0,
              v1=3000.0, bump=0.05),
        # demigration at the size of one least-squares iteration
        _case("adjoint_cube", kind="adjoint", n_il=101, n_xl=101, n_t=1001),
        # demigration of a padded image at odd sizes
        _case("adjoint_ragged", kind="adjoint", n_il=87, n_xl=64, n_t=417, d_xl=20.0, dt=0.004,
              angle=35.0, v0=1600.0, v1=2500.0, bump=0.1, pad_il=5, pad_xl=2),
        # a whole least-squares migration: 5 iterations of forward and adjoint
        _case("lsm_cube", kind="lsm", n_il=61, n_xl=61, n_t=501, iters=5),
        # a velocity scan: constant-velocity panels over one cube, and sub-volumes with a Vrms
        _case("batch_scan", kind="batch", n_il=101, n_xl=101, n_t=501, panels=8, subs=2,
              v0=1800.0, v1=3350.0),
        # the per-inline kernel of an existing host program, one output inline a call
        _case("inline_dropin", kind="inline", n_il=47, n_xl=101, n_t=501, v0=1800.0, v1=2400.0,
              pad_xl=4),
        # SEG-Y records (IBM floats) and 54 table points in, image out
        _case("job_segy", kind="job", n_il=81, n_xl=93, n_t=626, fmt=1, points=54, v0=1600.0,
              v1=2800.0, angle=35.0, pad_il=2, pad_xl=2),
    ]


def draw(rng):
    """One more case: sizes log-uniform over each kind's range, odd ones among them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["device", "device", "device", "resident", "resident", "host", "adjoint",
                       "adjoint", "lsm", "batch", "inline", "job"])
    top = {"device": (260, 1001), "resident": (160, 1001), "host": (180, 1001),
           "adjoint": (120, 1001), "lsm": (70, 501), "batch": (110, 601), "inline": (90, 901),
           "job": (110, 801)}[kind]
    v0 = rng.uniform(1500.0, 2200.0)
    const = rng.random() < 0.25
    c = _case(kind=kind, n_il=size(17, top[0]), n_xl=size(17, top[0]), n_t=size(101, top[1]),
              dt=rng.choice([0.002, 0.002, 0.004]), d_il=rng.choice([12.5, 20.0, 25.0]),
              d_xl=rng.choice([12.5, 20.0, 25.0]), angle=rng.uniform(20.0, 45.0), v0=v0,
              v1=v0 if const else rng.uniform(2400.0, 3500.0),
              bump=0.0 if const else rng.choice([0.0, 0.05, 0.1]), amp=rng.random() < 0.8,
              pad_il=rng.choice([0, 0, 3, 11]), pad_xl=rng.choice([0, 0, 2, 7]))
    if kind == "resident":
        c["precision"] = rng.choice(["f32", "bf16", "f16"])
        c["compensated"] = rng.random() < 0.5
    if kind == "lsm":
        c["iters"] = rng.randint(2, 5)
    if kind == "batch":
        c.update(panels=rng.randint(3, 10), subs=rng.randint(0, 3), pad_il=0, pad_xl=0)
    if kind == "job":
        c.update(fmt=rng.choice([1, 5]), points=rng.randint(6, 60))
    largest = work(listed()[3])["flops"]
    while work(c)["flops"] > 0.5 * largest:  # smaller bins reach more traces: shrink the cube
        c["n_il"] = max(17, int(c["n_il"] * 0.8))
        c["n_xl"] = max(17, int(c["n_xl"] * 0.8))
    return c


# --------------------------------------------------------------------------- inputs


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + 17)
    return g


def _traces(g, n_il, n_xl, n_t, dt, f=30.0):
    """Band-limited reflectivity: sparse +-1 events convolved with a Ricker, 5% noise."""
    half = int(1.5 / f / dt)
    t = torch.arange(-half, half + 1, device=DEV, dtype=torch.float32) * dt
    a = (math.pi * f * t) ** 2
    w = ((1 - 2 * a) * torch.exp(-a)).view(1, 1, -1)
    out = torch.empty((n_il, n_xl, n_t), device=DEV)
    for i in range(0, n_il, 32):  # in blocks of inlines: bounded temporaries
        n = min(32, n_il - i)
        e = torch.randn((n * n_xl, 1, n_t), device=DEV, generator=g)
        e = torch.where(e.abs() > 1.9, e, torch.zeros((), device=DEV))
        x = torch.nn.functional.conv1d(e, w, padding=half)
        x += 0.05 * torch.randn(x.shape, device=DEV, generator=g)
        out[i:i + n] = x.view(n, n_xl, n_t)
    return out


def _vrms(case, n_il, n_xl, n_t):
    """Vrms(t) from v0 to v1 over the record, times 1 + bump * a Gaussian 2 km wide."""
    t = torch.arange(n_t, device=DEV, dtype=torch.float64) / max(n_t - 1, 1)
    vt = case["v0"] + (case["v1"] - case["v0"]) * t
    il = (torch.arange(n_il, device=DEV, dtype=torch.float64) - (n_il - 1) / 2) * case["d_il"]
    xl = (torch.arange(n_xl, device=DEV, dtype=torch.float64) - (n_xl - 1) / 2) * case["d_xl"]
    lat = 1 + case["bump"] * torch.exp(-(il[:, None] ** 2 + xl[None, :] ** 2) / (2 * 2000.0 ** 2))
    out = torch.empty((n_il, n_xl, n_t), device=DEV)
    for i in range(0, n_il, 32):
        out[i:i + 32] = (lat[i:i + 32, :, None] * vt).float()
    return out


def _geometry(case, n_il, n_xl, n_t, max_v):
    import dataclasses
    g = plan_geometry(n_il, n_xl, n_t, case["dt"], case["d_il"], case["d_xl"], case["angle"],
                      max_v, case["pad_il"], case["pad_xl"], case["amp"],
                      precision=case["precision"])
    return dataclasses.replace(g, compensated=bool(case["compensated"]))


class _DeviceArray:
    """Device memory owned by the library, as torch reads it without a copy; the tensor keeps
    the owner alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape),
                                         "typestr": "<f4", "version": 2}


def _view(ptr, shape, owner):
    return torch.as_tensor(_DeviceArray(ptr, shape, owner), device=DEV)


def _table_points(case, seed):
    """(il, xl, time, v) rows of a velocity table over the cube's labels."""
    r = np.random.RandomState(seed % (2 ** 31))
    n = case["points"]
    t_max = (case["n_t"] - 1) * case["dt"]
    t = r.uniform(0.0, t_max, n)
    v = case["v0"] + (case["v1"] - case["v0"]) * t / t_max
    return [(int(a), int(b), float(np.round(tt, 3)), float(np.float32(vv)))
            for a, b, tt, vv in zip(r.randint(1, case["n_il"] + 1, n),
                                    r.randint(1, case["n_xl"] + 1, n), t, v)]


def _ibm_words(x):
    """float32 -> IBM System/360 single words (truncated fraction)."""
    a = np.abs(x.astype(np.float64))
    nz = a > 0
    e = np.zeros(a.shape, dtype=np.int64)
    e[nz] = np.floor(np.log2(a[nz]) / 4.0).astype(np.int64) + 1
    f = a / np.power(16.0, e)
    e = e + (f >= 1.0) - (nz & (f < 1.0 / 16.0))
    f = np.floor(a / np.power(16.0, e) * 16777216.0).astype(np.int64)
    w = ((x < 0).astype(np.int64) << 31) | ((e + 64) << 24) | f
    return np.where(nz, w, 0).astype(np.uint32)


def _ibm_values(w):
    """The values of IBM words, in 64 bits."""
    w = w.astype(np.int64)
    return np.where(w >> 31, -1.0, 1.0) * (w & 0xFFFFFF) / 16777216.0 * \
        np.power(16.0, ((w >> 24) & 0x7F) - 64.0)


def _job_inputs(case, seed):
    """Records in file order, their positions, the cube they decode to (fp32), table rows."""
    n_il, n_xl, n_t = case["n_il"], case["n_xl"], case["n_t"]
    d = _traces(_gen(seed), n_il, n_xl, n_t, case["dt"]).cpu().numpy().reshape(-1, n_t)
    if case["fmt"] == 1:
        words = _ibm_words(d)
        d = _ibm_values(words).astype(np.float32)
    else:
        words = d.view(np.uint32)
    rec = np.zeros((n_il * n_xl, 240 + 4 * n_t), dtype=np.uint8)
    rec[:, 240:] = words.astype(">u4").view(np.uint8).reshape(n_il * n_xl, 4 * n_t)
    order = np.random.RandomState(seed % (2 ** 31)).permutation(n_il * n_xl).astype(np.int32)
    return rec[order], order, d.reshape(n_il, n_xl, n_t), _table_points(case, seed)


def _batch_problems(case, seed):
    """Constant-velocity panels over one cube, then sub-volumes with their own Vrms cube:
    [(geometry, traces tensor, Vrms tensor or None, velocity)]."""
    n_il, n_xl, n_t = case["n_il"], case["n_xl"], case["n_t"]
    g = _gen(seed)
    cube = _traces(g, n_il, n_xl, n_t, case["dt"])
    out = []
    for k in range(case["panels"]):
        v = float(np.float32(case["v0"] + (case["v1"] - case["v0"]) * k
                             / max(case["panels"] - 1, 1)))
        out.append((_geometry(case, n_il, n_xl, n_t, v), cube, None, v))
    for k in range(case["subs"]):
        ni, nx, nt = n_il * (5 + 2 * k) // 12 + 1, n_xl * (9 - 2 * k) // 12 + 1, n_t * 3 // 4 + k
        v = _vrms(case, ni, nx, nt)
        out.append((_geometry(case, ni, nx, nt, estimate_max_velocity(v.cpu().numpy())),
                    _traces(g, ni, nx, nt, case["dt"]), v, 0.0))
    return out


def _inline_inputs(case, seed):
    """One output inline's buffer, velocity slice and positions, as the host driver makes
    them: n_il inlines around the output inline, n_xl real crosslines."""
    n_il, n_xl, n_t = case["n_il"], case["n_xl"], case["n_t"]
    buf = _traces(_gen(seed), n_il, n_xl, n_t, case["dt"])
    vel = _vrms(case, 1, n_xl, n_t)[0]
    return buf, vel, n_il // 2


# --------------------------------------------------------------------------- prepare, run


def prepare(case, seed):
    kind = case["kind"]
    n_il, n_xl, n_t = case["n_il"], case["n_xl"], case["n_t"]
    if kind == "inline":
        buf, vel, cur = _inline_inputs(case, seed)
        t0 = np.array([np.float32(i * case["dt"]) for i in range(n_t)], dtype=np.float32)
        g = _geometry(case, n_il, n_xl, n_t, case["v1"])
        return dict(kind=kind, args=(buf.cpu().numpy(), n_il, n_xl, n_t, vel.cpu().numpy(),
                                     np.empty((n_xl + 2 * case["pad_xl"], n_t), np.float32),
                                     np.arange(n_il, dtype=np.int32), None, cur,
                                     -case["pad_xl"], np.float32(case["dt"]), t0, g.tan2,
                                     case["d_il"], case["d_xl"], case["amp"]))
    m = Migrator(0)
    if kind == "batch":
        problems, hosts = [], {}
        for g, tr, vr, v in _batch_problems(case, seed):
            h = hosts.setdefault(id(tr), tr.cpu().numpy())  # panels share one host cube
            problems.append(Problem(g, h, None if vr is None else vr.cpu().numpy(), v))
        b = Batch(m, problems)
        b.autotune()
        images = [_view(b.image_device_ptr(i), (p.geom.n_oi, p.geom.n_ox, p.geom.n_t), (b, m))
                  for i, p in enumerate(problems)]
        return dict(kind=kind, b=b, m=m, images=images)
    if kind == "job":
        rec, pos, _, points = _job_inputs(case, seed)
        m.set_geometry(_geometry(case, n_il, n_xl, n_t, case["v1"]))
        return dict(kind=kind, m=m, rec=rec, pos=pos, points=points, fmt=case["fmt"],
                    il=np.arange(1, n_il + 1, dtype=np.int32),
                    xl=np.arange(1, n_xl + 1, dtype=np.int32),
                    out=np.empty(m.image_shape(), dtype=np.float32))
    gen = _gen(seed)
    vr = _vrms(case, n_il, n_xl, n_t).cpu().numpy()
    g = _geometry(case, n_il, n_xl, n_t, estimate_max_velocity(vr))
    m.set_geometry(g)
    s = dict(kind=kind, m=m)
    if kind == "adjoint":
        m.set_vrms(vr)
        s["img"] = _traces(gen, g.n_oi, g.n_ox, n_t, case["dt"])
        s["out"] = torch.empty((n_il, n_xl, n_t), device=DEV)
        return s
    d = _traces(gen, n_il, n_xl, n_t, case["dt"])
    if kind == "host":
        s["d"] = d.cpu().pin_memory()
        s["v"] = torch.from_numpy(vr).pin_memory()
        s["out"] = torch.empty(m.image_shape(), dtype=torch.float32).pin_memory()
        return s
    m.set_vrms(vr)
    if kind == "device":
        s["d"] = d
        s["out"] = torch.empty(m.image_shape(), device=DEV)
    elif kind == "resident":
        m.set_traces(d.cpu().numpy())
        s["out"] = _view(m.image_device_ptr(), m.image_shape(), m)
    else:
        s["d"] = d.cpu().numpy()
        s["iters"] = case["iters"]
    return s


def run(state):
    kind, m = state["kind"], state.get("m")
    if kind == "device":
        m.forward_device(state["d"].data_ptr(), state["out"].data_ptr())
        return state["out"]
    if kind == "resident":
        m.forward_async()
        return state["out"]
    if kind == "host":
        return m.forward_host(state["d"], state["v"], state["out"])
    if kind == "adjoint":
        m.adjoint_device(state["img"].data_ptr(), state["out"].data_ptr())
        return state["out"]
    if kind == "lsm":
        return m.lsm_cg(state["d"], state["iters"])
    if kind == "batch":
        state["b"].run_async()
        return state["images"]
    if kind == "inline":
        return MigrationKernel.kirchhoff_kernel_3d_with_padding(*state["args"])
    m.set_traces_segy(state["rec"], state["fmt"], state["pos"])
    m.set_vrms_table(state["points"], state["il"], state["xl"])
    return m.forward(state["out"])


# --------------------------------------------------------------------------- work


def _terms(case, n_il, n_xl, n_t, v0, v1, one_inline=False):
    """Summed samples: (output sample, input trace) pairs inside the aperture and the record,
    over the real output points, from the vertical velocity law at 48 times."""
    dt, t_max = case["dt"], (n_t - 1) * case["dt"]
    di = np.arange(-(n_il - 1), n_il)
    dk = np.arange(-(n_xl - 1), n_xl)
    if one_inline:
        di = np.arange(n_il) - n_il // 2
        wi = np.ones(len(di))
    else:
        wi = n_il - np.abs(di).astype(np.float64)
    r2 = ((di[:, None] * case["d_il"]) ** 2 + (dk[None, :] * case["d_xl"]) ** 2).ravel()
    w = (wi[:, None] * (n_xl - np.abs(dk))[None, :]).ravel()
    order = np.argsort(r2)
    r2, cum = r2[order], np.cumsum(w[order])
    tan2 = math.tan(math.radians(case["angle"])) ** 2
    total = 0.0
    m = min(48, n_t)
    for k in range(m):
        t = (k + 0.5) / m * t_max
        v = v0 + (v1 - v0) * t / t_max
        lim = min((v * t / 2) ** 2 * tan2, (t_max ** 2 - t ** 2) * v * v / 4)
        i = int(np.searchsorted(r2, lim, side="right"))
        total += (cum[i - 1] if i else 0.0) * n_t / m
    return total


def work(case):
    kind = case["kind"]
    n_il, n_xl, n_t = case["n_il"], case["n_xl"], case["n_t"]
    cube = 4.0 * n_il * n_xl * n_t
    image = 4.0 * (n_il + 2 * case["pad_il"]) * (n_xl + 2 * case["pad_xl"]) * n_t
    per = 10.0  # t^2, rsqrt, t/dt, floor and fraction, interpolation, weighted sum
    if kind == "batch":
        terms, nbytes = 0.0, cube
        for k in range(case["panels"]):
            v = case["v0"] + (case["v1"] - case["v0"]) * k / max(case["panels"] - 1, 1)
            terms += _terms(case, n_il, n_xl, n_t, v, v)
            nbytes += cube
        for k in range(case["subs"]):
            s = (n_il * (5 + 2 * k) // 12 + 1, n_xl * (9 - 2 * k) // 12 + 1, n_t * 3 // 4 + k)
            terms += _terms(case, *s, case["v0"], case["v1"])
            nbytes += 12.0 * s[0] * s[1] * s[2]
        return {"bytes": nbytes, "flops": per * terms}
    if kind == "inline":
        t = _terms(case, n_il, n_xl, n_t, case["v0"], case["v1"], one_inline=True)
        return {"bytes": cube + 8.0 * (n_xl + case["pad_xl"]) * n_t, "flops": per * t}
    t = _terms(case, n_il, n_xl, n_t, case["v0"], case["v1"])
    stored = cube / 2 if kind == "resident" and case["precision"] != "f32" else cube
    if kind == "lsm":
        it = case["iters"]
        return {"bytes": 2 * cube + image + it * (6 * cube + 4 * image),
                "flops": per * t * (2 * it + 1)}
    if kind == "job":
        return {"bytes": cube + image, "flops": per * t + 12.0 * case["points"] * cube / 4}
    return {"bytes": stored + cube + image, "flops": per * t}


# --------------------------------------------------------------------------- 64-bit values


def _operator(g, vrms):
    """Terms of the operator for every offset (inline, crossline) between output point and
    trace: yields (output slices, trace slices, lower index, fraction, weight)
    over the distinct output inlines.  Weight 0 where a mask drops the term; the masks are
    fp32, in the operator's order, the values fp64."""
    n_il, n_xl, n_t = g.n_il, g.n_xl, g.n_t
    f32, f64 = torch.float32, torch.float64
    t0 = torch.tensor(g.t0(), device=DEV)
    dt = np.float32(g.dt_seconds)
    inv_dt = torch.tensor(np.float32(1.0) / dt, device=DEV)
    tan2 = torch.tensor(np.float32(g.tan2), device=DEV)
    ntm1 = float(n_t - 1)
    v = vrms  # [n_il or 1][n_xl][n_t] fp32
    eps = torch.tensor(1e-10, dtype=f32, device=DEV).to(f64)
    f4 = (1.0 / (v.to(f64) * v.to(f64) + eps).to(f32)) * 4.0
    half = v * t0 * 0.5
    md2 = half * half * tan2
    md2 = torch.where((v >= 1e-5) & (t0 >= 1e-5), md2, torch.full_like(md2, -1.0))
    peak = md2.amax(dim=(0, 1)).cpu().numpy()  # largest aperture at each sample
    t0sq = t0 * t0
    reach = float(md2.max())
    reach_il = g.m_il + g.pad_il
    for di in range(-min(n_il - 1, reach_il), min(n_il - 1, reach_il) + 1):
        dx = np.float32(np.float32(di) * np.float32(g.d_il))
        dx2 = np.float32(dx * dx)
        if dx2 > reach:
            continue
        # output inlines c with trace inline c + di in the cube
        c0, c1 = max(0, -di), min(n_il, n_il - di)
        for dk in range(-(n_xl - 1), n_xl):
            dy = np.float32(np.float32(dk) * np.float32(g.d_xl))
            r2 = np.float32(np.float64(dy) * np.float64(dy) + np.float64(dx2))
            if r2 > reach:
                continue
            ok = np.nonzero(peak >= r2)[0]
            if not len(ok):
                continue
            a = int(ok[0])  # the shallowest sample any output point passes at
            x0, x1 = max(0, -dk), min(n_xl, n_xl - dk)
            sl = (slice(c0, c1), slice(x0, x1), slice(a, n_t))
            vv = v[sl]
            r = torch.tensor(r2, device=DEV)
            rad = (f4[sl].to(f64) * r.to(f64) + t0sq[a:].to(f64)).to(f32)
            keep = (r <= md2[sl]) & (torch.sqrt(rad) * inv_dt < ntm1)
            t = torch.sqrt(t0[a:].to(f64) ** 2 + 4.0 * r.to(f64) / (vv.to(f64) ** 2))
            s = t / float(dt)
            lo = torch.floor(s).clamp_(0, n_t - 2)
            w = 1.0 / (t * vv.to(f64) ** 2) if g.amp else torch.ones_like(t)
            w = torch.where(keep, w, torch.zeros_like(w))
            yield sl, (slice(c0 + di, c1 + di), slice(x0 + dk, x1 + dk)), lo.long(), s - lo, w


def _cost(g, vmax):
    """Elements the 64-bit evaluation touches."""
    rad = vmax * (g.n_t - 1) * g.dt_seconds / 2 * math.sqrt(g.tan2)
    ni = 2 * min(g.n_il - 1, rad / g.d_il, g.m_il + g.pad_il) + 1
    nk = 2 * min(g.n_xl - 1, rad / g.d_xl) + 1
    return 0.6 * ni * nk * g.n_il * g.n_xl * g.n_t


LIMIT = 5.0e11  # above this the 64-bit evaluation takes over about 20 seconds


def _expand(g, img):
    """Image of the distinct inlines -> output rows (padded inlines repeat the edge inline,
    padded crosslines are zero)."""
    out = torch.zeros((g.n_oi, g.n_ox, g.n_t), dtype=torch.float64, device=DEV)
    rows = torch.as_tensor(np.asarray(g.out_center), device=DEV, dtype=torch.long)
    out[:, g.pad_xl:g.pad_xl + g.n_xl] = img[rows]
    return out


def _fold(g, rows):
    """The transpose of _expand."""
    out = torch.zeros((g.n_il, g.n_xl, g.n_t), dtype=torch.float64, device=DEV)
    idx = torch.as_tensor(np.asarray(g.out_center), device=DEV, dtype=torch.long)
    return out.index_add_(0, idx, rows[:, g.pad_xl:g.pad_xl + g.n_xl].double())


def _forward64(g, data, vrms):
    """data fp64 [n_il][n_xl][n_t], vrms fp32 -> image fp64 of the distinct inlines."""
    img = torch.zeros((g.n_il, g.n_xl, g.n_t), dtype=torch.float64, device=DEV)
    for out, tr, lo, fr, w in _operator(g, vrms):
        d = data[tr]
        x = torch.gather(d, 2, lo)
        x = x + fr * (torch.gather(d, 2, lo + 1) - x)
        img[out] += torch.where(w > 0, x * w, torch.zeros_like(w))
    return img


def _adjoint64(g, img, vrms):
    data = torch.zeros((g.n_il, g.n_xl, g.n_t), dtype=torch.float64, device=DEV)
    for out, tr, lo, fr, w in _operator(g, vrms):
        c = torch.where(w > 0, img[out] * w, torch.zeros_like(w))
        d = data[tr]
        d.scatter_add_(2, lo, c * (1.0 - fr))
        d.scatter_add_(2, lo + 1, c * fr)
    return data


def _stored(d, precision):
    """The samples as 16-bit storage holds them: value / max|trace| rounded, times max."""
    if precision == "f32":
        return d.double()
    scale = d.abs().amax(dim=2, keepdim=True)
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    q = (d / scale).to(torch.bfloat16 if precision == "bf16" else torch.float16)
    return q.double() * scale.double()


def _table64(case, points):
    """Inverse-distance blend of the table points at every sample (fp64, then fp32: the
    velocity the operator is given)."""
    n_il, n_xl, n_t = case["n_il"], case["n_xl"], case["n_t"]
    il = torch.arange(1, n_il + 1, device=DEV, dtype=torch.float64)[:, None, None]
    xl = torch.arange(1, n_xl + 1, device=DEV, dtype=torch.float64)[None, :, None]
    t = torch.arange(n_t, device=DEV, dtype=torch.float64) * case["dt"]
    sv = torch.zeros((n_il, n_xl, n_t), device=DEV)
    sw = torch.zeros((n_il, n_xl, n_t), device=DEV)
    hit = torch.zeros((n_il, n_xl, n_t), dtype=torch.bool, device=DEV)
    hv = torch.zeros((n_il, n_xl, n_t), device=DEV)
    for p_il, p_xl, p_t, p_v in points:
        d = torch.sqrt((p_il - il) ** 2 + (p_xl - xl) ** 2 + (p_t - t) ** 2)
        w = 1.0 / (1.0 + d.float())
        sv += p_v * w
        sw += w
        new = (d < 1e-10) & ~hit
        hv = torch.where(new, torch.full_like(hv, p_v), hv)
        hit |= new
    return torch.where(hit, hv, sv / sw)


def exact(case, seed):
    kind = case["kind"]
    n_il, n_xl, n_t = case["n_il"], case["n_xl"], case["n_t"]
    if kind == "batch":
        out = []
        problems = _batch_problems(case, seed)
        if sum(_cost(g, v or case["v1"]) for g, _, _, v in problems) > LIMIT:
            return None
        for g, tr, vr, v in problems:
            if vr is None:
                vr = torch.full((g.n_il, g.n_xl, g.n_t), v, dtype=torch.float32, device=DEV)
            out.append(_expand(g, _forward64(g, tr.double(), vr)))
        return out
    if kind == "inline":
        buf, vel, cur = _inline_inputs(case, seed)
        g = _geometry(case, n_il, n_xl, n_t, case["v1"])
        g.m_il = n_il  # the whole buffer is read
        vr = vel[None].expand(n_il, n_xl, n_t)
        if _cost(g, case["v1"]) > LIMIT:
            return None
        img = _forward64(g, buf.double(), vr)[cur]
        out = torch.zeros((n_xl + 2 * case["pad_xl"], n_t), dtype=torch.float64, device=DEV)
        out[case["pad_xl"]:case["pad_xl"] + n_xl] = img
        return out.cpu()
    if kind == "job":
        _, _, d, points = _job_inputs(case, seed)
        g = _geometry(case, n_il, n_xl, n_t, case["v1"])
        if _cost(g, case["v1"]) > LIMIT:
            return None
        img = _forward64(g, torch.from_numpy(d).to(DEV).double(), _table64(case, points))
        return _expand(g, img).cpu()
    gen = _gen(seed)
    vr = _vrms(case, n_il, n_xl, n_t)
    g = _geometry(case, n_il, n_xl, n_t, estimate_max_velocity(vr.cpu().numpy()))
    passes = 2 * case["iters"] + 1 if kind == "lsm" else 1
    if passes * _cost(g, case["v1"] * (1 + case["bump"])) > LIMIT:
        return None
    if kind == "adjoint":
        img = _traces(gen, g.n_oi, g.n_ox, n_t, case["dt"])
        return _adjoint64(g, _fold(g, img), vr)
    d = _traces(gen, n_il, n_xl, n_t, case["dt"])
    if kind != "lsm":
        out = _expand(g, _forward64(g, _stored(d, case["precision"]), vr))
        return out.cpu() if kind == "host" else out
    # least squares: CG on min ||M^T m - d||, from m = 0
    r = d.double()
    hist = [float(r.norm())]
    s = _expand(g, _forward64(g, r, vr))
    m, p = torch.zeros_like(s), s
    gamma = float((s * s).sum())
    for _ in range(case["iters"]):
        q = _adjoint64(g, _fold(g, p), vr)
        delta = float((q * q).sum())
        alpha = gamma / delta if delta > 0 else 0.0
        m = m + alpha * p
        r = r - alpha * q
        hist.append(float(r.norm()))
        s = _expand(g, _forward64(g, r, vr))
        new = float((s * s).sum())
        p = s + (new / gamma if gamma > 0 else 0.0) * p
        gamma = new
    return m.cpu(), np.array(hist)
