"""The calls by which the framework's speed is followed, and their inputs.

What a program does with this framework is advance ARW states that live on
the GPU by whole large steps and bring the prognostic fields back: one domain
or an ensemble of uneven ones, in the plain FP32 form or with FP64 column
recursions, with periodic, walled or open sides, with few or many
positive-definite species, with the damping and diffusion options of the
namelist; a host model may also hand its state over at every step.  Each kind
is a case here, from a domain that one wave of blocks covers many times over
to one that needs tens of gigabytes.

The initial states follow wrf_gb300.cases (Weisman-Klemp supercell, f-plane
jet channel), built on the GPU: the horizontally uniform columns come from a
small case of that module, the perturbations are drawn from the seed, and
every column is put back into hydrostatic balance.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from wrf_gb300 import abi, cases
from wrf_gb300 import gpu as G

H = abi.HALO
DRY = ("u_2", "v_2", "w_2", "t_2", "ph_2", "mu_2", "p", "al")
ONES2 = ("msfux", "msfuy", "msfvx", "msfvx_inv", "msfvy", "msftx", "msfty", "cosa")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind="run", state="supercell", nx=64, ny=64, kde=41, scalars=0, steps=1, lateral="periodic", form="plain",
          options="none", members=1):
    return dict(kind=kind, state=state, nx=nx, ny=ny, kde=kde, scalars=scalars, steps=steps, lateral=lateral, form=form,
                options=options, members=members)


def listed():
    return [
        # one step of the smallest benchmark domain and its fields back: a
        # call whose cost is its launches and their latency
        dict(_case(nx=41, ny=41, kde=41, steps=1), name="step_41x41x41"),
        # ten steps of a small domain with many tracers, uneven in every direction
        dict(_case(nx=100, ny=70, kde=30, scalars=10, steps=10), name="run_100x70x30_s10"),
        # the tallest column the solver takes, narrow, with FP64 column recursions
        dict(_case(nx=75, ny=90, kde=128, scalars=2, steps=4, form="mixed"), name="run_75x90x128_mixed"),
        # a limited-area storm: open sides, w damping and the Rayleigh layer
        dict(_case(nx=190, ny=161, kde=60, scalars=3, steps=3, lateral="open", options="damp"), name="run_190x161x60_open"),
        # a rotating channel between walls with map factors, both diffusions and the implicit w damping
        dict(_case(state="channel", nx=160, ny=144, kde=64, scalars=1, steps=3, options="diffuse"),
             name="channel_160x144x64_diffuse"),
        # an ordinary storm run with tracers, on a quarter of the benchmark's area
        dict(_case(nx=256, ny=256, kde=80, scalars=10, steps=4), name="run_256x256x80_s10"),
        # the benchmark's own workload
        dict(_case(nx=512, ny=512, kde=80, scalars=10, steps=4), name="run_512x512x80_s10"),
        # the largest single domain: the jet channel, water vapour only
        dict(_case(state="channel", nx=1024, ny=1024, kde=96, steps=2), name="channel_1024x1024x96"),
        # an ensemble of uneven storms in the batched mixed form (sizes of the benchmark's ensemble)
        dict(_case(nx=256, ny=256, kde=80, scalars=3, steps=3, form="mixed", members=16), name="ensemble_16_mixed"),
        # an ensemble of many small domains, storms and channels, plain
        dict(_case(state="both", nx=96, ny=96, kde=60, scalars=7, steps=4, members=24), name="ensemble_24_small"),
        # a host time loop: every field over the link, one step, every field back, four times
        dict(_case(kind="loop", nx=256, ny=256, kde=80, scalars=10, steps=4), name="loop_256x256x80_s10"),
        # a device-resident caller's positive-definite transport of one field
        dict(_case(kind="pd", nx=231, ny=180, kde=64), name="pd_231x180x64"),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 7 + ["loop", "pd", "pd"])
    state = rng.choice(["supercell", "supercell", "channel"])
    lateral = rng.choice(["periodic", "periodic", "open", "openx"]) if state == "supercell" else "periodic"
    kde = _between(rng, 14, 128)
    if kind == "pd":
        # the entry point's limit is 8 Mi points, halo included
        nx = _between(rng, 16, 480)
        ny = _between(rng, 16, min(480, 7_500_000 // ((nx + 9) * kde) - 9))
        return _case(kind="pd", state=state, nx=nx, ny=ny, kde=kde)
    members = rng.choice([1, 1, 1, 1, 2, 5, 16]) if kind == "run" else 1
    scalars = rng.choice([0, 1, 2, 3, 4, 7, 10])
    # no more cells than the benchmark's domain with its eleven species
    cells = 16_000_000 // members if scalars > 4 else 20_000_000 // members
    nx = _between(rng, 16, 640)
    ny = max(16, min(_between(rng, 16, 640), cells // (nx * kde)))
    steps = max(1, min(rng.choice([1, 2, 4, 10]), 60_000_000 // (members * nx * ny * kde)))
    return _case(kind=kind, state=state, nx=nx, ny=ny, kde=kde, scalars=scalars, steps=steps, lateral=lateral,
                 form=rng.choice(["plain", "plain", "mixed"]), options=rng.choice(["none", "none", "none", "damp", "diffuse"]),
                 members=members)


# ---------------------------------------------------------------------------
# initial states
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _columns(state, ny, kde):
    """Balanced columns without perturbations: the description and 1-D fields
    of a small case, and its rows of theta, qv, u, v and dry mass."""
    rng = np.random.Generator(np.random.PCG64(1))
    if state == "channel":
        rows = 24  # the channel's rows at this many places; a row in between is interpolated
        small = cases.channel_state(8, rows, kde, 4000.0 * ny / rows, 20.0, 25000.0, rng, noise=0.0)
    else:
        rows = 8
        small = cases.supercell_state(8, rows, kde, 2000.0, 12.0, 20000.0, [], rng, noise=0.0)
    f = small.fields
    nk = kde - 1
    qv = small.species[0][0][H:H + rows, :nk, H]
    th = (f["t_1"][H:H + rows, :nk, H] + cases.T0) / (1.0 + (cases.R_V / cases.R_D) * qv) - cases.T0
    row = dict(th=th, qv=qv, u=f["u_1"][H:H + rows, :nk, H], v=f["v_1"][H:H + rows, :nk, H],
               mu=f["mu_1"][H:H + rows, H:H + 1])
    if state == "channel":
        at = (np.arange(ny) + 0.5) / ny * rows - 0.5
        for nm, a in row.items():
            row[nm] = np.stack([np.interp(at, np.arange(rows), a[:, k]) for k in range(a.shape[1])], axis=1)
    else:
        row = {nm: np.repeat(a[:1], ny, axis=0) for nm, a in row.items()}
    return small, row


def _index(n, mode, device):
    """Interior point (0-based) each memory point 1-4 .. n+1+4 holds initially."""
    p = torch.arange(-H, n + 1 + H, device=device)
    if mode == "periodic":
        return p % n
    if mode == "wall":
        p = torch.where(p < 0, -1 - p, p)
        return torch.where(p >= n, 2 * n - 1 - p, p).clamp(0, n - 1)
    return p.clamp(0, n - 1)


class _Member:
    """One domain: its description and its fields, float32 in memory layout."""

    def __init__(self, case, state, nx, ny, kde, seed):
        dev = torch.device("cuda")
        g = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 17)
        small, row = _columns(state, ny, kde)
        channel = state == "channel"
        dx, dt = (4000.0, 20.0) if channel else ((1000.0, 6.0) if nx * ny > 40000 else (2000.0, 12.0))
        self.desc = d = type(small.desc).from_buffer_copy(small.desc)
        d.ide, d.jde, d.kde, d.n_scalar = nx + 1, ny + 1, kde, case["scalars"]
        s, c = d.scalars, d.config
        s.dt, s.dx, s.dy, s.rdx, s.rdy = dt, dx, dx, 1.0 / dx, 1.0 / dx
        xmode, ymode = "periodic", "wall" if channel else "periodic"
        if case["lateral"] in ("open", "openx") and not channel:
            c.periodic_x, c.open_xs, c.open_xe = 0, 1, 1
            xmode = "open"
            if case["lateral"] == "open":
                c.periodic_y, c.open_ys, c.open_ye = 0, 1, 1
                ymode = "open"
        if case["options"] == "damp":
            c.w_damping, c.damp_opt, c.dampcoef, c.zdamp = 1, 2, 0.003, 5000.0
        if case["options"] == "diffuse":
            c.damp_opt, c.dampcoef, c.zdamp = 3, 0.2, 5000.0
            c.diff_6th_opt, c.diff_6th_factor = 2, 0.12
            c.diff_opt, c.km_opt, c.khdif, c.kvdif = 1, 1, 75.0, 5.0
        ix, iy = _index(nx, xmode, dev), _index(ny, ymode, dev)
        nk = kde - 1
        f1 = {nm: small.fields[nm] for nm in abi.F1D if nm in small.fields}
        col = {nm: torch.from_numpy(np.ascontiguousarray(small.fields[nm][H, :, H])).to(dev)
               for nm in ("phb", "pb", "alb", "t_init")}
        mub = float(small.fields["mub"][H, H])
        rows = {nm: torch.from_numpy(np.ascontiguousarray(a)).to(dev) for nm, a in row.items()}

        def rand(*shape):
            return torch.rand(*shape, generator=g, device=dev, dtype=torch.float64)

        th = rows["th"][:, :, None].expand(ny, nk, nx).clone()
        qv = rows["qv"][:, :, None].expand(ny, nk, nx)
        mu1 = rows["mu"].expand(ny, nx)
        z = 0.5 * (col["phb"][:-1] + col["phb"][1:]) / cases.G
        if channel:
            th += torch.where(z < 2000.0, 1.0, 0.0)[None, :, None] * (2.0 * rand(ny, nk, nx) - 1.0)
        else:
            xs = (torch.arange(nx, device=dev, dtype=torch.float64) + 0.5) * dx
            ys = (torch.arange(ny, device=dev, dtype=torch.float64) + 0.5) * dx
            at = rand(4, 3)
            for b in range(4 if nx * ny > 40000 else 1):
                r = torch.sqrt(((xs - at[b, 0] * nx * dx) / 1.0e4)[None, None, :] ** 2 +
                               ((ys - at[b, 1] * ny * dx) / 1.0e4)[:, None, None] ** 2 +
                               ((z - 1500.0) / 1500.0)[None, :, None] ** 2)
                th += torch.where(r <= 1.0, (1.0 + 3.0 * at[b, 2]) * torch.cos(0.5 * math.pi * r) ** 2, 0.0)
            th += 0.01 * (2.0 * rand(ny, nk, nx) - 1.0)
        ph, al, p = self._balance(f1, col, mub, mu1, th, qv, s.p_top, kde)
        tm = (th + cases.T0) * (1.0 + (cases.R_V / cases.R_D) * qv) - cases.T0
        del th

        def mem3(a):
            a = a.float()
            if a.shape[1] < kde:
                a = torch.cat([a, a.new_zeros(a.shape[0], kde - a.shape[1], a.shape[2])], dim=1)
            return a[iy][:, :, ix].contiguous()

        def wide(v):  # one column for the whole domain
            a = torch.zeros(kde, device=dev)
            a[:v.shape[0]] = v.float()
            return a[None, :, None].expand(ny + 1 + 2 * H, kde, nx + 1 + 2 * H).contiguous()

        def mem2(a):
            return a.float()[iy][:, ix].contiguous()

        self.fields = F = {}
        F["u_1"] = F["u_2"] = mem3(rows["u"][:, :, None].expand(ny, nk, nx))
        F["v_1"] = F["v_2"] = mem3(rows["v"][:, :, None].expand(ny, nk, nx))
        F["t_1"] = F["t_2"] = mem3(tm)
        F["ph_1"] = F["ph_2"] = mem3(ph)
        F["p"], F["al"] = mem3(p), mem3(al)
        F["alt"] = mem3(al + col["alb"][None, :nk, None])
        for nm in ("phb", "pb", "alb", "t_init"):
            F[nm] = wide(col[nm] if nm == "phb" else col[nm][:nk])
        F["mu_1"] = F["mu_2"] = mem2(mu1)
        F["mub"] = mem2(torch.full((ny, nx), mub, device=dev, dtype=torch.float64))
        msf = torch.ones(ny, nx, device=dev, dtype=torch.float64)
        if case["options"] == "diffuse":  # a smooth map scale factor that depends on the row
            msf += 0.02 * torch.cos(math.pi * (torch.arange(ny, device=dev) + 0.5) / ny)[:, None]
        for nm in ONES2:
            F[nm] = mem2(torch.ones_like(msf) if nm == "cosa" else 1.0 / msf if nm == "msfvx_inv" else msf)
        F["f"] = mem2(torch.full_like(msf, 1.0e-4 if channel else 0.0))
        for nm, a in f1.items():
            F[nm] = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32))
        self.species = [mem3(qv)]
        for _ in range(case["scalars"]):
            q = torch.randn(ny, nk, nx, generator=g, device=dev)
            self.species.append(mem3(1.0e-6 * torch.exp(q)))

    @staticmethod
    def _balance(f1, col, mub, mu1, th, qv, p_top, kde):
        """Geopotential in hydrostatic balance with theta, qv and the column's
        dry mass, then the specific volume and pressure that it gives
        (as wrf_gb300.cases does on the host)."""
        c1f, c2f, c1h, c2h = f1["c1f"], f1["c2f"], f1["c1h"], f1["c2h"]
        c3f, c4f, c3h, c4h = f1["c3f"], f1["c4f"], f1["c3h"], f1["c4h"]
        nk = kde - 1
        ny, _, nx = th.shape
        p = torch.zeros_like(th)
        al = torch.zeros_like(th)
        for k in range(nk - 1, -1, -1):
            qf = 0.5 * (qv[:, k] + qv[:, min(k + 1, nk - 1)])
            q2 = 1.0 / (1.0 + qf)
            load = (c1f[k + 1] * mu1 + qf * q2 * (c1f[k + 1] * mub + c2f[k + 1])) / q2
            p[:, k] = -0.5 * load / f1["rdnw"][k] if k == nk - 1 else p[:, k + 1] - load / f1["rdn"][k + 1]
            al[:, k] = (cases.R_D / cases.P1000) * (th[:, k] + cases.T0) * (1.0 + cases.RVOVRD * qv[:, k]) * (
                (p[:, k] + col["pb"][k]) / cases.P1000) ** cases.CVPM - col["alb"][k]
        ph = torch.zeros(ny, kde, nx, device=th.device, dtype=torch.float64)
        for k in range(nk):
            full = c1h[k] * mub + c2h[k] + c1h[k] * mu1
            ph[:, k + 1] = ph[:, k] - f1["dnw"][k] * (full * al[:, k] + c1h[k] * mu1 * col["alb"][k])
        mut = mub + mu1
        for k in range(nk):
            up = c3f[k + 1] * mut + c4f[k + 1] + p_top
            down = c3f[k] * mut + c4f[k] + p_top
            mid = c3h[k] * mut + c4h[k] + p_top
            alt = (ph[:, k + 1] - ph[:, k] + col["phb"][k + 1] - col["phb"][k]) / mid / torch.log(down / up)
            tm = (th[:, k] + cases.T0) * (1.0 + (cases.R_V / cases.R_D) * qv[:, k])
            al[:, k] = alt - col["alb"][k]
            p[:, k] = cases.P1000 * (cases.R_D * tm / (cases.P1000 * alt)) ** cases.CPOVCV - col["pb"][k]
        return ph, al, p


def _members(case, seed):
    """(state, nx, ny, kde, seed) of every member: one of the case's own size,
    or an uneven ensemble up to it."""
    if case["members"] == 1:
        state = "supercell" if case["state"] == "both" else case["state"]
        return [(state, case["nx"], case["ny"], case["kde"], seed)]
    rng = np.random.Generator(np.random.PCG64(case["members"]))
    out = []
    for m in range(case["members"]):
        nx = int(rng.integers(max(16, case["nx"] // 4), case["nx"] + 1))
        ny = int(rng.integers(max(16, case["ny"] // 4), case["ny"] + 1))
        kde = int(rng.integers(max(14, case["kde"] // 2), case["kde"] + 1))
        state = ("supercell", "channel")[int(rng.integers(0, 2))] if case["state"] == "both" else case["state"]
        out.append((state, nx, ny, kde, seed * 1000 + m))
    return out


class _Run:
    """A program's handle on a resident state and its page-locked host buffers."""

    def __init__(self, case, seed):
        self.steps, self.loop = case["steps"], case["kind"] == "loop"
        sizes = _members(case, seed)
        first = _Member(case, *sizes[0])
        descs = [first.desc]
        for state, nx, ny, kde, _ in sizes[1:]:
            d = type(first.desc).from_buffer_copy(_columns(state, ny, kde)[0].desc)
            descs.append(d)
        members = [first]
        # the descriptions of all members are needed before the first field is set
        for m in range(1, len(sizes)):
            members.append(_Member(case, *sizes[m]))
            descs[m] = members[m].desc
        self.dom = G.Ensemble(descs, flags=G.FLAG_MIXED if case["form"] == "mixed" else 0)
        self.out = {}
        for m, mem in enumerate(members):
            items = [(abi.FIELD_ID[nm], a) for nm, a in mem.fields.items()]
            for sp, q in enumerate(mem.species):
                items += [(abi.species_id(sp), q), (abi.species_id(sp, old=True), q)]
            staged, of = None, None
            for fid, a in items:
                if a is not of:
                    if staged is None or staged.numel() != a.numel():
                        staged = torch.empty(a.numel(), dtype=torch.float32, pin_memory=True)
                    staged.copy_(a.reshape(-1))
                    of = a
                self.dom.set(m, fid, staged.numpy())
            fids = [abi.FIELD_ID[nm] for nm in DRY] + [abi.species_id(sp) for sp in range(len(mem.species))]
            bufs = [torch.empty(self.dom.field_size(m, fid), dtype=torch.float32, pin_memory=True) for fid in fids]
            if self.loop:
                for fid, b in zip(fids, bufs):
                    b.copy_(torch.from_numpy(self.dom.get(m, fid)))
            outs = [b.numpy() for b in bufs]
            self.dom.bind_host_state(m, fids, outs if self.loop else [None] * len(outs), outs)
            # a run with many members gives back its leading ones' fields
            # whole through the same call; all are copied out
            self.out.update({"%d.%d" % (m, fid): b for fid, b in zip(fids, bufs) if len(self.out) < 60})
            members[m] = None

    def __call__(self):
        if self.loop:
            self.dom.step_host(self.steps)
        else:
            if self.steps > 1:
                self.dom.step(self.steps - 1)
            self.dom.step_host(1)
        return self.out


class _Pd:
    """Device arrays of a caller that transports one positive-definite field:
    a smooth mass-flux field, a log-normal tracer, and a tendency array."""

    def __init__(self, case, seed):
        nx, ny, kde = case["nx"], case["ny"], case["kde"]
        dev = torch.device("cuda")
        g = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 29)
        ymode = "wall" if case["state"] == "channel" else "periodic"
        small, _ = _columns("supercell", ny, kde)
        self.cfg = abi.default_config(True, ymode == "periodic", ymode == "wall")
        ix, iy = _index(nx, "periodic", dev), _index(ny, ymode, dev)
        nk = kde - 1

        def mem3(a, stag=""):
            full = torch.zeros(ny + 1 + 2 * H, kde, nx + 1 + 2 * H, device=dev)
            full[:, :a.shape[1]] = a.float()[iy][:, :, ix]
            if stag == "v" and ymode == "wall":  # no flow through the walls; mirrored with its sign behind them
                full[H], full[H + ny] = 0.0, 0.0
                for o in range(1, H + 1):
                    full[H - o], full[H + ny + o] = -full[H + o], -full[H + ny - o]
            return full.contiguous()

        self.dx, self.dt = 1000.0, 6.0
        mub = float(small.fields["mub"][H, H])
        q = 1.0e-6 * torch.exp(torch.randn(ny, nk, nx, generator=g, device=dev))
        q = torch.where(torch.rand(ny, nk, nx, generator=g, device=dev) < 0.2, torch.zeros_like(q), q)
        x = torch.arange(nx, device=dev) / nx
        y = torch.arange(ny, device=dev) / ny
        k = torch.arange(kde, device=dev) / nk
        a = torch.rand(6, generator=g, device=dev) * 6.28
        u = 20.0 * torch.sin(6.28 * y + a[0])[:, None, None] * torch.cos(3.0 * k[:nk] + a[1])[None, :, None] + \
            5.0 * torch.sin(6.28 * x + a[2])[None, None, :]
        v = 15.0 * torch.sin(6.28 * x + a[3])[None, None, :] * torch.cos(3.0 * k[:nk] + a[4])[None, :, None] * torch.ones_like(u)
        # eta velocity, zero at the model's bottom and top
        w = 2.0e-3 * torch.sin(3.14159265 * k)[None, :, None] * torch.sin(12.56 * x + a[5])[None, None, :] * \
            torch.cos(6.28 * y)[:, None, None]
        w[:, -1] = 0.0
        mu1 = 200.0 * torch.sin(6.28 * (x[None, :] + y[:, None]))

        def mem2(b):
            return b.float()[iy][:, ix].contiguous()

        self.a = A = {}
        A["q"] = mem3(q)
        A["q_old"] = mem3(q * (1.0 + 0.02 * torch.rand(ny, nk, nx, generator=g, device=dev)))
        A["ru"], A["rv"], A["rom"] = mem3(mub * u), mem3(mub * v, "v"), mem3(mub * w)
        A["mut"], A["mub"] = mem2(mub + mu1), mem2(torch.full((ny, nx), mub, device=dev))
        A["mu_old"] = mem2(mu1 + 2.0 * torch.cos(6.28 * x)[None, :])
        A["msftx"] = A["msfty"] = mem2(torch.ones(ny, nx, device=dev))
        for nm, key in (("c1", "c1h"), ("c2", "c2h"), ("fzm", "fnm"), ("fzp", "fnp"), ("rdzw", "rdnw")):
            A[nm] = torch.from_numpy(np.ascontiguousarray(small.fields[key], dtype=np.float32)).to(dev)
        self.tend = torch.zeros_like(A["q"])
        dims = [1, nx + 1, 1, ny + 1, 1, kde, 1 - H, nx + 1 + H, 1 - H, ny + 1 + H, 1, kde, 1, nx + 1, 1, ny + 1, 1, kde]
        self.keep = [C.c_float(1.0 / self.dx), C.c_float(1.0 / self.dx), C.c_float(self.dt)] + [C.c_int(d) for d in dims]
        ptr = [C.c_void_p(A[nm].data_ptr()) for nm in ("q", "q_old")] + [C.c_void_p(self.tend.data_ptr())]
        ptr += [C.c_void_p(A[nm].data_ptr()) for nm in ("ru", "rv", "rom", "c1", "c2", "mut", "mub", "mu_old")]
        ptr += [C.cast(C.pointer(self.cfg), C.c_void_p)]
        ptr += [C.c_void_p(A[nm].data_ptr()) for nm in ("msftx", "msfty", "fzm", "fzp")]
        ref = [C.cast(C.pointer(v), C.c_void_p) for v in self.keep]
        self.args = ptr + ref[:2] + [C.c_void_p(A["rdzw"].data_ptr())] + ref[2:]
        self.fn = G.load().wrfgpu_advect_scalar_pd_noalloc
        self.fn.restype = C.c_int
        self.fn.argtypes = [C.c_void_p] * (len(self.args) + 1)

    def __call__(self):
        self.tend.zero_()
        rc = self.fn(*self.args, C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise G.WrfGpuError("wrfgpu_advect_scalar_pd_noalloc failed: %d" % rc)
        return self.tend


def prepare(case, seed):
    return _Pd(case, seed) if case["kind"] == "pd" else _Run(case, seed)


def run(state):
    return state()


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its result in 64 bits
# ---------------------------------------------------------------------------
def work(case):
    if case["kind"] == "pd":
        pts = case["nx"] * case["ny"] * (case["kde"] - 1)
        # q, q_old, the three mass fluxes read, the tendency written (cleared by the caller, then accumulated)
        return {"bytes": 4.0 * 7 * pts, "flops": 170.0 * pts}
    cells = sum(nx * ny * (kde - 1) for _, nx, ny, kde, _ in _members(case, 1))
    nsp = 1 + case["scalars"]
    # a step reads the prognostic fields (u, v, w, theta, ph, p, al), the base
    # state (phb, pb, alb) and the species, and writes the prognostic fields,
    # their values one step back (5) and the species
    per_step = 4.0 * (7 + 3 + nsp + 7 + 5 + nsp)
    # three stages of five tendencies (about 100 each), the preparation and the
    # equation of state, seven acoustic steps (about 150 each); per species
    # three transports (about 60 each) and the limiter
    flops = 3 * (500 + 100) + 7 * 150 + nsp * (3 * 60 + 110)
    return {"bytes": per_step * cells * case["steps"], "flops": float(flops) * cells * case["steps"]}


def exact(case, seed):
    """The positive-definite transport in 64 bits.  A whole large step has no
    such value: restating the model's step is a second model, and p, al and w
    of any two roundings of it part by 1e-3 within a step (the adjustment of
    the initial state's top layers)."""
    if case["kind"] != "pd":
        return None
    s = _Pd(case, seed)
    A = {nm: a.double() for nm, a in s.a.items()}
    nx, ny, nk = case["nx"], case["ny"], case["kde"] - 1
    rd, dt = float(s.keep[0].value), s.dt
    q, qo, ru, rv, rom = A["q"][:, :nk], A["q_old"][:, :nk], A["ru"][:, :nk], A["rv"][:, :nk], A["rom"]
    c1, c2, rdzw = A["c1"][:nk, None], A["c2"][:nk, None], A["rdzw"][:nk, None]
    mass = c1 * A["mut"][:, None, :] + c2
    mass_old = c1 * (A["mub"] + A["mu_old"])[:, None, :] + c2

    def at(a, di=0, dj=0, xi=0, xj=0):
        """Cells 0 .. n+1 of both directions, moved by (di, dj), (xi, xj) longer."""
        return a[H - 1 + dj:H + 1 + ny + dj + xj, :, H - 1 + di:H + 1 + nx + di + xi]

    def upwind(lo, hi, cr):
        return 0.5 * torch.clamp(cr + cr.abs(), max=1.0) * lo + 0.5 * torch.clamp(cr - cr.abs(), min=-1.0) * hi

    def sign(v):
        return torch.where(torch.signbit(v), -1.0, 1.0).double()

    def faces(a_vel, axis):
        """Low-order flux and the rest of the fifth-order one at the lower face of every cell, and one face more."""
        sh = (lambda a, d: at(a, d, 0, 1, 0)) if axis == 2 else (lambda a, d: at(a, 0, d, 0, 1))
        vel, mu = sh(a_vel, 0), 0.5 * (sh(mass, 0) + sh(mass, -1))
        low = mu / (dt * rd) * upwind(sh(qo, -1), sh(qo, 0), vel * dt * rd / mu)
        m3, m2, m1, c, p1, p2 = (sh(q, d) for d in (-3, -2, -1, 0, 1, 2))
        high = 37.0 / 60.0 * (c + m1) - 2.0 / 15.0 * (p1 + m2) + 1.0 / 60.0 * (p2 + m3) - \
            sign(vel) / 60.0 * ((p2 - m3) - 5.0 * (p1 - m2) + 10.0 * (c - m1))
        return low, vel * high - low

    lx, hx = faces(ru, 2)
    ly, hy = faces(rv, 0)
    qc, qoc, mc, vel = at(q), at(qo), at(mass), at(rom)
    lz, hz = torch.zeros_like(vel), torch.zeros_like(vel)
    dz = 2.0 / (rdzw[1:] + rdzw[:-1])
    w, mu = vel[:, 1:nk], mc[:, 1:]
    lz[:, 1:nk] = mu * dz / dt * upwind(qoc[:, :-1], qoc[:, 1:], w * dt / dz / mu)
    hz[:, 1:nk] = w * (A["fzm"][1:nk, None] * qc[:, 1:] + A["fzp"][1:nk, None] * qc[:, :-1])
    w = vel[:, 2:nk - 1]
    hz[:, 2:nk - 1] = w * (7.0 / 12.0 * (qc[:, 2:-1] + qc[:, 1:-2]) - 1.0 / 12.0 * (qc[:, 3:] + qc[:, :-3]) +
                           sign(-w) / 12.0 * ((qc[:, 3:] - qc[:, :-3]) - 3.0 * (qc[:, 2:-1] - qc[:, 1:-2])))
    hz -= lz
    # what leaves a cell may not exceed what the low-order step leaves in it
    left = at(mass_old) * qoc - dt * (rd * (lx[:, :, 1:] - lx[:, :, :-1]) + rd * (ly[1:] - ly[:-1]) +
                                      rdzw * (lz[:, 1:] - lz[:, :-1]))
    out = dt * (rd * (hx[:, :, 1:].clamp(min=0) - hx[:, :, :-1].clamp(max=0)) +
                rd * (hy[1:].clamp(min=0) - hy[:-1].clamp(max=0)) +
                rdzw * (hz[:, 1:].clamp(max=0) - hz[:, :-1].clamp(min=0)))
    scale = torch.where(out > left, (left / (out + 1.0e-20)).clamp(min=0), 1.0)
    hx[:, :, 1:] *= torch.where(hx[:, :, 1:] > 0, scale, 1.0)
    hx[:, :, :-1] *= torch.where(hx[:, :, :-1] < 0, scale, 1.0)
    hy[1:] *= torch.where(hy[1:] > 0, scale, 1.0)
    hy[:-1] *= torch.where(hy[:-1] < 0, scale, 1.0)
    hz[:, 1:] *= torch.where(hz[:, 1:] < 0, scale, 1.0)
    hz[:, :-1] *= torch.where(hz[:, :-1] > 0, scale, 1.0)
    x, y, z = hx + lx, hy + ly, hz + lz
    tend = -rd * (x[:, :, 1:] - x[:, :, :-1]) - rd * (y[1:] - y[:-1]) - rdzw * (z[:, 1:] - z[:, :-1])
    whole = torch.zeros(s.tend.shape, dtype=torch.float64, device=tend.device)
    whole[H:H + ny, :nk, H:H + nx] = tend[1:-1, :, 1:-1]
    return whole
