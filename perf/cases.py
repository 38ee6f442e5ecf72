"""Performance cases of the lattice-Boltzmann step library: the work its users have it do.

Each case is one call pattern of the public interface over a state that a program keeps between
calls (a level, a hierarchy, a batch or an octree): ``prepare`` builds that state from a seed,
``run`` advances it by the case's steps, ``exact`` gives the same state in 64-bit arithmetic from
the equations alone. Sizes are those of this repository's configurations, tests and benchmark, or
generic ones between them.

Families (the ``kind`` of a case):

* ``box``      periodic box of the D3Q27 cumulant operator (decaying turbulence, Taylor-Green);
* ``channel``  sphere channel: velocity inlet, zero-gradient outlet, lateral mirrors, half-way
               walls, the FP64 drag of every step; optionally the spectral-viscosity filter;
* ``arrays``   the same channel stepped on caller-owned arrays in the reference's layout;
* ``batch``    many periodic boxes of uneven size stepped together, then read back;
* ``amr``      two-level block refinement around the sphere of a channel;
* ``kbc_box``, ``kbc_channel``  the D3Q39 entropic operator;
* ``oct_box``, ``oct_wing``     the D3Q19 octree operator, one periodic level or a wing on levels.
"""
import ctypes as C
import math

import numpy as np
import torch

from openaerolab_alpha_01_b200 import _capi as capi
from openaerolab_alpha_01_b200 import octree
from openaerolab_alpha_01_b200.amr import Hierarchy, blocks_in_box, refine
from openaerolab_alpha_01_b200.solver import (Batch, Geometry, Level, apply_analytic_sphere_obstacle, build_box,
                                              default_entropic_params, default_step_params)

ITEM = {"f16": 2, "bf16": 2, "f32": 4, "f64": 8}


def listed():
    return [
        # a small periodic box stepped call by call, as an interactive or coupled program does
        dict(name="box_small", kind="box", n=16, storage="f32", steps=4, c_wale=0.0, graph=False),
        # the 64^3 double-precision Taylor-Green accuracy run
        dict(name="box_f64", kind="box", n=64, storage="f64", steps=10, c_wale=0.2, graph=True),
        # the standard sphere channel, stepped with the drag of each step read by a monitor
        dict(name="channel_f16", kind="channel", nx=256, ny=128, nz=128, storage="f16", steps=5, graph=False, svv=0.0),
        # a channel of odd block counts in FP32, an odd count of steps as one call
        dict(name="channel_f32", kind="channel", nx=200, ny=88, nz=104, storage="f32", steps=5, graph=True, svv=0.0),
        # the channel with the spectral-viscosity filter of the reference's fine levels
        dict(name="channel_svv", kind="channel", nx=256, ny=128, nz=128, storage="f16", steps=2, graph=True, svv=0.004),
        # the drop-in call: a host program's own arrays in the reference's layout
        dict(name="arrays_f32", kind="arrays", nx=192, ny=96, nz=96, storage="f32", steps=2),
        # a parameter sweep of uneven boxes advanced together, the fields read at the end
        dict(name="batch_f16", kind="batch", members=16, n_min=16, n_max=64, storage="f16", steps=200),
        # two-level refinement around the sphere
        dict(name="amr_f16", kind="amr", nx=256, ny=128, nz=128, storage="f16", steps=2),
        # the entropic operator on a periodic box and on a channel
        dict(name="kbc_box", kind="kbc_box", n=96, steps=2),
        dict(name="kbc_channel", kind="kbc_channel", nx=96, ny=48, nz=56, steps=2),
        # the octree operator: a large periodic level, and a wing section on three levels
        dict(name="oct_box_f32", kind="oct_box", n0=192, n1=192, n2=192, precision="f32", steps=2),
        dict(name="oct_wing", kind="oct_wing", chord=128, precision="f32", steps=4),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["box", "box", "channel", "channel", "arrays", "batch", "amr", "kbc_box", "kbc_channel",
                       "oct_box", "oct_box", "oct_wing"])
    edge = lambda lo, hi: 8 * max(lo // 8, round(_log(rng, lo, hi) / 8))  # noqa: E731
    if kind == "box":
        n = edge(16, 128)
        return dict(kind=kind, n=n, storage=rng.choice(["f32", "f64", "f16", "bf16"]), steps=rng.randint(1, 12),
                    c_wale=rng.choice([0.0, 0.2]), graph=rng.random() < 0.5)
    if kind in ("channel", "arrays"):
        ny, nz = edge(40, 128), edge(40, 128)
        case = dict(kind=kind, nx=edge(64, 256), ny=ny, nz=nz, steps=rng.randint(1, 4))
        if kind == "arrays":
            case["storage"] = rng.choice(["f32", "f64"])
            return case
        case.update(storage=rng.choice(["f16", "f32", "bf16"]), graph=rng.random() < 0.5,
                    svv=rng.choice([0.0, 0.0, 0.0, 0.004]))
        return case
    if kind == "batch":
        return dict(kind=kind, members=rng.randint(3, 16), n_min=16, n_max=edge(24, 64),
                    storage=rng.choice(["f16", "f32"]), steps=round(_log(rng, 10, 200)))
    if kind == "amr":
        return dict(kind=kind, nx=edge(96, 256), ny=edge(64, 128), nz=edge(64, 128),
                    storage=rng.choice(["f16", "f32", "f64"]), steps=rng.randint(1, 3))
    if kind == "kbc_box":
        return dict(kind=kind, n=edge(16, 96), steps=rng.randint(1, 2))
    if kind == "kbc_channel":
        return dict(kind=kind, nx=edge(48, 96), ny=edge(32, 56), nz=edge(32, 56), steps=rng.randint(1, 3))
    if kind == "oct_box":
        even = lambda: 2 * round(_log(rng, 24, 192) / 2)  # noqa: E731
        return dict(kind=kind, n0=even(), n1=even(), n2=even(), precision=rng.choice(["f32", "f64"]),
                    steps=rng.randint(1, 4))
    return dict(kind=kind, chord=rng.choice([48, 64, 96, 128]), precision=rng.choice(["f32", "f64"]),
                steps=rng.randint(1, 4))


# ---- inputs ----------------------------------------------------------------------------------
def _modes(seed, count=6):
    """Random long-wave modes: (wave numbers per axis, phase, amplitude of rho, u, v, w)."""
    r = np.random.default_rng(seed)
    return [(r.integers(-3, 4, 3), r.uniform(0, 2 * np.pi), r.normal(size=4)) for _ in range(count)]


def _flow(seed, shape, u0, mean, scale=1.0):
    """Density and velocity of a smooth random flow around the mean x velocity on a box of `shape`
    cells of size 1 / scale, as (4, nx, ny, nz) float64 on the GPU."""
    ax = [torch.arange(s, dtype=torch.float64, device="cuda") + 0.5 for s in shape]
    x, y, z = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    out = torch.zeros((4,) + tuple(shape), dtype=torch.float64, device="cuda")
    for k, ph, am in _modes(seed):
        if not k.any():
            continue
        arg = 2 * math.pi * (k[0] * x / shape[0] + k[1] * y / shape[1] + k[2] * z / shape[2]) + ph
        w = torch.sin(arg)
        amp = am.copy()
        amp[1:] -= k * (amp[1:] @ k) / (k @ k)  # solenoidal
        for c in range(4):
            out[c] += float(amp[c]) * w
    out *= u0 / (out[1:].abs().max() + 1e-30)
    out[0] = 1.0 + 0.1 * out[0].clamp(-1, 1) * u0 / max(u0, 1e-30)
    out[1] += mean
    return out


def _to_blocks(a):
    """(..., nx, ny, nz) -> (..., nb, 512): blocks sorted by (bx, by, bz), cell = x + 8 y + 64 z."""
    lead, (nx, ny, nz) = a.shape[:-3], a.shape[-3:]
    n = len(lead)
    a = a.reshape(*lead, nx // 8, 8, ny // 8, 8, nz // 8, 8)
    a = a.permute(*range(n), n, n + 2, n + 4, n + 5, n + 3, n + 1)
    return a.reshape(*lead, (nx // 8) * (ny // 8) * (nz // 8), 512)


def _box_mask(shape, centre, radius):
    """Solid cells of a sphere, (nx, ny, nz) bool."""
    ax = [torch.arange(s, dtype=torch.float64, device="cuda") + 0.5 - c for s, c in zip(shape, centre)]
    return (ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2) <= radius * radius


def _host(a):
    return np.ascontiguousarray(a.cpu().numpy())


class _View:
    """A device array of the library as the array interface that torch reads; `owner` (the object whose
    memory it is) lives as long as the tensors made from it."""

    def __init__(self, ptr, shape, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=tuple(shape), typestr=kind, version=3)


def _tensor(ptr, shape, storage, owner):
    kind = {"f16": "<f2", "bf16": "<u2", "f32": "<f4", "f64": "<f8"}[storage]
    t = torch.as_tensor(_View(ptr, shape, kind, owner), device="cuda")
    return t.view(torch.bfloat16) if storage == "bf16" else t


class _LevelViews:
    """Torch views of a level's current populations, density and velocity (the state's buffers)."""

    def __init__(self, level, nb, q, storage, tree=None):
        self.level, self.nb, self.q, self.storage = level, nb, q, storage
        self.owner = tree or level  # a hierarchy owns its levels
        self.macro = "f64" if storage == "f64" else "f32"
        self.p = [C.c_void_p() for _ in range(3)]
        self.refs = [C.byref(v) for v in self.p]
        self.kept = {}

    def __call__(self):
        capi.check(capi.lib().oal_level_device_state(self.level.handle, *self.refs))
        f, r, v = (a.value for a in self.p)
        if f not in self.kept:
            self.kept[f] = (_tensor(f, (self.nb, self.q, 512), self.storage, self.owner),
                            _tensor(r, (self.nb, 512), self.macro, self.owner),
                            _tensor(v, (3, self.nb, 512), self.macro, self.owner))
        return self.kept[f]


def _sphere_of(case):
    """Centre and diameter of the channel's sphere: a quarter of the length in, about a fifth of the height."""
    d = max(8.0, 0.1875 * min(case["ny"], case["nz"]))
    return (case["nx"] / 4.0, case["ny"] / 2.0, case["nz"] / 2.0), d


def _channel_fields(case, seed, u):
    shape = (case["nx"], case["ny"], case["nz"])
    centre, d = _sphere_of(case)
    m = _flow(seed, shape, 0.2 * u, u)
    solid = _box_mask(shape, centre, d / 2.0)
    m[1:, solid] = 0.0
    return m, solid, d


U_CHANNEL, RE_CHANNEL = 0.05, 1000.0


def _channel_params(case, d, svv=0.0):
    nu = U_CHANNEL * d / RE_CHANNEL
    return default_step_params(tau=3.0 * nu + 0.5, c_wale=0.2, u_inlet=U_CHANNEL, solid_bc=capi.OAL_SOLID_HALFWAY,
                               collect_forces=1, svv_yz_epsilon=svv)


def _box_tau(n, u0, re):
    return 3.0 * (u0 * n / (2 * math.pi) / re) + 0.5


def _batch_edges(case, seed):
    r = np.random.default_rng(1000 + case["members"])
    choice = [e for e in (16, 24, 32, 40, 48, 64) if case["n_min"] <= e <= case["n_max"]]
    return [int(r.choice(choice)) for _ in range(case["members"])]


def _amr_box(case):
    """The refined box of coarse cells, aligned to blocks, away from the domain faces."""
    ax = (case["nx"], case["ny"], case["nz"])
    lo = [8 * max(2, round(n / 8 / 8)) if i == 0 else 8 * max(2, round(n / 4 / 8)) for i, n in enumerate(ax)]
    hi = [max(lo[i] + 16, min(n - 16, 8 * round((n / 2 if i == 0 else 3 * n / 4) / 8))) for i, n in enumerate(ax)]
    return lo, hi


def _wing(case):
    s = case["chord"] / 128.0
    up = lambda v: 16 * max(1, round(v / 16))  # noqa: E731
    dom = (float(up(1024 * s)), float(up(512 * s)), float(24 if case["chord"] < 128 else 40))
    return octree.naca_case(chord=case["chord"], levels=3, domain=dom, leading_edge_x=320.0 * s,
                            precision=np.float64 if case["precision"] == "f64" else np.float32)


# ---- prepare / run ----------------------------------------------------------------------------
class _State:
    """What a user's program keeps between calls."""


def prepare(case, seed):
    s = _State()
    s.kind, s.case = case["kind"], case
    k = case["kind"]
    if k in ("box", "kbc_box"):
        n = case["n"]
        m = _flow(seed, (n, n, n), 0.05, 0.0)
        dom = build_box(n // 8, n // 8, n // 8, periodic=(True, True, True))
        s.geom = Geometry(dom)
        if k == "box":
            s.params = default_step_params(tau=_box_tau(n, 0.05, 1000.0), c_wale=case["c_wale"], u_inlet=0.0)
            s.level = Level(s.geom, storage=case["storage"])
            s.views = _LevelViews(s.level, dom.n_blocks, 27, case["storage"])
        else:
            s.params = default_entropic_params(tau=0.5 + 0.5 * (_box_tau(n, 0.05, 1000.0) - 0.5), c_wale=0.2, u_inlet=0.0)
            s.level = Level(s.geom, "entropic")
            s.views = _LevelViews(s.level, dom.n_blocks, 39, "f32")
        b = _to_blocks(m)
        s.level.init_equilibrium(_host(b[0]), _host(b[1:]))
    elif k in ("channel", "arrays", "kbc_channel"):
        m, solid, d = _channel_fields(case, seed, U_CHANNEL)
        dom = build_box(case["nx"] // 8, case["ny"] // 8, case["nz"] // 8)
        apply_analytic_sphere_obstacle(dom, _sphere_of(case)[0], d / 2.0)
        s.geom = Geometry(dom)
        b = _to_blocks(m)
        if k == "arrays":
            s.params = _channel_params(case, d)
            dt = torch.float64 if case["storage"] == "f64" else torch.float32
            nb = dom.n_blocks
            q = _q27()
            s.f = [torch.stack([_feq(q, b[0], b[1], b[2], b[3], i) for i in range(27)]).to(dt), None]
            s.f[1] = torch.empty_like(s.f[0])
            s.vel = [b[1:].to(dt).contiguous(), torch.empty((3, nb, 512), dtype=dt, device="cuda")]
            s.rho = torch.empty((nb, 512), dtype=dt, device="cuda")
            s.force = torch.zeros(3, dtype=torch.float64, device="cuda")
            s.nb = nb
        else:
            if k == "channel":
                s.params = _channel_params(case, d, case["svv"])
                s.level = Level(s.geom, storage=case["storage"])
                s.views = _LevelViews(s.level, dom.n_blocks, 27, case["storage"])
                s.drag = torch.zeros(3, dtype=torch.float64).pin_memory()
            else:
                nu = U_CHANNEL * d / RE_CHANNEL
                s.params = default_entropic_params(tau=0.5 + 1.5 * nu, c_wale=0.2, u_inlet=U_CHANNEL)
                s.level = Level(s.geom, "entropic")
                s.views = _LevelViews(s.level, dom.n_blocks, 39, "f32")
            s.level.init_equilibrium(_host(b[0]), _host(b[1:]))
    elif k == "batch":
        edges = _batch_edges(case, seed)
        s.geoms = [Geometry(build_box(n // 8, n // 8, n // 8, periodic=(True, True, True))) for n in edges]
        use = [g.blocks() for g in s.geoms]
        s.batch = Batch(storage=case["storage"], max_real_blocks=sum(u[0] for u in use),
                        max_ghost_blocks=max(1, sum(u[1] for u in use)), max_mask_blocks=max(1, sum(u[2] for u in use)),
                        max_members=len(edges))
        s.ids, s.out = [], []
        for i, (n, g) in enumerate(zip(edges, s.geoms)):
            b = _to_blocks(_flow(seed * 1000 + i, (n, n, n), 0.05, 0.0))
            p = default_step_params(tau=_box_tau(n, 0.05, 500.0 + 50.0 * i), c_wale=0.0, u_inlet=0.0)
            s.ids.append(s.batch.add(g, p, _host(b[0]), _host(b[1:])))
            s.out.append((np.empty((g.dom.n_blocks, 512)), np.empty((3, g.dom.n_blocks, 512))))
    elif k == "amr":
        coarse = build_box(case["nx"] // 8, case["ny"] // 8, case["nz"] // 8)
        centre, d = _sphere_of(case)
        apply_analytic_sphere_obstacle(coarse, centre, d / 2.0)
        lo, hi = _amr_box(case)
        fine = refine(coarse, blocks_in_box(coarse, lo, hi))
        apply_analytic_sphere_obstacle(fine, tuple(2 * c for c in centre), float(d))
        s.tree = Hierarchy([coarse, fine], storage=case["storage"])
        s.params = [default_step_params(tau=t, c_wale=0.2, u_inlet=U_CHANNEL, solid_bc=capi.OAL_SOLID_HALFWAY)
                    for t in _amr_taus(d)]
        for l, m in enumerate(_amr_fields(case, seed)):
            b = _to_blocks(m)
            s.tree.level(l).init_equilibrium(_host(b[0]), _host(b[1:]))
        s.views = [_LevelViews(s.tree.level(l), dd.n_blocks, 27, case["storage"], s.tree)
                   for l, dd in enumerate((coarse, fine))]
    elif k in ("oct_box", "oct_wing"):
        dt = np.float64 if case["precision"] == "f64" else np.float32
        if k == "oct_box":
            box = octree.PeriodicBox(case["n0"], case["n1"], case["n2"])
            s.state = octree.State(box, octree.test_case_config(box, nu_lattice=0.001, precision=dt, sgs="wale",
                                                                hrr_sigma=0.98))
            m = _flow(seed, box.n, 0.05, 0.0)
            pick = torch.as_tensor(_oct_cells(box.n), device="cuda")
            flat = m.reshape(4, -1)[:, pick.reshape(-1)].reshape(4, -1, 8)
            rho, u = _host(flat[0]), _host(flat[1:].permute(1, 0, 2))
            it = iter([(rho, u[:, 0], u[:, 1], u[:, 2])])
            s.state.initialise(lambda x, y, z: next(it), nonequilibrium=False)
        else:
            mesh, cfg = _wing(case)
            s.state = octree.State(mesh, cfg)
            md = _modes(seed)
            ext = [float(e) for e in mesh.spec.domain]

            def init(x, y, z):
                a = sum(0.2 * float(am[0]) * np.sin(2 * np.pi * (k3[0] * x / ext[0] + k3[1] * y / ext[1] + k3[2] * z / ext[2]) + ph)
                        for k3, ph, am in md)
                return 1.0 + 0.0 * x, cfg.u_lattice * (1.0 + 0.2 * a), 0.1 * cfg.u_lattice * a, 0.0 * x

            s.state.initialise(init, nonequilibrium=False)
        s.kept = [dict() for _ in range(s.state.nlevels)]
    else:
        raise ValueError(k)
    torch.cuda.synchronize()
    return s


def _oct_views(s):
    out = []
    for l in range(1, s.state.nlevels + 1):
        f, u, r, _ = s.state.device_state(l)
        kept = s.kept[l - 1]
        if f not in kept:
            no, p = s.state.level_meshes[l - 1].nocts, s.case["precision"]
            kept[f] = (_tensor(f, (no, 19, 8), p, s.state), _tensor(u, (no, 3, 8), p, s.state), _tensor(r, (no, 8), p, s.state))
        out.append(kept[f])
    return out


def run(s):
    case, k = s.case, s.kind
    n = case["steps"]
    if k in ("box", "channel", "kbc_box", "kbc_channel"):
        p = s.params
        if k == "channel" and not case["graph"]:
            for _ in range(n):
                s.level.perform_timestep(p)
                s.level.forces_async(s.drag.data_ptr())
        elif case.get("graph", True):
            s.level.execute_timestep_batch(p, n)
        else:
            for _ in range(n):
                s.level.perform_timestep(p)
        if k == "channel":
            if case["graph"]:
                s.level.forces_async(s.drag.data_ptr())
            return s.views() + (s.drag,)
        return s.views()
    if k == "arrays":
        nb, st = s.nb, capi.STORAGE_NAMES[case["storage"]]
        for _ in range(n):
            fl = capi.LevelFields(s.f[0].data_ptr(), s.f[1].data_ptr(), None, s.rho.data_ptr(), s.vel[1].data_ptr(),
                                  s.vel[0].data_ptr(), st, 0, 512, 512 * nb, 512 * nb, s.force.data_ptr())
            capi.check(capi.lib().oal_stream_collide(s.geom.handle, C.byref(fl), C.byref(s.params),
                                                     torch.cuda.current_stream().cuda_stream))
            s.f.reverse()
            s.vel.reverse()
        return s.f[0], s.rho, s.vel[0], s.force
    if k == "batch":
        s.batch.advance(n)
        for m, (r, v) in zip(s.ids, s.out):
            capi.check(capi.lib().oal_batch_get_state(s.batch.handle, m, None, r.ctypes.data, v.ctypes.data))
        return s.out
    if k == "amr":
        s.tree.advance(s.params, n)
        return [v() for v in s.views]
    s.state.advance(n)
    return _oct_views(s)


# ---- the cost of a pass ------------------------------------------------------------------------
FLOPS = {"d3q27": 700, "d3q39": 5000, "d3q19": 500}  # of one cell update, as the equations are written


def _level_work(cells, steps, q, item, macro, flops, extra=0):
    # per step: the populations read and written, density and velocity written, velocity read
    return dict(bytes=cells * steps * (2 * q * item + (1 + 3 + 3) * macro + extra), flops=cells * steps * flops)


def work(case):
    k, n = case["kind"], case["steps"]
    if k in ("box", "channel", "arrays"):
        cells = case["n"] ** 3 if k == "box" else case["nx"] * case["ny"] * case["nz"]
        it = ITEM[case["storage"]]
        w = _level_work(cells, n, 27, it, max(4, it), FLOPS["d3q27"])
        if case.get("svv", 0.0) > 0.0:
            w["flops"] += cells * n * 27 * 20
        return w
    if k in ("kbc_box", "kbc_channel"):
        cells = case["n"] ** 3 if k == "kbc_box" else case["nx"] * case["ny"] * case["nz"]
        return _level_work(cells, n, 39, 4, 4, FLOPS["d3q39"], extra=2 * 13 * 4)
    if k == "batch":
        cells = sum(e ** 3 for e in _batch_edges(case, 0))
        w = _level_work(cells, n, 27, ITEM[case["storage"]], 4, FLOPS["d3q27"])
        w["bytes"] += cells * 4 * 8
        return w
    if k == "amr":
        lo, hi = _amr_box(case)
        cells = case["nx"] * case["ny"] * case["nz"] + 2 * 8 * math.prod(h - l for l, h in zip(lo, hi))
        it = ITEM[case["storage"]]
        return _level_work(cells, n, 27, it, max(4, it), FLOPS["d3q27"])
    it = 8 if case["precision"] == "f64" else 4
    if k == "oct_box":
        return _level_work(case["n0"] * case["n1"] * case["n2"], n, 19, it, it, FLOPS["d3q19"], extra=it)
    return _level_work(_wing(case)[0].work_W(), n, 19, it, it, FLOPS["d3q19"], extra=it)


def tolerance(case):
    # About four times the distance from the 64-bit result measured over the ranges of draw().
    # 16-bit populations are deviations from the weights, rounded stochastically at every step: their
    # last place is 2^-11 (bf16: 2^-8) of the value, and another order of the sums draws other
    # rounding bits. The entropic operator's alpha is the root of an entropy difference that is of the
    # order of the FP32 rounding of its sums near equilibrium, so its results carry that noise. The
    # drag of a small sphere is a sum that nearly cancels in the first steps of a channel.
    k = case["kind"]
    if k in ("oct_box", "oct_wing"):
        return {"rel": 2e-14, "max": 3e-13} if case["precision"] == "f64" else {"rel": 1e-6, "max": 1e-5}
    if k in ("kbc_box", "kbc_channel"):
        return {"rel": 1.3e-2, "max": 0.1}
    f32 = {"rel": 1e-5, "max": 6e-5} if k in ("box", "batch", "amr") else {"rel": 1.6e-4, "max": 2e-4}
    return {"f64": {"rel": 2e-13, "max": 2e-12}, "f32": f32, "f16": {"rel": 2e-3, "max": 2e-2},
            "bf16": {"rel": 2e-2, "max": 0.1}}[case["storage"]]


# ---- the same results in 64 bits -----------------------------------------------------------------
def _q27():
    c = [(k % 3 - 1, (k // 3) % 3 - 1, k // 9 - 1) for k in range(27)]
    return c, [(8 / 27, 2 / 27, 1 / 54, 1 / 216)[sum(abs(v) for v in ck)] for ck in c]


def _feq(q, rho, ux, uy, uz, k):
    (cx, cy, cz), w = q[0][k], q[1][k]
    cu = cx * ux + cy * uy + cz * uz
    return w * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (ux * ux + uy * uy + uz * uz))


def _f32(v):
    return float(np.float32(v))


def _grad(vel, periodic, solid=None):
    """g[a][b] = d u_a / d x_b by central differences; a missing or solid neighbour counts as the cell."""
    def at(a, ax, d):
        r = torch.roll(a, -d, ax)
        own = torch.zeros_like(a, dtype=torch.bool)
        if not periodic:
            own.select(ax, -1 if d > 0 else 0).fill_(True)
        if solid is not None:
            own |= torch.roll(solid, -d, ax)
        return torch.where(own, a, r)
    return [[0.5 * (at(vel[a], b, 1) - at(vel[a], b, -1)) for b in range(3)] for a in range(3)]


def _wale(g, c_wale, eps):
    sq = [[sum(g[i][k] * g[k][j] for k in range(3)) for j in range(3)] for i in range(3)]
    tr = (sq[0][0] + sq[1][1] + sq[2][2]) / 3
    dd = sum((0.5 * (sq[i][j] + sq[j][i]) - (tr if i == j else 0.0)) ** 2 for i in range(3) for j in range(3))
    ss = sum((0.5 * (g[i][j] + g[j][i])) ** 2 for i in range(3) for j in range(3))
    if eps is None:  # D3Q19: a small constant in the denominator
        return c_wale ** 2 * dd ** 1.5 / (ss ** 2.5 + dd ** 1.25 + 1e-20)
    den = ss * ss * ss.clamp(min=eps).sqrt() + dd * dd.clamp(min=eps).sqrt().sqrt()
    nu = c_wale ** 2 * dd ** 1.5 / den.clamp(min=1e-300)
    return torch.where((dd > eps) & (den > eps), nu, torch.zeros_like(nu))


def _cumulant(A, rho, u, om1, lam=1.0 / 6.0):
    """The cumulant collision of the populations A (27, ...) with omega_1, the other rates 1, adaptive
    omega_4 of the diagonal group and the factored limiter."""
    M = {(a, b, c): A[(a + 1) + 3 * (b + 1) + 9 * (c + 1)] for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)}
    for ax in range(3):
        N = {}
        for key in M:
            if key[ax] != 0:
                continue
            tri = [M[key[:ax] + (d,) + key[ax + 1:]] for d in (-1, 0, 1)]
            for p in range(3):
                mom = sum(((d - u[ax]) ** p if p else 1.0) * v for d, v in zip((-1, 0, 1), tri))
                N[key[:ax] + (p - 10,) + key[ax + 1:]] = mom
        M = N
    K = {tuple(p + 10 for p in key): v for key, v in M.items()}
    r = K[0, 0, 0]
    inv = 1.0 / r.clamp(min=0.01)
    k = {key: v * inv for key, v in K.items()}
    a4 = (-(om1 - 2) ** 2 / (lam * om1 + 1e-10)).clamp(0.01, 2.0)
    C2 = {}
    for (i, j) in ((0, 1), (0, 2), (1, 2)):
        kk = lambda *p: k[tuple(p.count(n) for n in range(3))]  # noqa: E731
        C2[i, j] = kk(i, i, j, j) - kk(i, i) * kk(j, j) - 2 * kk(i, j) ** 2
    mo = lambda *p: k[tuple(p.count(n) for n in range(3))]  # noqa: E731
    d1, d2 = (1 - om1) * (mo(0, 0) - mo(1, 1)), (1 - om1) * (mo(0, 0) - mo(2, 2))
    s = {(0, 0): (1 + d1 + d2) / 3, (1, 1): (1 - 2 * d1 + d2) / 3, (2, 2): (1 + d1 - 2 * d2) / 3}
    for (i, j) in ((0, 1), (0, 2), (1, 2)):
        b = (s[i, i] * s[j, j]).clamp(min=0).sqrt()
        v = (1 - om1) * mo(i, j)
        s[i, j] = torch.maximum(torch.minimum(v, b), -b)
    z = torch.zeros_like(r)
    out = {key: z for key in K}
    out[0, 0, 0] = torch.ones_like(r)
    put = lambda v, *p: out.__setitem__(tuple(p.count(n) for n in range(3)), v)  # noqa: E731
    for key, v in s.items():
        put(v, *key)
    C4 = {key: (1 - a4) * v for key, v in C2.items()}
    for (i, j) in C4:
        put(C4[i, j] + s[i, i] * s[j, j] + 2 * s[i, j] ** 2, i, i, j, j)
    x, y, w = s[0, 1], s[0, 2], s[1, 2]
    put(s[0, 0] * w + 2 * x * y, 0, 0, 1, 2)
    put(s[1, 1] * y + 2 * x * w, 0, 1, 1, 2)
    put(s[2, 2] * x + 2 * y * w, 0, 1, 2, 2)
    c222 = s[0, 0] * C4[1, 2] + s[1, 1] * C4[0, 2] + s[2, 2] * C4[0, 1]
    c222 = c222 + 8 * x * y * w + 2 * (s[2, 2] * x * x + s[1, 1] * y * y + s[0, 0] * w * w) + s[0, 0] * s[1, 1] * s[2, 2]
    out[2, 2, 2] = c222
    out = {key: v * r for key, v in out.items()}
    for ax in range(3):
        N = {}
        for key in out:
            if key[ax] != 0:
                continue
            m = [out[key[:ax] + (p,) + key[ax + 1:]] for p in range(3)]
            v = u[ax]
            m1, m2 = m[1] + v * m[0], m[2] + 2 * v * m[1] + v * v * m[0]
            for d, f in ((-11, 0.5 * (m2 - m1)), (-10, m[0] - m2), (-9, 0.5 * (m2 + m1))):
                N[key[:ax] + (d,) + key[ax + 1:]] = f
        out = N
    return torch.stack([out[a - 10, b - 10, c - 10] for c in (-1, 0, 1) for b in (-1, 0, 1) for a in (-1, 0, 1)])


def _step27(f, vel, p, periodic, solid=None, source=None):
    """One D3Q27 step on a dense box: f (27, nx, ny, nz), the previous velocity; `source`: the field the
    pulls read, one cell larger on each side (a refined level), instead of the domain faces."""
    q = _q27()
    shape = f.shape[1:]
    A = torch.empty_like(f)
    force = torch.zeros(3, dtype=torch.float64, device=f.device)
    for k, (cx, cy, cz) in enumerate(q[0]):
        if source is not None:
            v = source[k][1 - cx:1 - cx + shape[0], 1 - cy:1 - cy + shape[1], 1 - cz:1 - cz + shape[2]].clone()
        else:
            v = torch.roll(f[k], (cx, cy, cz), (0, 1, 2))
            if not periodic:
                if cz:
                    e = 0 if cz > 0 else -1
                    v[:, :, e] = f[(k % 9) + 9 * (2 - k // 9)][:, :, e]
                if cy:
                    e = 0 if cy > 0 else -1
                    v[:, e] = f[(k % 3) + 3 * (2 - (k // 3) % 3) + 9 * (k // 9)][:, e]
                if cx < 0:
                    v[-1] = f[k][-1]
                if cx > 0:
                    one = torch.ones((), dtype=torch.float64)
                    v[0] = float(_feq(q, one, p["u"] * one, 0 * one, 0 * one, k))
        if solid is not None and k != 13:
            cut = torch.roll(solid, (cx, cy, cz), (0, 1, 2)) & ~solid
            v = torch.where(cut, f[26 - k], v)
            m = 2.0 * (f[26 - k] * cut).sum()
            force -= m * torch.tensor([cx, cy, cz], dtype=torch.float64, device=f.device)
        A[k] = v
    rho = A.sum(0).clamp(min=0.01)
    u = [sum(ck[a] * A[k] for k, ck in enumerate(q[0]) if ck[a]) / rho for a in range(3)]
    nu = _wale(_grad(vel, periodic, solid), p["c_wale"], 1e-12) if p["c_wale"] else torch.zeros_like(rho)
    om = 1.0 / (3 * ((p["tau"] - 0.5) / 3 + nu) + 0.5).clamp(min=0.500001)
    out = _cumulant(A, rho, u, om, p["lam"])
    vout = torch.stack(u)
    if solid is not None:
        for k in range(27):
            out[k][solid] = q[1][k]
        rho = torch.where(solid, torch.ones_like(rho), rho)
        vout[:, solid] = 0.0
    return out, rho, vout, force


def _svv(fin, f, eps, solid):
    """The 5-point bi-Laplacian filter of f along y and z, the taps from the step's input."""
    q = _q27()
    new = torch.empty_like(f)
    dr = torch.zeros_like(f[0])
    dj = [torch.zeros_like(f[0]) for _ in range(3)]
    own = {}
    for ax in (1, 2):
        for d in (-2, -1, 1, 2):
            o = torch.roll(solid, -d, ax).clone()
            o.narrow(ax, o.shape[ax] - d if d > 0 else 0, abs(d)).fill_(True)
            own[ax, d] = o
    for k, ck in enumerate(q[0]):
        t = {(ax, d): torch.where(own[ax, d], fin[k], torch.roll(fin[k], -d, ax)) for ax, d in own}
        b = sum(t[ax, -2] - 4 * t[ax, -1] + 6 * f[k] - 4 * t[ax, 1] + t[ax, 2] for ax in (1, 2))
        new[k] = f[k] - eps * b
        e = new[k] - f[k]
        dr += e
        for a in range(3):
            dj[a] += ck[a] * e
    for k, ck in enumerate(q[0]):
        v = new[k] - q[1][k] * (dr + 3 * sum(ck[a] * dj[a] for a in range(3)))
        new[k] = torch.where(solid, f[k], v.clamp(min=1e-12))
    return new


def _pops(f, storage):
    """The stored form, (nb, 27, 512): 16-bit storage keeps f / w - 1."""
    if storage in ("f16", "bf16"):
        w = torch.tensor(_q27()[1], dtype=torch.float64, device=f.device)[:, None, None, None]
        f = f / w - 1.0
    return _to_blocks(f).permute(1, 0, 2).contiguous()


def _start27(m):
    q = _q27()
    return torch.stack([_feq(q, m[0], m[1], m[2], m[3], k) for k in range(27)])


def _p27(params):
    return dict(tau=float(params.tau), c_wale=float(params.c_wale), u=float(params.u_inlet), lam=float(params.lambda_param))


def _exact_box(case, seed, n, c_wale, re=1000.0):
    p = default_step_params(tau=_box_tau(n, 0.05, re), c_wale=c_wale, u_inlet=0.0)
    m = _flow(seed, (n, n, n), 0.05, 0.0)
    f, vel = _start27(m), m[1:]
    for _ in range(case["steps"]):
        f, rho, vel, _ = _step27(f, vel, _p27(p), True)
    return f, rho, vel


def _exact_channel(case, seed):
    m, solid, d = _channel_fields(case, seed, U_CHANNEL)
    svv = _f32(case.get("svv", 0.0))
    p = _p27(_channel_params(case, d))
    f, vel = _start27(m), m[1:]
    for _ in range(case["steps"]):
        g, rho, vel, force = _step27(f, vel, p, False, solid)
        f = _svv(f, g, svv, solid) if svv > 0 else g
    if case["kind"] == "arrays":
        return _to_blocks(f), _to_blocks(rho), _to_blocks(vel), force
    return _pops(f, case["storage"]), _to_blocks(rho), _to_blocks(vel), force.cpu()


def _amr_taus(d):
    nu = U_CHANNEL * 2 * d / RE_CHANNEL
    fine = 3.0 * nu + 0.5
    return [0.5 + 2 * (fine - 0.5), fine]


def _amr_fields(case, seed):
    lo, hi = _amr_box(case)
    shape = (case["nx"], case["ny"], case["nz"])
    centre, d = _sphere_of(case)
    out = []
    for s in (1, 2):
        m = _flow(seed, [s * n for n in shape], 0.2 * U_CHANNEL, U_CHANNEL)
        m[1:, _box_mask([s * n for n in shape], [s * c for c in centre], s * d / 2.0)] = 0.0
        if s == 2:
            m = m[:, 2 * lo[0]:2 * hi[0], 2 * lo[1]:2 * hi[1], 2 * lo[2]:2 * hi[2]].contiguous()
        out.append(m)
    return out


def _cubic_up(a, lo, hi):
    """Cubic Lagrange interpolation of the coarse field a (..., nx, ny, nz) at the fine cells of the
    coarse box [lo, hi) and one fine cell around it."""
    def wts(w):
        return [-w * (w - 1) * (w - 2) / 6, (w + 1) * (w - 1) * (w - 2) / 2, -w * (w + 1) * (w - 2) / 2,
                w * (w + 1) * (w - 1) / 6]
    for ax in range(3):
        dim = a.dim() - 3 + ax
        g = np.arange(2 * lo[ax], 2 * hi[ax] + 2)  # 1-based fine index of the cells with one more each side
        pc = 0.5 * g + 0.25
        i0 = np.floor(pc).astype(int)
        w = torch.as_tensor(pc - i0, device=a.device, dtype=a.dtype)
        shape = [1] * a.dim()
        shape[dim] = -1
        out = 0
        for j, wj in enumerate(wts(w)):
            out = out + wj.reshape(shape) * a.index_select(dim, torch.as_tensor(i0 - 1 + j - 1, device=a.device))
        a = out
    return a


def _exact_amr(case, seed):
    q = _q27()
    lo, hi = _amr_box(case)
    shape = (case["nx"], case["ny"], case["nz"])
    centre, d = _sphere_of(case)
    taus = [_f32(t) for t in _amr_taus(d)]
    solid = [_box_mask([s * n for n in shape], [s * c for c in centre], s * d / 2.0) for s in (1, 2)]
    sl = [slice(2 * l, 2 * h) for l, h in zip(lo, hi)]
    solid[1] = solid[1][sl[0], sl[1], sl[2]].contiguous()
    ms = _amr_fields(case, seed)
    f, vel, rho = [_start27(m) for m in ms], [m[1:] for m in ms], [m[0] for m in ms]
    P = [dict(tau=t, c_wale=_f32(0.2), u=_f32(U_CHANNEL), lam=_f32(1 / 6)) for t in taus]
    omc, omf = 1 / taus[0], 1 / taus[1]
    scale = (taus[1] - 0.5) / (taus[0] - 0.5) * (1 - omf) / (1 - omc)
    ratio = (taus[0] - 0.5) / (taus[1] - 0.5) * (1 - omc) / (1 - omf)
    cbox = [slice(l - 4, h + 4) for l, h in zip(lo, hi)]
    clo, chi = [4] * 3, [4 + h - l for l, h in zip(lo, hi)]
    for _ in range(case["steps"]):
        old = (f[0], rho[0], vel[0])
        f[0], rho[0], vel[0], _ = _step27(f[0], vel[0], P[0], False, solid[0])
        new = (f[0], rho[0], vel[0])
        for tw in (0.0, 0.5):
            part = lambda a: a[..., cbox[0], cbox[1], cbox[2]]  # noqa: E731
            cf, cr, cv = (part(o) * (1 - tw) + part(n) * tw for o, n in zip(old, new))
            up = _cubic_up(torch.cat([cr[None], cv]), clo, chi)
            src = torch.empty((27,) + tuple(up.shape[1:]), dtype=torch.float64, device=up.device)
            for k in range(27):
                neq = cf[k] - _feq(q, cr, cv[0], cv[1], cv[2], k)
                src[k] = _feq(q, up[0], up[1], up[2], up[3], k) + scale * _cubic_up(neq, clo, chi)
            src[:, 1:-1, 1:-1, 1:-1] = f[1]
            f[1], rho[1], vel[1], _ = _step27(f[1], vel[1], P[1], False, solid[1], source=src)
        fluid = (~solid[1]).double()
        sh = f[1].shape[1:]
        fold = lambda a: a.reshape(*a.shape[:-3], sh[0] // 2, 2, sh[1] // 2, 2, sh[2] // 2, 2).sum((-1, -3, -5))  # noqa: E731
        cnt = fold(fluid)
        avg = fold(f[1] * fluid) / cnt.clamp(min=1)
        r = avg.sum(0).clamp(min=0.01)
        u = [sum(ck[a] * avg[k] for k, ck in enumerate(q[0]) if ck[a]) / r for a in range(3)]
        box = tuple(slice(l, h) for l, h in zip(lo, hi))
        f[0], rho[0], vel[0] = f[0].clone(), rho[0].clone(), vel[0].clone()
        for k in range(27):
            fe = _feq(q, r, u[0], u[1], u[2], k)
            f[0][(k,) + box] = torch.where(cnt > 0, (fe + ratio * (avg[k] - fe)).clamp(min=1e-10), f[0][(k,) + box])
        rho[0][box] = torch.where(cnt > 0, r, rho[0][box])
        for a in range(3):
            vel[0][(a,) + box] = torch.where(cnt > 0, u[a], vel[0][(a,) + box])
    return [(_pops(f[l], case["storage"]), _to_blocks(rho[l]), _to_blocks(vel[l])) for l in range(2)]


C19 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, -1, 0),
       (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)]
W19 = [(1 / 3, 1 / 18, 1 / 36)[sum(abs(v) for v in c)] for c in C19]


def _oct_cells(n):
    """(nocts, 8) linear index into the (n0, n1, n2) cells of each slot, octs in Morton order."""
    m = [v // 2 for v in n]
    i, j, k = (a.reshape(-1) for a in np.meshgrid(*(np.arange(v) for v in m), indexing="ij"))

    def spread(v):
        out = np.zeros(v.shape, np.uint64)
        for b in range(20):
            out |= ((v.astype(np.uint64) >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b)
        return out
    key = spread(i + 1) | (spread(j + 1) << np.uint64(1)) | (spread(k + 1) << np.uint64(2))
    o = np.argsort(key, kind="stable")
    s = np.arange(8)
    x, y, z = 2 * i[o][:, None] + (s & 1), 2 * j[o][:, None] + ((s >> 1) & 1), 2 * k[o][:, None] + (s >> 2)
    return ((x * n[1] + y) * n[2] + z).astype(np.int64)


def _rr19(rho, u, pi, keep):
    """Recursive-regularised D3Q19 populations less the weights: second- and third-order Hermite terms."""
    d = torch.float64
    drho = rho - 1.0
    out = torch.empty((19,) + tuple(rho.shape), dtype=d, device=rho.device)
    idx = {(0, 0): 0, (1, 1): 1, (2, 2): 2, (0, 1): 3, (0, 2): 4, (1, 2): 5}
    P = lambda a, b: pi[idx[min(a, b), max(a, b)]]  # noqa: E731
    usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    # third-order non-equilibrium coefficients a_aab = 2 u_a P_ab + u_b P_aa
    a3 = {(a, b): 2 * u[a] * P(a, b) + u[b] * P(a, a) for a in range(3) for b in range(3) if a != b}
    for i, c in enumerate(C19):
        w = W19[i]
        cu = sum(c[a] * u[a] for a in range(3))
        h2 = sum((c[a] * c[b] - (1 / 3 if a == b else 0.0)) * P(a, b) for a in range(3) for b in range(3))
        # the six Hermite polynomials H_aab of the lattice, (c_a^2 - 1/3) c_b
        h3 = sum((c[a] * c[a] - 1 / 3) * c[b] * v for (a, b), v in a3.items())
        out[i] = w * (drho + rho * (3 * cu + 4.5 * cu * cu - 1.5 * usq) + keep * (4.5 * h2 + 13.5 * h3))
    return out


def _exact_oct_box(case, seed):
    n = (case["n0"], case["n1"], case["n2"])
    if math.prod(n) > 8_000_000:
        return None
    dt = torch.float64 if case["precision"] == "f64" else torch.float32
    m = _flow(seed, n, 0.05, 0.0).to(dt).double()
    one = lambda v: v if case["precision"] == "f64" else _f32(v)  # noqa: E731
    nu0, cw, sigma = one(0.001), one(0.5), one(0.98)
    rho, u = m[0], m[1:]
    zero = torch.zeros((6,) + tuple(n), dtype=torch.float64, device="cuda")
    f = _rr19(rho, u, zero, 0.0)
    for _ in range(case["steps"]):
        A = torch.stack([torch.roll(f[i], c, (0, 1, 2)) for i, c in enumerate(C19)])
        g = _grad(u, True)
        nut = _wale(g, cw, None)
        tau = 3 * (nu0 + nut) + 0.5
        prev = rho
        rho = 1.0 + A.sum(0)
        un = [sum(c[a] * A[i] for i, c in enumerate(C19) if c[a]) / rho for a in range(3)]
        pi = []
        for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)):
            raw = sum(c[a] * c[b] * A[i] for i, c in enumerate(C19) if c[a] * c[b])
            p = raw - ((rho - 1.0) / 3 if a == b else 0.0) - rho * un[a] * un[b]
            fd = -prev * tau / 3 * (g[a][b] + g[b][a])
            pi.append(sigma * p + (1 - sigma) * fd)
        f = _rr19(rho, un, pi, 1 - 1 / tau)
        u = torch.stack(un)
    pick = torch.as_tensor(_oct_cells(n), device="cuda").reshape(-1)
    slots = lambda a: a.reshape(a.shape[0], -1)[:, pick].reshape(a.shape[0], -1, 8).permute(1, 0, 2).contiguous()  # noqa: E731
    return [(slots(f), slots(u), slots(rho[None])[:, 0].contiguous())]


C39 = ([(0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)]
       + [(x, y, z) for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)]
       + [(-2, 0, 0), (2, 0, 0), (0, -2, 0), (0, 2, 0), (0, 0, -2), (0, 0, 2)]
       + [(-2, -2, 0), (-2, 2, 0), (2, -2, 0), (2, 2, 0), (-2, 0, -2), (-2, 0, 2), (2, 0, -2), (2, 0, 2), (0, -2, -2),
          (0, -2, 2), (0, 2, -2), (0, 2, 2)]
       + [(-3, 0, 0), (3, 0, 0), (0, -3, 0), (0, 3, 0), (0, 0, -3), (0, 0, 3)])
W39 = [{0: 1 / 12, 1: 1 / 12, 3: 1 / 27, 4: 2 / 135, 8: 1 / 432, 9: 1 / 1620}[sum(v * v for v in c)] for c in C39]
CS39 = 2.0 / 3.0


def _eq39(rho, u):
    """The 13-moment entropic equilibrium w exp(sum of multipliers times basis), by Newton's method."""
    c = torch.tensor(C39, dtype=torch.float64, device=rho.device)
    w = torch.tensor(W39, dtype=torch.float64, device=rho.device)
    efl = (c ** 2).sum(1) - 5 * CS39
    B = torch.stack([torch.ones_like(efl), *c.T, *(c.T ** 2 - CS39), c[:, 0] * c[:, 1], c[:, 0] * c[:, 2],
                     c[:, 1] * c[:, 2], *(c.T * efl)], 1)  # (39, 13)
    shape = rho.shape
    r = rho.reshape(-1)
    ux, uy, uz = (v.reshape(-1) for v in u)
    usq = ux * ux + uy * uy + uz * uz
    out = torch.empty((39, r.numel()), dtype=torch.float64, device=rho.device)
    for a in range(0, r.numel(), 1 << 17):
        s = slice(a, a + (1 << 17))
        x, y, z, q, rr = ux[s], uy[s], uz[s], usq[s], r[s]
        mt = rr[:, None] * torch.stack([torch.ones_like(x), x, y, z, x * x, y * y, z * z, x * y, x * z, y * z, x * q, y * q, z * q], 1)
        i1, i2 = 1 / CS39, 1 / CS39 ** 2
        o = torch.zeros_like(x)
        la = torch.stack([-0.5 * q * i1, x * i1, y * i1, z * i1, 0.5 * i2 * x * x, 0.5 * i2 * y * y, 0.5 * i2 * z * z,
                          i2 * x * y, i2 * x * z, i2 * y * z, o, o, o], 1)
        for _ in range(6):
            f = rr[:, None] * w * torch.exp(la @ B.T)
            H = torch.einsum("nk,ki,kj->nij", f, B, B)
            la = la + torch.linalg.solve(H, mt - f @ B)
        f = rr[:, None] * w * torch.exp(la @ B.T)
        out[:, s] = (f * (rr / f.sum(1))[:, None]).T
    return out.reshape((39,) + tuple(shape))


def _exact_kbc_box(case, seed):
    n = case["n"]
    p = default_entropic_params(tau=0.5 + 0.5 * (_box_tau(n, 0.05, 1000.0) - 0.5), c_wale=0.2, u_inlet=0.0)
    m = _flow(seed, (n, n, n), 0.05, 0.0).float().double()
    f, vel = _eq39(m[0], m[1:]), m[1:]
    opp = [C39.index(tuple(-v for v in c)) for c in C39]
    w = torch.tensor(W39, dtype=torch.float64, device="cuda")[:, None, None, None]
    H = lambda a: (a.clamp(min=1e-15) * (a.clamp(min=1e-15) / w).log()).sum(0)  # noqa: E731
    for _ in range(case["steps"]):
        A = torch.stack([torch.roll(f[i], c, (0, 1, 2)) for i, c in enumerate(C39)])
        rho = A.sum(0)
        u = torch.stack([sum(c[a] * A[i] for i, c in enumerate(C39) if c[a]) / rho for a in range(3)])
        fe = _eq39(rho, u)
        nu = _wale(_grad(vel, True), _f32(0.2), 1e-12)
        tau = 0.5 + ((float(p.tau) - 0.5) * CS39 + nu) / CS39
        beta = 0.5 / tau.clamp(min=0.500001)
        pre = H(A)
        df = A - fe
        s, h = 0.5 * (df + df[opp]), 0.5 * (df - df[opp])
        base = fe + (1 - 2 * beta) * s
        ib = 0.5 / beta.clamp(min=0.01)
        l, r = (ib - 0.1).clamp(min=0.1), (ib + 3.0).clamp(min=4.0)
        res = lambda al: H(base + (1 - 2 * beta * al) * h) - pre  # noqa: E731
        hl, hr = res(l), res(r)
        found = hl * hr < 0
        open_ = found.clone()
        for _ in range(10):
            mid = 0.5 * (l + r)
            hm = res(mid)
            up = hm * hl > 0
            l = torch.where(open_ & up, mid, l)
            hl = torch.where(open_ & up, hm, hl)
            r = torch.where(open_ & ~up, mid, r)
            open_ &= (r - l) >= 0.005 * (ib + 1e-6)
        al = torch.where(found, 0.5 * (l + r), ib)
        al = torch.minimum(torch.maximum(al, ib), torch.full_like(al, 6.0))
        al = torch.where((h ** 2).sum(0) > 1e-20, al, torch.full_like(al, 2.0))
        f = base + (1 - 2 * beta * al) * h
        vel = u
    return _to_blocks(f).permute(1, 0, 2).contiguous(), _to_blocks(rho), _to_blocks(vel)


def exact(case, seed):
    """The state after the case's steps in 64 bits; None for the octree wing (its mesh, walls and level
    transfers are data of the generator) and the entropic channel, and above the sizes noted."""
    k = case["kind"]
    if k == "box":
        f, rho, vel = _exact_box(case, seed, case["n"], _f32(case["c_wale"]))
        return _pops(f, case["storage"]), _to_blocks(rho), _to_blocks(vel)
    if k in ("channel", "arrays"):
        return _exact_channel(case, seed)
    if k == "batch":
        if case["members"] * case["steps"] > 1500:
            return None
        out = []
        for i, n in enumerate(_batch_edges(case, seed)):
            _, rho, vel = _exact_box(case, seed * 1000 + i, n, 0.0, 500.0 + 50.0 * i)
            out.append((_to_blocks(rho), _to_blocks(vel)))
        return out
    if k == "amr":
        return _exact_amr(case, seed)
    if k == "kbc_box":
        return _exact_kbc_box(case, seed)
    if k == "oct_box":
        return _exact_oct_box(case, seed)
    return None
