"""oal_stream_collide on caller-owned arrays: interior blocks on the uniform kernels with the caller's
strides, the rest on the general kernel, against the general kernel on every block. Arrays that start
off a pair, odd strides and a requested f_post_collision keep the general kernel everywhere, so the
same step on both kinds of arrays compares the two routes over what each accepts."""
import ctypes as C

import numpy as np
import pytest

from openaerolab_alpha_01_b200 import _capi as capi
from openaerolab_alpha_01_b200.cases import sphere_channel_case, taylor_green_case
from openaerolab_alpha_01_b200.solver import Geometry

pytestmark = pytest.mark.gpu

STEPS = 3
# FP32 and FP64 as the parity tests; 16-bit: the routes round the sums differently, so a stored
# deviation may fall to the neighbouring value (2^-10, bf16 2^-7, of the largest) at every step
TOL = {"f32": 2e-5, "f64": 1e-11, "f16": STEPS * 2.0 ** -10, "bf16": STEPS * 2.0 ** -7}


def weights():
    c = np.stack(np.meshgrid(*(np.arange(3) - 1,) * 3, indexing="ij"), -1).reshape(27, 3)
    return np.array([(8 / 27, 2 / 27, 1 / 54, 1 / 216)[int(np.abs(k).sum())] for k in c])


def run(case, storage, steps, off=0, block_stride=512, pad=0, post=False, dir_stride=None, svv=(0.0, 0.0)):
    """The case's populations, density, velocity and force after `steps`, in caller-owned arrays that
    start `off` elements into their buffers, with `pad` extra elements between directions (or directions
    `dir_stride` apart), the spectral-viscosity filter of strengths `svv` after each."""
    import torch
    dt = {"f32": torch.float32, "f64": torch.float64, "f16": torch.float16, "bf16": torch.bfloat16}[storage]
    mt = torch.float64 if storage == "f64" else torch.float32
    g, nb = Geometry(case.dom), case.dom.n_blocks
    kst = dir_stride or block_stride * nb + pad
    w = weights()
    c = np.stack(np.meshgrid(*(np.arange(3) - 1,) * 3, indexing="ij"), -1).reshape(27, 3)[:, ::-1]  # x fastest
    cu = np.tensordot(c.astype(float), case.vel, 1)
    f0 = w[:, None, None] * case.rho * (1 + 3 * cu + 4.5 * cu ** 2 - 1.5 * (case.vel ** 2).sum(0))
    if storage in ("f16", "bf16"):
        f0 = f0 / w[:, None, None] - 1.0
    size = max(27 * kst, (nb - 1) * block_stride + 26 * kst + 512) + off
    buf = [torch.zeros(size, dtype=dt, device="cuda") for _ in range(3 if post else 2)]
    view = lambda b: torch.as_strided(b, (27, nb, 512), (kst, block_stride, 1), off)  # noqa: E731
    view(buf[0]).copy_(torch.tensor(f0).to(dt))
    vel = [torch.zeros(3 * nb * 512 + off, dtype=mt, device="cuda") for _ in range(2)]
    vel[0][off:].copy_(torch.tensor(case.vel).reshape(-1).to(mt))
    rho = torch.zeros(nb * 512 + off, dtype=mt, device="cuda")
    force = torch.zeros(3, dtype=torch.float64, device="cuda")
    p = capi.StepParams.from_buffer_copy(case.params)
    p.store_post_collision = int(post)
    p.svv_x_epsilon, p.svv_yz_epsilon = svv
    at = lambda t: t.data_ptr() + off * t.element_size()  # noqa: E731
    for _ in range(steps):
        fl = capi.LevelFields(at(buf[0]), at(buf[1]), at(buf[2]) if post else None, at(rho), at(vel[1]), at(vel[0]),
                              capi.STORAGE_NAMES[storage], 0, block_stride, kst, 512 * nb, force.data_ptr())
        capi.check(capi.lib().oal_stream_collide(g.handle, C.byref(fl), C.byref(p), None))
        buf[0], buf[1] = buf[1], buf[0]
        vel.reverse()
    torch.cuda.synchronize()
    out = [view(buf[0]).double().cpu().numpy(), rho[off:].double().cpu().numpy(), vel[0][off:].double().cpu().numpy(),
           force.cpu().numpy()]
    g.close()
    return out


def cases():
    # every block interior (periodic), a domain with one interior block, none, and a channel with a sphere
    yield "periodic", taylor_green_case(24, c_wale=0.2)
    yield "one_interior", sphere_channel_case(24, 24, 24, diameter=4.0, centre_x=4.0, re=100.0)
    yield "thin", sphere_channel_case(32, 16, 16, diameter=6.0, centre_x=10.0, re=100.0)
    yield "channel", sphere_channel_case(56, 40, 32, diameter=8.0, centre_x=16.0, re=100.0)
    c = sphere_channel_case(40, 40, 40, diameter=8.0, centre_x=16.0, re=100.0, omega3=1.1,
                            limiter_type=capi.OAL_LIMITER_POSITIVITY)
    yield "general_rates", c
    # enough interior blocks for a launch of their own: 504, FP64's 448 among them, and 125 of the 112 elsewhere
    yield "split", sphere_channel_case(128, 64, 64, diameter=16.0, centre_x=32.0, re=100.0)
    yield "split_rates", sphere_channel_case(128, 64, 64, diameter=16.0, centre_x=32.0, re=100.0, omega3=1.1,
                                             limiter_type=capi.OAL_LIMITER_POSITIVITY)
    yield "split_least", sphere_channel_case(56, 56, 56, diameter=8.0, centre_x=16.0, re=100.0)


@pytest.mark.parametrize("storage", ["f32", "f64", "f16", "bf16"])
@pytest.mark.parametrize("name,case", list(cases()), ids=[n for n, _ in cases()])
def test_uniform_and_general_routes_agree(oal, storage, name, case):
    want = run(case, storage, STEPS, post=True)  # the general kernel on every block
    for kw in (dict(), dict(off=2), dict(block_stride=520), dict(pad=6)):
        got = run(case, storage, STEPS, **kw)
        for a, b in zip(got[:3], want[:3]):
            assert np.max(np.abs(a - b)) < TOL[storage] * np.max(np.abs(want[0])), kw
        scale = max(np.max(np.abs(want[3])), 1e-30)
        assert np.max(np.abs(got[3] - want[3])) <= 10 * TOL[storage] * max(scale, 1e-2), kw


@pytest.mark.parametrize("kw", [dict(off=1), dict(pad=1), dict(off=1, pad=3)])
@pytest.mark.parametrize("edge", [40, 64])
def test_unpaired_arrays_keep_the_general_route(oal, kw, edge):
    case = sphere_channel_case(edge, edge, edge, diameter=8.0, centre_x=16.0, re=100.0)
    want, got = run(case, "f32", STEPS, post=True), run(case, "f32", STEPS, **kw)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def holed(case):
    """The case's domain without some of its blocks: missing neighbours inside the domain."""
    from openaerolab_alpha_01_b200.amr import neighbor_table
    from openaerolab_alpha_01_b200.cases import Case
    from openaerolab_alpha_01_b200.solver import BlockDomain
    d = case.dom
    keep = [i for i, c in enumerate(d.coords.tolist()) if c not in ([2, 2, 2], [4, 1, 3], [5, 5, 5])]
    coords = np.ascontiguousarray(d.coords[keep])
    dom = BlockDomain(d.bx_max, d.by_max, d.bz_max, coords, neighbor_table(coords, (d.bx_max, d.by_max, d.bz_max)),
                      obstacle=None if d.obstacle is None else np.ascontiguousarray(d.obstacle[keep]))
    return Case(case.name, dom, np.ascontiguousarray(case.rho[keep]), np.ascontiguousarray(case.vel[:, keep]), case.params)


# the default face values come from the pull's address, every other option from the full face logic
OPTIONS = [dict(), dict(inlet_turbulence=0.05, time_step_seed=3), dict(compressible_corr=1), dict(zwall_bc=1),
           dict(zwall_bc=2), dict(ymin_wall_bc=1), dict(transverse_freestream=1, transverse_freestream_blend=0.4)]


@pytest.mark.parametrize("storage", ["f32", "f64"])
@pytest.mark.parametrize("options", OPTIONS, ids=lambda o: "-".join(o) or "default")
@pytest.mark.parametrize("holes", [False, True])
@pytest.mark.parametrize("shape", [(40, 40, 40), (128, 64, 64)])
def test_face_values_match_the_ghost_filled_level(oal, storage, options, holes, shape):
    from openaerolab_alpha_01_b200.solver import Level
    case = sphere_channel_case(*shape, diameter=8.0, centre_x=16.0, re=100.0, **options)
    if holes:
        case = holed(case)
    r = np.random.default_rng(5)
    case.vel = case.vel + 0.01 * r.standard_normal(case.vel.shape) * (case.dom.obstacle == 0)
    case.params.compressible_corr = options.get("compressible_corr", 0)
    got = run(case, storage, STEPS)
    g = Geometry(case.dom)
    L = Level(g, storage=storage)
    L.init_equilibrium(case.rho, case.vel)
    for _ in range(STEPS):
        L.perform_timestep(case.params)
    f, rho, vel = L.state()
    force = L.forces()
    for a, b in zip(got[:3], (f, rho.reshape(-1), vel.reshape(-1))):
        assert np.max(np.abs(a - b)) < TOL[storage] * np.max(np.abs(b))
    assert np.max(np.abs(got[3] - force)) <= 10 * TOL[storage] * max(np.max(np.abs(force)), 1e-2)
    L.close()
    g.close()


class ShortDomain:
    """A block domain whose cell extent ends inside its last blocks."""

    def __init__(self, dom, shape):
        self.dom, self.shape = dom, shape

    def __getattr__(self, name):
        return getattr(self.dom, name)


@pytest.mark.parametrize("storage", ["f32", "f64"])
@pytest.mark.parametrize("shape", [(37, 40, 40), (40, 33, 40), (40, 40, 38), (36, 35, 39)])
def test_face_values_of_extents_inside_a_block(oal, storage, shape):
    from openaerolab_alpha_01_b200.solver import Level
    case = sphere_channel_case(40, 40, 40, diameter=8.0, centre_x=16.0, re=100.0)
    case.dom = ShortDomain(case.dom, shape)
    r = np.random.default_rng(5)
    case.vel = case.vel + 0.01 * r.standard_normal(case.vel.shape) * (case.dom.obstacle == 0)
    case.params.compressible_corr = 0
    got = run(case, storage, STEPS)
    g = Geometry(case.dom)
    L = Level(g, storage=storage)
    L.init_equilibrium(case.rho, case.vel)
    for _ in range(STEPS):
        L.perform_timestep(case.params)
    f, rho, vel = L.state()
    for a, b in zip(got[:3], (f, rho.reshape(-1), vel.reshape(-1))):
        assert np.max(np.abs(a - b)) < TOL[storage] * np.max(np.abs(b))
    L.close()
    g.close()


WIDE = 2 * (2 ** 31 // 26 + 1)  # elements apart: 27 directions, or 27 blocks, span more than 2^32 elements


@pytest.mark.parametrize("svv", [(0.0, 0.0), (0.0, 0.004), (0.003, 0.004)])
@pytest.mark.parametrize("options", [dict(), dict(omega3=1.1, limiter_type=capi.OAL_LIMITER_POSITIVITY)],
                         ids=["default", "general_rates"])
@pytest.mark.parametrize("strides", [dict(dir_stride=WIDE), dict(block_stride=WIDE, dir_stride=512)],
                         ids=["directions", "blocks"])
@pytest.mark.parametrize("storage", ["f32", "f64", "f16", "bf16"])
def test_arrays_past_2_32_elements_keep_their_bits(oal, storage, strides, options, svv):
    """Spans of more than 2^32 elements take the kernels' 64-bit index instances: the same arithmetic, so the
    bits of the compact arrays."""
    import torch
    case = taylor_green_case(24, c_wale=0.2)
    for k, v in options.items():
        setattr(case.params, k, v)
    try:
        want = run(case, storage, 2, svv=svv)
        got = run(case, storage, 2, svv=svv, **strides)
    finally:
        torch.cuda.empty_cache()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
