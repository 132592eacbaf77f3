"""Kernels at the sizes and values where they can go wrong: edges of their
tiles, remainders, the ends of their ranges.  Discrete results are compared
for equality with the numpy restatement or the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

from oracle.oracle import OracleScene
from taichi_dem_julia_port_gb300 import GlobalData, _abi, scenes
from taichi_dem_julia_port_gb300.config import DEMConfig
from taichi_dem_julia_port_gb300.scenes import ParticleInput

pytestmark = pytest.mark.gpu


def _bucket(pos, lo, cell, H):
    """src/utils.jl:1-2 in numpy: 0-based bucket of each column of pos."""
    m = np.zeros(pos.shape[1], np.int64)
    for c in range(3):
        k = np.ceil((pos[c] - lo[c]) / cell).astype(np.int64) - 1
        for b in range(10):
            m |= ((k >> b) & 1) << (3 * b + c)
    return (m + 1) % H


@pytest.mark.parametrize("H", [1, 1024, 1025, 50_021, 1 << 20])
@pytest.mark.parametrize("n,spread", [(1, "random"), (31, "one"), (4095, "random"),
                                      (4096, "lattice"), (4097, "one"), (20_011, "lattice"),
                                      (300_001, "random"), (1 << 20, "lattice")])
def test_bucket_sort_chunk_edges(gpu, n, spread, H):
    """Chunks of 4,096 particles in warps of 256: remainders, a full last
    chunk, the largest n; every particle in one bucket; coordinates on the
    cells' edges and centres (decided by the exact division)."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + H)
    cell, lo = 0.01, [-0.05, 0.0, 0.02]
    if spread == "random":
        pos = rng.uniform(-0.05, 0.4, (3, n))
    elif spread == "one":
        pos = np.full((3, n), 0.3141)
    else:
        pos = rng.integers(-10, 90, (3, n)) * (cell / 2) + np.array(lo)[:, None]
    p = [torch.tensor(x, device="cuda") for x in pos]
    bucket = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    order = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    lib = _abi.load_library()
    rc = lib.dem_bucket_sort_noalloc(p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(), n,
                                     (C.c_double * 3)(*lo), cell, H, bucket.data_ptr(),
                                     order.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == _abi.DEM_OK
    want = _bucket(pos, lo, cell, H)
    np.testing.assert_array_equal(bucket.cpu().numpy(), want + 1)
    np.testing.assert_array_equal(order.cpu().numpy(), np.argsort(want, kind="stable"))


@pytest.mark.parametrize("mul", [0.999, 1.0, 1.1, 1.25])
@pytest.mark.parametrize("spread", ["touching", "random"])
def test_bond_initialisation_distances(gpu, mul, spread):
    """Bonds join pairs closer than r₀ᵢ + r₀ⱼ, r₀ = mul·r: pairs within a few
    FP64 and FP32 roundings of that distance and pairs anywhere near it, far
    from the domain's origin too, as the oracle joins them."""
    rng = np.random.default_rng(int(mul * 1000))
    n = 1_500
    r = rng.uniform(0.004, 0.01, n)
    side = 12
    k = np.arange(n)
    pos = np.stack([k % side, (k // side) % side, k // side ** 2], axis=1) * 0.05
    # every odd sphere at (about) the bonding distance of the even one before it
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    d = mul * (r[0::2] + r[1::2])
    if spread == "touching":
        d = d * (1.0 + rng.integers(-4, 5, n // 2) * rng.choice([2.0 ** -52, 2.0 ** -24, 2.0 ** -19],
                                                                n // 2))
    else:
        d = d * rng.uniform(0.9, 1.1, n // 2)
    pos[1::2] = pos[0::2] + u[1::2] * d[:, None]
    pos += [3.0, -2.0, 0.0]
    cfg = DEMConfig(domain_min=[-1.0, -4.0, -1.0], domain_max=[5.0, 1.0, 2.0],
                    particle_contact_radius_multiplier=mul, wall_distance=10.0,
                    max_coordinate_number=16)
    p = ParticleInput.from_arrays(r, pos, np.zeros((n, 3)), 2500.0)
    g, o = GlobalData(cfg, p), OracleScene(cfg, p)
    g.initialize()
    o.initialize()
    cg, co = g.contacts(), o.contacts()
    order = np.lexsort((co["j"], co["i"]))
    np.testing.assert_array_equal(cg["i"], np.asarray(co["i"])[order])
    np.testing.assert_array_equal(cg["j"], np.asarray(co["j"])[order])
    assert cg["bonded"].all() and len(cg["i"]) > n // 8
    g.close()


STATE = ("pos", "vel", "omega", "quat", "force", "moment", "wall_shear")
PAIRS = ("i", "j", "active", "bonded", "force", "shear", "torque_i", "torque_j", "point")


def _columns(n, seed=1, **kw):
    """n spheres of 0.5-2 mm in touching columns of ten on the plane, in slow
    motion; every tenth one starts free, above its column."""
    rng = np.random.default_rng(seed)
    r = rng.uniform(0.5e-3, 2e-3, n)
    side = int(np.ceil(np.sqrt(n / 10)))
    k = np.arange(n)
    col, level = k // 10, k % 10
    pos = np.zeros((n, 3))
    pos[:, 0] = (col % side + 0.5) * 4.3e-3
    pos[:, 1] = (col // side + 0.5) * 4.3e-3
    z = 0.999 * r
    for v in range(1, 10):
        at = np.flatnonzero(level == v)
        z[at] = z[at - 1] + 0.999 * (r[at] + r[at - 1])
    z[level == 9] += 3e-3
    pos[:, 2] = z
    vel, omega = rng.normal(0.0, 0.05, (n, 3)), rng.normal(0.0, 5.0, (n, 3))
    cfg = DEMConfig(domain_min=[-0.05] * 3, domain_max=(pos.max(axis=0) + 0.05).tolist(),
                    wall_normal=[0.0, 0.0, -1.0], wall_distance=0.0, dt=2e-7,
                    max_coordinate_number=16, gravity=[0.0, 0.0, -9.81], **kw)
    return cfg, ParticleInput.from_arrays(r, pos, vel, 2500.0), omega


def _result(g):
    c = g.contacts()
    order = np.lexsort((c["j"], c["i"]))
    return g.particles(), {f: np.asarray(v)[order] for f, v in c.items() if f in PAIRS}, g.stats()


def _same(got, want, what):
    for a, b in zip(got[:2], want[:2]):
        assert a.keys() == b.keys()
        for f in a:
            np.testing.assert_array_equal(a[f], b[f], err_msg=f"{what} {f}")


def _run(cfg, p, omega, calls, shape=None, precision="fp64", bonds=False, skin=None):
    with GlobalData(cfg, p, precision=precision) as g:
        if shape:
            g.set_launch_shape(**shape)
        if skin is not None:
            g.set_skin_factor(skin)
        g.set_particles(omega=omega)
        if bonds:
            g.initialize()
        for k in calls:
            g.simulate(k)
        return _result(g)


# warps, blocks of 128, 256 and 512 threads of a cooperative step (152 SMs),
# its largest scene, the list update in a launch of its own and its two
# register budgets, each with a remainder
@pytest.mark.parametrize("n", [1, 31, 32, 33, 4863, 4865, 9729, 38_912, 38_913, 77_825, 155_649])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_step_layouts_agree(gpu, n, precision):
    """The layouts that the sizes choose and the forced ones take the same
    steps, bit for bit, with bonds and without."""
    cfg, p, omega = _columns(n, seed=n)
    for bonds in (False, True):
        want = _run(cfg, p, omega, [9], None, precision, bonds)
        assert n < 100 or len(want[1]["i"]) > n // 2
        for shape in (dict(list_lanes=4, integrate_lanes=4), dict(list_lanes=1, integrate_lanes=1),
                      dict(list_lanes=4, integrate_lanes=1, dependent_launch=1)):
            got = _run(cfg, p, omega, [9], shape, precision, bonds)
            _same(got, want, f"n={n} bonds={bonds} {shape}")


@pytest.mark.parametrize("n", [3001, 50_001])
def test_calls_of_any_length(gpu, n):
    """Steps of a call share launches (up to 64 of a cooperative launch, 8 of
    a graph) and only a call's last step reports: any split of 65 steps gives
    the same state and contacts."""
    cfg, p, omega = _columns(n, seed=2)
    want = _run(cfg, p, omega, [1] * 65)
    for calls in ([65], [64, 1], [8, 8, 49], [7, 9, 17, 32]):
        _same(_run(cfg, p, omega, calls), want, f"{calls}")


def test_touched_bits_follow_the_layout(gpu):
    """Spins, orientations and wall shears written by the caller and by the
    layouts that keep no bits of them are found by the one that does."""
    cfg, p, omega = _columns(500, seed=3)
    rng = np.random.default_rng(4)
    quat = rng.normal(size=(500, 4))
    quat /= np.linalg.norm(quat, axis=1)[:, None]
    still = np.zeros((500, 3))

    def run(shapes):
        with GlobalData(cfg, p) as g:
            for k, shape in enumerate(shapes):
                g.set_launch_shape(**shape)
                g.simulate(3)
                if k == 1:
                    g.set_particles(omega=omega, wall_shear=1e-9 * omega)
                elif k == 3:
                    g.set_particles(omega=still, quat=quat)
                g.simulate(3)
            return _result(g)

    one, four = dict(list_lanes=1, integrate_lanes=1), dict(list_lanes=4, integrate_lanes=4)
    free = dict(list_lanes=0, integrate_lanes=0)
    want = run([four] * 6)
    for shapes in ([one] * 6, [free] * 6, [one, four, one, free, one, one],
                   [free, one, one, four, one, free]):
        _same(run(shapes), want, f"{shapes}")


@pytest.mark.parametrize("n", [31, 33, 320])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_lanes_of_a_warp_that_differ(gpu, n, precision):
    """Warps whose lanes spin or not, touch the plane or not, have partners or
    none and turn at different steps: each lane's bit survives the others'."""
    cfg, p, omega = _columns(n, seed=5)
    k = np.arange(n)
    omega[k % 3 != 0] = 0.0
    p.pos[k % 7 == 0, 2] += 0.5e-3  # off the plane and off their neighbours
    one, four = (_run(cfg, p, omega, [1, 4, 25], dict(list_lanes=m, integrate_lanes=m), precision)
                 for m in (1, 4))
    still = np.all(four[0]["quat"] == [1.0, 0.0, 0.0, 0.0], axis=1)
    assert 0 < still.sum() < n and np.any(four[0]["wall_shear"] != 0.0)
    _same(one, four, f"n={n} {precision}")


@pytest.mark.parametrize("small", [3, 4, 5, 20, 40])
def test_rows_longer_than_a_group(gpu, small):
    """A sphere in contact with more partners than a particle has lanes, and
    lists of more entries."""
    rng = np.random.default_rng(small)
    z, a = np.linspace(-0.9, 0.9, small), np.arange(small) * 2.4
    u = np.stack([np.cos(a) * np.sqrt(1 - z * z), np.sin(a) * np.sqrt(1 - z * z), z], axis=1)
    r = np.concatenate([[5e-3], np.full(small, 6e-4)])
    pos = np.concatenate([[[0.0, 0.0, 0.05]], [0.0, 0.0, 0.05] + u * 0.9995 * 5.6e-3])
    vel = np.concatenate([np.zeros((1, 3)), rng.normal(0.0, 0.5, (small, 3))])
    cfg = DEMConfig(domain_min=[-0.05] * 3, domain_max=[0.05, 0.05, 0.1], wall_distance=0.0,
                    wall_normal=[0.0, 0.0, -1.0], dt=2e-7, max_coordinate_number=64)
    p = ParticleInput.from_arrays(r, pos, vel, 2500.0)
    omega = rng.normal(0.0, 5.0, (small + 1, 3))
    want = _run(cfg, p, omega, [60], skin=0.0)  # a full search in every step
    assert want[2]["contacts_created"] >= small  # (they part again before the last step)
    for shape in (None, dict(list_lanes=4, integrate_lanes=4), dict(list_lanes=1, integrate_lanes=1)):
        _same(_run(cfg, p, omega, [60], shape), want, f"{small} {shape}")


def test_free_components_are_left_alone(gpu):
    """Spheres that nothing touches: components at rest, drifting, with -0
    in position and velocity, across gravity and along it; the integrator that
    leaves out what adds nothing against the one that computes it, as bits."""
    n = 256
    rng = np.random.default_rng(9)
    k = np.arange(n)
    pos = np.stack([k % 8, (k // 8) % 8, 1 + k // 64], axis=1) * 0.01 - [0.04, 0.0, 0.0]
    vals = np.array([0.0, -0.0, 0.25, -1e-3, 5e-324])
    vel = vals[rng.integers(0, 5, (n, 3))]
    vel[:64] = 0.0  # whole warps at rest
    vel[64:96, 0] = -0.0
    pos[128:160, 0] = -0.0
    cfg = DEMConfig(domain_min=[-0.05] * 3, domain_max=[0.1, 0.1, 0.1], wall_distance=0.0,
                    wall_normal=[0.0, 0.0, -1.0], dt=2e-7, max_coordinate_number=16,
                    gravity=[0.0, 0.0, -9.81])
    p = ParticleInput.from_arrays(np.full(n, 1e-3), pos, vel, 2500.0)
    for precision in ("fp64", "fp32"):
        got, want = (_run(cfg, p, np.zeros((n, 3)), [1, 6], dict(list_lanes=m, integrate_lanes=m),
                          precision)[0] for m in (1, 4))
        for f in STATE:
            np.testing.assert_array_equal(got[f].view(np.int64), want[f].view(np.int64), err_msg=f)


@pytest.mark.parametrize("n", [10, 1000, 40_000])
def test_not_a_number_asks_for_no_search(gpu, n):
    """A sphere that meets the plane without tangential motion gets NaN
    coordinates from the wall law; with neighbour lists the others go on as
    with a full search in every step, and the lists are kept."""
    cfg, p, omega = _columns(n, seed=6)
    p.pos[9] = [-0.03, -0.03, np.cbrt(0.75 * p.volume[9] / np.pi) + 1e-9]
    p.vel[9] = [0.0, 0.0, -0.01]
    omega[9] = 0.0
    steps = 200
    full, lists = (_run(cfg, p, omega, [steps], skin=s) for s in (0.0, 0.9))
    assert np.isnan(full[0]["pos"][9]).any() and np.isfinite(full[0]["pos"][:9]).all()
    _same(lists, full, f"n={n}")
    assert full[2]["full_searches"] == steps
    assert lists[2]["full_searches"] < steps // 4


@pytest.mark.parametrize("n", [2000, 40_000, 80_000])
def test_many_not_a_numbers_share_no_list(gpu, n):
    """More spheres with NaN coordinates than a neighbour list holds: a full
    search that finds them together in one bucket puts none on another's list,
    so the others go on as with a search in every step, and search as often as
    they do beside 40 spheres that have not landed."""
    nan, k = np.arange(9, 409, 10), np.arange(40)

    def run(gap, skin):
        cfg, p, omega = _columns(n, seed=8)
        r = np.cbrt(0.75 * p.volume[nan] / np.pi)
        p.pos[nan] = np.stack([-0.045 + 5e-3 * (k % 8), -0.045 + 5e-3 * (k // 8), r + gap], axis=1)
        p.vel[nan] = [0.0, 0.0, -0.01]
        omega[nan] = 0.0
        with GlobalData(cfg, p) as g:
            g.set_skin_factor(skin)
            g.set_particles(omega=omega)
            g.simulate(200)
            assert np.isnan(g.particles()["pos"][nan]).any(axis=1).all() == (gap < 1e-6)
            g.set_skin_factor(skin)  # the lists are built again
            before = g.stats()["full_searches"]
            g.simulate(60)
            return _result(g), g.stats()["full_searches"] - before

    (full, every), (lists, few), (_, beside) = run(1e-9, 0.0), run(1e-9, 0.9), run(1e-3, 0.9)
    _same(lists, full, f"n={n}")
    assert every == 60 and few == beside < 60


@pytest.mark.parametrize("n", [2000, 17_576])
def test_other_streams_get_their_turn(gpu, n):
    """A small kernel on a caller's own stream does not wait for dozens of
    steps of a scene that fills the GPU."""
    torch = pytest.importorskip("torch")
    import time
    cfg, p, omega = _columns(n, seed=10)
    x, s = torch.zeros(4096, device="cuda"), torch.cuda.Stream()
    with GlobalData(cfg, p) as g:
        step = g.simulate_timed(512) / 512 * 1e-3
        waits = []
        for _ in range(5):
            g.simulate(1000)
            for _ in range(4):
                t = time.perf_counter()
                with torch.cuda.stream(s):
                    x.add_(1.0)
                s.synchronize()
                waits.append(time.perf_counter() - t)
            g.sync()
    # the 16 steps of the launch in flight, as much again for the host's calls
    assert np.median(waits) < 32 * step + 1e-4, (np.median(waits), step)


@pytest.mark.parametrize("n", [2000, 7000, 17_576])
def test_two_handles_step_at_once(gpu, n):
    """Two threads, each stepping its own scene: as each alone."""
    import threading
    made = [_columns(n, seed=s) for s in (11, 12)]
    want = [_run(*m, [40, 40, 40]) for m in made]
    got = [None, None]

    def work(k):
        got[k] = _run(*made[k], [40, 40, 40])

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(got, want):
        _same(a, b, f"n={n}")
