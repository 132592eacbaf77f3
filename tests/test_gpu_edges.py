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
