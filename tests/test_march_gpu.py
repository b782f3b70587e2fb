"""The marching launchers (adjoint derivatives, density gradient, type1 adjoint)
at the edges of their tiles and chunks: extents around 32 columns and 16 rows,
chunks of 1 to 3 planes (small grids) and of 13 with a remainder (91 tiles x 37
planes), single cells, and ranges inside a larger allocation, against the oracle.  Tolerance: FP32 rounding of one kernel's sums, the same
2e-6 relative L2 as the other launcher tests."""
import numpy as np
import pytest

import miniappsforhpe_b200 as P
from oracle import Layout, Oracle
from tests.helpers import random_field, random_model, rel_l2, sponge_ab

H, DT, TOL = (10.0, 12.5, 8.0), 1e-3, 2e-6
DK = ("d1x", "d1y", "d1z", "d2x", "d2y", "d2z")
DIMS = ((1, 1, 1), (31, 15, 7), (32, 16, 8), (33, 17, 9), (65, 3, 130), (5, 50, 16), (40, 33, 17),
        (48, 40, 41), (200, 200, 37))


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def setup(dims):
    lay, rng = Layout(*dims), np.random.default_rng(sum(dims))
    return lay, random_model(lay, rng), [random_field(lay, rng) for _ in range(10)], rng


@pytest.mark.gpu
@pytest.mark.parametrize("dims", DIMS)
def test_adjoint_derivatives(dims):
    lay, m, f, _ = setup(dims)
    want = {k: lay.zeros() for k in DK}
    r3, r4 = lay.zeros(), lay.zeros()
    Oracle("f32").adj_drv(lay, want, r3, r4, f[0], f[1], m, H)
    t = {k: dev(v) for k, v in m.items()}
    d, g3, g4 = {k: dev(lay.zeros()) for k in DK}, dev(lay.zeros()), dev(lay.zeros())
    inv = [1 / h for h in H]
    P.launch_adj_kernel2_drv(d["d1x"], d["d2x"], d["d1y"], d["d2y"], d["d1z"], d["d2z"], g3, g4, dev(f[0]), dev(f[1]),
                             t["irho"], t["m1"], t["m2"], t["m3"], t["m4"], t["rx"], t["ry"], t["rz"], *lay.ranges,
                             inv[0] ** 2, inv[1] ** 2, inv[2] ** 2, inv[0] * inv[1] / 4, inv[1] * inv[2] / 4,
                             inv[2] * inv[0] / 4, lay.ldimx, lay.ldimy, 8, DT, *inv)
    for k in DK:  # cells outside the range stay as they were (zero in both)
        assert rel_l2(d[k].cpu().numpy(), want[k]) < TOL, k
    assert rel_l2(g3.cpu().numpy(), r3) < TOL and rel_l2(g4.cpu().numpy(), r4) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("dims", DIMS)
def test_density_gradient(dims):
    lay, m, f, rng = setup(dims)
    fd = dict(zip(DK, f[2:8]))
    start = rng.standard_normal((lay.nz, lay.ny, lay.nx)).astype(np.float32)
    want = start.copy()
    Oracle("f32").rho_gradient(lay, want, fd, f[0], f[1], m, H, lay.nx, lay.ny)
    got, t, d = dev(start), {k: dev(v) for k, v in m.items()}, {k: dev(v) for k, v in fd.items()}
    P.launch_update_rho_gradient_rho(got, d["d1x"], d["d2x"], d["d1y"], d["d2y"], d["d1z"], d["d2z"], dev(f[0]),
                                     dev(f[1]), t["irho"], t["m1"], t["m2"], t["m3"], t["m4"], t["rx"], t["ry"],
                                     t["rz"], *lay.ranges, lay.ldimx, lay.ldimy, lay.nx, lay.ny, *H)
    assert rel_l2(got.cpu().numpy(), want) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("sponge", [False, True])
@pytest.mark.parametrize("dims", DIMS)
def test_type1_adjoint(dims, sponge):
    lay, m, f, rng = setup(dims)
    ab = [sponge_ab(n, rng) for n in (lay.ldimx, lay.ldimy, lay.ldimz)]
    w3, w4 = f[2].copy(), f[3].copy()
    Oracle("f32").t1_adj(lay, w3, w4, f[0], f[1], m, ab, np.float32(DT), H, sponge)
    o3, o4 = dev(f[2]), dev(f[3])
    P.launch_type1_adj(o3, o4, dev(f[0]), dev(f[1]), *[dev(m[k]) for k in ("m1", "m2", "m3", "m4", "rx", "ry", "rz")],
                       *[dev(a) for a in ab], *lay.ranges, lay.ldimx, lay.ldimy, lay.ldimz, DT, *H, use_sponge=sponge)
    for got, want in ((o3, w3), (o4, w4)):
        assert rel_l2(got.cpu().numpy(), want) < TOL


@pytest.mark.gpu
def test_a_range_inside_the_allocation_leaves_the_rest_alone():
    lay, m, f, _ = setup((50, 40, 30))
    r = (10, 40, 7, 23, 9, 20)
    full, part = [], []
    t = {k: dev(v) for k, v in m.items()}
    inv = [1 / h for h in H]
    for ranges, out in ((lay.ranges, full), (r, part)):
        out.extend(dev(np.full(lay.shape, 7.0, np.float32)) for _ in range(8))
        P.launch_adj_kernel2_drv(*out, dev(f[0]), dev(f[1]), t["irho"], t["m1"], t["m2"], t["m3"], t["m4"], t["rx"],
                                 t["ry"], t["rz"], *ranges, 1, 1, 1, inv[0] * inv[1] / 4, inv[1] * inv[2] / 4,
                                 inv[2] * inv[0] / 4, lay.ldimx, lay.ldimy, 8, DT, *inv)
    inside = (slice(r[4], r[5] + 1), slice(r[2], r[3] + 1), slice(r[0], r[1] + 1))
    for a, b in zip(full, part):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        np.testing.assert_array_equal(a[inside], b[inside])
        b[inside] = 7.0
        assert np.all(b == 7.0)
