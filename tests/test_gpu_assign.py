"""GPU mass assignment vs the oracle (through the C ABI).

Bar: sort keys and NGP counts bit-exact; CIC/TSC (and weighted NGP) meshes
within 1e-5 per cell relative to the FP64 oracle (cells below one
particle's mass judged against one particle's mass); bitwise determinism
across runs and particle orders.
"""
import numpy as np
import pytest

import oracle as orc
from conftest import rel_err_cells
from cosmicatlas_b200 import synth
from cosmicatlas_b200.api import CIC, F32, F64, NGP, TSC, CamError, make_grid

pytestmark = pytest.mark.gpu

SCHEMES = [NGP, CIC, TSC]


def edge_positions(box, n):
    """Positions on and around cell edges and box faces."""
    f = np.float32
    d = f(box) / f(n)
    base = [0.0, np.nextafter(f(box), f(0)), box, -1e-4, box + 1e-3, d, np.nextafter(d, f(0)),
            0.5 * d, np.nextafter(f(0.5) * d, f(0)), box - 0.5 * d, 3 * d, np.nan]
    return np.array(base, np.float32)


def mixed_inputs(n, box, npart, seed):
    x, y, z = synth.clumped(npart, box, max(npart // 50, 1), 1.0 * box / n, 0.8, seed)
    e = edge_positions(box, n)
    k = len(e)
    x[:k] = e
    y[k:2 * k] = e
    z[2 * k:3 * k] = e
    x[3 * k:4 * k] = e
    y[3 * k:4 * k] = e[::-1]
    return x, y, z


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("n,box", [(64, 1000.0), (48, 777.7), (17, 100.0)])
def test_keys_bit_exact(ctx, scheme, n, box):
    x, y, z = mixed_inputs(n, box, 100_000, seed=n)
    g = make_grid(n, box)
    got = ctx.cell_keys(x, y, z, g, scheme)
    want = orc.keys(scheme, x, y, z, orc.Grid.cubic(n, box))
    assert np.array_equal(got, want)


def test_keys_non_cubic_with_origin(ctx):
    rng = np.random.default_rng(5)
    n, L, mn = (32, 48, 20), (300.0, 450.0, 200.0), (-10.0, 5.0, 100.0)
    x = rng.uniform(mn[0] - 5, mn[0] + L[0] + 5, 50_000).astype(np.float32)
    y = rng.uniform(mn[1] - 5, mn[1] + L[1] + 5, 50_000).astype(np.float32)
    z = rng.uniform(mn[2] - 5, mn[2] + L[2] + 5, 50_000).astype(np.float32)
    g = make_grid(n, L, None, mn)
    og = orc.Grid(n, L, tuple(g.d), mn)
    for s in SCHEMES:
        assert np.array_equal(ctx.cell_keys(x, y, z, g, s), orc.keys(s, x, y, z, og))


@pytest.mark.parametrize("n,box", [(128, 1000.0), (192, 1500.0)])
def test_ngp_counts_bit_exact(ctx, n, box):
    x, y, z = mixed_inputs(n, box, 400_000, seed=7)
    g = make_grid(n, box)
    r = ctx.count_ngp(x, y, z, g)
    k = orc.keys(NGP, x, y, z, orc.Grid.cubic(n, box))
    want = np.bincount(k[k < n ** 3], minlength=n ** 3).reshape(n, n, n).astype(np.uint32)
    assert np.array_equal(r.mesh, want)
    assert r.n_lost == int((k == n ** 3).sum())
    assert r.n_in + r.n_lost == x.size


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("precision", [F32, F64])
def test_mesh_vs_oracle(ctx, scheme, weighted, precision):
    n, box = 64, 1000.0
    x, y, z = mixed_inputs(n, box, 300_000, seed=11)
    w = synth.halo_masses(x.size, seed=3) if weighted else None
    g = make_grid(n, box)
    r = ctx.assign(x, y, z, w, g, scheme, precision)
    ref, lost = orc.assign_f64(scheme, x, y, z, w, orc.Grid.cubic(n, box))
    assert r.n_lost == lost
    err = rel_err_cells(r.mesh, ref, 1.0 if w is None else float(np.mean(w)))
    assert err <= 1e-5, err
    assert abs(r.sum_mesh - ref.sum()) <= 1e-9 * ref.sum()


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("n", [2, 3, 4, 5, 7, 33, 35])
def test_small_and_ragged_meshes(ctx, scheme, n):
    # meshes smaller than a brick, and meshes whose last brick is partial
    box = 10.0 * n
    x, y, z = mixed_inputs(n, box, 20_000, seed=n)
    g = make_grid(n, box)
    r = ctx.assign(x, y, z, None, g, scheme, F64)
    ref, lost = orc.assign_f64(scheme, x, y, z, None, orc.Grid.cubic(n, box))
    assert r.n_lost == lost
    assert rel_err_cells(r.mesh, ref, 1.0) <= 1e-5


def test_non_cubic_mesh(ctx):
    rng = np.random.default_rng(9)
    n, L, mn = (40, 24, 56), (400.0, 240.0, 560.0), (0.0, 0.0, 0.0)
    x = rng.uniform(0, L[0], 80_000).astype(np.float32)
    y = rng.uniform(0, L[1], 80_000).astype(np.float32)
    z = rng.uniform(0, L[2], 80_000).astype(np.float32)
    g = make_grid(n, L, None, mn)
    for s in SCHEMES:
        r = ctx.assign(x, y, z, None, g, s, F32)
        ref, lost = orc.assign_f64(s, x, y, z, None, orc.Grid(n, L, tuple(g.d), mn))
        assert rel_err_cells(r.mesh, ref, 1.0) <= 1e-5


def test_empty_and_all_lost(ctx):
    g = make_grid(32, 100.0)
    e = np.zeros(0, np.float32)
    r = ctx.assign(e, e, e, None, g, CIC, F32)
    assert r.n_in == 0 and r.n_lost == 0 and not np.any(r.mesh)
    far = np.full(1000, 1e6, np.float32)
    r = ctx.assign(far, far, far, None, g, TSC, F32)
    assert r.n_lost == 1000 and not np.any(r.mesh)


@pytest.mark.parametrize("scheme", SCHEMES)
def test_bitwise_deterministic(ctx, scheme):
    n, box = 96, 1000.0
    x, y, z = synth.clumped(500_000, box, 2_000, 3.0, 0.8, seed=21)
    w = synth.halo_masses(x.size, seed=22)
    g = make_grid(n, box)
    a = ctx.assign(x, y, z, w, g, scheme, F32).mesh
    b = ctx.assign(x, y, z, w, g, scheme, F32).mesh
    # same particles in a different order: same integer sums, same bits
    p = np.random.default_rng(1).permutation(x.size)
    c = ctx.assign(x[p], y[p], z[p], w[p], g, scheme, F32).mesh
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert np.array_equal(a.view(np.uint32), c.view(np.uint32))


@pytest.mark.parametrize("scheme", SCHEMES)
def test_signed_weights_vs_oracle(ctx, scheme):
    # some negative weights: the deposit's signed fixed-point path
    n, box = 64, 1000.0
    x, y, z = mixed_inputs(n, box, 300_000, seed=41)
    w = synth.halo_masses(x.size, seed=42)
    w[np.random.default_rng(43).random(x.size) < 0.2] *= -1.0
    g = make_grid(n, box)
    r = ctx.assign(x, y, z, w, g, scheme, F64)
    ref, lost = orc.assign_f64(scheme, x, y, z, w, orc.Grid.cubic(n, box))
    assert r.n_lost == lost
    err = rel_err_cells(r.mesh, ref, float(np.mean(np.abs(w))))
    assert err <= 1e-5, err


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("n", [96, 32])
def test_many_particles_vs_oracle(ctx, scheme, n):
    # 4.5 M weighted particles (clumped, plus the edge positions).  At n = 32
    # the bricks shrink to 4 x 4 x 32 cells, so TSC stencils cross brick
    # faces for most particles (several payload records per particle).
    box = 1000.0
    x, y, z = mixed_inputs(n, box, 4_500_000, seed=31 + n)
    w = synth.halo_masses(x.size, seed=32)
    g = make_grid(n, box)
    r = ctx.assign(x, y, z, w, g, scheme, F32)
    ref, lost = orc.assign_f64(scheme, x, y, z, w, orc.Grid.cubic(n, box))
    assert r.n_lost == lost
    err = rel_err_cells(r.mesh, ref, float(np.mean(w)))
    assert err <= 1e-5, err
    p = np.random.default_rng(2).permutation(x.size)
    c = ctx.assign(x[p], y[p], z[p], w[p], g, scheme, F32).mesh
    assert np.array_equal(r.mesh.view(np.uint32), c.view(np.uint32))


def test_device_arrays_roundtrip(ctx):
    import torch
    n, box = 64, 500.0
    x, y, z = synth.clumped(100_000, box, 500, 2.0, 0.8, seed=4)
    g = make_grid(n, box)
    host = ctx.assign(x, y, z, None, g, CIC, F32).mesh
    dx, dy, dz = (torch.from_numpy(v).cuda() for v in (x, y, z))
    dev = ctx.assign(dx, dy, dz, None, g, CIC, F32).mesh
    assert dev.is_cuda
    assert np.array_equal(dev.cpu().numpy(), host)


def test_nonfinite_weight_rejected(ctx):
    x = np.array([1.0, 2.0], np.float32)
    w = np.array([1.0, np.inf], np.float32)
    with pytest.raises(CamError) as e:
        ctx.assign(x, x, x, w, make_grid(8, 10.0), CIC, F32)
    assert e.value.code == -8


def test_invalid_arguments(ctx):
    x = np.ones(4, np.float32)
    with pytest.raises(CamError) as e:
        ctx.assign(x, x, x, None, make_grid(8, 10.0), 7, F32)
    assert e.value.code == -1
    g = make_grid(8, 10.0)
    g.L[0] = -1.0
    with pytest.raises(CamError) as e:
        ctx.assign(x, x, x, None, g, CIC, F32)
    assert e.value.code == -1


# ---- against the reference's own getDensity_* (golden fixture) ------------
def _golden():
    import os
    return np.load(os.path.join(os.path.dirname(__file__), "golden", "getdensity_ref.npz"))


@pytest.mark.parametrize("case", ["bulk", "shift", "edges"])
def test_ngp_counts_equal_reference_getdensity(ctx, case):
    # counts bit-exact against the meshes the reference's getDensity_NGP wrote
    G = _golden()
    n, L, mn = G[f"{case}_grid"]
    n = int(n)
    g = make_grid(n, float(L), None, float(mn))
    got = ctx.count_ngp(G[f"{case}_x"], G[f"{case}_y"], G[f"{case}_z"], g).mesh
    assert np.array_equal(np.asarray(got).astype(np.float32), G[f"{case}_ngp_unit"])


@pytest.mark.parametrize("case", ["bulk", "shift"])
@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("weighted", [False, True])
def test_mesh_vs_reference_getdensity(ctx, case, scheme, weighted):
    # within 1e-5 per cell of the reference's own float meshes
    G = _golden()
    n, L, mn = G[f"{case}_grid"]
    g = make_grid(int(n), float(L), None, float(mn))
    w = G[f"{case}_w"] if weighted else None
    got = ctx.assign(G[f"{case}_x"], G[f"{case}_y"], G[f"{case}_z"], w, g, scheme, F32).mesh
    want = G[f"{case}_{('ngp', 'cic', 'tsc')[scheme]}_{'mass' if weighted else 'unit'}"]
    unit = float(np.mean(w, dtype=np.float64)) if weighted else 1.0
    assert rel_err_cells(got, want, unit) <= 1e-5


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("n", [96, 384])
def test_unaligned_arrays_and_lost_particles_vs_oracle(ctx, scheme, n):
    # device arrays off the 16-byte boundary (scalar loads instead of
    # float4) and particles outside the box (counted as lost, never
    # written): the scatter takes exactly the particles its count pass
    # counted
    import torch
    box = 500.0
    rng = np.random.default_rng(n + scheme)
    npart = 400_001
    buf = rng.uniform(0.0, box, size=(4, npart + 1)).astype(np.float32)
    # every tenth particle anywhere in [-1.5 L, 2.5 L): outside the box even
    # after CIC's one periodic wrap
    buf[:3, ::10] = rng.uniform(-1.5 * box, 2.5 * box, size=(3, buf[:, ::10].shape[1])).astype(np.float32)
    buf[3] = rng.lognormal(0.0, 1.0, npart + 1).astype(np.float32)
    dbuf = torch.from_numpy(buf).cuda()
    xd, yd, zd, wd = dbuf[0, 1:], dbuf[1, 1:], dbuf[2, 1:], dbuf[3, 1:]
    assert xd.data_ptr() % 16 != 0
    x, y, z, w = buf[0, 1:], buf[1, 1:], buf[2, 1:], buf[3, 1:]
    a = ctx.assign(xd, yd, zd, wd, make_grid(n, box), scheme, F32)
    am = a.mesh.cpu().numpy()
    ref, lost = orc.assign_f64_mt(scheme, x, y, z, w, orc.Grid.cubic(n, box))
    assert a.n_lost == lost and lost > 0
    assert rel_err_cells(am, ref, float(np.mean(w, dtype=np.float64))) <= 1e-5


@pytest.mark.parametrize("scheme", [CIC, TSC])
def test_mesh_384_vs_oracle(ctx, scheme):
    # 384^3 (6,912 bricks: the count histogram and scan of a larger mesh)
    n, box = 384, 1000.0
    x, y, z = synth.clumped(3_000_000, box, 30_000, 2.0, 0.8, seed=77 + scheme)
    w = synth.halo_masses(x.size, seed=78)
    got = ctx.assign(x, y, z, w, make_grid(n, box), scheme, F32)
    ref, lost = orc.assign_f64_mt(scheme, x, y, z, w, orc.Grid.cubic(n, box))
    assert got.n_lost == lost
    assert rel_err_cells(got.mesh, ref, float(np.mean(w, dtype=np.float64))) <= 1e-5


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("signed", [False, True])
@pytest.mark.parametrize("n", [(1, 5, 33), (16, 1, 64), (2, 40, 31), (17, 34, 65), (3, 3, 3)])
def test_deposit_tile_edges(ctx, scheme, signed, n):
    # axes that one brick spans (the tile's halo is folded back, down to one
    # cell per axis), bricks of 2 and 15 cells, rows of 2 to 32 cells, both
    # forms of the deposit (signed weights take the general one)
    rng = np.random.default_rng(100 * n[0] + n[2] + scheme)
    L = tuple(10.0 * k for k in n)
    npart = 20_000
    xs = [rng.uniform(0.0, side, npart).astype(np.float32) for side in L]
    for a in range(3):
        e = edge_positions(L[a], n[a])
        xs[a][a * 20:a * 20 + len(e)] = e
    w = synth.halo_masses(npart, seed=12) if signed else None
    if signed:
        w[::3] *= -1.0
    g = make_grid(n, L)
    r = ctx.assign(*xs, w, g, scheme, F64)
    ref, lost = orc.assign_f64(scheme, *xs, w, orc.Grid(n, L, tuple(g.d), (0.0, 0.0, 0.0)))
    assert r.n_lost == lost
    unit = 1.0 if w is None else float(np.mean(np.abs(w)))
    assert rel_err_cells(r.mesh, ref, unit) <= 1e-5


@pytest.mark.parametrize("n,box,mn", [(33, 777.7, 0.0), (400, 1000.0, 0.0), (100, 313.1, -40.0), (96, 250.0, 17.5)])
def test_cells_next_to_every_face(ctx, n, box, mn):
    # positions within three float steps of every cell face: the common-case
    # floor, the exact quotient beside faces and the periodic images must give
    # the oracle's keys (NGP counts) and meshes
    f = np.float32
    d = f(f(box) / f(n))
    face = (np.arange(n + 1, dtype=np.float64) * float(d) + mn).astype(f)
    steps = [face]
    for toward in (f(-np.inf), f(np.inf)):
        v = face
        for _ in range(3):
            v = np.nextafter(v, toward)
            steps.append(v)
    x = np.concatenate(steps + [(face + f(0.5) * d).astype(f), (face + f(0.25) * d).astype(f)])
    rng = np.random.default_rng(n)
    y, z = (rng.permutation(x) for _ in range(2))
    g = make_grid(n, box, None, mn)
    og = orc.Grid((n,) * 3, (box,) * 3, tuple(g.d), (mn,) * 3)
    r = ctx.count_ngp(x, y, z, g)
    k = orc.keys(NGP, x, y, z, og)
    assert np.array_equal(r.mesh.reshape(-1), np.bincount(k[k < n ** 3], minlength=n ** 3).astype(np.uint32))
    for s in (CIC, TSC):
        a = ctx.assign(x, y, z, None, g, s, F64)
        ref, lost = orc.assign_f64(s, x, y, z, None, og)
        assert a.n_lost == lost
        assert rel_err_cells(a.mesh, ref, 1.0) <= 1e-5


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("weighted", [False, True])
def test_two_level_sort_vs_oracle(ctx, scheme, weighted):
    # 384 x 320 x 400 cells are more bricks than one tile counts, and 1.2 M
    # particles enough for the two-level sort: clumps, cell and box faces,
    # particles outside the box (their own bin) and NaN positions
    n, L = (384, 320, 400), (960.0, 800.0, 1000.0)
    npart = 1_200_007
    rng = np.random.default_rng(50 + scheme)
    xs = [rng.uniform(-0.02 * s, 1.02 * s, npart).astype(np.float32) for s in L]
    xs[0][: npart // 2] = (xs[0][: npart // 2] * 0.1).astype(np.float32)  # a dense slab
    for a in range(3):
        e = edge_positions(L[a], n[a])
        xs[a][a * 20:a * 20 + len(e)] = e
    w = synth.halo_masses(npart, seed=51) if weighted else None
    g = make_grid(n, L)
    r = ctx.assign(*xs, w, g, scheme, F32)
    ref, lost = orc.assign_f64_mt(scheme, *xs, w, orc.Grid(n, L, tuple(g.d), (0.0, 0.0, 0.0)))
    assert r.n_lost == lost and lost > 0
    assert rel_err_cells(r.mesh, ref, 1.0 if w is None else float(np.mean(w, dtype=np.float64))) <= 1e-5
    p = rng.permutation(npart)
    again = ctx.assign(*(v[p] for v in xs), None if w is None else w[p], g, scheme, F32)
    assert np.array_equal(r.mesh.view(np.uint32), again.mesh.view(np.uint32))


@pytest.mark.parametrize("scheme", [NGP, TSC])
def test_many_super_bricks_too_clumped_for_slabs(scheme):
    # 768^3 sorts by more than 128 super-bricks; a catalogue whose fullest
    # brick no slab holds is sorted in two levels once and counted in one
    # after that: the same mesh, bit for bit
    import torch
    from cosmicatlas_b200.api import Context
    n, L, npart = 768, 1000.0, 1_100_003
    gen = torch.Generator(device="cuda").manual_seed(scheme + 1)
    xs = [torch.rand(npart, device="cuda", generator=gen) * (40.0 if a else 1000.0) for a in range(3)]
    c = Context()
    try:
        g = make_grid(n, L)
        c.profile(True)
        c.profile_read(True)
        first = c.assign(*xs, None, g, scheme, F32)
        assert "assign_super_sort" in c.profile_read(True)
        again = c.assign(*xs, None, g, scheme, F32)
        names = c.profile_read(True)
        assert "assign_super_sort" not in names and "assign_bin_count" in names
        assert first.n_lost == again.n_lost and first.sum_mesh == again.sum_mesh
        assert np.array_equal(np.asarray(first.mesh.cpu()), np.asarray(again.mesh.cpu()))
    finally:
        c.close()


@pytest.mark.parametrize("mn", [0.0, 12.5])
@pytest.mark.parametrize("n,box,d", [(256, 505.0, 1.97265), (256, 505.0, 1.97266), (64, 1000.0, 15.62494),
                                     (64, 1000.0, 15.62506), (130, 777.7, 5.98232)])
def test_cell_size_off_box_over_cells(ctx, n, box, d, mn):
    # a cell size of one to four parts in 10^6 off L/N, as a caller that
    # rounds it passes: positions in and around the first and the last half
    # cell, where CIC takes periodic images, and anywhere
    f = np.float32
    rng = np.random.default_rng(n)
    edge = np.concatenate([rng.uniform(0.0, 1.0, 20_000), 0.5 + rng.uniform(-2e-3, 2e-3, 20_000),
                           n + rng.uniform(-1.0, 0.0, 20_000), n - 0.5 + rng.uniform(-2e-3, 2e-3, 20_000)]) * d
    x = (np.concatenate([edge, rng.uniform(0.0, box, 40_000)]) + mn).astype(f)
    y, z = (rng.permutation(x) for _ in range(2))
    g = make_grid(n, box, d, mn)
    og = orc.Grid((n,) * 3, (box,) * 3, tuple(g.d), (mn,) * 3)
    for s in SCHEMES:
        a = ctx.assign(x, y, z, None, g, s, F64)
        ref, lost = orc.assign_f64_mt(s, x, y, z, None, og)
        assert a.n_lost == lost
        assert rel_err_cells(a.mesh, ref, 1.0) <= 1e-5


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("n", [(61, 61, 61), (49, 49, 49), (13, 25, 64), (37, 10, 33), (85, 73, 31)])
def test_small_bricks_with_one_cell_left(ctx, scheme, n):
    # particles enough to make the bricks 4 or 3 cells along axes that either
    # leaves one cell of: a TSC stencil would span three bricks there
    box = 1000.0
    npart = 1_300_000
    rng = np.random.default_rng(n[0])
    x, y, z = (rng.uniform(0.0, box, npart).astype(np.float32) for _ in range(3))
    x[:npart // 4] *= np.float32(0.02)  # and the cells beside the box face
    y[npart // 8:npart // 2] = np.float32(box) - y[npart // 8:npart // 2] * np.float32(0.03)
    g = make_grid(n, box)
    r = ctx.assign(x, y, z, None, g, scheme, F64)
    ref, lost = orc.assign_f64_mt(scheme, x, y, z, None, orc.Grid(n, (box,) * 3, tuple(g.d), (0.0,) * 3))
    assert r.n_lost == lost
    assert abs(r.sum_mesh - (npart - lost)) <= 1e-9 * npart
    assert rel_err_cells(r.mesh, ref, 1.0) <= 1e-5


@pytest.mark.parametrize("n,npart", [(64, 200_000), (416, 1_200_000)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_nonfinite_weight_leaves_the_mesh(n, npart, bad):
    # the caller's device mesh is not written before the weights are refused:
    # exact and slab runs, one and two levels, with and without an overflow
    import torch
    from cosmicatlas_b200.api import Context
    gen = torch.Generator(device="cuda").manual_seed(n)
    xs = [torch.rand(npart, device="cuda", generator=gen) * 100.0 for _ in range(3)]
    w = torch.ones(npart, device="cuda")
    wrong = w.clone()
    wrong[npart // 2] = float(bad)
    clumped = [v * 0.1 for v in xs]
    c = Context()
    try:
        g = make_grid(n, 100.0)
        mesh = torch.full((n, n, n), -7.0, device="cuda")
        for pos in (xs, xs, clumped):
            with pytest.raises(CamError) as e:
                c.assign(*pos, wrong, g, CIC, F32, out=mesh)
            assert e.value.code == -8
            assert bool((mesh == -7.0).all())
            if pos is xs:
                c.assign(*xs, w, g, CIC, F32)  # measures the slabs of the calls after it
        c.assign(*xs, w, g, CIC, F32, out=mesh)
        assert abs(float(mesh.double().sum()) - npart) <= 1e-5 * npart
    finally:
        c.close()


def _deposits(c, call):
    """(result, deposit launches) of one call: two when it ran again exactly."""
    c.profile(True)
    c.profile_read(True)
    r = call()
    n = c.profile_read(True)["assign_deposit"][0]
    c.profile(False)
    return r, n


def _layered(npart, box, period, seed):
    """Uniform in x and z, the lower half of every `period` along y."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    xs = [torch.rand(npart, device="cuda", generator=gen) * box for _ in range(3)]
    xs[1] = (xs[1] / period).floor() * period + (xs[1] % period) * 0.5
    return xs


def test_slabs_are_kept_by_brick_extent():
    # layers 8 cells apart: even over bricks of 8 cells, which a million
    # particles get, twice the mean in every second brick of 4, which five
    # million get.  Calls of both in turn settle on slabs for the one and
    # exact counts for the other, none runs twice.
    from cosmicatlas_b200.api import Context
    n, box = 64, 64.0
    few, many = _layered(1_050_000, box, 8.0, 1), _layered(5_000_000, box, 8.0, 2)
    g = make_grid(n, box)
    c = Context()
    try:
        runs = [_deposits(c, lambda: c.assign(*xs, None, g, NGP, F32))[1] for _ in range(5) for xs in (few, many)]
        assert runs[4:] == [1] * 6, runs
    finally:
        c.close()


@pytest.mark.parametrize("n,npart", [(64, 1_050_000), (384, 1_200_000)])
def test_alternating_catalogues_run_once(n, npart):
    # a smooth and a clumped catalogue of one mesh in turn (one level of
    # sorting and two): after the first pair none runs twice; once only
    # smooth ones come, slabs are used again
    import torch
    from cosmicatlas_b200.api import Context
    gen = torch.Generator(device="cuda").manual_seed(n)
    smooth = [torch.rand(npart, device="cuda", generator=gen) * 100.0 for _ in range(3)]
    clumped = [v.clone() for v in smooth]
    clumped[0][: npart // 2] *= 0.125
    g = make_grid(n, 100.0)
    c = Context()
    try:
        runs = [_deposits(c, lambda: c.assign(*xs, None, g, NGP, F32))[1] for _ in range(5) for xs in (smooth, clumped)]
        assert runs[2:] == [1] * 8, runs
        for _ in range(6):
            c.assign(*smooth, None, g, NGP, F32)
        c.profile(True)
        c.profile_read(True)
        c.assign(*smooth, None, g, NGP, F32)
        assert "assign_bin_count" not in c.profile_read(True)
    finally:
        c.close()


def test_super_bricks_are_measured_again():
    # 768^3 sorts by more than 128 super-bricks: after clumped catalogues,
    # which run exactly in one level, smooth ones come back to slabs
    import torch
    from cosmicatlas_b200.api import Context
    n, npart = 768, 4_000_000
    gen = torch.Generator(device="cuda").manual_seed(5)
    smooth = [torch.rand(npart, device="cuda", generator=gen) * 1000.0 for _ in range(3)]
    clumped = [smooth[0] * 0.04, smooth[1], smooth[2]]
    g = make_grid(n, 1000.0)
    mesh = torch.empty((n, n, n), device="cuda")
    c = Context()
    try:
        for xs in [clumped] * 2 + [smooth] * 8:
            c.assign(*xs, None, g, NGP, F32, out=mesh)
        c.profile(True)
        c.profile_read(True)
        c.assign(*smooth, None, g, NGP, F32, out=mesh)
        names = c.profile_read(True)
        assert "assign_super_sort" in names and "assign_bin_count" not in names, sorted(names)
    finally:
        c.close()


@pytest.mark.parametrize("job", [False, True])
def test_short_of_memory_runs_exactly(job):
    # All but 0.9 GB of the device is taken.  30 M particles: 0.56 GB of CIC
    # records on 512^3, for which the two-level sort wants 0.48 GB beside
    # them and the payload estimate a quarter more; 0.65 GB of TSC records and
    # 0.14 GB of mesh and spectrum of a 256^3 job.
    import torch
    from cosmicatlas_b200 import _lib as L
    from cosmicatlas_b200.api import Context, alloc_stats
    npart = 30_000_000
    gen = torch.Generator(device="cuda").manual_seed(8)
    xs = [torch.rand(npart, device="cuda", generator=gen) * 1000.0 for _ in range(3)]
    mesh = None if job else torch.empty((512, 512, 512), device="cuda")

    def call(c):
        if job:
            return c.job(*xs, None, make_grid(256, 1000.0), TSC, F32, pk=Context.pk_opts(TSC, nbins=128))["pk"].pk
        c.assign(*xs, None, make_grid(512, 1000.0), CIC, F32, out=mesh)
        return mesh.cpu().numpy()

    c = Context()
    want = call(c)
    c.close()
    c = Context()
    hog = None
    try:
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        assert L.lib().cam_pool_trim(0) == L.CAM_OK
        hog = torch.empty(torch.cuda.mem_get_info()[0] - 900_000_000, dtype=torch.uint8, device="cuda")
        alloc_stats(reset=True)
        got = [call(c) for _ in range(3)]
        assert alloc_stats()["failures"] > 0
        del hog
        torch.cuda.empty_cache()
        got.append(call(c))
        assert all(np.array_equal(g, want) for g in got)
    finally:
        hog = None
        c.close()
        torch.cuda.empty_cache()
        L.lib().cam_pool_trim(0)


def test_sorted_particles_make_room_for_other_calls():
    # a 512^3 assignment leaves 0.5 GB of sorted particles in its context;
    # with 0.15 GB free the 0.23 GB spectrum of a 384^3 transform takes
    # their place, and the next assignment is the same again
    import torch
    from cosmicatlas_b200 import _lib as L
    from cosmicatlas_b200.api import Context
    gen = torch.Generator(device="cuda").manual_seed(9)
    xs = [torch.rand(30_000_000, device="cuda", generator=gen) * 1000.0 for _ in range(3)]
    mesh = torch.empty((512, 512, 512), device="cuda")
    field = torch.randn((384, 384, 384), device="cuda", generator=gen)
    spec = torch.empty((384, 384, 193), dtype=torch.complex64, device="cuda")
    g = make_grid(512, 1000.0)
    c = Context()
    hog = None

    def transform():
        c._check(c._lib.cam_fft_r2c(c.h, 384, F32, L.ptr(field), L.ptr(spec), L.MEM_DEVICE))
        return spec.cpu().numpy()

    try:
        want = Context()
        try:
            want_spec = want.fft_r2c(field).cpu().numpy()
        finally:
            want.close()
        c.assign(*xs, None, g, CIC, F32, out=mesh)
        want_mesh = mesh.cpu().numpy()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        assert L.lib().cam_pool_trim(0) == L.CAM_OK
        hog = torch.empty(torch.cuda.mem_get_info()[0] - 150_000_000, dtype=torch.uint8, device="cuda")
        assert np.array_equal(transform().view(np.float32), want_spec.view(np.float32))
        del hog
        torch.cuda.empty_cache()
        c.assign(*xs, None, g, CIC, F32, out=mesh)
        assert np.array_equal(mesh.cpu().numpy(), want_mesh)
    finally:
        hog = None
        c.close()
        torch.cuda.empty_cache()
        L.lib().cam_pool_trim(0)


def test_slabs_near_their_limit():
    # bricks of 4 cells along x whose fullest holds 1.9 times the mean: more
    # than the limit of two with the margin of 9/8, less without it.  In turn
    # with an even catalogue both use slabs, the exact mesh is the same.
    import torch
    from cosmicatlas_b200.api import Context
    npart = 1_050_000
    gen = torch.Generator(device="cuda").manual_seed(3)
    even = [torch.rand(npart, device="cuda", generator=gen) * 64.0 for _ in range(3)]
    layer = [v.clone() for v in even]
    layer[0][: int(0.06 * npart)] /= 16.0
    g = make_grid(64, 64.0)
    c, exact = Context(), Context()
    try:
        want = {id(xs): exact.assign(*xs, None, g, NGP, F32).mesh for xs in (even, layer)}
        for _ in range(2):
            for xs in (even, layer):
                c.assign(*xs, None, g, NGP, F32)
        for xs in (even, layer) * 2:
            c.profile(True)
            c.profile_read(True)
            got = c.assign(*xs, None, g, NGP, F32).mesh
            names = c.profile_read(True)
            c.profile(False)
            assert names["assign_deposit"][0] == 1 and "assign_bin_count" not in names
            assert bool((got == want[id(xs)]).all())
    finally:
        c.close()
        exact.close()
