"""The grouped and fused forms of the FP64 kernels at the sizes where they can go wrong: deposits
summed per cell inside a warp (any row order, weights, partial warps, non-finite values), the
cycle's fused push and centre mass, the history row's chunk edges, long runs of the cell sort,
the scan's two forms, the exchanges' variable groups and the clouds' slots on odd blocks --
against the CPU oracle; the mixed stage's window against the FP64 form."""
import numpy as np
import pytest

from athenak_b200.inputs import make_state
from athenak_b200.mesh import dir_index, uniform_mesh
from oracle.oracle import Oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12                    # FP64 sums in another order, of the field's scale


def fields(a, b):
    return max(np.abs(a[:, v] - b[:, v]).max() / max(np.abs(b[:, v]).max(), 1e-300)
               for v in range(a.shape[1]))


def state(cells, block, ppc, seed=5, **kw):
    d = 0.01
    ms = uniform_mesh(cells, block, 2, tuple(-0.5 * d * n for n in cells),
                      tuple(0.5 * d * n for n in cells))
    return ms, make_state(ms, [0.01, 0.3], [1.0, 0.5], ppc, seed=seed, vel_noise=0.05,
                          gas_noise=1e-2, **kw)


def permute(st, order):
    st.pr[:, :st.npart] = st.pr[:, order]
    st.pi[:, :st.npart] = st.pi[:, order]


def clump(st, n, seed=3):
    """the first n particles into one cell of block 0"""
    rng = np.random.default_rng(seed)
    mb = st.mesh.mb_size[0]
    c = [st.mesh.nx[0] - 1, 0, st.mesh.nx[2] // 2]
    for a, (r, r1) in enumerate(((0, 6), (2, 8), (4, 10))):
        if a == 2 and not st.mesh.three_d:
            continue
        x = mb[a] + (c[a] + rng.random(n)) * mb[6 + a]
        st.pr[r, :n] = st.pr[r1, :n] = x
    st.pi[0, :n] = 0


def pair(st, phys):
    from athenak_b200.drag import DeviceDust
    return Oracle(st, phys), DeviceDust(st, phys)


@pytest.mark.parametrize("order", ["cell", "drawn", "reversed", "clumped"])
@pytest.mark.parametrize("scheme,cells,block", [(2, (10, 14, 6), (5, 7, 6)), (1, (12, 18, 1), (12, 9, 1)),
                                                (0, (8, 6, 6), (4, 6, 3))])
def test_deposits_of_every_row_order(order, scheme, cells, block):
    ms, st = state(cells, block, 3)
    if order == "clumped":
        clump(st, min(300, st.npart))
    phys = dict(scheme=scheme, drag_solver=2)
    if order != "drawn":
        o = Oracle(st, phys)
        by_cell, _ = o.sort_order()
        permute(st, by_cell if order != "reversed" else by_cell[::-1].copy())
    o, g = pair(st, phys)
    a_dt = 2e-3
    o.register_copy(); g.register_copy()
    assert o.pc2_predictor(a_dt) == 0
    g.pc2_predictor(a_dt)
    assert fields(g.host("qdep")[:, 1:], o.qdep[:, 1:]) < TOL
    assert o.deposit_qp(a_dt) == 0
    g.deposit_qp(a_dt)
    assert fields(g.host("qdep")[:, :4], o.qdep[:, :4]) < TOL
    for s in (o, g):
        s.ghost_add("qdep", 5); s.solve_ustar(); s.dc1_sweep(a_dt); s.ghost_copy("ustar", 3)
    assert fields(g.host("ustar"), o.ustar) < TOL
    o.gather_kick_pmbr(a_dt); g.gather_kick_pmbr(a_dt)
    assert fields(g.host("dmom"), o.dmom) < TOL
    assert g.error_word() == 0


@pytest.mark.parametrize("cells,block", [((40, 6, 4), (40, 6, 4)), ((26, 10, 1), (26, 5, 1)), ((8, 8, 8), (4, 8, 8))])
def test_deposits_of_a_lattice(cells, block):
    """One particle per cell, cell after cell: rows of consecutive anchors add by themselves, the
    batches that cross several rows through the windows."""
    ms, st = state(cells, block, 1, placement="lattice")
    o, g = pair(st, dict(scheme=2, drag_solver=2))
    assert o.deposit_qp(2e-3) == 0
    g.deposit_qp(2e-3)
    assert fields(g.host("qdep")[:, :4], o.qdep[:, :4]) < TOL
    for _ in range(2):
        assert o.imex_cycle(2e-3) == 0
        g.imex_cycle(2e-3)
    assert fields(g.host("u0"), o.u0) < 1e-11
    assert g.error_word() == 0

@pytest.mark.parametrize("order", ["cell", "drawn", "reversed", "lattice"])
@pytest.mark.parametrize("scheme,cells,block,ppc", [(2, (26, 28, 18), (13, 14, 9), 1), (1, (18, 20, 12), (9, 10, 6), 4),
                                                    (2, (96, 64, 1), (48, 32, 1), 2), (0, (40, 72, 1), (20, 9, 1), 8)])
def test_deposits_of_more_than_two_warps_per_sm(order, scheme, cells, block, ppc):
    """Launches beyond the direct form's 9472 particles: the windows in cell order, the direct form
    of 2-D batches that change cell often (drawn) and of lattices; the cycle's centre mass too."""
    if order == "lattice":
        ppc = 1
        cells = tuple(2 * c if c > 1 else 1 for c in cells)
        block = tuple(2 * b if b > 1 else 1 for b in block)
    ms, st = state(cells, block, ppc, seed=15, placement="lattice" if order == "lattice" else "random")
    assert st.npart > 9472
    phys = dict(scheme=scheme, drag_solver=2)
    if order in ("cell", "reversed"):
        by_cell = Oracle(st, phys).sort_order()[0]
        permute(st, by_cell if order == "cell" else by_cell[::-1].copy())
    o, g = pair(st, phys)
    a_dt = 2e-3
    o.register_copy(); g.register_copy()
    for rate_dep in (1, 0):
        assert o.pc2_predictor(a_dt, rate_dep) == 0
        g.pc2_predictor(a_dt, rate_dep)
        assert fields(g.host("qdep")[:, 1:4], o.qdep[:, 1:4]) < TOL
        assert np.abs(g.host("qdep")[:, 4] - o.qdep[:, 4]).max() <= TOL * np.abs(o.qdep[:, 4]).max()
    assert o.deposit_qp(a_dt) == 0
    g.deposit_qp(a_dt)
    assert fields(g.host("qdep")[:, :4], o.qdep[:, :4]) < TOL
    for s in (o, g):
        s.ghost_add("qdep", 5); s.solve_ustar(); s.dc1_sweep(a_dt); s.ghost_copy("ustar", 3)
    assert fields(g.host("ustar"), o.ustar) < TOL
    o.gather_kick_pmbr(a_dt); g.gather_kick_pmbr(a_dt)
    assert fields(g.host("dmom"), o.dmom) < TOL
    assert o.imex_cycle(a_dt) == 0
    g.imex_cycle(a_dt)
    assert fields(g.host("u0"), o.u0) < 1e-11
    assert g.error_word() == 0


@pytest.mark.parametrize("order", ["cell", "drawn"])
@pytest.mark.parametrize("scheme,bad", [(0, np.inf), (1, np.nan), (2, np.inf)])
def test_values_that_are_not_finite_beside_the_windows(scheme, bad, order):
    """The batches of such a value add lane by lane, the others through the windows."""
    ms, st = state((16, 16, 16), (8, 16, 16), 3, seed=4)
    assert st.npart > 9472
    if order == "cell":
        permute(st, Oracle(st, {}).sort_order()[0])
    st.pr[1, 7] = bad
    st.pr[5, 7000] = -bad
    o, g = pair(st, dict(scheme=scheme))

    def same(a, b):
        ok = np.isfinite(b)
        np.testing.assert_array_equal(np.isfinite(a), ok)
        assert np.abs(a[ok] - b[ok]).max() < TOL * np.abs(b[ok]).max()

    out, err = o.point_science_fields()
    assert err == 0
    same(g.point_science_fields().cpu().numpy(), out)
    assert o.deposit_qp(1e-3) == 0
    g.deposit_qp(1e-3)
    same(g.host("qdep")[:, :4], o.qdep[:, :4])
    assert g.error_word() == 0


def test_deposit_on_more_cells_than_32_bit_keys():
    """Two cells 2^32 apart in the pack's padded cells: their particles stay apart.  Needs 69 GB for
    the density and its halo."""
    from athenak_b200.drag import DeviceDust
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 80 GB of free device memory")
    torch.cuda.empty_cache()
    ms = uniform_mesh((1792, 1792, 1280), (256, 256, 256), 2, (0.0,) * 3, (1792.0, 1792.0, 1280.0))
    per = 260 ** 3
    assert ms.nmb * per > 2 ** 32
    a = np.array([0, 20, 10, 10])                # block, padded k, j, i
    at = (a[1] * 260 + a[2]) * 260 + a[3] + 2 ** 32
    b = np.array([at // per, at % per // 260 ** 2, at % 260 ** 2 // 260, at % 260])
    assert b[0] == ms.nmb - 1 and (b[1:] >= 4).all() and (b[1:] < 256).all()
    n = 12000                                    # (beyond the launches that add lane by lane)
    g = DeviceDust.__new__(DeviceDust)
    from athenak_b200 import capi
    g.lib, g.mesh, g.device, g.npart, g.nspecies, g.stride = capi.load(), ms, torch.device("cuda"), n, 1, n
    f64 = dict(dtype=torch.float64, device="cuda")
    g.t = {k: torch.zeros(1, **f64) for k in ("u0", "u1", "qdep", "ustar", "dmom", "resid", "work", "sb_gid", "scalar")}
    g.t.update(pr=torch.zeros((17, n), **f64), pi=torch.zeros((5, n), dtype=torch.int32, device="cuda"),
               mb_size=torch.from_numpy(ms.mb_size).cuda(), nghbr=torch.from_numpy(ms.nghbr).cuda(),
               err=torch.zeros(1, dtype=torch.int32, device="cuda"), x3_removed=torch.zeros(2, **f64))
    g.phys = dict(scheme=2)
    g._rebuild_ctx()
    for q, c in enumerate((a, b)):               # a particle of each in turn, at the cells' centres
        g.t["pi"][0, q::2] = int(c[0])
        for x in range(3):
            g.t["pr"][2 * x, q::2] = float(ms.mb_size[c[0], x]) + float(c[3 - x]) - 2.0 + 0.5
    g.t["pr"][16] = 1.0
    g.t["pr"][16, 1::2] = 2.0
    rho = g.point_gravity_density()
    assert g.error_word() == 0
    w = np.array([0.125, 0.75, 0.125])
    w = w[:, None, None] * w[None, :, None] * w[None, None, :] * (n // 2)
    total = 0.0
    for c, m in ((a, 1.0), (b, 2.0)):
        got = rho[c[0], 0, c[1] - 1:c[1] + 2, c[2] - 1:c[2] + 2, c[3] - 1:c[3] + 2].cpu().numpy()
        np.testing.assert_allclose(got, m * w, rtol=TOL)
        total += m * n / 2
    assert abs(float(sum(rho[m].sum() for m in range(ms.nmb))) - total) < TOL * total
    del rho, g
    torch.cuda.empty_cache()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129])
def test_partial_warps_and_fused_cycle(n):
    ms, st = state((8, 8, 8), (4, 8, 8), 1, seed=8)
    st.npart = n
    phys = dict(scheme=2, drag_solver=2)
    o, g = pair(st, phys)
    for _ in range(2):
        assert o.imex_cycle(2e-3) == 0
        g.imex_cycle(2e-3)
    gp, gi = g.host("pr"), g.host("pi")
    np.testing.assert_array_equal(gi, o.st.pi[:, :n])
    for r in range(17):
        sc = max(np.abs(o.st.pr[r, :n]).max(), 1e-300)
        assert np.abs(gp[r] - o.st.pr[r, :n]).max() <= TOL * sc, r
    assert fields(g.host("u0"), o.u0) < 1e-11
    assert g.error_word() == 0


def test_zero_weights_keep_non_finite_values_out():
    """NGP: a particle with an infinite velocity reaches its own cell alone."""
    ms, st = state((8, 8, 8), (8, 8, 8), 2, seed=4)
    st.pr[1, 7] = np.inf
    phys = dict(scheme=0)
    o, g = pair(st, phys)
    assert o.deposit_qp(1e-3) == 0
    g.deposit_qp(1e-3)
    np.testing.assert_array_equal(np.isfinite(g.host("qdep")[:, :4]), np.isfinite(o.qdep[:, :4]))

@pytest.mark.parametrize("placement", ["random", "lattice"])
@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_science_fields_skip_cells_of_zero_weight(scheme, placement, bad):
    """A velocity that is not finite reaches the cells of nonzero weight alone, along x too, in
    a batch of any order (the lattice: rows of consecutive cells)."""
    ms, st = state((32, 6, 6), (32, 6, 6), 1, seed=4, placement=placement)
    st.pr[1, 7] = bad
    st.pr[5, 70] = -bad
    o, g = pair(st, dict(scheme=scheme))
    out, err = o.point_science_fields()
    got = g.point_science_fields().cpu().numpy()
    assert err == 0 and g.error_word() == 0
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(out))
    ok = np.isfinite(out)
    assert np.abs(got[ok] - out[ok]).max() < TOL * np.abs(out[ok]).max()


@pytest.mark.parametrize("row,bad", [(1, np.inf), (3, np.nan), (16, np.inf), (16, np.nan), ("massless", np.inf)])
@pytest.mark.parametrize("cells,block", [((10, 14, 6), (5, 7, 6)), ((12, 18, 1), (4, 9, 1))])
def test_clouds_skip_cells_of_zero_weight(cells, block, row, bad):
    """Clouds of levels 0 to 3 with a velocity or a mass that is not finite: the leaves of nonzero
    weight alone take them, in Q/P and the kick's back-reaction."""
    ms, st = state(cells, block, 3, seed=13)
    st.pi[3, :st.npart] = np.arange(st.npart) % 4
    for p in (5, 34, 63):                      # (levels 1, 2 and 3)
        if row == "massless":
            st.pr[16, p], st.pr[1, p] = 0.0, bad
        else:
            st.pr[row, p] = bad
    o, g = pair(st, dict(scheme=2))

    def same(a, b):
        ok = np.isfinite(b)
        np.testing.assert_array_equal(np.isfinite(a), ok)
        assert np.abs(a[ok] - b[ok]).max() < TOL * np.abs(b[ok]).max()

    assert o.cloud_deposit_qp(1.3e-3, 0.0) == 0
    g.cloud_deposit_qp(1.3e-3, 0.0)
    same(g.host("qdep")[:, :4], o.qdep[:, :4])
    us = np.random.default_rng(6).standard_normal(o.ustar.shape) * 0.05
    o.ustar[...] = us
    g.t["ustar"].copy_(torch.from_numpy(us))
    o.ghost_copy("ustar", 3, 0); g.ghost_copy("ustar", 3, 0)
    assert o.cloud_gather_kick(2e-3, 0.0, o.gather_pack()) == 0
    g.cloud_gather_kick(2e-3, 0.0)
    same(g.host("dmom"), o.dmom)
    assert g.error_word() == 0


@pytest.mark.parametrize("mass", [0.0, 1e-7])
@pytest.mark.parametrize("offset,missing", [((0.9, 0.9, 0.0), (1, 1, 0)), ((0.0, 0.9, 0.9), (0, 1, 1)),
                                            ((0.9, 0.9, 0.9), (1, 1, 1)), ((0.9, 0.9, 0.0), (1, 0, 0))])
def test_clouds_that_reach_an_unowned_cell(offset, missing, mass):
    """A block without one of its edge or corner neighbours: a cloud that reaches into it sets the
    error bit, a massless one too (a missing face ends the cloud there instead)."""
    ms, st = state((8, 8, 8), (4, 4, 4), 1, seed=3)
    ms.nghbr[0, dir_index(*missing)] = -1
    st.npart = 40
    st.pi[0, :40] = 0
    mb = ms.mb_size[0]
    for a in range(3):                          # (all at the centre of the block but one)
        st.pr[2 * a, :40] = mb[a] + 2.0 * mb[6 + a]
        st.pr[2 * a, 17] += 1.9 * mb[6 + a] * (offset[a] > 0)
    st.pr[16, 17] = mass
    o, g = pair(st, dict(scheme=2))
    err = o.cloud_deposit_qp(1.3e-3, 0.0)
    assert bool(err) == (missing != (1, 0, 0))
    g.cloud_deposit_qp(1.3e-3, 0.0)
    assert g.error_word() == err
    assert fields(g.host("qdep")[:, :4], o.qdep[:, :4]) < TOL


@pytest.mark.parametrize("n", [1, 127, 128, 129, 4095, 4096, 4097, 8300])
def test_history_row_at_chunk_edges(n):
    ms, st = state((16, 16, 16), (16, 16, 16), 2, seed=9)
    st.npart = n
    st.pr[16, n // 2] = 0.0 if n > 1 else st.pr[16, 0]
    o, g = pair(st, dict(scheme=2))
    rg = g.phst().cpu().numpy()
    ro, err = o.phst()
    assert err == 0 and g.error_word() == 0
    np.testing.assert_array_equal(rg[:7], ro[:7])
    np.testing.assert_array_equal(rg[8:12], ro[8:12])


@pytest.mark.parametrize("run", [47, 48, 49, 128, 129, 256, 257, 1024, 1025])
def test_sort_of_long_runs(run):
    ms, st = state((8, 8, 8), (8, 8, 8), 2, seed=6)
    clump(st, min(run, st.npart))
    rng = np.random.default_rng(run)
    permute(st, rng.permutation(st.npart))
    o, g = pair(st, {})
    np.testing.assert_array_equal(g.cell_index()[0].cpu().numpy(), o.sort_order()[0])


@pytest.mark.parametrize("cells", [(256, 256, 192), (256, 256, 256)])
def test_scan_on_both_sides_of_the_two_launch_limit(cells):
    """3073 and 4097 tiles of 4096 bins: the bins' starts against a count on the host."""
    from athenak_b200.drag import DeviceDust
    ms = uniform_mesh(cells, (64, 64, 64), 2, tuple(-0.5 * n for n in cells),
                      tuple(0.5 * n for n in cells))
    g = DeviceDust.empty(ms, 5000, {}, nspecies=1)
    rng = np.random.default_rng(2)
    c = np.stack([rng.integers(0, n, 5000) for n in cells])
    b = c // 64
    blk = (b[2] * ms.nblocks[1] + b[1]) * ms.nblocks[0] + b[0]
    l = c % 64
    key = ((blk * 64 + l[2]) * 64 + l[1]) * 64 + l[0]
    for a in range(3):
        g.t["pr"][2 * a].copy_(torch.from_numpy(c[a] + 0.5 - 0.5 * cells[a]))
    g.t["pi"][0].copy_(torch.from_numpy(blk.astype(np.int32)))
    order, cstart = g.cell_index()
    np.testing.assert_array_equal(order.cpu().numpy(), np.argsort(key, kind="stable"))
    cs = cstart.cpu().numpy()
    assert cs[-1] == 5000
    np.testing.assert_array_equal(np.diff(cs)[np.unique(key)], np.unique(key, return_counts=True)[1])


@pytest.mark.parametrize("x3bc,shear", [(0, False), (1, False), (2, True)])
def test_additive_exchange_in_any_number_of_variables(x3bc, shear):
    """The variables are taken five, three or one at a time: 7 together as each alone."""
    from athenak_b200.drag import DeviceDust
    ms = uniform_mesh((8, 12, 8), (4, 4, 4), 2, (-0.5,) * 3, (0.5,) * 3, x3bc=x3bc, shear_x1=shear)
    st = make_state(ms, [0.1], [1.0], 1, seed=2)
    g = DeviceDust(st, dict(scheme=2, shearing_box=shear))
    g.set_time(0.37)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    for nv in (1, 2, 3, 4, 5, 7):
        f = torch.randn(ms.field_shape(nv), dtype=torch.float64, device="cuda", generator=gen)
        g.t["many"] = f.clone()
        g.ghost_add("many", nv)
        one = torch.empty_like(f)
        for v in range(nv):
            g.t["single"] = f[:, v:v + 1].contiguous()
            g.ghost_add("single", 1)
            one[:, v:v + 1] = g.t["single"]
        assert torch.equal(g.t["many"], one), nv


@pytest.mark.parametrize("cells,block,x3bc", [((4, 6, 8), (2, 2, 2), 0), ((300, 4, 1), (300, 2, 1), 0),
                                              ((4, 300, 1), (2, 300, 1), 0), ((70, 3, 9), (35, 3, 3), 1)])
def test_copy_exchange_of_flat_and_tiny_blocks(cells, block, x3bc):
    """The ghost cells' enumeration at its smallest and flattest blocks, in 1 to 7 variables: bit for
    bit the oracle's, variable by variable."""
    ms = uniform_mesh(cells, block, 2, (-0.5,) * 3, (0.5,) * 3, x3bc=x3bc)
    st = make_state(ms, [0.1], [1.0], 1, seed=2)
    o, g = pair(st, dict(scheme=2))
    f = np.random.default_rng(5).standard_normal(ms.field_shape(7))
    want = np.empty_like(f)
    for v in range(7):
        o.ustar[...] = f[:, v:v + 1]
        o.ghost_copy("ustar", 3, 0)
        want[:, v] = o.ustar[:, 0]
    for nv in (1, 3, 4, 5, 7):
        g.t["many"] = torch.from_numpy(np.ascontiguousarray(f[:, :nv])).cuda()
        g.ghost_copy("many", nv, 0)
        np.testing.assert_array_equal(g.t["many"].cpu().numpy(), want[:, :nv])


@pytest.mark.parametrize("cells,block", [((10, 14, 6), (5, 7, 6)), ((12, 18, 1), (4, 9, 1)),
                                         ((6, 4, 8), (2, 2, 4))])
def test_cloud_slots_on_odd_blocks(cells, block):
    """Levels 0 to 3 in the drawn order: the gathered velocities bit for bit, the deposits to
    their order."""
    ms, st = state(cells, block, 3, seed=13)
    st.pi[3, :st.npart] = np.arange(st.npart) % 4
    o, g = pair(st, dict(scheme=2))
    assert o.cloud_deposit_qp(1.3e-3, 0.0) == 0
    g.cloud_deposit_qp(1.3e-3, 0.0)
    assert fields(g.host("qdep")[:, :4], o.qdep[:, :4]) < TOL
    us = np.random.default_rng(6).standard_normal(o.ustar.shape) * 0.05
    o.ustar[...] = us
    g.t["ustar"].copy_(torch.from_numpy(us))
    o.ghost_copy("ustar", 3, 0); g.ghost_copy("ustar", 3, 0)
    assert o.cloud_gather_kick(2e-3, 0.0, o.gather_pack()) == 0
    g.cloud_gather_kick(2e-3, 0.0)
    for r in (1, 3, 5, 12, 13, 14):
        np.testing.assert_array_equal(g.host("pr")[r], o.st.pr[r, :st.npart])
    assert fields(g.host("dmom"), o.dmom) < TOL
    assert g.error_word() == 0


@pytest.mark.parametrize("placement", ["random", "lattice"])
@pytest.mark.parametrize("levels", [[0], [1], [2], [1, 2, 3], [0, 1]])
@pytest.mark.parametrize("cells,block", [((32, 6, 4), (32, 3, 4)), ((30, 8, 1), (10, 4, 1)), ((4, 6, 8), (2, 2, 2))])
def test_clouds_of_one_kind_and_lattices(cells, block, levels, placement):
    """Batches whose clouds are all narrow, and lattices in cell order, add leaf by leaf: the
    deposits to their order, the gathered velocities (narrow clouds on two slots) bit for bit.
    At the centre of a cell a cloud of level 1 or more has its edges on faces or near them: a
    neighbour listed or not by rounding changes a coefficient by its moment's rounding, some 2 eps
    of each of up to 19 leaves and 3 coefficients, here times velocities and differences up to 0.3."""
    ms, st = state(cells, block, 1, seed=13, placement=placement)
    st.pi[3, :st.npart] = np.resize(levels, st.npart)
    if placement == "lattice":
        o = Oracle(st, dict(scheme=2))
        permute(st, o.sort_order()[0])
    o, g = pair(st, dict(scheme=2))
    assert o.cloud_deposit_qp(1.3e-3, 0.0) == 0
    g.cloud_deposit_qp(1.3e-3, 0.0)
    assert fields(g.host("qdep")[:, :4], o.qdep[:, :4]) < TOL
    us = np.random.default_rng(6).standard_normal(o.ustar.shape) * 0.05
    o.ustar[...] = us
    g.t["ustar"].copy_(torch.from_numpy(us))
    o.ghost_copy("ustar", 3, 0); g.ghost_copy("ustar", 3, 0)
    assert o.cloud_gather_kick(2e-3, 0.0, o.gather_pack()) == 0
    g.cloud_gather_kick(2e-3, 0.0)
    for r in (1, 3, 5):
        a, b = g.host("pr")[r], o.st.pr[r, :st.npart]
        if placement == "random":
            np.testing.assert_array_equal(a, b)
        else:
            assert np.abs(a - b).max() <= 2 * 19 * 3 * 0.3 * np.finfo(float).eps
    assert fields(g.host("dmom"), o.dmom) < TOL
    assert g.error_word() == 0


@pytest.mark.parametrize("cells,block,ppc", [
    ((6, 10, 14), (6, 10, 14), 3),      # one block, its own neighbour on every side
    ((4, 6, 4), (2, 6, 2), 5),          # blocks of two cells: every cell at a face
    ((64, 36, 1), (64, 9, 1), 2),       # 2-D, few particles per tile: one pass
    ((64, 8, 1), (64, 4, 1), 40),       # 2-D, dense: several passes
])
def test_mixed_stage_matches_fp64(cells, block, ppc):
    """The window written by the solves: every velocity and the gas within
    the mixed form's 1e-5 of the largest (plain back-reaction, two cycles)."""
    from athenak_b200.drag import DeviceDust
    from athenak_b200.mixed import MixedDust
    ms, st = state(cells, block, ppc, seed=17)
    phys = dict(scheme=2, drag_solver=3, consistent_gas=False)
    ref, mx = DeviceDust(st, phys), MixedDust(st, phys)
    for _ in range(2):
        ref.imex_cycle(2e-3)
        mx.imex_cycle(2e-3)
    mx.export()
    assert ref.error_word() == 0 and mx.error_word() == 0
    a, b = mx.dev.host("pr"), ref.host("pr")
    for r in (1, 3, 5):
        assert np.abs(a[r] - b[r]).max() < 1e-5 * np.abs(b[[1, 3, 5]]).max(), r
    ua, ub = ms.active(mx.dev.host("u0")), ms.active(ref.host("u0"))
    for v in range(1, 4):
        assert np.abs(ua[:, v] - ub[:, v]).max() < 1e-5 * max(np.abs(ub[:, v]).max(), 1e-300), v
