"""The dispatches of the kernels at the sizes where they switch or leave a remainder, against the
CPU oracle (bit for bit where the results are integers or follow its rounding)."""
import numpy as np
import pytest

from rtlib_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _t(a, dev):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


@pytest.mark.parametrize("n", [1, 33, 227329, 909315])
def test_record_root_only(cuda, oracle, n):
    """A cleared tree sums its records in registers, four grid strides (227328 each) at a time."""
    from rtlib_b200.sdtree import SDTree
    rec = W.sdtree_records(n, n)
    rec["radiance"][::7] = np.nan
    wo = np.where(np.arange(n) % 5 == 0, 0.0, 2.0).astype(np.float32)
    sw = np.where(np.arange(n) % 11 == 0, -1.0, 0.5).astype(np.float32)
    delta = (np.arange(n) % 13 == 0).astype(np.uint8)
    g, o = SDTree((0, 0, 0), (1, 1, 1)), oracle.sdtree((0, 0, 0), (1, 1, 1))
    g.record(*(_t(rec[k], cuda) for k in ("pos", "uv", "radiance")), _t(wo, cuda), _t(sw, cuda), _t(delta, cuda))
    o.record(rec["pos"], rec["uv"], rec["radiance"], wo, sw, delta)
    eg, eo = g.export(sampling=False), o.export(sampling=False)
    np.testing.assert_array_equal(eg.scalars, eo.scalars)
    np.testing.assert_array_equal(eg.dsums, eo.dsums)


@pytest.mark.parametrize("threshold", [1 << 30, 4000, 300, 3])
def test_record_counter_placement(cuda, oracle, threshold):
    """One DTree of many quadrants (all counters in shared memory), tens and hundreds of DTrees
    (stat-weights only) and thousands (neither)."""
    from rtlib_b200.sdtree import SDTree
    rec = W.sdtree_records(1 << 15, 5)
    g, o = SDTree((0, 0, 0), (1, 1, 1)), oracle.sdtree((0, 0, 0), (1, 1, 1))
    args = [_t(rec[k], cuda) for k in ("pos", "uv", "radiance")]
    for _ in range(2):
        g.record(*args)
        o.record(rec["pos"], rec["uv"], rec["radiance"])
        g.build()
        o.build()
        g.refine(threshold)
        o.refine(threshold)
    g.record(*args)
    o.record(rec["pos"], rec["uv"], rec["radiance"])
    eg, eo = g.export(sampling=False), o.export(sampling=False)
    assert eg.topology == eo.topology
    np.testing.assert_array_equal(eg.scalars, eo.scalars)
    np.testing.assert_array_equal(eg.dsums, eo.dsums)
    assert g.status() == 0


@pytest.mark.parametrize("level", [1, 2, 3, 4, 5, 6, 7])
def test_morton_build_skips_only_clean_cells(cuda, oracle, level):
    """Few cells of an odd number recorded, then others, then none: cells in use are rebuilt,
    cells no longer in use go back to zero, leaves end cleared; samples follow the pyramid."""
    import torch
    from rtlib_b200.hashgrid import MortonQuadTrees
    rng = np.random.default_rng(level)
    ncell = 37 if level < 6 else 5
    m = MortonQuadTrees(ncell, level=level)
    for used in ([0, 3, ncell - 1], [3, 4], []):
        n = 2000 if used else 0
        cell = np.array(used, np.uint32)[rng.integers(0, len(used), n)] if n else np.zeros(0, np.uint32)
        uv, val = rng.random((n, 2), dtype=np.float32), rng.lognormal(0, 2, n).astype(np.float32)
        leaves = np.zeros(ncell << (2 * level), np.int64)
        if n:
            m.record(_t(cell, cuda), _t(uv, cuda), _t(val, cuda))
            oracle.mqt_record(level, 24, leaves, cell, uv, val)
        m.update()
        want = oracle.mqt_build(ncell, level, 24, leaves)
        got_leaves, got = m.export()
        np.testing.assert_array_equal(got, want)
        assert not got_leaves.any()
        q = np.arange(5000, dtype=np.uint32) % (ncell + 1)
        seeds = rng.integers(1, 2**32, q.size, dtype=np.uint64).astype(np.uint32)
        o_uv = torch.empty((q.size, 2), dtype=torch.float32, device=cuda)
        o_pdf = torch.empty(q.size, dtype=torch.float32, device=cuda)
        m.sample_pdf(_t(q, cuda), _t(seeds, cuda), out_uv=o_uv, out_pdf_tree=o_pdf)
        in_range = q < ncell
        uv_w, pdf_w, _ = oracle.mqt_sample_pdf(level, want, q[in_range], seeds[in_range])
        np.testing.assert_array_equal(o_uv.cpu().numpy()[in_range], uv_w)
        np.testing.assert_array_equal(o_pdf.cpu().numpy()[in_range], pdf_w)


def test_morton_choice_at_its_margins(cuda, oracle):
    """Quadrant sums for which boundary and second comparison fall on representable draws (equal
    quarters and halves, zero quadrants, one quadrant alone): the divisions decide, as the oracle."""
    import torch
    from rtlib_b200.hashgrid import MortonQuadTrees
    sums = [(1, 1, 1, 1), (1, 0, 0, 0), (0, 0, 0, 2), (0, 3, 0, 3), (3, 0, 1, 0), (1, 1, 0, 0), (0, 0, 1, 1), (1, 2, 3, 2),
            (1e-6, 1, 1e-6, 1), (1, 1e-6, 1, 1e-6), (5, 0, 0, 7)]
    m = MortonQuadTrees(len(sums), level=1)
    cell = np.repeat(np.arange(len(sums), dtype=np.uint32), 4)
    uv = np.tile(np.array([[0.1, 0.1], [0.9, 0.1], [0.1, 0.9], [0.9, 0.9]], np.float32), (len(sums), 1))
    val = np.array(sums, np.float32).ravel()
    leaves = np.zeros(4 * len(sums), np.int64)
    m.record(_t(cell, cuda), _t(uv, cuda), _t(val, cuda))
    oracle.mqt_record(1, 24, leaves, cell, uv, val)
    m.update()
    pyr = oracle.mqt_build(len(sums), 1, 24, leaves)
    q = (np.arange(1 << 20) % len(sums)).astype(np.uint32)
    seeds = np.random.default_rng(1).integers(1, 2**32, q.size, dtype=np.uint64).astype(np.uint32)
    o_uv = torch.empty((q.size, 2), dtype=torch.float32, device=cuda)
    m.sample_pdf(_t(q, cuda), _t(seeds, cuda), out_uv=o_uv)
    np.testing.assert_array_equal(o_uv.cpu().numpy(), oracle.mqt_sample_pdf(1, pyr, q, seeds)[0])


@pytest.mark.parametrize("ncell,level,n", [(10, 2, 16 * 160), (10, 2, 16 * 160 - 1), (64, 4, 1 << 18), (65, 4, 1 << 18),
                                           (3, 1, 1), (16384, 4, 300001)])
def test_morton_record_routes(cuda, oracle, ncell, level, n):
    """Private sums (few leaves, many records) and one atomic per record, at the line between them;
    sums past 32 bits carry into the high word; every recorded cell is rebuilt."""
    from rtlib_b200.hashgrid import MortonQuadTrees
    rng = np.random.default_rng(n)
    m = MortonQuadTrees(ncell, level=level)
    cell = np.minimum((rng.random(n) ** 2 * (ncell + 1)).astype(np.uint32), ncell)  # ncell: outside, skipped
    cell[::17] = 0xFFFFFFFF
    uv, val = rng.random((n, 2), dtype=np.float32), rng.lognormal(3, 3, n).astype(np.float32)
    val[::19] = np.nan
    leaves = np.zeros(ncell << (2 * level), np.int64)
    m.record(_t(cell, cuda), _t(uv, cuda), _t(val, cuda))
    ok = cell < ncell
    oracle.mqt_record(level, 24, leaves, cell[ok], uv[ok], val[ok])
    np.testing.assert_array_equal(m.export()[0], leaves)
    m.update()
    np.testing.assert_array_equal(m.export()[1], oracle.mqt_build(ncell, level, 24, leaves))


@pytest.mark.parametrize("n", [64, 65, 66, 73, 500, 3000])
def test_hierarchy_hits(cuda, oracle, n):
    """Hits of the eight-wide hierarchy against brute force over soups of mixed sizes (walls among
    small triangles), with degenerate, duplicate, flat and non-finite triangles, rays along the axes,
    from far outside and with their own bounds: the same distance bit for bit."""
    import torch
    from rtlib_b200.tracer import Scene
    rng = np.random.default_rng(n)
    tri = (rng.normal(size=(n, 3, 3)) * 0.15 + rng.uniform(-3, 3, (n, 1, 3))).astype(np.float32)
    tri[0] = [[-4, -4, 3], [4, -4, 3], [4, 4, 3]]
    tri[1] = [[-4, -3, -4], [4, -3, 4], [4, -3, -4]]
    tri[2] = tri[3]                       # duplicates
    tri[4, 2] = tri[4, 1]                 # no area
    tri[5, :, 1] = 0.25                   # flat box
    if n > 65:
        tri[6, 0, 0], tri[7, 1, 2], tri[8, 2] = np.nan, np.inf, -np.inf
    q = 20000
    org = rng.uniform(-3.5, 3.5, (q, 3)).astype(np.float32)
    org[:200] *= 100.0
    d = rng.normal(size=(q, 3)).astype(np.float32)
    d[200:500] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, 300)] * rng.choice([-1, 1], (300, 1)).astype(np.float32)
    d[:200] = -org[:200]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    sc = Scene(_t(tri.reshape(n, 9), cuda))
    t, p, occ = torch.empty(q, device=cuda), torch.empty(q, dtype=torch.int32, device=cuda), torch.empty(q, dtype=torch.int32, device=cuda)
    for tmin, tmax in ((0.0, 1e20), (0.5, 2.0)):
        lo, hi = _t(np.full(q, tmin, np.float32), cuda), _t(np.full(q, tmax, np.float32), cuda)
        sc.intersect(_t(org, cuda), _t(d, cuda), lo, hi, out_t=t, out_prim=p)
        sc.intersect(_t(org, cuda), _t(d, cuda), lo, hi, any_hit=True, out_prim=occ)
        want_t, want_p = oracle.intersect(tri.reshape(n, 9), org, d, tmin, tmax)[:2]
        got_p = p.cpu().numpy().view(np.uint32)
        # duplicates may answer for one another
        same = (got_p == want_p) | (np.isin(got_p, (2, 3)) & np.isin(want_p, (2, 3)))
        assert same.all(), np.flatnonzero(~same)[:5]
        hit = want_p != 0xFFFFFFFF
        np.testing.assert_array_equal(t.cpu().numpy()[hit], want_t[hit])
        np.testing.assert_array_equal(occ.cpu().numpy() != -1, hit)


def test_hierarchy_of_coincident_triangles(cuda):
    """Equal boxes everywhere: clustering still pairs, the depth stays bounded, rays end."""
    import torch
    from rtlib_b200.tracer import Scene
    tri = np.tile(np.array([[0, 0, 1, 1, 0, 1, 0, 1, 1]], np.float32), (5000, 1))
    sc = Scene(_t(tri, cuda))
    org = _t(np.tile(np.array([[0.2, 0.2, 0.0]], np.float32), (4097, 1)), cuda)
    d = _t(np.tile(np.array([[0, 0, 1]], np.float32), (4097, 1)), cuda)
    t, p = torch.empty(4097, device=cuda), torch.empty(4097, dtype=torch.int32, device=cuda)
    sc.intersect(org, d, out_t=t, out_prim=p)
    assert (t == 1.0).all() and (p == p[0]).all()


@pytest.mark.parametrize("w,h,spp", [(1, 1, 3), (33, 7, 2), (148 * 7, 128, 1), (148 * 7, 129, 1)])
def test_whole_path_waves_equal_bounce_waves(cuda, w, h, spp):
    """Images, path depths and counters on both sides of the path-per-thread limit (7 CTAs of 128 per
    SM): the same as a launch per bounce gives."""
    from rtlib_b200 import scenes
    from rtlib_b200.tracer import FLAG_NEE, Tracer
    sc = scenes.cornell_box(w, h)
    tr = Tracer(sc, cuda, max_depth=6, width=w, height=h, seed=3)
    tr.render(spp, FLAG_NEE)
    img, depth, cnt = tr.image64().cpu().numpy(), tr.path_depths().cpu().numpy(), tr.counters()
    ref = Tracer(sc, cuda, max_depth=6, width=w, height=h, seed=3)
    ref.set_timing(True)  # measures the groups of a wave: always a launch per bounce
    ref.render(spp, FLAG_NEE)
    np.testing.assert_array_equal(img, ref.image64().cpu().numpy())
    np.testing.assert_array_equal(depth, ref.path_depths().cpu().numpy())
    assert cnt == ref.counters()


@pytest.mark.parametrize("w,h,ris", [(3, 1, 1), (9, 1, 0), (148, 80, 0), (149, 80, 1)])
@pytest.mark.parametrize("ntri", [36, 35, 1])
def test_lanes_that_share_a_path(cuda, w, h, ris, ntri):
    """Both sides of the limit of four lanes per path (80 paths per SM), an odd number of triangles and
    fewer pairs than lanes, coincident triangles: images, depths and counters as from a launch per
    bounce."""
    from rtlib_b200 import scenes
    from rtlib_b200.tracer import FLAG_NEE, FLAG_RIS, Tracer
    sc = scenes.cornell_box(w, h)
    sc["tri_v"] = sc["tri_v"].copy()
    sc["tri_v"][20:24] = sc["tri_v"][4:8]  # equal distances: the lowest index wins
    light = int(sc["light_tris"][0])
    keep = np.r_[np.arange(ntri - 1), light]
    sc = dict(sc, tri_v=sc["tri_v"][keep], tri_mat=sc["tri_mat"][keep], tri_uv=sc["tri_uv"][keep],
              light_tris=np.array([ntri - 1], np.uint32), light_first=np.zeros(1, np.uint32),
              light_count=np.ones(1, np.uint32))
    flags = FLAG_NEE | (FLAG_RIS if ris else 0)
    got = []
    for timing in (False, True):  # measured waves are always a launch per bounce
        tr = Tracer(sc, cuda, max_depth=6, width=w, height=h, seed=8)
        tr.set_timing(timing)
        tr.render(3, flags)
        got.append((tr.image64().cpu().numpy(), tr.path_depths().cpu().numpy(), tr.counters()))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    assert got[0][2] == got[1][2]


@pytest.mark.parametrize("counts", [[578], [1, 6, 571], [2] * 256 + [3, 63], [1] * 64])
def test_packed_lights_sample_like_indexed_ones(cuda, counts):
    """Light meshes of one and of many triangles, powers of two and not.  Entries in front of the
    lights, more than there are paths, rule the packed copy out; the image is the same.  The caller's
    index array is read at each render."""
    from rtlib_b200 import scenes
    from rtlib_b200.tracer import FLAG_NEE, FLAG_RIS, Tracer
    w, h = 148 * 7, 129  # past the path-per-thread limit
    sc = scenes.cornell_box(w, h, light_grid=17)
    rng = np.random.default_rng(len(counts))
    sc["light_tris"] = sc["light_tris"][:sum(counts)]
    sc["light_count"] = np.array(counts, np.uint32)
    sc["light_first"] = (np.cumsum(counts) - counts).astype(np.uint32)
    sc["light_emission"] = rng.uniform(1, 9, (len(counts), 3)).astype(np.float32)
    flags = FLAG_NEE | FLAG_RIS
    tr = Tracer(sc, cuda, max_depth=3, seed=4)
    far = dict(sc, light_tris=np.concatenate([np.zeros(w * h, np.uint32), sc["light_tris"]]),
               light_first=sc["light_first"] + np.uint32(w * h))
    ref = Tracer(far, cuda, max_depth=3, seed=4)
    for _ in range(2):
        tr.render(1, flags)
        ref.render(1, flags)
        np.testing.assert_array_equal(tr.image64().cpu().numpy(), ref.image64().cpu().numpy())
        tr.light_tris.copy_(tr.light_tris.flip(0))
        ref.light_tris[w * h:] = tr.light_tris


def test_lights_that_share_triangles(cuda):
    """Two meshes over the same entries, each with its own radiance: as the same entries twice."""
    from rtlib_b200 import scenes
    from rtlib_b200.tracer import FLAG_NEE, FLAG_RIS, Tracer
    w, h = 148 * 7, 129
    sc = scenes.cornell_box(w, h, light_grid=17)
    lt = sc["light_tris"]
    sc["light_emission"] = np.array([[9, 1, 1], [1, 1, 9]], np.float32)
    sc["light_count"] = np.full(2, len(lt), np.uint32)
    img = []
    for tris, first in ((lt, [0, 0]), (np.concatenate([lt, lt]), [0, len(lt)])):
        tr = Tracer(dict(sc, light_tris=tris, light_first=np.array(first, np.uint32)), cuda, max_depth=3, seed=4)
        tr.render(1, FLAG_NEE | FLAG_RIS)
        img.append(tr.image64().cpu().numpy())
    np.testing.assert_array_equal(img[0], img[1])


@pytest.mark.parametrize("grid,w,h", [(1, 40, 40), (16, 33, 20), (17, 33, 20), (2, 1100, 1)])
def test_emitter_gradients_add_up(cuda, grid, w, h):
    """The image is linear in the emitters' radiances, so gradients times radiances add up to the
    loss, in flat and hierarchy scenes, small and ragged images.  Both sides are the same products in
    another order: float rounding of about 1e5 terms, 1e-4 with room to spare."""
    import torch
    from rtlib_b200 import scenes
    from rtlib_b200.tracer import FLAG_NEE, Tracer
    sc = scenes.cornell_box(w, h, light_grid=grid)
    tr = Tracer(sc, cuda, max_depth=5, width=w, height=h, seed=5)
    d_img = _t(np.random.default_rng(grid).uniform(0.5, 1.0, (h, w, 3)).astype(np.float32), cuda)
    tr.render(8, FLAG_NEE)
    img = tr.image64()
    g = torch.zeros((grid * grid, 3), device=cuda)
    tr.clear()
    tr.render_adjoint(8, d_img, FLAG_NEE, -1, None, g)
    got = (g.double().cpu().numpy() * np.asarray(sc["light_emission"], np.float64).reshape(-1, 3)).sum(0)
    want = (img * d_img.double()).sum(dim=(0, 1)).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=1e-4)


@pytest.mark.parametrize("n,slots", [(1, 32), (128, 32), (129, 32), (5000, 1024), (4096, 1024), (4097, 1024), (70000, 1 << 16),
                                     (3000, 96), (300, 96)])
def test_hashgrid_insert_routes(cuda, oracle, n, slots):
    """Batches staged in the temporary table (at most four points per slot) and sorted ones give the
    slots of sequential insertion: overfull buckets, repeated cells, a table that is half full, a
    number of buckets that is no power of two."""
    from rtlib_b200.hashgrid import KEY_MORTON, HashGrid
    rng = np.random.default_rng(n)
    mn, mx, bounds = np.zeros(3, np.float32), np.full(3, 5, np.float32), [300, 40, 2000]
    hg = HashGrid(mn, mx, bounds, slots, keying=KEY_MORTON)
    cur = np.zeros(slots, np.uint64)
    import torch
    full = False
    for batch in range(3):
        pos = (rng.random((n, 3), dtype=np.float32) * 6 - 0.5).astype(np.float32)
        pos[n // 2:] = pos[rng.integers(0, n // 2 + 1, n - n // 2)]
        out = torch.empty(n, dtype=torch.int32, device=cuda)
        hg.insert(_t(pos, cuda), out)
        want, _ = oracle.mhash_insert(pos, mn, mx - mn, bounds, slots, cur)
        full |= bool((want == 0xFFFFFFFF).any())
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), want)
        np.testing.assert_array_equal(hg.export(), cur)
    assert bool(hg.status() & 0x10) == full


@pytest.mark.parametrize("offset", [0, 1, 3])
def test_hashgrid_noalloc_table_alignment(cuda, oracle, offset):
    """A caller's table need not lie on a 32-byte boundary."""
    import torch
    from rtlib_b200.hashgrid import KEY_MORTON, insert_noalloc
    rng = np.random.default_rng(offset)
    mn, mx, bounds, slots, n = np.zeros(3, np.float32), np.ones(3, np.float32), [64, 64, 64], 4096, 2500
    store = torch.zeros(slots + 8, dtype=torch.int64, device=cuda)
    table = store[offset:offset + slots]
    cur = np.zeros(slots, np.uint64)
    for _ in range(2):
        pos = rng.random((n, 3), dtype=np.float32)
        out = torch.empty(n, dtype=torch.int32, device=cuda)
        insert_noalloc(mn, mx, bounds, table, _t(pos, cuda), out, keying=KEY_MORTON)
        want, _ = oracle.mhash_insert(pos, mn, mx - mn, bounds, slots, cur)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), want)
    np.testing.assert_array_equal(table.cpu().numpy().view(np.uint64), cur)
    assert not store[:offset].any() and not store[offset + slots:].any()


@pytest.mark.parametrize("n", [1, 127, 129, 592 * 128 + 5])
def test_network_tile_edges(cuda, n):
    """Partial tiles, one tile per CTA and a CTA's second tile: each sample's row equals the one a
    single-tile call gives, raw outputs and lobes, into arrays with and without 16-byte alignment."""
    import torch
    from rtlib_b200._lib import call, ptr, stream_ptr
    from rtlib_b200.mlp import MLPGuide
    rng = np.random.default_rng(n)
    g = MLPGuide((0, 0, 0), (1, 1, 1), seed=4)
    unit = lambda: (lambda v: (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32))(rng.normal(size=(n, 3)))
    pos, nrm, wo = _t(rng.random((n, 3), dtype=np.float32), cuda), _t(unit(), cuda), _t(unit(), cuda)
    raw, lobes = g.eval(pos, nrm, wo), g.eval(pos, nrm, wo, raw=False)
    for a in sorted({0, n // 2, max(0, n - 100)}):
        sl = slice(a, min(n, a + 100))
        one = [x[sl].contiguous() for x in (pos, nrm, wo)]
        assert torch.equal(g.eval(*one), raw[sl]) and torch.equal(g.eval(*one, raw=False), lobes[sl])
    store = torch.full((n * 48 + 8,), 7.0, device=cuda)
    call("rtpg_mlp_eval", g.h, n, ptr(pos), ptr(nrm), ptr(wo), ptr(store) + 4, None, stream_ptr())
    assert torch.equal(store[1:1 + n * 48].view(n, 48), raw) and (store[1 + n * 48:] == 7.0).all()
    assert g.status() == 0


@pytest.mark.parametrize("steps", [255, 256, 257, 600])
def test_training_groups_of_minibatches(cuda, steps):
    """Weight sums are formed for 256 minibatches at a time and launches chained within them: steps
    taken in one call equal the same steps taken in several, bit for bit (one record per step: every
    gradient element is added once, so nothing depends on the order of atomics)."""
    from rtlib_b200.mlp import MLPGuide
    rng = np.random.default_rng(steps)
    unit = lambda: (lambda v: (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32))(rng.normal(size=(steps, 3)))
    rec = [_t(a, cuda) for a in (rng.random((steps, 3), dtype=np.float32), unit(), unit(), unit(),
                                 rng.lognormal(0, 1, steps).astype(np.float32))]
    a, b = MLPGuide((0, 0, 0), (1, 1, 1), seed=9), MLPGuide((0, 0, 0), (1, 1, 1), seed=9)
    la = a.train(rec, batch=1, epochs=1)
    for s in (0, 100, 101, steps):
        if s == steps:
            break
        e = {0: 100, 100: 101, 101: steps}[s]
        lb = b.train([x[s:e].contiguous() for x in rec], batch=1, epochs=1)
    np.testing.assert_array_equal(a.params(), b.params())
    assert la == lb and a.status() == 0 and b.status() == 0


@pytest.mark.parametrize("n", [1, 128, 129, 148 * 128 + 77])
def test_gradient_is_the_sum_of_its_tiles(cuda, n):
    """Partial tiles and a CTA's second tile: the gradient over all records is the weighted sum of the
    gradients over single tiles, up to the rounding of float sums."""
    import torch
    from rtlib_b200.mlp import MLPGuide
    rng = np.random.default_rng(n)
    unit = lambda: (lambda v: (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32))(rng.normal(size=(n, 3)))
    w = np.ones(n, np.float32)  # equal weights: no clamp, and the same scale in both sums
    rec = [_t(a, cuda) for a in (rng.random((n, 3), dtype=np.float32), unit(), unit(), unit(), w)]
    g = MLPGuide((0, 0, 0), (1, 1, 1), seed=2)
    loss, grad = g.loss_grad(*rec)
    want, wloss = torch.zeros(16384, device=cuda, dtype=torch.float64), 0.0
    for s in range(0, n, 128):
        part = [x[s:s + 128].contiguous() for x in rec]
        l, p = g.loss_grad(*part)
        want += p.double() * len(part[0]) / n
        wloss += l * len(part[0]) / n
    # the output gradients enter as bf16 (2^-9 relative) at another scale per call
    assert (grad.double() - want).norm() < 0.01 * want.norm()
    assert abs(loss - wloss) < 1e-4 * abs(wloss) and g.status() == 0


def test_sampling_thresholds_near_and_past_boundaries(cuda, oracle):
    """Quadrant sums whose boundary or second quotient lies on a draw, at 0 or at 1, on one side only
    or many orders apart: samples and pdfs of single-node trees equal the oracle's divisions."""
    import torch
    from rtlib_b200.sdtree import SDTree
    rng = np.random.default_rng(8)
    sums = [(1, 1, 1, 1), (1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 1, 0), (0, 0, 0, 1), (1, 0, 1, 0), (0, 1, 0, 1), (3, 1, 0, 2),
            (1e-5, 1, 1e-5, 1), (1, 1e-5, 1, 1e-5), (1e-6, 1, 3e-6, 1e5), (0.1, 0.2, 0.3, 0.4), (1e-7, 1e-7, 1e-7, 4e6)]
    sums += [tuple(rng.lognormal(0, 6, 4)) for _ in range(24)]
    uv = np.array([[0.2, 0.2], [0.7, 0.2], [0.2, 0.7], [0.7, 0.7]], np.float32)
    pos = np.full((4, 3), 0.5, np.float32)
    q = W.sdtree_queries(20000, 3)
    for s in sums:
        g, o = SDTree((0, 0, 0), (1, 1, 1)), oracle.sdtree((0, 0, 0), (1, 1, 1))
        r = np.array(s, np.float32)
        g.record(_t(pos, cuda), _t(uv, cuda), _t(r, cuda))
        o.record(pos, uv, r)
        g.build()
        o.build()
        a = torch.empty((20000, 2), device=cuda)
        p = torch.empty(20000, device=cuda)
        g.sample_pdf(_t(q["pos"], cuda), _t(q["seeds"], cuda), out_uv=a, out_pdf_uv=p)
        wa, wp = o.sample_pdf(q["pos"], q["seeds"])[:2]
        np.testing.assert_array_equal(a.cpu().numpy(), wa)
        np.testing.assert_array_equal(p.cpu().numpy(), wp)


def _records(n, seed, dev):
    rng = np.random.default_rng(seed)
    unit = lambda: (lambda v: (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32))(rng.normal(size=(n, 3)))
    return [_t(a, dev) for a in (rng.random((n, 3), dtype=np.float32), unit(), unit(), unit(),
                                 rng.lognormal(0, 2, n).astype(np.float32))]


@pytest.mark.parametrize("n,batch", [(1, 4096), (700, 256), (40000, 16384), (148 * 128 * 2 + 5, 148 * 128 + 1), (5000, 1 << 20)])
def test_training_repeats_bit_for_bit(cuda, n, batch):
    """Weight sums, gradients and loss are added in a fixed order whatever order the CTAs finish in: the
    same records give the same parameters, gradient and loss each time (one tile, one and several per
    CTA, ragged last minibatches).  Gradients are added to what is there."""
    import torch
    from rtlib_b200.mlp import MLPGuide
    rec = _records(n, n, cuda)
    got = []
    for _ in range(4):
        g = MLPGuide((0, 0, 0), (1, 1, 1), seed=9)
        loss, grad = g.loss_grad(*rec)
        got.append((g.train(rec, batch=batch, epochs=3), g.params(), loss, grad))
        assert g.status() == 0
    for loss, params, l0, g0 in got[1:]:
        assert loss == got[0][0] and l0 == got[0][2]
        np.testing.assert_array_equal(params, got[0][1])
        assert torch.equal(g0, got[0][3])
    # the same gradient added to ones, in the caller's buffer
    from rtlib_b200._lib import call, ptr, stream_ptr
    g = MLPGuide((0, 0, 0), (1, 1, 1), seed=9)
    more = torch.ones(16384, device=cuda)
    call("rtpg_mlp_loss_grad", g.h, n, *[ptr(x) for x in rec], ptr(more), None, stream_ptr())
    assert torch.equal(more, got[0][3] + 1.0)


@pytest.mark.parametrize("batch,steps", [(100, 40), (5000, 12), (148 * 128 + 1, 5)])
def test_chained_steps_see_the_step_before(cuda, batch, steps):
    """Within a call a step's launch starts while the previous step's Adam runs; its CTAs read the
    weights that Adam leaves: the steps of one call equal calls of one step each, bit for bit, with one
    tile, many CTAs and several tiles per CTA."""
    from rtlib_b200.mlp import MLPGuide
    n = batch * steps - batch // 3
    rec = _records(n, steps, cuda)
    a, b = MLPGuide((0, 0, 0), (1, 1, 1), seed=9), MLPGuide((0, 0, 0), (1, 1, 1), seed=9)
    la = a.train(rec, batch=batch, epochs=1)
    for s in range(0, n, batch):
        lb = b.train([x[s:s + batch].contiguous() for x in rec], batch=batch, epochs=1)
    np.testing.assert_array_equal(a.params(), b.params())
    assert la == lb and a.status() == 0 and b.status() == 0


@pytest.mark.parametrize("nested,others", [(130, 0), (200, 0), (200, 3000), (1000, 500)])
def test_hierarchy_of_nested_triangles(cuda, oracle, nested, others):
    """Boxes that contain one another merge one pair a round, so clustering runs out of rounds and
    pairs what is left by order: hits equal brute force, alone and beside other triangles."""
    import torch
    from rtlib_b200.tracer import Scene
    rng = np.random.default_rng(nested + others)
    size = (1.0 + 0.02 * np.arange(nested, dtype=np.float32))[:, None, None]
    tri = np.array([[[-1, -1, -1], [2, -1, -1], [-1, 2, 2]]], np.float32) * size
    soup = rng.normal(size=(others, 3, 3)) * 0.2 + rng.uniform(-9, 9, (others, 1, 3))
    tri = np.concatenate([tri, soup.astype(np.float32)]).reshape(-1, 9)
    tri = tri[rng.permutation(len(tri))]
    q = 20000
    org, d = rng.uniform(-10, 10, (q, 3)).astype(np.float32), rng.normal(size=(q, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    sc = Scene(_t(tri, cuda))
    t, p, occ = torch.empty(q, device=cuda), torch.empty(q, dtype=torch.int32, device=cuda), torch.empty(q, dtype=torch.int32, device=cuda)
    sc.intersect(_t(org, cuda), _t(d, cuda), out_t=t, out_prim=p)
    sc.intersect(_t(org, cuda), _t(d, cuda), any_hit=True, out_prim=occ)
    want_t, want_p = oracle.intersect(tri, org, d, 0.0, 1e20)[:2]
    hit, got_p = want_p != 0xFFFFFFFF, p.cpu().numpy().view(np.uint32)
    np.testing.assert_array_equal(got_p != 0xFFFFFFFF, hit)
    np.testing.assert_array_equal(t.cpu().numpy()[hit], want_t[hit])
    np.testing.assert_array_equal(occ.cpu().numpy() != -1, hit)
    # the triangles share a plane: another one than the lowest index may answer, at the same distance
    for i in np.flatnonzero(got_p != want_p):
        alone = oracle.intersect(tri[got_p[i]:got_p[i] + 1], org[i:i + 1], d[i:i + 1], 0.0, 1e20)[0]
        assert alone[0] == want_t[i]


@pytest.mark.parametrize("n", [65, 1024, 1025, 2048, 2049, 4097, 33000])
def test_hierarchy_build_sizes(cuda, oracle, n):
    """Clustering by one CTA (up to 2048 clusters, one or two a thread) and by launches of all SMs before
    that: every triangle is found."""
    import torch
    from rtlib_b200.tracer import Scene
    rng = np.random.default_rng(n)
    centre = rng.uniform(-3, 3, (n, 1, 3))
    tri = (rng.normal(size=(n, 3, 3)) * 0.02 + centre).astype(np.float32).reshape(n, 9)
    q = min(n, 3000)
    aim = rng.permutation(n)[:q]  # rays at as many triangles
    org = rng.uniform(-4, 4, (q, 3)).astype(np.float32)
    d = tri[aim].reshape(q, 3, 3).mean(1) - org
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    sc = Scene(_t(tri, cuda))
    t, p = torch.empty(q, device=cuda), torch.empty(q, dtype=torch.int32, device=cuda)
    sc.intersect(_t(org, cuda), _t(d, cuda), out_t=t, out_prim=p)
    want_t, want_p = oracle.intersect(tri, org, d, 0.0, 1e20)[:2]
    np.testing.assert_array_equal(p.cpu().numpy().view(np.uint32), want_p)
    np.testing.assert_array_equal(t.cpu().numpy(), want_t)
    assert (want_p != 0xFFFFFFFF).mean() > 0.99


@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1e-3, 0.0), (1e3, 0.0), (1.0, 50.0), (1e-3, 0.05)])
def test_hierarchy_planes_keep_every_hit(cuda, oracle, scale, offset):
    """Quantised boxes of nodes whose children lie on their walls (a room of many small tiles, flat boxes
    that share planes), at several scales and away from the origin; rays start on the walls and run
    along them: hits equal brute force."""
    import torch
    from rtlib_b200.tracer import Scene
    rng = np.random.default_rng(int(scale * 1000) + int(offset * 100))
    k = 12
    g = (np.stack(np.meshgrid(np.arange(k), np.arange(k), indexing="ij"), -1).reshape(-1, 2) / k).astype(np.float32)
    quads = []
    for axis in range(3):
        for side in (0.0, 1.0):
            c = np.empty((len(g), 4, 3), np.float32)
            for j, (du, dv) in enumerate(((0, 0), (1, 0), (1, 1), (0, 1))):
                c[:, j, axis] = side
                c[:, j, (axis + 1) % 3] = g[:, 0] + du / k
                c[:, j, (axis + 2) % 3] = g[:, 1] + dv / k
            quads.append(c)
    c = np.concatenate(quads)
    tri = np.concatenate([c[:, [0, 1, 2]], c[:, [0, 2, 3]]])
    inner = rng.normal(size=(300, 3, 3)) * 0.05 + rng.uniform(0.2, 0.8, (300, 1, 3))
    tri = (np.concatenate([tri, inner.astype(np.float32)]) * np.float32(scale) + np.float32(offset)).astype(np.float32).reshape(-1, 9)
    q = 6000
    on = tri.reshape(-1, 3, 3)[rng.integers(0, len(tri), (2, q))]
    b = rng.dirichlet((1, 1, 1), (2, q, 1))[:, :, 0, :, None]
    p = (on * b).sum(2).astype(np.float32)  # points of two triangles: from one towards the other
    org, d = p[0], p[1] - p[0]
    far = np.linalg.norm(d, axis=1)
    keep = far > 1e-2 * scale
    org, d = org[keep], (d[keep] / far[keep, None]).astype(np.float32)
    sc = Scene(_t(tri, cuda))
    n = len(org)
    t, prim, occ = torch.empty(n, device=cuda), torch.empty(n, dtype=torch.int32, device=cuda), torch.empty(n, dtype=torch.int32, device=cuda)
    tmin, tmax = np.float32(1e-4 * scale), np.float32(10.0 * scale)
    lo, hi = _t(np.full(n, tmin), cuda), _t(np.full(n, tmax), cuda)
    sc.intersect(_t(org, cuda), _t(d, cuda), lo, hi, out_t=t, out_prim=prim)
    sc.intersect(_t(org, cuda), _t(d, cuda), lo, hi, any_hit=True, out_prim=occ)
    want_t, want_p = oracle.intersect(tri, org, d, tmin, tmax)[:2]
    hit = want_p != 0xFFFFFFFF
    np.testing.assert_array_equal(prim.cpu().numpy().view(np.uint32) != 0xFFFFFFFF, hit)
    np.testing.assert_array_equal(t.cpu().numpy()[hit], want_t[hit])
    np.testing.assert_array_equal(occ.cpu().numpy() != -1, hit)


def test_training_scratch_is_given_back(cuda):
    """Forty guides at once hold 9.8 MB of training scratch each; when they are gone at most the 32 MB that
    the pool keeps stay with the process (and what the allocator rounds up to), and new guides train on
    it as on new memory."""
    import torch
    from rtlib_b200.mlp import MLPGuide
    rec = _records(5000, 3, cuda)
    def train():
        g = MLPGuide((0, 0, 0), (1, 1, 1), seed=9)
        return g.train(rec, batch=2000, epochs=1), g.params()
    want = train()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    guides = [MLPGuide((0, 0, 0), (1, 1, 1), seed=k) for k in range(40)]
    for g in guides:
        g.train(rec, batch=2000, epochs=1)
    held = before - torch.cuda.mem_get_info()[0]
    del guides, g
    torch.cuda.synchronize()
    kept = before - torch.cuda.mem_get_info()[0]
    assert held > 300e6 and kept < 80e6, (held, kept)
    got = train()
    assert got[0] == want[0]
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("ncell,level", [(1, 1), (52429, 1), (12483, 2), (50000, 2), (3084, 3), (13, 7)])
def test_morton_export_chunks(cuda, oracle, ncell, level):
    """Pyramids leave the device in chunks of 2^18 floats: less than one, exactly one cell past one, and
    several whose ends lie inside cells."""
    from rtlib_b200.hashgrid import MortonQuadTrees
    rng = np.random.default_rng(ncell)
    n = 20000
    m = MortonQuadTrees(ncell, level=level)
    cell, uv, val = rng.integers(0, ncell, n).astype(np.uint32), rng.random((n, 2), dtype=np.float32), rng.random(n, dtype=np.float32)
    cell[:2] = 0, ncell - 1
    leaves = np.zeros(ncell << (2 * level), np.int64)
    m.record(_t(cell, cuda), _t(uv, cuda), _t(val, cuda))
    oracle.mqt_record(level, 24, leaves, cell, uv, val)
    np.testing.assert_array_equal(m.export()[0], leaves)
    m.update()
    got_leaves, got = m.export()
    assert not got_leaves.any()
    np.testing.assert_array_equal(got, oracle.mqt_build(ncell, level, 24, leaves))
