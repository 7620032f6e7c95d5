"""The four-wide walker (trace mode 3 on box hierarchies) against the
one-thread-per-ray escape walk (mode 0) and the oracle: identical bits at the
sizes and on the rays where the two could part."""
import numpy as np
import pytest

import oracle
from gpugi_gb300 import bvh, cuda, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = cuda.Context(0)
    yield c
    c.close()


def grid_scene(n=12):
    """Axis-aligned quads and boxes on a dyadic grid: flat leaf boxes whose planes bound their
    ancestors, many coplanar faces."""
    v, t = [], []

    def quad(o, a, b):
        k = len(v)
        v.extend([o, o + a, o + a + b, o + b])
        t.extend([[k, k + 1, k + 2, 0], [k, k + 2, k + 3, 0]])

    e = np.eye(3)
    for i in range(n):
        for j in range(n):
            o = np.array([i / 8, 0.0, j / 8])
            quad(o, e[0] / 8, e[2] / 8)
            if (i + j) % 3 == 0:
                for a in range(3):
                    quad(o + e[1] / 4, e[a] / 16, e[(a + 1) % 3] / 16)
                    quad(o + e[1] / 4 + e[(a + 2) % 3] / 16, e[a] / 16, e[(a + 1) % 3] / 16)
    return np.array(v, np.float32), np.array(t, np.uint32)


def soup(n, seed, size):
    """Large overlapping triangles: rays hit most boxes, so walks hold deep stacks."""
    r = np.random.default_rng(seed)
    c = r.uniform(-1, 1, (n, 1, 3))
    p = (c + size * r.uniform(-1, 1, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
    t = np.concatenate([np.arange(3 * n).reshape(n, 3), np.zeros((n, 1), int)], 1).astype(np.uint32)
    return p, t


def make_rays(o, d, tmax):
    a = np.concatenate([o, d, np.broadcast_to(np.asarray(tmax, np.float32).reshape(-1, 1), (len(o), 1))], 1)
    a = np.ascontiguousarray(a.astype(np.float32).T)
    return {k: np.ascontiguousarray(a[i]) for i, k in enumerate(cuda.RAY_KEYS)}


def special_rays(pos, seed, n):
    """Axis-parallel directions, origins on box planes and vertices, tiny and signed-zero components,
    finite, zero and infinite tmax, and non-finite rays."""
    r = np.random.default_rng(seed)
    o = r.uniform(pos.min(0) - 0.5, pos.max(0) + 0.5, (n, 3)).astype(np.float32)
    on = r.random((n, 3)) < 0.5
    o = np.where(on, pos[r.integers(0, len(pos), n)], o)
    d = r.normal(size=(n, 3)).astype(np.float32)
    d = np.where(r.random((n, 3)) < 0.4, np.float32(0), d)
    d = np.where(r.random((n, 3)) < 0.2, -np.abs(d) * np.float32(0), d)  # signed zeros
    d = np.where(r.random((n, 3)) < 0.03, d * np.float32(1e-40), d)      # denormals: 1 / d overflows
    d[np.all(d == 0, 1), 1] = -1
    tmax = r.choice(np.array([np.inf, 3.4e38, 1.0, 0.25, 0.0, 1e-4], np.float32), n)
    bad = r.integers(0, n, max(1, n // 50))
    d[bad, r.integers(0, 3, len(bad))] = r.choice(np.array([np.nan, np.inf, -np.inf], np.float32), len(bad))
    bad = r.integers(0, n, max(1, n // 50))
    o[bad, r.integers(0, 3, len(bad))] = r.choice(np.array([np.nan, np.inf, -np.inf], np.float32), len(bad))
    return make_rays(o, d, tmax)


def both_modes(ctx, ds, rays):
    got = {}
    for mode in (3, 0):
        ctx.set_trace_config(mode, 128)
        got[mode] = (cuda.trace_closest(ctx, ds, rays), cuda.trace_any(ctx, ds, rays))
    ctx.set_trace_config(3, 128)
    return got[3], got[0]


def same(a, b):
    for k in ("slot", "t", "u", "v"):
        assert np.array_equal(a[0][k].view(np.uint32), b[0][k].view(np.uint32)), k
    assert np.array_equal(a[1], b[1])


SCENES = {
    "grid": lambda: grid_scene(),
    "icosphere": lambda: (lambda s: (s["positions"], s["triangles"]))(scenes.displaced_icosphere(4096, seed=2)),
    "soup": lambda: soup(6000, 3, 0.8),
    "two": lambda: soup(2, 5, 1.0),
}


@pytest.mark.parametrize("watertight", [False, True])
@pytest.mark.parametrize("leaf", [1, 2, 8, 32])
@pytest.mark.parametrize("name", list(SCENES))
def test_equals_escape_walk(ctx, name, leaf, watertight):
    pos, tri = SCENES[name]()
    for b in ([bvh.build_bvh(pos, tri, method="sweep", leaf_size=leaf)] if leaf != 8 else
              [bvh.build_bvh(pos, tri, method=m, leaf_size=8) for m in ("sweep", "kdtree")]):
        ds = ctx.upload_scene(b, pos)
        ds.set_triangle_test(watertight)
        for rays in (special_rays(pos, 11, 20011), scenes.aimed_rays(4099, pos, seed=6)):
            a, z = both_modes(ctx, ds, rays)
            same(a, z)
        if not watertight:
            o = oracle.trace_closest(b, pos, rays)
            assert np.array_equal(a[0]["slot"], o["slot"])
            assert np.array_equal(a[0]["t"].view(np.uint32), o["t"].view(np.uint32))
            assert np.array_equal(a[1], oracle.trace_any(b, pos, rays)["occluded"])
        ds.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 4863, 4865, 20000, 155649, 700001])
def test_queue_lengths(ctx, n):
    """One ray per warp, part-filled warps, one full pass of the grid, and refills."""
    s = scenes.displaced_icosphere(16384, seed=4)
    ds = ctx.build_scene(s["positions"], s["triangles"])
    a, z = both_modes(ctx, ds, scenes.aimed_rays(n, s["positions"], seed=n))
    same(a, z)
    ds.close()


@pytest.mark.parametrize("fit", ["ellipsoid", "obox"])
@pytest.mark.parametrize("n", [3, 67000, 69000, 155649, 400001])
def test_binary_queue_lengths(ctx, fit, n):
    """Trees without a wide copy: both sides of the rule between groups and lanes (68,096 rays on 152
    SMs), one full pass of the grid and refills."""
    s = scenes.instanced_scene(seed=3, num_triangles=8000)
    b = bvh.build_bvh(s["positions"], s["triangles"], method="sweep", fit=fit)
    ds = ctx.upload_scene(b, s["positions"])
    a, z = both_modes(ctx, ds, scenes.aimed_rays(n, s["positions"], seed=n, spread=0.8))
    same(a, z)
    rays = special_rays(s["positions"], 5, min(n, 80001))
    same(*both_modes(ctx, ds, rays))
    ds.close()


@pytest.mark.parametrize("broken", ["not nested", "empty box", "nan box", "escape"])
def test_trees_that_do_not_nest(ctx, broken):
    """Hierarchies the upload accepts but the wide copy must not be made of."""
    s = scenes.displaced_icosphere(2048, seed=7)
    b = bvh.build_bvh(s["positions"], s["triangles"], method="sweep", leaf_size=8)
    h = b.hierarchy.copy()
    inner = np.nonzero((h[:, 3].view(np.uint32) & 0x80000000) == 0)[0]
    i = inner[len(inner) // 3]
    if broken == "not nested":
        h[i, 0:3] = 0.6 * h[i, 0:3] + 0.4 * h[i, 4:7]
    elif broken == "empty box":
        h[i, [0, 4]] = h[i, [4, 0]]
    elif broken == "nan box":
        h[i, 5] = np.nan
    else:  # a left child that escapes past its sibling
        left = h[i, 3].view(np.uint32)
        right = h[left, 7].view(np.uint32)
        h[left, 7] = h[right, 7]
    b.hierarchy = h
    ds = ctx.upload_scene(b, s["positions"])
    rays = scenes.aimed_rays(30011, s["positions"], seed=9)
    a, z = both_modes(ctx, ds, rays)
    same(a, z)
    o = oracle.trace_closest(b, s["positions"], rays)
    assert np.array_equal(a[0]["slot"], o["slot"])
    ds.close()


def test_chain_hierarchy(ctx):
    """A chain deeper than the walk's stack allows (geometric spacing makes the sweep peel one leaf
    at a time): whichever walker takes it, results are the escape walk's."""
    r = np.random.default_rng(8)
    x = np.cumsum(1.25 ** np.arange(160))
    p = (r.uniform(-0.3, 0.3, (160, 3, 3)) + np.stack([x, 0 * x, 0 * x], 1)[:, None]).reshape(-1, 3).astype(np.float32)
    t = np.concatenate([np.arange(480).reshape(160, 3), np.zeros((160, 1), int)], 1).astype(np.uint32)
    b = bvh.build_bvh(p, t, method="sweep", leaf_size=1)
    ds = ctx.upload_scene(b, p)
    rays = scenes.aimed_rays(20000, p[:60], seed=3)
    same(*both_modes(ctx, ds, rays))
    ds.close()


@pytest.mark.parametrize("size,samples", [(7, 1), (64, 1), (200, 5)])
def test_passes_and_batches(ctx, size, samples):
    """PT and LT images, singly and batched over two scenes, against the same calls on the binary
    walkers (trace mode 2): the same paths, so images differ only by the order of at most a few
    hundred float additions per pixel (2^-24 each, on sums of non-negative terms)."""
    from gpugi_gb300 import render
    sets = []
    for level, grid in ((3, 6), (2, 4)):
        s = scenes.cornell_room(seed=1, sphere_level=level, wall_grid=grid)
        b = bvh.build_bvh(s["positions"], s["triangles"], method="sweep")
        sets.append(ctx.upload_scene(b, s["positions"], cuda.vertex_info(s["normals"], s["texcoords"]), s["materials"]))
    cam = render.camera_lookat(*scenes.CORNELL_CAMERA, size, size)
    images = {}
    for mode in (2, 3):
        ctx.set_trace_config(mode, 128)
        out = []
        for pass_ in ("PT", "LT"):
            img = render.Image(ctx, size, size)
            render.render(ctx, sets[0], cam, img, pass_, max_path_length=6, samples=samples, rng_state=[5])
            out.append(img.read())
        jobs = [dict(scene=sets[k % 2], camera=cam, image=render.Image(ctx, size, size), pass_=("PT", "LT", "PT")[k],
                     samples=samples, max_path_length=6, rng_state=[7 + k]) for k in range(3)]
        render.render_batch(ctx, jobs)
        out += [j["image"].read() for j in jobs]
        images[mode] = out
    ctx.set_trace_config(3, 128)
    for a, z in zip(images[3], images[2]):
        assert z[..., :3].any()
        assert np.abs(a - z).max() <= 512 * 2.0 ** -24 * max(1.0, float(np.abs(z).max()))
    for s in sets:
        s.close()


@pytest.mark.parametrize("n", [1, 151, 153, 607, 609, 9728, 9729])
def test_direct_and_queued_small_calls(ctx, n):
    """Both sides of the rule between one launch and prefilter plus queue (two rays per warp of the
    full grid, 9,728 on 152 SMs), one block per SM and one more; unaligned arrays; a caller's stream."""
    import torch
    s = scenes.closed_icosphere(4, seed=2)
    ds = ctx.build_scene(s["positions"], s["triangles"])
    rays = special_rays(s["positions"], n, n)
    want = both_modes(ctx, ds, rays)[1]
    dev = {k: torch.from_numpy(np.concatenate([v[:1], v])).cuda()[1:] for k, v in rays.items()}  # 4-B aligned
    out = {k: torch.zeros(n + 1, dtype=torch.int32 if k == "slot" else torch.float32, device="cuda")[1:]
           for k in ("slot", "t", "u", "v")}
    occ = torch.zeros(n + 1, dtype=torch.uint8, device="cuda")[1:]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    cuda.trace_closest_device_async(ctx, ds, dev, out, stream.cuda_stream)
    cuda.trace_any_device_async(ctx, ds, dev, occ, stream.cuda_stream)
    torch.cuda.synchronize()
    same(({k: v.cpu().numpy() for k, v in out.items()}, occ.cpu().numpy()), want)
    ds.close()


@pytest.mark.parametrize("watertight", [False, True])
@pytest.mark.parametrize("leaf", [9, 16, 32])
@pytest.mark.parametrize("n", [3001, 20001, 200001])
def test_leaves_of_several_passes(ctx, n, leaf, watertight):
    """Overlapping coplanar triangles, up to 32 in a leaf: rounding puts hits just before the leaf's flat
    box, after which a closer one in a later pass of the same leaf still counts. A warp per ray (one
    launch, and from a queue) and the last rays of a lane walk."""
    r = np.random.default_rng(leaf)
    k = 64  # clusters of `leaf` triangles, each in its own plane z = const
    p = r.uniform(-1, 1, (k, leaf, 3, 3))
    p[..., 2] = r.uniform(-0.4, 0.4, (k, 1, 1))
    p += np.stack(np.meshgrid(4 * np.arange(8), 4 * np.arange(8), [0], indexing="ij"), -1).reshape(k, 1, 1, 3)
    p = p.reshape(-1, 3).astype(np.float32)
    t = np.concatenate([np.arange(len(p)).reshape(-1, 3), np.zeros((k * leaf, 1), int)], 1).astype(np.uint32)
    b = bvh.build_bvh(p, t, method="sweep", leaf_size=leaf)
    full = b.slots.reshape(-1, leaf, 4)
    assert ((full[..., 0] != full[..., 1]).sum(1) > 8).any()
    ds = ctx.upload_scene(b, p)
    ds.set_triangle_test(watertight)
    at = r.integers(0, k, n)
    target = p.reshape(k, -1, 3)[at].mean(1) + np.concatenate([r.uniform(-0.6, 0.6, (n, 2)), np.zeros((n, 1))], 1)
    o = target + np.concatenate([r.uniform(-1, 1, (n, 2)), r.uniform(1, 3, (n, 1)) * r.choice([-1, 1], (n, 1))], 1)
    d = target - o
    rays = make_rays(o, d / np.linalg.norm(d, axis=1, keepdims=True), np.full(n, np.inf))
    same(*both_modes(ctx, ds, rays))
    ds.close()


def entering_rays(pos, tri, n, seed):
    """Rays at triangles from outside: every one enters the scene's root bounds, so it is queued."""
    r = np.random.default_rng(seed)
    target = pos[tri[r.integers(0, len(tri), n), :3].astype(np.int64)].astype(np.float64).mean(1)
    d = r.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return make_rays(target - d * np.linalg.norm(np.ptp(pos, axis=0)), d, np.full(n, np.inf))


@pytest.mark.parametrize("name", ["grid", "icosphere", "soup"])
def test_scenes_have_a_wide_copy(ctx, name):
    """The other tests compare modes, which agree whichever walker serves mode 3: here it is seen that
    the builders' trees have the wide copy, with at most one wide node per inner node and the numbers
    that the root's block of 256 leaves unused."""
    pos, tri = SCENES[name]()
    made = [ctx.upload_scene(bvh.build_bvh(pos, tri, method=m, leaf_size=leaf), pos)
            for m, leaf in (("sweep", 1), ("sweep", 8), ("sweep", 32), ("kdtree", 8))]
    for ds in made + [ctx.build_scene(pos, tri)]:
        inner = (ds.num_nodes - 1) // 2
        assert (inner - 1) // 3 <= ds.wide_nodes() <= inner + 256
        ds.close()
    two = ctx.upload_scene(bvh.build_bvh(*SCENES["two"](), method="sweep", leaf_size=2), SCENES["two"]()[0])
    assert two.num_nodes == 1 and two.wide_nodes() == 0
    two.close()
    ds = ctx.upload_scene(bvh.build_bvh(pos, tri, method="sweep", fit="ellipsoid"), pos)
    assert ds.wide_nodes() == 0
    ds.close()


@pytest.mark.parametrize("broken", ["not nested", "empty box", "nan box", "escape"])
def test_broken_trees_have_no_wide_copy(ctx, broken):
    s = scenes.displaced_icosphere(2048, seed=7)
    b = bvh.build_bvh(s["positions"], s["triangles"], method="sweep", leaf_size=8)
    ok = ctx.upload_scene(b, s["positions"])
    assert ok.wide_nodes() > 0
    ok.close()
    h = b.hierarchy.copy()
    word = h[:, 3].view(np.uint32)
    inner = np.nonzero((word & 0x80000000) == 0)[0]
    for i in (inner[0], inner[len(inner) // 3], inner[-1]):
        g = h.copy()
        if broken == "not nested":  # one child sticks out by one float
            left = word[i]
            g[left, 4] = np.nextafter(g[i, 4], np.float32(np.inf))
        elif broken == "empty box":
            g[word[i], [0, 4]] = [g[i, 4], g[i, 0]]
        elif broken == "nan box":
            g[word[i], 5] = np.nan
        else:
            left = word[i]
            g[left, 7] = g[g[left, 7].view(np.uint32), 7]
        b.hierarchy = g
        ds = ctx.upload_scene(b, s["positions"])
        assert ds.wide_nodes() == 0, i
        ds.close()


@pytest.mark.parametrize("inner", [71, 72, 73, 100])
def test_chains_at_the_depth_limit(ctx, inner):
    """A chain of inner nodes, each with one leaf: three of them per wide level, so 72 are the 24 levels
    that the walk's stack holds and 73 keep the binary walkers. Boxes that all overlap fill the stack."""
    r = np.random.default_rng(inner)
    p = r.uniform(-1, 1, (inner + 1, 3, 3)).astype(np.float32)
    lo, hi = p.min(1), p.max(1)
    h = np.zeros((2 * inner + 1, 8), np.float32)
    for k in range(inner + 1):
        leaf = 2 * k + 1 if k < inner else 2 * inner
        h[leaf, 0:3], h[leaf, 4:7] = lo[k], hi[k]
        h[leaf, 3] = np.uint32(0x80000000 | k).view(np.float32)
        h[leaf, 7] = np.uint32(2 * k + 2 if k < inner else 0).view(np.float32)
        if k < inner:
            h[2 * k, 0:3], h[2 * k, 4:7] = lo[k:].min(0), hi[k:].max(0)
            h[2 * k, 3] = np.uint32(2 * k + 1).view(np.float32)  # its escape is 0: the last child of the last child
    slots = np.concatenate([np.arange(3 * (inner + 1)).reshape(-1, 3), np.zeros((inner + 1, 1), int)], 1).astype(np.int32)
    pos = p.reshape(-1, 3)
    b = bvh.build_bvh(pos, slots.astype(np.uint32), method="sweep", leaf_size=1)
    b.hierarchy, b.slots = h, slots
    ds = ctx.upload_scene(b, pos)
    assert (ds.wide_nodes() > 0) == (inner <= 72)
    for n in (999, 30001):
        same(*both_modes(ctx, ds, entering_rays(pos, slots, n, n)))
    ds.close()


@pytest.mark.parametrize("per_warp", [2, 5, 8, 32])
def test_rules_on_rays_per_warp(ctx, per_warp):
    """Both sides of each rule on the queue's length in rays per warp of the full grid (eight blocks of
    four warps per SM): one launch without a queue up to 2, whole warps up to 5 (any hit) and 8
    (closest hit), one ray per lane up to 32."""
    import torch
    s = scenes.displaced_icosphere(16384, seed=4)
    ds = ctx.build_scene(s["positions"], s["triangles"])
    assert ds.wide_nodes() > 0
    at = per_warp * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    for n in (at, at + 1):
        same(*both_modes(ctx, ds, entering_rays(s["positions"], s["triangles"], n, n)))
    ds.close()


def test_memory_of_the_wide_copy():
    """Trees of a million nodes, where the copy's upper bound (64 B a node) and its scratch (20 B) are
    tens of megabytes: an accepted scene holds 128 B per wide node beside its arrays, one that fails the
    checks nothing, and no scratch stays behind. 8 MiB of slack for the allocator's rounding."""
    import torch
    mib = 1 << 20
    s = scenes.heightfield_boxes(seed=1, grid=500)
    pos, tri = s["positions"], s["triangles"]
    c = cuda.Context(0)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info(0)[0]

    first = c.build_scene(pos, tri, leaf_size=1)  # modules and the builder's own buffers are loaded
    b = first.export()
    first.close()
    before = free()
    arrays = 32 * len(b.hierarchy) + (16 + 48) * len(b.slots) + 12 * len(pos)
    assert len(b.hierarchy) > 1_000_000
    ds = c.upload_scene(b, pos)
    wide = ds.wide_nodes()
    assert wide > 0 and before - free() <= arrays + 128 * wide + 8 * mib
    ds.close()
    assert before - free() <= 8 * mib
    b.hierarchy[b.hierarchy[0, 3].view(np.uint32), 4] = np.nextafter(b.hierarchy[0, 4], np.float32(np.inf))
    ds = c.upload_scene(b, pos)
    assert ds.wide_nodes() == 0 and before - free() <= arrays + 8 * mib
    ds.close()
    c.close()
    # the scratch of a build goes with the call
    c = cuda.Context(0)
    small = c.build_scene(pos, tri[:1000], leaf_size=1)
    before = free()
    ds = c.build_scene(pos, tri, leaf_size=1)
    assert ds.wide_nodes() > 0
    ds.close()
    assert before - free() <= 8 * mib
    small.close()
    c.close()


@pytest.mark.parametrize("watertight", [False, True])
@pytest.mark.parametrize("fit", ["ellipsoid", "obox"])
def test_group_and_lane_rule(ctx, fit, watertight):
    """Trees without a wide copy: queues on both sides of the rule between 8-lane groups and lanes (48
    rays per block, eight blocks per SM: 58,368 on 152 SMs), every ray entering the scene."""
    import torch
    s = scenes.instanced_scene(seed=3, num_triangles=8000)
    pos, tri = s["positions"], s["triangles"]
    ds = ctx.upload_scene(bvh.build_bvh(pos, tri, method="sweep", fit=fit), pos)
    ds.set_triangle_test(watertight)
    assert ds.wide_nodes() == 0
    at = 48 * 8 * torch.cuda.get_device_properties(0).multi_processor_count
    for n in (at - 1, at):
        same(*both_modes(ctx, ds, entering_rays(pos, tri, n, n)))
    ds.close()


@pytest.mark.parametrize("share", [1, 50, 99, 100])
@pytest.mark.parametrize("streams", [1, 3, 4, 9])
def test_shares_over_streams(ctx, streams, share):
    """Stream-ordered walks on every grid that the share and the number of streams lead to, more streams
    than the context has scratch sets for among them: the synchronous calls' results."""
    import torch
    s = scenes.displaced_icosphere(16384, seed=4)
    ds = ctx.build_scene(s["positions"], s["triangles"])
    assert ds.wide_nodes() > 0
    n = [30001, 70001]
    host = [entering_rays(s["positions"], s["triangles"], k, k) for k in n]
    want = [(cuda.trace_closest(ctx, ds, r), cuda.trace_any(ctx, ds, r)) for r in host]
    dev = [{k: torch.from_numpy(v).cuda() for k, v in r.items()} for r in host]
    calls = 2 * streams + 9
    outs = [({k: torch.empty(n[i % 2], dtype=torch.int32 if k == "slot" else torch.float32, device="cuda")
              for k in ("slot", "t", "u", "v")}, torch.empty(n[i % 2], dtype=torch.uint8, device="cuda"))
            for i in range(calls)]
    queue = [torch.cuda.Stream() for _ in range(streams)]
    torch.cuda.synchronize()
    ctx.set_async_walker_share(share)
    for i, (o, occ) in enumerate(outs):
        cuda.trace_closest_device_async(ctx, ds, dev[i % 2], o, queue[i % streams].cuda_stream)
        cuda.trace_any_device_async(ctx, ds, dev[i % 2], occ, queue[i % streams].cuda_stream)
    torch.cuda.synchronize()
    ctx.set_async_walker_share(50)
    for i, (o, occ) in enumerate(outs):
        same(({k: v.cpu().numpy() for k, v in o.items()}, occ.cpu().numpy()), want[i % 2])
    assert ctx.device_error_bits() == 0
    ds.close()


@pytest.mark.parametrize("streams", [2, 4])
@pytest.mark.parametrize("entering", [0, 1, 5000, 70000, 400000])
def test_long_host_batches_over_streams(ctx, streams, entering):
    """2^20 + 1 rays in page-locked arrays of which 0 to 400,000 enter the scene: the walker's whole grid,
    the least part of it and the part that the queue's length gives (three streams and more)."""
    import ctypes

    import torch
    s = scenes.displaced_icosphere(16384, seed=4)
    pos, tri = s["positions"], s["triangles"]
    ds = ctx.build_scene(pos, tri)
    n = (1 << 20) + 1
    away = make_rays(np.full((n, 3), 10.0) * np.ptp(pos, axis=0).max(), np.full((n, 3), 3 ** -0.5), np.full(n, np.inf))
    at = np.sort(np.random.default_rng(entering).permutation(n)[:entering])
    rays = torch.empty((7, n)).pin_memory().numpy()
    hit = entering_rays(pos, tri, max(1, entering), 3)
    for k, key in enumerate(cuda.RAY_KEYS):
        rays[k] = away[key]
        rays[k, at] = hit[key][:entering]
    want = cuda.trace_closest(ctx, ds, dict(zip(cuda.RAY_KEYS, rays)))
    want_any = cuda.trace_any(ctx, ds, dict(zip(cuda.RAY_KEYS, rays)))
    queue = [torch.cuda.Stream() for _ in range(streams)]
    out = [torch.empty((4, n)).pin_memory().numpy() for _ in range(streams)]
    occ = [torch.empty(n, dtype=torch.uint8).pin_memory().numpy() for _ in range(streams)]
    lib, P = cuda.lib(), ctypes.c_void_p
    lib.gpugi_trace_closest_async.argtypes = [P] * 9 + [ctypes.c_uint64] + [P] * 5
    lib.gpugi_trace_any_async.argtypes = [P] * 9 + [ctypes.c_uint64] + [P] * 2
    for _ in range(4):
        for q, o, c in zip(queue, out, occ):
            src = [r.ctypes.data for r in rays]
            ctx.check(lib.gpugi_trace_closest_async(ctx.handle, ds.handle, *src, n, *[r.ctypes.data for r in o],
                                                    q.cuda_stream))
            ctx.check(lib.gpugi_trace_any_async(ctx.handle, ds.handle, *src, n, c.ctypes.data, q.cuda_stream))
    torch.cuda.synchronize()
    assert (want["slot"] >= 0).sum() >= 0.5 * entering
    for o, c in zip(out, occ):
        same((dict(zip(("slot", "t", "u", "v"), o)), c), (want, want_any))
    assert ctx.device_error_bits() == 0
    ds.close()
