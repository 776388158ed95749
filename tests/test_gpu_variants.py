"""Edges of the kernels' variants: tile remainders, the ends of each range that
a dispatch covers, and the calls on either side of its lines, each against the
oracle or against the general path of the same library."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# ---- partition and sort ------------------------------------------------------
# id bits: the batch bits inside one digit, across two, and at a digit's end
@pytest.mark.parametrize("id_bits", [1, 5, 6, 7, 8, 13, 14, 24])
@pytest.mark.parametrize("n", [0, 1, 4095, 4096, 4097, 33000])
def test_partition_at_digit_and_tile_edges(cuda, oracle, n, id_bits):
    from meturay_b200._lib import check, lib
    torch = cuda
    rng = np.random.default_rng(100 * id_bits + n)
    batch = rng.choice([0, 1, 2, 4, 6], n).astype(np.uint32)  # some batches absent
    keys = (batch << 24) | rng.integers(0, 1 << id_bits, n).astype(np.uint32)
    keys[batch == 0] = 0
    sid, sd = (torch.full((max(n, 1),), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    po, pe = (torch.full((8,), 77, dtype=torch.int32, device="cuda") for _ in range(2))
    nn = torch.full((1,), 77, dtype=torch.int32, device="cuda")
    tb = lib.mrb_partition_temp_bytes(n, id_bits)
    tmp = torch.zeros(tb, dtype=torch.uint8, device="cuda")
    check(lib.mrb_partition(_dev(torch, keys.view(np.int32)).data_ptr() if n else None, n, id_bits,
                            sid.data_ptr(), sd.data_ptr(), po.data_ptr(), pe.data_ptr(),
                            nn.data_ptr(), tmp.data_ptr(), tb, None))
    torch.cuda.synchronize()
    dense = ((keys >> 24) << id_bits) | (keys & ((1 << id_bits) - 1))
    order = np.argsort(-dense.astype(np.int64), kind="stable")
    assert np.array_equal(sid.cpu().numpy()[:n], order)
    assert np.array_equal(sd.cpu().numpy()[:n].view(np.uint32), dense[order])
    sorted_batch = batch[order]
    for b in range(8):
        at = np.nonzero(sorted_batch == b)[0]
        want = (at[0], at[-1] + 1) if len(at) else (0, 0)
        assert (int(po[b]), int(pe[b])) == want, b
    assert int(nn[0]) == n - int((batch == 0).sum())


def _sorted_on_device(torch, n, bits, seed):
    from meturay_b200._lib import check, lib
    gen = torch.Generator(device="cuda").manual_seed(seed)
    keys = torch.randint(0, 1 << bits, (n,), generator=gen, dtype=torch.int32, device="cuda")
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    orig = keys.clone()
    tb = lib.mrb_radix_sort_temp_bytes(n, 4, 0, bits)
    tmp = torch.empty(tb, dtype=torch.uint8, device="cuda")
    check(lib.mrb_radix_sort_pairs_u32(keys.data_ptr(), vals.data_ptr(), n, 0, bits, 0,
                                       tmp.data_ptr(), tb, None))
    torch.cuda.synchronize()
    return orig, keys, vals


# the lines between tiles of 1,024, 2,048 and 4,096 elements
@pytest.mark.parametrize("n", [1, 1024, 1025, 204_800, 204_801, 409_600, 409_601, 655_360, 655_361])
def test_sort_at_tile_size_lines(cuda, n):
    torch = cuda
    orig, keys, vals = _sorted_on_device(torch, n, 20, n)
    want, order = torch.sort(orig, stable=True)
    assert torch.equal(keys, want)
    assert torch.equal(vals.long(), order)


def _sorted_long_keys(torch, keys):
    """Stable sort by 63 bits; sorted keys, order and the microseconds of one."""
    from meturay_b200._lib import check, lib
    n = keys.shape[0]
    tb = lib.mrb_radix_sort_temp_bytes(n, 8, 0, 63)
    tmp = torch.empty(tb, dtype=torch.uint8, device="cuda")
    k, v = keys.clone(), torch.empty(n, dtype=torch.int32, device="cuda")
    best = float("inf")
    for _ in range(8):
        k.copy_(keys)
        torch.arange(n, out=v)
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        check(lib.mrb_radix_sort_pairs_u64(k.data_ptr(), v.data_ptr(), n, 0, 63, 0, tmp.data_ptr(),
                                           tb, None))
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return k, v, best


# a digit shared by a whole warp is ranked at once in the largest tiles only
@pytest.mark.parametrize("n", [5000, 300_000, 409_601, 1_000_003])
@pytest.mark.parametrize("distinct", [1, 40, 1 << 20, 1 << 62])
def test_sort_of_long_keys_with_few_and_many_digits(cuda, n, distinct):
    torch = cuda
    gen = torch.Generator(device="cuda").manual_seed(n)
    keys = torch.randint(0, distinct, (n,), generator=gen, device="cuda")
    if distinct == 40:
        keys <<= 50  # the distinct digit in one of the last passes
    k, v, _ = _sorted_long_keys(torch, keys)
    want, order = torch.sort(keys, stable=True)
    assert torch.equal(k, want) and torch.equal(v.long(), order)


def test_sort_of_few_distinct_long_keys_is_the_quicker_one(cuda):
    """All digits but one are the same in every key: 0.74 of the time of random
    keys with matches, 0.99 with a vote per bit of every digit."""
    torch = cuda
    gen = torch.Generator(device="cuda").manual_seed(1)
    few = torch.randint(0, 40, (4_000_000,), generator=gen, device="cuda")
    rand = torch.randint(0, 1 << 62, (4_000_000,), generator=gen, device="cuda")
    a, b = _sorted_long_keys(torch, few)[2], _sorted_long_keys(torch, rand)[2]
    assert a < 0.92 * b, (a, b)


def test_sort_beyond_the_numbered_flags(cuda):
    """More pairs than the pass-numbered tile flags hold (2^27): the words are
    cleared for every pass instead.  Values are the indices, so a stable sort
    leaves them ascending among equal keys."""
    torch = cuda
    n = (1 << 27) + 4097
    orig, keys, vals = _sorted_on_device(torch, n, 12, 4)
    assert bool((keys[1:] >= keys[:-1]).all())
    assert bool(((keys[1:] > keys[:-1]) | (vals[1:] > vals[:-1])).all())
    assert bool((orig[vals.long()] == keys).all())
    assert int(vals.long().sum()) == n * (n - 1) // 2


# ---- guiding network ---------------------------------------------------------
def _network_batch(seed, n):
    from oracle import mlp as M
    rng = np.random.default_rng(seed)
    x = M.encode(rng.uniform(0, 1, (n, 3)), M.sample_sphere(rng, n), M.sample_sphere(rng, n))
    t = np.zeros((n, 4), np.float32)
    t[:, :3] = M.sample_sphere(rng, n)
    t[:, 3] = rng.uniform(0.1, 2.0, n)
    t[rng.uniform(size=n) < 0.1, 3] = 0.0
    return x, t


# a lone row, the edges of a 128-row tile, and blocks with a second tile
# (592 inference blocks, 148 training blocks)
@pytest.mark.parametrize("n", [1, 127, 128, 129, 592 * 128 + 1])
def test_network_inference_at_tile_edges(system, cuda, n):
    from meturay_b200.learned import GuideMLP
    from oracle import mlp as M
    p = M.init_params(3)
    x, _ = _network_batch(n, n)
    out = cuda.full((n + 1, 40), -7.0, dtype=cuda.float32, device="cuda")
    GuideMLP(system, p).forward(_dev(cuda, x), out)
    cuda.cuda.synchronize()
    ref, _ = M.forward(p, x, quantize=True)
    got = out.cpu().numpy()
    # as test_gpu_mlp: rounding of the FP32 sums, and a bf16 flip that follows
    assert np.abs(got[:n] - ref).mean() < 1e-3 * np.abs(ref).mean()
    assert (got[n] == -7.0).all()  # nothing past the last row


@pytest.mark.parametrize("n", [1, 127, 129, 148 * 128 + 1])
def test_network_gradients_at_tile_edges(system, cuda, n):
    from meturay_b200.learned import PARAM_COUNT, GuideMLP
    from oracle import mlp as M
    p = M.init_params(5)
    x, t = _network_batch(7 * n, n)
    t[0, 3] = 1.0
    grad = cuda.zeros(PARAM_COUNT, dtype=cuda.float32, device="cuda")
    loss = cuda.zeros(2, dtype=cuda.float32, device="cuda")
    GuideMLP(system, p).gradients(_dev(cuda, x), _dev(cuda, t), grad, loss)
    cuda.cuda.synchronize()
    ref, lsum, wsum = M.gradients(p, x, t, quantize=True)
    got = grad.cpu().numpy().astype(np.float64)
    # the bound of test_gpu_mlp's gradients, over the whole vector
    assert np.linalg.norm(got - ref) < 2e-2 * np.linalg.norm(ref)
    assert abs(float(loss[0]) - lsum) < 1e-3 * abs(lsum) + 1e-3
    assert abs(float(loss[1]) - wsum) < 1e-4 * wsum
    assert (got[M.frozen_mask()] == 0).all()


# ---- traversal tree ----------------------------------------------------------
def _ploc_reference(boxes, radius=16):
    """Clustering steps and the sum of the inner boxes' half areas, in the same
    32-bit arithmetic."""
    c, steps, total = boxes.astype(np.float32), 0, 0.0
    while len(c) > 1:
        m = len(c)
        best, at = np.full(m, np.inf, np.float32), np.where(np.arange(m) == 0, 1, np.arange(m) - 1)
        for d in [*range(-radius, 0), *range(1, radius + 1)]:
            i = np.arange(max(0, -d), min(m, m - d))
            e = np.maximum(c[i, 3:], c[i + d, 3:]) - np.minimum(c[i, :3], c[i + d, :3])
            a = e[:, 0] * e[:, 1] + e[:, 1] * e[:, 2] + e[:, 2] * e[:, 0]
            less = a < best[i]
            best[i[less]], at[i[less]] = a[less], i[less] + d
        mutual = at[at] == np.arange(m)
        low, high = mutual & (np.arange(m) < at), mutual & (np.arange(m) > at)
        j = at[low]
        c[low] = np.concatenate([np.minimum(c[low, :3], c[j, :3]),
                                 np.maximum(c[low, 3:], c[j, 3:])], 1)
        e = c[low, 3:].astype(np.float64) - c[low, :3]
        total += float((e[:, 0] * e[:, 1] + e[:, 1] * e[:, 2] + e[:, 2] * e[:, 0]).sum())
        c, steps = c[~high], steps + 1
    return steps, total


# one block's range (1,024 clusters), the first step beyond it, tile remainders
@pytest.mark.parametrize("n", [2, 3, 33, 1023, 1024, 1025, 1281, 6000])
def test_ploc_steps_and_areas(system, cuda, n):
    from meturay_b200 import GPUScene, scenes
    scene = scenes.random_triangles(n, n)
    g = GPUScene(system, scene)
    g.set_wide_tree(1)
    g.construct_accelerators()
    a = g.export_accel()
    steps, area = _ploc_reference(a["tri_aabbs"][a["sorted_idx"]])
    info = g.accel_info()
    assert info["ploc_steps"] == steps
    # the same boxes, summed in double in another order
    assert abs(info["inner_area_ploc"] - area) <= n * 2.0 ** -52 * area
    g.construct_accelerators()  # again over the built scene
    assert g.accel_info()["ploc_steps"] == steps


def test_a_small_build_without_probes_does_not_pay_for_them(system, cuda):
    """A scene whose tree, collapse and kernel are named is built without the probe
    rays.  Their 3.4 MB allocated all the same made the build of ten triangles take
    0.8 of the time of one with probes; it takes 0.1 to 0.2 of it."""
    import time
    import meturay_b200 as m

    def seconds(probes):
        g = m.GPUScene(system, m.scenes.random_triangles(10, 10))
        if not probes:
            g.set_wide_tree(0)
            g.set_wide_collapse(0)
            g.set_wide_order("octant")
        g.construct_accelerators()
        best = float("inf")
        for _ in range(20):
            cuda.cuda.synchronize()
            t = time.perf_counter()
            g.construct_accelerators()
            cuda.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best

    plain, probed = seconds(False), seconds(True)
    assert plain < 0.5 * probed, (plain, probed)


# ---- reconstruction splat ----------------------------------------------------
def _bits_equal(a, b):
    return np.array_equal(np.asarray(a, np.float32).view(np.uint32),
                          np.asarray(b, np.float32).view(np.uint32))


def _splat(torch, ftype, radius, params, values, coords, res, segment=None):
    import meturay_b200 as m
    img = m.ImageMemory(res[0], res[1], 1 if values.ndim == 1 else 4)
    if segment is not None:
        ox, oy, w, h = segment
        img.reportion((ox, oy), (ox + w, oy + h))
    m.ReconFilter(ftype, radius, params).filter_to_img(img, _dev(torch, values),
                                                       _dev(torch, coords), coords.shape[0])
    torch.cuda.synchronize()
    return img.get_image()


def _longest_run(radius, coords, segment):
    """The most samples whose window touches one tile of 8 x 8 pixels."""
    import meturay_b200 as m
    wh = m.filter_pixel_wh(radius)
    ox, oy, w, h = segment
    c = coords[(np.abs(coords) < 1e9).all(1)]
    i = np.trunc(c).astype(np.int64)
    lo = i - (wh - 1) // 2 - ((wh % 2 == 0) & (c - i < 0.5)) - [ox, oy]
    hi = lo + wh
    lo, hi = np.maximum(lo, 0), np.minimum(hi, [w, h])
    keep = (lo < hi).all(1)
    a, b = lo[keep] // 8, (hi[keep] - 1) // 8
    runs = np.zeros(((h + 7) // 8 + 1, (w + 7) // 8 + 1), np.int64)  # as a 2D difference
    for x, y, v in ((a[:, 0], a[:, 1], 1), (b[:, 0] + 1, a[:, 1], -1), (a[:, 0], b[:, 1] + 1, -1),
                    (b[:, 0] + 1, b[:, 1] + 1, 1)):
        np.add.at(runs, (y, x), v)
    return int(runs.cumsum(0).cumsum(1).max())


CROWD = 128  # samples on a tile beyond which a block takes it and not two warps


# Radii below 0.75 go by pairs of pixel and sample, from there on by tiles of
# 8 x 8 pixels; windows of 1 to 5 pixels and one wider than a tile.  The numbers of
# samples give tiles of less than a warp's round, of several, and of one and several
# rounds of a block.
@pytest.mark.parametrize("ftype,radius,params", [
    ("Box", 0.0, {}), ("Box", 0.25, {}), ("Box", 0.5, {}), ("Tent", 0.74, {}), ("Tent", 0.75, {}),
    ("Tent", 1.0, {}), ("Box", 1.25, {}), ("Gaussian", 1.25, {"alpha": 1.0}),
    ("Mitchell", 2.0, {"b": 1 / 3, "c": 1 / 3}), ("Tent", 9.25, {})])
@pytest.mark.parametrize("channels", [1, 4])
@pytest.mark.parametrize("n", [300, 2000, 9000, 60_000])
def test_splat_windows_at_image_edges(cuda, oracle, ftype, radius, params, channels, n):
    import meturay_b200 as m
    rng = np.random.default_rng(int(radius * 100) + channels)
    w, h = 67, 41
    coords = np.stack([rng.uniform(-4, w + 4, n), rng.uniform(-4, h + 4, n)], 1).astype(np.float32)
    coords[:6] = [[0, 0], [w, h], [np.nan, 3], [3, np.inf], [2e9, 1], [-0.5, -0.5]]
    values = rng.uniform(0, 8, (n, channels)).astype(np.float32)
    values = values if channels == 4 else values[:, 0]
    seg = (5, 3, 50, 30)
    px, cnt = _splat(cuda, ftype, radius, params, values, coords, (w, h), seg)
    rp, rc = oracle.filter_to_img(ftype, radius, values, coords, (w, h), segment=seg, **params)
    assert _bits_equal(px, rp) and _bits_equal(cnt, rc)
    # the route that this case stands for: pairs and their sort's second copy fill
    # 16 bytes for each pixel of a window, tiles far less
    flt = m.ReconFilter(ftype, radius, params)
    img = m.ImageMemory(w, h, channels)
    img.reportion(seg[:2], (seg[0] + seg[2], seg[1] + seg[3]))
    flt.filter_to_img(img, _dev(cuda, values), _dev(cuda, coords), n)
    cuda.cuda.synchronize()
    if n >= 2000:
        assert (flt.used_gpu_memory() > 16 * n * m.filter_pixel_wh(radius) ** 2) == (radius < 0.75)
    if radius >= 0.75:
        blocks = n >= 9000 or (n >= 2000 and radius > 9.0)
        assert (_longest_run(radius, coords, seg) > CROWD) == blocks


# few and many crowded tiles (1,024 is the line), the many with and without runs
# that a block takes all the same (over 1,024 samples)
@pytest.mark.parametrize("w,h,per", [(40, 30, 7.9), (40, 30, 8.1), (256, 255, 8.1),
                                     (256, 256, 8.1), (280, 280, 8.1), (280, 280, 40.0)])
def test_splat_of_dense_samples(cuda, oracle, w, h, per):
    rng = np.random.default_rng(w + h)
    n = int(per * w * h / np.pi)  # radius 1
    coords = np.stack([rng.uniform(0, w, n), rng.uniform(0, h, n)], 1).astype(np.float32)
    values = rng.uniform(0, 4, (n, 4)).astype(np.float32)
    px, cnt = _splat(cuda, "Tent", 1.0, {}, values, coords, (w, h))
    rp, rc = oracle.filter_to_img("Tent", 1.0, values, coords, (w, h))
    assert _bits_equal(px, rp) and _bits_equal(cnt, rc)


def test_splat_of_crowded_pixels(cuda, oracle):
    """From none to hundreds of samples at a pixel; each pixel's sum is in the
    samples' order, so the bits are the oracle's."""
    rng = np.random.default_rng(8)
    w, h = 200, 150
    spots = [(20.5, 30.5, 9), (60.2, 70.9, 40), (120.0, 100.0, 700), (199.9, 149.9, 90)]
    coords = [np.array([x, y]) + rng.uniform(-1.2, 1.2, (k, 2)) for x, y, k in spots]
    coords.append(np.stack([rng.uniform(0, w, 3000), rng.uniform(0, h, 3000)], 1))
    coords = rng.permutation(np.concatenate(coords)).astype(np.float32)
    values = rng.uniform(0, 4, (len(coords), 4)).astype(np.float32)
    for ftype, radius, params in (("Tent", 1.0, {}), ("Gaussian", 2.0, {"alpha": 0.5})):
        px, cnt = _splat(cuda, ftype, radius, params, values, coords, (w, h))
        rp, rc = oracle.filter_to_img(ftype, radius, values, coords, (w, h), **params)
        assert _bits_equal(px, rp) and _bits_equal(cnt, rc)


def _splat_us(torch, coords, values, radius, res):
    """Microseconds of a splat, the best of some on the device."""
    import meturay_b200 as m
    img, flt = m.ImageMemory(res[0], res[1], 4), m.ReconFilter("Tent", radius)
    c, v = _dev(torch, coords), _dev(torch, values)
    best = float("inf")
    for _ in range(12):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        for _ in range(4):
            flt.filter_to_img(img, v, c, len(coords))
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 250.0)
    return best


def test_crowded_samples_cost_little_more_than_spread_ones(cuda):
    """200,000 samples on 30 x 30 pixels of a large image and all over it.  With a
    pair per pixel that a sample reaches the first took 2 to 2.5 times the second,
    and 8 times with one warp for every 8 x 4 pixels."""
    rng = np.random.default_rng(4)
    n, w, h = 200_000, 1920, 1080
    spread = rng.uniform(0, 1, (n, 2)).astype(np.float32)
    values = rng.uniform(0, 1, (n, 4)).astype(np.float32)
    few = _splat_us(cuda, spread * np.float32([w, h]), values, 1.0, (w, h))
    crowd = _splat_us(cuda, spread * np.float32(30.0) + np.float32([900, 500]), values, 1.0, (w, h))
    assert crowd < 4.0 * few, (crowd, few)


# ---- shadow rays -------------------------------------------------------------
@pytest.mark.parametrize("order", range(4))
@pytest.mark.parametrize("shielded,mis", [(False, 1), (True, 0)])
def test_shadow_rays_see_what_the_binary_traversal_sees(system, cuda, order, shielded, mis):
    """The 8-wide kernels report a next-event ray that its light's triangle does
    not end as a miss, the binary traversal reports what it hit.  Both run the
    same triangle test, so pixels differ by the order of their sums (a few ulp)
    but for paths that pass through two triangles at the same distance."""
    import meturay_b200 as m
    g = m.GPUScene(system, m.scenes.cornell(seed=1, shielded=shielded))
    g.construct_accelerators()

    def image(traversal):
        g.set_traversal(traversal)
        t = m.PathTracer(system, g)
        t.set_options({"Samples": 2, "MaxDepth": 4, "NextEventEstimation": 1,
                       "DirectLightMIS": mis, "RussianRouletteStart": 3, "Seed": 7})
        t.set_resolution(160, 120)
        for _ in range(4):
            t.render_frame()
        out = np.array(t.image())
        t.close()
        return out

    g.set_wide_order(order)
    wide, binary = image(1), image(0)
    assert wide[..., :3].sum() > 0
    differ = (np.abs(wide - binary) > 1e-5 * (1.0 + np.abs(binary))).any(-1)
    assert differ.mean() < 2e-3


# ---- few rays ----------------------------------------------------------------
# the lines are at 4,096 rays below 64 triangles, 8,192 below 256, 16,384 below 900,
# 24,576 below 3,000, and 32,768
@pytest.mark.parametrize("name,n", [
    *((s, n) for s in ("clusters", "cornell") for n in (1, 3, 4, 5, 2000, 32767, 32768, 32769)),
    *((s, n) for s in (2, 63) for n in (1, 4096, 4097)), (64, 8192), (255, 8193), (256, 16384),
    (899, 16385), (900, 24576), (2999, 24577), (3000, 32768)])
def test_few_rays_hit_what_a_lane_per_ray_hits(system, cuda, name, n):
    """Up to 32,768 rays, fewer over small scenes, a warp traces each ray, with the
    same triangle test: the distances are the same bits, and the triangles too but
    for ties."""
    import meturay_b200 as m
    torch = cuda
    scene = (m.scenes.clusters(1, n_clusters=40) if name == "clusters" else
             m.scenes.cornell(seed=1) if name == "cornell" else
             m.scenes.random_triangles(name, name))
    size = 100.0 if name == "clusters" else 1.0 if name == "cornell" else 10.0
    g = m.GPUScene(system, scene)
    g.construct_accelerators()
    gen = torch.Generator(device="cuda").manual_seed(n)
    o = torch.rand((n, 4), generator=gen, device="cuda") * size
    d = torch.randn((n, 4), generator=gen, device="cuda")
    d[:, :3] /= d[:, :3].norm(dim=1, keepdim=True)
    d[::5, 0] = 0.0  # directions within a plane and along an axis
    d[::10, 1] = 0.0
    o[:, 3] = 0.0
    d[:, 3] = 1000.0
    d[::7, 3] = 0.05 * size  # short rays

    def hits(order):
        g.set_wide_order(order)
        out = [torch.full((n,), -7, dtype=torch.int32, device="cuda") for _ in range(2)]
        out += [torch.full((n,), -7.0, device="cuda"), torch.full((n, 2), -7.0, device="cuda")]
        g.hit(o.data_ptr(), d.data_ptr(), n, *(x.data_ptr() for x in out))
        torch.cuda.synchronize()
        return out

    few, lanes = hits("auto"), hits("sorted")
    assert torch.equal(few[2], lanes[2])
    same = few[1] == lanes[1]
    assert int((~same).sum()) <= 1 + n // 1000
    assert torch.equal(few[0][same], lanes[0][same])
    assert torch.equal(few[3][same], lanes[3][same])


@pytest.mark.parametrize("triangles,n", [(12, 32768), (100, 32768), (300, 32768)])
def test_many_rays_over_a_small_scene_cost_no_more_than_a_lane_each(system, cuda, triangles, n):
    """A warp per ray took 1.5 to 2.4 times the fastest form of a lane per ray here."""
    import meturay_b200 as m
    torch = cuda
    g = m.GPUScene(system, m.scenes.random_triangles(triangles, triangles))
    g.construct_accelerators()
    gen = torch.Generator(device="cuda").manual_seed(n)
    o = torch.rand((n, 4), generator=gen, device="cuda") * 10.0
    d = torch.randn((n, 4), generator=gen, device="cuda")
    d[:, :3] /= d[:, :3].norm(dim=1, keepdim=True)
    o[:, 3], d[:, 3] = 0.0, 1000.0
    out = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2)]
    out += [torch.zeros(n, device="cuda"), torch.zeros((n, 2), device="cuda")]

    def micros(order):
        g.set_wide_order(order)
        best = float("inf")
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(20):
                g.hit(o.data_ptr(), d.data_ptr(), n, *(x.data_ptr() for x in out))
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 50.0)
        return best

    auto, lanes = micros("auto"), min(micros("sorted"), micros("octant"))
    assert auto < 1.3 * lanes, (auto, lanes)
