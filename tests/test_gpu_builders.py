"""The volume's builders (baked NEE grid, HG table, TR levels, occupancy and
pyramid) at the sizes and inputs where their kernels take another branch,
against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def blob(R, lo, hi, seed=3, negative=False):
    """Zero but for the box [lo, hi) per axis."""
    d = np.zeros((R, R, R), np.float32)
    rng = np.random.default_rng(seed)
    d[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = rng.uniform(-0.1 if negative else 0.05, 1.0,
                                                            [h - l for l, h in zip(lo, hi)])
    return d


@pytest.mark.parametrize("light", [(0.0, 1.0, 0.0), (0.0, 0.0, -1.0), (0.36, -0.48, 0.8)])
@pytest.mark.parametrize("replicate", [True, False])
@pytest.mark.parametrize("R,lo,hi,storage", [(24, (2, 9, 3), (9, 20, 24), "fp32"), (17, (0, 0, 0), (17, 17, 17), "fp16"),
                                             (24, (0, 0, 0), (0, 0, 0), "fp32"), (40, (30, 1, 12), (31, 2, 13), "fp32")])
def test_baked_voxels(light, replicate, R, lo, hi, storage):
    """Every voxel's estimate follows the oracle's draws.  A logarithm's last
    bit moves a step by up to 2^-23 and its density by that times R times the
    voxel-to-voxel slope (below 1), a few steps a walk: below 1e-4; a walk
    takes another course where a comparison falls into such a gap: far below
    1 % of the voxels.  Lights along an axis, an off-centre and a one-voxel
    box, a full one and an empty one."""
    import mrpnn_b200 as M
    M.init()
    B, alpha = 13, 40.0
    data = blob(R, lo, hi)
    if storage == "fp16":
        data = data.astype(np.float16).astype(np.float32)
    v = M.VolumeRender(R, storage=storage)
    v.set_data(data)
    v.Update()
    v.SetBakeResolution(B, replicate)
    v.Update_CachedTR(light, alpha)
    got = v.read(M.api.RES_BAKED_TR)
    sc = O.SceneBuf(data.ravel(), R, v.max_density)
    ref = O.baked_tr_voxels(sc, alpha, np.array(light, np.float32), B, 0, np.arange(B ** 3), replicate)
    assert np.mean(np.abs(got - ref) > 1e-4) < 0.01


@pytest.mark.parametrize("g,seed", [(0.857, 5), (0.65, 0), (0.0, 1), (-0.8, 2), (0.00005, 3)])
def test_hg_table_texels(g, seed):
    """The table's kinds of sample (only cone samples at g = 0 and below 0.6,
    both above), its corners and a random choice, with the bars of the
    existing table test: a texel can flip one of its 1024 samples between the
    kinds when a transcendental differs in the last bit."""
    import mrpnn_b200 as M
    M.init()
    rng = np.random.default_rng(seed)
    tex = np.unique(np.concatenate([[0, 511, 512 * 511, 512 * 512 - 1, 127, 128, 255, 256],
                                    rng.choice(512 * 512, 1500, replace=False)])).astype(np.int32)
    v = M.VolumeRender(16)
    v.SetSeed(seed)
    v.UpdateHGLut(g)
    got = v.read(M.api.RES_LUT)[tex]
    ref = O.hg_lut_texels(g, seed, tex)
    rel = np.abs(got - ref) / np.maximum(np.abs(ref), 1e-6)
    assert np.mean(rel < 1e-4) > 0.995, np.sort(rel)[-10:]
    assert np.max(rel) < 0.05


@pytest.mark.parametrize("g,texels", [(2.0, (224430, 245486, 246279, 250037, 251486)), (-3.0, (242611, 250729)),
                                      (-1.25, (254390, 261580)), (40.0, (220822, 233584, 234644))])
def test_hg_table_infinite_cosine(g, texels):
    """An asymmetry above 1, which the entry points accept: one phase sample
    of each of these texels divides by 1 - g + 2 g e = 0.  Its direction is
    not a number and counts as 0.  The texels are 1e9 and more from samples
    beside the pole, whose cosine takes IEEE operations alone, so the bar is
    that of the table test's texels without a flipped sample."""
    import mrpnn_b200 as M
    M.init()
    tex = np.array(texels, np.int32)
    v = M.VolumeRender(16)
    v.UpdateHGLut(g)
    ref = O.hg_lut_texels(g, 0, tex)
    assert np.all(ref > 1e9) and np.all(np.isfinite(ref))
    np.testing.assert_allclose(v.read(M.api.RES_LUT)[tex], ref, rtol=1e-4)


@pytest.mark.parametrize("light", [(0.0, 1.0, 0.0), (0.0, 0.0, -1.0), (0.36, -0.48, 0.8), (-0.99, 0.1, 0.1)])
@pytest.mark.parametrize("R,lo,hi", [(64, (0, 0, 0), (64, 64, 64)), (40, (30, 1, 12), (31, 2, 13)),
                                     (33, (0, 31, 7), (5, 33, 26)), (24, (0, 0, 0), (0, 0, 0))])
def test_tr_levels(light, R, lo, hi):
    """All eight levels, rays along an axis and along the grid's faces, dense
    to the border, in one corner, a single voxel and an empty grid; the
    exponential's last bits are what may differ (the bar of the existing TR
    test)."""
    import mrpnn_b200 as M
    M.init()
    data = blob(R, lo, hi)
    v = M.VolumeRender(R)
    v.set_data(data)
    v.Update()
    v.Update_TR(light, 48.0)
    mips = np.concatenate([v.read(M.api.RES_MIP, m) for m in range(9)])
    got = np.concatenate([v.read(M.api.RES_TR, m) for m in range(8)])
    ref = O.tr_mips(mips, 48.0, np.array(light, np.float32))
    np.testing.assert_allclose(got, ref, rtol=2e-6, atol=1e-7)


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
@pytest.mark.parametrize("R", [2, 7, 8, 9, 31, 33, 64, 70, 129, 1030])
def test_scan(R, storage):
    """Occupancy bricks and majorant at grid edges around the bricks' and the
    row masks' sizes (8, 32 and 1024 voxels), from voxels at corners, at brick
    and mask borders and inside: a brick is set exactly when a nonzero voxel
    lies in [8 b - 1, 8 b + 9] per axis; a negative voxel and a NaN count as
    nonzero and never as the majorant."""
    import torch

    import mrpnn_b200 as M
    M.init()
    if R > 1024 and storage == "fp32":
        pytest.skip("one storage type is enough for the long rows")
    rng = np.random.default_rng(R)
    at = {(0, 0, 0), (R - 1, R - 1, R - 1), (R // 2, 0, R - 1), (min(7, R - 1), min(8, R - 1), min(9, R - 1)),
          (0, R - 1, min(31, R - 1)), (0, R // 3, min(32, R - 1)), (R - 1, R // 3, min(1023, R - 1)),
          (R // 3, 1, min(1024, R - 1))} | {tuple(rng.integers(0, R, 3)) for _ in range(6)}
    d = torch.zeros((R, R, R), device="cuda")
    vals = [-0.5, float("nan")] + [0.25 + 0.125 * k for k in range(len(at))]
    nb = (R + 7) // 8
    want = np.zeros((nb, nb, nb), np.uint8)
    top = 1e-5
    for (x, y, z), val in zip(sorted(at), vals):
        d[x, y, z] = val
        top = max(top, val) if val == val else top
        r = [[b for b in range(nb) if 8 * b - 1 <= c <= 8 * b + 9] for c in (x, y, z)]
        want[np.ix_(*r)] = 1
    v = M.VolumeRender(R, storage=storage)
    torch.cuda.synchronize()
    v.set_data(d)
    v.Update(process_mips=R <= 129)
    np.testing.assert_array_equal(v.read(M.api.RES_OCCUPANCY).reshape(nb, nb, nb), want)
    assert v.max_density == np.float32(top)


@pytest.mark.parametrize("R", [2, 3, 100, 255, 257, 300])
def test_pyramid_levels(R):
    """The pyramid of grids below, at and above 256 and of two voxels,
    negative voxels among them: bit-exact against the oracle."""
    import mrpnn_b200 as M
    M.init()
    data = np.random.default_rng(R).uniform(-0.2, 1.0, R ** 3).astype(np.float32)
    v = M.VolumeRender(R)
    v.set_data(data)
    v.Update()
    ref = O.split_levels(O.build_pyramid(data, R), O.mip_sizes())
    for m in range(9):
        np.testing.assert_array_equal(v.read(M.api.RES_MIP, m), ref[m].ravel(), err_msg=f"mip {m}")


def bake(R, data, B, light, alpha, replicate, tr_scale=1.0, majorant=None):
    """A baked grid and the oracle's, from the same draws."""
    import mrpnn_b200 as M
    M.init()
    v = M.VolumeRender(R)
    v.set_data(data)
    v.Update()
    if majorant is not None:
        v.max_density = majorant
    v.SetTrScale(tr_scale)
    v.SetBakeResolution(B, replicate)
    v.Update_CachedTR(light, alpha)
    sc = O.SceneBuf(data.ravel(), R, v.max_density, tr_scale=tr_scale)
    return (v.read(M.api.RES_BAKED_TR),
            O.baked_tr_voxels(sc, alpha, np.array(light, np.float32), B, 0, np.arange(B ** 3), replicate))


@pytest.mark.parametrize("replicate", [True, False])
@pytest.mark.parametrize("alpha,tr_scale", [(-40.0, 1.0), (40.0, -0.5)])
def test_bake_walks_backwards(alpha, tr_scale, replicate):
    """A negative extinction or step scale, which the entry points accept,
    walks away from the light: the oracle's draws and its estimate.  The bar
    is test_baked_voxels'; a third of the voxels and more see the blob
    behind them."""
    got, ref = bake(24, blob(24, (6, 6, 6), (18, 18, 18)), 9, (0.36, -0.48, 0.8), alpha, replicate, tr_scale)
    assert np.mean(ref < 1.0) > 0.2
    assert np.mean(np.abs(got - ref) > 1e-4) < 0.01


@pytest.mark.parametrize("replicate", [True, False])
@pytest.mark.parametrize("alpha,tr_scale", [(-8.0, 1.0), (8.0, -0.5)])
def test_bake_walks_back_and_forth(alpha, tr_scale, replicate):
    """A backward walk into a negative density (a distance) is carried forward
    by it, here past the far side, from where its next steps bring it back
    into the cloud.  Both densities are constant, so a jump moves by no more
    than its step's rounding; only in the one voxel between them does it
    stretch that (by 2 a voxel's length, 48), once or twice a walk: below
    1e-4, and the bar of the other walks holds."""
    data = np.full((24, 24, 24), -1.5, np.float32)
    data[:, :, 12:] = 0.25
    got, ref = bake(24, data, 9, (0.0, 0.0, 1.0), alpha, replicate, tr_scale)
    assert np.mean(np.abs(got - ref) > 1e-4) < 0.01


@pytest.mark.parametrize("R,storage", [(2, "fp32"), (64, "fp16"), (200, "fp32"), (1030, "fp16")])
def test_device_bytes(R, storage):
    """mrp_volume_info counts what a volume holds from its creation on and
    the baked grid: the grid, the pyramid and TR levels with their padded,
    paired and z-paired copies, the LUT with its tables, the occupancy with
    its scratch rows."""
    import mrpnn_b200 as M
    M.init()
    pad = 11 ** 3 + 7 ** 3 + 5 ** 3
    floats = sum((256 >> m) ** 3 for m in range(9)) + pad + sum((128 >> m) ** 3 for m in range(8)) + pad
    floats += 512 * 512 + 160 + 192 * 514
    pairs = sum((256 >> m) ** 3 for m in range(1, 5)) + sum(((128 >> m) + 2) ** 3 for m in range(8)) + pad
    rows = max(R * R * -(-R // 1024), sum((256 >> m) ** 2 for m in range(5)))
    nb = -(-R // 8)
    flags = sum((32 >> m) ** 3 for m in range(5)) + nb ** 3 + (-(-nb // 4)) ** 3 + 32
    want = R ** 3 * (2 if storage == "fp16" else 4) + 4 * floats + 8 * pairs + 16 * rows + flags
    v = M.VolumeRender(R, storage=storage)
    held = v.info().device_bytes
    assert want <= held < want + 5 * 256      # (five parts, each from a 256-byte boundary on)
    if R == 64:
        v.set_data(np.zeros((R, R, R), np.float32))
        v.Update()
        v.SetBakeResolution(21)
        v.Update_CachedTR((0.0, 1.0, 0.0), 1.0)
        assert v.info().device_bytes == held + 21 ** 3 * 4


@pytest.mark.parametrize("light", [(0.0, 1.0, 0.0), (0.0, 0.0, -1.0), (0.36, -0.48, 0.8)])
@pytest.mark.parametrize("R,lo,hi,B", [(40, (30, 26, 12), (31, 27, 13), 53), (24, (17, 3, 9), (20, 6, 12), 29),
                                       (32, (3, 9, 20), (4, 28, 21), 41)])
def test_bake_small_boxes(light, R, lo, hi, B):
    """One voxel, a small cube and a line of voxels, and a bake grid fine
    enough that a hundred voxels and more see them.  The steps are far
    shorter than a voxel, so the estimates' bar of 1e-4 holds as in
    test_baked_voxels, and walks that take another course stay below 1 % of
    the voxels that see the box."""
    got, ref = bake(R, blob(R, lo, hi), B, light, 400.0, True)
    seen = int(np.count_nonzero(ref < 1.0))
    assert seen >= 100
    assert np.count_nonzero(np.abs(got - ref) > 1e-4) <= 0.01 * seen


@pytest.mark.parametrize("replicate", [True, False])
def test_bake_majorant_below_density(replicate):
    """A majorant set below the density makes single estimates negative (the
    ratio factor 1 - S / majorant is); they enter the mean as they are."""
    got, ref = bake(24, blob(24, (6, 6, 6), (18, 18, 18)), 13, (0.36, -0.48, 0.8), 40.0, replicate, majorant=0.4)
    assert np.mean(ref < 0.0) > 0.01
    assert np.mean(np.abs(got - ref) > 1e-4) < 0.01


@pytest.mark.parametrize("light", [(float("nan"), 0.6, 0.8), (0.6, 0.8, float("nan")), (0.0, 0.0, 0.0)])
def test_tr_levels_odd_lights(light):
    """A light with a component that is not a number, whose rays have no place
    in the cube and go by the general fetches, and one of no length, whose
    steps stay where they are: what the oracle's fetches give (not a number
    for the first two)."""
    import mrpnn_b200 as M
    M.init()
    v = M.VolumeRender(24)
    v.set_data(blob(24, (6, 6, 6), (18, 18, 18)))
    v.Update()
    v.Update_TR(light, 48.0)
    mips = np.concatenate([v.read(M.api.RES_MIP, m) for m in range(9)])
    got = np.concatenate([v.read(M.api.RES_TR, m) for m in range(8)])
    ref = O.tr_mips(mips, 48.0, np.array(light, np.float32))
    np.testing.assert_allclose(got, ref, rtol=2e-6, atol=1e-7)


@pytest.mark.parametrize("axis,start", [(0, 0), (0, 1027), (1, 1027), (2, 0), (2, 1022), (2, 1027)])
def test_scan_long_rows(axis, start):
    """Rows longer than one mask segment (1024 voxels) in fp32: the occupancy
    of a slab of three voxels, and its bounds, which decide where the walks of
    a bake begin and end.  A ray toward the slab has 11 expected steps in it
    (3 voxels of 1 / 1030 at 4000 a unit length) and reads 1 only where none
    falls there: one voxel of 100 000; with bounds that miss the slab, every
    one does."""
    import torch

    import mrpnn_b200 as M
    M.init()
    R, nb = 1030, 129
    d = torch.zeros((R, R, R), device="cuda")
    d.narrow(axis, start, 3).fill_(1.0)
    v = M.VolumeRender(R)
    torch.cuda.synchronize()
    v.set_data(d)
    del d
    torch.cuda.empty_cache()
    v.Update(process_mips=False)
    want = np.zeros((nb, nb, nb), np.uint8)
    bricks = [b for b in range(nb) if 8 * b - 1 <= start + 2 and start <= 8 * b + 9]
    np.moveaxis(want, axis, 0)[bricks] = 1
    np.testing.assert_array_equal(v.read(M.api.RES_OCCUPANCY).reshape(nb, nb, nb), want)
    assert v.max_density == 1.0
    light = np.zeros(3, np.float32)
    light[axis] = 1.0 if start else -1.0
    v.SetBakeResolution(13)
    v.Update_CachedTR(light, 4000.0)
    assert np.mean(v.read(M.api.RES_BAKED_TR) < 1.0) > 0.99
