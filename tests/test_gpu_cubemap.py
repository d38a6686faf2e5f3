"""Cube maps on the GPU (gbsp_create_cube_map / gbsp_create_irradiance_cube_map)
against the CPU restatement of src/cubemap.cpp, which matches the
reference's own code bit for bit on the same host.  The device uses CUDA's
sinf/cosf/atan2f, whose last bits differ from glibc's, so the bar is a
relative error: mean <= 1e-5 for the direct resampling, <= 1e-4 for the
irradiance integrals."""

import numpy as np
import pytest

from oracle import pyoracle
from vk_cinematic_gb300 import gbsp, scenes

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    d = np.abs(a[..., :3].astype(np.float64) - b[..., :3])
    return d / np.maximum(np.abs(b[..., :3]), 1e-3)


@pytest.fixture(scope="module")
def hdri():
    pyoracle.build_port()
    return scenes.equirect_hdri(512, 256)


def test_cube_map_matches_oracle(gpu_lib, hdri):
    import torch

    eq = torch.from_numpy(hdri).cuda()
    got = gbsp.create_cube_map(eq, 64, 48).cpu().numpy()
    ref = pyoracle.create_cube_map(hdri, 64, 48)
    e = rel_err(got, ref)
    print(f"cube map: mean rel err {e.mean():.3e}, max {e.max():.3e}")
    assert e.mean() <= 1e-5
    assert np.mean(e > 1e-3) < 1e-3  # only seam texels may move by a texel
    assert np.array_equal(got[..., 3], ref[..., 3])


@pytest.mark.parametrize("width,height", [(1, 1), (31, 9), (33, 7), (64, 8), (65, 1)])
def test_cube_map_ragged_sizes(gpu_lib, hdri, width, height):
    # blocks of 32 x 8 texels: one texel, a row and a column short, one over, exact;
    # the source's odd width leaves its rows at every alignment of a texel pair
    import torch

    src = np.ascontiguousarray(hdri[:255, :509])
    got = gbsp.create_cube_map(torch.from_numpy(src).cuda(), width, height).cpu().numpy()
    ref = pyoracle.create_cube_map(src, width, height)
    e = rel_err(got, ref)
    assert got.shape == ref.shape
    assert np.median(e) <= 1e-5
    assert np.mean(e > 1e-3) <= max(1e-3, 3 / e.size)


@pytest.mark.parametrize("mode,size,spp", [(gbsp.IRRADIANCE_UNIFORM, 12, 0),
                                           (gbsp.IRRADIANCE_RANDOM, 16, 32)])
def test_irradiance_matches_oracle(gpu_lib, hdri, mode, size, spp):
    import torch

    eq = torch.from_numpy(hdri).cuda()
    got = gbsp.create_irradiance_cube_map(eq, size, size, spp, mode).cpu().numpy()
    ref = pyoracle.create_irradiance_cube_map(hdri, size, size, spp, mode)
    e = rel_err(got, ref)
    print(f"irradiance mode {mode}: mean rel err {e.mean():.3e}, max {e.max():.3e}")
    assert e.mean() <= 1e-4
    assert np.all(got[..., 3] == 1.0)


def test_irradiance_random_stream_is_the_references(gpu_lib):
    # a constant environment: every sample is min(c * cosine, 10), so the
    # only inputs are the random offsets; texels far down the stream check
    # the GF(2) jump-ahead against the sequential stream of the oracle
    import torch

    flat = np.ones((32, 64, 4), np.float32)
    eq = torch.from_numpy(flat).cuda()
    got = gbsp.create_irradiance_cube_map(eq, 20, 20, 3, gbsp.IRRADIANCE_RANDOM).cpu().numpy()
    ref = pyoracle.create_irradiance_cube_map(flat, 20, 20, 3, 1)
    assert np.abs(got - ref).max() <= 1e-6


@pytest.mark.parametrize("width,height", [(700, 333), (1030, 517)])
def test_cube_map_rows_per_thread(gpu_lib, hdri, width, height):
    # sizes at which a thread takes two and four rows, the last ones past the map
    import torch

    src = np.ascontiguousarray(hdri[::4, ::4])
    got = gbsp.create_cube_map(torch.from_numpy(src).cuda(), width, height).cpu().numpy()
    ref = pyoracle.create_cube_map(src, width, height)
    e = rel_err(got, ref)
    assert e.mean() <= 1e-5
    assert np.mean(e > 1e-3) < 1e-3
    assert np.array_equal(got[..., 3], ref[..., 3])


@pytest.mark.parametrize("width,height,spp", [(5, 3, 1), (7, 2, 31), (6, 6, 33), (9, 4, 65), (33, 1, 64)])
def test_irradiance_random_splits_the_stream(gpu_lib, hdri, width, height, spp):
    # a warp per texel, a run of samples per lane: one sample, a lane short, a run
    # of two with idle lanes, a ragged last run, full runs
    import torch

    got = gbsp.create_irradiance_cube_map(torch.from_numpy(hdri).cuda(), width, height, spp,
                                          gbsp.IRRADIANCE_RANDOM).cpu().numpy()
    ref = pyoracle.create_irradiance_cube_map(hdri, width, height, spp, gbsp.IRRADIANCE_RANDOM)
    assert rel_err(got, ref).mean() <= 1e-4


@pytest.mark.parametrize("width,height,spp", [(65, 67, 1), (65, 67, 8), (65, 67, 33), (33, 31, 1), (131, 1, 1),
                                              (160, 90, 100), (64, 64, 34), (64, 64, 35)])
def test_irradiance_random_lane_per_texel(gpu_lib, hdri, width, height, spp):
    """Maps around the size from which a lane takes a whole texel, with a last
    warp that is partly past the map, at sample counts of one run and of
    several: the oracle's values.  With a constant image a texel is a sum of
    spp cosines over spp, whose float sums are off by at most spp 2^-24 on
    either side, besides the samples' own rounding (1e-6)."""
    import torch

    flat = np.ones((32, 64, 4), np.float32)
    got = gbsp.create_irradiance_cube_map(torch.from_numpy(flat).cuda(), width, height, spp,
                                          gbsp.IRRADIANCE_RANDOM).cpu().numpy()
    ref = pyoracle.create_irradiance_cube_map(flat, width, height, spp, gbsp.IRRADIANCE_RANDOM)
    assert np.abs(got - ref).max() <= 1e-6 + 2 * spp * 2.0 ** -24
    got = gbsp.create_irradiance_cube_map(torch.from_numpy(hdri).cuda(), width, height, spp,
                                          gbsp.IRRADIANCE_RANDOM).cpu().numpy()
    ref = pyoracle.create_irradiance_cube_map(hdri, width, height, spp, gbsp.IRRADIANCE_RANDOM)
    assert rel_err(got, ref).mean() <= 1e-4


@pytest.mark.parametrize("width,height", [(1, 700), (2, 257), (3, 129), (7, 64), (9, 33), (17, 40), (41, 300)])
def test_cube_map_narrow_blocks(gpu_lib, hdri, width, height):
    # widths for which a block is 1, 2, 8 and 16 texels wide, partly past the map's rows
    import torch

    got = gbsp.create_cube_map(torch.from_numpy(hdri).cuda(), width, height).cpu().numpy()
    ref = pyoracle.create_cube_map(hdri, width, height)
    e = rel_err(got, ref)
    assert np.median(e) <= 1e-5
    assert np.mean(e > 1e-3) <= max(1e-3, 3 / e.size)


def test_rejects_bad_arguments(gpu_lib):
    import torch

    eq = torch.zeros((8, 16, 4), dtype=torch.float32, device="cuda")
    with pytest.raises(gbsp.GbspError, match="mode"):
        gbsp.create_irradiance_cube_map(eq, 4, 4, 1, mode=7)
    with pytest.raises(gbsp.GbspError, match="empty"):
        gbsp.create_cube_map(eq, 0, 4)
