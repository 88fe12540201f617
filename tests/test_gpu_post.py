"""Image post-processing at sizes and addresses that fill no vector, warp or
block: batches of odd images behind a float's and an RGB byte's offset, more
images than a group, a single pixel, constant and non-positive images."""
import numpy as np
import pytest

import oracle as O
from libmeshlessvis_b200 import _lib as L
from libmeshlessvis_b200 import meshless as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,nx,ny", [(1, 1, 1), (3, 5, 7), (2, 33, 127), (5, 64, 64), (70, 31, 9), (1, 257, 513)])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_post_at_odd_sizes(count, nx, ny, offset):
    import torch

    rng = np.random.default_rng(nx * ny + offset)
    imgs = rng.uniform(-1.0, 9.0, (count, nx, ny)).astype(np.float32)
    imgs[0, 0, 0] = 12.0
    if count > 2:
        imgs[1] = 2.5
    n = imgs.size
    d_img = torch.zeros(n + offset, dtype=torch.float32, device="cuda")[offset:]
    d_img.copy_(torch.from_numpy(imgs.ravel()))
    whole = torch.full((3 * n + 2 * offset + 1,), -7.0, dtype=torch.float32, device="cuda")
    d_rgb = whole[offset:offset + 3 * n]
    cfg = M.Config(step=(1.0, 1.0), cutoff=(8, 4), samples=(16, 16), block_length=64)
    lib = M.lib()

    def rgb():
        cfg.synchronize()
        got = d_rgb.cpu().numpy().reshape(count, nx, ny, 3)
        rest = torch.cat((whole[:offset], whole[offset + 3 * n:])).cpu().numpy()
        assert np.all(rest == -7.0)  # nothing written past the images
        return got

    torch.cuda.synchronize()
    assert lib.vis_images_normalize_to_rgb(cfg.ptr, d_img.data_ptr(), count, L.int2(nx, ny), d_rgb.data_ptr()) == 0
    np.testing.assert_allclose(rgb(), O.normalize_to_rgb(imgs), rtol=1e-6, atol=1e-7)
    # 3e-7 of the value going in, 1e-6 of the logarithm quotient, through slopes of at most 10
    for log_scale, color_map in ((0, 1), (1, 2), (1, 3)):
        assert lib.vis_images_colormap(cfg.ptr, d_img.data_ptr(), count, L.int2(nx, ny), -1.0, 9.0, log_scale, color_map,
                                       d_rgb.data_ptr()) == 0
        np.testing.assert_allclose(rgb(), O.colormap(imgs, -1.0, 9.0, log_scale, color_map), rtol=2e-5, atol=2e-5)
    cfg.close()


def _rgb(cfg, call, imgs, *args):
    import torch

    d_img = torch.from_numpy(imgs).cuda()
    d_rgb = torch.empty(imgs.shape + (3,), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert call(cfg.ptr, d_img.data_ptr(), len(imgs), L.int2(*imgs.shape[1:]), *args, d_rgb.data_ptr()) == 0
    cfg.synchronize()
    return d_rgb.cpu().numpy()


@pytest.mark.parametrize("log_scale,color_map", [(0, 1), (1, 2), (0, 3)])
@pytest.mark.parametrize("scale", [1.0, 1e-29])
def test_colormap_of_infinities_nans_and_small_ranges(log_scale, color_map, scale):
    """Intensities below the range, and NaNs, take the first colour, those above
    it the last; a range as small as 1e-29 keeps its quotients."""
    rng = np.random.default_rng(color_map)
    imgs = (rng.uniform(-1.0, 4.0, (2, 33, 31)) * scale).astype(np.float32)
    imgs[0, 0, :3] = np.inf, -np.inf, np.nan
    imgs[1, 32, 30] = np.nan
    lo, hi = np.float32(0.0), np.float32(3.0 * scale)
    cfg = M.Config(step=(1.0, 1.0), cutoff=(8, 4), samples=(16, 16), block_length=64)
    got = _rgb(cfg, M.lib().vis_images_colormap, imgs, float(lo), float(hi), log_scale, color_map)
    cfg.close()
    finite = np.where(np.isnan(imgs) | (imgs == -np.inf), np.float32(-1.0 * scale), imgs)
    finite = np.where(imgs == np.inf, np.float32(9.0 * scale), finite)
    np.testing.assert_allclose(got, O.colormap(finite, float(lo), float(hi), log_scale, color_map), rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("shape", [(2, 25, 41), (1, 3, 683), (2, 64, 64), (3, 5, 7)])
@pytest.mark.parametrize("where", ["first", "first rows", "all", "infinite"])
def test_maximum_passes_over_nans(shape, where):
    """The scan from the first sample on passes over NaNs, also where a block has
    no pixels but the first sample (1025 and 2049 of them); an image of NaNs has
    none other, and an infinite maximum leaves zeros."""
    rng = np.random.default_rng(shape[2])
    imgs = rng.uniform(-1.0, 9.0, shape).astype(np.float32)
    if where == "first":
        imgs[:, 0, 0] = np.nan
    elif where == "first rows":
        imgs[:, :2] = np.nan
    elif where == "all":
        imgs[-1] = np.nan
    else:
        imgs[:, -1, -1] = np.inf
    cfg = M.Config(step=(1.0, 1.0), cutoff=(8, 4), samples=(16, 16), block_length=64)
    got = _rgb(cfg, M.lib().vis_images_normalize_to_rgb, imgs)
    cfg.close()
    expected = np.empty(shape)
    for e, img in zip(expected, imgs.astype(np.float64)):
        m = np.nan if np.isnan(img).all() else np.nanmax(img)
        e[:] = np.divide(np.maximum(img, 0.0), m, out=np.full(img.shape, np.nan), where=img < np.inf)
    np.testing.assert_allclose(got, np.repeat(expected[..., None], 3, axis=3), rtol=1e-6, atol=1e-7)
