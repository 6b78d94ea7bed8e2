"""cf_render_lit where one warp holds pixels that end at different places of
the shader: off the canvas, on bare canvas far from paint, near paint, and
lanes outside the picture.  Every block has to pass its barriers together, and
each pixel is the one a view of many more pixels holds at the same place, bit
for bit, where whole blocks end alike."""
import numpy as np
import pytest

from canvaz_film import camera, capi

pytestmark = pytest.mark.gpu

W, H, VIEW = 40, 32, (9, 35)
PAINTED = 2  # the tile column that holds paint: columns 0-15 are far from it


def film():
    import __graft_entry__ as g
    g.build()
    from canvaz_film.film import Film
    f = Film(capi.Settings.default(width_m=W * 1e-3, height_m=H * 1e-3), W, H, capi.CF_PREC_FP32)
    rng = np.random.default_rng(3)
    x, y = np.meshgrid(np.arange(W), np.arange(H))
    h = np.where(x >= 16 * PAINTED, 4e-4 * rng.random((H, W)), 0.0)
    f.set_plane("h", h)
    f.set_plane("m", 2e-5 * rng.random((H, W)))
    f.set_plane("color", np.concatenate([rng.random((H, W, 3)), np.full((H, W, 1), 0.4)], 2))
    method = rng.integers(1, 5, (H, W)) + 0.8 * rng.random((H, W))
    f.set_plane("detail", np.stack([np.where(h > 0, method, 0), 0.3 * (h > 0), 40.0 * (h > 0), h], 2))
    f.set_plane("tile_flags", np.array([int(t % 3 == PAINTED) for t in range(6)]))
    return f


def view(kind):
    c = camera.render_cam(W, H, W * 1e-3, H * 1e-3, 1e-3, yaw=0.6, aspect=VIEW[0] / VIEW[1])
    if kind != "persp":
        c.ortho[0] = 1.0
        c.jitter[0] = 0.5  # a quarter of the picture is off the canvas
    c.jitter[2] = float(kind == "beauty")
    return c


def render(f, cam, w, h):
    import torch
    out = torch.full((h, w, 4), -7.0, device="cuda")
    u8 = torch.zeros((h, w), dtype=torch.int32, device="cuda")
    f.render_lit(cam, w, h, out.data_ptr(), u8.data_ptr())
    torch.cuda.synchronize()
    return out.cpu().numpy(), u8.cpu().numpy()


def test_the_view_mixes_the_ends_in_a_warp():
    """The columns of the orthographic view: far, near and off the canvas, in
    the 16 columns a warp takes (the last 7 lie outside the picture)."""
    x = ((2.0 * (np.arange(VIEW[0]) + 0.5) / VIEW[0] - 1.0 + 0.5) * 0.5 + 0.5) * W
    kinds = {"off" if v > W else "near" if v >= 16 else "far" for v in x}
    assert kinds == {"off", "near", "far"} and VIEW[0] < 16


@pytest.mark.parametrize("kind", ["ortho", "persp", "beauty"])
# times in x and y (odd): few and many pixels, the last two in the tall blocks
@pytest.mark.parametrize("tx,ty", [(3, 3), (1, 1523), (39, 39)])
def test_pixels_do_not_depend_on_their_warp(kind, tx, ty):
    f = film()
    small, b = render(f, view(kind), *VIEW)
    large, bl = render(f, view(kind), VIEW[0] * tx, VIEW[1] * ty)
    assert np.isfinite(large).all() and (large[..., 3] == 1.0).all()
    assert np.array_equal(large[ty // 2::ty, tx // 2::tx], small)
    assert np.array_equal(bl[ty // 2::ty, tx // 2::tx], b)
    assert len(np.unique(small.reshape(-1, 4), axis=0)) > 20
    f.close()
