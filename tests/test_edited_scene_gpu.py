"""GPU: a scene edited in place, behind unchanged pointers and counts, is rendered as edited: the film
equals the one of a fresh upload of the same content. Each edit changes one record or a few that a
strided sample of a large table would miss, and of every table that the device keeps a copy of. A record
that the edit makes invalid is refused although the device holds a valid copy of the scene."""

import ctypes as C

import numpy as np
import pytest

from prgpu import abi, hostscene, render, scenes, spectra

pytestmark = pytest.mark.gpu

W = H = 32


def _film(h, ext=None, spp=4):
    return render.render_ex(h, W, H, spp, seed=3, max_depth=5, ext=ext)


def _other_scene():
    """Takes the scene's place on the device."""
    _film(hostscene.build_box_scene(scenes.box_scene(seed=99, width=W, height=H, subdiv=0)), spp=1)


def _box():
    return hostscene.build_box_scene(scenes.box_scene(seed=1, width=W, height=H, subdiv=3)), None


def _outdoor():
    return hostscene.build_large_scene(W, H, terrain_res=80, cloud_res=64, spheres=3, sky_resolution=512)


def _wall_prims(h):
    """Triangles of the four walls that the camera sees; the scene has 44,814."""
    return [k for k in range(12) if k % 10]


def _edit_material(h, ext):
    h.prim_array["material"][_wall_prims(h)] = 2


def _edit_normals(h, ext):
    k = np.flatnonzero(np.abs(h.prim_array["n0"]).sum(1) > 0)
    k = k[(k % 10 != 0)]
    for n in ("n0", "n1", "n2"):
        h.prim_array[n][k] = h.prim_array[n][k][:, [1, 2, 0]]


def _edit_medium_side(h, ext):
    h.prim_array["mediumInside"][_wall_prims(h)] = -1  # unchanged values: nothing may change ...
    h.prim_array["light"][13] = -1                     # ... but one half of the ceiling light goes dark


def _edit_node(h, ext):
    """A subtree's box collapsed to a point: what it holds is no longer seen."""
    k = next(i for i in range(3, len(h.nodes)) if h.nodes[i]["nPrims"] == 0 and i % 2 and
             h.nodes[i]["offset"] - i > 2000)
    h.nodes["bmin"][k] = h.nodes["bmax"][k] = 50.0


def _edit_order(h, ext):
    """Two leaves of equal size trade their primitives (and no longer hold what their boxes say)."""
    big = [int(h.nodes[i]["offset"]) for i in range(len(h.nodes)) if h.nodes[i]["nPrims"] > 0]
    step = len(h.order) // 4096
    s = [o for o in big if o % step and (h.order[o] < 12)]
    t = [o for o in big if o % step and (h.order[o] >= 200)]
    for a, b in zip(s, t):
        h.order[a], h.order[b] = h.order[b], h.order[a]


def _edit_cloud(h, ext):
    d = ext._keep[-1]  # the density, (64, 64, 64)
    flat = d.reshape(-1)
    flat[1::2] = flat[1::2][::-1].copy()


def _edit_sky(h, ext):
    texels = ext._keep[-4]
    assert texels.shape == (256, 512, 4)
    texels.reshape(-1, 4)[1::2, 3] *= 2.0


def _textured():
    h = hostscene.build_box_scene(scenes.box_scene(seed=1, width=W, height=H, subdiv=0))
    rng = np.random.default_rng(5)
    img = rng.random((400, 400, 3)).astype(np.float32)
    table = np.zeros(64 + 3 * 64 ** 3 * 3, np.float32)
    table[:64] = np.linspace(0, 1, 64)
    table[64:] = rng.uniform(-1, 1, len(table) - 64) * np.tile([1e-6, 1e-3, 1.0], 3 * 64 ** 3)
    mt = [(0, -1, 1.0, False)] + [(-1, -1, 1.0, False)] * (len(h.mat_array) - 1)
    ext = render.make_ext(textures=[render.image_texture(img)], material_textures=mt, rgb_to_spectrum=table)
    ext._arrays = (img, table)
    return h, ext


def _edit_texture(h, ext):
    ext._arrays[0].reshape(-1, 3)[1::2] = 0.02


def _edit_rgb_table(h, ext):
    ext._arrays[1][64:].reshape(-1, 3)[:, 2] -= 2.0


def _sheen():
    h = hostscene.build_box_scene(scenes.box_scene(seed=1, width=W, height=H, subdiv=0))
    h.mat_array["sheenWeight"][0] = 1.0
    h.mat_array["sheenRoughness"][0] = 0.5
    h.mat_array["sheenColor"][0] = 0
    h.sheen = np.zeros(512, np.float32)
    abi.gpu_lib().prgpu_sheen_albedo_table(abi.ptr(h.sheen))
    h.desc().sheenAlbedo = h.sheen.ctypes.data
    return h, None


def _edit_sheen_table(h, ext):
    h.sheen *= 0.3


def _outdoor_cie():
    h, ext = _outdoor()
    h.cie = np.ascontiguousarray(spectra.cie_xyz(spectra.LAMBDA), np.float32)
    h.desc().cie = h.cie.ctypes.data
    return h, ext


def _edit_cie(h, ext):
    h.cie[1, 40:] = 0.0  # other sampling probabilities of the sky's texels


EDITS = {
    "material": (_box, _edit_material), "normals": (_box, _edit_normals), "light": (_box, _edit_medium_side),
    "node": (_box, _edit_node), "order": (_box, _edit_order), "cloud": (_outdoor, _edit_cloud),
    "sky": (_outdoor, _edit_sky), "texture": (_textured, _edit_texture), "rgb_table": (_textured, _edit_rgb_table),
    "sheen_table": (_sheen, _edit_sheen_table), "cie": (_outdoor_cie, _edit_cie),
}


@pytest.mark.parametrize("name", sorted(EDITS))
def test_an_edit_in_place_shows(gpu, name):
    make, edit = EDITS[name]
    h, ext = make()
    before = _film(h, ext)
    np.testing.assert_array_equal(_film(h, ext), before)
    edit(h, ext)
    after = _film(h, ext)
    _other_scene()
    fresh = _film(h, ext)
    assert (fresh != before).any()
    np.testing.assert_array_equal(after, fresh)


def test_a_batch_sees_the_edit(gpu):
    h, _ = _box()

    def batch():
        film = np.zeros((H, W, 3))
        render.render_batch([(h, None, dict(spp=4, seed=3, max_depth=5), film)], config=render.batch_config(1 << 14, 256))
        return film

    before = batch()
    _edit_material(h, None)
    after = batch()
    assert (after != before).any()
    np.testing.assert_array_equal(after, _film(h))


def test_a_guide_buffer_sees_the_edit(gpu):
    h, _ = _box()
    before = render.render_aov(h, W, H, render.AOV_NORMAL, 2)
    _edit_normals(h, None)
    after = render.render_aov(h, W, H, render.AOV_NORMAL, 2)
    _other_scene()
    fresh = render.render_aov(h, W, H, render.AOV_NORMAL, 2)
    assert (fresh != before).any()
    np.testing.assert_array_equal(after, fresh)


@pytest.mark.parametrize("field,value", [("material", 1 << 20), ("material", -1), ("light", 77), ("mediumInside", 3),
                                         ("mediumOutside", -2), ("type", 9)])
def test_an_edit_that_breaks_the_scene_is_refused(gpu, field, value):
    h, _ = _box()
    good = _film(h)
    k = 33333
    was = h.prim_array[field][k].copy()
    h.prim_array[field][k] = value
    with pytest.raises(abi.PrgpuError):
        _film(h)
    h.prim_array[field][k] = was
    np.testing.assert_array_equal(_film(h), good)
