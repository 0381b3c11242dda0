"""Splatted images at the edges of the splat loops, bit for bit: sprites of under one pixel, of
a few and of more pixels than the image, image widths off the lanes' stride, images that are
only 4-byte aligned, sets of 0, 1 and 1000 particles; the whole fluid view against its stages
(whose own results other tests hold against the CPU restatement)."""
import ctypes as C

import numpy as np
import pytest
import torch

from snowsimulation_b200 import _native, render, scene
from snowsimulation_b200.export import SNOW_RGB

pytestmark = pytest.mark.gpu

CASES = {   # width, height, point size, filter radius, water and snow particles drawn
    "small sprites": (97, 61, 0.3, 10.0, 1000, 1000),
    "7 px": (131, 70, 2.5, 10.0, 1000, 1000),
    "whole image": (33, 17, 90.0, 3.5, 40, 40),
    "one of each": (64, 48, 8.0, 0.0, 1, 1),
    "no water": (40, 30, 4.0, 10.0, 0, 1000),
    "no snow": (40, 30, 4.0, 256.0, 1000, 0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_splats(cuda, name):
    from oracle import render_oracle
    from snowsimulation_b200.world import Simulation
    W, H, ps, radius, ns, nd = CASES[name]
    sim = Simulation(scene.scene_drop((6, 6, 6), (9, 9, 9), seed=2, snow_jitter=0.002, water_jitter=0.002, name=name)).setup()
    ns, nd = min(ns, sim.n_sph), min(nd, sim.n_dem)
    cam = render.camera(eye=(0.2, 0.25, 0.5), center=(0.0, 0.1, 0.0), width=W, height=H, point_size=ps)
    ss = render.ssfr_params(sphere_radius=0.01, filter_radius=radius)
    lib, a = sim.lib, C.addressof
    pc = render.colour(SNOW_RGB)
    host = sim.to_host()

    def alloc(skew, *shape):   # skew: floats past the 16-byte boundary
        t = torch.full((int(np.prod(shape)) + 8,), 7.0, dtype=torch.float32, device=sim.device)
        return t[skew:skew + int(np.prod(shape))].view(*shape)

    outs = []
    for skew in (0, 1):
        rgba, out = alloc(skew, H, W, 4), alloc(skew, H, W, 4)
        zb = torch.empty((H, W), dtype=torch.int64, device=sim.device)
        thick = torch.empty_like(zb)
        sdep, fdep, tmp, sm = (alloc(0, H, W) for _ in range(4))
        dem, sph = C.byref(sim._s[1]), C.byref(sim._s[0])
        for rc in (lib.snowb_render_clear_colour(a(cam), a(ss.clear_color), rgba.data_ptr(), zb.data_ptr()),
                   lib.snowb_render_points(dem, nd, a(cam), a(pc), 0, rgba.data_ptr(), zb.data_ptr()),
                   lib.snowb_ssfr_clear(a(cam), sdep.data_ptr(), thick.data_ptr()),
                   lib.snowb_ssfr_clear(a(cam), fdep.data_ptr(), None),
                   lib.snowb_ssfr_sphere_depth(dem, nd, a(cam), a(ss), sdep.data_ptr()),
                   lib.snowb_ssfr_sphere_depth(sph, ns, a(cam), a(ss), fdep.data_ptr()),
                   lib.snowb_ssfr_smooth(a(cam), a(ss), fdep.data_ptr(), tmp.data_ptr(), sm.data_ptr()),
                   lib.snowb_ssfr_thickness(sph, ns, a(cam), thick.data_ptr()),
                   lib.snowb_ssfr_compose(a(cam), a(ss), sm.data_ptr(), thick.data_ptr(), rgba.data_ptr(),
                                          sdep.data_ptr(), out.data_ptr())):
            _native.check(rc)
        view = alloc(skew, H, W, 4)
        nbytes = C.c_uint64(0)
        _native.check(lib.snowb_ssfr_workspace_bytes(a(cam), C.byref(nbytes)))
        ws = torch.empty(int(nbytes.value) // 4, dtype=torch.float32, device=sim.device)
        _native.check(lib.snowb_render_fluid(sph, ns, dem, nd, a(cam), a(pc), a(ss), ws.data_ptr(), view.data_ptr()))
        outs.append([t.cpu().numpy() for t in (rgba, out, view)])
    for x, y in zip(*outs):
        assert np.array_equal(x, y, equal_nan=True)
    rgba, out, view = outs[0]
    assert np.array_equal(view, out, equal_nan=True)
    if nd:
        ref = render_oracle.render(render.camera_dict(cam), [(host.dem["positions"][:nd], None, {"rgb": SNOW_RGB})])
        hit = ref[..., 3] > 0
        assert np.array_equal(rgba[hit], ref[hit])
        assert (rgba[~hit] == np.array(list(ss.clear_color), np.float32)).all()
