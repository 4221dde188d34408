"""Specular resampling over hits as far away as a renderer may put them (misses on a sky
sphere): squared distances beyond 2^60, which stay within the branch-free arithmetic, and
beyond binary32, which leave it. Against the oracle, bit for bit: the per-pass entries of the
reference form, and frames of the float forms."""
import ctypes as C

import numpy as np
import pytest

import violet_gb300 as vg
from oracle import pyoracle as po
from tests.helpers import d2h, dev_zeros, first_float_mismatch, upload
from tests.test_gpu_spec_ranges import dev, reservoirs, same_bits, vp

pytestmark = pytest.mark.gpu

SCALES = pytest.mark.parametrize("scale", [1e9, 1e12, 1e18, 3e19])


def far(hit, n, share, scale):
    """A share of the hits (n records of four floats) `scale` times as far."""
    h = hit.reshape(n, 4).copy()
    at = np.random.default_rng(n).random(n) < share
    h[at, :3] *= np.float32(scale)
    return np.ascontiguousarray(h.reshape(-1))


@SCALES
@pytest.mark.parametrize("share", [0.02, 1.0])
def test_spec_passes_far_hits(share, scale):
    import torch

    w, h = 128, 48
    n = w * h
    P, fp, cur, prev, rsv, hit, rad = reservoirs(w, h, "none")
    hit = far(hit, n, share, scale)
    new_hit = far(cur["spec_hit_pos"], n, share, scale)
    calls = {
        "vlt_ind_spec_spatial_resample": ((cur["gbuffer"], cur["depth"], rsv, hit, rad), (4, 2, 8, 16, 4), (77,),
                                          (("lighting", np.uint32), ("ray length", np.float16),
                                           ("reservoir", np.uint32), ("hit", np.float32), ("radiance", np.uint32))),
        "vlt_ind_spec_temporal_resample": ((prev["depth"], prev["gbuffer"], cur["depth"], cur["gbuffer"], rsv, hit,
                                            rad, new_hit, cur["spec_hit_radiance"]), (8, 16, 4), (31, 1),
                                           (("reservoir", np.uint32), ("hit", np.float32), ("radiance", np.uint32))),
    }
    for name, (src, sizes, tail, outs) in calls.items():
        want = [np.zeros(k * n, np.uint8) for k in sizes]
        got = [torch.zeros(k * n, dtype=torch.uint8, device="cuda") for k in sizes]
        keep = [dev(a) for a in src]
        getattr(po.lib(), name.replace("vlt_", "vlto_"))(C.byref(fp), w, h, C.byref(P), *[po.ptr(a) for a in src],
                                                         *[po.ptr(a) for a in want], *tail)
        assert getattr(vg.lib(), name)(C.byref(fp), w, h, C.byref(P), *[vp(t) for t in keep], *[vp(t) for t in got],
                                       *tail, None) == 0
        torch.cuda.synchronize()
        for (what, dt), a, b in zip(outs, got, want):
            same_bits("%s %s" % (name, what) if what != "reservoir" else what, a.cpu().numpy(), b, dt)


@pytest.mark.parametrize("scale", [1e12, 3e19])
@pytest.mark.parametrize("form", ["f32", "f16"])
def test_float_frames_far_hits(form, scale):
    import torch

    w, h = 96, 64
    n, px = w * h, {"f32": 16, "f16": 8}[form]
    ctx = vg.Context(0)
    params = vg.params_reference()
    scene = vg.Scene(31, w, h, disocclusion_frac=0.02)
    view, oview = vg.View(ctx, w, h, form, params), po.OracleView(w, h, params, form)
    try:
        for f in range(4):
            host = scene.generate_host(f)
            host["spec_hit_pos"] = far(host["spec_hit_pos"], n, 0.1, scale)
            fp = scene.frame_params(f)
            out_dev = {k: dev_zeros(px * n) for k in ("diffuse", "specular")}
            out_host = {k: np.zeros(px * n, np.uint8) for k in ("diffuse", "specular")}
            view.run(fp, f, upload(host), out_dev)
            oview.run(fp, f, host, out_host)
            torch.cuda.synchronize()
            for name, words in (("spec_hit_pos", 4), ("spec_reservoir", 2), ("spec_radiance", 1)):
                ptr, nb = view.buffer(name)
                msg = first_float_mismatch(d2h(ptr, nb, np.uint32), oview.buffer(name, np.uint8).view(np.uint32), w,
                                           words)
                assert msg is None, "frame %d %s: %s" % (f, name, msg)
    finally:
        view.close()
        oview.close()
        ctx.close()
