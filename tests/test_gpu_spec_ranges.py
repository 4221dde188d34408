"""Specular resampling (per-pass entries) against the oracle with reservoirs outside the
range of its branch-free arithmetic: hits at the surface, zero, tiny, huge and infinite
target functions and weights, zero and huge M, infinite radiance. Pixels that meet such a
value take the IEEE operations; every output must still equal the oracle's bits."""
import ctypes as C

import numpy as np
import pytest

import violet_gb300 as vg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def vp(t):
    return C.c_void_p(t.data_ptr())


def reservoirs(w, h, kind):
    """Frame 2 of a scene, its params and the resident specular reservoir with a share of
    its values replaced."""
    n = w * h
    P = vg.params_reference()
    scene = vg.Scene(7, w, h, disocclusion_frac=0.05)
    ov = po.OracleView(w, h, P)
    prev = None
    for f in range(3):
        if f == 2:
            prev = cur
        cur = scene.generate_host(f)
        ov.run(scene.frame_params(f), f, cur)
    fp = scene.frame_params(2)
    rsv = ov.buffer("spec_reservoir").view(np.uint32).copy().reshape(n, 2)
    hit = ov.buffer("spec_hit_pos").view(np.float32).copy().reshape(n, 4)
    rad = ov.buffer("spec_radiance").view(np.uint32).copy()
    ov.close()
    rng = np.random.default_rng(n)
    share = {"none": 0.0, "few": 0.02, "many": 0.5}[kind]

    def at():
        return rng.random(n) < share / 8

    values = np.array([0.0, 1e-38, 1e-25, 1e25, 3e38, np.inf], np.float32)
    rsv[at(), 0] = 0
    rsv[at(), 0] = 0xFFFFFFFF
    m = at()
    rsv[m, 1] = rng.choice(values, m.sum()).view(np.uint32)
    m = at()
    hit[m, 3] = rng.choice(values, m.sum())
    hit[at(), :3] = 1e-20
    hit[at(), :3] = 1e20
    rad[at()] = 0
    rad[at()] = 31 << 6
    rsv, hit = np.ascontiguousarray(rsv.reshape(-1)), np.ascontiguousarray(hit.reshape(-1))
    return P, fp, cur, prev, rsv, hit, rad


def same_bits(name, x, y, dt):
    if name == "reservoir":  # {M, W}: W is a float
        n = x.nbytes // 8
        np.testing.assert_array_equal(x.view(np.uint32).reshape(n, 2)[:, 0], y.view(np.uint32).reshape(n, 2)[:, 0])
        x, y = (np.ascontiguousarray(v.view(np.float32).reshape(n, 2)[:, 1]).view(np.uint8) for v in (x, y))
        dt = np.float32
    same = x.view(dt).view("u%d" % np.dtype(dt).itemsize) == y.view(dt).view("u%d" % np.dtype(dt).itemsize)
    if np.dtype(dt).kind == "f":
        same |= np.isnan(x.view(dt)) & np.isnan(y.view(dt))
    assert same.all(), "%s: %d differ" % (name, (~same).sum())


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()


KINDS = pytest.mark.parametrize("kind", ["none", "few", "many"])
SIZES = pytest.mark.parametrize("w,h", [(33, 17), (128, 48)])


@KINDS
@SIZES
def test_spec_spatial_special_reservoirs(w, h, kind):
    import torch

    n = w * h
    P, fp, cur, _, rsv, hit, rad = reservoirs(w, h, kind)
    want = [np.zeros(k * n, np.uint8) for k in (4, 2, 8, 16, 4)]
    got = [torch.zeros(k * n, dtype=torch.uint8, device="cuda") for k in (4, 2, 8, 16, 4)]
    src = (cur["gbuffer"], cur["depth"], rsv, hit, rad)
    keep = [dev(a) for a in src]
    po.lib().vlto_ind_spec_spatial_resample(C.byref(fp), w, h, C.byref(P), *[po.ptr(a) for a in src],
                                            *[po.ptr(a) for a in want], 77)
    assert vg.lib().vlt_ind_spec_spatial_resample(C.byref(fp), w, h, C.byref(P), *[vp(t) for t in keep],
                                                  *[vp(t) for t in got], 77, None) == 0
    torch.cuda.synchronize()
    for name, a, b, dt in zip(("lighting", "ray length", "reservoir", "hit position", "radiance"), got, want,
                              (np.uint32, np.float16, np.uint32, np.float32, np.uint32)):
        same_bits(name, a.cpu().numpy(), b, dt)


@KINDS
@SIZES
def test_spec_temporal_special_reservoirs(w, h, kind):
    import torch

    n = w * h
    P, fp, cur, prev, rsv, hit, rad = reservoirs(w, h, kind)
    new_hit, new_rad = cur["spec_hit_pos"].copy().reshape(n, 4), cur["spec_hit_radiance"].copy()
    rng = np.random.default_rng(n + 1)
    share = {"none": 0.0, "few": 0.01, "many": 0.2}[kind]
    new_rad[rng.random(n) < share] = 0
    new_hit[rng.random(n) < share, :3] = 1e-20
    new_hit[rng.random(n) < share, :3] = 1e20
    new_hit = np.ascontiguousarray(new_hit.reshape(-1))
    src = (prev["depth"], prev["gbuffer"], cur["depth"], cur["gbuffer"], rsv, hit, rad, new_hit, new_rad)
    keep = [dev(a) for a in src]
    want = [np.zeros(k * n, np.uint8) for k in (8, 16, 4)]
    got = [torch.zeros(k * n, dtype=torch.uint8, device="cuda") for k in (8, 16, 4)]
    po.lib().vlto_ind_spec_temporal_resample(C.byref(fp), w, h, C.byref(P), *[po.ptr(a) for a in src],
                                             *[po.ptr(a) for a in want], 31, 1)
    assert vg.lib().vlt_ind_spec_temporal_resample(C.byref(fp), w, h, C.byref(P), *[vp(t) for t in keep],
                                                   *[vp(t) for t in got], 31, 1, None) == 0
    torch.cuda.synchronize()
    for name, a, b, dt in zip(("reservoir", "hit position", "radiance"), got, want,
                              (np.uint32, np.float32, np.uint32)):
        same_bits(name, a.cpu().numpy(), b, dt)
