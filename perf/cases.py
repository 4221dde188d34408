"""Performance cases of the lighting back end.

Whole frames go through the view API (`View.run_bound`, `View.run_sequence`,
`View.trace` + `View.run`, `Batch.run`); blocks of passes go through the per-pass C
entry points, which stand in for the reference renderer's render-graph nodes. Frames
come from the seeded synthetic scene: a ring of four scene frames walked forth and back
by a moving, jittered camera, with 2 % disocclusion, fireflies in the candidates and a
history that the view has built up over the frames before.

Kinds (`kind` of a case) and what they stand for:
  frame     one frame of one view, device-resident inputs and outputs
  sequence  a few frames of one view handed over in one call
  traced    a frame in traced mode: ray generation, the scene's tracer in the caller's
            place, shading of the hits with both validations, the rest of the frame
  batch     one frame of a dozen small views of uneven size as one batched step
  diffuse   the diffuse block: AO generation and filter, temporal and spatial resampling
  specular  the specular block: temporal and spatial resampling
  denoise   the denoiser's front: temporal filter, disocclusion fix, fast-history clamp,
            spatial fallback
  atrous    the denoiser's a-trous filter, three iterations
  hashgrid  the radiance cache: decay, query selection, compaction, update, emission
"""
import ctypes
import math

import numpy as np
import torch

import violet_gb300 as vg

RING = (0, 1, 2, 3, 2, 1)  # scene frames of a walk forth and back
WARM = 8                   # frames a view has run before it is timed
FORM_LIGHT = {"ref": (torch.int32, 1), "f32": (torch.float32, 4), "f16": (torch.float16, 4)}


# ------------------------------------------------------------------ cases

def listed():
    return [
        # The smallest configured workload: launches and latency count.
        {"name": "frame f32 320x180", "kind": "frame", "form": "f32", "knobs": "plain0", "w": 320, "h": 180,
         "post": 0, "fast": 0},
        # What the reference renderer runs by default, with final lighting and TAA.
        {"name": "frame ref 1280x720 post", "kind": "frame", "form": "ref", "knobs": "reference", "w": 1280,
         "h": 720, "post": 2, "fast": 0},
        # The headline workload.
        {"name": "frame f32 1920x1080", "kind": "frame", "form": "f32", "knobs": "plain1", "w": 1920, "h": 1080,
         "post": 0, "fast": 0},
        # The precision form at its configured size: the largest.
        {"name": "frame f16 3840x2160", "kind": "frame", "form": "f16", "knobs": "plain1", "w": 3840, "h": 2160,
         "post": 0, "fast": 0},
        # Frames that a caller already holds, run as one pipelined call, ragged width.
        {"name": "sequence f32 853x479", "kind": "sequence", "form": "f32", "knobs": "plain1", "w": 853, "h": 479,
         "n": 4},
        # Traced mode with both validations, odd size.
        {"name": "traced ref 961x541", "kind": "traced", "form": "ref", "knobs": "reference", "w": 961, "h": 541},
        # Many small views in one step, as a server runs them.
        {"name": "batch f16 12 views", "kind": "batch", "form": "f16", "knobs": "plain1", "views": 12, "w_max": 640},
        # The drop-in passes of the reference renderer, block by block.
        {"name": "diffuse 1280x720", "kind": "diffuse", "w": 1280, "h": 720, "knobs": "reference"},
        {"name": "specular 1920x1080", "kind": "specular", "w": 1920, "h": 1080, "knobs": "reference"},
        {"name": "denoise 1365x767", "kind": "denoise", "w": 1365, "h": 767, "fast": 1},
        {"name": "atrous 1920x1080", "kind": "atrous", "w": 1920, "h": 1080, "iterations": 3},
        # One query per pixel of a 720p frame against 2^22 cells.
        {"name": "hash grid 1280x720", "kind": "hashgrid", "w": 1280, "h": 720, "log2_buckets": 18},
    ]


def draw(rng):
    def size(lo, hi):
        w = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        h = max(1, int(round(w / rng.choice((16 / 9, 4 / 3, 21 / 9, 1.0)))) + rng.randint(-2, 2))
        return w, h

    kind = rng.choice(("frame", "frame", "frame", "sequence", "traced", "batch", "diffuse", "specular", "denoise",
                       "atrous", "hashgrid"))
    form = rng.choice(("ref", "f32", "f16"))
    knobs = rng.choice(("reference", "plain0", "plain1"))
    if kind == "frame":
        w, h = size(160, 2560)
        return {"kind": kind, "form": form, "knobs": knobs, "w": w, "h": h, "post": rng.choice((0, 0, 2)),
                "fast": rng.choice((0, 0, 1))}
    if kind == "sequence":
        w, h = size(160, 1280)
        return {"kind": kind, "form": form, "knobs": knobs, "w": w, "h": h, "n": rng.randint(2, 6)}
    if kind == "traced":
        w, h = size(160, 1920)
        return {"kind": kind, "form": form, "knobs": knobs, "w": w, "h": h}
    if kind == "batch":
        return {"kind": kind, "form": form, "knobs": knobs, "views": rng.randint(2, 24),
                "w_max": rng.randint(280, 900)}
    w, h = size(160, 2560)
    if kind in ("diffuse", "specular"):
        return {"kind": kind, "w": w, "h": h, "knobs": knobs}
    if kind == "denoise":
        return {"kind": kind, "w": w, "h": h, "fast": rng.choice((0, 1))}
    if kind == "atrous":
        return {"kind": kind, "w": w, "h": h, "iterations": rng.randint(1, 5)}
    return {"kind": kind, "w": w, "h": h, "log2_buckets": rng.randint(14, 18)}


# ---------------------------------------------------------------- helpers

def _knobs(case):
    p = {"reference": vg.params_reference, "plain0": lambda: vg.params_plain(0),
         "plain1": lambda: vg.params_plain(1)}[case["knobs"]]()
    p.post = case.get("post", 0)
    p.fast_history_clamp = case.get("fast", 0)
    return p


def _empty(n, dtype):
    return torch.empty(n, dtype=dtype, device="cuda")


def _bytes(n):
    return torch.zeros(max(int(n), 16), dtype=torch.uint8, device="cuda")


class _Resident:
    """Device memory of a view as a tensor's storage; keeps the view alive."""

    def __init__(self, view, ptr, n, typestr):
        self.view = view
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


_TYPES = {"<i4": 4, "<f4": 4, "<f2": 2, "|u1": 1}


def _resident(state, name, typestr):
    """A buffer of the view's resident state as a tensor (the view swaps its buffers
    between frames, so a tensor per address)."""
    view = state["view"]
    ptr, nbytes = view.buffer(name)
    t = state["tensors"].get((name, ptr))
    if t is None:
        t = torch.as_tensor(_Resident(view, ptr, nbytes // _TYPES[typestr], typestr), device="cuda")
        state["tensors"][(name, ptr)] = t
    return t


def _ring(seed, w, h):
    """The ring of frames: device inputs and the frame parameters of each step, whose
    previous-frame fields are those of the step before it."""
    scene = vg.Scene(seed, w, h, disocclusion_frac=0.02)
    n = w * h
    inputs = {}
    for f in sorted(set(RING)):
        bufs = {k: _empty(n * c * np.dtype(dt).itemsize, torch.uint8) for k, (dt, c) in vg.FRAME_BUFFERS.items()}
        scene.generate_device(f, bufs)
        inputs[f] = bufs
    steps = []
    for i, f in enumerate(RING):
        fp, prev = scene.frame_params(f), scene.frame_params(RING[i - 1])
        fp.prev_view_proj = prev.view_proj
        fp.prev_inv_view_proj = prev.inv_view_proj
        fp.prev_view_pos = prev.view_pos
        fp.jitter[2], fp.jitter[3] = prev.jitter[0], prev.jitter[1]
        steps.append((fp, inputs[f]))
    return scene, steps


def _outputs(form, w, h, params):
    dt, c = FORM_LIGHT[form]
    names = ("diffuse", "specular") + (("color",) if params.post >= 1 else ()) + (("taa",) if params.post >= 2 else ())
    return {k: torch.zeros(w * h * c, dtype=dt, device="cuda") for k in names}


def _view_state(case, seed):
    params = _knobs(case)
    ctx = vg.Context(0)
    w, h, form = case["w"], case["h"], case["form"]
    scene, steps = _ring(seed, w, h)
    out = _outputs(form, w, h, params)
    view = vg.View(ctx, w, h, form, params)
    return {"case": case, "ctx": ctx, "view": view, "scene": scene, "steps": steps, "out": out, "frame": 0,
            "params": params, "tensors": {}}


def _frame_outputs(state):
    res = dict(state["out"])
    form = state["case"]["form"]
    res["diff_reservoir"] = _resident(state, "diff_reservoir", "|u1" if form == "f16" else "<i4")
    res["spec_reservoir"] = _resident(state, "spec_reservoir", "<i4")
    if form == "ref":
        res["history"] = _resident(state, "hist_color", "<i4")
    else:
        res["history"] = _resident(state, "hist_record", "<f4" if form == "f32" else "<f2")
    if state["params"].hg_enable:
        res["cells"] = _resident(state, "hg_storage", "<i4")
    return res


def _vp(t):
    return ctypes.c_void_p(t if isinstance(t, int) else (t.data_ptr() if t is not None else None))


def _call(name, *args):
    st = getattr(vg.lib(), name)(*args)
    if st != 0:
        raise RuntimeError("%s: status %d" % (name, st))


def _owned(view, name, dtype=torch.uint8):
    ptr, nbytes = view.buffer(name)
    return torch.as_tensor(_Resident(view, ptr, nbytes, "|u1"), device="cuda").clone().view(dtype)


def _reference_state(seed, w, h, names, **knobs):
    """Copies of a reference-form view's resident buffers after WARM frames, with the
    parameters and inputs of the frame before and of the frame that comes next."""
    params = vg.params_reference()
    for k, v in knobs.items():
        setattr(params, k, v)
    ctx = vg.Context(0)
    scene, steps = _ring(seed, w, h)
    view = vg.View(ctx, w, h, "ref", params)
    for f in range(WARM):
        fp, bufs = steps[f % len(steps)]
        view.run(fp, f, bufs)
    torch.cuda.synchronize()
    got = {k: _owned(view, k) for k in names}
    torch.cuda.synchronize()
    view.close()
    fp, cur = steps[WARM % len(steps)]
    prev = steps[(WARM - 1) % len(steps)][1]
    return ctx, fp, cur, prev, got


# ---------------------------------------------------------------- prepare

def prepare(case, seed):
    return {"frame": _prepare_frame, "sequence": _prepare_sequence, "traced": _prepare_traced,
            "batch": _prepare_batch, "diffuse": _prepare_diffuse, "specular": _prepare_specular,
            "denoise": _prepare_denoise, "atrous": _prepare_atrous, "hashgrid": _prepare_hashgrid}[case["kind"]](
                case, seed)


def _prepare_frame(case, seed):
    s = _view_state(case, seed)
    s["bound"] = [(vg.FrameBinding(bufs, s["out"]), fp) for fp, bufs in s["steps"]]
    for _ in range(WARM):
        _run_frame(s)
    torch.cuda.synchronize()
    return s


def _prepare_sequence(case, seed):
    s = _view_state(case, seed)
    dt, c = FORM_LIGHT[case["form"]]
    n = case["w"] * case["h"]
    s["outs"] = [{k: torch.zeros(n * c, dtype=dt, device="cuda") for k in ("diffuse", "specular")}
                 for _ in range(case["n"])]
    for _ in range(-(-WARM // case["n"])):
        _run_sequence(s)
    torch.cuda.synchronize()
    return s


def _prepare_traced(case, seed):
    # diffuse and specular validation on, as the reference renderer runs
    params = _knobs(case)
    params.trace = params.diff_validate = params.spec_validate = 1
    ctx = vg.Context(0)
    w, h = case["w"], case["h"]
    n = w * h
    scene, steps = _ring(seed, w, h)
    view = vg.View(ctx, w, h, case["form"], params)
    rays = {"cache": _bytes(max(view.cache_ray_capacity, 1) * 32), "diffuse": _bytes(n * 32),
            "spec_validate": _bytes(n * 32)}
    hits = {k: _bytes(t.numel() * 2) for k, t in rays.items()}
    s = {"case": case, "ctx": ctx, "view": view, "scene": scene, "steps": steps, "rays": rays, "hits": hits,
         "out": _outputs(case["form"], w, h, params), "frame": 0, "params": params, "tensors": {}}
    for _ in range(WARM):
        _run_traced(s)
    torch.cuda.synchronize()
    return s


def _batch_sizes(case):
    """View sizes spread over the logarithm of [256, w_max], aspects in turn."""
    sizes = []
    for k in range(case["views"]):
        u = (k * 0.6180339887498949) % 1.0
        w = int(round(256 * math.exp(u * math.log(case["w_max"] / 256))))
        sizes.append((w, int(round(w / (16 / 9, 4 / 3, 1.0)[k % 3]))))
    return sizes


def _prepare_batch(case, seed):
    ctx = vg.Context(0)
    views, rings, outs = [], [], []
    for k, (w, h) in enumerate(_batch_sizes(case)):
        params = _knobs(case)
        params.hg_log2_buckets = 14
        _, steps = _ring(seed * 64 + k, w, h)
        views.append(vg.View(ctx, w, h, case["form"], params))
        rings.append(steps)
        outs.append(_outputs(case["form"], w, h, params))
    s = {"case": case, "ctx": ctx, "views": views, "rings": rings, "outs": outs, "frame": 0, "batch": vg.Batch(ctx),
         "stream": torch.cuda.Stream()}
    torch.cuda.synchronize()
    for _ in range(WARM):
        _run_batch(s)
    torch.cuda.synchronize()
    return s


def _prepare_diffuse(case, seed):
    w, h = case["w"], case["h"]
    n = w * h
    ctx, fp, cur, prev, got = _reference_state(seed, w, h, ("diff_reservoir", "ao_history"))
    return {"case": case, "ctx": ctx, "fp": fp, "cur": cur, "prev": prev, "got": got, "params": _knobs(case),
            "ao": _empty(2 * n, torch.float16), "ao_filtered": _empty(n, torch.float16),
            "temporal": _empty(4 * n, torch.int32), "reservoir": _empty(4 * n, torch.int32),
            "lighting": _empty(n, torch.int32), "frame": 0}


def _prepare_specular(case, seed):
    w, h = case["w"], case["h"]
    n = w * h
    ctx, fp, cur, prev, got = _reference_state(seed, w, h, ("spec_hit_pos", "spec_reservoir", "spec_radiance"))
    return {"case": case, "ctx": ctx, "fp": fp, "cur": cur, "prev": prev, "got": got, "params": _knobs(case),
            "reservoir": _empty(2 * n, torch.int32), "hit_pos": _empty(4 * n, torch.float32),
            "radiance": _empty(n, torch.int32), "lighting": _empty(n, torch.int32),
            "ray_len": _empty(n, torch.float16), "frame": 0}


def _prepare_denoise(case, seed):
    w, h = case["w"], case["h"]
    n = w * h
    ctx, fp, cur, prev, got = _reference_state(
        seed, w, h, ("raw_diffuse", "raw_specular", "spec_ray_len", "hist_color", "hist_moments", "hist_len"),
        fast_history_clamp=case["fast"])
    s = {"case": case, "ctx": ctx, "fp": fp, "cur": cur, "prev": prev, "got": got, "params": vg.params_reference(),
         "color": _empty(2 * n, torch.int32), "moments": _empty(2 * n, torch.float16),
         "length": _empty(n, torch.uint8), "fast": _empty(2 * n, torch.int32) if case["fast"] else None,
         "fixed": _empty(2 * n, torch.int32), "fixed_moments": _empty(2 * n, torch.float16),
         "filtered": _empty(2 * n, torch.int32), "variance": _empty(2 * n, torch.float16)}
    s["params"].fast_history_clamp = case["fast"]
    return s


def _prepare_atrous(case, seed):
    w, h = case["w"], case["h"]
    n = w * h
    ctx, _, cur, prev, got = _reference_state(seed, w, h, ("hist_color", "hist_moments", "hist_len"))
    frame = prev  # the frame whose history it is
    color, variance = _empty(2 * n, torch.int32), _empty(2 * n, torch.float16)
    _call("vlt_denoise_spatial_fallback", w, h, _vp(frame["depth"]), _vp(frame["gbuffer"]), _vp(got["hist_len"]),
          _vp(got["hist_color"]), _vp(got["hist_moments"]), _vp(color), _vp(variance), None)
    # the variance of a scene whose moments stay within binary16
    variance = torch.nan_to_num(variance, nan=0.0, posinf=4096.0).clamp_(max=4096.0)
    return {"case": case, "ctx": ctx, "cur": frame, "color": color, "variance": variance,
            "ping": [(_empty(2 * n, torch.int32), _empty(2 * n, torch.float16)) for _ in range(2)]}


def _prepare_hashgrid(case, seed):
    w, h, lb = case["w"], case["h"], case["log2_buckets"]
    n, cells = w * h, 16 << case["log2_buckets"]
    ctx = vg.Context(0)
    _, steps = _ring(seed, w, h)
    s = {"case": case, "ctx": ctx, "steps": steps, "frame": 0, "storage": torch.zeros(4 * cells, dtype=torch.int32,
                                                                                    device="cuda"),
         "decay": torch.zeros(cells, dtype=torch.uint8, device="cuda"),
         "selection": torch.zeros(cells, dtype=torch.int32, device="cuda"),
         "queries": torch.zeros(8 * n, dtype=torch.int32, device="cuda"),
         "count": torch.zeros(1, dtype=torch.int32, device="cuda"),
         "index": _empty(min(n, cells), torch.int32), "addr": _empty(min(n, cells), torch.int32),
         "compact": torch.zeros(1, dtype=torch.int32, device="cuda"),
         "scratch": _bytes(vg.lib().vlt_hg_select_scratch_bytes(lb, n))}
    for _ in range(WARM):
        _run_hashgrid(s)
    torch.cuda.synchronize()
    return s


# -------------------------------------------------------------------- run

def run(state):
    return _RUN[state["case"]["kind"]](state)


def _run_frame(s):
    f = s["frame"]
    s["frame"] = f + 1
    binding, fp = s["bound"][f % len(s["bound"])]
    s["view"].run_bound(binding, fp, f)
    return _frame_outputs(s)


def _run_sequence(s):
    f, n, steps = s["frame"], s["case"]["n"], s["steps"]
    s["frame"] = f + n
    at = [steps[(f + k) % len(steps)] for k in range(n)]
    seq = vg.FrameSequence([fp for fp, _ in at], list(range(f, f + n)), [b for _, b in at], s["outs"])
    s["view"].run_sequence(seq)
    res = _frame_outputs(dict(s, out={}))
    res["frames"] = s["outs"]
    return res


def _run_traced(s):
    f = s["frame"]
    s["frame"] = f + 1
    fp, bufs = s["steps"][f % len(s["steps"])]
    counts = s["view"].trace(fp, f, bufs, s["rays"])
    inp = dict(bufs)
    for k, name in (("cache", "cache_hits"), ("diffuse", "diffuse_hits"), ("spec_validate", "spec_validate_hits")):
        if counts[k]:
            s["scene"].trace_device(fp, s["rays"][k], counts[k], s["hits"][k])
            inp[name] = s["hits"][k]
    s["view"].run(fp, f, inp, s["out"])
    return _frame_outputs(s)


def _run_batch(s):
    f = s["frame"]
    s["frame"] = f + 1
    at = [r[f % len(r)] for r in s["rings"]]
    s["batch"].run(s["views"], [fp for fp, _ in at], [f] * len(at), [b for _, b in at], s["outs"],
                   s["stream"].cuda_stream)
    return s["outs"]


def _run_diffuse(s):
    w, h, cur, prev, got = s["case"]["w"], s["case"]["h"], s["cur"], s["prev"], s["got"]
    fp, params = ctypes.byref(s["fp"]), ctypes.byref(s["params"])
    f = s["frame"]
    s["frame"] = f + 1
    _call("vlt_ao_gen", fp, w, h, _vp(cur["diff_hit_pos_normal"]), _vp(cur["depth"]), _vp(got["ao_history"]),
          _vp(s["ao"]), 1, 1, ctypes.c_float(s["params"].ao_radius), None)
    _call("vlt_ao_filter", w, h, _vp(cur["depth"]), _vp(s["ao"]), _vp(s["ao_filtered"]), None)
    _call("vlt_ind_diff_temporal_resample", fp, w, h, params, _vp(prev["depth"]), _vp(cur["depth"]),
          _vp(cur["diff_hit_pos_normal"]), _vp(cur["diff_hit_radiance"]), _vp(cur["diff_source_pdf"]),
          _vp(got["diff_reservoir"]), _vp(s["temporal"]), 2 * f + 17, 1, 1, None)
    _call("vlt_ind_diff_spatial_resample", fp, w, h, params, _vp(cur["gbuffer"]), _vp(cur["depth"]),
          _vp(s["ao_filtered"]), _vp(s["temporal"]), _vp(s["reservoir"]), _vp(s["lighting"]), 2 * f + 18, None)
    return {k: s[k] for k in ("ao", "ao_filtered", "reservoir", "lighting")}


def _run_specular(s):
    w, h, cur, prev, got = s["case"]["w"], s["case"]["h"], s["cur"], s["prev"], s["got"]
    fp, params = ctypes.byref(s["fp"]), ctypes.byref(s["params"])
    f = s["frame"]
    s["frame"] = f + 1
    _call("vlt_ind_spec_temporal_resample", fp, w, h, params, _vp(prev["depth"]), _vp(prev["gbuffer"]),
          _vp(cur["depth"]), _vp(cur["gbuffer"]), _vp(got["spec_reservoir"]), _vp(got["spec_hit_pos"]),
          _vp(got["spec_radiance"]), _vp(cur["spec_hit_pos"]), _vp(cur["spec_hit_radiance"]), _vp(s["reservoir"]),
          _vp(s["hit_pos"]), _vp(s["radiance"]), 2 * f + 21, 1, None)
    _call("vlt_ind_spec_spatial_resample", fp, w, h, params, _vp(cur["gbuffer"]), _vp(cur["depth"]),
          _vp(s["reservoir"]), _vp(s["hit_pos"]), _vp(s["radiance"]), _vp(s["lighting"]), _vp(s["ray_len"]), None,
          None, None, 2 * f + 22, None)
    return {k: s[k] for k in ("reservoir", "hit_pos", "radiance", "lighting", "ray_len")}


def _run_denoise(s):
    w, h, cur, prev, got = s["case"]["w"], s["case"]["h"], s["cur"], s["prev"], s["got"]
    fast = s["case"]["fast"]
    depth, gbuf = _vp(cur["depth"]), _vp(cur["gbuffer"])
    # the colour history stands in for a fast history
    _call("vlt_denoise_temporal", ctypes.byref(s["fp"]), w, h, ctypes.byref(s["params"]), depth, gbuf,
          _vp(got["raw_diffuse"]), _vp(got["raw_specular"]), _vp(got["spec_ray_len"]), _vp(prev["depth"]),
          _vp(prev["gbuffer"]), _vp(got["hist_color"]), _vp(got["hist_moments"]), _vp(got["hist_len"]),
          _vp(got["hist_color"] if fast else None), _vp(s["color"]), _vp(s["moments"]), _vp(s["length"]),
          _vp(s["fast"]), 1, fast, None)
    _call("vlt_denoise_disocclusion_fix", w, h, depth, gbuf, _vp(s["length"]), _vp(s["color"]), _vp(s["moments"]),
          _vp(s["fixed"]), _vp(s["fixed_moments"]), None)
    if fast:
        _call("vlt_denoise_fast_history_clamp", w, h, _vp(s["fast"]), _vp(s["fixed"]), None)
    _call("vlt_denoise_spatial_fallback", w, h, depth, gbuf, _vp(s["length"]), _vp(s["fixed"]),
          _vp(s["fixed_moments"]), _vp(s["filtered"]), _vp(s["variance"]), None)
    return {k: s[k] for k in ("length", "fast", "fixed", "fixed_moments", "filtered", "variance")}


def _run_atrous(s):
    w, h, cur = s["case"]["w"], s["case"]["h"], s["cur"]
    src = (s["color"], s["variance"])
    for k in range(s["case"]["iterations"]):
        dst = s["ping"][k & 1]
        _call("vlt_denoise_atrous", w, h, _vp(cur["depth"]), _vp(cur["gbuffer"]), _vp(src[0]), _vp(src[1]),
              _vp(dst[0]), _vp(dst[1]), 1 << k, None)
        src = dst
    return {"color": src[0], "variance": src[1]}


def _run_hashgrid(s):
    case = s["case"]
    w, h, lb = case["w"], case["h"], case["log2_buckets"]
    n, f = w * h, s["frame"]
    s["frame"] = f + 1
    fp, bufs = s["steps"][f % len(s["steps"])]
    storage, decay, sel, queries, count = (_vp(s[k]) for k in ("storage", "decay", "selection", "queries", "count"))
    _call("vlt_hg_decay", lb, decay, storage, None)
    s["selection"].zero_()
    s["compact"].zero_()
    _call("vlt_hg_query_select", lb, n, queries, count, storage, sel, (f * 2654435761 + 97) & 0xFFFFFFFF,
          _vp(s["scratch"]), None)
    _call("vlt_hg_query_compact", lb, n, sel, _vp(s["index"]), _vp(s["addr"]), _vp(s["compact"]), None)
    _call("vlt_hg_update", n, queries, _vp(s["index"]), _vp(s["addr"]), _vp(s["compact"]), storage, decay, None)
    _call("vlt_hg_emit_queries", ctypes.byref(fp), w, h, lb, 1, n, _vp(bufs["depth"]),
          _vp(bufs["diff_hit_pos_normal"]), _vp(bufs["diff_hit_radiance"]), queries, count, None)
    # the compacted lists' order is unspecified, so the cells and the queries stand for them
    return {k: s[k] for k in ("storage", "decay", "selection", "queries", "count", "compact")}


_RUN = {"frame": _run_frame, "sequence": _run_sequence, "traced": _run_traced, "batch": _run_batch,
        "diffuse": _run_diffuse, "specular": _run_specular, "denoise": _run_denoise, "atrous": _run_atrous,
        "hashgrid": _run_hashgrid}


# ------------------------------------------------------------------- work

# Bytes per pixel from the record layouts of vlt.h. Inputs of a frame: depth 4,
# G-buffer 16, previous depth 4 and G-buffer 16, diffuse candidate 16, specular
# candidate 20. State, read and written: diffuse reservoir, specular reservoir, AO
# history, denoiser history. Outputs: two lighting images.
_FRAME_BYTES = {"ref": 76 + 2 * (16 + 28 + 4 + 13) + 8, "f32": 76 + 2 * (48 + 28 + 8 + 33) + 32,
                "f16": 76 + 2 * (17 + 28 + 4 + 17) + 16}
_LIGHT = {"ref": 4, "f32": 16, "f16": 8}
# Operations per tap and per pixel, counted from the reference's shaders (a
# transcendental, a division and a square root count as one each).
_DIFF_TAP, _SPEC_TAP, _ATROUS_TAP, _PIXEL = 90, 160, 45, 600


def _frame_flops(p):
    # a specular pixel runs taps x roughness taps: half of them on average
    return (p.diff_spatial_passes * p.diff_spatial_taps * _DIFF_TAP
            + p.spec_spatial_passes * p.spec_spatial_taps * _SPEC_TAP // 2
            + p.atrous_iterations * 20 * _ATROUS_TAP + _PIXEL)


def _frame_work(case, n, p):
    cells = (16 << p.hg_log2_buckets) if p.hg_enable else 0
    queries = min(n, p.hg_max_queries or n) if p.hg_enable else 0
    b = (_FRAME_BYTES[case["form"]] + (2 * _LIGHT[case["form"]] if p.post else 0)
         + (2 * _LIGHT[case["form"]] if p.post == 2 else 0)) * n + 2 * cells + 64 * queries
    return {"bytes": b, "flops": n * _frame_flops(p)}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = sum(w * h for w, h in _batch_sizes(case))
        p = _knobs(case)
        p.hg_log2_buckets = 14
        one = _frame_work(case, n, p)
        return {"bytes": one["bytes"] + (case["views"] - 1) * 2 * (16 << 14), "flops": one["flops"]}
    n = case["w"] * case["h"]
    if kind == "frame":
        return _frame_work(case, n, _knobs(case))
    if kind == "sequence":
        one = _frame_work(case, n, _knobs(case))
        return {k: v * case["n"] for k, v in one.items()}
    if kind == "traced":
        p = _knobs(case)
        one = _frame_work(case, n, p)
        rays = 2 * n + min(16 << p.hg_log2_buckets, p.hg_max_queries or n)
        return {"bytes": one["bytes"] + rays * (32 + 64) * 2, "flops": one["flops"] + rays * 150}
    if kind == "diffuse":
        p = _knobs(case)
        return {"bytes": n * (4 + 4 + 4 + 16 + 4 + 16 + 4 + 2 + 16 + 4), "flops": n * (p.diff_spatial_taps * _DIFF_TAP + 250)}
    if kind == "specular":
        p = _knobs(case)
        return {"bytes": n * (4 + 4 + 8 + 8 + 28 + 20 + 28 + 6), "flops": n * (p.spec_spatial_taps * _SPEC_TAP // 2 + 500)}
    if kind == "denoise":
        fast = 8 if case["fast"] else 0
        return {"bytes": n * (4 + 8 + 4 + 4 + 2 + 4 + 8 + 8 + 4 + 1 + fast + 1 + fast + 12 + 12), "flops": n * 400}
    if kind == "atrous":
        return {"bytes": n * (4 + 8 + 12 + 12), "flops": n * case["iterations"] * 20 * _ATROUS_TAP}
    cells = 16 << case["log2_buckets"]
    return {"bytes": n * (16 + 32 + 32) + cells * (2 + 8), "flops": n * 120}


# ------------------------------------------------------------------ exact

def exact(case, seed):
    """Binary64 values of the computed (binary16) outputs of the AO passes and of the
    a-trous filter. The other float outputs depend on random-walk decisions (reservoirs,
    and with them everything a frame computes), which have no value of their own."""
    if case["kind"] == "diffuse":
        ao, filtered = _exact_ao(prepare(case, seed))
        return {"ao": ao, "ao_filtered": filtered, "reservoir": None, "lighting": None}
    if case["kind"] == "atrous":
        return {"color": None, "variance": _exact_atrous(prepare(case, seed))}
    return None


def _matrix(m):
    return torch.tensor(list(m), dtype=torch.float64, device="cuda").view(4, 4)  # rows are columns


def _exact_ao(s):
    w, h = s["case"]["w"], s["case"]["h"]
    fp, dev = s["fp"], "cuda"
    depth = s["cur"]["depth"].view(torch.float32).double().view(h, w)
    hist = s["got"]["ao_history"].view(torch.float16).double().view(h, w, 2)
    y, x = torch.meshgrid(torch.arange(h, device=dev).double(), torch.arange(w, device=dev).double(), indexing="ij")
    uv = torch.stack([(x + 0.5) / w, (y + 0.5) / h], -1)

    def project(m, p):
        q = torch.cat([p, torch.ones_like(p[..., :1])], -1) @ _matrix(m)
        return q[..., :3] / q[..., 3:]

    pos = project(fp.inv_view_proj, torch.cat([uv * 2 - 1, depth[..., None]], -1))
    j = [float(v) for v in fp.jitter]
    ndc = project(fp.view_proj, pos)[..., :2] - torch.tensor(j[:2], device=dev).double()
    ndc_p = project(fp.prev_view_proj, pos)[..., :2] - torch.tensor(j[2:], device=dev).double()
    huv = uv - (ndc - ndc_p) * 0.5
    inside = ((huv >= 0) & (huv <= 1)).all(-1)
    st = torch.where(inside[..., None], huv, torch.zeros_like(huv)) * torch.tensor([w, h], device=dev) - 0.5
    fl = torch.floor(st)
    fr = (st - fl)[..., None]
    x0, y0 = fl[..., 0].long(), fl[..., 1].long()

    def tap(yy, xx):
        return hist[yy.clamp(0, h - 1), xx.clamp(0, w - 1)]

    top = torch.lerp(tap(y0, x0), tap(y0, x0 + 1), fr[..., 0, :])
    bottom = torch.lerp(tap(y0 + 1, x0), tap(y0 + 1, x0 + 1), fr[..., 0, :])
    old = torch.lerp(top, bottom, fr[..., 1, :]) * inside[..., None]
    word = s["cur"]["diff_hit_pos_normal"].view(torch.float16).view(h, w, 4)[..., :3].double()
    near = ((word - pos).norm(dim=-1) >= s["params"].ao_radius).double()
    ao = near + (31.0 / 32.0) * old[..., 1] * (old[..., 0] - near)
    sky = depth == 0
    ao = torch.where(sky, torch.zeros_like(ao), ao)
    full = torch.stack([ao, (~sky).double()], -1)

    # 3x3 taps: a neighbour across a depth step counts as the centre; a coordinate below
    # zero is out of range, one past the end clamps out of range, and both read zero
    def shifted(img, dy, dx):
        out = torch.zeros_like(img)
        ys, yd = slice(max(dy, 0), h + min(dy, 0)), slice(max(-dy, 0), h + min(-dy, 0))
        xs, xd = slice(max(dx, 0), w + min(dx, 0)), slice(max(-dx, 0), w + min(-dx, 0))
        out[yd, xd] = img[ys, xs]
        return out

    med, lo, hi = [], [], []
    for dy in (-1, 0, 1):
        row = [torch.where((depth - shifted(depth, dy, dx)).abs() > 0.0005, ao, shifted(ao, dy, dx))
               for dx in (-1, 0, 1)]
        med.append(torch.minimum(torch.maximum(row[0], row[1]), row[2]))
        lo.append(torch.minimum(torch.minimum(row[0], row[1]), row[2]))
        hi.append(torch.maximum(torch.maximum(row[0], row[1]), row[2]))
    a = torch.minimum(torch.minimum(hi[0], hi[1]), hi[2])
    b = torch.maximum(torch.maximum(lo[0], lo[1]), lo[2])
    c = torch.minimum(torch.maximum(med[0], med[1]), med[2])
    m = torch.minimum(torch.maximum(c, a), b)
    mn = torch.minimum(torch.minimum(lo[0], lo[1]), lo[2])
    filtered = torch.where(sky, torch.zeros_like(m), 0.5 * (m + mn))
    return full.reshape(-1), filtered.reshape(-1)


def _small_float(bits, mantissa):
    e, m = bits >> mantissa, (bits & ((1 << mantissa) - 1)).double()
    return torch.where(e == 0, m * 2.0 ** (-14 - mantissa),
                       (1 + m * 2.0 ** -mantissa) * torch.pow(torch.tensor(2.0, device="cuda").double(), (e - 15).double()))


def _unpack(word):
    u = word.long() & 0xFFFFFFFF
    return torch.stack([_small_float(u & 0x7FF, 6), _small_float((u >> 11) & 0x7FF, 6), _small_float(u >> 22, 5)], -1)


def _as_stored(c):
    """The values that an unsigned small-float image (11, 11 and 10 bits) keeps."""
    out = []
    for k, mantissa in ((0, 6), (1, 6), (2, 5)):
        v = torch.nan_to_num(c[..., k], nan=0.0).clamp(min=0.0)
        step = torch.pow(torch.tensor(2.0, device="cuda").double(), torch.floor(torch.log2(v.clamp(min=2.0 ** -14))) - mantissa)
        top = (2 - 2.0 ** -mantissa) * 2.0 ** 15
        out.append((torch.round(v / step) * step).clamp(max=top))
    return torch.stack(out, -1)


def _exact_atrous(s):
    w, h = s["case"]["w"], s["case"]["h"]
    dev = "cuda"
    depth = s["cur"]["depth"].view(torch.float32).double().view(h, w)
    g = s["cur"]["gbuffer"].view(torch.int32).view(4, h, w).long() & 0xFFFFFFFF
    fx, fy = (g[1] & 0xFFF).double() / 4095 * 2 - 1, ((g[1] >> 12) & 0xFFF).double() / 4095 * 2 - 1
    nz = 1 - fx.abs() - fy.abs()
    t = (-nz).clamp(0, 1)
    normal = torch.stack([fx - torch.where(fx >= 0, t, -t), fy - torch.where(fy >= 0, t, -t), nz], -1)
    normal = normal / normal.norm(dim=-1, keepdim=True)
    fwz = (g[2] & 0xFFFF).to(torch.int32).to(torch.int16).view(torch.float16).double()
    color = s["color"].view(h, w, 2)
    col = torch.stack([_unpack(color[..., 0]), _unpack(color[..., 1])], -2)  # h, w, channel, rgb
    var = s["variance"].double().view(h, w, 2)
    lum_w = torch.tensor([0.2126, 0.7152, 0.0722], device=dev).double()
    kernel = (1.0, 2.0 / 3.0, 1.0 / 6.0)
    for it in range(s["case"]["iterations"]):
        step = 1 << it
        lum = col @ lum_w
        rcp = 1 / (4 * var.sqrt() + 1e-8)
        csum, vsum, wsum = col.clone(), var.clone(), torch.ones_like(var)
        for oy in (-2, -1, 1, 2):
            for ox in (-2, -1, 1, 2):
                dy, dx = oy * step, ox * step
                if abs(dy) >= h or abs(dx) >= w:
                    continue
                yc, xc = slice(max(-dy, 0), h - max(dy, 0)), slice(max(-dx, 0), w - max(dx, 0))
                yt, xt = slice(max(dy, 0), h - max(-dy, 0)), slice(max(dx, 0), w - max(-dx, 0))
                dist = math.sqrt(dx * dx + dy * dy)
                wz = -(depth[yt, xt] - depth[yc, xc]).abs() / (fwz[yc, xc] * dist + 1e-8)
                nd = (normal[yt, xt] * normal[yc, xc]).sum(-1).clamp(0, 1) ** 128
                wl = -(lum[yt, xt] - lum[yc, xc]).abs() * rcp[yc, xc]
                wt = kernel[abs(oy)] * kernel[abs(ox)] * nd[..., None] * torch.exp(wz[..., None] + wl)
                csum[yc, xc] += wt[..., None] * col[yt, xt]
                vsum[yc, xc] += wt * wt * var[yt, xt]
                wsum[yc, xc] += wt
        col = torch.stack([_as_stored(csum[..., k, :] / wsum[..., k, None]) for k in (0, 1)], -2)
        var = (vsum / (wsum * wsum)).half().double()
    return var.reshape(-1)
