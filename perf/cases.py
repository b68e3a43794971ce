"""The render path's performance cases: what a program that uses this library has it do, from a thumbnail to
a 24-megapixel photograph.

Every case goes through the public C ABI by its ctypes binding (spk_ctypes) or the torch binding
(spk_torch). A case is a dict of plain values; its "kind" says which call a pass makes:

  render    spk_render of an open session: develop, print, scan, result in pinned host memory
  reprint   spk_set_params (a print slider) and spk_reprint of the cached negative
  open      spk_open_device, spk_render of the live tier, spk_session_release: a photograph is looked at
  print     spkx_print_negative: densities to RGBA16 in device memory (no copy to the host)
  vjp       spk_render_vjp: the adjoint of the render, host arrays in and out
  fit       spk_torch.render_linear, a loss and its backward pass: one step of a parameter fit
  batch     spkx_render_batch of frames of mixed sizes

"look" is the parameter set: "bench" the benchmark's (halation mixture given in pixels, no couplers, no
glare), "defaults" the engine's own defaults (auto exposure, DIR couplers, halation preset, glare).
"scene" is the picture: "noise" the benchmark's log-uniform RGB in [2^-8, 2^2], every pixel its own;
"photo" smooth shading, flat regions with edges, and sensor noise over the same range.
"""

import json
import math
import os
import random
import sys

import numpy as np
import torch

# the package folder's name is not an identifier: its modules are imported from the folder itself
sys.path.insert(0, os.path.join(os.getcwd(), "spektralab-engine_b200"))

import spk_ctypes as sc  # noqa: E402
import spk_torch  # noqa: E402
import synth_resources  # noqa: E402

STOCKS = {"film_stock": "synthetic_negative_400", "print_stock": "synthetic_paper"}
BENCH = dict(STOCKS, auto_exposure=False, dir_couplers_active=False, glare_active=False)
FILM_SEED = 7
SLIDER = (1.2, 0.85, 1.0, 1.35)  # print exposures a user drags through
NODES = 3 * 16  # density-curve parameters of the adjoint

_engine = None


def engine():
    """One engine for the process, as a host application keeps it."""
    global _engine
    if _engine is None:
        _engine = sc.load().engine(synth_resources.ensure(sc.RESOURCES), device=0)
    return _engine


# ---- the cases --------------------------------------------------------------------------------------


def listed():
    return [
        # a contact-sheet thumbnail: launches and host work count, not pixels; odd size
        {"name": "thumb_131x97", "kind": "render", "w": 131, "h": 97, "look": "bench", "scene": "photo",
         "sigma0": 3.5, "sigma1": 17.0, "lens": 0.0, "grain": True, "tier": "full"},
        # the preview workload: 512 x 512, halation sigma 8 and 40 px
        {"name": "preview_512", "kind": "render", "w": 512, "h": 512, "look": "bench", "scene": "noise",
         "sigma0": 8.0, "sigma1": 40.0, "lens": 0.0, "grain": True, "tier": "preview"},
        # the headline workload's render
        {"name": "render_4k", "kind": "render", "w": 3840, "h": 2160, "look": "bench", "scene": "noise",
         "sigma0": 20.0, "sigma1": 120.0, "lens": 1.5, "grain": True, "tier": "full"},
        # the headline workload's reprint: a print slider is dragged on a developed 4K frame
        {"name": "reprint_4k", "kind": "reprint", "w": 3840, "h": 2160, "look": "bench", "scene": "noise",
         "sigma0": 20.0, "sigma1": 120.0, "lens": 1.5, "grain": True, "tier": "full"},
        # the engine's defaults on a small photograph whose width is odd
        {"name": "defaults_1999x1333", "kind": "render", "w": 1999, "h": 1333, "look": "defaults", "scene": "photo",
         "sigma0": 0.0, "sigma1": 0.0, "lens": 0.0, "grain": True, "tier": "full"},
        # a 24-megapixel photograph is opened and looked at: meter, live tier, defaults
        {"name": "open_24mp_live", "kind": "open", "w": 6000, "h": 4000, "look": "defaults", "scene": "photo",
         "sigma0": 0.0, "sigma1": 0.0, "lens": 0.0, "grain": True, "tier": "live"},
        # the same photograph exported at full size
        {"name": "export_24mp", "kind": "render", "w": 6000, "h": 4000, "look": "defaults", "scene": "photo",
         "sigma0": 0.0, "sigma1": 0.0, "lens": 0.0, "grain": True, "tier": "full"},
        # the print side alone on device buffers, for a host that shows the picture from device memory
        {"name": "print_24mp", "kind": "print", "w": 6144, "h": 4096, "mode": "fp32", "bins": 81, "lens": 1.5},
        # the same at 1 nm with the spectral integrals on the tensor cores (split BF16)
        {"name": "print_401_bf16x3", "kind": "print", "w": 2048, "h": 1365, "mode": "bf16x3", "bins": 401, "lens": 0.0},
        # the adjoint workload: 1024 x 1024, 55 parameters
        {"name": "vjp_1024", "kind": "vjp", "w": 1024, "h": 1024, "scene": "noise", "sigma0": 8.0, "sigma1": 40.0,
         "lens": 1.5},
        # one step of fitting print and halation parameters to a small odd crop, through torch
        {"name": "fit_333x250", "kind": "fit", "w": 333, "h": 250, "scene": "photo", "sigma0": 4.0, "sigma1": 21.0,
         "lens": 0.0},
        # a folder of frames of mixed sizes, each with its own halation and print exposure
        {"name": "batch_12", "kind": "batch", "scene": "photo", "lens": 1.5,
         "sizes": "256x256,401x307,640x427,800x1200,1023x683,1280x720,1365x2048,1501x1001,1920x1080,2048x1365,333x2500,2731x1820"},
    ]


def _size(rng, lo_px, hi_px):
    """A width and height of lo_px .. hi_px pixels, spread over the logarithm, aspect 2:3 .. 16:9, any parity."""
    px = math.exp(rng.uniform(math.log(lo_px), math.log(hi_px)))
    aspect = rng.choice((2 / 3, 3 / 4, 1.0, 4 / 3, 3 / 2, 16 / 9)) * rng.uniform(0.97, 1.03)
    w, h = max(16, round(math.sqrt(px * aspect))), max(16, round(math.sqrt(px / aspect)))
    if rng.random() < 0.5:  # a size as cameras and displays have it
        w, h = max(16, w // 4 * 4), max(16, h // 2 * 2)
    return w, h


def draw(rng):
    kind = rng.choice(("render", "render", "render", "reprint", "open", "print", "vjp", "fit", "batch"))
    if kind == "batch":
        return {"kind": kind, "scene": "photo", "lens": rng.choice((0.0, 1.5)),
                "sizes": ",".join("%dx%d" % _size(rng, 60e3, 3.5e6) for _ in range(rng.randint(3, 10)))}
    if kind == "print":
        mode, bins = rng.choice((("fp32", 81), ("fp32", 81), ("bf16x3", 81), ("bf16x3", 401)))
        w, h = _size(rng, 100e3, 25e6 if bins == 81 and mode == "fp32" else 4e6)
        return {"kind": kind, "w": w, "h": h, "mode": mode, "bins": bins, "lens": rng.choice((0.0, 0.7, 1.5))}
    if kind in ("vjp", "fit"):
        w, h = _size(rng, 12e3, 1.05e6 if kind == "vjp" else 150e3)
        s0 = rng.uniform(3.2, 12.0)
        return {"kind": kind, "w": w, "h": h, "scene": rng.choice(("noise", "photo")), "sigma0": round(s0, 2),
                "sigma1": round(s0 * rng.uniform(3.0, 5.0), 2), "lens": rng.choice((0.0, 1.5))}
    look = "defaults" if kind == "open" else rng.choice(("bench", "defaults"))
    lo, hi = (3e6, 24e6) if kind == "open" else (12e3, 24e6)
    w, h = _size(rng, lo, hi)
    s0 = max(w, h) / 200.0 * rng.uniform(0.7, 1.5) if look == "bench" else 0.0
    return {"kind": kind, "w": w, "h": h, "look": look, "scene": rng.choice(("noise", "photo")), "sigma0": round(max(s0, 0.8), 2) if s0 else 0.0,
            "sigma1": round(max(s0, 0.8) * rng.uniform(3.0, 6.0), 2) if s0 else 0.0, "lens": rng.choice((0.0, 0.0, 1.5, 0.7)),
            "grain": rng.random() < 0.8, "tier": "live" if kind == "open" else "full"}


# ---- inputs -----------------------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def picture(scene, w, h, seed):
    """Linear ProPhoto RGB in [2^-8, 2^2], (h, w, 3) float32 on the GPU."""
    g = _generator(seed)
    if scene == "noise":
        return torch.exp2(torch.rand((h, w, 3), generator=g, device="cuda") * 10.0 - 8.0)
    grow = torch.nn.functional.interpolate
    ev = torch.zeros((1, 3, h, w), device="cuda")
    for cells, amount in ((4, 2.2), (24, 0.9)):  # shading
        grid = torch.randn((1, 1, cells, cells), generator=g, device="cuda") * amount
        ev += grow(grid, size=(h, w), mode="bicubic", align_corners=True)
    for cells, amount in ((9, 0.9), (60, 0.35)):  # objects: flat regions with a colour each
        grid = torch.randn((1, 3, cells, cells), generator=g, device="cuda") * amount
        ev += grow(grid, size=(h, w), mode="nearest")
    ev += torch.randn((1, 3, h, w), generator=g, device="cuda") * 0.06  # sensor noise
    return torch.exp2((ev - 3.0).clamp_(-8.0, 2.0))[0].permute(1, 2, 0).contiguous()


def densities(w, h, seed):
    """Dye densities of a negative: (h, w, 3) float32 in [0, 3] on the GPU."""
    return torch.rand((h, w, 3), generator=_generator(seed), device="cuda") * 3.0


def open_device(frame, delta):
    """spk_open_device on a GPU tensor (h, w, 3): a Session."""
    e = engine()
    h, w, c = frame.shape
    torch.cuda.current_stream().synchronize()  # the frame is read on the session's stream
    image = sc.SpkDeviceImage(frame.data_ptr(), w, h, c)
    handle = e.L.lib.spk_open_device(e.h, image, json.dumps(delta).encode(), None)
    if not handle:
        raise sc.SpkError(-2, e.L.last_error())
    return sc.Session(e, handle, None, (h, w))


def delta_of(case, long_edge):
    if case.get("look") == "defaults":
        return dict(STOCKS, grain_active=case["grain"], scanner_lens_blur=case["lens"])
    # the benchmark's film format: about 600 grains per pixel and sub-layer
    return dict(BENCH, film_format_mm=round(min(200.0, max(4.0, 92.5877 * long_edge / 3840.0)), 4),
                grain_active=case.get("grain", True), scanner_lens_blur=case["lens"])


def set_halation(session, case, weight):
    if case.get("sigma0"):
        session.set_halation([((weight,) * 3, (case["sigma0"],) * 3), ((weight,) * 3, (case["sigma1"],) * 3)],
                             (0.03, 0.03, 0.03))


class State:
    """What the caller's program holds: sessions, inputs, and the last results until the next ones come."""

    def __init__(self, case):
        self.case, self.sessions, self.results, self.passes = case, [], [], 0

    def keep(self, results):
        old, self.results = self.results, results
        for r in old:
            r.free()

    def __del__(self):
        self.keep([])
        for s in self.sessions:
            s.close()


def prepare(case, seed):
    st = State(case)
    kind = case["kind"]
    if kind == "batch":
        rng = random.Random(seed)
        for i, size in enumerate(case["sizes"].split(",")):
            w, h = (int(v) for v in size.split("x"))
            s = open_device(picture(case["scene"], w, h, seed * 64 + i),
                            dict(BENCH, film_format_mm=35.0, print_exposure=rng.uniform(0.7, 1.4), scanner_lens_blur=case["lens"]))
            s.set_halation([((1, 1, 1), (rng.uniform(5, 30),) * 3), ((1, 1, 1), (rng.uniform(40, 160),) * 3)],
                           (0.03, 0.03, 0.03))
            st.sessions.append(s)
        return st
    w, h = case["w"], case["h"]
    if kind == "print":
        st.negative = densities(w, h, seed)
        st.stride = (w + 31) // 32 * 32
        st.out = torch.zeros((h, st.stride, 4), dtype=torch.int16, device="cuda")
        s = open_device(picture("photo", 64, 48, 1), dict(BENCH, scanner_lens_blur=case["lens"]))
        s.set_print_mode(case["mode"], case["bins"])
        st.sessions.append(s)
        torch.cuda.synchronize()
        return st
    frame = picture(case["scene"], w, h, seed)
    delta = delta_of(case, max(w, h))
    if kind == "open":
        st.frame, st.delta = frame, delta
        return st
    if kind == "fit":
        st.image = frame.cpu().requires_grad_(True)
        st.params = torch.tensor([1.1, 0.02, -0.01, 0.8, 1.2, case["sigma0"], case["sigma1"]], dtype=torch.float64,
                                 requires_grad=True)
        st.delta = delta
        st.target = frame.cpu() * 0.5 + 0.05
        return st
    s = open_device(frame, delta)
    st.sessions.append(s)
    set_halation(s, case, 0.02 if kind == "vjp" else 1.0)
    if kind == "vjp":
        st.grad = (picture("photo", w, h, seed + 1) - 0.3).cpu().numpy()
    if kind == "reprint":
        st.keep([s.render_result(case["tier"])])
    return st


# ---- one pass ---------------------------------------------------------------------------------------


def run(state):
    case, kind = state.case, state.case["kind"]
    state.passes += 1
    if kind == "render":
        state.keep([state.sessions[0].render_result(case["tier"])])
        return state.results[0].pixels
    if kind == "reprint":
        state.sessions[0].set_params({"print_exposure": SLIDER[state.passes % len(SLIDER)]})
        state.keep([state.sessions[0].render_result(case["tier"], reprint=True)])
        return state.results[0].pixels
    if kind == "open":
        with open_device(state.frame, state.delta) as s:
            state.keep([s.render_result(case["tier"])])
        return state.results[0].pixels
    if kind == "print":
        state.sessions[0].print_negative(state.negative.data_ptr(), case["w"], case["h"], state.out.data_ptr(),
                                         state.stride)
        return state.out[:, : case["w"]]
    if kind == "vjp":
        return state.sessions[0].render_vjp(state.grad, FILM_SEED, 7 + NODES, want_output=True)
    if kind == "fit":
        state.image.grad = state.params.grad = None
        y = spk_torch.render_linear(state.image, state.params, engine(), state.delta)
        loss = torch.square(y - state.target).sum()
        loss.backward()
        return {"output": y.detach(), "loss": loss.detach(), "image": state.image.grad, "params": state.params.grad}
    results, _ = engine().render_batch(state.sessions, "full")
    state.keep(results)
    return [r.pixels for r in results]


# ---- the least a pass can move and compute ----------------------------------------------------------

# Per pixel: the expose lookup (16 texels of the spectral table, 3 channels), the density curves and nine
# Poisson draws, the two spectral integrals (exponent, exponential and three sums per wavelength), the
# gamut stage, a scanner FIR, and a halation component (third-order recursion, both ways, rows and columns).
EXPOSE, DEVELOP, DRAW, GAMUT, SCAN, COMPONENT = 200, 80, 100, 300, 100, 4 * 3 * 8


def _film(case):
    components = 2 if case.get("sigma0") else (8 if case.get("look") == "defaults" else 0)
    return EXPOSE + DEVELOP + (9 * DRAW if case.get("grain", True) else 0) + components * COMPONENT


def _print(bins):
    return 2 * bins * 13 + GAMUT + SCAN


def work(case):
    kind = case["kind"]
    if kind == "batch":
        px = sum(int(s.split("x")[0]) * int(s.split("x")[1]) for s in case["sizes"].split(","))
        return {"bytes": px * (12 + 12 + 8), "flops": px * (_film({"sigma0": 1}) + _print(81))}
    px = case["w"] * case["h"]
    if kind == "render":  # the frame in, the negative kept, the RGBA16 result out
        return {"bytes": px * (12 + 12 + 8), "flops": px * (_film(case) + _print(81))}
    if kind == "reprint" or kind == "print":
        return {"bytes": px * (12 + 8), "flops": px * _print(case.get("bins", 81))}
    if kind == "open":  # the frame in and kept; the live tier's pixels developed and printed
        live = px * min(1.0, 1600.0 / max(case["w"], case["h"])) ** 2
        return {"bytes": px * 24 + live * 32, "flops": px * 40 + live * (_film(case) + _print(81))}
    # the adjoint: the forward, and the print's tangents along three densities and three parameters
    flops = _film({"sigma0": 1}) + _print(81) + 2 * 81 * 70 + 3000
    if kind == "fit":
        return {"bytes": px * 4 * 12, "flops": px * (flops + _film({"sigma0": 1}) + _print(81))}
    return {"bytes": px * 4 * 12, "flops": px * flops}


def exact(case, seed):
    """No case has a value in 64 bits: the pictures are whole numbers, and the adjoint's outputs hang on
    the Poisson counts of the binary32 sampler, which only the library draws."""
    return None
