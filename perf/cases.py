"""The work a user of this framework has it do, as timed cases.

Every case goes through a public entry point of `unblending_b200`: the
device-resident passes, the host-buffer API, the batched first pass, the
allocation-free first pass and the warm-start network. Images come from the
repository's own seeded generator (`unblending_b200.synthetic`), with its
blend-mode stacks, blob sizes and radii. A case is a dict of plain values:

  kind       which entry points run (see `run`)
  width, height (or sides of a batch), modes (bottom to top)
  sigma_lo, sigma_hi, noise     the generator's blob sizes and colour noise
  and the options that the entry points take.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import unblending_b200 as U
from unblending_b200 import synthetic as syn

L3 = "normal,multiply,screen"
L5 = "normal,multiply,screen,overlay,color_dodge"
L6 = "normal,multiply,screen,overlay,color_dodge,soft_light"
L8 = "normal,multiply,screen,overlay,color_dodge,soft_light,color_burn,hard_light"


def listed():
    return [
        # The smallest call: a preview tile, the first pass on a device-resident image. Latency.
        dict(name="unmix_tile", kind="unmix", width=37, height=23, modes=L3, sigma_lo=10.0, sigma_hi=60.0),
        # The three-layer 256x256 configuration, both passes, refinement radius 4.
        dict(name="decompose_rgb256_l3", kind="decompose", width=256, height=256, modes=L3, sigma_lo=10.0,
             sigma_hi=60.0, radius=4, smooth=True),
        # The five-layer 1024x1024 configuration (the repository's benchmark), both passes, the reference's radius.
        dict(name="decompose_rgb1024_l5", kind="decompose", width=1024, height=1024, modes=L5, sigma_lo=20.0,
             sigma_hi=200.0, radius=-1, smooth=True),
        # The six-layer configuration with colour noise (radius 8) at 1280x960: the largest case here.
        dict(name="decompose_noise_l6", kind="decompose", width=1280, height=960, modes=L6, sigma_lo=50.0,
             sigma_hi=800.0, noise=0.01, radius=8, smooth=True),
        # A C++ or Python host program on plain heap buffers, odd sizes: the reference's two calls.
        dict(name="host_two_calls_l4", kind="host", width=683, height=431, modes="normal,multiply,overlay,color_burn",
             sigma_lo=20.0, sigma_hi=200.0, smooth=True),
        # Plus-composited layers over a background that may be transparent, the background kept as solved.
        dict(name="decompose_plus_l3", kind="decompose", width=517, height=389, modes="normal,multiply,lighten",
             sigma_lo=20.0, sigma_hi=120.0, radius=-1, smooth=False, opaque=False, plus=True),
        # Eight layers, the most the library takes, from three solver starts.
        dict(name="unmix_l8_starts3", kind="unmix", width=211, height=160, modes=L8, sigma_lo=20.0, sigma_hi=120.0,
             starts=3),
        # The batched first pass over images of uneven size and layer count, three to six layers.
        dict(name="batch_uneven", kind="batch", count=10, side_lo=128, side_hi=512, layers_lo=3, layers_hi=6),
        # The FP32 option: an FP32 solve and the FP64 re-solve of its misses, both passes.
        dict(name="decompose_fp32_l5", kind="decompose", width=640, height=480, modes=L5, sigma_lo=20.0,
             sigma_hi=200.0, radius=-1, smooth=True, fp32=True),
        # The first pass for callers that cannot allocate device memory.
        dict(name="unmix_noalloc_l5", kind="noalloc", width=400, height=300, modes=L5, sigma_lo=20.0, sigma_hi=200.0),
        # The warm-start network's predictions for a photograph-sized image.
        dict(name="mlp_predict", kind="predict", width=1280, height=853, modes=L5, sigma_lo=20.0, sigma_hi=200.0),
        # One forward and backward pass of the warm-start network over its default training batch.
        dict(name="mlp_loss_grad", kind="loss_grad", count=8192, layers=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _modes(rng, layers):
    return ",".join(["normal"] + [rng.choice(["normal", "multiply", "screen", "overlay", "color_dodge", "soft_light",
                                              "color_burn", "hard_light", "lighten"]) for _ in range(layers - 1)])


def draw(rng):
    kind = rng.choice(["unmix", "decompose", "decompose", "decompose", "host", "batch", "noalloc", "predict",
                       "loss_grad"])
    if kind == "loss_grad":
        return dict(kind=kind, count=_log_int(rng, 128, 16384), layers=rng.randint(2, 8))
    if kind == "batch":
        lo = rng.randint(2, 4)
        return dict(kind=kind, count=rng.randint(2, 12), side_lo=rng.randint(32, 128), side_hi=rng.randint(160, 448),
                    layers_lo=lo, layers_hi=rng.randint(lo, 6))
    layers = rng.randint(2, 8 if kind in ("unmix", "predict") else 6)
    # Sides over the range, with fewer pixels where there are more layers: a drawn case stays below the largest listed.
    most = {"predict": 1300, "noalloc": 420, "host": 640}.get(kind, 1000 if layers <= 4 else 640)
    height = _log_int(rng, 16, most)
    width = max(8, min(most, int(round(height * rng.uniform(0.75, 1.5)))))
    case = dict(kind=kind, width=width, height=height, modes=_modes(rng, layers), sigma_lo=10.0,
                sigma_hi=float(rng.randint(60, 200)))
    if kind == "decompose":
        plus = rng.random() < 0.2
        case.update(radius=rng.choice([-1, -1, 4, 8]), smooth=not plus and rng.random() < 0.7, plus=plus,
                    opaque=not plus, fp32=rng.random() < 0.25, noise=rng.choice([0.0, 0.0, 0.01]))
    elif kind == "unmix":
        case.update(fp32=rng.random() < 0.25, starts=rng.choice([1, 1, 2, 3]) if width * height < 100000 else 1)
    return case


# ------------------------------------------------------------------ inputs --
_STREAM = None


def _stream():
    """The program's one CUDA stream (the library's calls on a device share its scratch)."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def _image(case, seed):
    return syn.generate(case["width"], case["height"], [syn.MODES[m] for m in case["modes"].split(",")],
                        (case["sigma_lo"], case["sigma_hi"]), seed=seed, noise=case.get("noise", 0.0),
                        comp=syn.PLUS if case.get("plus") else syn.SOURCE_OVER)


def _batch(case, seed):
    """Images as `syn.batch` draws them: sizes, layer counts and modes of the case, colours and alphas of the seed."""
    rng = np.random.default_rng([case["count"], case["side_lo"], case["side_hi"], 17])
    for k in range(case["count"]):
        side = int(rng.integers(case["side_lo"], case["side_hi"] + 1))
        w, h = side, max(1, int(round(side / rng.uniform(1.0, 4.0 / 3.0))))
        if rng.random() < 0.5:
            w, h = h, w
        layers = int(rng.integers(case["layers_lo"], case["layers_hi"] + 1))
        modes = [syn.MODES["normal"]] + [int(m) for m in rng.choice(syn.BATCH_MODES, size=layers - 1)]
        yield syn.generate(w, h, modes, (20.0, 200.0), seed=1000 * seed + k)


def _network(layers, seed):
    """A network with the initialization that training starts from, as float arrays by field name."""
    rng = np.random.default_rng([seed, 11])
    net = {}
    for k, (rows, cols) in enumerate(((64, 32), (64, 64), (64, 64), (32, 64))):
        used = rows if k < 3 else 4 * layers
        bound = math.sqrt(6.0 / (30 if k == 0 else cols)) if k < 3 else math.sqrt(6.0 / (cols + used))
        w = rng.uniform(-bound, bound, (rows, cols)).astype(np.float32)
        b = rng.uniform(-0.1, 0.1, rows).astype(np.float32)
        w[used:] = 0.0
        b[used:] = 0.0
        net["w%d" % (k + 1)], net["b%d" % (k + 1)] = w, b
    return net


def _mlp(layers, seed):
    model = U.Mlp.new()
    model.layer_count = layers
    for name, value in _network(layers, seed).items():
        model.set(name, value)
    return model


def _samples(case, seed):
    """Features (count, 32) and targets (count, 4L) of a training batch: colours of a neighbourhood, start points."""
    rng = np.random.default_rng([seed, 13])
    n, outs = case["count"], 4 * case["layers"]
    f = np.zeros((n, 32), np.float32)
    centre = rng.uniform(0.0, 1.0, (n, 3))
    f[:, :27] = np.clip(np.tile(centre, (1, 9)) + rng.normal(0.0, 0.1, (n, 27)), 0.0, 1.0)
    f[:, 12:15] = centre
    f[:, 27:30] = np.log(f[:, 12:15] + np.float32(1.0 / 256.0))
    return f, rng.uniform(0.0, 1.0, (n, outs)).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "loss_grad":
        f, t = _samples(case, seed)
        s.update(model=_mlp(case["layers"], seed), features=torch.from_numpy(f).cuda(),
                 targets=torch.from_numpy(t).cuda())
        torch.cuda.synchronize()
        return s
    if kind == "batch":
        jobs = []
        for wl in _batch(case, seed):
            image = torch.from_numpy(wl.image).cuda()
            out = torch.empty((len(wl.layers), wl.height, wl.width, 4), dtype=torch.float64, device="cuda")
            status = torch.empty(wl.pixels, dtype=torch.int32, device="cuda")
            jobs.append(dict(width=wl.width, height=wl.height, d_image=image.data_ptr(),
                             layers=syn.layer_array(wl.layers), d_output=out.data_ptr(),
                             d_status=status.data_ptr(), image=image, out=out, status=status))
        s.update(jobs=jobs, solver=U.solver_options())
        torch.cuda.synchronize()
        return s
    wl = _image(case, seed)
    n, layers = wl.pixels, len(wl.layers)
    s.update(width=wl.width, height=wl.height, layers=syn.layer_array(wl.layers), opaque=case.get("opaque", True),
             smooth=case.get("smooth", False))
    if kind == "host":
        s.update(image=wl.image)
        return s
    s.update(image=torch.from_numpy(wl.image).cuda())
    if kind == "predict":
        s.update(model=_mlp(layers, seed), out=torch.empty((n, 4 * layers), dtype=torch.float32, device="cuda"))
        torch.cuda.synchronize()
        return s
    s.update(solver=U.solver_options(precision=U.PRECISION_FP32 if case.get("fp32") else U.PRECISION_FP64,
                                     radius=case.get("radius", -1), starts=case.get("starts", 1)),
             first=torch.empty((layers, wl.height, wl.width, 4), dtype=torch.float64, device="cuda"),
             status=torch.empty(n, dtype=torch.int32, device="cuda"))
    if kind == "decompose":
        s.update(final=torch.empty_like(s["first"]), status2=torch.empty_like(s["status"]))
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "host":
        first = U.compute_color_unmixing(s["image"], s["layers"], s["opaque"])
        final = U.perform_matte_refinement(s["image"], first, s["layers"], s["opaque"], s["smooth"])
        return {"first": first, "final": final}
    if kind == "loss_grad":
        g = U.mlp_loss_grad_device(s["model"], s["case"]["count"], s["features"].data_ptr(), s["targets"].data_ptr())
        return {"loss": float(g.loss), **{name: g.get(name) for name in g.SHAPES}}
    stream = _stream().cuda_stream
    if kind == "batch":
        U.unmix_batch_device(s["jobs"], solver=s["solver"], stream=stream)
        return [{"out": j["out"], "status": j["status"]} for j in s["jobs"]]
    w, h, image = s["width"], s["height"], s["image"].data_ptr()
    if kind == "predict":
        U.mlp_predict_device(s["model"], w, h, image, s["out"].data_ptr(), stream=stream)
        return s["out"]
    if kind == "noalloc":
        U.unmix_device_noalloc(w, h, image, s["layers"], s["first"].data_ptr(), opaque=s["opaque"],
                               solver=s["solver"], d_status=s["status"].data_ptr(), stream=stream)
        return {"first": s["first"], "status": s["status"]}
    U.unmix_device(w, h, image, s["layers"], s["first"].data_ptr(), opaque=s["opaque"], solver=s["solver"],
                   d_status=s["status"].data_ptr(), stream=stream)
    if kind == "unmix":
        return {"first": s["first"], "status": s["status"]}
    U.refine_device(w, h, image, s["layers"], s["first"].data_ptr(), s["final"].data_ptr(), opaque=s["opaque"],
                    smooth=s["smooth"], solver=s["solver"], d_status=s["status2"].data_ptr(), stream=stream)
    return {"first": s["first"], "status": s["status"], "final": s["final"], "status2": s["status2"]}


# -------------------------------------------------------------------- work --
# Evaluations a pixel takes in one pass of the method, and how many of them need a gradient (a pixel that converges).
VALUES, GRADIENTS = 110, 25


def _solve_flops(modes):
    """Flops of one pass for one pixel: the composite, the colour prior and the constraint rows of an evaluation,
    the reverse sweep of a gradient (add, multiply, divide: one each)."""
    layers = len(modes)
    value = (layers - 1) * (7 + 3 * 15) + layers * 26 + 20
    gradient = layers * 21 + (layers - 1) * (8 + 3 * 35)
    return VALUES * value + GRADIENTS * gradient


def work(case):
    kind = case["kind"]
    macs = 32 * 64 + 64 * 64 * 2 + 64 * 32
    if kind == "loss_grad":
        n = case["count"]
        return {"bytes": n * (32 + 4 * case["layers"]) * 4 + 2 * (macs + 224) * 4, "flops": 2 * n * macs * 3}
    if kind == "batch":
        side = 0.5 * (case["side_lo"] + case["side_hi"])
        n = case["count"] * side * side / 1.17
        layers = (case["layers_lo"] + case["layers_hi"]) // 2
        return {"bytes": n * (24 + 32 * layers + 4), "flops": n * _solve_flops(["normal"] * layers)}
    n = case["width"] * case["height"]
    modes = case["modes"].split(",")
    layers = len(modes)
    if kind == "predict":
        return {"bytes": n * (24 + 16 * layers) + macs * 4, "flops": 2 * n * macs}
    passes = 2 if kind in ("decompose", "host") else 1
    return {"bytes": n * (24 + 32 * layers + 4) + (passes - 1) * n * (24 + 64 * layers + 4),
            "flops": n * passes * _solve_flops(modes) * case.get("starts", 1)}


# ------------------------------------------------------------------- exact --
def _forward(net, f):
    """Activations of the network's four layers in 64 bits (GELU, then sigmoid), and the pre-activations."""
    h, hs, zs = f, [f], []
    for k in range(1, 5):
        z = h @ net["w%d" % k].astype(np.float64).T + net["b%d" % k].astype(np.float64)
        zs.append(z)
        if k < 4:
            h = 0.5 * z * (1.0 + torch.erf(torch.from_numpy(z / math.sqrt(2.0))).numpy())
            hs.append(h)
    return 1.0 / (1.0 + np.exp(-zs[3])), hs, zs


def exact(case, seed):
    """The warm-start network in 64 bits. The solves have no such value: the method stops at its own tolerance, so
    where it ends is defined by its arithmetic alone."""
    if case["kind"] == "predict":
        img = _image(case, seed).image
        layers = len(case["modes"].split(","))
        net = _network(layers, seed)
        h, w, _ = img.shape
        pad = np.pad(img, ((1, 1), (1, 1), (0, 0)), mode="edge")
        f = np.zeros((h * w, 32))
        k = 0
        for dy in range(3):
            for dx in range(3):
                f[:, k:k + 3] = pad[dy:dy + h, dx:dx + w].reshape(-1, 3)
                k += 3
        f[:, 27:30] = np.log(img.reshape(-1, 3) + 1.0 / 256.0)
        out = np.empty((h * w, 4 * layers))
        for i in range(0, h * w, 65536):
            out[i:i + 65536] = _forward(net, f[i:i + 65536])[0][:, :4 * layers]
        return out
    if case["kind"] == "loss_grad":
        f, t = (a.astype(np.float64) for a in _samples(case, seed))
        net = _network(case["layers"], seed)
        n, outs = t.shape
        y, hs, zs = _forward(net, f)
        e = y[:, :outs] - t
        d = np.zeros_like(y)
        d[:, :outs] = 2.0 / (n * outs) * e * y[:, :outs] * (1.0 - y[:, :outs])
        g = {"loss": float(np.mean(e * e))}
        for k in (4, 3, 2, 1):
            g["w%d" % k], g["b%d" % k] = d.T @ hs[k - 1], d.sum(axis=0)
            if k > 1:
                z = zs[k - 2]
                slope = 0.5 * (1.0 + torch.erf(torch.from_numpy(z / math.sqrt(2.0))).numpy()) + \
                    z * np.exp(-0.5 * z * z) / math.sqrt(2.0 * math.pi)
                d = (d @ net["w%d" % k].astype(np.float64)) * slope
        return g
    return None
