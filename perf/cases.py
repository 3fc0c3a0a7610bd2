"""Performance cases: the reconstructions a user of the engine runs, through its public entry points.

listed() names the cases, draw() makes more of the same ranges, prepare()/run() do one, work() states the
bytes and operations one pass cannot do without, tolerance() how far two correct implementations may
differ, exact() the result in 64 bits from plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ufo-filters_b200"))

import ufob  # noqa: E402
from ufob import cnn  # noqa: E402

DEV = "cuda"
I0 = 1.0e4  # photons per ray of the noisy phantoms


# ------------------------------------------------------------------------------------------ cases

def listed():
    return [
        # the reference task's unit of work, one sinogram per call (the smallest call: launches and
        # latency count): 512 px, 512 angles, axis between the middle pixels
        dict(name="slice_512", kind="fbp", Z=1, P=512, W=512, axis=255.5, storage="f32"),
        # a group of slices of a full-size scan in the plain form
        dict(name="stack_f32", kind="fbp", Z=32, P=1500, W=2048, axis=1023.5, storage="f32"),
        # a larger group of the same scan with filtered sinograms stored in 16 bits, the form a whole
        # volume is reconstructed in
        dict(name="stack_f16", kind="fbp", Z=64, P=1500, W=2048, axis=1023.5, storage="f16"),
        # the same from pinned host memory and back, as a program with volumes larger than the GPU does
        dict(name="host_f16", kind="host", Z=32, P=1500, W=2048, axis=1023.5, storage="f16"),
        # raw projections of a cropped detector (odd width, rows and angle count, off-centre axis):
        # flat-field correction, transposition, filter and backprojection
        dict(name="raw_odd_f16", kind="raw", Z=13, P=721, W=1001, axis=487.25, storage="f16"),
        # the filter stage alone, rows out (a graph that does its own backprojection)
        dict(name="filter_rows", kind="filter", Z=64, P=1500, W=2048, storage="f32"),
        # cone-beam reconstruction: weighting, filter, general backprojection of a circular scan
        dict(name="cone_fdk", kind="cone", P=360, H=512, W=512, N=256, NZ=256),
        # laminography of a flat sample: a slab of slices tilted by 30 degrees about the beam
        dict(name="lamino_slab", kind="lamino", P=1024, H=1024, W=1024, N=512, NZ=96),
        # search for the rotation centre: one slice at many centre positions
        dict(name="centre_sweep", kind="sweep", P=360, H=512, W=512, N=512, NZ=40),
        # an uneven batch of independent sinograms in one call
        dict(name="batch_uneven", kind="batch", jobs=32, mix=2024, wmax=2048, pmax=1800, storage="f32"),
        # the learned sparse-view correction of a batch of slices
        dict(name="net_forward", kind="net", B=64, H=512, W=512),
        # its training: steps on pairs of sparse and dense slices
        dict(name="net_train", kind="train", B=16, H=512, W=512, steps=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _axis(rng, W):
    return round(W / 2.0 + rng.uniform(-0.04, 0.04) * W, 2)


def draw(rng):
    """One more case of the listed ranges; none does more than the largest listed one."""
    kind = rng.choice(["slice", "fbp", "fbp", "fbp", "host", "raw", "raw", "filter", "cone", "lamino", "sweep", "batch",
                       "net", "train"])
    storage = rng.choice(["f32", "f16"])
    if kind == "slice":
        W = _log_int(rng, 256, 2048)
        return dict(kind="fbp", Z=1, P=rng.randint(W // 3, W), W=W, axis=_axis(rng, W), storage=storage)
    if kind in ("fbp", "host", "raw"):
        W = _log_int(rng, 320, 2048)
        P = rng.randint(max(90, W // 3), min(1500, W + W // 2))
        room = 9.0e10 if storage == "f32" else 1.5e11
        Z = _log_int(rng, 2, max(3, min(96, int(room / (float(W) * W * P)))))
        return dict(kind=kind, Z=Z, P=P, W=W, axis=_axis(rng, W), storage=storage)
    if kind == "filter":
        W = _log_int(rng, 256, 4096)
        P = rng.randint(max(90, W // 3), min(1500, W))
        return dict(kind="filter", Z=_log_int(rng, 1, max(2, min(64, int(1.9e8 / (P * W))))), P=P, W=W,
                    storage=storage)
    if kind == "cone":
        W, H, N = rng.randint(90, 160) * 4, rng.randint(300, 640), rng.randint(120, 288)
        return dict(kind="cone", P=rng.randint(180, 480), H=H, W=W, N=N, NZ=rng.randint(24, N))
    if kind == "lamino":
        W, H, N = rng.randint(120, 256) * 4, rng.randint(400, 1024), rng.randint(200, 512)
        return dict(kind="lamino", P=rng.randint(300, 1024), H=H, W=W, N=N, NZ=rng.randint(16, 96))
    if kind == "sweep":
        W = rng.randint(80, 192) * 4
        return dict(kind="sweep", P=rng.randint(180, 480), H=rng.randint(256, 640), W=W, N=rng.randint(200, 512),
                    NZ=rng.randint(9, 48))
    if kind == "batch":
        return dict(kind="batch", jobs=rng.randint(4, 32), mix=rng.randint(1, 10 ** 6), wmax=rng.choice([512, 1024, 2048]),
                    pmax=rng.randint(400, 1800), storage=storage)
    if kind == "net":
        return dict(kind="net", B=_log_int(rng, 1, 64), H=32 * rng.randint(8, 20), W=32 * rng.randint(8, 20))
    return dict(kind="train", B=rng.randint(2, 16), H=32 * rng.randint(8, 16), W=32 * rng.randint(8, 16), steps=1)


# ----------------------------------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _ellipsoids(seed, n):
    """Random ellipsoids: centres uniform in the unit disc, semi-axes 0.05 to 0.4, densities -0.5 to 1."""
    rng = np.random.default_rng(seed)
    r, t = np.sqrt(rng.uniform(0, 1, n)), rng.uniform(0, 2 * math.pi, n)
    return np.stack([r * np.cos(t), r * np.sin(t), rng.uniform(-0.6, 0.6, n), rng.uniform(0.05, 0.4, n),
                     rng.uniform(0.05, 0.4, n), rng.uniform(0.2, 0.6, n), rng.uniform(0, math.pi, n),
                     rng.uniform(-0.5, 1.0, n)], axis=1)


def _sinograms(seed, Z, P, W, axis, n=12):
    """Noisy line integrals [Z, P, W] (pixel lengths) of ellipsoids, slices spread over the sample."""
    scale = 0.45 * W
    th = torch.arange(P, device=DEV, dtype=torch.float32)[:, None] * (math.pi / P)
    u = (torch.arange(W, device=DEV, dtype=torch.float32)[None, :] + 0.5 - axis) / scale
    z = (torch.arange(Z, device=DEV, dtype=torch.float32) + 0.5) / Z - 0.5
    out = torch.zeros(Z, P, W, device=DEV)
    for cx, cy, cz, a, b, c, phi, rho in _ellipsoids(seed, n):
        s2 = a * a * torch.cos(th - phi) ** 2 + b * b * torch.sin(th - phi) ** 2
        d2 = (u - cx * torch.cos(th) - cy * torch.sin(th)) ** 2 / s2
        k = 2.0 * rho * a * b / torch.sqrt(s2)
        for i in range(Z):
            f2 = 1.0 - (float(z[i]) - cz) ** 2 / (c * c)
            if f2 > 0:
                out[i] += k * torch.sqrt(torch.clamp(f2 - d2, min=0.0))
    out *= 1.0 / 2.4  # attenuation of a few units along the densest rays
    counts = torch.poisson(I0 * torch.exp(-torch.clamp(out, -2.0, 8.0)), generator=_gen(seed))
    return (-torch.log(torch.clamp(counts, min=0.5) / I0) * scale).contiguous()


def _projections(seed, P, H, W):
    """Projections [P, H, W] of balls turning about the vertical axis, with 1% noise."""
    rng = np.random.default_rng(seed)
    out = torch.randn(P, H, W, device=DEV, generator=_gen(seed)) * 0.01
    v = torch.arange(H, device=DEV, dtype=torch.float32)[:, None] + 0.5 - H / 2.0
    u = torch.arange(W, device=DEV, dtype=torch.float32)[None, :] + 0.5 - W / 2.0
    th = torch.arange(P, device=DEV, dtype=torch.float32)[:, None, None] * (2 * math.pi / P)
    for _ in range(6):
        r, t = 0.35 * W * math.sqrt(rng.uniform()), rng.uniform(0, 2 * math.pi)
        cz, rad, rho = rng.uniform(-0.3, 0.3) * H, rng.uniform(0.05, 0.2) * min(H, W), rng.uniform(0.2, 1.0)
        for p0 in range(0, P, 128):
            d2 = (u - r * torch.cos(th[p0:p0 + 128] + t)) ** 2 + (v - cz) ** 2
            out[p0:p0 + 128] += (2.0 * rho / rad) * torch.sqrt(torch.clamp(rad * rad - d2, min=0.0))
    return out


def _pow2(W):
    return 1 << (W - 1).bit_length()


def _fft_props(W):
    """The graph's fft size-x and ifft crop-width: the filter needs a power-of-two spectrum."""
    return {} if W == _pow2(W) else {"size_x": _pow2(W), "crop_width": W}


def _jobs(case):
    rng = np.random.default_rng(case["mix"])
    widths = [w for w in (256, 512, 1024, 1536, 2048) if w <= case["wmax"]]
    return [(int(rng.choice(widths)), int(rng.integers(180, case["pmax"] + 1))) for _ in range(case["jobs"])]


def _gbp_props(case):
    """Properties of the general backprojection: detector centre, region of interest, geometry."""
    N, NZ, W, H = case["N"], case["NZ"], case["W"], case["H"]
    p = {"center-position-x": W / 2.0 + 0.25, "center-position-z": H / 2.0,
         "x-region": (-N / 2.0, N / 2.0, 1.0), "y-region": (-N / 2.0, N / 2.0, 1.0)}
    if case["kind"] == "sweep":  # quarter-pixel steps around the nominal centre of one slice
        p.update({"parameter": "center-position-x", "z": 0.1 * H,
                  "region": (W / 2.0 - NZ / 8.0, W / 2.0 - NZ / 8.0 + NZ * 0.25 - 0.1, 0.25)})
        return p
    p["region"] = (-NZ / 2.0, NZ / 2.0, 1.0)
    if case["kind"] == "cone":  # source and detector distances of the 1024 px geometry, scaled
        p.update({"source-position-y": -800.0 * W / 512, "detector-position-y": 200.0 * W / 512})
    else:
        p["axis-angle-x"] = math.pi / 6
    return p


def _cone_weight(case):
    W, H = case["W"], case["H"]
    return {"center_position_x": W / 2.0 + 0.25, "center_position_z": H / 2.0, "source_distance": 800.0 * W / 512,
            "detector_distance": 200.0 * W / 512}


def _net_params(seed):
    """He-initialised parameters as one vector (per layer weights [Cout][9][Cin], then the bias)."""
    rng = np.random.default_rng(seed)
    out = []
    for ci, co, _ in LAYERS:
        out.append(rng.normal(0.0, math.sqrt(2.0 / (9.0 * ci)), size=co * 9 * ci))
        out.append(rng.normal(0.0, 0.02, size=co))
    return np.concatenate(out).astype(np.float32)


LAYERS = [(16, 32, True), (32, 64, True), (64, 128, True), (128, 256, True), (256, 128, True), (128, 64, True),
          (64, 32, True), (32, 16, False)]


def _slices(seed, B, H, W):
    """Reconstruction-like images (smooth objects) and the same with streaks and noise."""
    g = _gen(seed)
    rng = np.random.default_rng(seed)
    y = torch.arange(H, device=DEV, dtype=torch.float32)[:, None] / H - 0.5
    x = torch.arange(W, device=DEV, dtype=torch.float32)[None, :] / W - 0.5
    clean = torch.zeros(B, H, W, device=DEV)
    for i in range(B):
        for cx, cy, _, a, b, _, phi, rho in _ellipsoids(int(rng.integers(1 << 30)), 8):
            xr = (x - 0.4 * cx) * math.cos(phi) + (y - 0.4 * cy) * math.sin(phi)
            yr = -(x - 0.4 * cx) * math.sin(phi) + (y - 0.4 * cy) * math.cos(phi)
            clean[i] += rho * ((xr / a) ** 2 + (yr / b) ** 2 < 0.25)
    noisy = clean + 0.05 * torch.randn(B, H, W, device=DEV, generator=g)
    noisy += 0.1 * torch.sin(40.0 * (x + 0.3 * y))
    return noisy.contiguous(), clean.contiguous()


STORAGE = {"f32": ufob.F32, "f16": ufob.F16}


# ------------------------------------------------------------------------------------ prepare, run

def prepare(case, seed):
    """What a program holds before the call: inputs on the GPU (host memory for `host`), task objects
    and result buffers."""
    k = case["kind"]
    if k in ("fbp", "host", "raw"):
        Z, P, W = case["Z"], case["P"], case["W"]
        s = {"case": case, "fbp": ufob.FBP(filter_props=_fft_props(W), bp_props={"axis_pos": case["axis"]},
                                           storage=STORAGE[case["storage"]])}
        sino = _sinograms(seed, Z, P, W, case["axis"])
        if k == "fbp":
            s["sino"] = sino[0] if Z == 1 else sino
            s["out"] = torch.empty(Z, W, W, device=DEV)
        elif k == "host":
            s["sino"] = torch.empty(Z, P, W, pin_memory=True)
            s["sino"].copy_(sino)
            s["out"] = torch.empty(Z, W, W, pin_memory=True)
        else:
            g = _gen(seed + 1)
            s["dark"] = 100.0 + 10.0 * torch.rand(Z, W, device=DEV, generator=g)
            s["flat"] = s["dark"] + 10000.0 + 2000.0 * torch.rand(Z, W, device=DEV, generator=g)
            att = (sino / (0.45 * W)).transpose(0, 1)
            s["proj"] = (s["dark"] + (s["flat"] - s["dark"]) * torch.exp(-att)).contiguous()
            s["ffc"] = ufob.FlatFieldCorrectTask(absorption_correct=1)
            s["out"] = torch.empty(Z, W, W, device=DEV)
        return s
    if k == "filter":
        Z, P, W = case["Z"], case["P"], case["W"]
        return {"case": case, "task": ufob.FilterTask(**_fft_props(W)), "sino": _sinograms(seed, Z, P, W, W / 2.0),
                "out": torch.empty(Z, P, W, device=DEV,
                                   dtype=torch.float32 if case["storage"] == "f32" else torch.float16)}
    if k in ("cone", "lamino", "sweep"):
        t = ufob.GeneralBackprojectTask(num_projections=case["P"])
        for name, v in _gbp_props(case).items():
            t.set_property(name, v)
        s = {"case": case, "task": t, "proj": _projections(seed, case["P"], case["H"], case["W"]),
             "out": torch.empty(case["NZ"], case["N"], case["N"], device=DEV)}
        if k == "cone":
            s["weight"] = ufob.ConeBeamProjectionWeightTask(**_cone_weight(case))
            s["filter"] = ufob.FilterTask(**_fft_props(case["W"]))
            s["filtered"] = torch.empty_like(s["proj"])
        return s
    if k == "batch":
        jobs = []
        for i, (W, P) in enumerate(_jobs(case)):
            jobs.append({"sino": _sinograms(seed * 1000 + i, 1, P, W, W / 2.0, n=10)[0],
                         "out": torch.empty(W, W, device=DEV)})
        return {"case": case, "batch": ufob.Batch(storage=STORAGE[case["storage"]]), "jobs": jobs}
    net = cnn.SparseViewNet(seed=1)
    net.set_state(cnn.PARAMS, _net_params(seed))
    noisy, clean = _slices(seed, case["B"], case["H"], case["W"])
    s = {"case": case, "net": net, "x": noisy, "y": clean}
    if k == "net":
        s["out"] = torch.empty_like(noisy)
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "fbp":
        out = s["out"][0] if case["Z"] == 1 else s["out"]
        s["fbp"].process(s["sino"] if case["Z"] > 1 else s["sino"][None], out=s["out"])
        return out
    if k == "host":
        return s["fbp"].process_host(s["sino"], out=s["out"])
    if k == "raw":
        return s["fbp"].process_projections(s["proj"], ffc=s["ffc"], dark=s["dark"], flat=s["flat"], out=s["out"])
    if k == "filter":
        return s["task"].process(s["sino"], dtype=STORAGE[case["storage"]], out=s["out"])
    if k == "cone":
        f = s["filter"].process_projections(s["proj"], cone=s["weight"], sinograms=False, out=s["filtered"])
        return s["task"].process(f, out=s["out"])
    if k in ("lamino", "sweep"):
        return s["task"].process(s["proj"], out=s["out"])
    if k == "batch":
        s["batch"].run(s["jobs"])
        return [j["out"] for j in s["jobs"]]
    if k == "net":
        return s["net"].forward(s["x"], out=s["out"])
    # training steps at the schedule's final learning rate, then the gradients a checkpoint or a monitor reads
    for _ in range(case["steps"]):
        loss = s["net"].train_step(s["x"], s["y"], 1e-5)
    return {"loss": loss, "grads": s["net"].get_state(cnn.GRADS)}


# ----------------------------------------------------------------------------------------- bounds

def _fft_flops(rows, N):
    return 5.0 * rows * N * math.log2(N)  # a real transform there and back


def work(case):
    """Each input read once, each output written once; 4 operations per voxel-angle update in parallel
    beam (two multiply-adds), 8 in the general geometry (bilinear sample and weight)."""
    k = case["kind"]
    if k in ("fbp", "host", "raw", "filter"):
        Z, P, W = case["Z"], case["P"], case["W"]
        fl = _fft_flops(Z * P, _pow2(W))
        if k == "filter":
            return {"bytes": Z * P * W * (8.0 if case["storage"] == "f32" else 6.0), "flops": fl}
        by = 4.0 * Z * P * W + 4.0 * Z * W * W + (8.0 * Z * W if k == "raw" else 0.0)
        return {"bytes": by, "flops": fl + 4.0 * Z * W * W * P}
    if k in ("cone", "lamino", "sweep"):
        P, H, W, N, NZ = (case[c] for c in ("P", "H", "W", "N", "NZ"))
        fl = 8.0 * N * N * NZ * P + (_fft_flops(P * H, _pow2(W)) if k == "cone" else 0.0)
        return {"bytes": 4.0 * P * H * W + 4.0 * N * N * NZ, "flops": fl}
    if k == "batch":
        js = _jobs(case)
        return {"bytes": sum(4.0 * W * P + 4.0 * W * W for W, P in js),
                "flops": sum(_fft_flops(P, _pow2(W)) + 4.0 * W * W * P for W, P in js)}
    B, H, W = case["B"], case["H"], case["W"]
    px, conv = B * H * W / 16.0, 0.0
    for (ci, co, _), level in zip(LAYERS, (0, 1, 2, 3, 3, 2, 1, 0)):
        conv += 18.0 * ci * co * px / 4 ** level
    n = sum(co * 9 * ci + co for ci, co, _ in LAYERS)
    if k == "net":
        return {"bytes": 8.0 * B * H * W + 4.0 * n, "flops": conv}
    return {"bytes": case["steps"] * (8.0 * B * H * W + 28.0 * n), "flops": case["steps"] * 3.0 * conv}


def tolerance(case):
    """About four times the largest distance from exact() measured over listed and drawn cases."""
    k = case["kind"]
    if k == "net":
        return {"rel": 1.4e-2}  # BF16 weights and activations through eight layers
    if k == "train":
        return {"rel": 2e-2}  # the same and the gradients back
    if k == "filter":
        return {"rel": 3e-6} if case["storage"] == "f32" else {"rel": 1.5e-3}
    if k in ("cone", "lamino", "sweep"):
        return {"rel": 1.5e-5}
    if case["storage"] == "f16":
        return {"rel": 3e-3}  # filtered sinograms rounded to 11 bits, as many in the weights
    return {"rel": 1.5e-4}  # 32-bit detector coordinates on noisy data, sums over up to 1800 angles


# ------------------------------------------------------------------------------------------ exact

def _ramp(N, device):
    """The ramp filter built from its real-space kernel (the filter task's default), 32-bit kernel values."""
    h = np.zeros(N, dtype=np.float32)
    h[0] = 0.25
    k = np.arange(1, N // 2 + 1)
    h[1:N // 2 + 1] = np.where(k % 2 == 1, -1.0 / (k * k * math.pi * math.pi), 0.0)
    h[N // 2 + 1:] = h[1:N // 2][::-1]
    z = np.fft.fft(h.astype(np.float64) * (1 + 1j))
    return torch.from_numpy(z.real.copy()).to(device), torch.from_numpy(z.imag.copy()).to(device)


def _filtered(rows, W):
    """`fft ! filter ! ifft` of double rows along the last axis."""
    N = _pow2(W)
    cr, ci = _ramp(N, rows.device)
    X = torch.fft.fft(rows, n=N, dim=-1)
    return torch.fft.ifft(torch.complex(X.real * cr, X.imag * ci), dim=-1).real[..., :W].contiguous()


def _backprojected(sino, axis):
    """`backproject` of filtered sinograms [Z, P, W] in double onto W x W slices."""
    Z, P, W = sino.shape
    axis = float(np.float32(axis))
    c = torch.arange(W, device=sino.device, dtype=torch.float64) + 0.5 - axis
    out = torch.zeros(Z, W * W, device=sino.device, dtype=torch.float64)
    pad = torch.zeros(Z, P, W + 2, device=sino.device, dtype=torch.float64)
    pad[..., 1:W + 1] = sino
    for p in range(P):
        s, co = math.sin(p * math.pi / P), math.cos(p * math.pi / P)
        h = (c[:, None] * s + c[None, :] * co).reshape(-1) + (axis - 0.5)
        f = torch.floor(h)
        w = h - f
        i = f.to(torch.int64) + 1
        row = pad[:, p]
        a = torch.index_select(row, 1, i.clamp(0, W + 1))
        b = torch.index_select(row, 1, (i + 1).clamp(0, W + 1))
        out += torch.lerp(a, b, w)
    return (out * (math.pi / P)).reshape(Z, W, W)


def _exact_fbp(sino, W, axis):
    """Filter and backproject [Z, P, W] (any float type) by groups of slices."""
    out = []
    for z in range(0, sino.shape[0], 8):
        out.append(_backprojected(_filtered(sino[z:z + 8].double(), W), axis))
    return torch.cat(out)


def _exact_general(case, proj):
    """General backprojection of double projections [P, H, W] (bilinear samples, zero outside)."""
    P, H, W, N, NZ = (case[c] for c in ("P", "H", "W", "N", "NZ"))
    pr = _gbp_props(case)
    dev, f64 = proj.device, torch.float64
    cx, cz = pr["center-position-x"], pr["center-position-z"]
    x = (torch.arange(N, device=dev, dtype=f64) - N / 2.0)[None, None, :]
    y = (torch.arange(N, device=dev, dtype=f64) - N / 2.0)[None, :, None]
    start, _, step = pr["region"]
    sv = (start + torch.arange(NZ, device=dev, dtype=f64) * step)[:, None, None]
    z = torch.full_like(sv, pr["z"]) if case["kind"] == "sweep" else sv
    out = torch.zeros(NZ, N, N, device=dev, dtype=f64)
    pad = torch.zeros(H + 2, W + 2, device=dev, dtype=f64)
    for i in range(P):
        a = i / P * 2 * math.pi
        s, c = math.sin(a), math.cos(a)
        wgt = 1.0
        if case["kind"] == "cone":
            sy, dy = pr["source-position-y"], pr["detector-position-y"]
            m = -sy / (dy - sy)
            vx, vy, vz = m * (c * x - s * y), m * (s * x + c * y), m * z
            t = (dy - sy) / (vy - sy)
            u, v, wgt = t * vx + cx, t * vz + cz, ((sy - dy) / (sy - vy)) ** 2
        elif case["kind"] == "lamino":
            al = pr["axis-angle-x"]
            u, v = c * x - s * y + cx, math.sin(al) * (s * x + c * y) + math.cos(al) * z + cz
        else:
            u, v = c * x - s * y + sv, z + cz
        u, v = (u - 0.5).expand(NZ, N, N), (v - 0.5).expand(NZ, N, N)
        fu, fv = torch.floor(u), torch.floor(v)
        pad[1:H + 1, 1:W + 1] = proj[i]
        iu, iv = fu.to(torch.int64) + 1, fv.to(torch.int64) + 1
        u0, u1 = iu.clamp(0, W + 1), (iu + 1).clamp(0, W + 1)
        v0, v1 = iv.clamp(0, H + 1) * (W + 2), (iv + 1).clamp(0, H + 1) * (W + 2)
        q, fu, fv = pad.reshape(-1), u - fu, v - fv
        top = torch.lerp(q[v0 + u0], q[v0 + u1], fu)
        out += wgt * torch.lerp(top, torch.lerp(q[v1 + u0], q[v1 + u1], fu), fv)
    return out * (2 * math.pi / P)


def _exact_net(params, x, scale=1.0):
    """The correction network in double from the 32-bit parameters: prediction for [B, H, W]."""
    F = torch.nn.functional
    B, H, W = x.shape
    off, layers = 0, []
    for ci, co, _ in LAYERS:
        w = params[off:off + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        off += co * 9 * ci
        layers.append((w, params[off:off + co]))
        off += co

    def conv(i, t):
        # a 3x3 convolution as nine products of matrices
        w, b = layers[i]
        n, ci, h, wd = t.shape
        tp = F.pad(t, (1, 1, 1, 1))
        out = b[None, :, None, None]
        for dy in range(3):
            for dx in range(3):
                out = out + torch.einsum("oc,nchw->nohw", w[:, :, dy, dx], tp[:, :, dy:dy + h, dx:dx + wd])
        return torch.relu(out) if LAYERS[i][2] else out

    def up(t):
        return t.repeat_interleave(2, 2).repeat_interleave(2, 3)

    a = F.pixel_unshuffle((x / scale)[:, None], 4)
    e1 = conv(0, a)
    e2 = conv(1, F.avg_pool2d(e1, 2))
    e3 = conv(2, F.avg_pool2d(e2, 2))
    d3 = conv(4, conv(3, F.avg_pool2d(e3, 2)))
    d2 = conv(5, up(d3) + e3)
    d1 = conv(6, up(d2) + e2)
    return x + scale * F.pixel_shuffle(conv(7, up(d1) + e1), 4)[:, 0]


def _inputs(s):
    """The inputs of a prepared state without its handles and buffers."""
    keep = {n: s[n] for n in ("sino", "proj", "dark", "flat", "x", "y") if n in s}
    if "jobs" in s:
        keep["sinos"] = [j["sino"] for j in s["jobs"]]
    return keep


def exact(case, seed):
    k = case["kind"]
    w = work(case)
    if w["flops"] > 2.0e12 and k in ("fbp", "host", "raw"):
        return None  # half a minute and more in 64 bits
    d = _inputs(prepare(case, seed))
    if k in ("fbp", "host"):
        sino = d["sino"].to(DEV)
        out = _exact_fbp(sino if sino.dim() == 3 else sino[None], case["W"], case["axis"])
        return out[0] if case["Z"] == 1 and k == "fbp" else out
    if k == "raw":
        dark, flat = d["dark"].double(), d["flat"].double()
        sino = torch.log((flat - dark) / (d["proj"].double() - dark)).transpose(0, 1)
        return _exact_fbp(sino, case["W"], case["axis"])
    if k == "filter":
        return torch.cat([_filtered(d["sino"][z:z + 8].double(), case["W"]) for z in range(0, case["Z"], 8)])
    if k == "cone":
        cw, W, H = _cone_weight(case), case["W"], case["H"]
        sd = cw["source_distance"]
        mag = sd / (sd + cw["detector_distance"])
        u = (torch.arange(W, device=DEV, dtype=torch.float64)[None, :] - cw["center_position_x"] + 0.5) * mag
        v = (torch.arange(H, device=DEV, dtype=torch.float64)[:, None] - cw["center_position_z"] + 0.5) * mag
        wgt = sd / torch.sqrt(sd * sd + u * u + v * v)
        f = torch.cat([_filtered(d["proj"][i:i + 32].double() * wgt, W) for i in range(0, case["P"], 32)])
        return _exact_general(case, f)
    if k in ("lamino", "sweep"):
        return _exact_general(case, d["proj"].double())
    if k == "batch":
        return [_exact_fbp(q[None], q.shape[-1], q.shape[-1] / 2.0)[0] for q in d["sinos"]]
    params = torch.from_numpy(_net_params(seed)).to(DEV).double()
    if k == "net":
        return torch.cat([_exact_net(params, d["x"][i:i + 4].double()) for i in range(0, case["B"], 4)])
    if case["steps"] > 1:
        return None  # later steps see updated weights
    params.requires_grad_(True)
    n, loss = d["x"].numel(), 0.0
    for i in range(0, case["B"], 4):
        part = ((_exact_net(params, d["x"][i:i + 4].double()) - d["y"][i:i + 4].double()) ** 2).sum() / n
        part.backward()
        loss += float(part.detach())
    return {"loss": loss, "grads": params.grad}
