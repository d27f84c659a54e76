"""Performance cases: the reconstructions a user of libmtr runs, through the
public Python binding (mtr.py), over the sizes, geometries, precisions and
entry points that the library is used with.

A case names an entry point and one or more tilt series.  A series is written
"X:Y:Z:PX:PY:N:phi/phi/..": volume and detector size, number of tilts over
+-60 degrees, and the in-plane angle of each tilt axis.  `maps` says how the
linear maps were obtained:
    plain    an ideal tilt series (the benchmark's and the tests' geometry)
    aligned  per-view 2-D alignment transforms (rotation, magnification,
             shift) turned into maps of the raw views, as IMOD .tlt/.xf users
             do; detector y then depends weakly on Z
    leaning  a tilt axis that leans out of the XY plane (y-maps with a Z term)
"""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
PKG = ROOT / "multi-tilt-reconstuction_gb300"
if str(PKG) not in sys.path:
    sys.path.insert(0, str(PKG))

import mtr  # noqa: E402
import phantom  # noqa: E402

PRECISIONS = {"fp32": mtr.PREC_FP32, "bf16": mtr.PREC_MIXED_BF16, "fp16": mtr.PREC_MIXED_FP16}


def _case(name, entry, series, precision="fp32", maps="plain", noise="gaussian", outer=1, inner=10, sirt_step=0.5,
          mace_step=0.7, graph=False):
    return dict(name=name, entry=entry, series=series, precision=precision, maps=maps, noise=noise, outer=outer,
                inner=inner, sirt_step=sirt_step, mace_step=mace_step, graph=graph)


def listed() -> list[dict]:
    return [
        # the smallest benchmark configuration: one axis, preview size, one replayed graph; launches and latency count
        _case("single_128", "run", "128:128:32:128:128:61:0", graph=True),
        # an ordinary single-axis tilt series in the recommended mixed precision
        _case("single_256_fp16", "run", "256:256:64:256:256:61:0", "fp16", inner=8),
        # dual-axis tomography (two orthogonal series), sizes no multiple of any tile, low-dose counts
        _case("dual_ragged", "run", "301:277:61:340:330:41:0/90", noise="poisson", outer=2, inner=4),
        # three oblique axes, FP32, a MACE run of ordinary size
        _case("tri_256", "run", "256:256:64:256:256:61:0/60/120", outer=2, inner=4, mace_step=0.8),
        # the headline benchmark configuration: a whole mixed-precision MACE run
        _case("tri_512_fp16", "run", "512:512:128:512:512:61:0/60/120", "fp16", outer=2, mace_step=0.8, graph=True),
        # a real data set's geometry: every view has its own alignment transform
        _case("aligned_320", "run", "320:300:72:344:322:51:12", maps="aligned", inner=5),
        # a leaning tilt axis, two oblique axes, BF16 volume copies
        _case("leaning_192_bf16", "run", "192:160:48:224:210:41:30/135", "bf16", "leaning", inner=5),
        # the reference-shaped single-axis entries on host buffers: weighted back-projection of a slab ...
        _case("wbp_slab", "wbp", "400:384:40:420:400:61:90"),
        # ... and SIRT iterations on a slab, in place
        _case("sirt_slab", "sirt", "320:288:48:336:300:45:60", inner=6),
        # one call from host projections to host volume (set-up, upload, run, download)
        _case("reconstruct_host", "reconstruct", "256:320:64:300:340:61:0/45", outer=2, inner=3),
        # many uneven series as one batch
        _case("batch_uneven", "batch", "128:120:40:136:128:41:0;200:176:64:216:212:61:0/90;96:100:32:128:128:81:45;"
              "310:256:48:320:300:51:60/150", "fp16", outer=1, inner=5, graph=True),
        # the largest: four axes, fine tilts, low dose
        _case("quad_1024", "run", "1024:1024:192:1024:1024:121:0/45/90/135", noise="poisson", outer=1, inner=2),
    ]


def _cost(case: dict) -> float:
    """Voxel-angle visits of one pass, and a floor for its fixed parts."""
    its = 2 * case["outer"] * case["inner"] if case["entry"] != "wbp" else 0
    return sum(s["X"] * s["Y"] * s["Z"] * s["N"] * len(s["phis"]) * (1 + its) for s in _series(case))


def draw(rng) -> dict:
    """A case of the same ranges: any entry point, lateral sizes 40-1100, depths 6-200, 9-121 tilts."""
    def log_int(lo, hi):
        return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))

    limit = 0.7 * max(_cost(c) for c in listed())
    while True:
        entry = rng.choice(["run", "run", "run", "run", "wbp", "sirt", "reconstruct", "batch"])
        specs = []
        for _ in range(rng.randint(2, 4) if entry == "batch" else 1):
            x = log_int(40, 1100 if entry == "run" else 420)
            y = max(40, int(x * rng.uniform(0.75, 1.25)))
            z = min(log_int(6, 200), max(6, x // 2))
            # (the detector covers the volume seen along each orthogonal axis; the corners of oblique axes fall off it)
            px, py = (int(max(x, y) * rng.uniform(1.0, 1.15)) + 6 for _ in range(2))
            phis = rng.choice(["0", "90", "0/90", "60", "0/60/120", "0/45/90/135", "17.5", "30/120", "89.3/1.1"])
            if entry in ("wbp", "sirt"):
                phis = phis.split("/")[-1]
            specs.append(f"{x}:{y}:{z}:{px}:{py}:{rng.randint(4, 60) * 2 + 1}:{phis}")
        single = entry in ("wbp", "sirt")
        case = _case("", entry, ";".join(specs), "fp32" if single else rng.choice(["fp32", "fp32", "fp16", "bf16"]),
                     rng.choice(["plain", "plain", "plain", "aligned", "leaning"]),
                     rng.choice(["gaussian", "poisson"]), 1 if single else rng.randint(1, 2), rng.randint(1, 8),
                     rng.choice([0.3, 0.5, 0.8]), rng.choice([0.5, 0.7, 0.8]), rng.random() < 0.3)
        del case["name"]
        if _cost(case) <= limit:
            return case


# ---- inputs -----------------------------------------------------------------------------
def _series(case: dict) -> list[dict]:
    out = []
    for text in case["series"].split(";"):
        x, y, z, px, py, n, phis = text.split(":")
        out.append(dict(X=int(x), Y=int(y), Z=int(z), PX=int(px), PY=int(py), N=int(n),
                        phis=[float(p) for p in phis.split("/")]))
    return out


def _maps(s: dict, vol, phi: float, kind: str, rng) -> tuple[np.ndarray, np.ndarray]:
    tilts = np.linspace(-60.0, 60.0, s["N"])
    if kind != "aligned":
        xc, yc = phantom.axis_maps(s["PX"], s["PY"], tilts, phi, vol)
        if kind == "leaning":
            yc[3::4] += 0.04
        return xc, yc
    n = s["N"]
    rot, mag = np.deg2rad(rng.normal(0.0, 0.4, n)), 1.0 + rng.normal(0.0, 0.004, n)
    xf = np.stack([mag * np.cos(rot), -mag * np.sin(rot), mag * np.sin(rot), mag * np.cos(rot),
                   rng.normal(0.0, 2.0, n), rng.normal(0.0, 2.0, n)], axis=1)
    return mtr.geometry_from_tilts(tilts, phi, s["PX"], s["PY"], vol, xf)


def _inputs(case: dict, seed: int) -> list[tuple]:
    """[(volume frame, [(x maps, y maps, projections on the GPU)])] of every series."""
    made = []
    for i, s in enumerate(_series(case)):
        rng = np.random.default_rng([seed, i])
        vol = mtr.VolumeSize.make(0, s["X"], 0, s["Y"], 0, s["Z"])
        ell = phantom.random_ellipsoids(rng, 12, vol)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed * 101 + i)
        # the microscope's geometry belongs to the case, what it saw to the seed
        geometry = np.random.default_rng([7, i])
        axes = []
        for phi in s["phis"]:
            xc, yc = _maps(s, vol, phi, case["maps"], geometry)
            proj = phantom.line_integrals_torch(ell, xc, yc, s["PX"], s["PY"], "cuda")
            top = max(float(proj.max()), 1e-6)
            if case["noise"] == "poisson":  # dose 50 per pixel, at most two attenuation lengths
                counts = torch.poisson(50.0 * torch.exp(-2.0 / top * proj), generator=gen)
                proj = -torch.log(torch.clamp(counts, min=1.0) / 50.0) * (top / 2.0)
            else:
                proj = proj + 0.03 * top * torch.randn(proj.shape, generator=gen, device="cuda")
            axes.append((xc, yc, proj.contiguous()))
        made.append((vol, axes))
    return made


# ---- what a program keeps, and one pass ----------------------------------------------------
_program: dict = {}


def _context() -> tuple:
    """The program's one library context, on a stream of its own."""
    if not _program:
        _program["stream"] = torch.cuda.Stream()
        _program["ctx"] = mtr.Context(torch.cuda.current_device())
        _program["ctx"].set_stream(_program["stream"].cuda_stream)
    return _program["ctx"], _program["stream"]


def _slab_start(shape: tuple, seed: int) -> np.ndarray:
    return np.random.default_rng([seed, 99]).random(shape, dtype=np.float32)


def prepare(case: dict, seed: int) -> dict:
    ctx, stream = _context()
    series = _inputs(case, seed)
    torch.cuda.synchronize()
    p = mtr.params(case["outer"], case["inner"], case["sirt_step"], case["mace_step"], PRECISIONS[case["precision"]],
                   mtr.FLAG_GRAPH if case["graph"] else 0)
    st = dict(case=case, ctx=ctx, stream=stream, p=p)
    if case["entry"] == "run":
        vol, axes = series[0]
        st["recon"] = mtr.Recon(ctx, [mtr.AxisData(*a) for a in axes], vol, p, mtr.MEM_DEVICE)
        st["out"] = torch.empty(vol.shape, dtype=torch.float32, device="cuda")
    elif case["entry"] == "batch":
        st["batch"] = mtr.Batch(ctx, [([mtr.AxisData(*a) for a in axes], vol) for vol, axes in series], p,
                                mtr.MEM_DEVICE)
        st["outs"] = [torch.empty(vol.shape, dtype=torch.float32, device="cuda") for vol, _ in series]
    else:  # the entries on host buffers
        vol, axes = series[0]
        st["vol"] = vol
        # projections as a loader leaves them: pinned host memory
        st["pinned"] = [d.cpu().pin_memory() for _, _, d in axes]
        st["axes"] = [mtr.AxisData(xc, yc, d.numpy()) for (xc, yc, _), d in zip(axes, st["pinned"])]
        if case["entry"] == "sirt":
            st["slab"] = _slab_start(vol.shape, seed)
    torch.cuda.synchronize()
    return st


def run(st: dict):
    case, ctx, stream = st["case"], st["ctx"], st["stream"]
    if case["entry"] == "reconstruct":
        return ctx.reconstruct(st["axes"], st["vol"], st["p"])
    if case["entry"] == "wbp":
        return ctx.wbp(st["axes"][0], st["vol"])
    if case["entry"] == "sirt":
        return ctx.sirt(st["axes"][0], st["vol"], st["slab"], case["inner"], case["sirt_step"])
    caller = torch.cuda.current_stream()
    stream.wait_stream(caller)
    if case["entry"] == "run":
        st["recon"].run()
        out = st["recon"].download(st["out"], mtr.MEM_DEVICE)
    else:
        st["batch"].run()
        out = [st["batch"].download(i, o, mtr.MEM_DEVICE) for i, o in enumerate(st["outs"])]
    caller.wait_stream(stream)
    return out


def work(case: dict) -> dict:
    """Each input read once and each output written once; four taps of a multiply and an add per voxel and angle for
    each back-projection and forward projection (WBP, then two per SIRT iteration)."""
    values = flops = 0.0
    for s in _series(case):
        v, k = float(s["X"] * s["Y"] * s["Z"]), len(s["phis"])
        values += k * s["PX"] * s["PY"] * s["N"] + v * (2 if case["entry"] == "sirt" else 1)
        its = 0 if case["entry"] == "wbp" else 2 * case["outer"] * case["inner"]
        flops += 8.0 * v * s["N"] * k * (its if case["entry"] == "sirt" else 1 + its)
    return {"bytes": 4.0 * values, "flops": flops}


# ---- the same computation in 64 bits, in plain torch ---------------------------------------
class _Axis64:
    """Projector pair of one axis in FP64: bilinear taps, dropped off the detector."""

    def __init__(self, vol, xc, yc, proj):
        self.vol, self.b = vol, proj.double()
        self.xc, self.yc = np.asarray(xc).reshape(-1, 4), np.asarray(yc).reshape(-1, 4)
        f64 = dict(dtype=torch.float64, device="cuda")
        self.X = torch.arange(vol.Xstart, vol.Xend, **f64)[None, None, :]
        self.Y = torch.arange(vol.Ystart, vol.Yend, **f64)[None, :, None]
        self.Z = torch.arange(vol.Zstart, vol.Zend, **f64)[:, None, None]

    def taps(self, a):
        """(pixel index, weight) of the four taps of every voxel at angle a; weight 0 off the detector."""
        _, py, px = self.b.shape
        x = self.xc[a, 0] - 1.0 + self.xc[a, 1] * self.X + self.xc[a, 2] * self.Y + self.xc[a, 3] * self.Z
        y = self.yc[a, 0] - 1.0 + self.yc[a, 1] * self.X + self.yc[a, 2] * self.Y + self.yc[a, 3] * self.Z
        x0, y0 = torch.floor(x), torch.floor(y)
        for dx in (0, 1):
            for dy in (0, 1):
                wx = (x - x0) if dx else 1.0 - (x - x0)
                wy = (y - y0) if dy else 1.0 - (y - y0)
                ix, iy = (x0 + dx).long(), (y0 + dy).long()
                ok = (ix >= 0) & (ix < px) & (iy >= 0) & (iy < py)
                yield torch.where(ok, iy * px + ix, 0), torch.where(ok, wx * wy, 0.0)

    def back(self, img):
        out = torch.zeros(self.vol.shape, dtype=torch.float64, device="cuda")
        for a in range(img.shape[0]):
            flat = img[a].reshape(-1)
            for i, w in self.taps(a):
                out += w * flat[i]
        return out

    def weights(self):
        out = torch.zeros(self.vol.shape, dtype=torch.float64, device="cuda")
        for a in range(self.b.shape[0]):
            for _, w in self.taps(a):
                out += w
        return out

    def forward(self, vol):
        out = torch.zeros_like(self.b)
        for a in range(self.b.shape[0]):
            flat = out[a].reshape(-1)
            for i, w in self.taps(a):
                flat.index_add_(0, i.reshape(-1), (w * vol).reshape(-1))
        return out


def _ratio(num, den, where_zero):
    return torch.where(den != 0, num / torch.where(den != 0, den, 1.0), where_zero)


def _wbp64(ax):
    ax.c = ax.weights()
    return _ratio(ax.back(ax.b), ax.c, torch.zeros_like(ax.c))


def _sirt64(ax, x, n, step):
    if not hasattr(ax, "rows"):
        ax.rows = ax.forward(torch.ones(ax.vol.shape, dtype=torch.float64, device="cuda"))
    for _ in range(n):
        s = ax.forward(x)
        g = ax.back(ax.b - _ratio(s, ax.rows, s))
        x = x + step * _ratio(g, ax.c, torch.zeros_like(g))
    return x


def exact(case: dict, seed: int):
    # (a pass of 64-bit taps in plain torch visits about 1.5e9 voxel-angles a second)
    if _cost(case) > 1.4e10:
        return None
    outs = []
    step, rho = float(np.float32(case["sirt_step"])), float(np.float32(case["mace_step"]))
    for vol, axes in _inputs(case, seed):
        ax = [_Axis64(vol, *a) for a in axes]
        if case["entry"] == "wbp":
            return _wbp64(ax[0]).cpu().numpy()
        if case["entry"] == "sirt":
            ax[0].c = ax[0].weights()
            start = torch.from_numpy(_slab_start(vol.shape, seed)).cuda().double()
            return _sirt64(ax[0], start, case["inner"], step).cpu().numpy()
        mean = sum(_wbp64(a) for a in ax)
        state = [mean.clone() for _ in ax]
        for _ in range(case["outer"]):
            for k, a in enumerate(ax):
                z = 2.0 * mean - state[k]
                v = _sirt64(a, z, case["inner"], step)
                state[k] = rho * (2.0 * v - z) + (1.0 - rho) * state[k]
            mean = sum(state) / len(ax)
        outs.append(mean)
    if case["entry"] == "reconstruct":
        return outs[0].cpu().numpy()
    return outs[0] if case["entry"] == "run" else outs
