"""Performance cases of the beamformer: what a station's program has it do.

Every case is one call (or the two calls that belong together) of the public
Python entry points on data as a telescope delivers it: packed int4 voltages
of Gaussian noise with a source in the field, geometric beam weights, and
the weights, workspaces and output buffers that such a program keeps from
block to block.  `listed` gives the fixed cases, `draw` others of the same
ranges, `prepare` a case's inputs and buffers on the GPU, `run` one pass,
`work` what a pass cannot do without, and `exact` its results in 64 bits
from plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from beamform_project_b200 import api, serve

F = 336                     # channels of a shard
C_LIGHT = 299_792_458.0
TWO_PI = 6.283185307179586476925286766559


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # The plain grid on a short block of a 32-element line: 13 MB of
        # voltage, where launches and latency count.
        dict(name="plain_grid_short", kind="tensor", ant=32, time=1024, beams=16, spectra=10, shards=1, codes=False),
        # The grid behind an upchannelizer (10 spectra per product, float
        # product) at the largest beam count; the last window is partial.
        dict(name="upchannelized_grid", kind="tensor", ant=64, time=8195, beams=128, spectra=10, shards=1,
             codes=False),
        # The largest array the interface takes, products quantized.
        dict(name="wide_array_grid", kind="tensor", ant=256, time=8192, beams=64, spectra=320, shards=1, codes=True),
        # An ordinary block of one shard on the checked grid, odd sizes.
        dict(name="checked_block", kind="checked", ant=64, time=2570, beams=72, spectra=320, shards=1, codes=True),
        # The full band: two shards, 128 beams, float and int8 products.
        dict(name="checked_full_band", kind="checked", ant=64, time=32768, beams=128, spectra=320, shards=2,
             codes=True),
        # The drop-in for the reference's pipeline at its default
        # dimensions: tiled weights, 320 spectra, int8 quantizer.
        dict(name="drop_in_integrated", kind="exact", ant=64, time=15360, beams=64, spectra=320, tiled=True,
             codes=True),
        # The drop-in's per-spectrum powers, an odd beam count.
        dict(name="drop_in_spectra", kind="exact", ant=64, time=1000, beams=37, spectra=0, tiled=False, codes=False),
        # A drifting source followed over a long run, one product per 1024
        # spectra: the voltage is read once from memory.
        dict(name="tracker_long", kind="tracker", ant=64, time=131072, spectra=1024, mode=1, intensity=False),
        # The tracker at the upchannelized cadence (new weights every 10
        # spectra) with its per-spectrum power.
        dict(name="tracker_short_windows", kind="tracker", ant=64, time=15360, spectra=10, mode=1, intensity=True),
        # Direction finding: block covariances and the Bartlett and Capon
        # scans of 16 blocks on 1801 points.
        dict(name="doa_blocks", kind="doa", ant=64, block=4096, blocks=16, sub=8, points=1801),
        # The adaptive tracker: per window a coarse-to-fine search, then
        # the beam along the estimate.
        dict(name="doa_track", kind="track", ant=64, block=256, blocks=32, sub=8, capon=True, grid=16, levels=2,
             intensity=True),
        # The server: a mix of grid and tracker jobs through their life,
        # results read back.
        dict(name="served_mix", kind="served", jobs=8, windows=8, pick=26),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tensor", "tensor", "checked", "checked", "exact", "exact", "tracker", "tracker", "doa",
                       "track", "served"])
    if kind == "tensor":
        return dict(kind=kind, ant=rng.choice([32, 64, 64, 128, 256]), time=_log(rng, 320, 8192),
                    beams=rng.randint(1, 128), spectra=rng.choice([10, 10, 16, 64, 320]), shards=rng.choice([1, 2]),
                    codes=rng.random() < 0.5)
    if kind == "checked":
        return dict(kind=kind, ant=64, time=_log(rng, 640, 32768), beams=rng.randint(8, 128),
                    spectra=rng.choice([64, 128, 320, 320, 640]), shards=rng.choice([1, 2]), codes=True)
    if kind == "exact":
        ant = rng.choice([32, 64, 64, 128, 256])
        spectra = rng.choice([0, 10, 320, 320])
        return dict(kind=kind, ant=ant, time=_log(rng, 64, 8192 * 64 // ant), beams=rng.randint(1, 64),
                    spectra=spectra, tiled=rng.random() < 0.5, codes=spectra > 0 and rng.random() < 0.5)
    if kind == "tracker":
        ant = rng.choice([32, 64, 64, 128])
        return dict(kind=kind, ant=ant, time=_log(rng, 640, 65536 * 64 // ant),
                    spectra=rng.choice([10, 10, 100, 320, 1024]), mode=rng.choice([1, 1, 1, 0]),
                    intensity=rng.random() < 0.5)
    if kind == "doa":
        blocks = rng.randint(1, 16)
        return dict(kind=kind, ant=rng.choice([32, 64]), block=128 * _log(rng, 2, 32), blocks=blocks,
                    sub=rng.randint(4, 16), points=_log(rng, 181, 1801))
    if kind == "track":
        return dict(kind=kind, ant=rng.choice([32, 64]), block=128 * _log(rng, 1, 8), blocks=rng.randint(4, 32),
                    sub=rng.choice([8, 8, 12, 16]), capon=rng.random() < 0.5, grid=rng.choice([8, 12, 16, 24]),
                    levels=rng.randint(0, 3), intensity=rng.random() < 0.5)
    return dict(kind=kind, jobs=rng.randint(2, 8), windows=rng.randint(2, 8), pick=rng.randint(2, 1000000))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _positions(ant):
    """A line at half a wavelength of 600 MHz (32), a 2 x 32 grid at half a
    wavelength of 800 MHz (64), 0.6 m grids above."""
    pos = np.zeros((ant, 3), np.float32)
    for a in range(ant):
        if ant == 32:
            pos[a, 0] = a * 0.5 * C_LIGHT / 600e6
        elif ant == 64:
            pos[a, :2] = (a % 32) * 0.5 * C_LIGHT / 800e6, (a // 32) * 0.5 * C_LIGHT / 800e6
        else:
            pos[a, :2] = (a % 16) * 0.6, (a // 16) * 0.6
    return pos


def _frequencies(n):
    return (400e6 + np.arange(n) * (400e6 / max(1, n - 1))).astype(np.float32)


def _wave_numbers(freq):
    return TWO_PI * freq.astype(np.float64) / C_LIGHT


def _phases(pos, kw, dirs):
    """k (p . d) in FP64: [directions][channels][antennas]."""
    p, k, d = (torch.as_tensor(np.asarray(x, np.float64), device="cuda") for x in (pos, kw, dirs))
    return k[None, :, None] * (d @ p.T)[:, None, :]


def _unit(lm):
    lm = np.asarray(lm, np.float32)
    n = np.sqrt(np.float32(1) - (lm[:, 0] * lm[:, 0] + lm[:, 1] * lm[:, 1])).astype(np.float32)
    return np.concatenate([lm, n[:, None]], axis=1).astype(np.float32)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _pack(x):
    """complex64 -> bytes, low nibble real, high nibble imaginary."""
    q = torch.view_as_real(x).round_().clamp_(-8, 7).to(torch.int8)
    return (q[..., 0] & 15 | (q[..., 1] << 4)).view(torch.uint8)


def _voltage(seed, time, pos, kw, sources, sigma, step=None):
    """Packed voltages [time][channels][antennas]: noise of standard deviation
    sigma per component and, per source (direction at spectrum t, amplitude),
    a Gaussian waveform along exp(-i k p.d)."""
    g = _generator(seed)
    n_ch, ant = len(kw), len(pos)
    out = torch.empty((time, n_ch, ant), dtype=torch.uint8, device="cuda")
    step = step or max(1, (1 << 25) // (n_ch * ant))
    for t in range(0, time, step):
        n = min(step, time - t)
        x = torch.randn((n, n_ch, ant), dtype=torch.complex64, device="cuda", generator=g) * (sigma * math.sqrt(2.0))
        for direction, amplitude in sources:
            w = torch.randn((n, n_ch, 1), dtype=torch.complex64, device="cuda", generator=g) * amplitude
            ph = _phases(pos, kw, direction(t)[None])[0]
            x.addcmul_(w, torch.polar(torch.ones_like(ph), -ph).to(torch.complex64)[None])
        out[t:t + n] = _pack(x)
    return out


def _fixed(lm):
    d = _unit([lm])[0]
    return lambda t: d


def _weights(pos, kw, dirs, shards):
    """complex64 [shard][beam][channel][antenna], as (re, im) float32."""
    ph = _phases(pos, kw, dirs)                                        # [B][shards F][A]
    w = torch.stack([ph.cos(), ph.sin()], -1).to(torch.float32)
    return w.reshape(len(dirs), shards, F, len(pos), 2).transpose(0, 1).contiguous()


def _grid_inputs(case, seed):
    shards = case.get("shards", 1)
    rng = np.random.default_rng(seed)
    pos, kw = _positions(case["ant"]), _wave_numbers(_frequencies(shards * F))
    dirs = _unit(rng.uniform(-0.5, 0.5, size=(case["beams"], 2)))
    source = _fixed(dirs[rng.integers(0, case["beams"]), :2])
    volt = torch.stack([_voltage(seed + 7919 * s, case["time"], pos, kw[s * F:(s + 1) * F],
                                 [(source, 2.5 * math.sqrt(2 * 5.0))], 2.5) for s in range(shards)])
    return volt, _weights(pos, kw, dirs, shards)


def _drift(case, seed):
    """Window directions [W][3] of a source that drifts by 0.02 over the run."""
    rng = np.random.default_rng(seed)
    l0, m0 = rng.uniform(-0.2, 0.2, 2).astype(np.float32)
    t = np.arange(0, case["time"], case["spectra"]).astype(np.float32)
    rate = np.float32(0.02 / case["time"])
    return _unit(np.stack([l0 + t * rate, m0 - t * rate], axis=1))


def _tracker_inputs(case, seed):
    pos, kw = _positions(case["ant"]), _wave_numbers(_frequencies(F))
    dirs = _drift(case, seed)
    volt = _voltage(seed, case["time"], pos, kw,
                    [(lambda t: dirs[t // case["spectra"]], 2.0 * math.sqrt(2 * 3.0))], 2.0, step=1000)
    return volt, pos, kw, dirs


def _doa_inputs(case, seed):
    pos, kw = _positions(case["ant"]), _wave_numbers(_frequencies(2 * F)[:F])
    rng = np.random.default_rng(seed)
    l, m = rng.uniform(-0.12, 0.12, 2)
    far = _fixed((rng.uniform(0.4, 0.6), 0.0))
    volt = _voltage(seed, case["block"] * case["blocks"], pos, kw,
                    [(_fixed((l, m if case["kind"] == "track" else 0.0)), 2.0 * math.sqrt(2 * 2.0)), (far, 1.5)], 2.0)
    return volt, pos, kw


POOL, WINDOW, MAX_SHARDS = 2560, 320, 2


def _served_jobs(case):
    """The mix: antennas, shards, grid beams or tracker sources, integration."""
    rng = np.random.default_rng(case["pick"])
    jobs = []
    for i in range(case["jobs"]):
        ant, shards, spectra = int(rng.choice([32, 64])), int(rng.integers(1, MAX_SHARDS + 1)), int(rng.choice([10, 320]))
        n = case["windows"] * WINDOW
        offset = int(rng.integers(0, POOL // WINDOW)) * WINDOW
        pos, freq = serve.array_positions(ant), _frequencies(shards * F)
        if i % 2 == 0:
            dirs = _unit(rng.uniform(-0.3, 0.3, size=(int(rng.choice([1, 8, 32, 128])), 2)))
            jobs.append(serve.JobSpec(serve.GRID, ant, shards, len(dirs), n, spectra, pos, freq, directions=dirs,
                                      pool_offset=offset))
        else:
            tr = np.zeros((int(rng.integers(1, 17)), 4), np.float32)
            tr[:, :2] = rng.uniform(-0.3, 0.3, size=(len(tr), 2))
            tr[:, 2:] = rng.uniform(-0.02, 0.02, size=(len(tr), 2)) / n
            jobs.append(serve.JobSpec(serve.TRACKER, ant, shards, len(tr), n, spectra, pos, freq, trajectories=tr,
                                      pool_offset=offset))
    return jobs


def _served_pool(seed, ant):
    kw = _wave_numbers(_frequencies(MAX_SHARDS * F))
    return _voltage(seed + ant, POOL, _positions(ant), kw, [(_fixed((0.1, -0.05)), 2.0)], 2.0)


# --------------------------------------------------------------------------
# prepare and run
# --------------------------------------------------------------------------

def _empty(n, dtype):
    return torch.empty(int(n), dtype=dtype, device="cuda")


def _product_buffers(s, dims, windows, shards, codes):
    n = shards * windows * dims.n_freq * dims.n_beams
    s["out"] = _empty(n, torch.float32)
    s["codes"] = s["params"] = None
    if codes:
        s["qdims"] = api.Dimensions(windows, dims.n_freq, dims.n_ant, dims.n_beams)
        s["codes"] = _empty(n, torch.int8)
        s["params"] = _empty(2 * shards * api.quantization_parameter_count(s["qdims"]), torch.float32)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("tensor", "checked", "exact"):
        shards, spectra = case.get("shards", 1), case["spectra"]
        d = s["dims"] = api.Dimensions(case["time"], F, case["ant"], case["beams"])
        s["volt"], w = _grid_inputs(case, seed)
        windows = api.integrated_time_count(d.n_time, spectra) if spectra else d.n_time
        _product_buffers(s, d, windows, shards, case["codes"])
        if kind == "tensor":
            s["weights"] = _empty(api.split_weight_bytes(d, shards), torch.uint8)
            api.prepare_split_weights(None, w, s["weights"], d, shards)
        elif kind == "checked":
            s["weights"] = _empty(api.auto_weight_bytes(d, shards), torch.uint8)
            api.prepare_auto_weights(None, w, s["weights"], d, shards)
            s["work"] = torch.zeros(max(256, api.grid_auto_workspace_bytes(d, spectra, shards)), dtype=torch.uint8,
                                    device="cuda")
        elif case["tiled"]:
            tiles = -(-d.n_beams // 32)
            t = torch.zeros((F, tiles, d.n_ant, 32, 2), dtype=torch.float32, device="cuda")
            for b in range(d.n_beams):
                t[:, b // 32, :, b % 32] = w[0, b]
            s["weights"] = t
        else:
            s["weights"] = w
    elif kind == "tracker":
        s["volt"], pos, kw, dirs = _tracker_inputs(case, seed)
        s["dims"] = api.Dimensions(case["time"], F, case["ant"], 1)
        s["pos"], s["kw"], s["dirs"] = (torch.from_numpy(x).cuda() for x in (pos, kw, dirs))
        s["out"] = _empty(len(dirs) * F, torch.float32)
        s["intensity"] = _empty(case["time"] * F, torch.float32) if case["intensity"] else None
    elif kind == "doa":
        s["volt"], pos, kw = _doa_inputs(case, seed)
        d = s["dims"] = api.Dimensions(case["block"] * case["blocks"], F, case["ant"], 1)
        s["pos"], s["kw"] = torch.from_numpy(pos[:case["sub"]].copy()).cuda(), torch.from_numpy(kw).cuda()
        s["cov"] = _empty(case["blocks"] * F * case["ant"] ** 2 * 2, torch.int32)
        s["bartlett"], s["capon"] = (_empty(case["blocks"] * case["points"], torch.float64) for _ in range(2))
        s["peaks"] = _empty(2 * case["blocks"], torch.float64)
        s["work"] = _empty(api.doa_workspace_bytes(d, case["block"], case["sub"]), torch.uint8)
    elif kind == "track":
        s["volt"], pos, kw = _doa_inputs(case, seed)
        d = s["dims"] = api.Dimensions(case["block"] * case["blocks"], F, case["ant"], 1)
        s["config"] = api.doa_track_config(case["block"], subarray=case["sub"], capon=case["capon"],
                                           grid=case["grid"], levels=case["levels"], fov_l=0.15, fov_m=0.15,
                                           forgetting=0.9, diag_load=1e-3)
        s["pos"], s["kw"] = torch.from_numpy(pos).cuda(), torch.from_numpy(kw).cuda()
        s["dirs"] = _empty(3 * case["blocks"], torch.float32)
        s["intensity"] = _empty(d.n_time * F, torch.float32) if case["intensity"] else None
        s["work"] = _empty(api.doa_track_workspace_bytes(d, s["config"]), torch.uint8)
    else:
        s["jobs"] = _served_jobs(case)
        s["server"] = serve.Server(2 << 30, max_jobs=16, window_spectra=WINDOW, pool_spectra=POOL,
                                   shard_channels=F, max_shards=MAX_SHARDS)
        for ant in (32, 64):
            s["server"].pool(ant).copy_(_served_pool(seed, ant))
        torch.cuda.synchronize()
    return s


def _doa_scan_grid(case):
    return -0.9, 1.8 / (case["points"] - 1)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "tensor":
        api.grid_tensor_integrated(None, s["volt"], s["weights"], s["out"], s["codes"], s["params"], s["dims"],
                                   case["spectra"], case["shards"])
        return [s["out"], s["codes"], s["params"]]
    if kind == "checked":
        api.grid_auto_integrated(None, s["volt"], s["weights"], s["out"], s["codes"], s["params"], s["work"],
                                 s["dims"], case["spectra"], case["shards"])
        return [s["out"], s["codes"], s["params"]]
    if kind == "exact":
        kernel = api.CudaBeamformerKernel.Tiled if case["tiled"] else api.CudaBeamformerKernel.Direct
        if not case["spectra"]:
            api.launch_packed_beamformer(kernel, None, s["volt"], s["weights"], s["out"], s["dims"])
            return [s["out"], None, None]
        api.launch_packed_integrated_beamformer(kernel, None, s["volt"], s["weights"], s["out"], s["dims"],
                                                case["spectra"])
        if case["codes"]:
            api.launch_quantize_integrated_intensity(None, s["out"], s["codes"], s["params"], s["qdims"])
        return [s["out"], s["codes"], s["params"]]
    if kind == "tracker":
        api.tracker(None, case["mode"], s["volt"], s["pos"], s["kw"], s["dirs"], s["intensity"], s["out"], s["dims"],
                    case["spectra"])
        return [s["out"], s["intensity"]]
    if kind == "doa":
        first, step = _doa_scan_grid(case)
        api.doa_covariance_i32(None, s["volt"], s["cov"], s["dims"], case["block"])
        api.doa_scan(None, s["cov"], s["pos"], s["kw"], s["dims"], case["block"], case["sub"], 0.9, 1e-3, first, step,
                     case["points"], 0.0, s["bartlett"], s["capon"], s["peaks"], s["work"])
        return [s["cov"], s["bartlett"], s["capon"], s["peaks"]]
    if kind == "track":
        api.doa_track(None, s["volt"], s["pos"], s["kw"], s["dims"], s["config"], s["dirs"], s["intensity"], s["work"])
        return [s["dirs"], s["intensity"]]
    server = s["server"]
    ids = [server.submit(job) for job in s["jobs"]]
    while server.step():
        pass
    server.sync()
    outs = []
    for jid in ids:
        outs.append(list(server.result(jid, floats=False)))
        server.release(jid)
    return outs


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def _grid_work(ant, time, beams, spectra, shards, codes):
    windows = -(-time // spectra) if spectra else time
    n_out = shards * windows * F * beams
    return (shards * F * ant * (time + 8 * beams) + n_out * (5 if codes else 4),
            shards * time * F * beams * (8 * ant + 3))


def work(case):
    kind = case["kind"]
    if kind in ("tensor", "checked", "exact"):
        b, f = _grid_work(case["ant"], case["time"], case["beams"], case["spectra"], case.get("shards", 1),
                          case["codes"])
    elif kind == "tracker":
        windows = -(-case["time"] // case["spectra"])
        b = F * (case["time"] * case["ant"] + 4 * windows + (4 * case["time"] if case["intensity"] else 0))
        f = case["time"] * F * (8 * case["ant"] + 3)
    elif kind == "doa":
        ant, n = case["ant"], case["block"] * case["blocks"]
        b = n * F * ant + 8 * case["blocks"] * F * ant * ant + 16 * case["blocks"] * case["points"]
        f = 4 * n * F * ant * (ant + 1) + 16 * case["blocks"] * F * case["points"] * (case["sub"] - 1)
    elif kind == "track":
        ant, n = case["ant"], case["block"] * case["blocks"]
        points = case["grid"] ** 2 + 9 * case["levels"]
        b = F * (n * ant + (4 * n if case["intensity"] else 0)) + 12 * case["blocks"]
        f = 4 * n * F * ant * (ant + 1) + 4 * case["blocks"] * F * points * case["sub"] ** 2 \
            + (n * F * (8 * ant + 3) if case["intensity"] else 0)
    else:
        b = f = 0
        for j in _served_jobs(case):
            if j.kind == serve.GRID:
                x, y = _grid_work(j.n_ant, j.n_spectra, j.n_beams, j.integration_spectra, j.n_shards, True)
            else:
                x = j.n_shards * F * (j.n_spectra * j.n_ant
                                      + 4 * j.n_beams * (j.n_spectra // j.integration_spectra))
                y = j.n_shards * F * j.n_spectra * j.n_beams * (8 * j.n_ant + 3)
            b, f = b + x, f + y
    return {"bytes": float(b), "flops": float(f)}


# --------------------------------------------------------------------------
# the results in 64 bits
# --------------------------------------------------------------------------

def _complex(v):
    """bytes -> complex128"""
    s = v.view(torch.int8)
    return torch.complex(((s << 4) >> 4).double(), (s >> 4).double())


def _window_sums(p, spectra):
    """[time][...] -> [windows][...], the last window as long as it is."""
    time = p.shape[0]
    windows = -(-time // spectra)
    pad = torch.zeros((windows * spectra - time,) + p.shape[1:], dtype=p.dtype, device=p.device)
    return torch.cat([p, pad]).reshape((windows, spectra) + p.shape[1:]).sum(1)


def _grid_powers(volt, w, spectra):
    """[time][channels][antennas], [beams][channels][antennas] complex -> [windows][channels][beams]."""
    out = []
    for f in range(volt.shape[1]):
        p = (_complex(volt[:, f]) @ w[:, f].T).abs().square()
        out.append(_window_sums(p, spectra) if spectra else p)
    return torch.stack(out, 1)


def _chunk_params(x):
    """(offset, scale) of every 1 x 16 x 16 chunk of [windows][channels][beams]."""
    windows, n_ch, beams = x.shape
    pad = (0, -beams % 16, 0, -n_ch % 16)

    def chunks(fill):
        y = torch.nn.functional.pad(x, pad, value=fill)
        return y.reshape(windows, y.shape[1] // 16, 16, y.shape[2] // 16, 16)

    lo, hi = chunks(math.inf).amin((2, 4)), chunks(-math.inf).amax((2, 4))
    scale = (hi - lo) / 255.0
    return torch.stack([lo + 127.5 * scale, scale], -1)


def _tracker_powers(volt, pos, kw, dirs, spectra):
    """[time][channels] along the window directions."""
    p = torch.empty(volt.shape[:2], dtype=torch.float64, device="cuda")
    group = max(1, 512 // spectra)
    for w0 in range(0, len(dirs), group):
        ph = _phases(pos, kw, dirs[w0:w0 + group])
        w = torch.polar(torch.ones_like(ph), ph)
        t0, t1 = w0 * spectra, min(volt.shape[0], (w0 + group) * spectra)
        which = torch.arange(t1 - t0, device="cuda") // spectra
        for a in range(t0, t1, 512):
            b = min(t1, a + 512)
            wt = w[which[a - t0:b - t0]] if len(ph) > 1 else w
            p[a:b] = (_complex(volt[a:b]) * wt).sum(-1).abs().square()
    return p


def _doa_spectra(case, volt, pos, kw):
    blocks, K, A, M = case["blocks"], case["block"], case["ant"], case["sub"]
    L = A - M + 1
    first, step = _doa_scan_grid(case)
    grid = first + torch.arange(case["points"], dtype=torch.float64, device="cuda") * step
    x = torch.as_tensor(pos[:M, 0].astype(np.float64), device="cuda")
    bart = torch.zeros((blocks, case["points"]), dtype=torch.float64, device="cuda")
    cap = torch.zeros_like(bart)
    for f in range(F):
        v = _complex(volt[:, f]).reshape(blocks, K, A)
        R = v.transpose(1, 2) @ v.conj() / K
        S = sum(R[:, i:i + M, i:i + M] for i in range(L)) / L
        if L > 1:
            S = (S + S.flip(1, 2).conj()) / 2
        eps = 1e-3 * torch.diagonal(S, dim1=1, dim2=2).real.sum(1) / M
        for b in range(1, blocks):
            S[b] = 0.9 * S[b - 1] + 0.1 * S[b]
            eps[b] = 0.9 * eps[b - 1] + 0.1 * eps[b]
        Q = torch.linalg.inv(S + eps[:, None, None] * torch.eye(M, dtype=torch.float64, device="cuda"))
        ph = -float(kw[f]) * grid[:, None] * x[None]
        a = torch.polar(torch.ones_like(ph), ph)
        bart += torch.einsum("nr,brc,nc->bn", a.conj(), S, a).real
        cap += 1.0 / torch.einsum("nr,brc,nc->bn", a.conj(), Q, a).real
    peaks = []
    for P in (bart, cap):
        i = P.argmax(1, keepdim=True)
        lo, mid, hi = (P.gather(1, (i + o).clamp(0, P.shape[1] - 1)) for o in (-1, 0, 1))
        den = lo - 2 * mid + hi
        off = torch.where(den < 0, (0.5 * (lo - hi) / den).clamp(-0.5, 0.5), torch.zeros_like(den))
        off = torch.where((i > 0) & (i + 1 < P.shape[1]), off, torch.zeros_like(off))
        peaks.append(first + (i + off) * step)
    return bart.reshape(-1), cap.reshape(-1), torch.cat(peaks, 1).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("tensor", "checked", "exact"):
        volt, w = _grid_inputs(case, seed)
        wc = torch.view_as_complex(w.double().contiguous())
        p = torch.stack([_grid_powers(volt[i], wc[i], case["spectra"]) for i in range(len(volt))])
        params = torch.cat([_chunk_params(x).reshape(-1) for x in p]) if case["codes"] else None
        return [p.reshape(-1), None, params]
    if kind == "tracker":
        volt, pos, kw, dirs = _tracker_inputs(case, seed)
        p = _tracker_powers(volt, pos, kw, dirs, case["spectra"])
        return [_window_sums(p, case["spectra"]).reshape(-1), p.reshape(-1) if case["intensity"] else None]
    if kind == "doa":
        volt, pos, kw = _doa_inputs(case, seed)
        return [None, *_doa_spectra(case, volt, pos, kw)]
    if kind == "track":
        return None     # a search: each direction hangs on decisions between neighbouring cells
    pools = {ant: _served_pool(seed, ant) for ant in (32, 64)}
    outs = []
    for j in _served_jobs(case):
        n_ch = j.n_shards * F
        rows = (j.pool_offset + torch.arange(j.n_spectra, device="cuda")) % POOL
        volt = pools[j.n_ant][rows][:, :n_ch].contiguous()
        kw = _wave_numbers(j.frequencies)
        if j.kind == serve.GRID:
            ph = _phases(j.positions, kw, j.directions)
            p = _grid_powers(volt, torch.polar(torch.ones_like(ph), ph), j.integration_spectra)
            p = p.reshape(len(p), j.n_shards, F, j.n_beams).transpose(0, 1)
            outs.append([None, None, torch.cat([_chunk_params(x).reshape(-1) for x in p])])
        else:
            t = np.arange(0, j.n_spectra, j.integration_spectra).astype(np.float32)
            per = []
            for l0, m0, dl, dm in j.trajectories:
                dirs = _unit(np.stack([l0 + t * dl, m0 + t * dm], axis=1))
                per.append(_window_sums(_tracker_powers(volt, j.positions, kw, dirs, j.integration_spectra),
                                        j.integration_spectra))
            outs.append([torch.stack(per, -1), None, None])
    return outs
