"""The work that users of this package have it do, as timed cases.

Every case goes through public entry points: ``run_transport`` (scenes with
the source sampled on the device, the tally grids back on the host), the
device-array entry ``cc_transport_photons_device``, ``BatchedRun`` (many
scenes in one launch), and for the learned denoiser the layer calls
``ccu_conv3d`` / ``ccu_conv3d_wgrad`` and ``UNet3D``'s forward and backward
passes.  Scenes and sizes are those of ``chatcarlo_b200.workloads``,
``chatcarlo_b200.phantoms`` and ``chatcarlo_b200.denoiser.LAYERS``; ``draw``
spreads the same kinds of work over the sizes in between, ragged volumes
among them.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from chatcarlo_b200 import _native as N
from chatcarlo_b200 import _unet_native as U
from chatcarlo_b200 import ct_denoise as CD
from chatcarlo_b200 import denoiser as DN
from chatcarlo_b200 import phantoms as PH
from chatcarlo_b200 import workloads as W
from chatcarlo_b200.batched import BatchedRun
from chatcarlo_b200.distributed import device_grid_tensors
from chatcarlo_b200.geometry import Geometry
from chatcarlo_b200.tally import VoxelGrid
from chatcarlo_b200.transport import default_engine, run_transport

DEV = "cuda"


def listed() -> list[dict]:
    return [
        # the call a newcomer makes: run_transport's own defaults (100,000
        # histories, 5 cm voxels), a new host grid each time
        {"name": "room_default", "kind": "run", "scene": "room", "n": 100_000, "voxel_cm": 5.0, "own_grid": False},
        # a shielding study: 20 batches of 200,000 histories in the room,
        # batch statistics, one page-locked grid kept between runs
        {"name": "room_4e6", "kind": "run", "scene": "room", "n": 4_000_000, "voxel_cm": 5.0, "own_grid": True},
        # a CT dose scan on the full 1 mm grid, 553 MB of tallies back each time
        {"name": "ct_scan_2e6", "kind": "run", "scene": "ct", "n": 2_000_000, "voxel_cm": 0.1, "own_grid": True},
        # photons of another program, already on the device, through the room
        {"name": "photons_1e6", "kind": "photons", "n": 1_000_000},
        # a parameter sweep: two dozen random scenes in one launch
        {"name": "scenes_24", "kind": "batch", "scenes": 24, "hist_lo": 20_000, "hist_hi": 400_000, "scenes_seed": 2026},
        # denoiser layers: the network's first convolution on the CT volume,
        # a decoder layer on a minibatch (skip + upsampled input), the
        # deepest layer on a small volume
        {"name": "conv_e0_ct", "kind": "conv", "ca": 16, "cb": 0, "cout": 16, "b": 1, "d": 320, "h": 320, "w": 152},
        {"name": "conv_d1a_4x32", "kind": "conv", "ca": 32, "cb": 64, "cout": 32, "b": 4, "d": 32, "h": 32, "w": 32},
        {"name": "conv_b3_8x8", "kind": "conv", "ca": 128, "cb": 0, "cout": 128, "b": 8, "d": 8, "h": 8, "w": 8},
        # training: data gradient of the last decoder level's first layer
        # (48 channels split over skip and upsampled parts), weight gradient
        # of a full-resolution layer
        {"name": "dgrad_d0a_4x64", "kind": "dgrad", "ca": 16, "cb": 32, "cout": 16, "b": 4, "d": 64, "h": 64, "w": 64},
        {"name": "wgrad_e0_4x64", "kind": "wgrad", "ca": 16, "cb": 0, "cout": 16, "b": 4, "d": 64, "h": 64, "w": 64},
        # the whole network: one prediction of the CT volume, and the
        # gradient of a training minibatch
        {"name": "predict_ct", "kind": "predict", "net": "ct", "b": 1, "d": 320, "h": 320, "w": 152},
        {"name": "gradient_4x64", "kind": "gradient", "b": 4, "d": 64, "h": 64, "w": 64},
    ]


def _log_int(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# (full-resolution, upsampled and output channels) of the network's layers
_LAYERS = sorted({(L.ca, L.cb, L.cout) for L in DN.LAYERS})


def _volume(rng, most: float, even: bool, of8: bool = False) -> dict:
    """A batch of volumes of at most `most` voxels: sides of 8 to 160, ragged
    unless the layer needs even sides or the network multiples of 8."""
    while True:
        b = rng.choice([1, 1, 2, 3, 4, 8])
        s = [_log_int(rng, 8, 160) for _ in range(3)]
        if of8:
            s = [8 * max(1, round(x / 8)) for x in s]
        elif even:
            s = [x + x % 2 for x in s]
        if 512 <= b * s[0] * s[1] * s[2] <= most:
            return {"b": b, "d": s[0], "h": s[1], "w": s[2]}


def draw(rng) -> dict:
    kind = rng.choice(["run", "run", "run", "photons", "batch", "conv", "conv", "dgrad", "wgrad", "predict", "gradient"])
    if kind == "run":
        scene = rng.choice(["room", "room", "ct", "plain", "phantom"])
        n = _log_int(rng, 20_000, 2_000_000 if scene == "ct" else 4_000_000)
        lo, hi = {"room": (4.0, 12.0), "ct": (0.1, 0.5), "plain": (0.5, 1.5), "phantom": (0.5, 1.0)}[scene]
        voxel = round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 3)
        return {"kind": "run", "scene": scene, "n": n, "voxel_cm": voxel,
                "own_grid": scene != "room" or rng.random() < 0.5}
    if kind == "photons":
        return {"kind": "photons", "n": _log_int(rng, 5_000, 2_000_000)}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(2, 28), "hist_lo": 10_000,
                "hist_hi": _log_int(rng, 20_000, 400_000), "scenes_seed": rng.randrange(1 << 20)}
    if kind in ("predict", "gradient"):
        c = {"kind": kind}
        if kind == "predict":
            c["net"] = rng.choice(["ct", "phantom"])
        return {**c, **_volume(rng, 4e6 if kind == "predict" else 1e6, True, of8=True)}
    ca, cb, cout = rng.choice(_LAYERS)
    return {"kind": kind, "ca": ca, "cb": cb, "cout": cout, **_volume(rng, 6e7 / (ca + cb + cout), cb > 0)}


# ---------------------------------------------------------------------------
# transport
# ---------------------------------------------------------------------------

# track segments per history, and centimetres of track inside the grid per
# history (voxel visits ~ 1.5 x track / voxel edge), as the engine counts them
_SEGMENTS = {"room": 5.3, "ct": 2.7, "plain": 4.5, "phantom": 4.0}
_TRACK_CM = {"room": 160.0, "ct": 6.2, "plain": 15.0, "phantom": 25.0}


def _scene(case: dict, seed: int) -> tuple[dict, tuple, tuple]:
    """(scene dict, grid origin, grid extent in cm)."""
    name = case["scene"]
    if name == "phantom":
        raw, g = PH.phantom(np.random.default_rng(seed))
    else:
        raw = {"room": W.room, "ct": W.ct, "plain": W.plain_mc}[name]()
        g = {"room": W.ROOM_GRID, "ct": W.CT_GRID, "plain": W.PLAIN_MC_GRID}[name]
    return raw, g["origin"], tuple(s * g["voxel_cm"] for s in g["shape"])


def _run_shape(case: dict) -> tuple:
    h = case["voxel_cm"]
    if not case["own_grid"]:                 # run_transport's grid covers the scene's bounding box
        g = Geometry(_scene(case, 0)[0]["geometry"])
        ext = np.asarray(g.bbox_max, dtype=float) - np.asarray(g.bbox_min, dtype=float)
    else:
        ext = _scene(case, 0)[2]
    return tuple(max(1, int(math.ceil(x / h - 1e-9))) for x in ext)


def _prepare_run(case: dict, seed: int) -> dict:
    raw, origin, ext = _scene(case, seed)
    st = {"raw": raw, "seed": seed, "grid": None}
    eng = default_engine()
    eng.tables(Geometry(raw["geometry"]).materials(), need_muen=True)
    if case["own_grid"]:
        st["grid"] = VoxelGrid(origin_cm=np.asarray(origin, dtype=float), shape=_run_shape(case),
                               voxel_size_cm=case["voxel_cm"], track_uncertainty=True, pinned=True)
    return st


def _run_run(case: dict, st: dict):
    r = run_transport(st["raw"], n_histories=case["n"], seed=st["seed"], dose_grid=True,
                      grid_resolution_cm=case["voxel_cm"], grid=st["grid"])
    g = r.grid
    return {"kerma": g.kerma_keV, "h10": g.h10_track_pSv_cm3, "kerma_sum2": g.kerma_sum2, "h10_sum2": g.h10_sum2,
            "hits": g.n_batches_hit, "n_batches": int(g.n_batches), "n_histories": int(g.n_histories),
            "edep_MeV": np.array([r.energy_deposited_MeV[k] for k in sorted(r.energy_deposited_MeV)]),
            "outcomes": np.array([r.fraction_absorbed, r.fraction_escaped, r.mean_scatter_events]),
            "n_fluorescence": int(r.n_fluorescence)}


def _prepare_photons(case: dict, seed: int) -> dict:
    raw = W.room()
    eng = default_engine()
    geo = Geometry(raw["geometry"])
    ts, th = eng.tables(geo.materials(), need_muen=False)
    n = case["n"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    u = torch.rand(n, 2, generator=g, device=DEV, dtype=torch.float64) - 0.5
    pos = torch.tensor([0.0, 0.0, 190.0], device=DEV, dtype=torch.float64).expand(n, 3).contiguous()
    d = torch.stack([35.0 * u[:, 0], 43.0 * u[:, 1], torch.full_like(u[:, 0], -180.0)], 1)
    d = d / d.norm(dim=1, keepdim=True)
    sp = W.room_spectrum()
    e = torch.tensor([s["energy_keV"] for s in sp], device=DEV, dtype=torch.float64)
    w = torch.tensor([s["weight"] for s in sp], device=DEV, dtype=torch.float64)
    en = e[torch.multinomial(w, n, replacement=True, generator=g)]
    return {"eng": eng, "tables": th, "scene": eng.scene(geo, ts), "n_mat": len(ts.names), "seed": seed,
            "pos": pos, "dir": d.contiguous(), "energy": en.contiguous(),
            "nsc": torch.empty(n, dtype=torch.int32, device=DEV),
            "flags": torch.empty(2, n, dtype=torch.uint8, device=DEV)}


def _run_photons(case: dict, st: dict):
    # the photons are updated in place: the program keeps its own, and the
    # engine's stream starts once the copies are there
    p, d, e = st["pos"].clone(), st["dir"].clone(), st["energy"].clone()
    torch.cuda.current_stream().synchronize()
    eng = st["eng"]
    edep = np.zeros(st["n_mat"])
    nfl = C.c_int64(0)
    fn = eng.lib.cc_transport_photons_device
    arg = [C.cast(t.data_ptr(), a) if a is not C.c_void_p else t.data_ptr()
           for t, a in zip((p, d, e), fn.argtypes[5:8])]
    out = [C.cast(t.data_ptr(), a) if a is not C.c_void_p else t.data_ptr()
           for t, a in zip((st["nsc"], st["flags"][0], st["flags"][1]), fn.argtypes[11:14])]
    N.check(fn(eng.ctx, st["scene"], st["tables"], None, case["n"], *arg, st["seed"], 0, 1, *out, N.dptr(edep),
               C.byref(nfl)), eng.lib)
    return {"pos": p, "dir": d, "energy": e, "n_scatter": st["nsc"], "absorbed": st["flags"][0],
            "escaped": st["flags"][1], "edep": edep, "n_fluorescence": int(nfl.value)}


def _batch_scenes(case: dict):
    return W.batched_scenes(n_scenes=case["scenes"], seed=case["scenes_seed"], hist_lo=case["hist_lo"],
                            hist_hi=case["hist_hi"])


def _prepare_batch(case: dict, seed: int) -> dict:
    scenes, specs, counts = _batch_scenes(case)
    br = BatchedRun(scenes, specs, counts)
    return {"br": br, "seed": seed, "totals": [device_grid_tensors(d)["totals"] for d in br.dgrids]}


def _run_batch(case: dict, st: dict):
    br = st["br"]
    br.reset()
    counts, _ = br.run(seed=st["seed"])
    return {"counts": counts, "totals": st["totals"]}       # the tallies stay on the device


# ---------------------------------------------------------------------------
# denoiser
# ---------------------------------------------------------------------------

def _act(g, n: int, c: int) -> torch.Tensor:
    """ReLU activations."""
    return torch.randn(n, c, generator=g, device=DEV).relu_().to(torch.bfloat16)


def _prepare_layer(case: dict, seed: int) -> dict:
    g = torch.Generator(device=DEV).manual_seed(seed)
    ca, cb, cout = case["ca"], case["cb"], case["cout"]
    cin = ca + cb
    n = case["b"] * case["d"] * case["h"] * case["w"]
    w32 = torch.randn(27, cout, cin, generator=g, device=DEV) * math.sqrt(2.0 / (27 * cin))
    st = {"w32": w32, "n": n, "a": _act(g, n, ca), "b": _act(g, n // 8, cb) if cb else None}
    lib = U.lib()
    if case["kind"] == "wgrad":
        st["dz"] = (torch.randn(n, cout, generator=g, device=DEV) * 1e-3).to(torch.bfloat16)
        st["dz"] *= torch.rand(n, cout, generator=g, device=DEV) < 0.5
        st["dw"] = torch.zeros(27, cout, cin, device=DEV)
        st["slices"] = max(1, min(256, n // 2048))
        return st
    st["w"] = torch.empty(lib.ccu_packed_weight_elems(cout, cin), dtype=torch.bfloat16, device=DEV)
    st["wt"] = torch.empty(lib.ccu_packed_weight_elems(cin, cout), dtype=torch.bfloat16, device=DEV)
    U.check(lib.ccu_pack_weights(w32.data_ptr(), cout, cin, st["w"].data_ptr(), st["wt"].data_ptr(),
                                 torch.cuda.current_stream().cuda_stream))
    if case["kind"] == "conv":
        st["bias"] = torch.randn(cout, generator=g, device=DEV) * 0.1
        st["out"] = torch.empty(n, cout, dtype=torch.bfloat16, device=DEV)
    else:
        st["dz"] = (torch.randn(n, cout, generator=g, device=DEV) * 1e-3).to(torch.bfloat16)
        st["out"] = torch.empty(n, ca, dtype=torch.bfloat16, device=DEV)
        st["up"] = torch.empty(n, cb, dtype=torch.bfloat16, device=DEV) if cb else None
    return st


def _run_layer(case: dict, st: dict):
    lib, stream = U.lib(), torch.cuda.current_stream().cuda_stream
    ptr = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    dims = (case["b"], case["d"], case["h"], case["w"])
    ca, cb, cout = case["ca"], case["cb"], case["cout"]
    if case["kind"] == "conv":
        U.check(lib.ccu_conv3d(ptr(st["a"]), ca, ptr(st["b"]), cb, *dims, ptr(st["w"]), ptr(st["bias"]), cout, 1,
                               ptr(st["out"]), cout, None, None, stream))
        return st["out"]
    if case["kind"] == "dgrad":
        # into the ReLU output below (masked by it) and the upsampled part
        U.check(lib.ccu_conv3d(ptr(st["dz"]), cout, None, 0, *dims, ptr(st["wt"]), None, ca + cb, 0, ptr(st["out"]),
                               ca, ptr(st["a"]), ptr(st["up"]), stream))
        return [st["out"], st["up"]] if cb else [st["out"]]
    U.check(lib.ccu_zero(ptr(st["dw"]), st["dw"].numel() * 4, stream))
    U.check(lib.ccu_conv3d_wgrad(ptr(st["a"]), ca, ptr(st["b"]), cb, *dims, ptr(st["dz"]), cout, ptr(st["dw"]),
                                 st["slices"], stream))
    return st["dw"]


def _prepare_net(case: dict, seed: int) -> dict:
    """A low-history kerma map of an object (Poisson-like noise in log space
    over a smooth map), its densities and materials, and the network."""
    dims = (case["b"], case["d"], case["h"], case["w"])
    n = int(np.prod(dims))
    g = torch.Generator(device=DEV).manual_seed(seed)
    params = DN.load_params(CD.CT_PRETRAINED if case.get("net") == "ct" else None)[0]
    model = DN.UNet3D(params=params)
    coarse = torch.randn(dims[0], 1, *(max(2, s // 8) for s in dims[1:]), generator=g, device=DEV)
    smooth = torch.nn.functional.interpolate(coarse, size=dims[1:], mode="trilinear").reshape(-1)
    noise = torch.randn(n, generator=g, device=DEV)
    rel = 0.05 + 0.3 * torch.rand(n, generator=g, device=DEV)
    x = torch.log((torch.exp(0.5 * smooth) * (1.0 + rel * noise)).clamp_min(0.0) + DN.EPS)
    mat = (smooth > 0.8).to(torch.uint8) + (smooth > -0.5).to(torch.uint8)
    dens = torch.tensor([0.0012, 1.0, 1.85, 11.35], device=DEV)[mat.long()] * DN.DENSITY_SCALE
    model.set_input(None, None, None, dims[0], dims[1:], device_xlog=x, device_density=dens, device_mat=mat,
                    unc=rel.cpu().numpy())
    st = {"model": model, "x": x}
    if case["kind"] == "gradient":
        st["target"] = torch.log(torch.exp(0.5 * smooth) + DN.EPS)
        st["weight"] = torch.where(mat > 0, 1.0, 0.1)
        st["inv"] = 1.0 / float(st["weight"].sum())
    return st


def _run_net(case: dict, st: dict):
    m = st["model"]
    if case["kind"] == "predict":
        return m.predict()
    m.forward()
    m.backward(st["target"], st["weight"], st["inv"])
    return {"gradient": m.g, "loss": m.acc, "out": m.out}


# ---------------------------------------------------------------------------
# the interface
# ---------------------------------------------------------------------------

def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    make = {"run": _prepare_run, "photons": _prepare_photons, "batch": _prepare_batch, "predict": _prepare_net,
            "gradient": _prepare_net}.get(kind, _prepare_layer)
    return {"case": case, **make(case, seed)}


def run(state: dict):
    case = state["case"]
    go = {"run": _run_run, "photons": _run_photons, "batch": _run_batch, "predict": _run_net,
          "gradient": _run_net}.get(case["kind"], _run_layer)
    return go(case, state)


# FLOPs of one track segment (material, cross sections, boundaries, one
# interaction's samplers) and of one voxel visit
_SEG_FLOPS, _VISIT_FLOPS = 300.0, 15.0


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "run":
        s, h = case["scene"], case["voxel_cm"]
        visits = 1.5 * _TRACK_CM[s] / h
        return {"bytes": float(np.prod(_run_shape(case))) * 36.0,
                "flops": case["n"] * (_SEGMENTS[s] * _SEG_FLOPS + visits * _VISIT_FLOPS)}
    if kind == "photons":
        return {"bytes": case["n"] * (2 * 56.0 + 6.0), "flops": case["n"] * _SEGMENTS["room"] * _SEG_FLOPS}
    if kind == "batch":
        total = float(sum(_batch_scenes(case)[2]))
        return {"bytes": case["scenes"] * 64.0 ** 3 * 16.0, "flops": total * (2.8 * _SEG_FLOPS + 60.0 * _VISIT_FLOPS)}
    n = float(case["b"] * case["d"] * case["h"] * case["w"])
    if kind in ("predict", "gradient"):
        flops = sum(2.0 * 27 * L.cin * L.cout * n / 8 ** L.level for L in DN.LAYERS)
        p = DN.n_params()
        if kind == "predict":
            return {"bytes": n * (32.0 + 4.0 + 4.0) + 2.0 * p, "flops": flops}
        return {"bytes": n * (32.0 + 16.0) + 6.0 * p, "flops": 3.0 * flops}
    ca, cb, cout = case["ca"], case["cb"], case["cout"]
    flops = 2.0 * 27 * (ca + cb) * cout * n
    inp = n * 2.0 * (ca + cb / 8.0)
    if kind == "conv":
        return {"bytes": inp + n * 2.0 * cout + 54.0 * (ca + cb) * cout, "flops": flops}
    if kind == "dgrad":
        return {"bytes": n * 2.0 * (cout + 2 * ca + cb) + 54.0 * (ca + cb) * cout, "flops": flops}
    return {"bytes": inp + n * 2.0 * cout + 108.0 * (ca + cb) * cout, "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------

def _pad(x: torch.Tensor) -> torch.Tensor:
    """[B, D, H, W, C] with a voxel of zeros around each volume."""
    return torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))


def _taps(xp: torch.Tensor):
    """(tap, the padded volume shifted by it), taps in (dz, dy, dx) order."""
    d, h, w = (s - 2 for s in xp.shape[1:4])
    for t in range(27):
        z, y, x = t // 9, t // 3 % 3, t % 3
        yield t, xp[:, z:z + d, y:y + h, x:x + w]


def _conv64(x: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """3x3x3 "same" convolution of x [B, D, H, W, cin] with w [27, cout, cin]."""
    y = None
    for t, v in _taps(_pad(x)):
        u = v.reshape(-1, x.shape[-1]) @ w[t].T
        y = u if y is None else y + u
    return y.reshape(*x.shape[:4], w.shape[1])


def _up64(x: torch.Tensor) -> torch.Tensor:
    for a in (1, 2, 3):
        x = x.repeat_interleave(2, a)
    return x


def _pool64(x: torch.Tensor) -> torch.Tensor:
    b, d, h, w, c = x.shape
    return x.reshape(b, d // 2, 2, h // 2, 2, w // 2, 2, c).mean((2, 4, 6))


def _exact_layer(case: dict, seed: int):
    st = _prepare_layer(case, seed)
    dims = (case["b"], case["d"], case["h"], case["w"])
    vol = lambda t, div=1: t.double().reshape(dims[0], *(s // div for s in dims[1:]), -1)  # noqa: E731
    wb = st["w32"].to(torch.bfloat16).double()
    if case["kind"] == "dgrad":
        # taps flipped, channels transposed
        y = _conv64(vol(st["dz"]), wb.flip(0).transpose(1, 2)).reshape(st["n"], -1)
        out = [y[:, :case["ca"]] * (st["a"] > 0)]
        return out + [y[:, case["ca"]:].contiguous()] if case["cb"] else out
    x = vol(st["a"])
    if case["cb"]:
        x = torch.cat([x, _up64(vol(st["b"], 2))], -1)
    if case["kind"] == "conv":
        return (_conv64(x, wb) + st["bias"].double()).relu_().reshape(st["n"], -1)
    dz = st["dz"].double()
    return torch.stack([dz.T @ v.reshape(st["n"], -1) for _, v in _taps(_pad(x))])


def _exact_net(case: dict, seed: int):
    """The network with BF16 weights and inputs, everything else in 64 bits."""
    st = _prepare_net(case, seed)
    m = st["model"]
    p = m.p.double().requires_grad_(case["kind"] == "gradient")
    lay = DN.param_layout()

    def conv(name, x):
        o, n, bo, bn = lay[name]
        w = p[o:o + n]
        w = w + (w.detach().to(torch.bfloat16).double() - w.detach())     # BF16 values, gradients of the master copy
        return torch.relu(_conv64(x, w.reshape(27, bn, -1)) + p[bo:bo + bn])

    x = m.a["x0"].double().reshape(*m.shape, DN.IN_CH)
    e0 = conv("e0", conv("e0a", x))
    e1 = conv("e1", conv("e1a", _pool64(e0)))
    e2 = conv("e2", conv("e2a", _pool64(e1)))
    b3 = conv("b3", conv("b3a", _pool64(e2)))
    d2 = conv("d2", conv("d2a", torch.cat([e2, _up64(b3)], -1)))
    d1 = conv("d1", conv("d1a", torch.cat([e1, _up64(d2)], -1)))
    d0 = conv("d0", conv("d0a", torch.cat([e0, _up64(d1)], -1)))
    ho = lay["head"][0]
    out = st["x"].double() + d0.reshape(-1, 16) @ p[ho:ho + 16] + p[ho + 16]
    if case["kind"] == "predict":
        return out.detach()
    loss = (st["weight"].double() * (out - st["target"].double()) ** 2).sum() * st["inv"]
    loss.backward()
    return {"gradient": p.grad, "loss": loss.detach().reshape(1), "out": out.detach()}


def exact(case: dict, seed: int):
    """Transport is a random walk whose decisions follow 32-bit roundings: no
    64-bit value of its tallies exists for the same random numbers."""
    if case["kind"] in ("run", "photons", "batch"):
        return None
    with torch.set_grad_enabled(case["kind"] == "gradient"):
        return (_exact_net if case["kind"] in ("predict", "gradient") else _exact_layer)(case, seed)
