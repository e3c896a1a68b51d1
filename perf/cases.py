"""The work that users of this library have it do, as timed cases.

A survey's life is: Born modelling of a reflectivity (``born``), reverse-time
migration of recorded traces (``rtm``: source propagation, then the adjoint
with the source wavefield rebuilt), least-squares RTM on the linearised pair
(``pair``, ``linadj``) with its CG vector algebra (``vectors``), and the
learned preconditioner: generating training pairs (``pair``), training
(``unet_train`` and its single layers ``conv_fwd`` / ``conv_bwd``) and applying
the network to a search direction (``unet_infer``).

Propagation cases are windows of the full time loops: the first steps of a loop
of thousands, on the full grid, between the calls a shot makes around it
(image to the padded grid, traces to data, and back).  Velocities, sources,
receivers and interpolation tables are made here from the seed and handed to
the C ABI as any caller's own would be.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from sep_code_gb300 import gpu_funcs as gf
from sep_code_gb300 import learned
from sep_code_gb300 import unet
from sep_code_gb300._lib import check, lib
from sep_code_gb300.operator import RtmOperator

lib.sepx_batch_begin.argtypes = [C.c_int]
lib.sepx_batch_select.argtypes = [C.c_int]
lib.sepx_vec_scale_add2.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_longlong, C.c_double, C.c_double]
lib.sepx_vec_fill.argtypes = [C.c_void_p, C.c_longlong, C.c_float]
lib.sepx_set_receivers.argtypes = [C.c_int, C.c_int, C.c_int, C.c_void_p]
lib.sepx_op_image_to_padded.argtypes = [C.c_void_p] + [C.c_int] * 6
lib.sepx_op_padded_to_image.argtypes = [C.c_void_p] + [C.c_int] * 6
lib.sepx_op_traces_to_data.argtypes = [C.c_void_p, C.c_int, C.c_float]
lib.sepx_op_data_to_traces.argtypes = [C.c_void_p, C.c_int, C.c_float]

NB = 20            # absorbing cells on each side, as every workload here has
BC_A, BC_B = 50.0, 0.0005
DT = 0.001
NSLOT = 6          # device contexts kept for the propagation cases

# (input, output) channels of the network's 3x3x3 layers
LAYERS = ((8, 16), (16, 16), (16, 32), (32, 32), (32, 48), (48, 48), (48, 64), (64, 64), (112, 48),
          (80, 32), (48, 16))


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one CG iteration's inner product and update on a 64^3 model: the smallest calls
        {"name": "vectors_64", "kind": "vectors", "n": 64 ** 3},
        # the same on the traces of 4 shots, 128 x 128 receivers, 1000 samples (odd length)
        {"name": "vectors_traces", "kind": "vectors", "n": 4 * 128 * 128 * 1000 + 1},
        # a training pair: L'L m of the operator object on a 64^3 patch, host buffers in and out
        {"name": "pair_64", "kind": "pair", "m": 64, "nt": 300, "js": 4},
        # Born modelling on a small ragged model, two propagation steps per data sample
        {"name": "born_ragged", "kind": "born", "m1": 75, "m2": 53, "m3": 91, "jt": 2, "nt": 160},
        # Born modelling at survey size
        {"name": "born_512", "kind": "born", "m1": 512, "m2": 512, "m3": 400, "jt": 1, "nt": 60},
        # migration of one shot of the 128^3 model
        {"name": "rtm_128", "kind": "rtm", "m1": 128, "m2": 128, "m3": 128, "jt": 1, "nt": 150},
        # migration at survey size
        {"name": "rtm_512", "kind": "rtm", "m1": 512, "m2": 512, "m3": 400, "jt": 1, "nt": 40},
        # adjoint of the linearised pair, BF16 source snapshots
        {"name": "linadj_256_bf16", "kind": "linadj", "m1": 256, "m2": 256, "m3": 256, "jt": 1, "nt": 60,
         "js": 4, "prec": "bf16"},
        # the preconditioner applied to a 128^3 search direction
        {"name": "unet_infer_128", "kind": "unet_infer", "D": 128, "H": 128, "W": 128},
        # one training step on a batch of 64^3 patches
        {"name": "unet_train_64", "kind": "unet_train", "nb": 4, "D": 64, "H": 64, "W": 64},
        # the decoder's first fine layer on half a 384^3 direction per axis, odd row count
        {"name": "conv_fwd_48_16", "kind": "conv_fwd", "nb": 1, "D": 192, "H": 189, "W": 192, "cin": 48,
         "cout": 16, "ycs": 16, "yco": 0},
        # data and weight gradient of a second-level layer of the training batch
        {"name": "conv_bwd_32_32", "kind": "conv_bwd", "nb": 4, "D": 32, "H": 32, "W": 32, "cin": 32,
         "cout": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vectors", "pair", "born", "born", "rtm", "rtm", "linadj", "unet_infer", "unet_train",
                       "conv_fwd", "conv_fwd", "conv_bwd", "conv_bwd"])
    if kind == "vectors":
        return {"kind": kind, "n": _log(rng, 24 ** 3, 6.5e7)}
    if kind == "pair":
        return {"kind": kind, "m": 8 * rng.randint(4, 10), "nt": rng.randint(60, 200), "js": rng.choice([1, 2, 4])}
    if kind in ("born", "rtm", "linadj"):
        jt = rng.choice([1, 1, 2, 3])
        c = {"kind": kind, "m1": _log(rng, 20, 400), "m2": _log(rng, 20, 400), "m3": _log(rng, 24, 320),
             "jt": jt, "nt": jt * rng.randint(8, 24)}
        if kind == "linadj":
            c["m1"], c["m2"], c["m3"] = (min(v, 256) for v in (c["m1"], c["m2"], c["m3"]))
            c["js"] = rng.choice([1, 2, 4])
            c["prec"] = rng.choice(["f32", "bf16", "f16"])
        return c
    if kind == "unet_infer":
        return {"kind": kind, **{k: 8 * _log(rng, 4, 20) for k in "DHW"}}
    if kind == "unet_train":
        return {"kind": kind, "nb": rng.randint(1, 4), **{k: 8 * rng.randint(4, 8) for k in "DHW"}}
    cin, cout = rng.choice(LAYERS)
    big = 160 if cin * cout <= 1600 else 64
    c = {"kind": kind, "nb": rng.randint(1, 2), "D": _log(rng, 8, big), "H": _log(rng, 8, big),
         "W": _log(rng, 8, big), "cin": cin, "cout": cout}
    if kind == "conv_fwd":
        # some layers write a channel slice of a wider (concatenated) buffer
        c["yco"] = rng.choice([0, 0, 16])
        c["ycs"] = cout + c["yco"]
    return c


# ------------------------------------------------------------------ helpers
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _padded(m1, m2, m3, nb=NB):
    """padded grid of a model: boundary and halo cells, then the next multiples of 16"""
    up = lambda v: (v + 15) // 16 * 16  # noqa: E731
    f = nb + 4
    return up(m1 + 2 * f), up(m2 + 2 * f), up(m3 + 2 * f + 2 * nb + 8)


def _sinc(jt):
    """jt rows of 8 interpolation taps: row i reads the trace i/jt of a sample past tap 3"""
    k = np.arange(8)[None, :] - 3 - np.arange(jt)[:, None] / jt
    w = np.sinc(k) * np.cos(np.pi * np.clip(k / 4.5, -1, 1) / 2) ** 2
    return np.ascontiguousarray(w / w.sum(1, keepdims=True), np.float32)


def _velocity(n, g):
    """v^2 dt^2 on the padded grid: smooth in the model, random in the boundary"""
    n1, n2, n3 = n
    z = torch.arange(n3, device="cuda", dtype=torch.float32)[:, None, None]
    x = torch.arange(n1, device="cuda", dtype=torch.float32)[None, None, :]
    y = torch.arange(n2, device="cuda", dtype=torch.float32)[None, :, None]
    ph = torch.rand(3, device="cuda", generator=g) * 6.28
    v = 1600.0 + 2200.0 * z / n3 + 90.0 * torch.sin(x * 0.05 + ph[0]) * torch.cos(y * 0.06 + ph[1])
    e = torch.minimum(torch.minimum(x, n1 - 1 - x), torch.minimum(y, n2 - 1 - y))
    e = torch.minimum(e, torch.minimum(z, n3 - 1 - z))
    u = torch.rand((n3, n2, n1), device="cuda", generator=g)
    w = torch.clamp(1.0 - e / (NB + 4), 0.0, 1.0)
    v = v * (1.0 + w * 0.3 * (2.0 * u - 1.0))
    return (v * DT) ** 2


def _reflectivity(m, g):
    """flat horizons and sparse spikes"""
    m1, m2, m3 = m
    r = torch.zeros((m3, m2, m1), device="cuda")
    amp = 0.05 * torch.randn(6, device="cuda", generator=g)
    for i, iz in enumerate(torch.randint(m3 // 8 + 1, m3, (6,), device="cuda", generator=g).tolist()):
        r[iz] += amp[i]
    s = torch.rand(r.shape, device="cuda", generator=g) < 0.02
    return r + s * 0.05 * torch.randn(r.shape, device="cuda", generator=g)


def _shot(c, seed):
    """everything one shot hands to the C ABI, from the seed alone"""
    m = (c["m1"], c["m2"], c["m3"])
    n = _padded(*m)
    g = _gen(seed)
    f = NB + 4
    jt, nt = c["jt"], c["nt"]
    s = {"m": m, "n": n, "f": f, "jt": jt, "nt": nt, "ntd": nt // jt, "d": 10.0}
    s["vel"] = _velocity(n, g)
    cx, cy, cz = f + m[0] // 2, f + m[1] // 2, f + 3
    s["src"] = np.array([(cx + i) + n[0] * ((cy + j) + n[1] * cz) for j in (-1, 0, 1) for i in (-1, 0, 1)],
                        np.int32)
    ntr = s["ntd"] + 9
    t = np.arange(ntr) * DT * jt
    f0 = 0.08 / (DT * jt)   # a wavelet resolved by the trace sampling, inside the window
    a = (np.pi * f0 * (t - 0.9 / f0)) ** 2
    amp = (1.0 + 0.2 * torch.rand(9, device="cuda", generator=g)).cpu().numpy()
    s["wav"] = np.ascontiguousarray(1e3 * amp[:, None] * ((1 - 2 * a) * np.exp(-a))[None, :], np.float32)
    ix, iy = np.meshgrid(np.arange(m[0]), np.arange(m[1]))
    s["rec"] = np.ascontiguousarray((f + ix) + n[0] * ((f + iy) + n[1] * (f + 4)), np.int32).reshape(-1)
    s["refl"] = _reflectivity(m, g) if c["kind"] == "born" else None
    if c["kind"] != "born":
        k = torch.randn((m[0] * m[1], s["ntd"]), device="cuda", generator=g)
        s["data"] = torch.nn.functional.avg_pool1d(k[:, None, :], 3, 1, 1)[:, 0, :].contiguous()
    return s


class _Slot:
    """one of a few device contexts, held while a state lives"""
    free: list = []
    made = False

    def __init__(self):
        if not _Slot.made:
            gf.setup_cuda(1)
            check(lib.sepx_batch_begin(NSLOT))
            _Slot.made, _Slot.free = True, list(range(NSLOT))
        self.i = _Slot.free.pop(0)

    def __enter__(self):
        check(lib.sepx_batch_select(self.i))

    def __exit__(self, *a):
        lib.sepx_batch_select(-1)

    def __del__(self):
        _Slot.free.append(self.i)


_nets: dict = {}


def _net(what):
    if what not in _nets:
        gf.setup_cuda(1)
        _nets[what] = unet.UNet3D(params=unet.UNet3D.load_params(learned.WEIGHTS))
    return _nets[what]


def _direction(shape, g):
    """a migration-like volume (smeared horizons, noise) and the reflectivity behind it, unit RMS"""
    nb, D, H, W = shape
    y = torch.stack([_reflectivity((W, H, D), g) for _ in range(nb)])
    k = torch.tensor([-0.3, -0.7, 2.0, -0.7, -0.3], device="cuda")
    x = torch.nn.functional.conv3d(y[:, None], k.view(1, 1, 5, 1, 1), padding=(2, 0, 0))[:, 0]
    x = x + 0.02 * torch.randn(shape, device="cuda", generator=g)
    rms = lambda v: (v / v.square().mean().sqrt()).contiguous()  # noqa: E731
    return rms(x), rms(y)


def _layer(c, seed):
    """one layer's inputs: ReLU activations, He weights, bias, output gradient"""
    g = _gen(seed)
    V, cin, cout = c["nb"] * c["D"] * c["H"] * c["W"], c["cin"], c["cout"]
    x = torch.relu(torch.randn((V, cin), device="cuda", generator=g)).to(torch.bfloat16)
    w = torch.randn((27, cin, cout), device="cuda", generator=g) * math.sqrt(2.0 / (27 * cin))
    b = 0.1 * torch.randn(cout, device="cuda", generator=g)
    dy = (torch.randn((V, cout), device="cuda", generator=g) / V).to(torch.bfloat16) if c["kind"] == "conv_bwd" else None
    return x, w, b, dy


def _pack(w, cin, cout, transpose):
    pk = torch.zeros(lib.sepx_unet_packed_elems(cout, cin, 27, transpose), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    check(lib.sepx_unet_pack_weights(_ptr(w), cout, cin, 27, transpose, _ptr(pk), lib.sepx_get_stream()))
    gf.synchronize()
    return pk


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    k = case["kind"]
    gf.setup_cuda(1)
    if k == "vectors":
        g = _gen(seed)
        n = case["n"]
        return {"case": case, "a": torch.randn(n, device="cuda", generator=g),
                "b": torch.randn(n, device="cuda", generator=g) * 0.5 + 0.1, "y": torch.empty(n, device="cuda")}
    if k == "pair":
        rng = np.random.default_rng(seed)
        n = case["m"]
        vel = learned.velocity_model(rng, (n, n, n), 12.5)
        s = learned.patch_survey(np.minimum(vel, 4000.0), np.zeros_like(vel), 12.5, case["nt"])
        op = RtmOperator(s, mode="linear", snap_js=case["js"], snap_prec="f32")
        return {"case": case, "op": op, "m": learned.random_reflectivity(rng, (n, n, n))}
    if k in ("born", "rtm", "linadj"):
        s = _shot(case, seed)
        slot = _Slot()
        with slot:
            gf.create_gpu_space(s["d"], s["d"], s["d"], BC_A, BC_B, BC_B, *s["n"])
            gf.transfer_sinc_table_s(_sinc(s["jt"]))
            gf.transfer_sinc_table_d(_sinc(s["jt"]))
            gf.transfer_source_func(s["src"], s["wav"])
            gf.transfer_vel_func1(s["vel"].cpu().numpy())
            check(lib.sepx_set_receivers(s["m"][0], s["m"][1], s["ntd"] + 8,
                                         s["rec"].ctypes.data_as(C.c_void_p)))
        st = {"case": case, "slot": slot, "s": {q: s[q] for q in ("m", "f", "jt", "nt", "ntd")}}
        if k == "born":
            st["refl"] = s["refl"]
            st["out"] = torch.zeros((s["m"][0] * s["m"][1], s["ntd"]), device="cuda")
        else:
            st["data"] = s["data"]
            st["out"] = torch.zeros((s["m"][2], s["m"][1], s["m"][0]), device="cuda")
        return st
    if k == "unet_infer":
        net = _net("infer")
        x, _ = _direction((1, case["D"], case["H"], case["W"]), _gen(seed))
        return {"case": case, "net": net, "x": x}
    if k == "unet_train":
        net = _net("train")
        shape = (case["nb"], case["D"], case["H"], case["W"])
        x, y = _direction(shape, _gen(seed))
        if _nets.get("train_shape") != shape:   # the batch buffers of a captured step, as learned.train has them
            torch.cuda.synchronize()
            if "train_p" not in _nets:
                _nets["train_p"] = net.flat["p"].clone()
            _nets["train_io"] = (torch.empty(shape, device="cuda"), torch.empty(shape, device="cuda"))
            for buf, v in zip(_nets["train_io"], (x, y)):
                buf.copy_(v)
            torch.cuda.synchronize()
            net.capture_train_step(*_nets["train_io"])
            _nets["train_shape"] = shape
        return {"case": case, "net": net, "x": x, "y": y, "p": _nets["train_p"], "io": _nets["train_io"]}
    x, w, b, dy = _layer(case, seed)
    cin, cout, V = case["cin"], case["cout"], x.shape[0]
    st = {"case": case, "x": x, "b": b, "stream": torch.cuda.ExternalStream(lib.sepx_get_stream())}
    if k == "conv_fwd":
        st["pk"] = _pack(w, cin, cout, 0)
        st["out"] = torch.zeros((V, case["ycs"]), dtype=torch.bfloat16, device="cuda")
    else:
        st["pk"] = _pack(w, cin, cout, 1)
        st["dy"] = dy
        st["dx"] = torch.empty((V, cin), dtype=torch.bfloat16, device="cuda")
        st["dw"] = torch.empty((27, cin, cout), device="cuda")
        st["db"] = torch.empty(cout, device="cuda")
    return st


# ------------------------------------------------------------------ run
def run(state):
    c = state["case"]
    k = c["kind"]
    if k == "vectors":
        n = c["n"]
        r = C.c_double()
        check(lib.sepx_dot_f32(_ptr(state["a"]), _ptr(state["b"]), n, C.byref(r)))
        check(lib.sepx_vec_scale_add2(_ptr(state["y"]), _ptr(state["a"]), _ptr(state["b"]), n, 0.75, -1.5))
        return {"dot": r.value, "y": state["y"]}
    if k == "pair":
        d = state["op"].forward(state["m"])
        return {"data": d, "image": state["op"].adjoint(d)}
    if k in ("born", "rtm", "linadj"):
        s = state["s"]
        out, m, f = state["out"], s["m"], (-s["f"],) * 3
        with state["slot"]:
            check(lib.sepx_vec_fill(_ptr(out), out.numel(), 0.0))
            if k == "born":
                check(lib.sepx_zero_traces())
                check(lib.sepx_op_image_to_padded(_ptr(state["refl"]), *m, *f))
                check(lib.sepx_rtm_forward_resident(s["jt"], 9, s["nt"]))
                check(lib.sepx_op_traces_to_data(_ptr(out), s["ntd"], DT))
            else:
                check(lib.sepx_op_data_to_traces(_ptr(state["data"]), s["ntd"], DT))
                if k == "rtm":
                    check(lib.sepx_source_prop_resident(s["jt"], 9, s["nt"]))
                    check(lib.sepx_rtm_adjoint_resident(s["jt"], 9, s["nt"], 1))
                else:
                    gf.lin_source_pass(s["jt"], 9, s["nt"], c["js"], c["prec"])
                    gf.lin_adjoint(s["jt"], s["nt"], c["js"], c["prec"])
                check(lib.sepx_op_padded_to_image(_ptr(out), *m, *f))
        return out
    if k == "unet_infer":
        return state["net"].forward_device(state["x"])
    if k == "unet_train":
        # every pass starts from the same weights and moments, then does what a training loop does with
        # a batch: into the captured step's buffers, one step
        net = state["net"]
        with torch.cuda.stream(net.stream):
            net.flat["p"].copy_(state["p"])
            net.flat["m"].zero_()
            net.flat["v"].zero_()
            state["io"][0].copy_(state["x"])
            state["io"][1].copy_(state["y"])
        net.step_count = 0
        net.pack()
        loss = net.train_step(*state["io"])
        return {"loss": loss, "out": net.a["out"], "grad": net.flat["g"]}
    st = lib.sepx_get_stream()
    dims = (c["nb"], c["D"], c["H"], c["W"])
    cin, cout = c["cin"], c["cout"]
    if k == "conv_fwd":
        check(lib.sepx_unet_conv_fwd(_ptr(state["x"]), cin, 0, *dims, cin, 27, _ptr(state["pk"]), _ptr(state["b"]),
                                     cout, 1, _ptr(state["out"]), c["ycs"], c["yco"], None, None, st))
        return state["out"]
    with torch.cuda.stream(state["stream"]):
        state["dw"].zero_()
        state["db"].zero_()
    check(lib.sepx_unet_conv_fwd_masked(_ptr(state["dy"]), cout, 0, *dims, cout, 27, _ptr(state["pk"]), None, cin, 0,
                                        _ptr(state["dx"]), cin, 0, None, None, _ptr(state["x"]), cin, 0, st))
    check(lib.sepx_unet_conv_wgrad_bias(_ptr(state["x"]), cin, 0, *dims, cin, 27, _ptr(state["dy"]), cout, 0, cout,
                                        _ptr(state["dw"]), _ptr(state["db"]), st))
    return {"dx": state["dx"], "dw": state["dw"], "db": state["db"]}


# ------------------------------------------------------------------ work
_STENCIL = 41      # additions and multiplications of one 25-point update


def _cells(n):
    return (n[0] - 8) // 16 * 16 * ((n[1] - 8) // 16 * 16) * (n[2] - 12)


def work(case):
    """Bytes and operations of one pass.  Time loops: every step reads each
    field's two states, v^2 dt^2 and the image or snapshot it uses, and writes
    the new states, once per updated cell; loops whose volumes all fit the
    129 MB L2 count their inputs and outputs once instead."""
    k = case["kind"]
    if k == "vectors":
        return {"bytes": 20.0 * case["n"], "flops": 5.0 * case["n"]}
    if k == "pair":
        n, nt = _padded(case["m"], case["m"], case["m"]), case["nt"]
        cells = _cells(n)
        recs = case["m"] ** 2 * nt
        return {"bytes": 4.0 * (3 * n[0] * n[1] * n[2] + 2 * case["m"] ** 3 + 2 * recs + cells * nt / case["js"] * 2),
                "flops": 4.0 * _STENCIL * cells * nt}
    if k in ("born", "rtm", "linadj"):
        m, nt = (case["m1"], case["m2"], case["m3"]), case["nt"]
        n = _padded(*m)
        cells, vol = _cells(n), n[0] * n[1] * n[2]
        recs, mod = m[0] * m[1] * (nt // case["jt"]), m[0] * m[1] * m[2]
        big = 4.0 * vol * {"born": 6, "rtm": 6, "linadj": 5}[k] > 129e6
        images = (nt + case["jt"] - 1) // case["jt"] if k != "linadj" else (nt + case["js"] - 1) // case["js"]
        if k == "born":
            step, fields = 28.0 * cells * nt + 4.0 * cells * images, 2 * nt
        elif k == "rtm":
            step, fields = 16.0 * cells * (nt + 1) + 28.0 * cells * nt + 8.0 * cells * images, 3 * nt + 1
        else:
            q = 4 if case["prec"] == "f32" else 2
            step, fields = (16.0 + 20.0) * cells * nt + (2 * q + 8.0) * cells * images, 2 * nt
        return {"bytes": 4.0 * (recs + mod) + (step if big else 4.0 * vol), "flops": float(_STENCIL) * cells * fields}
    if k in ("unet_infer", "unet_train"):
        nb = case.get("nb", 1)
        V = nb * case["D"] * case["H"] * case["W"]
        lvl = {"e1": 0, "e2": 1, "e3": 2, "b4": 3, "d3": 2, "d2": 1, "d1": 0, "ou": 0}
        fl = sum(2.0 * (V >> (3 * lvl[L.name[:2]])) * L.ntap * L.cin * L.cout for L in unet.LAYERS)
        act = sum(2.0 * (V >> (3 * lvl[L.name[:2]])) * (L.cin_p + L.cout) for L in unet.LAYERS)
        if k == "unet_infer":
            return {"bytes": act + 8.0 * V, "flops": fl}
        # backward: each layer reads its input, its output gradient (twice) and writes its input's gradient
        return {"bytes": 3.0 * act + 12.0 * V, "flops": 3.0 * fl}
    V, cin, cout = case["nb"] * case["D"] * case["H"] * case["W"], case["cin"], case["cout"]
    fl, wb = 54.0 * V * cin * cout, 27.0 * cin * cout
    if k == "conv_fwd":
        return {"bytes": 2.0 * V * (cin + cout) + 2 * wb, "flops": fl}
    return {"bytes": 2.0 * V * (2 * cin + cout) + 6 * wb, "flops": 2 * fl}


# ------------------------------------------------------------------ exact
class _Grid64:
    """the propagation step in 64 bits"""

    def __init__(self, s):
        n1, n2, n3 = n = s["n"]
        self.n = n
        self.v = s["vel"].double()
        c = 8.0 / (5.0 * s["d"] ** 2)
        self.c = [-1025.0 / 576.0 * 3 * c, c, -c / 8.0, c / 63.0, -c / 896.0]
        self.xe, self.ye, self.ze = 4 + 16 * ((n1 - 8) // 16), 4 + 16 * ((n2 - 8) // 16), n3 - 8
        self.xg, self.yg = self.xe - 4, self.ye - 4
        x = torch.arange(n1, device="cuda")[None, None, :]
        y = torch.arange(n2, device="cuda")[None, :, None]
        z = torch.arange(n3, device="cuda")[:, None, None]
        e = torch.minimum(torch.minimum(x - 4, n1 - 4 - x), torch.minimum(y - 4, n2 - 4 - y))
        e = torch.minimum(e, torch.minimum(z - 4, n3 - 4 - z))
        t = torch.exp(-BC_B * (BC_A - e.double()))
        on = (x < self.xg) & (y < self.yg) & (e >= 0)
        self.t = torch.where(on & (t < 1.0), t, torch.ones((), dtype=torch.float64, device="cuda"))
        self.imask = (x < self.xg) & (y < self.yg)
        self.tab = torch.tensor(_sinc(s["jt"]), dtype=torch.float64, device="cuda")
        self.wav = torch.tensor(s["wav"], dtype=torch.float64, device="cuda")
        self.src = torch.tensor(s["src"], dtype=torch.long, device="cuda")
        self.rec = torch.tensor(s["rec"], dtype=torch.long, device="cuda")
        self.jt = s["jt"]

    def zeros(self):
        n1, n2, n3 = self.n
        return torch.zeros((n3, n2, n1), dtype=torch.float64, device="cuda")

    def inner(self, a, dx=0, dy=0, dz=0):
        return a[4 + dz:self.ze + dz, 4 + dy:self.ye + dy, 4 + dx:self.xe + dx]

    def lap(self, p):
        """25-point Laplacian at the updated cells, 0 elsewhere"""
        out = self.zeros()
        o = self.inner(out)
        o.add_(self.inner(p), alpha=self.c[0])
        for k in range(1, 5):
            for d in ((k, 0, 0), (-k, 0, 0), (0, k, 0), (0, -k, 0), (0, 0, k), (0, 0, -k)):
                o.add_(self.inner(p, *d), alpha=self.c[k])
        return out

    def keep(self, a):
        """a at the updated cells, 0 elsewhere"""
        out = self.zeros()
        self.inner(out).copy_(self.inner(a))
        return out

    def inj(self, j):
        return self.wav[:, j // self.jt:j // self.jt + 8] @ self.tab[j % self.jt]

    def add_src(self, p, j, sign=1.0):
        p.view(-1).index_add_(0, self.src, sign * self.inj(j))

    def add_rec(self, p, trc, it):
        i = it // self.jt
        p.view(-1).index_add_(0, self.rec, self.tab[it % self.jt] @ trc[i:i + 8])


def _loops64(case, s):
    G = _Grid64(s)
    nt, jt, ntd, rnx = s["nt"], s["jt"], s["ntd"], s["m"][0]
    n1, n2, n3 = s["n"]
    m1, m2, m3 = s["m"]
    f = s["f"]
    nrec = len(s["rec"])
    first = (torch.arange(nrec, device="cuda") % rnx == 0)
    dt = float(np.float32(DT))
    if case["kind"] == "born":
        e = G.zeros()
        e[f:f + m3, f:f + m2, f:f + m1] = s["refl"].double()
        img = torch.zeros_like(e)
        img[1:] += e[:-1]
        img[:-1] -= e[:-1]
        img *= G.imask
        trc = torch.zeros((ntd + 8, nrec), dtype=torch.float64, device="cuda")
        D0, D1, S0, S1 = (G.zeros() for _ in range(4))
        for it in range(nt):
            a = G.keep(2 * D1 - G.t * G.t * D0) + G.lap(G.v * D1)
            b = G.keep(2 * S1 - G.t * S0) + G.v * G.lap(S1)
            G.add_src(b, it)
            if it % jt == 0:
                a += 1e-6 * b * G.keep(img)
            i = it // jt
            trc[i:i + 8] += G.tab[it % jt][:, None] * a.view(-1)[G.rec][None, :]
            D0, D1, S0, S1 = D1, a * G.t * G.t, S1, b * G.t
        mt = (trc[4:4 + ntd] / dt).t()
        d = torch.empty_like(mt)
        d[:, 1:] = mt[:, :-1] - mt[:, 1:]
        spill = torch.cat([torch.zeros(1, dtype=torch.float64, device="cuda"), mt[:-1, -1]])
        d[:, 0] = spill - mt[:, 0] - first * mt[:, 0]
        d[:, 1] += first * mt[:, 0]
        return d.contiguous()
    data = s["data"].double()
    nxt = torch.cat([data[:, 1:], torch.cat([data[1:, :1], torch.zeros((1, 1), dtype=torch.float64, device="cuda")])], 1)
    g = (nxt - data) / dt
    g[:, 0] *= 1.0 + first
    trc = torch.zeros((ntd + 8, nrec), dtype=torch.float64, device="cuda")
    trc[4:4 + ntd] = g.t()
    img = G.zeros()
    A, B = G.zeros(), G.zeros()
    if case["kind"] == "rtm":
        for it in range(nt + 1):
            u = G.keep(2 * B - A) + G.v * G.lap(B)
            G.add_src(u, it)
            A, B = B, u
        S0, S1 = B, A
        D0, D1 = G.zeros(), G.zeros()
        for it in range(nt - 1, -1, -1):
            a = G.keep(2 * D1 - G.t * D0) + G.v * G.lap(D1)
            G.add_rec(a, trc, it)
            if it == nt - 1:
                u = S0
            else:
                u = G.keep(2 * S1 - S0) + G.v * G.lap(S1)
            if it % jt == 0:
                img += G.keep(1e-6 * a * u * G.imask)
            if it != nt - 1:
                G.add_src(S1, it + 1, -1.0)
                S0, S1 = S1, u
            D0, D1 = D1, a * G.t
    else:
        js = case["js"]
        snaps = []
        for it in range(nt):
            u = G.keep(2 * B - A) + G.v * G.lap(B)
            G.add_src(u, it)
            if it % js == 0:
                snaps.append(u)
            A, B = B, u
        a, B = G.zeros(), G.zeros()
        for it in range(nt - 1, -1, -1):
            a = G.t * a + G.v * G.lap(B)
            G.add_rec(a, trc, it)
            b = B + a
            if it % js == 0:
                img += G.keep(1e-6 * b * snaps[it // js] * G.imask)
            B = G.t * b
    lap = torch.zeros_like(img)
    lap[:-1] = img[1:] - img[:-1]
    return lap[f:f + m3, f:f + m2, f:f + m1].contiguous()


def _conv64(x, w):
    """3x3x3 convolution in 64 bits: x [nb, D, H, W, cin], w [27, cin, cout]"""
    nb, D, H, W, cin = x.shape
    if w.shape[0] == 1:
        return x @ w[0]
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    out = None
    for t in range(27):
        z, y, q = t // 9, t // 3 % 3, t % 3
        v = p[:, z:z + D, y:y + H, q:q + W].reshape(-1, cin) @ w[t]
        out = v if out is None else out + v
    return out.view(nb, D, H, W, -1)


def _unet64(x, P):
    conv = lambda n, v: torch.relu(_conv64(v, P[n + "_w"]) + P[n + "_b"])  # noqa: E731
    first = lambda v, c: v.permute(0, 4, 1, 2, 3) if c else v.permute(0, 2, 3, 4, 1)  # noqa: E731
    pool = lambda v: first(torch.nn.functional.avg_pool3d(first(v, True), 2), False)  # noqa: E731
    up = lambda v: v.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)  # noqa: E731
    e1 = conv("e1b", conv("e1a", x[..., None]))
    e2 = conv("e2b", conv("e2a", pool(e1)))
    e3 = conv("e3b", conv("e3a", pool(e2)))
    b4 = conv("b4b", conv("b4a", pool(e3)))
    d3 = conv("d3b", conv("d3a", torch.cat([up(b4), e3], -1)))
    d2 = conv("d2b", conv("d2a", torch.cat([up(d3), e2], -1)))
    d1 = conv("d1b", conv("d1a", torch.cat([up(d2), e1], -1)))
    return x + (_conv64(d1, P["out_w"]) + P["out_b"])[..., 0]


def exact(case, seed):
    k = case["kind"]
    if k == "pair":   # the operator object prepares its own velocity boundary and tables
        return None
    if k == "vectors":
        g = _gen(seed)
        a = torch.randn(case["n"], device="cuda", generator=g)
        b = (torch.randn(case["n"], device="cuda", generator=g) * 0.5 + 0.1)
        return {"dot": float((a.double() * b.double()).sum()), "y": 0.75 * a.double() - 1.5 * b.double()}
    if k in ("born", "rtm", "linadj"):
        return _loops64(case, _shot(case, seed))
    if k in ("unet_infer", "unet_train"):
        z = np.load(learned.WEIGHTS)
        P, names = {}, []
        for L in unet.LAYERS:
            w = torch.tensor(z[L.name + "_w"], dtype=torch.float64, device="cuda").reshape(L.ntap, -1, L.cout)[:, :L.cin]
            P[L.name + "_w"] = w.contiguous()
            P[L.name + "_b"] = torch.tensor(z[L.name + "_b"], dtype=torch.float64, device="cuda").reshape(-1)
            names += [(L.name + "_w", L), (L.name + "_b", L)]
        nb = case.get("nb", 1)
        x, y = _direction((nb, case["D"], case["H"], case["W"]), _gen(seed))
        if k == "unet_infer":
            with torch.no_grad():
                return _unet64(x.double(), P).reshape(-1)
        for v in P.values():
            v.requires_grad_(True)
        out = _unet64(x.double(), P)
        loss = (out - y.double()).square().mean()
        loss.backward()
        grads = []
        for name, L in names:
            gr = P[name].grad
            if name.endswith("_w"):   # stored with the input channels rounded up to 8
                full = torch.zeros((L.ntap, L.cin_p, L.cout), dtype=torch.float64, device="cuda")
                full[:, :L.cin] = gr
                gr = full
            grads.append(gr.reshape(-1))
        return {"loss": float(loss), "out": out.detach().reshape(-1), "grad": torch.cat(grads)}
    x, w, b, dy = _layer(case, seed)
    dims = (case["nb"], case["D"], case["H"], case["W"])
    X = x.double().view(*dims, -1)
    W = w.double()
    if k == "conv_fwd":
        y = torch.relu(_conv64(X, W) + b.double()).view(X[..., 0].numel(), -1)
        return torch.cat([torch.zeros((y.shape[0], case["yco"]), dtype=torch.float64, device="cuda"), y], 1)
    dY = dy.double().view(*dims, -1)
    dx = _conv64(dY, W.flip(0).transpose(1, 2).contiguous()) * (X > 0)
    p = torch.nn.functional.pad(X, (0, 0, 1, 1, 1, 1, 1, 1))
    D, H, Wd = dims[1:]
    dw = torch.stack([p[:, t // 9:t // 9 + D, t // 3 % 3:t // 3 % 3 + H, t % 3:t % 3 + Wd].reshape(-1, X.shape[-1]).t()
                      @ dY.view(-1, dY.shape[-1]) for t in range(27)])
    return {"dx": dx.view(x.shape), "dw": dw, "db": dY.view(-1, dY.shape[-1]).sum(0)}
