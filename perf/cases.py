"""The work a user of this library has it do, as measurable cases: the U-Net forward from and to device memory, its queued host entry, the
sliding window over a volume, the conv entry points of the reference interface (plain, decoder form, stride 2), the joint of two network
levels (norm, down conv, transposed conv), the elementwise operators on MX tensors, and the front and back end of predict.

A case is a dict; "kind" names the family and the other keys its sizes and options.  Inputs are seeded stand-ins for what the path meets:
activations N(0, 1), Kaiming-normal weights, CT bytes clip(N(110, 40), 0, 255)."""
import ctypes as C
import itertools
import math

import torch

import ufsm_b200
from ufsm_b200 import Feather, Gnp, Shape5, Split, UnetCfg

F32, F16, MX8, MX4, U8OUT = 0, 2, 3, 4, 100
WIDTHS = [32, 64, 128, 256, 320]                  # the benchmark network's channels per level
NH = 7                                            # its head channels
G = 8                                             # GroupNorm groups of the MX operators
_wkeys = itertools.count(1)                       # split_t.wkey names one set of weights for the life of the process


def _lib():
    L = ufsm_b200.lib()
    if not getattr(_lib, "ready", False):
        if L.nn_init(0) != 0:
            raise RuntimeError((L.lp_check() or b"").decode())
        _lib.ready = True
    return L


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # a small network on a small patch, one at a time: what a quick look at one place of a volume costs; launches and latency count
        {"name": "unet_32_three_levels", "kind": "unet", "P": 32, "L": 3, "N": 1, "bits": 8, "out": "f32"},
        # the benchmark network on its 128^3 patch, every conv MX-fp8: the headline forward
        {"name": "unet_128_fp8", "kind": "unet", "P": 128, "L": 5, "N": 1, "bits": 8, "out": "f32"},
        # the same network with MX-fp4 interior convs on a batch of patches, fp16 logits: the throughput form
        {"name": "unet_128_fp4_batch", "kind": "unet", "P": 128, "L": 5, "N": 2, "bits": 4, "out": "h16"},
        # the call a predict loop makes: CT bytes in pinned host memory to probability bytes in pinned host memory, queued
        {"name": "unet_96_host_bytes", "kind": "host", "P": 96, "L": 4, "N": 1, "bits": 8},
        # a small volume through the sliding window with blending, host to host
        {"name": "window_176", "kind": "window", "V": 176, "P": 64, "overlap": 16, "L": 3, "batch": 2, "bits": 8, "out": "u8"},
        # the reference's conv entry on one layer of the benchmark's first configuration, fp16 in and out, weights known by their key
        {"name": "conv_32_64cube_fp8", "kind": "conv", "bits": 8, "N": 1, "ci": 32, "co": 32, "D": 64, "H": 64, "W": 64, "x": "h16", "y": "h16", "gn": False, "stats": False, "key": True},
        # a deep layer of a training-like caller: MX tensors in and out, the GroupNorm + SiLU input transform, statistics of the output,
        # weights that change between calls (no key); odd grid
        {"name": "conv_deep_fp4", "kind": "conv", "bits": 4, "N": 1, "ci": 256, "co": 256, "D": 15, "H": 18, "W": 20, "x": "mx", "y": "mx", "gn": True, "stats": True, "key": False},
        # the decoder conv of the reference's models on [upsample(silu(gn(coarse))) | silu(gn(skip))]
        {"name": "conv_decoder_fp8", "kind": "decoder", "bits": 8, "N": 1, "cx": 64, "c2": 32, "co": 32, "D": 64, "H": 64, "W": 64, "gn": True, "key": True},
        # the 3^3 stride-2 conv between two levels
        {"name": "conv_stride2_fp8", "kind": "stride2", "bits": 8, "N": 1, "ci": 32, "co": 64, "D": 96, "H": 96, "W": 96, "y": "mx"},
        # one joint of the U-Net: InstanceNorm + LeakyReLU + requantise with the space-to-depth copy, 2^3 stride-2 down conv, transposed conv
        # into the concat tensor; the sizes of the benchmark's second configuration
        {"name": "level_joint_fp4", "kind": "joint", "bits": 4, "N": 1, "c": 64, "cd": 128, "D": 96, "H": 96, "W": 96},
        # the elementwise operators of the reference interface one after the other: quantise, statistics, GroupNorm + SiLU, dequantise,
        # upsample, 1^3 conv to logits
        {"name": "mx_operators_fp8", "kind": "ops", "bits": 8, "N": 1, "c": 64, "co": 7, "D": 48, "H": 48, "W": 48},
        # predict's front and back end for one window: network input from CT bytes, material mask, placement of the probabilities, seam feather
        {"name": "predict_window_192", "kind": "predict", "W": 192, "halo": 16, "B": 16, "bits": 8, "axis": 1, "neighbours": 127},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _chan(rng, hi=320):
    """channel counts: mostly multiples of 32, some of 8"""
    c = _log(rng, 16, hi)
    return max(16, c // 8 * 8) if rng.random() < 0.25 else max(32, (c + 16) // 32 * 32)


def _grid(rng, lo, hi, even=False):
    g = [_log(rng, lo, hi) for _ in range(3)]
    return [v // 2 * 2 for v in g] if even else g


MOST_FLOPS, MOST_BYTES = {"window": 6e12}, 6e8    # a drawn case stays below the largest listed ones


def draw(rng):
    while True:
        kind = rng.choice(["unet", "unet", "host", "window", "conv", "conv", "decoder", "stride2", "joint", "ops", "predict"])
        bits = rng.choice([8, 4])
        if kind in ("unet", "host"):
            L = rng.randint(2, 5)
            m = 1 << (L - 1)
            c = {"kind": kind, "P": max(1, _log(rng, 16, 128) // m) * m, "L": L, "N": rng.randint(1, 4), "bits": bits}
            if c["P"] < 4 * m:                   # four voxels or more an axis at the bottom level
                continue
            if kind == "unet":
                c["out"] = rng.choice(["f32", "h16"])
        elif kind == "window":
            L = rng.randint(2, 4)
            P = rng.choice([32, 48, 64])
            c = {"kind": kind, "V": _log(rng, P + 1, 200), "P": P, "overlap": rng.choice([8, 16]), "L": L, "batch": rng.randint(1, 4), "bits": bits, "out": rng.choice(["u8", "h16"])}
        elif kind == "conv":
            D, H, W = _grid(rng, 4, 96)
            c = {"kind": kind, "bits": bits, "N": rng.randint(1, 2), "ci": _chan(rng), "co": _chan(rng), "D": D, "H": H, "W": W, "x": rng.choice(["h16", "mx"]), "y": rng.choice(["h16", "mx"]),
                 "gn": rng.random() < 0.4, "stats": False, "key": rng.random() < 0.6}
            c["stats"] = c["y"] == "mx" and rng.random() < 0.4
        elif kind == "decoder":
            D, H, W = _grid(rng, 8, 72, even=True)
            c = {"kind": kind, "bits": bits, "N": rng.randint(1, 2), "cx": rng.choice([32, 64, 128, 256]), "c2": rng.choice([32, 64, 128]), "co": rng.choice([32, 64, 128]), "D": D, "H": H, "W": W,
                 "gn": rng.random() < 0.7, "key": rng.random() < 0.6}
        elif kind == "stride2":
            D, H, W = _grid(rng, 8, 128)
            c = {"kind": kind, "bits": bits, "N": rng.randint(1, 2), "ci": _chan(rng, 256), "co": _chan(rng), "D": D, "H": H, "W": W, "y": rng.choice(["h16", "mx"])}
        elif kind == "joint":
            D, H, W = _grid(rng, 8, 128, even=True)
            ch = rng.choice([32, 64, 128, 256])
            c = {"kind": kind, "bits": bits, "N": rng.randint(1, 2), "c": ch, "cd": rng.choice([ch, 2 * ch]), "D": D, "H": H, "W": W}
        elif kind == "ops":
            D, H, W = _grid(rng, 4, 96)
            c = {"kind": kind, "bits": bits, "N": rng.randint(1, 2), "c": _chan(rng, 256), "co": rng.randint(1, 16), "D": D, "H": H, "W": W}
        else:
            W = _log(rng, 48, 256)
            c = {"kind": kind, "W": W, "halo": rng.choice([8, 12, 16]), "B": rng.choice([8, 16]), "bits": bits, "axis": rng.choice([-1, 0, 1]), "neighbours": rng.randint(0, 127)}
        w = work(c)
        if w["flops"] <= MOST_FLOPS.get(kind, 2e12) and w["bytes"] <= MOST_BYTES:
            return c


# ---------------------------------------------------------------- what one pass cannot do without
def _mxb(bits, n, c, s):
    """bytes of an MX tensor: rows of 8 / 16 / 32 channels and a scale byte each"""
    bw = 8 if c <= 8 else 16 if c <= 16 else 32
    return n * -(-c // bw) * s * (bw * bits // 8 + 1)


def _unet_work(c):
    P, L = c["P"], c["L"]
    cw, fl, nw = WIDTHS[:L], 0.0, 0
    for l in range(L):
        S, ci = (P >> l) ** 3, cw[l] if l else 1
        fl += 2.0 * S * 27 * (ci * cw[l] + cw[l] * cw[l])
        nw += 27 * (ci + cw[l]) * cw[l]
        if l < L - 1:
            fl += 2 * 2.0 * S * cw[l] * cw[l + 1] + 2.0 * S * 27 * 3 * cw[l] * cw[l]
            nw += 16 * cw[l] * cw[l + 1] + 27 * 3 * cw[l] * cw[l]
    return fl + 2.0 * P ** 3 * cw[0] * NH, nw


def _window_origins(c):
    V, P, s = c["V"], c["P"], c["P"] - c["overlap"]
    return 1 if V <= P else -(-(V - P) // s) + 1


def work(case):
    c, k = case, case["kind"]
    if k in ("unet", "host"):
        fl, nw = _unet_work(c)
        vox = c["N"] * c["P"] ** 3
        return {"bytes": vox * (1 + NH if k == "host" else 2 + NH * (4 if c["out"] == "f32" else 2)) + nw, "flops": fl * c["N"]}
    if k == "window":
        fl, nw = _unet_work(c)
        return {"bytes": c["V"] ** 3 * (1 + NH * (1 if c["out"] == "u8" else 2)) + nw, "flops": fl * _window_origins(c) ** 3}
    if k == "predict":
        n, E = c["W"] ** 3, c["W"] - 2 * c["halo"]
        S = E - c["B"]
        return {"bytes": n + _mxb(c["bits"], 1, 4, n) + E ** 3 * (2 + 0.125 + 1) + S ** 3 + 2.0 * (E ** 3 - S ** 3), "flops": 0}
    N, S = c["N"], c["D"] * c["H"] * c["W"]
    if k == "conv":
        xb = N * c["ci"] * S * 2 if c["x"] == "h16" else _mxb(c["bits"], N, c["ci"], S)
        yb = N * c["co"] * S * 2 if c["y"] == "h16" else _mxb(c["bits"], N, c["co"], S)
        return {"bytes": xb + yb + 27 * c["ci"] * c["co"] * 4, "flops": 2.0 * N * S * 27 * c["ci"] * c["co"]}
    if k == "decoder":
        xb = _mxb(c["bits"], N, c["cx"], S // 8) + _mxb(c["bits"], N, c["c2"], S)
        return {"bytes": xb + _mxb(c["bits"], N, c["co"], S) + 27 * (c["cx"] + c["c2"]) * c["co"] * 4, "flops": 2.0 * N * S * 27 * (c["cx"] + c["c2"]) * c["co"]}
    if k == "stride2":
        So = -(-c["D"] // 2) * -(-c["H"] // 2) * -(-c["W"] // 2)
        yb = N * c["co"] * So * 2 if c["y"] == "h16" else _mxb(c["bits"], N, c["co"], So)
        return {"bytes": _mxb(c["bits"], N, c["ci"], S) + yb + 27 * c["ci"] * c["co"] * 4, "flops": 2.0 * N * So * 27 * c["ci"] * c["co"]}
    if k == "joint":
        return {"bytes": N * c["c"] * S * 2 + _mxb(c["bits"], N, 2 * c["c"], S) + 2 * _mxb(c["bits"], N, c["cd"], S // 8) + 16 * c["c"] * c["cd"], "flops": 2 * 2.0 * N * S * c["c"] * c["cd"]}
    # ops: statistics need the whole tensor before the transform can start, but it is read at least once; every operator writes its result
    m = _mxb(c["bits"], N, c["c"], S)
    return {"bytes": N * c["c"] * S * (2 + 4) + m + m + _mxb(c["bits"], N, c["c"], 8 * S) + N * c["co"] * S * 2, "flops": 2.0 * N * S * c["c"] * c["co"]}


def tolerance(case):
    k = case["kind"]
    if k in ("unet", "host", "window"):
        # networks of MX convs: a value next to a rounding boundary takes the other 3-bit (1-bit) code when an fp32 sum changes in its last bit
        bytes_out = k == "host" or (k == "window" and case["out"] == "u8")
        return {"differ": 0.01} if bytes_out else {"rel": 0.02, "max": 0.9}
    if k == "predict":
        return {"differ": 1e-3}                   # a probability byte within the hardware exp's error of a tie
    # fp16 outputs: an fp32 sum in another order rounds to the neighbouring half now and then; MX codes and scale bytes likewise
    return {"rel": 1e-3, "max": 2e-2, "differ": 5e-3}


# ---------------------------------------------------------------- inputs and handles
class _Free:
    """calls fn(h) when the state goes away"""

    def __init__(self, fn, h):
        self.fn, self.h = fn, h

    def __del__(self):
        self.fn(self.h)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + 17)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _ct(g, n):
    return (_randn(g, n) * 40 + 110).round_().clamp_(0, 255).to(torch.uint8)


def _weights(g, co, ci, taps):
    return _randn(g, co * ci * taps) * math.sqrt(2.0 / (ci * taps))


def _mx(L, x, bits, N, Cn, S):
    """fp32 plane-major activations as an MX tensor of the reference's storage"""
    y = torch.empty((L.lp_mx8_bytes if bits == 8 else L.lp_mx4_bytes)(N, Cn, S), dtype=torch.uint8, device="cuda")
    (L.lp_f32_to_mx8 if bits == 8 else L.lp_f32_to_mx4)(x.data_ptr(), N, Cn, S, y.data_ptr())
    return y


def _gn(g, N, Cn, keep):
    """GroupNorm parameters and statistics of a tensor of Cn channels"""
    gp = Gnp()
    t = [1 + 0.2 * _randn(g, Cn), 0.1 * _randn(g, Cn), 0.1 * _randn(g, N * G), 0.8 + 0.4 * torch.rand(N * G, generator=g, device="cuda")]
    keep += t
    gp.gamma, gp.beta, gp.mean, gp.rstd, gp.G = t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(), G
    return gp


def _unet(L, g, c, max_batch):
    cfg = UnetCfg()
    cfg.L, cfg.nh, cfg.P = c["L"], NH, c["P"]
    for i, v in enumerate(WIDTHS[:c["L"]]):
        cfg.cw[i] = v
    cfg.bits_first, cfg.bits_mid, cfg.bits_last = 8, c["bits"], 8
    cw, parts = WIDTHS[:c["L"]], []

    def conv(co, ci, taps):
        parts.append(_weights(g, co, ci, taps))
        parts.append(0.01 * _randn(g, co))
    for l in range(c["L"]):
        conv(cw[l], cw[l] if l else 1, 27)
        conv(cw[l], cw[l], 27)
        if l < c["L"] - 1:
            conv(cw[l + 1], cw[l], 8)
    for l in range(c["L"] - 2, -1, -1):
        conv(cw[l], cw[l + 1], 8)
        conv(cw[l], 2 * cw[l], 27)
        conv(cw[l], cw[l], 27)
    conv(NH, cw[0], 1)
    w = torch.cat(parts).cpu().numpy()
    if w.size != L.umx_unet_nweights(C.byref(cfg)):
        raise RuntimeError("unet weights")
    u = L.umx_unet_create(C.byref(cfg), w.ctypes.data, max_batch)
    if not u:
        raise RuntimeError((L.lp_check() or b"").decode())
    return u


def prepare(case, seed):
    L, g, c, k = _lib(), _gen(seed), case, case["kind"]
    s = {"keep": []}
    keep = s["keep"]
    if k == "unet":
        N, V = c["N"], c["P"] ** 3
        u = _unet(L, g, c, N)
        x = (_ct(g, N * V).float() / 255).half()
        y = torch.empty((N, NH, V), dtype=torch.float32 if c["out"] == "f32" else torch.float16, device="cuda")
        keep += [_Free(L.umx_unet_free, u), x]
        fn, args = L.umx_unet_forward if c["out"] == "f32" else L.umx_unet_forward_h16, (u, x.data_ptr(), N, y.data_ptr())
        s["run"] = lambda: (fn(*args), y)[1]
    elif k == "host":
        N, V = c["N"], c["P"] ** 3
        u = _unet(L, g, c, N)
        x, y = torch.empty(N * V, dtype=torch.uint8, pin_memory=True), torch.empty((N, NH, V), dtype=torch.uint8, pin_memory=True)
        x.copy_(_ct(g, N * V))
        keep += [_Free(L.umx_unet_free, u), x]
        fn, args = L.umx_unet_submit_host_u8, (u, x.data_ptr(), N, y.data_ptr())
        s["run"] = lambda: (fn(*args), y)[1]
    elif k == "window":
        V, fmt, dt = c["V"], (U8OUT if c["out"] == "u8" else F16), (torch.uint8 if c["out"] == "u8" else torch.float16)
        u = _unet(L, g, c, c["batch"])
        w = L.umx_window_make(V, c["P"], c["overlap"])
        p = L.umx_wplan_create(C.byref(w), 0, 1, NH)
        vol, out = torch.empty(V ** 3, dtype=torch.uint8, pin_memory=True), torch.empty((NH, V, V, V), dtype=dt, pin_memory=True)
        vol.copy_(_ct(g, V ** 3))
        if L.umx_wplan_prepare(p, u, c["batch"], fmt) != 0:
            raise RuntimeError((L.lp_check() or b"").decode())
        keep += [_Free(L.umx_wplan_free, p), _Free(L.umx_unet_free, u), vol]
        fn, args = L.umx_window_run_fx, (u, p, vol.data_ptr(), c["batch"], fmt, out.data_ptr())
        s["run"] = lambda: (fn(*args), out)[1]
    elif k in ("conv", "decoder"):
        N, D, H, W, co, bits = c["N"], c["D"], c["H"], c["W"], c["co"], c["bits"]
        S, mx = D * H * W, (MX8 if bits == 8 else MX4)
        gp, sp = Gnp(), Split()
        if k == "conv":
            ci, xbf, ybf = c["ci"], (F16 if c["x"] == "h16" else mx), (F16 if c["y"] == "h16" else mx)
            x = _randn(g, N * ci * S)
            x = x.half() if c["x"] == "h16" else _mx(L, x, bits, N, ci, S)
            stats = c["stats"]
            if c["gn"]:
                gp = _gn(g, N, ci, keep)
        else:
            ci, xbf, ybf, stats = c["cx"] + c["c2"], mx, mx, True
            x = _mx(L, _randn(g, N * c["cx"] * (S // 8)), bits, N, c["cx"], S // 8)
            x2 = _mx(L, _randn(g, N * c["c2"] * S), bits, N, c["c2"], S)
            keep.append(x2)
            sp.x2, sp.c_split, sp.up = x2.data_ptr(), c["cx"], 1
            if c["gn"]:
                gp, sp.gp2 = _gn(g, N, c["cx"], keep), _gn(g, N, c["c2"], keep)
        w, b = _weights(g, co, ci, 27), 0.01 * _randn(g, co)
        sp.wkey = next(_wkeys) if c["key"] else 0
        y = torch.empty(N * co * S, dtype=torch.float16, device="cuda") if ybf == F16 else torch.empty((L.lp_mx8_bytes if bits == 8 else L.lp_mx4_bytes)(N, co, S), dtype=torch.uint8, device="cuda")
        keep += [x, w, b]
        fn = L.lp_conv_fwd_f8 if bits == 8 else L.lp_conv_fwd_f4
        if stats:
            # the statistics of the stored output for the GroupNorm that follows, as the model graph takes them
            sp.stored_stats = 1
            sums = torch.zeros(N * G * 2 * 3, dtype=torch.int64, device="cuda")
            mean, rstd = torch.empty(N * G, device="cuda"), torch.empty(N * G, device="cuda")
            zero, fin, nb = L.nn_zero, L.umx_gn_finalize, sums.numel() * 8
            args = (x.data_ptr(), xbf, Shape5(N, ci, D, H, W), w.data_ptr(), b.data_ptr(), co, y.data_ptr(), ybf, gp, sums.data_ptr(), G, sp)
            fargs = (sums.data_ptr(), N * G, co // G * S, 1e-5, mean.data_ptr(), rstd.data_ptr())

            def run_stats():
                zero(sums.data_ptr(), nb)
                fn(*args)
                fin(*fargs)
                return y, mean, rstd
            s["run"] = run_stats
        else:
            args = (x.data_ptr(), xbf, Shape5(N, ci, D, H, W), w.data_ptr(), b.data_ptr(), co, y.data_ptr(), ybf, gp, None, 0, sp)
            s["run"] = lambda: (fn(*args), y)[1]
    elif k == "stride2":
        N, D, H, W, ci, co, bits = c["N"], c["D"], c["H"], c["W"], c["ci"], c["co"], c["bits"]
        S, mx = D * H * W, (MX8 if bits == 8 else MX4)
        ys = Shape5(N, co, (D + 1) // 2, (H + 1) // 2, (W + 1) // 2)
        So = ys.d * ys.h * ys.w
        x = _mx(L, _randn(g, N * ci * S), bits, N, ci, S)
        w, b = _weights(g, co, ci, 27), 0.01 * _randn(g, co)
        ybf = F16 if c["y"] == "h16" else mx
        y = torch.empty(N * co * So, dtype=torch.float16, device="cuda") if ybf == F16 else torch.empty((L.lp_mx8_bytes if bits == 8 else L.lp_mx4_bytes)(N, co, So), dtype=torch.uint8, device="cuda")
        keep += [x, w, b]
        fn, args = L.lp_conv_fwd_s2_f8, (x.data_ptr(), mx, Shape5(N, ci, D, H, W), w.data_ptr(), b.data_ptr(), co, y.data_ptr(), ybf, ys, Gnp())
        s["run"] = lambda: (fn(*args), y)[1]
    elif k == "joint":
        N, D, H, W, ch, cd, bits = c["N"], c["D"], c["H"], c["W"], c["c"], c["cd"], c["bits"]
        S, nb = D * H * W, ch // 32
        x = _randn(g, N * ch * S).half()                                         # a conv's output, blocked fp16 [N][block][voxel][32]
        wd, bd = _weights(g, cd, ch, 8).cpu().numpy(), (0.01 * _randn(g, cd)).cpu().numpy()
        wu, bu = _weights(g, ch, cd, 8).cpu().numpy(), (0.01 * _randn(g, ch)).cpu().numpy()
        down, up = L.umx_conv_create(2, wd.ctypes.data, bd.ctypes.data, cd, ch, bits), L.umx_conv_create(3, wu.ctypes.data, bu.ctypes.data, ch, cd, bits)
        part = torch.empty(L.umx_stats_doubles(N, ch, D, H, W), dtype=torch.float64, device="cuda")
        coef = torch.empty(N * ch * 2, device="cuda")

        def mxt(n, s_):
            return torch.empty(L.umx_mx_bytes32(bits, N, n, s_), dtype=torch.uint8, device="cuda")
        cat, s2d, dn = mxt(2 * ch, S), mxt(8 * ch, S // 8), mxt(cd, S // 8)
        keep += [_Free(L.umx_conv_free, down), _Free(L.umx_conv_free, up), x, part, s2d]
        stat, apply_, fwd = L.umx_in_stats_coef, L.umx_in_apply, L.umx_conv_fwd
        a0 = (x.data_ptr(), N, ch, D, H, W, None, None, 1e-5, part.data_ptr(), coef.data_ptr())
        a1 = (x.data_ptr(), coef.data_ptr(), N, ch, D, H, W, 2, cat.data_ptr(), bits, 2 * nb, nb, s2d.data_ptr(), None, 1)
        a2 = (down, s2d.data_ptr(), N, D // 2, H // 2, W // 2, dn.data_ptr(), 1, bits, 0, 0, None, 3)
        a3 = (up, dn.data_ptr(), N, D // 2, H // 2, W // 2, cat.data_ptr(), 1, bits, 2 * nb, 0, None, 3)

        def run_joint():
            stat(*a0)
            apply_(*a1)
            fwd(*a2)
            fwd(*a3)
            return coef, cat, dn
        s["run"] = run_joint
    elif k == "ops":
        N, D, H, W, ch, co, bits = c["N"], c["D"], c["H"], c["W"], c["c"], c["co"], c["bits"]
        S, mx, sh = D * H * W, (MX8 if bits == 8 else MX4), Shape5(N, ch, D, H, W)
        raw = _randn(g, N * ch * S).half()
        gp = _gn(g, N, ch, keep)
        w, b = _randn(g, co * ch) / math.sqrt(ch), 0.01 * _randn(g, co)
        sums = torch.zeros(N * G * 2 * 3, dtype=torch.int64, device="cuda")
        mean, rstd = torch.empty(N * G, device="cuda"), torch.empty(N * G, device="cuda")
        gp.mean, gp.rstd = mean.data_ptr(), rstd.data_ptr()
        yb = L.lp_mx8_bytes if bits == 8 else L.lp_mx4_bytes
        x, act, fine = (torch.empty(yb(N, ch, m), dtype=torch.uint8, device="cuda") for m in (S, S, 8 * S))
        back = torch.empty((N, ch, S), device="cuda")
        logits = torch.empty((N, co, S), dtype=torch.float16, device="cuda")
        keep += [raw, w, b, sums]
        enc, dec = (L.lp_h16_to_mx8, L.lp_mx8_to_f32) if bits == 8 else (L.lp_h16_to_mx4, L.lp_mx4_to_f32)
        zero, stat, fin, silu, up2, head, none = L.nn_zero, L.lp_gn_sums_mx, L.umx_gn_finalize, L.lp_gn_silu_apply_mx, L.lp_up2_fwd_mx, L.lp_conv1_fwd_mx_h16, Gnp()
        nb = sums.numel() * 8
        ae, ad = (raw.data_ptr(), F16, N, ch, S, x.data_ptr()), (act.data_ptr(), N, ch, S, back.data_ptr())
        a0 = (x.data_ptr(), mx, N, ch, G, S, sums.data_ptr(), 0, S)
        a1 = (sums.data_ptr(), N * G, ch // G * S, 1e-5, mean.data_ptr(), rstd.data_ptr())
        a2 = (x.data_ptr(), mx, sh, G, gp.gamma, gp.beta, gp.mean, gp.rstd, act.data_ptr(), mx)
        a3 = (act.data_ptr(), mx, sh, fine.data_ptr(), mx, none)
        a4 = (x.data_ptr(), mx, sh, w.data_ptr(), b.data_ptr(), co, logits.data_ptr(), gp)

        def run_ops():
            enc(*ae)
            zero(sums.data_ptr(), nb)
            stat(*a0)
            fin(*a1)
            silu(*a2)
            dec(*ad)
            up2(*a3)
            head(*a4)
            return x, mean, rstd, act, back, fine, logits
        s["run"] = run_ops
    else:
        W, h, B, bits = c["W"], c["halo"], c["B"], c["bits"]
        n, E = W ** 3, W - 2 * h
        S = E - B
        ct = _ct(g, n)
        ct[torch.rand(n, generator=g, device="cuda") < 0.1] = 0                  # voxels that are not material
        lg = (2 * _randn(g, n)).half()
        dyo, dxo = 100 * _randn(g, W) - W, 100 * _randn(g, W) + W
        inp = torch.empty((L.lp_mx8_bytes if bits == 8 else L.lp_mx4_bytes)(1, 4, n), dtype=torch.uint8, device="cuda")
        mask = torch.empty((n + 31) // 32, dtype=torch.int32, device="cuda")
        e, out = torch.empty(E ** 3, dtype=torch.uint8, device="cuda"), torch.empty(S ** 3, dtype=torch.uint8, device="cuda")
        zs, ys, xs = (torch.empty(m, dtype=torch.uint8, device="cuda") for m in (B * E * E, S * B * E, S * S * B))
        old = [torch.randint(0, 256, (m,), generator=g, device="cuda", dtype=torch.uint8) for m in (B * E * E, S * B * E, S * S * B)]      # the spills of earlier windows
        f = Feather()
        f.S, f.B, f.e, f.osh, f.out = S, B, e.data_ptr(), S, out.data_ptr()
        for d in range(1, 8):
            f.nb[d] = old[0 if d & 4 else 1 if d & 2 else 2].data_ptr() if c["neighbours"] >> (d - 1) & 1 else None
        for d in range(3):
            f.oo[d], f.on[d] = 0, S
        keep += [ct, lg, dyo, dxo, old, f]
        front, mk, h16, place, blend, kp = L.lp_pred_input_mx, L.nn_pred_ctmask, L.nn_set_logits_h16, L.nn_pred_place_m, L.umx_feather_blend, L.umx_feather_keep
        a0 = (ct.data_ptr(), W, 110.0, 1.0 / 40.0, dyo.data_ptr(), dxo.data_ptr(), c["axis"], 0, W, inp.data_ptr(), 2, bits)
        a1 = (ct.data_ptr(), n, mask.data_ptr())
        a2 = (lg.data_ptr(), mask.data_ptr(), W, h, -h, -h, -h, E, E, E, E, e.data_ptr())
        a3 = (e.data_ptr(), S, B, zs.data_ptr(), ys.data_ptr(), xs.data_ptr())
        fr = C.byref(f)

        def run_predict():
            h16(1)
            front(*a0)
            mk(*a1)
            place(*a2)
            blend(fr)
            kp(*a3)
            return inp, mask, e, out, zs, ys, xs
        s["run"] = run_predict
    L.nn_sync()
    err = L.lp_check()
    if err:
        raise RuntimeError(err.decode())
    return s


def run(state):
    return state["run"]()
