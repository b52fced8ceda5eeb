"""CPU checks of the boundary: the library loads, exports every function include/ufsm_mx.h declares, the structs have the
reference's sizes, the host-only scheduler logic is right, and compute entries fail loudly without a B200."""
import ctypes as C
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

import ufsm_b200
from ufsm_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def header_functions():
    src = open(os.path.join(ROOT, "include", "ufsm_mx.h")).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b((?:lp|nn|umx)_[a-z0-9_]+)\s*\(", src)))


def test_every_declared_symbol_is_exported_and_bound():
    L = ufsm_b200.lib()
    names = header_functions()
    assert len(names) > 40
    for n in names:
        assert hasattr(L, n), "not exported: " + n
        assert n in _lib.SYMBOLS, "no ctypes signature: " + n
    for n in _lib.SYMBOLS:
        assert n in names, "bound but not declared in the header: " + n


def test_kernels_hold_their_tensor_memory_before_a_successor_may_start():
    """A kernel that lets its successor start early does so behind the barrier after its tcgen05.alloc, which waits without a limit: a successor's block that took the columns first would
    wait for this kernel, and this kernel for it."""
    csrc, seen = os.path.join(ROOT, "ufsm_b200", "csrc"), 0
    for f in sorted(os.listdir(csrc)):
        src = re.sub(r"/\*.*?\*/", "", open(os.path.join(csrc, f)).read(), flags=re.S)
        for body in re.split(r"\b__global__\b", src)[1:]:
            if "tmem_alloc(" in body and "pdl_trigger()" in body:
                at = body.index("__syncthreads()", body.index("tmem_alloc("))
                assert body.index("pdl_trigger()") > at, "%s: %s" % (f, body[:120])
                seen += 1
    assert seen == 5


def test_no_object_holds_more_than_a_form_of_the_z_marching_conv():
    """A process loads an object's kernels as a whole when it first launches one of them: all 24 instances in one made its first 3^3 conv take 10.6 ms."""
    objs = [os.path.join(ROOT, "build", f) for f in os.listdir(os.path.join(ROOT, "build")) if f.endswith(".cu.o")] if os.path.isdir(os.path.join(ROOT, "build")) else []
    if not objs or shutil.which("nm") is None:
        pytest.skip("the objects of the build are not here")
    counts = [len(re.findall(r"\bconv_mxr_k<", subprocess.run(["nm", "-C", o], stdout=subprocess.PIPE, text=True).stdout)) for o in objs]
    assert max(counts) <= 6 and sum(counts) >= 30


def test_struct_sizes_match_the_reference():
    assert C.sizeof(ufsm_b200.Shape5) == 20
    assert C.sizeof(ufsm_b200.Split) <= 128 and C.sizeof(ufsm_b200.Split) == 128   # static_assert of src/nn_lp.h:38-41
    assert C.sizeof(ufsm_b200.Gnp) == 56
    assert C.sizeof(ufsm_b200.Feather) == 120        # umx_feather_t: 2 ints, 9 pointers, 7 ints, padding, 1 pointer


def test_storage_sizes():
    L = ufsm_b200.lib()
    assert L.lp_mx8_bytes(1, 32, 64 ** 3) == 64 ** 3 * 33 and L.lp_mx4_bytes(1, 64, 96 ** 3) == 2 * 96 ** 3 * 17
    assert L.lp_mx8_bytes(2, 4, 10) == 2 * 10 * 9 and L.lp_mx4_bytes(1, 16, 10) == 10 * 9
    assert L.umx_mx_bytes32(8, 1, 1, 100) == 3300 and L.umx_mx_bytes32(4, 2, 40, 10) == 2 * 2 * 10 * 17


def test_window_plan():
    L = ufsm_b200.lib()
    w = L.umx_window_make(1024, 128, 16)
    assert (w.nper, w.npatch) == (9, 729)
    z, y, x = C.c_int(), C.c_int(), C.c_int()
    L.umx_window_origin(C.byref(w), 728, C.byref(z), C.byref(y), C.byref(x))
    assert (z.value, y.value, x.value) == (896, 896, 896)
    covered = np.zeros(1024, bool)
    for i in range(9):
        L.umx_window_origin(C.byref(w), i, C.byref(z), C.byref(y), C.byref(x))
        covered[x.value:x.value + 128] = True
    assert covered.all()
    for world in (1, 2, 3, 4, 8):
        f, c = C.c_int(), C.c_int()
        seen = []
        for r in range(world):
            L.umx_window_share(C.byref(w), r, world, C.byref(f), C.byref(c))
            assert c.value % 9 == 0                       # whole (z, y) rows
            seen += list(range(f.value, f.value + c.value))
        assert seen == list(range(729))                   # every patch once, contiguous z-slab order
    w2 = L.umx_window_make(300, 128, 16)                  # the last patch is pulled back to the edge
    L.umx_window_origin(C.byref(w2), w2.npatch - 1, C.byref(z), C.byref(y), C.byref(x))
    assert w2.nper == 3 and x.value == 300 - 128
    lo, hi = C.c_int(), C.c_int()
    L.umx_window_share(C.byref(w), 1, 8, C.byref(f), C.byref(c))
    L.umx_window_extent(C.byref(w), f.value, c.value, C.byref(lo), C.byref(hi))
    assert 0 <= lo.value < hi.value <= 1024 and (hi.value - lo.value) % 16 == 0


def test_network_sizes():
    L = ufsm_b200.lib()
    cfg = ufsm_b200.UnetCfg()
    cfg.L = 5
    for i, v in enumerate([32, 64, 128, 256, 320]):
        cfg.cw[i] = v
    cfg.nh, cfg.P, cfg.bits_first, cfg.bits_mid, cfg.bits_last = 7, 128, 8, 8, 8
    import orc
    assert L.umx_unet_nweights(C.byref(cfg)) == orc.unet_nweights(orc.unet_cfg(128, [32, 64, 128, 256, 320]))
    assert abs(L.umx_unet_flops(C.byref(cfg)) / 1e9 - 1012.8) < 0.5     # the benchmark's figure for one 128^3 patch


def test_upsample_tile_rows_are_exact():
    """the upsample finds a staged row's plane, line and place by multiplication: every row of every tile its search can return"""
    L = ufsm_b200.lib()
    buf, seen = (C.c_int * (3 * 896))(), 0
    for ux in range(1, 34):
        for uy in range(0, 34):
            for uz in range(0, 14):
                n = (uz + 1) * (uy + 1) * (ux + 1)
                ok = 2 <= ux <= 32 and 1 <= uy <= 64 // ux and 1 <= uz <= 12 and n <= 896
                assert L.umx_up2_tile_rows(uz, uy, ux, buf) == (n if ok else 0)
                if ok:
                    seen += 1
                    s, hx, hyx = np.arange(n), ux + 1, (ux + 1) * (uy + 1)
                    assert np.array_equal(np.ctypeslib.as_array(buf)[:3 * n].reshape(n, 3), np.stack([s // hyx, s % hyx // hx, s % hx], 1)), (uz, uy, ux)
    assert seen > 1000


def test_upsample_tile_is_the_cheapest():
    """the upsample's tile search skips what cannot win: the tile, and the one of equals, that a look at every tile finds (cost model of up2_tile)"""
    L = ufsm_b200.lib()
    L.umx_up2_tile.restype, L.umx_up2_tile.argtypes = None, [C.c_int] * 3 + [C.c_size_t, C.c_int, C.c_void_p]
    t = np.array([(x, y, z) for x in range(2, 33) for y in range(1, 64 // x + 1) for z in range(1, 13) if (x + 1) * (y + 1) * (z + 1) <= 896])
    x, y, z = t.T
    trips, r, out = ((x + 1) * (y + 1) * (z + 1) + 63) // 64, np.random.default_rng(4), (C.c_int * 3)()
    grids = [(1, 1, 1), (2, 3, 5), (8, 8, 8), (48, 48, 48), (54, 54, 54), (128, 128, 128)] + [tuple(int(2 ** r.uniform(0, 8)) for _ in range(3)) for _ in range(400)]
    for D, H, W in grids:
        for nbk, gn in ((1, 0), (2, 1), (int(2 ** r.uniform(0, 8)), int(r.integers(2)))):
            blocks = ((D + z) // z) * ((H + y) // y) * ((W + x) // x) * nbk
            whole, rest = blocks // 296, blocks % 296
            cost = (1000.0 + 800.0 * z + (150.0 if gn else 70.0) * trips) * (whole + np.where(rest == 0, 0.0, np.where(rest <= 148, 0.65, 1.0)))
            L.umx_up2_tile(D, H, W, nbk, gn, out)
            assert tuple(out) == tuple(int(v) for v in t[np.argmin(cost)][::-1]), (D, H, W, nbk, gn)


def test_norm_plan_keeps_a_sample_its_own():
    """the one-launch norm: what fixes the order of a sample's sums (the shares, their trips, the voxels of a trip) does not depend on the batch, every share has
    its block, and a launch has at most one block a multiprocessor and as many trips as a block can hold"""
    L = ufsm_b200.lib()
    L.umx_norm_plan.restype, L.umx_norm_plan.argtypes = None, [C.c_size_t] + [C.c_int] * 4 + [C.c_void_p]
    out, r, seen = (C.c_int * 8)(), np.random.default_rng(3), set()

    def plan(*a):
        L.umx_norm_plan(*a, out)
        return tuple(out)
    sizes = [1, 255, 256, 257, 1024, 1025, 4096, 4097, 8000, 16 ** 3, 24 ** 3, 32 ** 3, 64 ** 3, 148 * 4096, 148 * 4096 + 1, 96 ** 3] + [int(2 ** r.uniform(0, 21)) for _ in range(300)]
    for S in sizes:
        for nb in (1, 2, 3, 4, 8, 10, 74, 148, 149):
            for sms in (148, 132, 20, 600):
                one = plan(S, nb, 1, sms, 1)
                assert one[0] == (1 if S <= 4096 or min(sms // nb, 511) * 4096 >= S else 0)
                for N in (1, 2, 3, 4, 5, 7, 16, 200):
                    held, blocks, cl, ranks, per, vp, trips, most = plan(S, nb, N, sms, 1)
                    assert (held == 0) == (one[0] == 0)
                    if not held:
                        continue
                    assert (ranks, vp, trips) == (one[3], one[5], one[6]) and ranks * vp * trips >= S
                    if S <= 4096:
                        assert held == 1 and blocks == cl == ranks <= 16 and per == 1 and vp <= 256 and trips == most == 1
                        continue
                    assert cl == 1 and vp == 512 and ranks <= 511 and (ranks - 1) * vp < S
                    seen.add((held, per > 1, most > 2))
                    if held == 1:
                        assert blocks * nb * N <= sms and blocks * per >= ranks and most <= 8 and per <= 4
                        # the trips of each block, counted one by one
                        count = np.bincount(np.arange(0, S, vp) // vp % ranks % blocks, minlength=blocks)
                        assert count.max() == count[0] == most
    assert {(1, False, False), (1, False, True), (1, True, False), (1, True, True)} <= seen and any(s[0] == 2 for s in seen)


def test_zeroing_kernel_only_on_the_devices_own_memory():
    """nn_zero takes its kernel for 16-byte pieces of the current device's memory (type 2) alone; another device's (which need not be mapped), pinned (1), managed
    (3) and unregistered (0) memory go to memset"""
    L = ufsm_b200.lib()
    f = L.umx_zero_by_kernel
    f.restype, f.argtypes = C.c_int, [C.c_int, C.c_int, C.c_int, C.c_size_t, C.c_size_t]
    assert f(2, 0, 0, 4096, 64) and f(2, 3, 3, 16, 16)
    for other in [(2, 1, 0, 4096, 64), (2, 0, 1, 4096, 64), (1, 0, 0, 4096, 64), (3, 0, 0, 4096, 64), (0, -2, 0, 4096, 64), (2, 0, 0, 4104, 64), (2, 0, 0, 4096, 60), (2, 0, 0, 4096, 0)]:
        assert not f(*other), other


def test_no_cpu_fallback():
    """Without a B200 a compute entry must latch an error, not compute something."""
    import torch
    if torch.cuda.is_available():
        return
    L = ufsm_b200.lib()
    L.lp_check()
    buf = np.zeros(64, np.float32)
    out = np.zeros(128, np.uint8)
    L.lp_f32_to_mx8(buf.ctypes.data, 1, 32, 2, out.ctypes.data)
    e = L.lp_check()
    assert e and b"no CPU path" in e or b"no other path" in e
    assert not out.any()
