"""GPU: the debug flavour of the library on the forms that a table with rows of period 64 and short sums do not reach: expanded tables of
bytes with 256 rows, and the reference's order of additions with one to four pixels per lane and several units per CTA.  Every access
stays in its bounds, the outputs have the checker's bits, a wait that runs out is reported as status 3, and with the limit back the
same call is right again."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = r"""
import ctypes as C, sys
import numpy as np, torch
sys.path.insert(0, %r)
import tf_approximate_b200 as ax
from tf_approximate_b200 import _lib
from oracle import oracle as O
L = _lib.load()
rec = (C.c_uint32 * 4)()
assert L.axc_debug_bounds_record(0, rec) == 0, "not the debug flavour"
rng = np.random.Generator(np.random.PCG64(77))
a = np.arange(256)
# distances 0 .. 156 from the exact product, without a period
lut = np.minimum(a[:, None] * a[None, :] + rng.integers(0, 157, (256, 256)), 65535).astype(np.uint16).reshape(-1)
byte = ax.Table(array=lut)
noisy_lut = ax.noisy_table(9)
noisy = ax.Table(array=noisy_lut)

def operands(n, h, w, c, k, co, lo=-1.0):
    x = rng.uniform(lo, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (k, k, c, co)).astype(np.float32)
    return x, f, (lo, 1.0, float(f.min()), float(f.max())), torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()

def violations():
    torch.cuda.synchronize()
    assert L.axc_debug_bounds_record(0, rec) == 0
    print("violations", rec[0], "site", rec[1], "value", rec[2] | (rec[3] << 32))
    assert rec[0] == 0
""" % ROOT

BYTES = HEAD + r"""
seen = set()
for n, h, w, c, k, co, s, pad in [(1, 7, 7, 512, 1, 512, 1, "SAME"), (1, 64, 64, 3, 7, 64, 2, "SAME"), (3, 27, 31, 150, 1, 45, 1, "VALID"), (8, 56, 56, 16, 1, 24, 1, "SAME"),
                                  (40, 14, 14, 16, 3, 8, 1, "SAME"), (12, 7, 7, 8, 1, 2048, 1, "SAME"), (12, 14, 14, 8, 1, 512, 1, "SAME"), (2, 28, 28, 512, 3, 8, 1, "SAME"),
                                  (20, 28, 28, 32, 3, 8, 1, "SAME"), (12, 14, 14, 8, 1, 1024, 1, "SAME"), (4, 200, 200, 8, 1, 8, 1, "SAME"), (8, 14, 14, 128, 3, 256, 1, "SAME"),
                                  (40, 97, 97, 20, 1, 8, 1, "SAME")]:
    x, f, mm, xd, fd = operands(n, h, w, c, k, co)
    d = O.desc(n, h, w, c, k, k, co, (s, s), (1, 1), pad)
    ref = O.conv2d(d, lut, x, f, *mm, want=("out_exact",))["out_exact"]
    y, dbg = ax.approx_conv2d_with_min_max_vars(xd, fd, *mm, [1, s, s, 1], 8, byte, pad, debug=True)
    r = dbg["plan"]["route"]
    assert r["kernels"] == "expanded" and dbg["plan"]["status"] == 0
    seen.add((r["tile"], r["splits"] > 1, r["tables_in_global_memory"]))
    assert np.array_equal(y.cpu().numpy().view(np.uint32), ref.view(np.uint32)), (n, h, w, c, k, co)
    z = ax.approx_conv2d_with_min_max_vars(xd, fd, *mm, [1, s, s, 1], 8, byte, pad)
    assert torch.equal(z.view(torch.int32), y.view(torch.int32))
    p, q = rng.integers(0, 256, x.shape).astype(np.uint8), rng.integers(0, 256, f.shape).astype(np.uint8)
    got, _, _ = ax.ax_conv2d(torch.from_numpy(p).cuda(), torch.from_numpy(q).cuda(), -1.0, 2.0, -0.5, 0.5, [1, s, s, 1], pad, table=byte, ax_tune=False)
    assert np.array_equal(got.cpu().numpy(), O.qconv2d(d, lut, p, q, O.quantized_zero_point(-1.0, 2.0), O.quantized_zero_point(-0.5, 0.5))), (n, h, w, c, k, co)
print(sorted(seen))
own = {(256, True, False), (512, False, False), (1024, False, False), (1024, True, False), (2048, False, False), (2048, True, False)}
assert seen >= own | {(1024, False, True), (1024, True, True), (2048, False, True)}, seen
violations()
"""

REFERENCE = HEAD + r"""
# tiles of one to four pixels per lane (512 pixels each); the last has more units than CTAs
tiles = []
for n, h, w, c, k, co, s in [(1, 7, 7, 512, 3, 128, 1), (2, 40, 41, 3, 11, 24, 1), (3, 56, 55, 40, 3, 45, 1), (4, 56, 57, 96, 3, 72, 1), (9, 130, 129, 20, 5, 8, 1),
                             (1, 130, 129, 20, 5, 112, 1), (30, 130, 129, 29, 3, 8, 1)]:
    x, f, mm, xd, fd = operands(n, h, w, c, k, co, 0.0)
    ref = O.conv2d(O.desc(n, h, w, c, k, k, co, (s, s)), noisy_lut, x, f, *mm, want=("out_ref",))["out_ref"]
    y, dbg = ax.approx_conv2d_with_min_max_vars(xd, fd, *mm, [1, s, s, 1], 8, noisy, "SAME", accumulate="reference", debug=True)
    r = dbg["plan"]["route"]
    assert r["kernels"] == "expanded" and dbg["plan"]["status"] == 0
    m = n * -(-h // s) * -(-w // s)
    tiles.append((-(-r["tile"] // 512), -(-m // r["tile"]) * -(-co // 8)))
    assert np.array_equal(y.cpu().numpy().view(np.uint32), ref.view(np.uint32)), (n, h, w, c, k, co)
print(tiles)
assert {p for p, _ in tiles} == {1, 2, 3, 4} and max(u for _, u in tiles) > 148
violations()
"""

WAITS = HEAD + r"""
for table, values, opts, n, h, w, c, k, co, in_global in ((byte, lut, {}, 4, 56, 57, 32, 3, 64, True), (byte, lut, {}, 1, 7, 7, 512, 1, 512, False), (byte, lut, {}, 12, 14, 14, 8, 1, 1024, False),
                                                          (noisy, noisy_lut, {"accumulate": "reference"}, 2, 20, 20, 64, 3, 64, False)):
    x, f, mm, xd, fd = operands(n, h, w, c, k, co)
    key = "out_ref" if opts else "out_exact"
    ref = O.conv2d(O.desc(n, h, w, c, k, k, co), values, x, f, *mm, want=(key,))[key]
    for expand, convolution in ((0, -1), (-1, 0), (0, 0), (-1, -1)):
        assert L.axc_debug_wait_polls(0, expand, convolution) == 0
        y, dbg = ax.approx_conv2d_with_min_max_vars(xd, fd, *mm, [1, 1, 1, 1], 8, table, "SAME", debug=True, **opts)
        torch.cuda.synchronize()
        assert dbg["plan"]["route"]["kernels"] == "expanded" and dbg["plan"]["route"]["tables_in_global_memory"] == in_global, dbg["plan"]["route"]
        gave_up = convolution == 0 or (expand == 0 and in_global)
        assert dbg["plan"]["status"] == (3 if gave_up else 0), (n, h, c, expand, convolution, dbg["plan"])
        if not gave_up:
            assert np.array_equal(y.cpu().numpy().view(np.uint32), ref.view(np.uint32))
violations()
"""


@pytest.mark.parametrize("child", [BYTES, REFERENCE, WAITS], ids=["bytes", "reference", "waits"])
def test_checked_flavour(built, child):
    r = subprocess.run([sys.executable, "-c", child], env=dict(os.environ, AXC_LIBRARY_FLAVOUR="check"), capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert "violations 0" in r.stdout
