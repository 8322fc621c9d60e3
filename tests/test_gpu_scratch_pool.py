"""The launches' scratch pool: a device that was reset, memory given back, and
another thread's capture in progress while the pool is made."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")

from ultraprecise_b200 import abi, runtime
from ultraprecise_b200 import expr as E

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# without torch: its own state would not survive the reset
RESET = r"""
import ctypes as C
from ultraprecise_b200 import abi, codec
from ultraprecise_b200 import expr as E
rt = C.CDLL("libcudart.so.12")
lib = abi.load()
b = E.derive_types(E.build([E.col(0) * E.col(1)], [E.ColType(18, 2)] * 2))
h = C.c_void_p()
qa = (abi.UpQueryAgg * 1)((abi.UP_AGG_SUM, b.roots[0]))
abi.check(lib.up_query_compile(b.nodes, b.n_nodes, b.col_types, b.n_cols, qa, 1, None, C.byref(h)), "compile")
rows, groups = 2000, 700  # a kernel that asks for more than 48 KB of shared memory
raw = codec.encode([(0, i) for i in range(rows)], 18)

def device(data):
    p = C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(len(data))) == 0
    assert rt.cudaMemcpy(p, data, C.c_size_t(len(data)), 1) == 0
    return p

def launch():
    col = abi.UpColumn(device(raw), None, None, 0, None, 18, 2, 8, 0)
    gid = device(b"".join((i % groups).to_bytes(4, "little") for i in range(rows)))
    out = device(bytes(133 * groups))
    abi.check(lib.up_query_launch(h, (abi.UpColumn * 2)(col, col), 2, rows, gid, groups, (C.c_void_p * 1)(out), None, None), "launch")
    got = C.create_string_buffer(133 * groups)
    assert rt.cudaDeviceSynchronize() == 0 and rt.cudaMemcpy(got, out, C.c_size_t(133 * groups), 2) == 0
    for g in range(groups):
        assert int.from_bytes(got.raw[133 * g + 5:133 * (g + 1)], "little") == sum(i * i for i in range(g, rows, groups))

launch(); launch()
assert rt.cudaDeviceReset() == 0
launch(); launch()
print("same after the reset")
"""


def test_launches_after_a_device_reset():
    env = dict(os.environ, PYTHONPATH=ROOT)
    env["LD_LIBRARY_PATH"] = "/usr/local/cuda/lib64:" + env.get("LD_LIBRARY_PATH", "")
    r = subprocess.run([sys.executable, "-c", RESET], capture_output=True, text=True, timeout=300, cwd=ROOT, env=env)
    assert r.returncode == 0 and "same after the reset" in r.stdout, r.stdout + r.stderr


def _sum_module():
    q = runtime.compile_query([E.col(0) * E.col(1)], [(abi.UP_AGG_SUM, 0)], [E.ColType(18, 2)] * 2)
    cols = [runtime.DeviceColumn(runtime.gen_digits(5000, 18, k), 18, 2) for k in range(2)]
    return q, cols


def test_unused_scratch_is_given_back():
    groups = 600_000  # 19 MB of limb sums and more
    q, cols = _sum_module()
    gid = (torch.arange(5000, device="cuda") % groups).to(torch.int32)
    outs = [torch.zeros(groups * 133, dtype=torch.uint8, device="cuda")]
    q.launch(cols, gid, groups, outs=outs)
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    abi.load().up_module_cache_size(1)
    assert torch.cuda.mem_get_info()[0] >= held + (8 << 20)
    q.launch(cols, gid, groups, outs=outs)  # and allocated anew
    torch.cuda.synchronize()


# a process of its own, in which no launch has made the pool yet
CAPTURE = r"""
import threading, torch
from ultraprecise_b200 import abi, runtime
from ultraprecise_b200 import expr as E
q = runtime.compile_query([E.col(0) * E.col(1)], [(abi.UP_AGG_SUM, 0)], [E.ColType(18, 2)] * 2)
cols = [runtime.DeviceColumn(runtime.gen_digits(1000, 18, k), 18, 2) for k in range(2)]
gid = torch.zeros(1000, dtype=torch.int32, device="cuda")
outs = [[torch.zeros(133, dtype=torch.uint8, device="cuda")] for _ in range(2)]
x, side, graph, failed = torch.zeros(10, device="cuda"), torch.cuda.Stream(), torch.cuda.CUDAGraph(), []
torch.cuda.synchronize()

def other():
    try:
        q.launch(cols, gid, 1, outs=outs[0], stream=side)
    except Exception as e:
        failed.append(str(e))

with torch.cuda.graph(graph, capture_error_mode="thread_local"):
    x.add_(1)
    t = threading.Thread(target=other)
    t.start()
    t.join()
    x.add_(1)
graph.replay()
q.launch(cols, gid, 1, outs=outs[1])
torch.cuda.synchronize()
assert not failed and float(x[0]) == 2.0 and torch.equal(outs[0][0], outs[1][0])
print("both done")
"""


def test_first_launch_beside_a_capture():
    r = subprocess.run([sys.executable, "-c", CAPTURE], capture_output=True, text=True, timeout=300, cwd=ROOT,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and "both done" in r.stdout, r.stdout + r.stderr
