"""The torch binding and several Python threads: a call leaves the interpreter to the others while it is inside the library, and
first calls from several threads at once, each on its own stream, give what one thread gets."""
import os
import shutil
import subprocess
import sys

import pytest

from util import ROOT, nvk

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# A library with the same entry points.  nvk_linear stays inside until another thread lets it go, two seconds at most.
STAND_IN = """
#include <time.h>
static volatile int inside = 0, go = 0;
int nvk_test_inside(void) { return inside; }
void nvk_test_go(void) { go = 1; }
int nvk_linear(void) {
    inside = 1;
    for (int i = 0; i < 2000 && !go; ++i) { struct timespec t = {0, 1000000}; nanosleep(&t, 0); }
    return go ? 0 : 2;
}
const char* nvk_last_error(void) { return "nobody let the call go"; }
"""

CALLER = """
import ctypes, importlib.util, sys, threading, time
import torch
spec = importlib.util.spec_from_file_location("nvk_torch", sys.argv[1] + "/nvk_torch.so")
binding = importlib.util.module_from_spec(spec)
spec.loader.exec_module(binding)
lib = ctypes.CDLL(sys.argv[1] + "/libnvk.so")
x = torch.zeros(128, 128, device="cuda", dtype=torch.bfloat16)
failed = []
def call():
    try:
        binding.linear(x, x, x)
    except RuntimeError as e:
        failed.append(str(e))
t = threading.Thread(target=call)
t.start()
while not lib.nvk_test_inside():
    time.sleep(0.001)
lib.nvk_test_go()
t.join()
assert not failed, failed
"""


def test_a_call_does_not_hold_the_interpreter(tmp_path):
    others = [n for n in nvk().EXPORTED_SYMBOLS if n not in ("nvk_linear", "nvk_last_error")]
    (tmp_path / "stand_in.c").write_text(STAND_IN + "".join(f"int {n}(void) {{ return 0; }}\n" for n in others))
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "libnvk.so"), str(tmp_path / "stand_in.c")], check=True)
    shutil.copy(nvk().BINDING_PATH, tmp_path / "nvk_torch.so")   # finds the library beside it
    subprocess.run([sys.executable, "-c", CALLER, str(tmp_path)], check=True, timeout=120)

THREADS = """
import threading
import torch
from util import nvk, to_dev, workloads
bf, lib = torch.bfloat16, nvk()
d = workloads().make_decode_workload(5, 8, 2, 128, 256, 1, 3000, seed=1)
p = workloads().make_prefill_workload([300, 70], [256, 0], 8, 2, 128, 256, seed=2)
dev = {n: to_dev(d[n], bf) for n in ("q", "k_cache", "v_cache")}
pre = {n: to_dev(p[n], bf) for n in ("q", "k_cache", "v_cache")}
ctx, bt, cu_q, cu_k, pt = (to_dev(a) for a in (d["context_lens"], d["block_tables"], p["cu_q"], p["cu_k"], p["block_tables"]))
x, w = torch.randn(200, 512, device="cuda").to(bf), torch.randn(768, 512, device="cuda").to(bf)
torch.cuda.synchronize()
def work():
    ws = torch.empty(lib.decode_attention_workspace_bytes(5, 8, 2, 128, bt.shape[1], 256), dtype=torch.uint8, device="cuda")
    o = [torch.empty_like(dev["q"]), torch.empty_like(pre["q"]), torch.empty(200, 768, device="cuda", dtype=bf)]
    for _ in range(30):
        lib.launch_decode_attention_paged(dev["q"], dev["k_cache"], dev["v_cache"], ctx, bt, 2, 128, 256, d["scale"], o[0], ws)
        lib.launch_prefill_attention_paged(pre["q"], cu_q, pre["k_cache"], pre["v_cache"], cu_k, pt, 2, 128, 256, p["scale"], o[1])
        lib.linear(x, w, o[2])
    return o
got = [None] * 4
start = threading.Barrier(4)
def thread(i):
    with torch.cuda.stream(torch.cuda.Stream()):
        start.wait()
        got[i] = work()
        torch.cuda.current_stream().synchronize()
ts = [threading.Thread(target=thread, args=(i,)) for i in range(4)]
[t.start() for t in ts]
[t.join() for t in ts]
want = work()
torch.cuda.synchronize()
assert lib.prefill_status() == 0 and lib.gemm_status() == 0
for o in got:
    assert all(torch.equal(a, b) for a, b in zip(o, want))
"""


def test_first_calls_from_several_threads():
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.join(ROOT, "tests"), ROOT]))
    subprocess.run([sys.executable, "-c", THREADS], check=True, timeout=300, env=env, cwd=ROOT)
