"""The torch binding and several Python threads: a call leaves the interpreter to the others while it is inside the library."""
import shutil
import subprocess
import sys

import pytest

from util import nvk

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
